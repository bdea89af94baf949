"""Host build of the BN254 scalar decomposition (impeller_b200/csrc/glv.cuh).

The header is written for host and device alike; here g++ compiles it for the
CPU and every split is checked against Python's integers: the halves give the
scalar back modulo r, and stay below the 2^127 that the digit windows rely on.
"""
import ctypes
import os
import random
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "impeller_b200", "csrc")
R = 21888242871839275222246405745257275088548364400416034343698204186575808495617
P = 21888242871839275222246405745257275088696311157297823662689037894645226208583
LAMBDA = 0xB3C4D79D41A917585BFC41088D8DAAA78B17EA66B99C90DD
BETA = 0x59E26BCEA0D48BACD4F263F1ACDB5C4F5763473177FFFFFE

SHIM = r"""
#include "glv.cuh"
extern "C" void glv_split(const uint32_t *k, uint32_t *k1, uint32_t *k2, uint32_t *neg) {
    uint32_t a[8], b[4], c[4];
    for (int i = 0; i < 8; i++) a[i] = k[i];
    ec::glv::split(a, b, neg[0], c, neg[1]);
    for (int i = 0; i < 4; i++) k1[i] = b[i], k2[i] = c[i];
}
extern "C" uint32_t glv_windows(uint32_t c) { return ec::glv::windows(c); }
extern "C" void glv_beta(uint32_t *b) {
    const uint32_t v[8] = GLV_BETA;
    for (int i = 0; i < 8; i++) b[i] = v[i];
}
"""


@pytest.fixture(scope="module")
def lib():
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tempfile.mkdtemp(prefix="glv_")
    src, so = os.path.join(d, "shim.cpp"), os.path.join(d, "libglv.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, src, "-o", so], check=True)
    return ctypes.CDLL(so)


def split(lib, k):
    w = (ctypes.c_uint32 * 8)(*[(k >> (32 * i)) & 0xFFFFFFFF for i in range(8)])
    a, b, neg = (ctypes.c_uint32 * 4)(), (ctypes.c_uint32 * 4)(), (ctypes.c_uint32 * 2)()
    lib.glv_split(w, a, b, neg)
    value = lambda x: sum(int(v) << (32 * i) for i, v in enumerate(x))  # noqa: E731
    return (-1) ** neg[0] * value(a), (-1) ** neg[1] * value(b)


def test_constants(lib):
    assert (LAMBDA * LAMBDA + LAMBDA + 1) % R == 0 and pow(BETA, 3, P) == 1 and BETA != 1
    b = (ctypes.c_uint32 * 8)()
    lib.glv_beta(b)
    assert sum(int(v) << (32 * i) for i, v in enumerate(b)) == (BETA << 256) % P


def test_split_gives_the_scalar_back(lib):
    rng = random.Random(11)
    ks = [0, 1, 2, R - 1, R - 2, R // 2, R // 2 + 1, LAMBDA, R - LAMBDA, LAMBDA + 1, (1 << 253) - 1]
    ks += [1 << e for e in range(254) if 1 << e < R]
    # the corners of the lattice cell, where the halves are largest
    a, n1, n2 = 0x89D3256894D213E3, 0x6F4D8248EEB859FC8211BBEB7D4F1128, 0x6F4D8248EEB859FD0BE4E1541221250B
    for i in range(200):
        u, v = rng.randrange(1 << 64) * 2 + 1, rng.randrange(1 << 127) * 2 + 1
        half = ((u * a + v * n2) // 2 + LAMBDA * ((v * a - u * n1) // 2)) % R
        ks += [half, (half + 1) % R, (half - 1) % R]
    ks += [rng.randrange(R) for _ in range(5000)]
    for k in ks:
        k1, k2 = split(lib, k)
        assert (k1 + k2 * LAMBDA - k) % R == 0
        assert abs(k1) < 1 << 127 and abs(k2) < 1 << 127


@pytest.mark.parametrize("c", range(3, 32))
def test_windows_hold_a_127_bit_half(lib, c):
    w = lib.glv_windows(c)
    top = ((1 << 127) - 1) >> (c * (w - 1))
    assert top + 1 <= 1 << (c - 1)

"""The rules of csrc/launch.cuh, checked in the sources: what a kernel has to do
that is set up while the kernel before it still runs.  A kernel that breaks
them races with other work of its stream, so nothing here runs on a GPU.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "impeller_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"//[^\n]*", "", text)
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def kernels():
    """name -> (parameter list, body) of every __global__ function."""
    found = {}
    for f in FILES:
        text = source(f)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            params, start = text[m.end():at - 1], text.index("{", at)
            depth, end = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            found[m.group(1)] = (params, text[start + 1:end - 1])
    return found


KERNELS = kernels()


def chained():
    """Kernels launched so that they may be set up beside their predecessor."""
    names = set()
    for f in FILES:
        text = source(f)
        text = re.sub(r"#define (?:[^\n]*\\\n)*[^\n]*", "", text)
        for m in re.finditer(r"\b(?:CURVE_LAUNCH|DIGIT_LAUNCH|launch_next|launch_cluster)\s*\(([^;]*);", text):
            names |= set(re.findall(r"\bk_\w+", m.group(1)))
        # a kernel launched through a local name
        for m in re.finditer(r"auto\s+kern\s*=\s*(k_\w+)", text):
            names.add(m.group(1))
    return sorted(n for n in names if n in KERNELS)


def test_kernels_and_launches_are_found():
    assert {"k_accumulate", "k_ntt_pass", "k_ntt_small", "k_small_sort", "k_affine_pairs", "k_final"} <= set(chained())
    assert {"k_precompute", "k_combine", "k_omegas"} <= set(KERNELS)


@pytest.mark.parametrize("name", chained())
def test_chained_kernels_wait_for_their_predecessor_first(name):
    body = KERNELS[name][1].strip()
    assert re.match(r"(?:impeller::)?grid_wait\(\);", body), f"{name} does not start with grid_wait()"


# inputs that no kernel of a chain writes
READ_ONLY = {"descs", "points"}


@pytest.mark.parametrize("name", chained())
def test_chained_kernels_read_with_plain_loads(name):
    params, body = KERNELS[name]
    assert "__ldg" not in body and "ld.global.nc" not in body
    restrict = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s*(\w+)", params))
    assert restrict <= READ_ONLY, f"{name}: {sorted(restrict - READ_ONLY)}"


@pytest.mark.parametrize("name", ["msm_kernels.cuh", "affine_pairs.cuh", "lane_pairs.cuh", "bn254.cuh", "ntt.cu"])
def test_helpers_of_chained_kernels_read_with_plain_loads(name):
    text = source(name)
    assert "__ldg" not in text
    assert set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s*(\w+)", text)) <= READ_ONLY

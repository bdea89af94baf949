"""Plans of MSMs, built on the CPU: a small C++ program links the library, lays
plans out as its callers do, and the sizes and index ranges are checked.  No
GPU is needed (the layout assumes 148 SMs where there is no device).
"""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(HERE, "..", "impeller_b200")
CUDA = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))

SOURCE = r"""
#include <unistd.h>

#include <cstdio>
#include <cstring>
#include "engine.h"
#include "impeller_msm.h"
using namespace impeller;

// A context of len points as impeller_ctx_create makes it, without a device.
struct Context {
    impeller_ctx ctx;
    explicit Context(u64 len, u32 curve = CURVE_BN254) {
        ctx.len = len;
        ctx.curve = curve;
    }
    // what impeller_ctx_precompute changes
    void add_tables(u32 c) {
        const u64 have = ctx.tables ? ctx.tables_points : ctx.len;
        ctx.tables = reinterpret_cast<u32 *>(16);
        ctx.tables_points = have + (u64)digit_windows(c, ctx.curve) * ctx.len;
        ctx.sets.emplace_back(c, (u32)have);
    }
};

static int mixed_batch() {
    // a plain job, then tables, then a job on the tables and a plain one: what
    // a server holds when tables are added between its jobs' submissions
    Context k(5000);
    const MsmShape before = ctx_shape(&k.ctx, 3000, 13);
    k.add_tables(16);
    const MsmShape table = ctx_shape(&k.ctx, 5000, 16), after = ctx_shape(&k.ctx, 2000, 13);
    Plan p, q, r;
    const bool one = Plan::build(p, 0, {before, table}), two = Plan::build(q, 0, {before, after});
    const bool all = Plan::build(r, 0, {after, table, before});
    const u64 past_table = table.table_base + (u64)(digit_windows(16) - 1) * table.table_stride + table.n;
    std::printf("built %d %d %d\n", one, two, all);
    std::printf("images_past_points %d %d %d\n", p.phi_base >= past_table, q.phi_base >= 3000, r.phi_base >= past_table);
    std::printf("images %u %u %u\n", p.phi_points, q.phi_points, r.phi_points);
    return 0;
}

static int largest() {
    // sizes whose whole scalars' digits fit 32 bits and the halves' do not
    Context k(280000000);
    Plan p;
    const u32 n = (u32)k.ctx.len, c = ctx_window(&k.ctx, n);
    const bool one = Plan::build(p, 0, {ctx_shape(&k.ctx, n, c)});
    std::printf("single %d %u\n", one, p.phi_points);
    // the same of many MSMs together, through the call that makes a batch (it
    // gets as far as the device)
    if (!access("/dev/nvidiactl", F_OK)) {
        std::printf("batch skipped\n");
        return 0;
    }
    Context m(1 << 24);
    std::vector<uint64_t> sizes(16, 1 << 24);
    impeller_batch *b = nullptr;
    const cudaError_t e = impeller_batch_create(&b, &m.ctx, sizes.data(), nullptr, (u32)sizes.size(), 0);
    std::printf("batch %s\n", e == cudaErrorInvalidValue ? impeller_last_error() : "laid out");
    return 0;
}

static int refused() {
    // windows whose buckets do not fit are refused whether or not scalars are split
    Context k(1 << 16);
    for (u32 c : {28u, 29u, 30u, 31u}) {
        Plan p;
        const bool ok = Plan::build(p, 0, {ctx_shape(&k.ctx, 1000, c)});
        std::printf("c%u %d\n", c, ok);
    }
    return 0;
}

static int runs() {
    // a drop-in call sizes its buffer for its largest run; the last run has
    // fewer MSMs, and a streamed one fewer points
    u32 checked = 0, larger = 0, refused = 0, over = 0;
    for (u32 curve : {(u32)CURVE_BN254, (u32)CURVE_BLS12381})
        for (u32 c : {4u, 8u, 11u, 12u, 14u, 16u, 18u, 19u, 20u, 22u})
            for (u32 kind = 0; kind < 3; kind++)
                for (u32 n : {1u, 300u, 5000u, 100003u, 1000000u, 1u << 21})
                    for (u32 msms : {2u, 3u, 5u, 7u, 16u, 64u}) {
                        if ((u64)n * msms > 8000000) continue;
                        MsmShape s{n, c, kind == 0 ? 0 : kind == 1 ? 4u : 1u, n, 0, curve};
                        if (kind == 0) s.split = curve == CURVE_BN254;
                        RunSizes r;
                        Plan full;
                        if (!Plan::build(full, 0, std::vector<MsmShape>(msms, s)) || !run_sizes(0, s, msms, r)) continue;
                        for (u32 k = 1; k <= msms; k = k < 8 ? k + 1 : k * 5 / 4)
                            for (u32 m : {n, n - n / 10, n / 3 + 1, 1u}) {
                                Plan p;
                                MsmShape t = s;
                                t.n = m;
                                checked++;
                                if (!Plan::build_within(p, 0, std::vector<MsmShape>(k, t), r.scratch)) refused++;
                                else if (p.scratch_bytes() > r.scratch || p.image_bytes() > r.image) over++;
                                Plan q;
                                Plan::build(q, 0, std::vector<MsmShape>(k, t));
                                larger += q.scratch_bytes() > full.scratch_bytes() || q.image_bytes() > full.image_bytes();
                            }
                    }
    std::printf("checked %u\nlarger %u\nrefused %u\nover %u\n", checked, larger, refused, over);
    return 0;
}

int main(int argc, char **argv) {
    if (argc > 1 && !std::strcmp(argv[1], "runs")) return runs();
    if (argc > 1 && !std::strcmp(argv[1], "largest")) return largest();
    if (argc > 1 && !std::strcmp(argv[1], "refused")) return refused();
    if (argc > 1 && !std::strcmp(argv[1], "mixed_batch")) return mixed_batch();
    return 2;
}
"""


@pytest.fixture(scope="module")
def plans():
    from impeller_b200 import build
    gxx = shutil.which("g++")
    if gxx is None or not os.path.isdir(os.path.join(CUDA, "include")):
        pytest.skip("g++ or the CUDA headers are not available")
    build.build()
    d = tempfile.mkdtemp(prefix="plans_")
    src, exe = os.path.join(d, "plans.cpp"), os.path.join(d, "plans")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(HERE, "..", "include"),
                    "-I", os.path.join(CUDA, "include"), src,
                    "-o", exe, build.LIB, "-Wl,-rpath," + os.path.abspath(PKG), "-lpthread"], check=True)

    def run(what):
        r = subprocess.run([exe, what], capture_output=True, text=True, timeout=600, check=True)
        return dict(line.split(" ", 1) for line in r.stdout.splitlines())
    return run


def test_images_lie_past_every_point_of_a_batch(plans):
    """Virtual indices of endomorphism images must not meet real ones, whatever
    the context held when a job's shape was made, and no such mix is refused."""
    r = plans("mixed_batch")
    assert r["built"] == "1 1 1"
    assert r["images_past_points"] == "1 1 1"
    assert r["images"] == "3000 3000 3000"


def test_sizes_that_fit_with_whole_scalars_are_not_refused(plans):
    r = plans("largest")
    assert r["single"] == "1 0"
    assert r["batch"] in ("laid out", "skipped")


def test_windows_with_too_many_buckets_are_refused(plans):
    # 2^31 buckets of whole scalars: from window 29 on (9 windows of 2^28)
    assert plans("refused") == {"c28": "1", "c29": "0", "c30": "0", "c31": "0"}


def test_every_run_of_a_drop_in_call_fits_its_buffer(plans):
    r = plans("runs")
    assert int(r["checked"]) > 5000
    assert int(r["larger"]) > 0  # smaller runs that need more than the largest: the case in question
    assert r["refused"] == "0" and r["over"] == "0"

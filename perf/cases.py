"""What this framework is timed on: multi-scalar multiplications on both curves,
alone, batched and through the drop-in host call, the window tables, and the
number-theoretic transforms.

A case names a kind of call and its sizes.  Every output is whole numbers
(canonical affine points or field elements in Montgomery form as 32-bit
words), so two correct implementations give the same bytes, and no `exact`
in floating point exists.
"""
import math

import numpy as np
import torch

from impeller_b200 import msm as M
from impeller_b200 import ntt as NT

CURVES = {"bn254": M.BN254, "bls12381": M.BLS12381}
FIELDS = {"bn254_fr": NT.BN254_FR, "bls12381_fr": NT.BLS12381_FR}
UNIFORM, SKEWED = 0, 1  # scalars: uniform in the field; witness-like (many 0, 1 and small values)


def listed():
    return [
        # the smallest resident MSM a prover makes (a lookup or permutation
        # remainder): launches and the chain of dependent additions
        {"name": "msm_small", "kind": "msm", "curve": "bn254", "n": 1000, "tables": True, "dist": UNIFORM},
        # an odd size on a plain resident SRS (no window tables)
        {"name": "msm_plain_ragged", "kind": "msm", "curve": "bn254", "n": 100003, "tables": False, "dist": UNIFORM},
        # an ordinary commitment: a polynomial of a mid-size circuit, window tables resident
        {"name": "msm_mid", "kind": "msm", "curve": "bn254", "n": 1 << 18, "tables": True, "dist": UNIFORM},
        # a witness column: half of the scalars are 0, 1 or small
        {"name": "msm_skewed", "kind": "msm", "curve": "bn254", "n": 1 << 20, "tables": True, "dist": SKEWED},
        # the headline: 2^22 points, window tables resident
        {"name": "msm_large", "kind": "msm", "curve": "bn254", "n": 1 << 22, "tables": True, "dist": UNIFORM},
        # the second curve (381-bit base field)
        {"name": "msm_bls12381", "kind": "msm", "curve": "bls12381", "n": 1 << 20, "tables": True, "dist": UNIFORM},
        # a proof's commitments in one plan: 64 MSMs of uneven sizes, CUDA graph
        {"name": "batch", "kind": "batch", "curve": "bn254", "count": 64, "log2_min": 10, "log2_max": 20, "graph": True},
        # the drop-in call: host points and scalars uploaded each time
        {"name": "drop_in", "kind": "drop_in", "curve": "bn254", "n": 1 << 22},
        # window tables for the drop-in call, host points in, host tables out
        {"name": "precompute", "kind": "precompute", "curve": "bn254", "n": 1 << 17, "window": 13, "target": 4},
        # the smallest transform: one tile
        {"name": "ntt_small", "kind": "ntt", "field": "bn254_fr", "log_n": 10, "recompute": False},
        # the benchmark transform with a twiddle table
        {"name": "ntt_large", "kind": "ntt", "field": "bn254_fr", "log_n": 24, "recompute": False},
        # a coset extension without a twiddle table: powers of the shift, then
        # the transform with recomputed twiddles, on the other curve's field
        {"name": "ntt_coset", "kind": "coset", "field": "bls12381_fr", "log_n": 20},
    ]


def draw(rng):
    kind = rng.choice(["msm", "msm", "msm", "batch", "drop_in", "precompute", "ntt", "coset"])
    curve = rng.choice(["bn254", "bn254", "bls12381"])
    if kind == "msm":
        n = int(2 ** rng.uniform(10, 22 if curve == "bn254" else 20))
        return {"kind": kind, "curve": curve, "n": n, "tables": rng.random() < 0.6,
                "dist": SKEWED if rng.random() < 0.3 else UNIFORM}
    if kind == "batch":
        lo = rng.randint(10, 14)
        return {"kind": kind, "curve": curve, "count": rng.randint(2, 48 if curve == "bn254" else 16),
                "log2_min": lo, "log2_max": rng.randint(lo + 1, 19), "graph": rng.random() < 0.7}
    if kind == "drop_in":
        return {"kind": kind, "curve": curve, "n": int(2 ** rng.uniform(10, 22 if curve == "bn254" else 20))}
    if kind == "precompute":
        return {"kind": kind, "curve": curve, "n": int(2 ** rng.uniform(8, 16)), "window": rng.choice([13, 16]),
                "target": rng.choice([4, 8])}
    field = rng.choice(sorted(FIELDS))
    if kind == "ntt":
        return {"kind": kind, "field": field, "log_n": rng.randint(1, 23), "recompute": rng.random() < 0.4}
    return {"kind": kind, "field": field, "log_n": rng.randint(4, 22)}


def _msm_sizes(case):
    """Sizes of a batch: log-uniform between the bounds, the same for every seed."""
    r = np.random.RandomState(case["count"] * 64 + case["log2_max"])
    return [int(round(2 ** r.uniform(case["log2_min"], case["log2_max"]))) for _ in range(case["count"])]


def _pinned(t):
    """A pinned host copy of a device tensor, as uint32 words."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy().view(np.uint32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("ntt", "coset"):
        return _prepare_ntt(case, seed)
    curve = CURVES[case["curve"]]
    st = {"kind": kind}
    if kind == "msm":
        n = case["n"]
        ctx = M.MsmContext(M.gen_points_device(n, seed=seed, curve=curve), curve=curve)
        if case["tables"]:
            c = M.table_window(n)
            if c:
                ctx.precompute(c)
        st["ctx"] = ctx
        st["scalars"] = M.gen_scalars_device(n, seed=seed, dist=case["dist"], curve=curve)
        st["out"] = torch.empty(ctx.pw, dtype=torch.int32, device="cuda")
    elif kind == "batch":
        sizes = _msm_sizes(case)
        ctx = M.MsmContext(M.gen_points_device(max(sizes), seed=seed, curve=curve), curve=curve)
        for c in sorted({M.table_window(s) for s in sizes} - {0}):
            ctx.precompute(c)
        st["ctx"] = ctx
        st["scalars"] = [M.gen_scalars_device(s, seed=seed, stream_id=1000 + i, curve=curve)
                         for i, s in enumerate(sizes)]
        st["batch"] = ctx.batch(sizes, graph=case["graph"])
        st["out"] = torch.empty((len(sizes), ctx.pw), dtype=torch.int32, device="cuda")
    elif kind == "drop_in":
        n = case["n"]
        c = M.default_window(n, curve)
        cfg = M.MsmConfig(window_size=c, target_window=M.window_count(c, curve), curve=curve)
        st["op"] = M.MSM(cfg)
        st["buffer"], st["keep"] = M.alloc_gpu_buffer(st["op"].get_buffer_size(n)[0])
        st["points"] = _pinned(M.gen_points_device(n, seed=seed, curve=curve))
        st["scalars"] = _pinned(M.gen_scalars_device(n, seed=seed, curve=curve))
    elif kind == "precompute":
        n = case["n"]
        cfg = M.MsmConfig(window_size=case["window"], target_window=case["target"], curve=curve)
        st["op"] = M.MSMPrecompute(cfg).get_fn()
        st["n"] = n
        points = M.to_host(M.gen_points_device(n, seed=seed, curve=curve)).reshape(n, -1)
        st["tables"] = [points] + [np.zeros_like(points) for _ in range(cfg.get_precompute() - 1)]
    else:
        raise ValueError(kind)
    return st


def _prepare_ntt(case, seed):
    field, log_n = FIELDS[case["field"]], case["log_n"]
    n = 1 << log_n
    curve = M.BLS12381 if field == NT.BLS12381_FR else M.BN254
    st = {"kind": case["kind"], "x": M.gen_scalars_device(n, seed=seed, stream_id=11, curve=curve)}
    unit = NT.to_mont_limbs(NT.root_of_unity(log_n, field), field)
    if case["kind"] == "coset" or case["recompute"]:
        g = NT.GenPqOmegas(field)
        pq = np.zeros((g.get_pq_len(log_n), NT.WORDS), np.uint32)
        om = np.zeros((32, NT.WORDS), np.uint32)
        g.get_fn()(pq, om, n, unit)
        st["pq"], st["omegas"] = M.to_device(pq), M.to_device(om)
        st["fn"] = NT.RecomputeNtt(field).get_fn()
    else:
        tw = np.zeros((max(n // 2, 1), NT.WORDS), np.uint32)
        NT.SsipPrecompute(field).get_fn()(tw, unit)
        st["twiddle"] = M.to_device(tw)
        st["fn"] = NT.SsipNtt(field).get_fn()
    if case["kind"] == "coset":
        # powers of the coset shift, one per coefficient
        powers = np.zeros((n, NT.WORDS), np.uint32)
        NT.SsipPrecompute(field).get_fn()(powers, NT.to_mont_limbs(7, field))
        st["powers"] = M.to_device(powers)
        st["distribute"] = NT.DistributePowers(field).get_fn()
    return st


def run(state):
    kind = state["kind"]
    if kind == "msm":
        return state["ctx"].msm_device(state["scalars"], out=state["out"])
    if kind == "batch":
        return state["batch"].run(state["scalars"], out=state["out"])
    if kind == "drop_in":
        return state["op"].run([state["points"]], [state["scalars"]], [state["buffer"]])
    if kind == "precompute":
        state["op"](state["tables"], state["n"], 1)
        return state["tables"]
    if kind == "coset":
        state["distribute"](state["x"], state["powers"])
    if "twiddle" in state:
        state["fn"](state["x"], state["twiddle"])
    else:
        state["fn"](state["x"], state["pq"], state["omegas"])
    return state["x"]


def _msm_work(curve, n):
    """Scalars and points read once; Pippenger's bucket additions at a window
    near log2(n) - 2, six field products each (an affine addition whose
    inversion is shared), a product being 2 N^2 + N multiply-adds of N-limb
    numbers."""
    words = M.POINT_WORDS[curve]
    limbs = words // 2
    c = max(8, int(math.log2(n)) - 2)
    adds = n * M.window_count(c, curve)
    return {"bytes": n * (32 + 4 * words) + 4 * words, "flops": 2.0 * adds * 6 * (2 * limbs * limbs + limbs)}


def work(case):
    kind = case["kind"]
    if kind in ("msm", "drop_in"):
        return _msm_work(CURVES[case["curve"]], case["n"])
    if kind == "batch":
        each = [_msm_work(CURVES[case["curve"]], n) for n in _msm_sizes(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "precompute":
        curve = CURVES[case["curve"]]
        words = M.POINT_WORDS[curve]
        limbs = words // 2
        tables = M.n_precompute(case["window"], case["target"], curve)
        # per further table: window * target doublings (seven products each)
        # and an affine conversion with a shared inversion (seven)
        products = case["n"] * (tables - 1) * (7 * case["window"] * case["target"] + 7)
        return {"bytes": case["n"] * tables * words * 4, "flops": 2.0 * products * (2 * limbs * limbs + limbs)}
    log_n = case["log_n"]
    n = 1 << log_n
    products = NT.butterfly_products(log_n) + (n if kind == "coset" else 0)
    return {"bytes": (96 if kind == "coset" else 64) * n, "flops": 2.0 * products * 136}

// Pairwise affine additions inside the buckets, ahead of the XYZZ accumulation.
//
// A level takes a bucket-sorted list of affine points and adds neighbours
// 2j and 2j + 1 of every bucket (the last one of an odd bucket passes
// through), so that a bucket of m points leaves ceil(m / 2).  An affine
// addition whose inversion is shared (Montgomery's trick: one product per
// addition going forward, two going backward around one inversion) costs
// 5 products and 1 square, the XYZZ mixed addition 8 and 2.
#pragma once

#include "bn254.cuh"
#include "launch.cuh"

namespace impeller {

using namespace ec;

// Where bucket b's slots start after `level` levels.  Level l + 1 starts
// bucket b at (start_l + b) / 2: the buckets before it need at most
// sum ceil(m / 2) <= (start_l + b) / 2 slots, so no scan is needed, at the
// price of at most one unused slot per bucket.  Nested, that is
// (start_0 + (2^l - 1) b) / 2^l.
__host__ __device__ __forceinline__ u64 level_start(u64 start0, u64 b, u32 level) {
    return (start0 + (((u64)1 << level) - 1) * b) >> level;
}

// Points bucket b holds after `level` levels of a bucket of m.
__host__ __device__ __forceinline__ u32 level_count(u32 m, u32 level) {
    return (u32)(((u64)m + ((1u << level) - 1u)) >> level);
}

#ifndef PAIR_BLOCKS_PER_SM
#define PAIR_BLOCKS_PER_SM 4
#endif
#ifndef PAIR_BLOCKS_PER_SM_BLS
#define PAIR_BLOCKS_PER_SM_BLS 3
#endif
// Slots per lane and tile, at most; tiles are multiples of PAIR_UNIT slots per lane.
#ifndef PAIR_SLOTS
#define PAIR_SLOTS 128
#endif
#ifndef PAIR_UNIT
#define PAIR_UNIT 8
#endif
static constexpr u32 PAIR_BLOCK = 128;
static constexpr u32 PAIR_MAX_LEVELS = 6;
static constexpr u64 PAIR_SCRATCH_MAX = 16ull << 30;  // bytes of the first level's points
static constexpr u32 PAIR_NONE = 0xffffffffu;

// Where points come from: entries of the sort, entries among which indices
// from phi_base on stand for images under the endomorphism, or the previous
// level's points in order.
enum : int { FROM_ENTRIES = 0, FROM_IMAGES = 1, FROM_LEVEL = 2 };
template <class C>
struct PairShape {
    static constexpr u32 per_sm = C::XW == 32 ? PAIR_BLOCKS_PER_SM : PAIR_BLOCKS_PER_SM_BLS;
    static constexpr u32 planes = C::Fq::N / 4;
    // scratch of one block: a tile's running products and its pairs
    static constexpr u32 lanes = PAIR_BLOCK * PAIR_SLOTS;
    static constexpr size_t block_bytes = (size_t)lanes * (planes * 16 + 8);
    // shared memory: per warp two stages of 32 pairs and their running
    // products, a point padded by 16 bytes (an odd number of 16-byte units, so
    // that a warp's 16-byte reads hit every bank once); the threads' totals
    // take its place in between
    static constexpr u32 point_bytes = C::PW * 4 + 16;
    static constexpr u32 stage_bytes = 2 * 32 * point_bytes + 32 * planes * 16;
    static constexpr size_t smem = (size_t)(PAIR_BLOCK / 32) * 2 * stage_bytes;
    static_assert(smem >= (size_t)PAIR_BLOCK * planes * 16, "the totals share the stages' memory");
};

struct PairArgs {
    const u32 *offsets;  // nb + 1, level 0
    u32 nb;
    u32 level;           // of the input: 0 reads entries, later ones the previous level's points
    u32 sms;
    const u32 *entries;
    const u32 *points;   // level 0: the point array; else the previous level's points
    u32 *out;
    unsigned char *scratch;  // PairShape::block_bytes per block
    const u32 *phi;          // level 0: the images' abscissae, for entries of index phi_base + i
    u32 phi_base;
    const u32 *used;         // number of levels that run (k_pair_plan)
    u32 *next_unit;          // zero at launch
};

template <class F>
__device__ __forceinline__ void plane_store(uint4 *s, u32 plane, u32 i, const Fe<F> &a) {
#pragma unroll
    for (int k = 0; k < F::N / 4; k++)
        s[k * plane + i] = make_uint4(a.l[4 * k], a.l[4 * k + 1], a.l[4 * k + 2], a.l[4 * k + 3]);
}

template <class F>
__device__ __forceinline__ Fe<F> plane_load(const uint4 *s, u32 plane, u32 i) {
    Fe<F> r;
#pragma unroll
    for (int k = 0; k < F::N / 4; k++) {
        const uint4 v = s[k * plane + i];
        r.l[4 * k] = v.x;
        r.l[4 * k + 1] = v.y;
        r.l[4 * k + 2] = v.z;
        r.l[4 * k + 3] = v.w;
    }
    return r;
}

// Inverts the block's 128 totals in place: lane l of the warp takes threads
// l, l + 32, l + 64 and l + 96 around one inversion.
template <class F>
__device__ __noinline__ void invert_totals(uint4 *s, u32 plane, u32 lane) {
    static_assert(PAIR_BLOCK == 128, "four totals per lane");
    const Fe<F> a0 = plane_load<F>(s, plane, lane), a1 = plane_load<F>(s, plane, lane + 32);
    const Fe<F> a2 = plane_load<F>(s, plane, lane + 64), a3 = plane_load<F>(s, plane, lane + 96);
    const Fe<F> p1 = fe_mul_call<F>(a0, a1), p2 = fe_mul_call<F>(p1, a2);
    Fe<F> inv = fe_inv_divsteps<F>(fe_mul_call<F>(p2, a3), fe_rcube<F>());
    plane_store<F>(s, plane, lane + 96, fe_mul_call<F>(inv, p2));
    inv = fe_mul_call<F>(inv, a3);
    plane_store<F>(s, plane, lane + 64, fe_mul_call<F>(inv, p1));
    inv = fe_mul_call<F>(inv, a2);
    plane_store<F>(s, plane, lane + 32, fe_mul_call<F>(inv, a0));
    plane_store<F>(s, plane, lane, fe_mul_call<F>(inv, a1));
}

// The inputs of one output slot: entries (level 0) or indices of the previous
// level's points; y == PAIR_NONE for a lone one, x == PAIR_NONE for an unused
// slot.
//
// A warp looks up 32 consecutive slots at a time: its lanes read the starts
// of 32 consecutive buckets from the warp's current one and every lane finds
// its slot among them (a slot range of 32 spans few buckets).
struct PairWalk {
    const u32 *offsets, *entries;
    u32 nb, level, b;  // b: a bucket at or before the next slots'
    u32 window;        // offsets[b + lane], read ahead
    __device__ __forceinline__ PairWalk(const PairArgs &a, u32 s) : offsets(a.offsets), entries(a.entries), nb(a.nb), level(a.level) {
        u32 lo = 0, hi = nb;
        while (hi - lo > 1) {
            const u32 mid = (lo + hi) >> 1;
            if ((u32)level_start(offsets[mid], mid, level + 1) <= s) lo = mid;
            else hi = mid;
        }
        b = lo;
        window = offsets[min(b + (threadIdx.x & 31u), nb)];
    }
    // s: ascending over lanes and calls, below the last bucket's end
    template <int FROM>
    __device__ __forceinline__ uint2 at(u32 s, u32 lane) {
        u32 mine = NOT_FOUND, beg = 0, end = 0;
        for (;;) {
            const u32 o = window;
            const u32 start = (u32)level_start(o, min(b + lane, nb), level + 1);
            u32 r = 0;  // the last lane whose bucket starts at or before s
#pragma unroll
            for (u32 step = 16; step; step >>= 1) {
                const u32 v = __shfl_sync(0xffffffffu, start, r + step);
                if (v <= s) r += step;
            }
            const u32 ob = __shfl_sync(0xffffffffu, o, r), oe = __shfl_sync(0xffffffffu, o, (r + 1) & 31u);
            if (mine == NOT_FOUND && r < 31) {
                mine = b + r;
                beg = ob;
                end = oe;
            }
            if (__all_sync(0xffffffffu, mine != NOT_FOUND)) break;
            b += 31;
            window = offsets[min(b + lane, nb)];
        }
        b = __shfl_sync(0xffffffffu, mine, 31);
        window = offsets[min(b + lane, nb)];
        const u32 j = 2 * (s - (u32)level_start(beg, mine, level + 1)), cnt = level_count(end - beg, level);
        if (j >= cnt) return make_uint2(PAIR_NONE, PAIR_NONE);
        const u32 i = (u32)level_start(beg, mine, level) + j;
        const bool two = j + 1 < cnt;
        if constexpr (FROM != FROM_LEVEL) return make_uint2(entries[i], two ? entries[i + 1] : PAIR_NONE);
        else return make_uint2(i, two ? i + 1 : PAIR_NONE);
    }
    static constexpr u32 NOT_FOUND = 0xffffffffu;
};

// Where an entry's coordinates lie.  Index phi_base + i is the image of point
// i under the endomorphism (beta x, y): its abscissa lies in phi.
template <class C, bool IMAGES>
__device__ __forceinline__ void entry_coordinates(const u32 *points, u32 e, const u32 *phi, u32 phi_base,
                                                  const u32 *&px, const u32 *&py) {
    u32 i = e >> 1;
    if constexpr (IMAGES) {
        const bool image = i >= phi_base;
        if (image) i -= phi_base;
        py = points + (size_t)i * C::PW + C::Fq::N;
        px = image ? phi + (size_t)i * C::Fq::N : py - C::Fq::N;
    } else {
        px = points + (size_t)i * C::PW;
        py = px + C::Fq::N;
    }
}

template <class C, int FROM>
__device__ __forceinline__ void pair_coordinates(const PairArgs &a, u32 e, const u32 *&px, const u32 *&py) {
    if constexpr (FROM != FROM_LEVEL) {
        entry_coordinates<C, FROM == FROM_IMAGES>(a.points, e, a.phi, a.phi_base, px, py);
    } else {
        px = a.points + (size_t)e * C::PW;
        py = px + C::Fq::N;
    }
}

// Asynchronous copy of the leading CH 16-byte chunks of 32 points, one per
// lane, into the warp's stage at dst: neighbouring lanes copy neighbouring
// chunks of a point, so that a point costs one request.  (A random request
// that misses the TLB costs the same for one 32-byte sector as for the whole
// point: 38 G random requests/s over tables of 0.5 GB and more on B200, so
// lane-wise loads of a 64-byte point, two requests, reach 19 G points/s.)
template <class C, int FROM, u32 CH>
__device__ __forceinline__ void stage_points(const PairArgs &a, u32 e, u32 dst, u32 lane) {
#pragma unroll
    for (u32 j = 0; j < CH; j++) {
        const u32 c = lane + 32 * j, pt = c / CH, ch = c % CH;
        const u32 ee = __shfl_sync(0xffffffffu, e, pt);
        // no copy where there is no point: copies of one stand-in would all
        // queue at its L2 slice
        if (ee != PAIR_NONE) {
            const u32 *px, *py;
            pair_coordinates<C, FROM>(a, ee, px, py);
            const u32 *from = ch < C::Fq::N / 4 ? px + ch * 4 : py + ch * 4 - C::Fq::N;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + pt * PairShape<C>::point_bytes + ch * 16),
                         "l"(from)
                         : "memory");
        }
    }
}

// The lane's running product (16-byte planes at src) into the stage.
template <class C>
__device__ __forceinline__ void stage_product(const uint4 *src, u32 dst, u32 lane) {
#pragma unroll
    for (u32 k = 0; k < PairShape<C>::planes; k++)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (k * 32 + lane) * 16),
                     "l"(src + (size_t)k * PairShape<C>::lanes)
                     : "memory");
}

__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void stage_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
    __syncwarp();
}

// An affine point in 32-byte stores (whole sectors).
template <class F>
__device__ __forceinline__ void store32(u32 *p, const AffineT<F> &a) {
    u32 w[2 * F::N];
#pragma unroll
    for (int i = 0; i < F::N; i++) {
        w[i] = a.x.l[i];
        w[F::N + i] = a.y.l[i];
    }
#pragma unroll
    for (int i = 0; i < 2 * F::N; i += 8)
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p + i), "r"(w[i]), "r"(w[i + 1]),
                     "r"(w[i + 2]), "r"(w[i + 3]), "r"(w[i + 4]), "r"(w[i + 5]), "r"(w[i + 6]), "r"(w[i + 7])
                     : "memory");
}

// x1 == x2: a doubling when y1 == y2, else the sum is the identity (or one of
// the points is, and the sum the other).  d is the doubling's denominator or
// one: never zero, so that the shared product stays invertible.
template <class F>
__device__ __forceinline__ Fe<F> pair_equal_x(const Fe<F> &y1, const Fe<F> &y2, bool &dbl) {
    dbl = !fe_is_zero(y1) && fe_is_zero(fe_sub(y1, y2));
    return dbl ? fe_dbl(y1) : fe_one<F>();
}

// fe_is_zero and fe_is_zero_canonical behind a look at the low word (every
// slot takes these tests, and nearly none passes).
template <class F>
__device__ __forceinline__ bool pair_zero(const Fe<F> &a) {
    constexpr Words<F::N> m = words(F::M);
    return (a.l[0] == 0 || a.l[0] == m.v[0]) && fe_is_zero(a);
}
template <class F>
__device__ __forceinline__ bool pair_identity(const Fe<F> &y) {
    return y.l[0] == 0 && fe_is_zero_canonical(y);
}

template <class C, int FROM>
__device__ __forceinline__ Fe<typename C::Fq> pair_y(const u32 *py, u32 e) {
    const Fe<typename C::Fq> y = fe_load<typename C::Fq>(py);
    return FROM != FROM_LEVEL && (e & 1u) ? fe_neg(y) : y;
}

// One level.  A tile is 128 x kk consecutive output slots, 32 x kk of them a
// warp's: iteration k of a warp takes 32 consecutive slots.  Each lane
// multiplies its pairs' denominators together (the products before each go to
// the block's scratch), one warp inverts the 128 totals, and each lane goes
// back through its pairs.  Blocks take tiles from a counter.
template <class C, int FROM>
__global__ void __launch_bounds__(PAIR_BLOCK, PairShape<C>::per_sm) k_affine_pairs(PairArgs a) {
    grid_wait();
    using FQ = typename C::Fq;
    using S = PairShape<C>;
    extern __shared__ uint4 pair_smem[];
    __shared__ u32 tile_at, tile_units;
    uint4 *const totals = pair_smem;
    constexpr u32 plane = S::lanes, XCH = FQ::N / 4, PCH = 2 * XCH;
    uint4 *const pre = reinterpret_cast<uint4 *>(a.scratch + (size_t)blockIdx.x * S::block_bytes);
    uint2 *const src = reinterpret_cast<uint2 *>(pre + (size_t)S::planes * plane);
    const u32 tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
    // the warp's two stages: points 1 of the 32 pairs, then points 2
    unsigned char *const stage_ptr = reinterpret_cast<unsigned char *>(pair_smem) + wid * 2 * S::stage_bytes;
    const u32 stage = (u32)__cvta_generic_to_shared(stage_ptr);
    constexpr u32 SECOND = 32 * S::point_bytes, PRODUCT = 2 * SECOND;
    // co-resident blocks invert on different warps (and so on different schedulers)
    const u32 q = (blockIdx.x / a.sms) & 3u;
    if (a.level >= *a.used) return;
    const u32 total = (u32)level_start(a.offsets[a.nb], a.nb, a.level + 1);
    if (total == 0) return;
    // What fits one tile per block is split evenly; more is taken in tiles of
    // PAIR_SLOTS slots per lane that shrink towards the end, so that the
    // blocks end together.
    const bool single = total <= (u64)gridDim.x * S::lanes;
    const u32 unit = single ? (total + gridDim.x * PAIR_BLOCK - 1) / (gridDim.x * PAIR_BLOCK) : PAIR_UNIT;  // per lane
    const u32 units = (total + PAIR_BLOCK * unit - 1) / (PAIR_BLOCK * unit);

    for (;;) {
        if (tid == 0) {
            const u32 left = units - min(*(volatile u32 *)a.next_unit, units);
            const u32 want = single ? 1u : min(max((2 * left + 3 * gridDim.x - 1) / (3 * gridDim.x), 1u), (u32)(PAIR_SLOTS / PAIR_UNIT));
            tile_units = want;
            tile_at = atomicAdd(a.next_unit, want);
        }
        __syncthreads();
        const u32 first = tile_at, kk = tile_units * unit;
        if (first >= units) return;
        // this warp's slots
        const u64 w0 = (u64)first * unit * PAIR_BLOCK + (u64)wid * 32 * kk;
        const u32 s0 = (u32)min(w0, (u64)total), s1 = (u32)min(w0 + 32 * kk, (u64)total);
        const u32 n = (s1 - s0 + 31) / 32;
        uint4 *const my_pre = pre + (size_t)wid * 32 * kk + lane;
        uint2 *const my_src = src + (size_t)wid * 32 * kk + lane;
        Fe<FQ> run = fe_one<FQ>();
        if (n) {
            PairWalk walk(a, s0);
            auto look = [&](u32 k) {
                const u32 s = s0 + 32 * k + lane;
                uint2 e = walk.at<FROM>(min(s, total - 1), lane);
                if (s >= s1) e = make_uint2(PAIR_NONE, PAIR_NONE);
                return e;
            };
            // slot inputs are looked up two iterations ahead, their points copied one ahead
            uint2 e = look(0), next = make_uint2(PAIR_NONE, PAIR_NONE);
            stage_points<C, FROM, XCH>(a, e.x, stage, lane);
            stage_points<C, FROM, XCH>(a, e.y, stage + SECOND, lane);
            stage_commit();
            if (n > 1) next = look(1);
#pragma unroll 1
            for (u32 k = 0; k < n; k++) {
                if (k + 1 < n) {
                    const u32 at = stage + ((k + 1) & 1u) * S::stage_bytes;
                    stage_points<C, FROM, XCH>(a, next.x, at, lane);
                    stage_points<C, FROM, XCH>(a, next.y, at + SECOND, lane);
                }
                stage_commit();
                uint2 next2 = make_uint2(PAIR_NONE, PAIR_NONE);
                if (k + 2 < n) next2 = look(k + 2);
                my_src[32 * k] = e;
                stage_wait<1>();
                if (e.y != PAIR_NONE) {
                    const u32 *p = reinterpret_cast<const u32 *>(stage_ptr + (k & 1u) * S::stage_bytes + lane * S::point_bytes);
                    Fe<FQ> d = fe_sub(fe_load<FQ>(p + SECOND / 4), fe_load<FQ>(p));
                    if (pair_zero(d)) {
                        bool dbl;
                        const u32 *px, *py1, *py2;
                        pair_coordinates<C, FROM>(a, e.x, px, py1);
                        pair_coordinates<C, FROM>(a, e.y, px, py2);
                        d = pair_equal_x(pair_y<C, FROM>(py1, e.x), pair_y<C, FROM>(py2, e.y), dbl);
                    }
                    plane_store<FQ>(my_pre, plane, 32 * k, run);
                    run = fe_mul(run, d);
                }
                __syncwarp();  // the stage is overwritten by the next iteration's copies
                e = next;
                next = next2;
            }
        }
        __syncthreads();  // every warp is done with its stages
        plane_store<FQ>(totals, PAIR_BLOCK, tid, run);
        __syncthreads();
        if (wid == q) invert_totals<FQ>(totals, PAIR_BLOCK, lane);
        __syncthreads();
        Fe<FQ> inv = plane_load<FQ>(totals, PAIR_BLOCK, tid);
        __syncthreads();
        if (n) {
            uint2 e = my_src[32 * (n - 1)], next = n > 1 ? my_src[32 * (n - 2)] : e;
            stage_points<C, FROM, PCH>(a, e.x, stage + ((n - 1) & 1u) * S::stage_bytes, lane);
            stage_points<C, FROM, PCH>(a, e.y, stage + ((n - 1) & 1u) * S::stage_bytes + SECOND, lane);
            if (e.y != PAIR_NONE) stage_product<C>(my_pre + 32 * (n - 1), stage + ((n - 1) & 1u) * S::stage_bytes + PRODUCT, lane);
            stage_commit();
#pragma unroll 1
            for (u32 k = n; k-- > 0;) {
                uint2 next2 = next;
                if (k > 1) next2 = my_src[32 * (k - 2)];
                if (k) {
                    const u32 at = stage + ((k - 1) & 1u) * S::stage_bytes;
                    stage_points<C, FROM, PCH>(a, next.x, at, lane);
                    stage_points<C, FROM, PCH>(a, next.y, at + SECOND, lane);
                    if (next.y != PAIR_NONE) stage_product<C>(my_pre + 32 * (k - 1), at + PRODUCT, lane);
                }
                stage_commit();
                stage_wait<1>();
                const u32 *p1 = reinterpret_cast<const u32 *>(stage_ptr + (k & 1u) * S::stage_bytes + lane * S::point_bytes);
                const u32 *p2 = p1 + SECOND / 4;
                AffineT<FQ> r;
                if (e.y != PAIR_NONE) {
                    Fe<FQ> d = fe_sub(fe_load<FQ>(p2), fe_load<FQ>(p1));
                    bool dbl = false;
                    const bool same = pair_zero(d);
                    if (same) d = pair_equal_x(pair_y<C, FROM>(p1 + FQ::N, e.x), pair_y<C, FROM>(p2 + FQ::N, e.y), dbl);
                    const uint4 *pp = reinterpret_cast<const uint4 *>(stage_ptr + (k & 1u) * S::stage_bytes + PRODUCT);
                    const Fe<FQ> w = fe_mul(inv, plane_load<FQ>(pp, 32, lane));  // 1 / d
                    inv = fe_mul(inv, d);
                    const Fe<FQ> y1 = pair_y<C, FROM>(p1 + FQ::N, e.x), y2 = pair_y<C, FROM>(p2 + FQ::N, e.y);
                    Fe<FQ> num = fe_sub(y2, y1);
                    const Fe<FQ> x1 = fe_load<FQ>(p1), x2 = fe_load<FQ>(p2);
                    if (dbl) {
                        const Fe<FQ> xx = fe_sqr(x1);
                        num = fe_add(fe_dbl(xx), xx);
                    }
                    const Fe<FQ> l = fe_mul(num, w);
                    r.x = fe_sub(fe_sub(fe_sqr(l), x1), x2);
                    r.y = fe_sub(fe_mul(l, fe_sub(x1, r.x)), y1);
                    const bool id1 = pair_identity(y1), id2 = pair_identity(y2);
                    if (id1 || id2 || (same && !dbl)) {
                        // an identity input leaves the other point; opposite points the identity
                        r.x = id1 ? x2 : x1;
                        r.y = id1 ? y2 : y1;
                        if (!id1 && !id2) r.x = r.y = fe_zero<FQ>();
                    }
                } else if (e.x != PAIR_NONE) {
                    r.x = fe_load<FQ>(p1);
                    r.y = pair_y<C, FROM>(p1 + FQ::N, e.x);
                } else {
                    r.x = r.y = fe_zero<FQ>();  // unused slot: the identity
                }
                const u32 s = s0 + 32 * k + lane;
                if (s < s1) store32(a.out + (size_t)s * C::PW, r);
                __syncwarp();
                e = next;
                next = next2;
            }
        }
    }
}

// How many levels pay: while the buckets hold PAIR_MIN_BUCKET points and
// more on average (below, unused slots and lone points eat the gain) and the
// level's slots are at least slots_min (below, the levels' inversions do).
static constexpr u32 PAIR_MIN_BUCKET = 8;
__host__ __device__ __forceinline__ u32 pair_levels(u64 entries, u64 nb, u64 slots_min, u32 most) {
    u32 k = 0;
    while (k < most && entries >= ((u64)PAIR_MIN_BUCKET * nb << k) && level_start(entries, nb, k + 1) >= slots_min) k++;
    return k;
}

// The host sizes the levels by the digits the scalars can have; this decides
// by those they do have (skewed scalars have many zero digits).  out: the
// bucket starts after the last level; state: the number of levels, then the
// levels' tile counters.
__global__ void k_pair_plan(const u32 *offsets, u32 nb, u32 slots_min, u32 most, u32 *out, u32 *state) {
    grid_wait();
    const u32 used = pair_levels(offsets[nb], nb, slots_min, most);
    if (blockIdx.x == 0 && threadIdx.x <= PAIR_MAX_LEVELS) state[threadIdx.x] = threadIdx.x ? 0 : used;
    for (u32 b = blockIdx.x * blockDim.x + threadIdx.x; b <= nb; b += gridDim.x * blockDim.x)
        out[b] = (u32)level_start(offsets[b], b, used);
}

}  // namespace impeller

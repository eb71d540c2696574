/*
 * fsph_passes.cuh -- per-particle bodies of the PBF passes, shared by the
 * single-scene kernels (fsph_kernels.cu, one thread per particle) and the
 * batched persistent kernels (fsph_batch.cu, tiles of one scene per block).
 *
 * A body computes one particle i (a slot in device order) with the constants
 * of its scene, p.  `valid` is false for the padding lanes of a tile: they
 * run the loops on a clamped slot (so warp-wide shuffles stay convergent)
 * and write nothing.  LPP > 1 lets LPP adjacent lanes share one particle's
 * candidates (lane `sub` takes entries sub, sub + LPP, ...); their partial
 * sums are combined with shuffles, and lane 0 of the group writes.
 */
#pragma once
#include <cuda_fp16.h>

#include "fsph_kernels.cuh"

namespace fsph {

/* ---------------- candidate loop ---------------- */

/* Calls f(j, load(j)) for every candidate slot j of slot i handled by lane
 * `sub` of its LPP-lane group: the list entries sub, sub + LPP, ... or -- for
 * an overflowed list or when lists are off -- every LPP-th slot of the 27
 * cells around the current position.  List entries are taken kBatch at a
 * time: their indices are decoded and their positions loaded before any is
 * used, so each thread keeps kBatch independent loads in flight (the passes
 * are bound by load latency, not by arithmetic).  Load selects the load
 * flavour for x. */
#ifndef FSPH_KBATCH
#define FSPH_KBATCH 4
#endif

/* resident threads per SM the constraint passes are compiled for (single
 * scene and batched): 1536 cap them at 40 registers, 48 warps per SM
 * (measured best) */
#ifndef FSPH_PASS_THREADS
#define FSPH_PASS_THREADS 1536
#endif
#define FSPH_PASS_MINB (FSPH_PASS_THREADS / FSPH_PASS_BLOCK)
constexpr int kBatch = FSPH_KBATCH;

/* FSPH_FOLD 1: the constraint passes keep constant factors out of the pair
 * loop (fewer instructions per candidate; same results to rounding).
 * Measured on the 1M double dam break: lambda 82 -> 80 us, warm step
 * 2.855 -> 2.817 ms, plain step 10.25 -> 10.06 ms; on by default. */
#ifndef FSPH_FOLD
#define FSPH_FOLD 1
#endif
/* Neighbour-list loads do not allocate in L1 (ld.global.nc.L1::no_allocate):
 * a pass streams ≈ 160 B of list per particle once, while the gathered
 * positions (16 B per particle, each read ≈ 40 times per pass) keep L1 to
 * themselves.  FSPH_LIST_HINT 0 gives plain read-only loads. */
#ifndef FSPH_LIST_HINT
#define FSPH_LIST_HINT 1
#endif

__device__ __forceinline__ uint4 load_list_group(const uint4 *a) {
#if FSPH_LIST_HINT == 1
    uint4 r;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(a));
    return r;
#elif FSPH_LIST_HINT == 2
    /* also first in line for eviction from L2: the streamed lists make room
     * before the gathered positions do */
    uint4 r;
    unsigned long long pol;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(a), "l"(pol));
    return r;
#else
    return __ldg(a);
#endif
}

/* The list groups are prefetched into L2 kListAhead groups ahead of their
 * use (the lists stream from DRAM: they are larger than L2).  Measured at
 * 1 M particles: 2 groups ahead -2.3 % per step; 1, 3 or 4 ahead, or the
 * next group loaded into registers, gain less.  FSPH_LIST_PF 0 turns the
 * prefetch off. */
#ifndef FSPH_LIST_PF
#define FSPH_LIST_PF 1
#endif
constexpr int kListAhead = 2;

__device__ __forceinline__ void prefetch_list_group(const uint4 *a) {
#if FSPH_LIST_PF
    asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
#endif
}

/* DEEP: for launches that leave the GPU's warps few (kDeepMax): eight
 * candidates and the next two list groups in flight instead of four
 * candidates, so that a particle's chain of dependent loads is half as long;
 * it takes the registers that so few warps leave unused.  The order in which
 * f meets the candidates, and so the result, is the same. */
template <int LPP, bool DEEP = false, class Load, class F>
__device__ __forceinline__ void for_each_candidate(const DevParams &p, const unsigned int *__restrict__ cell_start,
                                                   const ListEntry *__restrict__ list,
                                                   const unsigned char *__restrict__ cnt, int i, float3 xi, int sub,
                                                   Load &&load, F &&f) {
    int k = list ? (int)cnt[i] : (int)kListOverflow;
#if FSPH_DEBUG_BOUNDS
    if (k > kListMax && k != (int)kListOverflow) { /* a count the build never writes: walk the cells */
        if (p.dbg) atomicOr(p.dbg, kBoundCount);
        k = (int)kListOverflow;
    }
#endif
    if (DEEP && k != (int)kListOverflow) {
        const uint4 *lg = reinterpret_cast<const uint4 *>(list) + i;
        const size_t n = (size_t)p.n;
        uint4 e[2];
        e[0] = load_list_group(lg);
        e[1] = load_list_group(k > 4 ? lg + n : lg);
        for (int t0 = 0; t0 < k; t0 += 8) {
            const uint4 *nx = lg + (size_t)((t0 >> 2) + 2) * n;
            uint4 g[2] = {e[0], e[0]};
            if (t0 + 8 < k) g[0] = load_list_group(nx);
            if (t0 + 12 < k) g[1] = load_list_group(nx + n);
            const unsigned int j[8] = {e[0].x, e[0].y, e[0].z, e[0].w, e[1].x, e[1].y, e[1].z, e[1].w};
            decltype(load(0u)) xj[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) xj[u] = load(bounded(p, j[u], (unsigned int)p.n, kBoundSlot));
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (t0 + u < k) f(bounded(p, j[u], (unsigned int)p.n, kBoundSlot), xj[u]);
            e[0] = g[0];
            e[1] = g[1];
        }
    } else if (LPP == 1 && kBatch == 4 && k != (int)kListOverflow) {
        /* one 16-byte load brings the next four entries (the tail group is
         * padded with a valid slot, so every load stays in bounds) */
        const uint4 *lg = reinterpret_cast<const uint4 *>(list) + i;
#pragma unroll
        for (int g = 1; g < kListAhead; ++g)
            if (4 * g < k) prefetch_list_group(lg + (size_t)g * (size_t)p.n);
        for (int t0 = 0; t0 < k; t0 += 4) {
            if (t0 + 4 * kListAhead < k) prefetch_list_group(lg + (size_t)((t0 >> 2) + kListAhead) * (size_t)p.n);
            const uint4 e = load_list_group(lg + (size_t)(t0 >> 2) * (size_t)p.n);
            const unsigned int j[4] = {bounded(p, e.x, (unsigned int)p.n, kBoundSlot),
                                       bounded(p, e.y, (unsigned int)p.n, kBoundSlot),
                                       bounded(p, e.z, (unsigned int)p.n, kBoundSlot),
                                       bounded(p, e.w, (unsigned int)p.n, kBoundSlot)};
            decltype(load(0u)) xj[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) xj[u] = load(j[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (t0 + u < k) f(j[u], xj[u]);
        }
    } else if (k != (int)kListOverflow) {
        for (int t0 = sub; t0 < k; t0 += kBatch * LPP) {
            unsigned int j[kBatch];
            decltype(load(0u)) xj[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const int t = t0 + u * LPP < k ? t0 + u * LPP : k - 1;
                j[u] = bounded(p, __ldg(list + list_at(t, i, p.n)), (unsigned int)p.n, kBoundSlot);
            }
#pragma unroll
            for (int u = 0; u < kBatch; ++u) xj[u] = load(j[u]);
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                if (t0 + u * LPP < k) f(j[u], xj[u]);
        }
    } else {
        const int3 c = cell_of(xi, p);
        for (int dz = -1; dz <= 1; ++dz)
            for (int dy = -1; dy <= 1; ++dy) {
                unsigned int s, e;
                row_range(cell_start, c, dy, dz, p, s, e);
                for (unsigned int j = s + (unsigned int)sub; j < e; j += LPP) f(j, load(j));
            }
    }
}

/* Calls f(b, bpos[b]) for every boundary slot b in the 27 cells around the
 * cell of x (nothing when no boundary particle is near that cell).  The
 * boundary is static and sorted by the same cells as the fluid, so a
 * boundary particle within h of x lies in those cells. */
template <class F>
__device__ __forceinline__ void for_each_boundary(const DevParams &p, float3 x, F &&f) {
    const int3 c = cell_of(x, p);
    const unsigned int ci = cell_index(c, p);
    if (!p.bnear[ci]) return;
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy) {
            const unsigned int base = ci + (unsigned int)((dz * p.gy + dy) * p.gx);
            if (!cell_row_ok(p, base)) continue;
            const unsigned int s = __ldg(p.bcell + base - 1);
            const unsigned int e = bounded(p, __ldg(p.bcell + base + 2), (unsigned int)p.nb + 1u, kBoundBoundary);
            for (unsigned int j = s; j < e; ++j) f(j, __ldg(p.bpos + j));
        }
}

/* sum over the LPP lanes of a group (every lane of the warp must call it) */
template <int LPP>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = LPP / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

/* Sums and products of two floats without their rounding errors: the result
 * and its error (Knuth; Dekker; the product's error from one fused operation),
 * with no contraction by the compiler. */
struct Split {
    float h, l; /* the value is h + l */
};
__device__ __forceinline__ Split two_sum(float a, float b) {
    const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
    return Split{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
/* group_sum of v + e, e the part of each lane's sum that v has lost: every lane
 * gets the same value (each addition is the same seen from either side) */
template <int LPP>
__device__ __forceinline__ float group_sum_split(float v, float e) {
#pragma unroll
    for (int o = LPP / 2; o > 0; o >>= 1) {
        const Split t = two_sum(v, __shfl_xor_sync(0xffffffffu, v, o));
        e = __fadd_rn(__fadd_rn(e, __shfl_xor_sync(0xffffffffu, e, o)), t.l);
        v = t.h;
    }
    return __fadd_rn(v, e);
}

/* ---------------- grid build ---------------- */

/* x* = walls(x + dt (v + dt a)), a = gravity when acc == NULL, then the
 * cell key and the slot's rank within the cell. */
__device__ __forceinline__ void predict_body(const DevParams &p, int i, const float4 *__restrict__ pos,
                                             const float4 *__restrict__ vel, const float4 *__restrict__ acc,
                                             float4 *__restrict__ ppos_out, unsigned int *__restrict__ key,
                                             unsigned int *__restrict__ rank, unsigned int *__restrict__ count,
                                             const float4 *__restrict__ dwarm, float4 *__restrict__ xpred_out) {
    float3 x = f3(pos[i]);
    float3 v = f3(vel[i]);
    float3 a = acc ? f3(acc[i]) : p.gravity;
    const float3 x_old = x;
    v = v + p.dt * a;
    x = x + p.dt * v;
    if (p.ntri) polygon_collide(x_old, x, v, p.dt, p);
    x = solid_project(x, p);
    if (xpred_out) xpred_out[i] = make_float4(x.x, x.y, x.z, 0.0f);
    /* warm start: the iterations begin from walls(x* + predicted correction);
     * the grid and lists are then built on that start */
    if (dwarm) x = solid_project(x + f3(dwarm[i]), p);
    ppos_out[i] = make_float4(x.x, x.y, x.z, 0.0f);
    unsigned int c = cell_index(cell_of(x, p), p);
    key[i] = c;
    rank[i] = atomicAdd(count + c, 1u);
}

__device__ __forceinline__ void hash_body(const DevParams &p, int i, float3 x, unsigned int *__restrict__ key,
                                          unsigned int *__restrict__ rank, unsigned int *__restrict__ count) {
    unsigned int c = cell_index(cell_of(x, p), p);
    key[i] = c;
    rank[i] = atomicAdd(count + c, 1u);
}

/* Calls f(j, load(j)) for every slot j of the 27 cells around `cell`, in ascending
 * order: a thread's own search, for the slots of a warp that do not search
 * together (warp_candidates).  Four positions and the bounds of three rows in
 * flight. */
template <class Load, class F>
__device__ __forceinline__ void walk_cells(const DevParams &p, const unsigned int *__restrict__ cell_start,
                                           unsigned int cell, Load &&load, F &&f) {
#pragma unroll 1
    for (int z = -1; z <= 1; ++z) {
        unsigned int s[3], e[3];
#pragma unroll
        for (int y = 0; y < 3; ++y) {
            const unsigned int base = cell + (unsigned int)((z * p.gy + (y - 1)) * p.gx);
            s[y] = e[y] = 0u;
            if (!cell_row_ok(p, base)) continue;
            s[y] = __ldg(cell_start + base - 1);
            e[y] = bounded(p, __ldg(cell_start + base + 2), (unsigned int)p.n + 1u, kBoundSlot);
        }
#pragma unroll
        for (int y = 0; y < 3; ++y)
            for (unsigned int j0 = s[y]; j0 < e[y]; j0 += 4) {
                float4 xc[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) xc[u] = load(min(j0 + u, e[y] - 1));
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (j0 + u < e[y]) f(j0 + u, xc[u]);
            }
    }
}

/* Every slot j within the list radius (= the cell width) of slot i at the
 * build positions xb, self included, in ascending order: one thread on its own. */
__device__ __forceinline__ void build_list_body(const DevParams &p, int i, const unsigned int *__restrict__ cell_start,
                                                const float4 *__restrict__ xb, unsigned int cell,
                                                ListEntry *__restrict__ list, unsigned char *__restrict__ cnt) {
    const float3 xi = f3(xb[i]);
    int k = 0;
    ListEntry last = 0;
    walk_cells(
        p, cell_start, cell, [&](unsigned int j) { return __ldg(xb + j); },
        [&](unsigned int j, const float4 &xj) {
            const float3 d = xi - f3(xj);
            if (!(dot3(d, d) < p.rl2)) return;
            last = j;
            if (k < kListMax) list[list_at(k, i, p.n)] = last;
            ++k;
        });
    const bool overflow = k > kListMax;
    if (!overflow) /* pad the last group (k >= 1: the slot itself is always listed) */
        for (int t = k; (t & 3) != 0; ++t) list[list_at(t, i, p.n)] = last;
    cnt[i] = overflow ? kListOverflow : (unsigned char)k;
}

/* The candidates of the 32 consecutive slots of a warp, searched together on
 * the tensor cores.  The slots lie in a run of a few cells along x, so in each
 * of the nine rows of cells their candidates are one range of slots, about 1.9
 * times what a lane's own three cells hold.  The warp takes 32 of them at a
 * time and computes all 32 x 32 values r^2 / rr^2 - 1 as products of 16 terms
 * (mma.m16n8k16): with coordinates relative to the warp, in units of the radius
 * and split into two halves of 11 bits each, r^2 = |xi|^2 + |xj|^2 - 2 xi.xj
 * needs the three products of the halves (the last, 2^-22, left out), the two
 * norms (split too) and the constant:
 *
 *   candidate  xh yh zh nh   xl yl zl nl   xh yh zh nh    1  1   1   1
 *   slot      -2xh   ..  1  -2xh   ..  1  -2xl   ..  0   nh nl  -1  -2^-12
 *
 * The error of a value is below 1e-4 (coordinates of at most 6, sums of 16
 * terms below 80) and the constant is 1 + 2^-12: every slot within the radius is
 * found, and one in some thousands that lies a hair beyond it, which a pass
 * evaluates to zero.  The signs shift into masks, eight candidates of four slots
 * a lane, which two shuffles turn into 32 candidates of one slot.
 * Tested two at a time in packed single precision 32 x 32 candidates took 170
 * instructions and the list build 266 us at 1 M particles, a thread walking its
 * own cells 291 us, both bound by instruction issue; this form takes 174 us, and
 * 16 instead of 33 at 6,912 particles.  Without the walk over the
 * masks and the rows' stores it takes 125, without the matrix instructions too 93:
 * reading, converting and staging the candidates is what is left. */
constexpr int kTileWords = 32; /* masks of a warp's candidates: 32 x 32 slots */
template <int W> /* the warps that share it */
struct __align__(16) PairTileOf {
    uint4 row[W][32];                   /* operand rows, eight terms each */
    unsigned int mask[kTileWords][32];  /* [w][lane], bit 31 - k: candidate k of word w is within the radius */
    unsigned int slot[kTileWords][32];  /* [w][k]: the candidates' slots */
    int cnt[W][32];                     /* what each warp found for a lane's slot (W > 1) */
};
using PairTile = PairTileOf<1>;

__device__ __forceinline__ unsigned int half_pair(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const unsigned int *>(&v);
}
__device__ __forceinline__ float2 pair_floats(unsigned int v) {
    return __half22float2(*reinterpret_cast<const __half2 *>(&v));
}
/* a point's terms: (xh, yh), (zh, nh) and the lower halves (xl, yl), (zl, nl) */
struct PairTerms {
    unsigned int h0, h1, l0, l1;
    float nn;
};
__device__ __forceinline__ PairTerms pair_terms(float x, float y, float z) {
    PairTerms t;
    t.nn = x * x + y * y + z * z;
    t.h0 = half_pair(x, y);
    t.h1 = half_pair(z, t.nn);
    const float2 a = pair_floats(t.h0), b = pair_floats(t.h1);
    t.l0 = half_pair(x - a.x, y - a.y);
    t.l1 = half_pair(z - b.x, t.nn - b.y);
    return t;
}
/* both halves times -2 (exact) */
__device__ __forceinline__ unsigned int times_m2(unsigned int v) {
    const __half2 r = __hmul2(*reinterpret_cast<const __half2 *>(&v), __float2half2_rn(-2.0f));
    return *reinterpret_cast<const unsigned int *>(&r);
}
__device__ __forceinline__ void load_matrices(unsigned int (&r)[4], const uint4 *row) {
    const unsigned int at = (unsigned int)__cvta_generic_to_shared(row);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(at)
                 : "memory");
}
/* m << 1 with the sign of v shifted in */
__device__ __forceinline__ unsigned int sign_in(unsigned int m, float v) {
    return __funnelshift_l(__float_as_uint(v), m, 1);
}
/* the four signs' masks of a 16 x 8 tile of tests: rows g and g + 8, columns
 * 2c and 2c + 1 (lane = 4g + c) */
__device__ __forceinline__ void test_tile(unsigned int &m0, unsigned int &m1, unsigned int a0, unsigned int a1,
                                          unsigned int a2, unsigned int a3, unsigned int b0, unsigned int b1) {
    float d0, d1, d2, d3;
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%10, %10, %10, %10};"
        : "=f"(d0), "=f"(d1), "=f"(d2), "=f"(d3)
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
    m0 = sign_in(sign_in(m0, d0), d1);
    m1 = sign_in(sign_in(m1, d2), d3);
}

/* One lane's candidates of a tile, ascending.  next() gives the `left`-th from the
 * end; called again after the last it keeps giving that one.  Selects instead of
 * branches: at almost every call some lane of a warp opens its next word. */
template <int W>
struct TileWalk {
    const PairTileOf<W> &t;
    unsigned int some, m = 0u;
    int w = 0, left;
    unsigned int last = 0u;
    __device__ __forceinline__ TileWalk(const PairTileOf<W> &tile, unsigned int words, int count)
        : t(tile), some(words), left(count) {}
    __device__ __forceinline__ unsigned int next() {
        const bool open = m == 0u;
        const int wn = __clz((int)some) & 31;
        const unsigned int mn = t.mask[wn][threadIdx.x & 31];
        w = open ? wn : w;
        m = open ? mn : m;
        some = open ? some & ~(0x80000000u >> wn) : some;
        const int b = __clz((int)m) & 31;
        m &= ~(0x80000000u >> b);
        const unsigned int j = t.slot[w][b];
        last = left > 0 ? j : last;
        --left;
        return last;
    }
};

/* Calls emit(found, first, count, total, walk) for each valid lane: found: the
 * lane's `count` candidates within sqrt(r2max) come from walk, ascending; else they
 * have to be looked for without the tile (lanes far apart, or a coordinate out of the
 * operands' range: a particle far outside the box, or not a number).  load(j): slot
 * j's position, a plain load where the kernel writes beside it.  xi, cell: the lane's
 * position and build cell, cells ascending over the lanes, padding lanes (valid =
 * false) after the valid ones; every lane of the warp calls it.  Lanes in different
 * rows of cells, or more than eight cells apart (a run that wraps), take turns: a
 * row's range then never reaches the next row, and no slot is met twice.  As many
 * turns as fit the tile are emitted together.
 *
 * W > 1: the W warps of a block share the same 32 slots (a lane's slot is the same
 * in each) and the tile.  Each takes a W-th of every turn's words and emits what it
 * found there: `count` of the lane's `total`, from the `first` on.  A warp's twenty
 * words in a row, latency bound, are the pass of a small scene: 16 us at 6,912 slots
 * with one warp, 10 with four.
 *
 * In compressed fluid a turn that does not fit the tile goes through it in parts, each
 * emitted with the total so far; found = false then starts a lane again (for W > 1 it
 * is for warp 0 to act on).  The lanes' own walks, which one warp of the four did,
 * took 178 us where the parts take 37: the density of a collapsing dam of 32,768
 * particles with 71 neighbours on average; of 512,000 with 106 444 and 291.
 *
 * In sparse fluid (spray) the lanes share few candidates and a warp takes up to 32
 * turns: there each lane looks for its own, once the cells between the lanes, at
 * most three a pair, are more than kTileApart (a lattice at rest has about 5).  The
 * list build in us, own / tile, at 1 M particles at random with one in (0.8 h)^3 129
 * / 128, h^3 125 / 143, (1.2 h)^3 100 / 145, (2 h)^3 58 / 252; with four warps, 30,000
 * particles, (0.8 h)^3 17 / 13, h^3 17 / 19, (1.2 h)^3 15 / 34, (2 h)^3 9 / 34. */
constexpr int kTileApart = 24, kTileApartSplit = 36; /* one warp, several */
template <int W, class Load, class Emit>
__device__ __forceinline__ void warp_candidates(const DevParams &p, const unsigned int *__restrict__ cell_start,
                                                Load &&load, float3 xi, unsigned int cell, bool valid, float r2max,
                                                PairTileOf<W> &t, Emit &&emit) {
    const int lane = threadIdx.x & 31, wid = W > 1 ? (int)(threadIdx.x >> 5) : 0;
    uint4 *const rows = t.row[wid];
    const unsigned int row = (cell - p.cell_off) / (unsigned int)p.gx;
    const float inv = rsqrtf(r2max);
    /* candidate 8 q + 2 s + b is column 2 q + b of step s; the rows are stored so
     * that neither the stores nor the loads of eight rows collide */
    uint4 *const st = rows + 8 * (lane >> 3) + 2 * ((lane >> 3) ^ ((lane >> 1) & 3)) + (lane & 1);
    const uint4 *const ld = rows + 8 * ((lane & 7) >> 1) + 2 * (((lane & 7) >> 1) ^ (lane >> 3)) + (lane & 1);
    const unsigned int pick1 = (lane & 2) ? 0x3726u : 0x5140u, pick2 = (lane & 1) ? 0x6273u : 0x0415u;
    const unsigned int ones = 0x3c003c00u; /* (1, 1) */
    const bool upper = (lane & 2) != 0;    /* terms 12-15 of a candidate are ones, 8-11 its terms 0-3 again */
    const int own = (lane >> 2) + 8 * (lane & 3); /* the slot whose 32 candidates this lane ends up with */
    /* lanes too far apart to share candidates look for their own */
    const unsigned int prev = __shfl_up_sync(0xffffffffu, cell, 1);
    const bool apart = __reduce_add_sync(0xffffffffu, valid && lane > 0 ? min(cell - prev, 3u) : 0u) >
                       (unsigned int)(W == 1 ? kTileApart : kTileApartSplit);
    unsigned int todo = __ballot_sync(0xffffffffu, valid);
    unsigned int resume = 0u; /* the word at which a turn in parts goes on */
    int base = 0;             /* what its earlier parts found for the lane */
    while (todo) {
        int cnt = 0, w = 0;
        unsigned int any = 0u, done = 0u, part = 0u;
        bool bad = false;
        if (apart) {
            done = todo;
            todo = 0u;
        }
        while (todo) { /* turns, until the tile is full */
            const int lead = __ffs((int)todo) - 1;
            const unsigned int lead_row = __shfl_sync(0xffffffffu, row, lead);
            const unsigned int first = __shfl_sync(0xffffffffu, cell, lead);
            const bool mine = (todo >> lane & 1u) && row == lead_row && cell - first <= 7u;
            const unsigned int grp = __ballot_sync(0xffffffffu, mine);
            const int tail = 31 - __clz((int)grp);
            const unsigned int last = __shfl_sync(0xffffffffu, cell, tail);
            /* lane r < 9: row r's cells first - 1 .. last + 1 hold the slots from s on; the
             * rows' candidates are numbered through, row r's from `from` on */
            unsigned int s = 0u, len = 0u;
            if (lane < 9) {
                const int o = ((lane / 3 - 1) * p.gy + (lane % 3 - 1)) * p.gx;
                const unsigned int a = (unsigned int)((int)first + o), b = (unsigned int)((int)last + o);
                if (cell_row_ok(p, a) && cell_row_ok(p, b)) {
                    s = __ldg(cell_start + (a - 1u));
                    len = bounded(p, __ldg(cell_start + (b + 2u)), (unsigned int)p.n + 1u, kBoundSlot) - s;
                }
            }
            unsigned int from = len;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                const unsigned int v = __shfl_up_sync(0xffffffffu, from, o);
                if (lane >= o) from += v;
            }
            const unsigned int total = __shfl_sync(0xffffffffu, from, 8);
            from -= len; /* lane 9 and on: the total */
            const unsigned int shift = s - from;
            /* the words from lo on, n of them */
            const unsigned int words = (total + 31u) >> 5, room = (unsigned int)(kTileWords - w), lo = resume;
            unsigned int n = words - lo;
            if (n > room) {
                if (w) break; /* after what the tile holds now */
                part = grp;
                n = room;
                resume = lo + room;
            } else {
                done |= grp;
                todo &= ~grp;
                resume = 0u;
            }
            const float ox = 0.5f * (__shfl_sync(0xffffffffu, xi.x, lead) + __shfl_sync(0xffffffffu, xi.x, tail));
            const float oy = __shfl_sync(0xffffffffu, xi.y, lead), oz = __shfl_sync(0xffffffffu, xi.z, lead);
            unsigned int a0[4], a1[4]; /* the slots' terms: rows 0-7, 8-15, 16-23, 24-31; terms 0-7 and 8-15 */
            {
                const PairTerms v = mine ? pair_terms((xi.x - ox) * inv, (xi.y - oy) * inv, (xi.z - oz) * inv)
                                         : PairTerms{0u, 0u, 0u, 0u, 0.0f};
                bad |= !(v.nn <= 64.0f);
                const unsigned int h0 = times_m2(v.h0), h1 = times_m2(v.h1), l0 = times_m2(v.l0), l1 = times_m2(v.l1);
                const unsigned int z1 = (h1 & 0xffffu) | (ones & 0xffff0000u); /* (-2 zh, 1) */
                __syncwarp(); /* the last operands of the turn before have been read */
                rows[lane] = make_uint4(h0, z1, h0, z1);
                __syncwarp();
                load_matrices(a0, rows + lane);
                __syncwarp();
                rows[lane] = make_uint4(l0, l1 & 0xffffu, __byte_perm(v.h1, v.l1, 0x7632),
                                         half_pair(-1.0f, -0x1p-12f));
                __syncwarp();
                load_matrices(a1, rows + lane);
            }
            const bool keep = (grp >> own & 1u) != 0u;
            int r = 0;
            /* this lane's candidate of the word from q0 on, its position on the way */
            auto fetch = [&](unsigned int q0, unsigned int &j) {
                const unsigned int q = q0 + (unsigned int)lane;
                j = q + __shfl_sync(0xffffffffu, shift, r);
                for (;;) { /* the rows that these 32 candidates reach into */
                    const unsigned int next = __shfl_sync(0xffffffffu, from, r + 1);
                    if (next >= q0 + 32u || r == 8) break;
                    ++r;
                    const unsigned int sh = __shfl_sync(0xffffffffu, shift, r);
                    if (q >= next) j = q + sh;
                }
                /* past the last candidate: some slot's position, not used */
                return load(min(q < total ? j : j - (q - total + 1u), (unsigned int)p.n - 1u));
            };
            /* this warp's words */
            const unsigned int begin = (lo + n * wid / W) * 32u, end = min(total, (lo + n * (wid + 1) / W) * 32u);
            unsigned int jn;
            float4 cn;
            if (W == 1 || begin < end) cn = fetch(begin, jn);
#pragma unroll 1
            for (unsigned int q0 = begin; q0 < end; q0 += 32u, w += W == 1 ? 1 : 0) {
                const int at = W == 1 ? w : w + (int)((q0 >> 5) - lo);
                const unsigned int q = q0 + (unsigned int)lane, j = jn;
                const float4 c = cn;
                if (q0 + 32u < end) cn = fetch(q0 + 32u, jn);
                PairTerms v{0x4f804f80u, 0x4f804f80u, 0u, 0u, 0.0f}; /* past the last candidate: 30 30 30, far away */
                if (q < total) {
                    v = pair_terms((c.x - ox) * inv, (c.y - oy) * inv, (c.z - oz) * inv);
                } else {
                    v.h1 = half_pair(30.0f, 2700.0f);
                }
                bad |= !(v.nn <= 64.0f);
                __syncwarp(); /* the operands of the last word have been read */
                *st = make_uint4(v.h0, v.h1, v.l0, v.l1);
                t.slot[at][lane] = j;
                __syncwarp();
                unsigned int b[4];
                load_matrices(b, ld);
                unsigned int m0 = 0u, m1 = 0u, m2 = 0u, m3 = 0u;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const unsigned int b1 = upper ? ones : b[k];
                    test_tile(m0, m1, a0[0], a0[1], a1[0], a1[1], b[k], b1);
                    test_tile(m2, m3, a0[2], a0[3], a1[2], a1[3], b[k], b1);
                }
                /* byte k of lane c: candidates 8c .. 8c + 7 of slot g + 8k; the quad's four
                 * lanes exchange bytes until lane c has all of slot g + 8c */
                unsigned int m = __byte_perm(__byte_perm(m0, m1, 0x0040), __byte_perm(m2, m3, 0x0040), 0x5410);
                m = __byte_perm(m, __shfl_xor_sync(0xffffffffu, m, 2), pick1);
                m = __byte_perm(m, __shfl_xor_sync(0xffffffffu, m, 1), pick2);
                if (!keep) m = 0u;
                t.mask[at][own] = m;
                cnt += __popc(m);
                if (m) any |= 0x80000000u >> at;
            }
            if (W > 1) w += (int)n;
            if (part) break;
        }
        const int holder = 4 * (lane & 7) + (lane >> 3); /* the lane that counted this lane's slot */
        const int count = __shfl_sync(0xffffffffu, cnt, holder);
        const unsigned int some = __shfl_sync(0xffffffffu, any, holder);
        int first = 0, all = count;
        bool found = !apart;
        if (W > 1) {
            t.cnt[wid][lane] = count;
            found = !__syncthreads_or(bad) && found;
            all = 0;
#pragma unroll
            for (int v = 0; v < W; ++v) {
                const int n = t.cnt[v][lane];
                if (v < wid) first += n;
                all += n;
            }
        } else {
            found = !__any_sync(0xffffffffu, bad) && found;
            __syncwarp();
        }
        if (!found) { /* whatever its earlier parts gave, the lane starts again */
            done |= part;
            todo &= ~part;
            part = resume = 0u;
        }
        if ((done | part) >> lane & 1u) {
            TileWalk<W> walk(t, some, count);
            emit(found, base + first, count, base + all, walk);
            base = (part >> lane & 1u) ? base + all : 0;
        }
        /* the tile is free again */
        if (W > 1)
            __syncthreads();
        else
            __syncwarp();
    }
}

/* The lists of a warp's 32 consecutive slots (i ascending over the lanes,
 * padding lanes last).  The entries leave four at a time, one 16-byte store
 * per lane and 512 consecutive bytes per warp; with W > 1 warps for the slots
 * one by one. */
template <int W>
__device__ __forceinline__ void build_list_warp(const DevParams &p, int i, bool valid,
                                                const unsigned int *__restrict__ cell_start,
                                                const float4 *__restrict__ xb,
                                                const unsigned int *__restrict__ cellb, ListEntry *__restrict__ list,
                                                unsigned char *__restrict__ cnt, PairTileOf<W> &t) {
    const float3 xi = valid ? f3(__ldg(xb + i)) : make_float3(0.f, 0.f, 0.f);
    const unsigned int cell = valid ? __ldg(cellb + i) : 0u;
    warp_candidates(p, cell_start, [&](unsigned int j) { return __ldg(xb + j); }, xi, cell, valid, p.rl2, t,
                    [&](bool found, int first, int count, int total, TileWalk<W> &walk) {
        if (!found) {
            if (W == 1 || threadIdx.x < 32u) build_list_body(p, i, cell_start, xb, cell, list, cnt);
            return;
        }
        if (W == 1 && first == 0) {
            const int most = min(count, kListMax);
            for (int k = 0; k < most; k += 4) {
                unsigned int v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = walk.next(); /* the last group is padded with its last entry */
                reinterpret_cast<uint4 *>(list)[(size_t)(k >> 2) * (size_t)p.n + (size_t)i] =
                    make_uint4(v[0], v[1], v[2], v[3]);
            }
        } else {
            unsigned int v = 0u;
            const int most = min(first + count, kListMax);
            for (int k = first; k < most; ++k) {
                v = walk.next();
                list[list_at(k, i, p.n)] = v;
            }
            if (count && first + count == total && total < kListMax) /* pad the last group */
                for (int k = total; (k & 3) != 0; ++k) list[list_at(k, i, p.n)] = v;
        }
        if (W == 1 || threadIdx.x < 32u) cnt[i] = total > kListMax ? kListOverflow : (unsigned char)total;
    });
}

/* ---------------- constraint iterations ---------------- */

/* Density, C, sum |grad C|^2 (with the k = i term) and lambda of one particle
 * at xi; returns C (every lane of a group gets the same values).
 * each(load, f) calls f(j, load(j)) for the lane's candidates. */
template <int LPP, bool KAHAN, class Each>
__device__ __forceinline__ float lambda_terms(const DevParams &p, const float4 *pp, float3 xi, Each &&each,
                                              float &rho_out, float &lam_out) {
    float wsum = 0.f, wc = 0.f, sd = 0.f;
    float3 gs = make_float3(0.f, 0.f, 0.f);
    const float agr = p.ag * p.inv_rest_dens;
#if FSPH_FOLD
    /* the pair loop sums g' = (h - r)^2 / r; the coefficient agr (grad W /
     * rho0 = agr g' d) multiplies the sums once after the loop */
    const float agl = 1.0f;
#else
    const float agl = agr;
#endif
    /* plain (L1-cached) loads: only the .w words of pp are written by this
     * pass, and the neighbour loop reads x, y, z */
    each(
        [&](unsigned int j) { return pp[j]; },
        [&](unsigned int, const float4 &xj4) {
            /* branch-free: outside h both q and t clamp to zero; the self
             * pair (d = 0) adds W(0) to the density and nothing else */
            const float3 d = xi - f3(xj4);
            const float r2 = dot3(d, d);
            const float q = fmaxf(p.h2 - r2, 0.0f);
            const float inv_r = pair_rsqrt(r2);
            const float t = fmaxf(p.h - r2 * inv_r, 0.0f);
            const float g = agl * t * t * inv_r; /* grad W / rho0 = (agr / agl) g d */
            if (KAHAN) { /* compensated sum of the density terms */
                const float y = q * q * q - wc;
                const float s = wsum + y;
                wc = (s - wsum) - y;
                wsum = s;
            } else {
                wsum += q * q * q;
            }
            gs = gs + g * d;
            sd += g * g * r2;
        });
    if (LPP > 1) {
        wsum = KAHAN ? group_sum_split<LPP>(wsum, -wc) : group_sum<LPP>(wsum);
        sd = group_sum<LPP>(sd);
        gs.x = group_sum<LPP>(gs.x);
        gs.y = group_sum<LPP>(gs.y);
        gs.z = group_sum<LPP>(gs.z);
    }
    float rho = p.mass * p.aw * wsum;
    /* the roundings spelt out: a compiler may fuse either product of x x + y y, or
     * this scaling with what is added below, and every kernel has to agree */
    sd = __fadd_rn(sd, __fmaf_rn(gs.z, gs.z, __fmaf_rn(gs.y, gs.y, __fmul_rn(gs.x, gs.x))));
#if FSPH_FOLD
    sd = __fmul_rn(sd, agr * agr);
#endif
    if (p.nb) {
        /* boundary particles (rx_sph_pbd.cpp:728-748, 795-818): density
         * rho0 psi_b W and |grad C|^2 terms of (rho0 psi_b / m) grad W / rho0,
         * each boundary neighbour counted once (rx_pbdsph_kernel.cu:577-664);
         * every lane of a group sums them (they are few) */
        float bw = 0.f;
        for_each_boundary(p, xi, [&](unsigned int, const float4 &b4) {
            const float3 d = xi - f3(b4);
            const float r2 = dot3(d, d);
            const float q = fmaxf(p.h2 - r2, 0.0f);
            const float inv_r = pair_rsqrt(r2);
            const float t = fmaxf(p.h - r2 * inv_r, 0.0f);
            const float gb = b4.w * agr * t * t * inv_r;
            bw += b4.w * q * q * q;
            sd += gb * gb * r2;
        });
        rho += p.mass * p.aw * bw;
    }
    float C = rho * p.inv_rest_dens - 1.0f;
    float Cc = (p.clamp_constraint && C < 0.0f) ? 0.0f : C;
    rho_out = rho;
    lam_out = -Cc / (sd + p.epsilon);
    return C;
}

/* lambda pass of one particle: lambda into x*.w and rho into dens (lane 0 of a
 * valid group).  Returns C (the caller turns it into the error terms). */
template <int LPP, bool KAHAN = false, bool DEEP = false>
__device__ __forceinline__ float lambda_body(const DevParams &p, const unsigned int *__restrict__ cell_start,
                                             float4 *pp, float *__restrict__ dens, DevCtl *ctl,
                                             const ListEntry *__restrict__ list,
                                             const unsigned char *__restrict__ cnt, int i, int sub, bool valid) {
    const float3 xi = f3(pp[i]);
    float rho, lam;
    const float C = lambda_terms<LPP, KAHAN>(
        p, pp, xi,
        [&](auto &&load, auto &&f) { for_each_candidate<LPP, DEEP>(p, cell_start, list, cnt, i, xi, sub, load, f); },
        rho, lam);
    if (valid && sub == 0) {
        reinterpret_cast<float *>(pp + i)[3] = lam;
        dens[i] = rho;
        if (!(rho == rho)) ctl->nan_flag = 1u;
    }
    return C;
}

/* End of the lambda pass: block partial errors; the last block reduces them
 * in a fixed order, advances the iteration counter and decides whether the
 * device-side loop continues (lp: the loop constants).  Every thread of the
 * block calls it. */
__device__ __forceinline__ void lambda_tail(const DevParams &lp, DevCtl *ctl, ErrPartial *part, float e1, float e2,
                                            float em, cudaGraphConditionalHandle hwhile, int use_graph) {
    __shared__ float sh1[32], sh2[32], shm[32];
    __shared__ double d1[32], d2[32];
    __shared__ int s_last;
    e1 = warp_sum(e1);
    e2 = warp_sum(e2);
    em = warp_max(em);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) { sh1[warp] = e1; sh2[warp] = e2; shm[warp] = em; }
    __syncthreads();
    if (threadIdx.x == 0) {
        float a = 0.f, b = 0.f, m = 0.f;
        for (int w = 0; w < nw; ++w) { a += sh1[w]; b += sh2[w]; m = fmaxf(m, shm[w]); }
        part[blockIdx.x] = ErrPartial{a, b, m, 0.f};
        __threadfence();
        unsigned int t = atomicAdd(&ctl->ticket, 1u);
        s_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    /* fixed-order reduction of the block partials (double): strided per
     * thread, a shuffle tree per warp, then the warps in order */
    double a = 0.0, b = 0.0;
    float m = 0.f;
    for (unsigned int k = threadIdx.x; k < gridDim.x; k += blockDim.x) {
        float4 v = __ldcg(reinterpret_cast<const float4 *>(part) + k);
        a += v.x; b += v.y; m = fmaxf(m, v.z);
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    if (lane == 0) { d1[warp] = a; d2[warp] = b; shm[warp] = m; }
    __syncthreads();
    if (threadIdx.x == 0) {
        a = 0.0; b = 0.0; m = 0.f;
        for (int w = 0; w < nw; ++w) { a += d1[w]; b += d2[w]; m = fmaxf(m, shm[w]); }
        float err1 = (float)(a / (double)lp.n);
        float err2 = (float)(b / (double)lp.n);
        ctl->err1 = err1;
        ctl->err2 = err2;
        ctl->errmax = m;
        unsigned int it = ctl->iter + 1u;
        ctl->iter = it;
        float err = lp.error_mode ? err2 : err1;
        int minit = lp.min_iter > 1 ? lp.min_iter : 1;
        int cont = ((int)it < lp.max_iter) && !(err <= lp.eta && (int)it >= minit);
        if (ctl->nan_flag) cont = 0;
        ctl->done = cont ? 0u : 1u;
        ctl->ticket = 0u;
        if (use_graph & 1) cudaGraphSetConditional(hwhile, cont ? 1u : 0u);
    }
}

/* |C| in units of 2^-32, saturating (a diverged step is caught by the NaN
 * flag and the error itself) */
__device__ __forceinline__ unsigned long long err_fix(float x) {
    return (unsigned long long)__float2ll_rn(fminf(x, 1024.0f) * 4294967296.0f);
}
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
/* The next 32 slots of a persistent pass (warp-uniform): round-robin while whole
 * rounds last (stat), the rest on demand, so that warps that finish early take the
 * leftovers; the error sums are fixed point (units of 2^-32), exact and so
 * independent of which warp ran which chunk. */
__device__ __forceinline__ int next_chunk(int c, int nw, int stat, unsigned int *ctr, int lane) {
    c += nw;
    if (c < stat) return c;
    unsigned int v = 0u;
    if (lane == 0) v = atomicAdd(ctr, 1u);
    return stat + (int)__shfl_sync(0xffffffffu, v, 0);
}

/* lambda_tail for fixed-point error sums: integer sums are exact, so the
 * block partials may combine in any order */
__device__ __forceinline__ void lambda_tail_fix(const DevParams &lp, DevCtl *ctl, ErrPartial *part,
                                                unsigned long long q1, unsigned long long q2, float em,
                                                cudaGraphConditionalHandle hwhile, int use_graph) {
    __shared__ unsigned long long sq1[32], sq2[32];
    __shared__ float shm[32];
    __shared__ int s_last;
    ErrPartialFix *pf = reinterpret_cast<ErrPartialFix *>(part);
    q1 = warp_sum_u64(q1);
    q2 = warp_sum_u64(q2);
    em = warp_max(em);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) { sq1[warp] = q1; sq2[warp] = q2; shm[warp] = em; }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long a = 0ull, b = 0ull;
        float m = 0.f;
        for (int w = 0; w < nw; ++w) { a += sq1[w]; b += sq2[w]; m = fmaxf(m, shm[w]); }
        pf[blockIdx.x].s1 = a;
        pf[blockIdx.x].s2 = b;
        pf[blockIdx.x].mx = m;
        __threadfence();
        unsigned int t = atomicAdd(&ctl->ticket, 1u);
        s_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    unsigned long long a = 0ull, b = 0ull;
    float m = 0.f;
    for (unsigned int k = threadIdx.x; k < gridDim.x; k += blockDim.x) {
        a += __ldcg(&pf[k].s1);
        b += __ldcg(&pf[k].s2);
        m = fmaxf(m, __ldcg(&pf[k].mx));
    }
    a = warp_sum_u64(a);
    b = warp_sum_u64(b);
    m = warp_max(m);
    __syncthreads(); /* every warp has read its shared entries above */
    if (lane == 0) { sq1[warp] = a; sq2[warp] = b; shm[warp] = m; }
    __syncthreads();
    if (threadIdx.x == 0) {
        a = 0ull; b = 0ull; m = 0.f;
        for (int w = 0; w < nw; ++w) { a += sq1[w]; b += sq2[w]; m = fmaxf(m, shm[w]); }
        float err1 = (float)((double)a * 0x1p-32 / (double)lp.n);
        float err2 = (float)((double)b * 0x1p-32 / (double)lp.n);
        ctl->err1 = err1;
        ctl->err2 = err2;
        ctl->errmax = m;
        unsigned int it = ctl->iter + 1u;
        ctl->iter = it;
        float err = lp.error_mode ? err2 : err1;
        int minit = lp.min_iter > 1 ? lp.min_iter : 1;
        int cont = ((int)it < lp.max_iter) && !(err <= lp.eta && (int)it >= minit);
        if (ctl->nan_flag) cont = 0;
        ctl->done = cont ? 0u : 1u;
        ctl->ticket = 0u;
        ctl->grab = 0u; /* every block has passed its loop: the counter is free for the next pass */
        if (use_graph & 1) cudaGraphSetConditional(hwhile, cont ? 1u : 0u);
    }
}

/* dp_i = sum_j (lambda_i + lambda_j + s_corr) grad W_ij / rho0 of one particle
 * at xi with lambda li (every lane of a group gets it). */
template <int LPP, class Each>
__device__ __forceinline__ float3 correction_terms(const DevParams &p, const float4 *src, float3 xi, float li,
                                                   Each &&each) {
    float3 acc = make_float3(0.f, 0.f, 0.f);
    const float k_dt2 = -p.ap_k * p.dt * p.dt;
    const float agr = p.ag * p.inv_rest_dens;
    const float awq = p.aw * p.inv_wq;
#if FSPH_FOLD
    /* agr multiplies the sum once after the loop; for n = 4 the tensile
     * term -k dt^2 (awq q^3)^4 is K q^12 with K = -k dt^2 awq^4 (|K| ~ 1e26
     * for the configured h, well inside FP32) */
    const float agl = 1.0f;
    const float awq2 = awq * awq;
    const float k12 = k_dt2 * (awq2 * awq2);
#else
    const float agl = agr;
#endif
    each(
        [&](unsigned int j) { return src[j]; },
        [&](unsigned int, const float4 &xj4) {
            /* branch-free: t = 0 outside h and d = 0 for the self pair */
            const float3 d = xi - f3(xj4);
            const float r2 = dot3(d, d);
            const float inv_r = pair_rsqrt(r2);
            const float t = fmaxf(p.h - r2 * inv_r, 0.0f);
            const float g = agl * t * t * inv_r;
            float coef = li + xj4.w;
            if (p.use_ap) {
                const float q = fmaxf(p.h2 - r2, 0.0f);
#if FSPH_FOLD
                if (p.ap_n == 4.0f) {
                    const float q2 = q * q, q4 = q2 * q2;
                    coef = fmaf(k12, (q4 * q4) * q4, coef);
                } else {
                    coef += k_dt2 * __powf(awq * q * q * q, p.ap_n);
                }
#else
                const float ww = awq * q * q * q;
                const float pw = (p.ap_n == 4.0f) ? (ww * ww) * (ww * ww) : __powf(ww, p.ap_n);
                coef += k_dt2 * pw;
#endif
            }
            acc = acc + (coef * g) * d;
        });
    if (LPP > 1) {
        acc.x = group_sum<LPP>(acc.x);
        acc.y = group_sum<LPP>(acc.y);
        acc.z = group_sum<LPP>(acc.z);
    }
#if FSPH_FOLD
    acc = make_float3(__fmul_rn(agr, acc.x), __fmul_rn(agr, acc.y), __fmul_rn(agr, acc.z)); /* as in lambda_terms */
#endif
    if (p.nb) {
        /* boundary terms (rx_sph_pbd.cpp:977-1019): lambda_b, and s_corr of
         * the (rho0 psi_b / m)-scaled W */
        float3 accb = make_float3(0.f, 0.f, 0.f);
        for_each_boundary(p, xi, [&](unsigned int b, const float4 &b4) {
            const float3 d = xi - f3(b4);
            const float r2 = dot3(d, d);
            const float inv_r = pair_rsqrt(r2);
            const float t = fmaxf(p.h - r2 * inv_r, 0.0f);
            const float g = agr * t * t * inv_r;
            float sc = 0.0f;
            if (p.use_ap) {
                const float q = fmaxf(p.h2 - r2, 0.0f);
                const float ww = b4.w * awq * q * q * q;
                const float pw = (p.ap_n == 4.0f) ? (ww * ww) * (ww * ww) : __powf(ww, p.ap_n);
                sc = k_dt2 * pw;
            }
            accb = accb + ((li + __ldg(p.blam + b) + sc) * g) * d;
        });
        acc = acc + accb;
    }
    return acc;
}

/* correction pass of one particle: x*_i <- walls(x*_i + dp_i) into dst (lane 0
 * of a valid group).  Returns |x*_i - xb_i|^2 (0 for the other lanes). */
template <int LPP, bool DEEP = false>
__device__ __forceinline__ float correction_body(const DevParams &p, const unsigned int *__restrict__ cell_start,
                                                 const float4 *__restrict__ src, float4 *__restrict__ dst,
                                                 const float4 *__restrict__ xb, DevCtl *ctl,
                                                 float4 *__restrict__ dp_out, const ListEntry *__restrict__ list,
                                                 const unsigned char *__restrict__ cnt, int i, int sub, bool valid) {
    const float4 xi4 = src[i];
    const float3 xi = f3(xi4);
    const float3 acc = correction_terms<LPP>(p, src, xi, xi4.w, [&](auto &&load, auto &&f) {
        for_each_candidate<LPP, DEEP>(
            p, cell_start, list, cnt, i, xi, sub, [&](unsigned int j) { return __ldg(src + j); }, f);
        (void)load;
    });
    if (!valid || sub != 0) return 0.0f;
    if (dp_out) dp_out[i] = make_float4(acc.x, acc.y, acc.z, 0.0f);
    float3 xn = solid_project(xi + acc, p);
    dst[i] = make_float4(xn.x, xn.y, xn.z, 0.0f);
    float3 dd = xn - f3(xb[i]);
    if (!(xn.x == xn.x && xn.y == xn.y && xn.z == xn.z)) ctl->nan_flag = 1u;
    return dot3(dd, dd);
}

/* End of the correction pass: the largest displacement measure of the block;
 * the last block compares the maximum with lp.skin2 (a rebuild is due above
 * it), flips the x* parity and sets the graph's rebuild conditions.  Every
 * thread of the block calls it. */
__device__ __forceinline__ void correction_tail(const DevParams &lp, DevCtl *ctl, float *part, float disp2,
                                                unsigned int par, cudaGraphConditionalHandle hif,
                                                cudaGraphConditionalHandle hif2, int use_graph) {
    __shared__ float shm[32];
    __shared__ int s_last;
    disp2 = warp_max(disp2);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) shm[warp] = disp2;
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = 0.f;
        for (int w = 0; w < nw; ++w) m = fmaxf(m, shm[w]);
        part[blockIdx.x] = m;
        __threadfence();
        unsigned int t = atomicAdd(&ctl->ticket2, 1u);
        s_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    float m = 0.f;
    for (unsigned int k = threadIdx.x; k < gridDim.x; k += blockDim.x) m = fmaxf(m, __ldcg(part + k));
    m = warp_max(m);
    __syncthreads(); /* every warp has read its shm entry above */
    if (lane == 0) shm[warp] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float md = 0.f;
        for (int w = 0; w < nw; ++w) md = fmaxf(md, shm[w]);
        ctl->disp2_bits = __float_as_uint(md);
        unsigned int rb = (md > lp.skin2 || !(md == md)) ? 1u : 0u;
        ctl->rebuild = rb;
        ctl->parity = 1u - par;
        ctl->ticket2 = 0u;
        if (use_graph & 1) {
            unsigned int more = ctl->done ? 0u : 1u;
            cudaGraphSetConditional(hif, rb & more);
            if (use_graph & 2) cudaGraphSetConditional(hif2, rb);
        }
    }
}

/* ---------------- end of step ---------------- */

/* omega_i = sum_j (m / rho_j)(v_j - v_i) x grad_j W_ij (grad_j = -grad_i):
 * the SPH curl of v, each neighbour weighted by its volume m / rho_j as in
 * the XSPH sum and the eta gradient below (Macklin & Mueller 2013, eq. 15,
 * writes the sum without the volume, whose scale their eps absorbs; in
 * SI units that sum is ~1e5 times the curl at h = 0.0457 and the configured
 * eps = 1e-4 then drives the flow unstable).  The XSPH update
 * v_i + c sum_j (m / rho_j)(v_j - v_i) W_ij, and (fo.feat) the warm-start
 * features of the particle. */
/* PRE: pos[j].w is m / rho_j (written once per particle by k_finalize, the
 * same correctly rounded quotient), and the pass leaves |omega_i| in mag for
 * vort_apply_body<true>; else a division per pair.  FEAT: the features are
 * wanted, NBR: with the neighbour means.
 * Both passes are bound as the constraint passes are, by the L1 wavefronts of
 * their gathers (78 % and 68 % of the unit's peak while active at 262,144
 * particles with m / rho in an array of its own and the features' sums always
 * kept): two gathers a pair here and one and a 4-byte one there, all of a
 * group's in flight before its first pair.  262,144 particles 37.0 -> 32.5 us
 * and 31.9 -> 26.8, 16.8 M particles 1656 -> 1554 and 1188 -> 1056. */
struct PosVel {
    float4 x, v;
};
template <bool FEAT, bool NBR, bool PRE, bool DEEP = false>
__device__ __forceinline__ void xsph_vort_body(const DevParams &p, int i, const unsigned int *__restrict__ cell_start,
                                               const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                                               const float *__restrict__ dens, float4 *__restrict__ vel_out,
                                               float4 *__restrict__ vort, const FeatureOut &fo,
                                               const ListEntry *__restrict__ list,
                                               const unsigned char *__restrict__ cnt, float *__restrict__ mag) {
    const float3 xi = f3(pos[i]), vi = f3(vel[i]);
    float3 om = make_float3(0.f, 0.f, 0.f), xs = make_float3(0.f, 0.f, 0.f);
    float3 off = make_float3(0.f, 0.f, 0.f), cg = make_float3(0.f, 0.f, 0.f);
    float cntf = 0.f;
    float wpred = 0.f; /* sum q^3 at the next step's predicted relative positions */
    /* poly6-weighted neighbour sums (self excluded) for the features:
     * weights, density, relative velocity, step correction */
    float nw = 0.f, nrho = 0.f;
    float3 nv = make_float3(0.f, 0.f, 0.f), nd = make_float3(0.f, 0.f, 0.f);
    /* branch-free pair terms: q and t clamp to zero outside h, and the self
     * pair (d = 0, v_ij = 0) adds only to the neighbour count */
    for_each_candidate<1, DEEP>(
        p, cell_start, list, cnt, i, xi, 0, [&](unsigned int j) { return PosVel{__ldg(pos + j), __ldg(vel + j)}; },
        [&](unsigned int j, const PosVel &b) {
            const float3 d = xi - f3(b.x);
            const float r2 = dot3(d, d);
            const float q = fmaxf(p.h2 - r2, 0.0f);
            const float inv_r = pair_rsqrt(r2);
            const float t = fmaxf(p.h - r2 * inv_r, 0.0f);
            const float g = p.ag * t * t * inv_r;
            const float3 vij = f3(b.v) - vi;
            const float rhoj = (NBR || !PRE) ? __ldg(dens + j) : 0.0f;
            const float mrho = PRE ? b.x.w : p.mass / rhoj;
            om = om + cross3(vij, (-g * mrho) * d);
            xs = xs + (p.aw * q * q * q * mrho) * vij;
            if (FEAT) {
                const float inside = r2 < p.h2 ? 1.0f : 0.0f;
                cntf += inside;
                off = off - inside * d;
                /* the pair at the next step's prediction x + dt v (gravity cancels
                 * in relative positions): poly6 and its spiky gradient there */
                const float3 ds = d - p.dt * vij;
                const float r2s = dot3(ds, ds);
                const float qs = fmaxf(p.h2 - r2s, 0.0f);
                const float inv_rs = pair_rsqrt(r2s);
                const float ts = fmaxf(p.h - r2s * inv_rs, 0.0f);
                wpred += qs * qs * qs;
                cg = cg + (p.ag * ts * ts * inv_rs) * ds;
                if (NBR) {
                    const float w = r2 > 0.0f ? q * q * q : 0.0f;
                    nw += w;
                    nrho += w * rhoj;
                    nv = nv + w * vij;
                    nd = nd + w * f3(__ldg(fo.dstep + j));
                }
            }
        });
    float3 vn = vi + p.xsph_c * xs;
    vel_out[i] = make_float4(vn.x, vn.y, vn.z, 0.0f);
    vort[i] = make_float4(om.x, om.y, om.z, 0.0f);
    if (PRE) mag[i] = sqrtf(dot3(om, om));
    if (FEAT) {
        cntf = fmaxf(cntf, 1.0f);
        /* warm-start features at the end of the step (dimensionless; see kFeatures) */
        const float inv_h = 1.0f / p.h;
        const float4 *pl = fo.ctl->parity ? fo.ppos0 : fo.ppos1; /* buffer of the last lambda pass */
        const float3 dd = f3(fo.dstep[i]);
        float f[kFeatures];
        f[0] = dens[i] * p.inv_rest_dens - 1.0f;
        f[1] = pl[i].w * p.rest_dens * p.h2;
        f[2] = cntf * (1.0f / 33.0f);
        f[3] = off.x * inv_h / cntf; f[4] = off.y * inv_h / cntf; f[5] = off.z * inv_h / cntf;
        f[6] = vi.x * p.dt * inv_h; f[7] = vi.y * p.dt * inv_h; f[8] = vi.z * p.dt * inv_h;
        f[9] = dd.x * inv_h; f[10] = dd.y * inv_h; f[11] = dd.z * inv_h;
        /* predicted constraint C' = rho' / rho0 - 1 and h grad_i C' at the next prediction */
        const float mr0 = p.mass * p.inv_rest_dens;
        f[12] = mr0 * p.aw * wpred - 1.0f;
        f[13] = mr0 * cg.x * p.h; f[14] = mr0 * cg.y * p.h; f[15] = mr0 * cg.z * p.h;
        /* weighted neighbour means of features 0, 6-8 and 9-11 (zero without neighbours) */
        const float inw = nw > 0.0f ? 1.0f / nw : 0.0f;
        const float vs = p.dt * inv_h;
        f[16] = nw > 0.0f ? nrho * inw * p.inv_rest_dens - 1.0f : 0.0f;
        f[17] = nw > 0.0f ? (vi.x + nv.x * inw) * vs : 0.0f;
        f[18] = nw > 0.0f ? (vi.y + nv.y * inw) * vs : 0.0f;
        f[19] = nw > 0.0f ? (vi.z + nv.z * inw) * vs : 0.0f;
        f[20] = nd.x * inw * inv_h; f[21] = nd.y * inw * inv_h; f[22] = nd.z * inw * inv_h;
#pragma unroll
        for (int k = 23; k < kFeatures; ++k) f[k] = 0.0f;
        float4 *out = reinterpret_cast<float4 *>(fo.feat + (size_t)i * kFeatures);
#pragma unroll
        for (int k = 0; k < kFeatures / 4; ++k) out[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
        if (i == 0) *fo.valid = 1u;
    }
}

/* eta_i = sum_j (m / rho_j)(|w_j| - |w_i|) grad_i W_ij; f = eps (eta/|eta|) x w_i;
 * v_i <- v_i + dt f. */
/* PRE: |omega_j| from mag (what xsph_vort_body wrote) and m / rho_j from
 * pos[j].w, so neither a division nor a square root per pair. */
template <bool PRE = false, bool DEEP = false>
__device__ __forceinline__ void vort_apply_body(const DevParams &p, int i, const unsigned int *__restrict__ cell_start,
                                                const float4 *__restrict__ pos, const float4 *__restrict__ vort,
                                                const float *__restrict__ dens, const float4 *__restrict__ vel_in,
                                                float4 *__restrict__ vel_out, const ListEntry *__restrict__ list,
                                                const unsigned char *__restrict__ cnt,
                                                const float *__restrict__ mag) {
    float4 v4 = vel_in[i];
    if (p.vort_eps != 0.0f) {
        const float3 xi = f3(pos[i]);
        const float3 wi = f3(vort[i]);
        const float wmi = sqrtf(dot3(wi, wi));
        float3 eta = make_float3(0.f, 0.f, 0.f);
        struct PosMag {
            float4 x;
            float w;
        };
        for_each_candidate<1, DEEP>(
            p, cell_start, list, cnt, i, xi, 0,
            [&](unsigned int j) { return PosMag{__ldg(pos + j), PRE ? __ldg(mag + j) : 0.0f}; },
            [&](unsigned int j, const PosMag &b) {
                const float3 d = xi - f3(b.x);
                const float r2 = dot3(d, d);
                const float inv_r = pair_rsqrt(r2);
                const float t = fmaxf(p.h - r2 * inv_r, 0.0f);
                const float g = p.ag * t * t * inv_r;
                float k;
                if (PRE) {
                    k = b.x.w * (b.w - wmi) * g;
                } else {
                    const float3 wj = f3(__ldg(vort + j));
                    k = p.mass / __ldg(dens + j) * (sqrtf(dot3(wj, wj)) - wmi) * g;
                }
                eta = eta + k * d;
            });
        float en = sqrtf(dot3(eta, eta));
        if (en > 1e-30f) {
            float3 N = (1.0f / en) * eta;
            float3 f = p.vort_eps * cross3(N, wi);
            v4.x += p.dt * f.x;
            v4.y += p.dt * f.y;
            v4.z += p.dt * f.z;
        }
    }
    vel_out[i] = v4;
}

}  // namespace fsph

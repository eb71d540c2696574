/*
 * fsph_kernels.cu -- sm_103a kernels of the fluid step.
 *
 * One thread per particle in device (cell-sorted) order: the 32 lanes of a
 * warp are 32 consecutive slots, i.e. neighbouring particles of the same few
 * cells, so their nine candidate row ranges mostly coincide and the
 * candidate float4 loads are served by L1 / L2 broadcasts (the whole x*
 * array of a 1M-particle scene is 16 MB and stays resident in the 126 MB L2).
 *
 * Kernel-by-kernel correspondence with the reference:
 *   k_predict_hash     rxPBDSPH::integrate (rx_sph_pbd.cpp:1409-1446) fused with
 *                      calcHashD2 (rx_sph_kernel.cu:54-73)
 *   k_scan / scatter   thrust::sort_by_key + reorderDataAndFindCellStartD
 *                      (rx_cu_funcs.cu:255-260, rx_sph_kernel.cu:108-153)
 *   k_lambda           calScalingFactor (rx_sph_pbd.cpp:699-914) fused with the
 *                      density-error reduction (rx_sph_pbd.cpp:448-454,
 *                      rx_pbdsph_kernel.cu:431-441) and the loop test
 *   k_correction       calPositionCorrection (rx_sph_pbd.cpp:925-1026) fused with
 *                      the position update and wall projection (rx_sph_pbd.cpp:436-445)
 *   k_finalize         velocity / position update (rx_sph_pbd.cpp:464-471)
 *   k_xsph_vort        xsphVisocosity (rx_pbdsph_kernel.cu:1130-1162) + vorticity
 *   k_sph_*            rxSPH::calDensity / calForce / integrate (rx_sph_cpu.cpp:495-1077)
 */
#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>

#include "fsph_kernels.cuh"
#include "fsph_passes.cuh"

namespace fsph {

/* ======================================================================== */
/* grid build                                                               */
/* ======================================================================== */

__global__ void k_predict_hash(DevParams p, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                               const float4 *__restrict__ acc, float4 *__restrict__ ppos_out,
                               unsigned int *__restrict__ key, unsigned int *__restrict__ rank,
                               unsigned int *__restrict__ count, const float4 *__restrict__ dwarm,
                               float4 *__restrict__ xpred_out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    predict_body(p, i, pos, vel, acc, ppos_out, key, rank, count, dwarm, xpred_out);
}

__global__ void k_hash(DevParams p, const float4 *__restrict__ x4, unsigned int *__restrict__ key,
                       unsigned int *__restrict__ rank, unsigned int *__restrict__ count) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    hash_body(p, i, f3(x4[i]), key, rank, count);
}

/* exclusive prefix of v over the 1024 threads of a block; total: the block's sum */
__device__ __forceinline__ unsigned int block_scan(unsigned int v, unsigned int &total) {
    __shared__ unsigned int warp_tot[32];
    __shared__ unsigned int s_total;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        unsigned int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        unsigned int w = warp_tot[lane];
        unsigned int wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            unsigned int y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        warp_tot[lane] = wi - w; /* exclusive prefix of the warps */
        if (lane == 31) s_total = wi;
    }
    __syncthreads();
    total = s_total;
    return warp_tot[warp] + incl - v;
}

/* Scan phase 1: a block scans kScanTile = 4096 counts and zeroes them; a thread
 * takes four 16-byte words 4 KB apart (count and out are 16-byte aligned arrays),
 * all in flight, and the 32 runs of 128 cells meet in one warp.  A table of one
 * tile ends here: the block also writes the grand total to out[ncells].  With 1024
 * threads of one word each, two blocks per SM waited at their barriers with
 * nothing in flight: 32.5 M cells 281 -> 111 us, 280,000 8.1 -> 4.1 (phase 3,
 * changed the same way, 38 -> 33 and 4.1 -> 3.3). */
__global__ void __launch_bounds__(kScanBlock) k_scan_local(unsigned int *__restrict__ count,
                                                           unsigned int *__restrict__ out,
                                                           unsigned int *__restrict__ block_sums,
                                                           unsigned int ncells) {
    __shared__ unsigned int run_tot[32], s_total;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int base = blockIdx.x * kScanTile + threadIdx.x * 4;
    uint4 v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const unsigned int at = base + r * (kScanBlock * 4);
        v[r] = make_uint4(0u, 0u, 0u, 0u);
        if (at + 4 <= ncells) {
            v[r] = *reinterpret_cast<const uint4 *>(count + at);
        } else if (at < ncells) {
            v[r].x = count[at];
            if (at + 1 < ncells) v[r].y = count[at + 1];
            if (at + 2 < ncells) v[r].z = count[at + 2];
        }
    }
    unsigned int before[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const unsigned int at = base + r * (kScanBlock * 4);
        if (at + 4 <= ncells) {
            *reinterpret_cast<uint4 *>(count + at) = make_uint4(0u, 0u, 0u, 0u);
        } else {
            for (unsigned int k = at; k < ncells; ++k) count[k] = 0u;
        }
        const unsigned int own = v[r].x + v[r].y + v[r].z + v[r].w;
        unsigned int incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        before[r] = incl - own;
        if (lane == 31) run_tot[r * (kScanBlock / 32) + warp] = incl;
    }
    __syncthreads();
    if (warp == 0) {
        const unsigned int own = run_tot[lane];
        unsigned int incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        run_tot[lane] = incl - own;
        if (lane == 31) s_total = incl;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const unsigned int at = base + r * (kScanBlock * 4);
        const unsigned int run = run_tot[r * (kScanBlock / 32) + warp] + before[r];
        const uint4 e = make_uint4(run, run + v[r].x, run + v[r].x + v[r].y, run + v[r].x + v[r].y + v[r].z);
        if (at + 4 <= ncells) {
            *reinterpret_cast<uint4 *>(out + at) = e;
        } else if (at < ncells) {
            out[at] = e.x;
            if (at + 1 < ncells) out[at + 1] = e.y;
            if (at + 2 < ncells) out[at + 2] = e.z;
        }
    }
    if (threadIdx.x == 0) {
        block_sums[blockIdx.x] = s_total;
        if (gridDim.x == 1) out[ncells] = s_total;
    }
}

/* Scan phase 2: one block scans the block totals; writes the grand total to out[ncells]. */
__global__ void __launch_bounds__(1024) k_scan_top(unsigned int *__restrict__ block_sums, unsigned int nblocks,
                                                   unsigned int *__restrict__ out, unsigned int ncells) {
    const int per = (nblocks + 1023) / 1024;
    const unsigned int start = threadIdx.x * per;
    unsigned int t = 0;
    for (int k = 0; k < per; ++k)
        if (start + k < nblocks) t += block_sums[start + k];
    unsigned int total;
    unsigned int run = block_scan(t, total);
    if (threadIdx.x == 0) out[ncells] = total;
    for (int k = 0; k < per; ++k)
        if (start + k < nblocks) {
            unsigned int b = block_sums[start + k];
            block_sums[start + k] = run;
            run += b;
        }
}

/* Scan phase 3: block b adds the total before its tile.  SUM: the totals are
 * still the tiles' own (no phase 2 has run), so the block sums the b totals
 * before it; the last block writes the grand total. */
template <bool SUM>
__global__ void __launch_bounds__(kScanBlock) k_scan_add(unsigned int *__restrict__ out,
                                                         const unsigned int *__restrict__ block_sums,
                                                         unsigned int ncells) {
    __shared__ unsigned int s_sum[kScanBlock / 32];
    const unsigned int base = blockIdx.x * kScanTile + threadIdx.x * 4;
    uint4 v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const unsigned int at = base + r * (kScanBlock * 4);
        if (at + 4 <= ncells) v[r] = *reinterpret_cast<const uint4 *>(out + at);
    }
    unsigned int add = 0u;
    if (SUM) {
        unsigned int t = 0u;
        for (unsigned int k = threadIdx.x; k < blockIdx.x; k += kScanBlock) t += block_sums[k];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = t;
        __syncthreads();
        for (int w = 0; w < kScanBlock / 32; ++w) add += s_sum[w];
        if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) out[ncells] = add + block_sums[blockIdx.x];
    } else {
        add = block_sums[blockIdx.x];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const unsigned int at = base + r * (kScanBlock * 4);
        if (at + 4 <= ncells) {
            v[r].x += add; v[r].y += add; v[r].z += add; v[r].w += add;
            *reinterpret_cast<uint4 *>(out + at) = v[r];
        } else {
            for (unsigned int k = at; k < ncells; ++k) out[k] += add;
        }
    }
}

__global__ void k_scatter(int n, const unsigned int *__restrict__ key, const unsigned int *__restrict__ rank,
                          const unsigned int *__restrict__ cell_start, unsigned int *__restrict__ perm) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    perm[cell_start[key[i]] + rank[i]] = (unsigned int)i;
}

/* The atomic ranks order a cell's slots arbitrarily.  Counting, for each
 * scattered entry, the smaller previous slots of its cell gives its place in
 * the stable order of the 64-bit key (cell << 32 | previous slot), identical
 * on every run.  Every entry counts for itself (about 10 independent loads,
 * one or two lines), so the kernel that moves the particles does it on the
 * way and no kernel sorts the cells.  One thread per cell, an insertion
 * sort in global memory (a serial chain of dependent loads and stores) had
 * taken 27 us at 4,096 particles, 37 us at 1 M and 110 us for the 4.7 M of a
 * batch; whole calls went from 102.6 to 83.7 us (lambda pass, 4,096), 568 to
 * 548 us (PBF step, 262 k) and 5,755 to 5,658 us (batch step).
 * s: the previous slot of scattered entry u; returns its slot in the order. */
__device__ __forceinline__ unsigned int ranked_slot(unsigned int u, const CellOrder &o, unsigned int &s) {
    s = o.perm[u];
    if (!o.key) return u; /* perm is the order itself (radix sort, partition) */
    const unsigned int c = o.key[s];
    const unsigned int a = o.cell_start[c], e = o.cell_start[c + 1];
    unsigned int d = a;
    for (unsigned int v = a; v < e; ++v) d += o.perm[v] < s ? 1u : 0u;
    return d;
}

__global__ void k_gather(int n, CellOrder o, Gather g, DevCtl *count_build) {
    int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u == 0 && count_build) count_build->builds += 1u;
    if (u >= n) return;
    unsigned int s;
    const unsigned int d = ranked_slot((unsigned int)u, o, s);
    if (o.sorted) o.sorted[d] = s;
#pragma unroll
    for (int k = 0; k < 6; ++k)
        if (k < g.n4) g.dst4[k][d] = g.src4[k][s];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k < g.n1) g.dst1[k][d] = g.src1[k][s];
}

/* The whole grid build of a small cloud in one block: cells counted, scanned,
 * filled and ranked in shared memory, x4 copied to its slots, the cell table
 * and the order written out.  The slot order is ranked_slot's.  Five launches
 * and a memset, each a few microseconds of launch and latency around almost no
 * work, become one: a call on 4,096 particles 36 -> 22 us. */
__global__ void __launch_bounds__(1024) k_small_grid(DevParams p, unsigned int ncells, const float4 *__restrict__ x4,
                                                     float4 *__restrict__ x_out, unsigned int *__restrict__ order,
                                                     unsigned int *__restrict__ cell_start) {
    extern __shared__ unsigned int s_mem[];
    unsigned int *s_start = s_mem, *s_perm = s_mem + ncells + 1;
    for (unsigned int c = threadIdx.x; c <= ncells; c += 1024u) s_start[c] = 0u;
    __syncthreads();
    unsigned int key[kSmallGrid / 1024], rank[kSmallGrid / 1024];
#pragma unroll
    for (int k = 0; k < kSmallGrid / 1024; ++k) {
        const int i = (int)threadIdx.x + 1024 * k;
        if (i >= p.n) break;
        key[k] = cell_index(cell_of(f3(__ldg(x4 + i)), p), p);
        rank[k] = atomicAdd(s_start + key[k], 1u);
    }
    __syncthreads();
    const unsigned int per = (ncells + 1023u) / 1024u, c0 = min(threadIdx.x * per, ncells), c1 = min(c0 + per, ncells);
    unsigned int sum = 0u, total;
    for (unsigned int c = c0; c < c1; ++c) sum += s_start[c];
    unsigned int run = block_scan(sum, total);
    for (unsigned int c = c0; c < c1; ++c) {
        const unsigned int v = s_start[c];
        s_start[c] = run;
        run += v;
    }
    if (threadIdx.x == 0) s_start[ncells] = total;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSmallGrid / 1024; ++k) {
        const int i = (int)threadIdx.x + 1024 * k;
        if (i >= p.n) break;
        s_perm[s_start[key[k]] + rank[k]] = (unsigned int)i;
    }
    for (unsigned int c = threadIdx.x; c <= ncells; c += 1024u) cell_start[c] = s_start[c];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSmallGrid / 1024; ++k) {
        const unsigned int i = threadIdx.x + 1024u * k;
        if (i >= (unsigned int)p.n) break;
        const unsigned int a = s_start[key[k]], e = s_start[key[k] + 1];
        unsigned int d = a;
        for (unsigned int v = a; v < e; ++v) d += s_perm[v] < i ? 1u : 0u;
        x_out[d] = __ldg(x4 + i);
        order[d] = i;
    }
}

/* In-loop grid rebuild: hash the current x* (the ping-pong buffer named by
 * ctl->parity, which only the device knows inside a captured loop). */
__global__ void k_hash_parity(DevParams p, const float4 *ppos0, const float4 *ppos1, const DevCtl *ctl,
                              unsigned int *__restrict__ key, unsigned int *__restrict__ rank,
                              unsigned int *__restrict__ count) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const float4 *x4 = ctl->parity ? ppos1 : ppos0;
    hash_body(p, i, f3(x4[i]), key, rank, count);
}

/* Gather every array carried through the iterations into temporaries. */
__global__ void k_rebuild_gather(int n, CellOrder o, const DevCtl *ctl,
                                 const float4 *__restrict__ pos, const float4 *ppos0, const float4 *ppos1,
                                 const unsigned int *__restrict__ id, const unsigned int *__restrict__ attr,
                                 const float *__restrict__ dens, float4 *__restrict__ t_pos,
                                 float4 *__restrict__ t_x, unsigned int *__restrict__ t_id,
                                 unsigned int *__restrict__ t_attr, float *__restrict__ t_dens,
                                 const unsigned int *__restrict__ key, unsigned int *__restrict__ cellb,
                                 const float4 *__restrict__ xpred, float4 *__restrict__ t_xpred,
                                 float *__restrict__ t_lam) {
    int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n) return;
    const float4 *x4 = ctl->parity ? ppos1 : ppos0;
    unsigned int s;
    const unsigned int d = ranked_slot((unsigned int)u, o, s);
    if (cellb) cellb[d] = key[s];
    if (xpred) t_xpred[d] = xpred[s];
    /* lambda of the last pass lives in the .w of the other buffer */
    if (t_lam) t_lam[d] = (ctl->parity ? ppos0 : ppos1)[s].w;
    t_pos[d] = pos[s];
    t_x[d] = x4[s];
    t_id[d] = id[s];
    t_attr[d] = attr[s];
    t_dens[d] = dens[s];
}

/* Copy the temporaries back; x* also becomes the new build reference xb. */
__global__ void k_rebuild_copy(int n, DevCtl *ctl, const float4 *__restrict__ t_pos, const float4 *__restrict__ t_x,
                               const unsigned int *__restrict__ t_id, const unsigned int *__restrict__ t_attr,
                               const float *__restrict__ t_dens, float4 *__restrict__ pos, float4 *ppos0,
                               float4 *ppos1, float4 *__restrict__ xb, unsigned int *__restrict__ id,
                               unsigned int *__restrict__ attr, float *__restrict__ dens,
                               const float4 *__restrict__ t_xpred, float4 *__restrict__ xpred,
                               const float *__restrict__ t_lam) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned int par = ctl->parity;
    if (d == 0) {
        ctl->builds += 1u;
        ctl->rebuild = 0u;
    }
    if (d >= n) return;
    if (xpred) xpred[d] = t_xpred[d];
    if (t_lam) (par ? ppos0 : ppos1)[d].w = t_lam[d];
    float4 *x4 = par ? ppos1 : ppos0;
    pos[d] = t_pos[d];
    float4 x = t_x[d];
    x4[d] = x;
    xb[d] = x;
    id[d] = t_id[d];
    attr[d] = t_attr[d];
    dens[d] = t_dens[d];
}

/* ======================================================================== */
/* neighbour lists                                                          */
/* ======================================================================== */

/* blocks per SM: seven of four warps (72 registers a thread), so that 32,768 slots
 * are one round of the GPU (the WCSPH density took 19.8 us there with 80 registers,
 * 16.8 with these); six of four tiles, what shared memory holds */
constexpr int kSplitBlocks = 7, kTileBlocks = 6;
/* The lists of every slot, W warps for 32 consecutive ones (build_list_warp). */
template <int W>
__global__ void __launch_bounds__(W == 1 ? kListBlock : 32 * W, W == 1 ? kTileBlocks : kSplitBlocks)
    k_build_list(DevParams p, const unsigned int *__restrict__ cell_start, const float4 *__restrict__ xb,
                 const unsigned int *__restrict__ cellb, ListEntry *__restrict__ list,
                 unsigned char *__restrict__ cnt) {
    __shared__ PairTileOf<W> s_tile[W == 1 ? kListBlock / 32 : 1];
    const int i = W == 1 ? blockIdx.x * kListBlock + threadIdx.x : blockIdx.x * 32 + (threadIdx.x & 31);
    build_list_warp<W>(p, i, i < p.n, cell_start, xb, cellb, list, cnt, s_tile[W == 1 ? threadIdx.x >> 5 : 0]);
}

/* ======================================================================== */
/* PBF                                                                      */
/* ======================================================================== */

/* rho_i = m aw sum_j (h^2 - r^2)^3 over r < h, self included. */
__global__ void k_pbf_density(DevParams p, const unsigned int *__restrict__ cell_start,
                              const float4 *__restrict__ pos, float *__restrict__ dens) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    float3 xi = f3(pos[i]);
    int3 c = cell_of(xi, p);
    float acc = 0.0f;
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy) {
            unsigned int s, e;
            row_range(cell_start, c, dy, dz, p, s, e);
            for (unsigned int j = s; j < e; ++j) {
                float3 d = xi - f3(__ldg(pos + j));
                float r2 = dot3(d, d);
                if (r2 < p.h2) {
                    float q = p.h2 - r2;
                    acc += q * q * q;
                }
            }
        }
    float rho = p.mass * p.aw * acc;
    if (p.nb) { /* + sum_b rho0 psi_b W (rx_sph_pbd.cpp:624-644) */
        float bw = 0.f;
        for_each_boundary(p, xi, [&](unsigned int, const float4 &b4) {
            const float3 d = xi - f3(b4);
            const float q = fmaxf(p.h2 - dot3(d, d), 0.0f);
            bw += b4.w * q * q * q;
        });
        rho += p.mass * p.aw * bw;
    }
    dens[i] = rho;
}

/* a_i = mu sum_{j != i} m (v_j - v_i) / rho_i lapW + g (rx_sph_pbd.cpp:651-689). */
__global__ void k_pbf_visc(DevParams p, const unsigned int *__restrict__ cell_start, const float4 *__restrict__ pos,
                           const float4 *__restrict__ vel, const float *__restrict__ dens,
                           float4 *__restrict__ acc) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    float3 xi = f3(pos[i]), vi = f3(vel[i]);
    int3 c = cell_of(xi, p);
    float3 f = make_float3(0.f, 0.f, 0.f);
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy) {
            unsigned int s, e;
            row_range(cell_start, c, dy, dz, p, s, e);
            for (unsigned int j = s; j < e; ++j) {
                if (j == (unsigned int)i) continue;
                float3 d = xi - f3(__ldg(pos + j));
                float r2 = dot3(d, d);
                if (r2 < p.h2 && r2 > 0.0f) {
                    float r = sqrtf(r2);
                    float lw = p.al * (p.h - r);
                    f = f + lw * (f3(__ldg(vel + j)) - vi);
                }
            }
        }
    float k = p.viscosity * p.mass / dens[i];
    float3 a = k * f + p.gravity;
    acc[i] = make_float4(a.x, a.y, a.z, 0.0f);
}

/* lambda pass: density, C, sum |grad C|^2 (with the k = i term), lambda
 * into x*.w, block partial errors; the last block reduces the errors in a
 * fixed order, advances the iteration counter and decides whether the
 * device-side loop continues.
 * As many blocks as are resident; each warp takes chunks of 32 slots, the first
 * and all but the last whole round in turn, the rest on demand.  At 1 M particles
 * 92 us as a plain grid, 82 round-robin, 78 with the leftovers on demand, 74 with
 * one more round (81 with every chunk: the counter contends; that form took 30.6
 * us at 221,184 particles, where there is one round, and takes 22.8 now). */
template <bool KAHAN, bool DEEP>
__global__ void __launch_bounds__(DEEP ? kDeepBlock : kPassBlock, DEEP ? kDeepMinB : FSPH_PASS_MINB) k_lambda(DevParams p, const unsigned int *__restrict__ cell_start,
                                                   float4 *ppos0, float4 *ppos1, float *__restrict__ dens,
                                                   DevCtl *ctl, ErrPartial *part,
                                                   cudaGraphConditionalHandle hwhile, int use_graph,
                                                   const ListEntry *__restrict__ list,
                                                   const unsigned char *__restrict__ cnt) {
    const unsigned int par = *((volatile unsigned int *)&ctl->parity);
    float4 *pp = par ? ppos1 : ppos0;
    /* DEEP: one chunk a warp, in order */
    unsigned long long q1 = 0ull, q2 = 0ull;
    float em = 0.f;
    const int lane = threadIdx.x & 31, warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)((gridDim.x * blockDim.x) >> 5), nchunks = (p.n + 31) >> 5;
    const int stat = max(nchunks / nw - 1, 1) * nw;
    for (int c = warp; c < nchunks;
         c = DEEP || stat >= nchunks ? nchunks : next_chunk(c, nw, stat, &ctl->grab, lane)) {
        const int i = c * 32 + lane;
        if (i < p.n) {
            const float C = lambda_body<1, KAHAN, DEEP>(p, cell_start, pp, dens, ctl, list, cnt, i, 0, true);
            q1 += err_fix(C > 0.0f ? C : 0.0f);
            q2 += err_fix(fabsf(C));
            em = fmaxf(em, fabsf(C));
        }
    }
    lambda_tail_fix(p, ctl, part, q1, q2, em, hwhile, use_graph);
}

/* Density and lambda of every slot by walking the cells, LPP lanes a particle,
 * written to the particle's place (order[slot]): the whole pass of the
 * allocation-free entry point, which keeps no lists.  One thread a particle
 * leaves 8 blocks and a serial walk of 290 candidates at 4,096 particles (47 us);
 * with 32 lanes a row of cells is one coalesced step.  The whole call went from
 * 84 to 36 us at 4,096 particles (21 with the grid built by one block).  The sums
 * are the lanes' partial sums, as in the batched passes with several lanes; KAHAN:
 * each compensated, and added with the errors of the additions. */
template <int LPP, bool KAHAN>
__global__ void __launch_bounds__(kBlock) k_lambda_walk(DevParams p, const unsigned int *__restrict__ cell_start,
                                                        const float4 *__restrict__ x,
                                                        const unsigned int *__restrict__ order,
                                                        float *__restrict__ dens, float *__restrict__ lambda) {
    const int t = blockIdx.x * kBlock + threadIdx.x;
    const int sub = t % LPP;
    const bool valid = t / LPP < p.n;
    const int i = valid ? t / LPP : p.n - 1; /* padding lanes run a real slot and write nothing */
    const float3 xi = f3(__ldg(x + i));
    float rho, lam;
    lambda_terms<LPP, KAHAN>(
        p, x, xi,
        [&](auto &&load, auto &&f) {
            for_each_candidate<LPP>(p, cell_start, nullptr, nullptr, i, xi, sub, load, f);
        },
        rho, lam);
    if (!valid || sub != 0) return;
    const unsigned int o = order[i];
    dens[o] = rho;
    lambda[o] = lam;
}

/* correction pass: dp_i = sum_j (lambda_i + lambda_j + s_corr) grad W_ij / rho0,
 * x*_i <- walls(x*_i + dp_i) into the other ping-pong buffer; the largest
 * displacement since the last grid build decides whether the grid must be
 * rebuilt before the next pass. */
template <bool DEEP>
__global__ void __launch_bounds__(DEEP ? kDeepBlock : kPassBlock, DEEP ? kDeepMinB : FSPH_PASS_MINB) k_correction(DevParams p, const unsigned int *__restrict__ cell_start,
                                                       float4 *ppos0, float4 *ppos1,
                                                       const float4 *__restrict__ xb, DevCtl *ctl, float *part,
                                                       cudaGraphConditionalHandle hif,
                                                       cudaGraphConditionalHandle hif2, int use_graph,
                                                       float4 *__restrict__ dp_out,
                                                       const ListEntry *__restrict__ list,
                                                       const unsigned char *__restrict__ cnt) {
    const unsigned int par = *((volatile unsigned int *)&ctl->parity);
    const float4 *__restrict__ src = par ? ppos1 : ppos0;
    float4 *__restrict__ dst = par ? ppos0 : ppos1;
    float disp2 = 0.f;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.n)
        disp2 = correction_body<1, DEEP>(p, cell_start, src, dst, xb, ctl, dp_out, list, cnt, i, 0, true);
    correction_tail(p, ctl, part, disp2, par, hif, hif2, use_graph);
}

/* v = (x* - x) / dt, x = x* (rx_sph_pbd.cpp:464-471); also brings id / attr
 * back to the step's home buffers. */
__global__ void k_finalize(DevParams p, const float4 *__restrict__ pos_b, const float4 *ppos0,
                           const float4 *ppos1, const DevCtl *ctl, const unsigned int *__restrict__ id_b,
                           const unsigned int *__restrict__ attr_b, float4 *__restrict__ pos_a,
                           float4 *__restrict__ vel_a, unsigned int *__restrict__ id_a,
                           unsigned int *__restrict__ attr_a, const float4 *__restrict__ xpred,
                           float4 *__restrict__ dstep, const float *__restrict__ dens, float4 *__restrict__ xm) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const float4 *pp = ctl->parity ? ppos1 : ppos0;
    float3 xs = f3(pp[i]);
    float3 x = f3(pos_b[i]);
    float3 v = p.inv_dt * (xs - x);
    pos_a[i] = make_float4(xs.x, xs.y, xs.z, 0.0f);
    if (xm) xm[i] = make_float4(xs.x, xs.y, xs.z, p.mass / dens[i]); /* what the XSPH and vorticity passes gather */
    vel_a[i] = make_float4(v.x, v.y, v.z, 0.0f);
    id_a[i] = id_b[i];
    attr_a[i] = attr_b[i];
    /* total correction of this step, x*_final - x*_predicted */
    if (dstep) {
        float3 dd = xs - f3(xpred[i]);
        dstep[i] = make_float4(dd.x, dd.y, dd.z, 0.0f);
    }
}

/* omega_i = sum_j (v_j - v_i) x grad_j W_ij (grad_j = -grad_i), and the
 * XSPH update v_i + c sum_j (m / rho_j)(v_j - v_i) W_ij. */
template <bool FEAT, bool NBR, bool PRE, bool DEEP>
__global__ void __launch_bounds__(DEEP ? kDeepBlock : kPostBlock) k_xsph_vort(DevParams p, const unsigned int *__restrict__ cell_start,
                                                      const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                                                      const float *__restrict__ dens, float4 *__restrict__ vel_out,
                                                      float4 *__restrict__ vort, FeatureOut fo,
                                                      const ListEntry *__restrict__ list,
                                                      const unsigned char *__restrict__ cnt,
                                                      float *__restrict__ mag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    xsph_vort_body<FEAT, NBR, PRE, DEEP>(p, i, cell_start, pos, vel, dens, vel_out, vort, fo, list, cnt, mag);
}

/* eta_i = sum_j (m / rho_j)(|w_j| - |w_i|) grad_i W_ij; f = eps (eta/|eta|) x w_i;
 * v_i <- v_i + dt f. */
template <bool PRE, bool DEEP>
__global__ void __launch_bounds__(DEEP ? kDeepBlock : kPostBlock) k_vort_apply(DevParams p, const unsigned int *__restrict__ cell_start,
                                                       const float4 *__restrict__ pos,
                                                       const float4 *__restrict__ vort,
                                                       const float *__restrict__ dens,
                                                       const float4 *__restrict__ vel_in,
                                                       float4 *__restrict__ vel_out,
                                                       const ListEntry *__restrict__ list,
                                                       const unsigned char *__restrict__ cnt,
                                                      const float *__restrict__ mag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    vort_apply_body<PRE, DEEP>(p, i, cell_start, pos, vort, dens, vel_in, vel_out, list, cnt, mag);
}

/* ======================================================================== */
/* static boundary particles                                                */
/* ======================================================================== */
/* p.n = the boundary count in these kernels; p.bpos etc. the sorted boundary */

/* psi_b = m / sum_b' m W(r_bb') (rx_sph_pbd.cpp:1061-1090); bscale[b] = rho0 psi_b / m */
__global__ void k_boundary_volume(DevParams p, float *__restrict__ bscale) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= p.n) return;
    const float3 xb = f3(__ldg(p.bpos + b));
    float wsum = 0.f;
    for_each_boundary(p, xb, [&](unsigned int, const float4 &c4) {
        const float3 d = xb - f3(c4);
        const float q = fmaxf(p.h2 - dot3(d, d), 0.0f);
        wsum += q * q * q;
    });
    const float mw = p.mass * p.aw * wsum; /* sum_b' m W, self included */
    bscale[b] = p.rest_dens / mw;          /* rho0 psi_b / m = rho0 / (sum m W) */
}

/* The boundary-boundary parts of lambda_b, fixed for a static boundary. */
__global__ void k_boundary_static(DevParams p, float2 *__restrict__ bstat) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= p.n) return;
    const float3 xb = f3(__ldg(p.bpos + b));
    const float agr = p.ag * p.inv_rest_dens;
    float bw = 0.f, sd = 0.f;
    for_each_boundary(p, xb, [&](unsigned int, const float4 &c4) {
        const float3 d = xb - f3(c4);
        const float r2 = dot3(d, d);
        const float q = fmaxf(p.h2 - r2, 0.0f);
        const float inv_r = pair_rsqrt(r2);
        const float t = fmaxf(p.h - r2 * inv_r, 0.0f);
        const float gb = c4.w * agr * t * t * inv_r;
        bw += c4.w * q * q * q;
        sd += gb * gb * r2;
    });
    bstat[b] = make_float2(p.mass * p.aw * bw, sd);
}

__global__ void k_boundary_near(DevParams p, unsigned int ncells, unsigned char *__restrict__ bnear) {
    unsigned int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    const int x = (int)(c % (unsigned int)p.gx), y = (int)((c / (unsigned int)p.gx) % (unsigned int)p.gy),
              z = (int)(c / ((unsigned int)p.gx * (unsigned int)p.gy));
    unsigned char any = 0;
    if (x >= 1 && y >= 1 && z >= 1 && x <= p.gx - 2 && y <= p.gy - 2 && z <= p.gz - 2) {
        for (int dz = -1; dz <= 1; ++dz)
            for (int dy = -1; dy <= 1; ++dy) {
                const unsigned int base = c + (unsigned int)((dz * p.gy + dy) * p.gx);
                if (p.bcell[base + 2] > p.bcell[base - 1]) any = 1;
            }
    }
    bnear[c] = any;
}

/* lambda_b = -C_b / (sd_b + eps): rho_b and sd_b from the fluid x* of the
 * current parity plus the static boundary parts (rx_sph_pbd.cpp:825-913,
 * fluid neighbours on the current positions as rx_pbdsph_kernel.cu:666-735). */
__global__ void __launch_bounds__(kBlock) k_boundary_lambda(DevParams p, const unsigned int *__restrict__ cell_start,
                                                            const float4 *ppos0, const float4 *ppos1,
                                                            const DevCtl *ctl, const float2 *__restrict__ bstat,
                                                            float *__restrict__ blam) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= p.nb) return;
    const float4 *pp = ctl->parity ? ppos1 : ppos0;
    const float3 xb = f3(__ldg(p.bpos + b));
    const float agr = p.ag * p.inv_rest_dens;
    float wsum = 0.f, sd = 0.f;
    for_each_candidate<1>(
        p, cell_start, nullptr, nullptr, 0, xb, 0, [&](unsigned int j) { return pp[j]; },
        [&](unsigned int, const float4 &xj4) {
            const float3 d = xb - f3(xj4);
            const float r2 = dot3(d, d);
            const float q = fmaxf(p.h2 - r2, 0.0f);
            const float inv_r = pair_rsqrt(r2);
            const float t = fmaxf(p.h - r2 * inv_r, 0.0f);
            const float g = agr * t * t * inv_r;
            wsum += q * q * q;
            sd += g * g * r2;
        });
    const float2 st = bstat[b];
    const float rho = p.mass * p.aw * wsum + st.x;
    sd += st.y;
    float C = rho * p.inv_rest_dens - 1.0f;
    if (p.clamp_constraint && C < 0.0f) C = 0.0f;
    blam[b] = -C / (sd + p.epsilon);
}

void launch_boundary_volume(const DevParams &p, float *bscale, cudaStream_t s) {
    k_boundary_volume<<<blocks_for(p.n), kBlock, 0, s>>>(p, bscale);
}
void launch_boundary_static(const DevParams &p, float2 *bstat, cudaStream_t s) {
    k_boundary_static<<<blocks_for(p.n), kBlock, 0, s>>>(p, bstat);
}
void launch_boundary_near(const DevParams &p, unsigned int ncells, unsigned char *bnear, cudaStream_t s) {
    k_boundary_near<<<blocks_for(ncells), kBlock, 0, s>>>(p, ncells, bnear);
}
void launch_boundary_lambda(const DevParams &p, const unsigned int *cell_start, const float4 *ppos0,
                            const float4 *ppos1, const DevCtl *ctl, const float2 *bstat, float *blam, cudaStream_t s) {
    if (p.nb <= 0) return;
    k_boundary_lambda<<<blocks_for(p.nb), kBlock, 0, s>>>(p, cell_start, ppos0, ppos1, ctl, bstat, blam);
}

/* the rest of the arithmetic of split floats (Split, two_sum: fsph_passes.cuh) */
__device__ __forceinline__ Split two_diff(float a, float b) { return two_sum(a, -b); }
__device__ __forceinline__ Split two_prod(float a, float b) {
    const float q = __fmul_rn(a, b);
    return Split{q, __fmaf_rn(a, b, -q)};
}
/* h + l with the error of the sum kept (|h| >= |l| or h = 0) */
__device__ __forceinline__ Split renorm(float h, float l) {
    const float s = __fadd_rn(h, l);
    return Split{s, __fsub_rn(l, __fsub_rn(s, h))};
}
__device__ __forceinline__ Split split_of(double v) {
    const float h = (float)v;
    return Split{h, (float)(v - (double)h)};
}

/* ======================================================================== */
/* WCSPH                                                                    */
/* ======================================================================== */

/* rho_i = m aw sum_j (h^2 - r^2)^3 (r < h, self included) and p_i = k (rho_i -
 * rho0) (rxSPH::calDensity, rx_sph_cpu.cpp:495-552, 569), in the same walk
 * over the 27 cells as the neighbour list of the following force pass
 * (every slot within the list radius, here the cell width h (1 + 1e-3));
 * the force pass's per-neighbour factors ride in the .w words of the sorted
 * copies: pos.w = p / rho^2, vel.w = 1 / rho.  Only .w words are written, so
 * the x, y, z the other threads read stay as they are; they read them by plain
 * loads (ld.global.nc is for what no thread of the launch writes beside). */
__device__ __forceinline__ void sph_density_out(const DevParams &p, int i, float acc, float4 *pos, float4 *vel,
                                                float *__restrict__ dens, float *__restrict__ pres) {
    const float rho = p.mass * p.aw * acc;
    const float prs = p.gas_k * (rho - p.rest_dens);
    dens[i] = rho;
    pres[i] = prs;
    reinterpret_cast<float *>(pos + i)[3] = prs / (rho * rho);
    reinterpret_cast<float *>(vel + i)[3] = 1.0f / rho;
}
/* W warps for 32 consecutive slots: their candidates from the tile
 * (warp_candidates), each evaluated from a gathered position, four at a time,
 * and listed; where the tile does not serve (spray), a thread's own walk.  A thread
 * testing all its candidates was bound by issue and took 205 us at 1,030,301
 * slots and 64.6 at 262,144, this form 171 and 59.5; in a collapsed dam (512,000
 * slots, 106 neighbours on average) 380 and 291. */
template <int W>
__global__ void __launch_bounds__(W == 1 ? kListBlock : 32 * W, W == 1 ? kTileBlocks : kSplitBlocks)
    k_sph_density(DevParams p, const unsigned int *__restrict__ cell_start, float4 *pos, float4 *vel,
                  float *__restrict__ dens, float *__restrict__ pres, ListEntry *__restrict__ list,
                  unsigned char *__restrict__ cnt) {
    __shared__ PairTileOf<W> s_tile[W == 1 ? kListBlock / 32 : 1];
    const int i = W == 1 ? blockIdx.x * kListBlock + threadIdx.x : blockIdx.x * 32 + (threadIdx.x & 31);
    const bool valid = i < p.n;
    const float3 xi = valid ? f3(pos[i]) : make_float3(0.f, 0.f, 0.f);
    const int3 c = cell_of(xi, p);
    /* W = 1: four partial sums, whose error is no larger than that of the lanes'; a
     * warp of several holds whole rows of cells, of very different weight, and keeps
     * its sum's error beside it */
    float acc[4] = {};
    auto add = [&](int u, const float4 &xj) {
        const float3 d = xi - f3(xj);
        const float r2 = dot3(d, d);
        if (r2 < p.h2) {
            const float q = p.h2 - r2;
            if (W == 1) {
                acc[u] += q * q * q;
            } else {
                const float y = q * q * q - acc[1], s = acc[0] + y;
                acc[1] = (s - acc[0]) - y;
                acc[0] = s;
            }
        }
        return r2;
    };
    warp_candidates(
        p, cell_start, [&](unsigned int j) { return pos[j]; }, xi, valid ? cell_index(c, p) : 0u, valid, p.rl2,
        s_tile[W == 1 ? threadIdx.x >> 5 : 0],
        [&](bool found, int first, int count, int total, TileWalk<W> &walk) {
            if (found) {
                unsigned int last = 0u;
                for (int k = 0; k < count; k += 4) {
                    unsigned int v[4];
                    float4 xj[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[u] = walk.next(); /* the last group is padded with its last entry */
#pragma unroll
                    for (int u = 0; u < 4; ++u) xj[u] = pos[v[u]];
                    if (W == 1 && first == 0) {
                        if (list && k < kListMax)
                            reinterpret_cast<uint4 *>(list)[(size_t)(k >> 2) * (size_t)p.n + (size_t)i] =
                                make_uint4(v[0], v[1], v[2], v[3]);
                    } else if (list) {
                        last = v[3];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (k + u < count && first + k + u < kListMax) list[list_at(first + k + u, i, p.n)] = v[u];
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (k + u < count) add(u, xj[u]);
                }
                if (W > 1 || first > 0) {
                    if (list && count && first + count == total && total < kListMax)
                        for (int k = total; (k & 3) != 0; ++k) list[list_at(k, i, p.n)] = last;
                    count = total;
                }
            } else {
                acc[0] = acc[1] = acc[2] = acc[3] = 0.0f;
                if (W > 1 && threadIdx.x >= 32u) return;
                unsigned int last = (unsigned int)i;
                count = 0;
                walk_cells(
                    p, cell_start, cell_index(c, p), [&](unsigned int j) { return pos[j]; },
                    [&](unsigned int j, const float4 &xj) {
                        if (!(add(0, xj) < p.rl2)) return;
                        last = j;
                        if (list && count < kListMax) list[list_at(count, i, p.n)] = last;
                        ++count;
                    });
                if (list && count <= kListMax) /* pad the last group (the slot itself is always listed) */
                    for (int k = count; (k & 3) != 0; ++k) list[list_at(k, i, p.n)] = last;
            }
            if (list && (W == 1 || threadIdx.x < 32u)) cnt[i] = count > kListMax ? kListOverflow : (unsigned char)count;
        });
    if (W == 1) {
        if (valid) sph_density_out(p, i, (acc[0] + acc[1]) + (acc[2] + acc[3]), pos, vel, dens, pres);
    } else {
        __shared__ double s_sum[W][32];
        s_sum[threadIdx.x >> 5][threadIdx.x & 31] = (double)acc[0] - (double)acc[1];
        __syncthreads();
        if (threadIdx.x >= 32u || !valid) return;
        double sum = 0.0;
#pragma unroll
        for (int w = 0; w < W; ++w) sum += s_sum[w][threadIdx.x];
        sph_density_out(p, i, (float)sum, pos, vel, dens, pres);
    }
}

/* The same with a warp per particle, for scenes that would leave the GPU idle: its
 * lanes take the candidates of each row side by side and a ballot ranks the hits,
 * so the list holds the same slots in the same order.  The density is the sum of
 * the lanes' partial sums (same terms, other order), the errors of their additions
 * kept. */
__global__ void __launch_bounds__(kBlock) k_sph_density_lanes(DevParams p, const unsigned int *__restrict__ cell_start,
                                                              float4 *pos, float4 *vel, float *__restrict__ dens,
                                                              float *__restrict__ pres, ListEntry *__restrict__ list,
                                                              unsigned char *__restrict__ cnt) {
    const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= p.n) return;
    const float3 xi = f3(pos[i]);
    const int3 c = cell_of(xi, p);
    float acc = 0.0f;
    int k = 0;
    unsigned int last = (unsigned int)i;
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy) {
            unsigned int s, e;
            row_range(cell_start, c, dy, dz, p, s, e);
            for (unsigned int j0 = s; j0 < e; j0 += 32) {
                const unsigned int j = j0 + (unsigned int)lane;
                bool hit = false;
                if (j < e) {
                    const float3 d = xi - f3(pos[j]);
                    const float r2 = dot3(d, d);
                    if (r2 < p.h2) {
                        const float q = p.h2 - r2;
                        acc += q * q * q;
                    }
                    hit = r2 < p.rl2;
                }
                if (list) {
                    const unsigned int m = __ballot_sync(0xffffffffu, hit);
                    if (m) {
                        if (hit) {
                            const int at = k + __popc(m & ((1u << lane) - 1u));
                            if (at < kListMax) list[list_at(at, i, p.n)] = (ListEntry)j;
                        }
                        last = j0 + (unsigned int)(31 - __clz((int)m));
                        k += __popc(m);
                    }
                }
            }
        }
    acc = group_sum_split<32>(acc, 0.0f);
    if (lane != 0) return;
    if (list) {
        const bool ovf = k > kListMax;
        if (!ovf) /* pad the last group (k >= 1: the slot itself is always listed) */
            for (int u = k; (u & 3) != 0; ++u) list[list_at(u, i, p.n)] = (ListEntry)last;
        cnt[i] = ovf ? kListOverflow : (unsigned char)k;
    }
    sph_density_out(p, i, acc, pos, vel, dens, pres);
}

/* a_i = -sum_j m (p_i/rho_i^2 + p_j/rho_j^2) grad W_ij + mu sum_j m (v_j - v_i)
 * lapW_ij / rho_j + g over 0 < r_ij < h (rxSPH::calForce, rx_sph_cpu.cpp:558-656),
 * from the list of the density pass (or the 27 cells when lists are off),
 * with LPP lanes per particle (small scenes then still fill the GPU).
 * Branch-free pair terms: t = max(h - r, 0) is 0 at and beyond h, and at
 * r = 0 too (h - 0 * rsqrt(0) is NaN, which fmaxf maps to 0), so the self
 * pair and coincident particles add nothing, as the reference skips them. */
template <int LPP>
__global__ void __launch_bounds__(kBlock) k_sph_force(DevParams p, const unsigned int *__restrict__ cell_start,
                                                      const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                                                      float4 *__restrict__ acc, const ListEntry *__restrict__ list,
                                                      const unsigned char *__restrict__ cnt) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int sub = t % LPP;
    const bool valid = t / LPP < p.n;
    const int i = valid ? t / LPP : p.n - 1; /* padding lanes run a real slot and write nothing */
    const float4 xi4 = pos[i], vi4 = vel[i];
    const float3 xi = f3(xi4), vi = f3(vi4);
    const float prsi = xi4.w;
    float3 fp = make_float3(0.f, 0.f, 0.f), fv = make_float3(0.f, 0.f, 0.f);
    for_each_candidate<LPP>(
        p, cell_start, list, cnt, i, xi, sub,
        [&](unsigned int j) { return PosVel{__ldg(pos + j), __ldg(vel + j)}; },
        [&](unsigned int, const PosVel &b) {
            const float3 d = xi - f3(b.x);
            const float r2 = dot3(d, d);
            const float inv_r = rsqrtf(r2);
            const float tt = fmaxf(fmaf(-r2, inv_r, p.h), 0.0f);
            const float g = p.ag * tt * tt * fminf(inv_r, 1e30f);
            fp = fp + ((prsi + b.x.w) * g) * d;
            fv = fv + (p.al * tt * b.v.w) * (f3(b.v) - vi);
        });
    if (LPP > 1) {
        fp.x = group_sum<LPP>(fp.x); fp.y = group_sum<LPP>(fp.y); fp.z = group_sum<LPP>(fp.z);
        fv.x = group_sum<LPP>(fv.x); fv.y = group_sum<LPP>(fv.y); fv.z = group_sum<LPP>(fv.z);
    }
    if (!valid || sub != 0) return;
    const float3 a = (-p.mass) * fp + (p.viscosity * p.mass) * fv + p.gravity;
    acc[i] = make_float4(a.x, a.y, a.z, 0.0f);
}
__global__ void k_sph_integrate(DevParams p, const float4 *__restrict__ pos_b, const float4 *__restrict__ vel_b,
                                const float4 *__restrict__ acc, const unsigned int *__restrict__ id_b,
                                const unsigned int *__restrict__ attr_b, float4 *__restrict__ pos_a,
                                float4 *__restrict__ vel_a, unsigned int *__restrict__ id_a,
                                unsigned int *__restrict__ attr_a) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    float3 v = f3(vel_b[i]) + p.dt * f3(acc[i]);
    float3 x = f3(pos_b[i]) + p.dt * v;
    if (p.ntri) polygon_collide(f3(pos_b[i]), x, v, p.dt, p); /* sphIntegrateWithPolygon, rx_sph_kernel.cu:852-895 */
    x = solid_project(x, p);
    pos_a[i] = make_float4(x.x, x.y, x.z, 0.0f);
    vel_a[i] = make_float4(v.x, v.y, v.z, 0.0f);
    id_a[i] = id_b[i];
    attr_a[i] = attr_b[i];
}

/* ======================================================================== */
/* neighbour sets, reference criterion                                      */
/* ======================================================================== */

/* fl32(|xi - xj|^2 in double) <= fl32(h*h) (rx_nnsearch.h:499-507): a float
 * test decides unless the float distance lies within 1e-5 of h^2, where the
 * double evaluation (separate multiplies and adds, no fusion) decides. */
__device__ inline bool ref_neighbor(float3 xi, float3 xj, float h2) {
    float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
    float d2 = dx * dx + dy * dy + dz * dz;
    if (d2 < h2 * (1.0f - 1e-5f)) return true;
    if (d2 > h2 * (1.0f + 1e-5f)) return false;
    double ex = (double)xi.x - (double)xj.x, ey = (double)xi.y - (double)xj.y, ez = (double)xi.z - (double)xj.z;
    double dd = __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez));
    return __double2float_rn(dd) <= h2;
}

/* Neighbour counts of a warp's 32 consecutive slots, in particle order
 * (cnt_p[id]), and the neighbours themselves in the list storage (up to
 * kListMax a slot; cnt = kListOverflow past that) for k_nb_rows: the search,
 * from the warp's tile (warp_candidates, a hair wider than the radius), is
 * done once.  total: the sum over all slots. */
__global__ void __launch_bounds__(kListBlock) k_nb_count(DevParams p, const unsigned int *__restrict__ cell_start,
                                                         const float4 *__restrict__ pos,
                                                         const unsigned int *__restrict__ id,
                                                         unsigned int *__restrict__ cnt_p,
                                                         unsigned long long *__restrict__ total,
                                                         ListEntry *__restrict__ list,
                                                         unsigned char *__restrict__ cnt) {
    __shared__ PairTile s_tile[kListBlock / 32];
    PairTile &t = s_tile[threadIdx.x >> 5];
    const int i = blockIdx.x * kListBlock + threadIdx.x;
    const bool valid = i < p.n;
    const float3 xi = valid ? f3(__ldg(pos + i)) : make_float3(0.f, 0.f, 0.f);
    const int3 c = cell_of(xi, p);
    unsigned int k = 0;
    warp_candidates(p, cell_start, [&](unsigned int j) { return __ldg(pos + j); }, xi,
                    valid ? cell_index(c, p) : 0u, valid, p.h2 * (1.0f + 1e-4f), t,
                    [&](bool found, int, int count, int, TileWalk<1> &walk) {
                        auto load = [&](unsigned int j) { return __ldg(pos + j); };
                        auto meet = [&](unsigned int j, const float4 &xj) {
                            if (ref_neighbor(xi, f3(xj), p.h2)) {
                                if (k < (unsigned int)kListMax) list[list_at((int)k, i, p.n)] = j;
                                ++k;
                            }
                        };
                        if (!found) k = 0;
                        if (found) {
                            for (int f = 0; f < count; ++f) {
                                const unsigned int j = walk.next();
                                meet(j, load(j));
                            }
                        } else {
                            walk_cells(p, cell_start, cell_index(c, p), load, meet);
                        }
                        cnt_p[id[i]] = k;
                        cnt[i] = k > (unsigned int)kListMax ? kListOverflow : (unsigned char)k;
                    });
    unsigned long long sum = k;
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(total, sum);
}

/* squared distance as the reference's rxNeigh::Dist2: the difference of the
 * float coordinates and its squares summed in double, x + y + z in that
 * order with no fused multiply-add, rounded to float (rx_nnsearch.h:499-507) */
__device__ inline float ref_dist2(float3 xi, float3 xj) {
    double ex = (double)xi.x - (double)xj.x, ey = (double)xi.y - (double)xj.y, ez = (double)xi.z - (double)xj.z;
    return __double2float_rn(__dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez)));
}

/* Rows of the neighbour sets, one warp per slot: the particle indices of its
 * neighbours in ascending order at out[offsets[particle] ...] (and each pair's
 * squared distance).  A row of up to kListMax entries is in the list storage:
 * each lane holds one or two and counts the smaller ones, which it reads four at
 * a time from shared memory (a shuffle for each took 62.7 us at 65,600 particles,
 * this 26.9).  Longer rows are found again by walking the cells and sorted in place
 * by one lane. */
__global__ void __launch_bounds__(kBlock) k_nb_rows(DevParams p, const unsigned int *__restrict__ cell_start,
                                                    const float4 *__restrict__ pos,
                                                    const unsigned int *__restrict__ id,
                                                    const unsigned int *__restrict__ offsets,
                                                    const ListEntry *__restrict__ list,
                                                    const unsigned char *__restrict__ cnt, int *__restrict__ out,
                                                    float *__restrict__ d2out) {
    __shared__ __align__(16) int s_row[kBlock / 32][kListMax];
    const int lane = threadIdx.x & 31;
    const int i = (int)(((long long)blockIdx.x * kBlock + threadIdx.x) >> 5);
    if (i >= p.n) return;
    const int k = (int)cnt[i];
    const size_t at = offsets[id[i]];
    const float3 xi = f3(__ldg(pos + i));
    if (k != (int)kListOverflow) {
        unsigned int j[2] = {0u, 0u};
        int v[2] = {INT_MAX, INT_MAX}, r[2] = {0, 0};
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (lane + 32 * u < k) {
                j[u] = __ldg(list + list_at(lane + 32 * u, i, p.n));
                v[u] = (int)__ldg(id + j[u]);
            }
        int *row = s_row[threadIdx.x >> 5];
        row[lane] = v[0];
        row[lane + 32] = v[1];
        __syncwarp();
        for (int t = 0; t < k; t += 4) { /* the places past k hold the largest number */
            const int4 w = *reinterpret_cast<const int4 *>(row + t);
            r[0] += (w.x < v[0]) + (w.y < v[0]) + (w.z < v[0]) + (w.w < v[0]);
            if (k > 32) r[1] += (w.x < v[1]) + (w.y < v[1]) + (w.z < v[1]) + (w.w < v[1]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (lane + 32 * u < k) {
                out[at + r[u]] = v[u];
                if (d2out) d2out[at + r[u]] = ref_dist2(xi, f3(__ldg(pos + j[u])));
            }
        return;
    }
    if (lane != 0) return;
    const int3 c = cell_of(xi, p);
    int m = 0; /* a heap of the entries met so far, the largest index first */
    auto swap = [&](int a, int b) {
        const int w = out[at + a];
        out[at + a] = out[at + b];
        out[at + b] = w;
        if (d2out) {
            const float f = d2out[at + a];
            d2out[at + a] = d2out[at + b];
            d2out[at + b] = f;
        }
    };
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy) {
            unsigned int s, e;
            row_range(cell_start, c, dy, dz, p, s, e);
            for (unsigned int j = s; j < e; ++j) {
                const float3 xj = f3(__ldg(pos + j));
                if (!ref_neighbor(xi, xj, p.h2)) continue;
                out[at + m] = (int)__ldg(id + j);
                if (d2out) d2out[at + m] = ref_dist2(xi, xj);
                for (int q = m++; q > 0 && out[at + (q - 1) / 2] < out[at + q]; q = (q - 1) / 2) swap(q, (q - 1) / 2);
            }
        }
    for (int end = m - 1; end > 0; --end) {
        swap(0, end);
        for (int q = 0;;) {
            int l = 2 * q + 1;
            if (l >= end) break;
            if (l + 1 < end && out[at + l + 1] > out[at + l]) ++l;
            if (out[at + q] >= out[at + l]) break;
            swap(q, l);
            q = l;
        }
    }
}

/* ======================================================================== */
/* deletion regions and the active / parked partition                       */
/* ======================================================================== */

/* Particles strictly inside a region [lo, hi] (checkDeletePB,
 * rx_pbdsph_kernel.cu:1171-1187) are deleted: attribute -1, parked at the
 * reference's far point (0, 0, 1e6) with zero velocity. */
__global__ void k_delete_regions(int n, float4 *__restrict__ pos, float4 *__restrict__ vel,
                                 unsigned int *__restrict__ attr, const float4 *__restrict__ reg, int nreg) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n || attr[d] == 0xffffffffu) return;
    const float4 x = pos[d];
    for (int r = 0; r < nreg; ++r) {
        const float4 lo = reg[2 * r], hi = reg[2 * r + 1];
        if (x.x > lo.x && x.x < hi.x && x.y > lo.y && x.y < hi.y && x.z > lo.z && x.z < hi.z) {
            pos[d] = make_float4(0.0f, 0.0f, 1e6f, 0.0f);
            vel[d] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            attr[d] = 0xffffffffu;
            return;
        }
    }
}

/* keep[d] = 1 for a particle that takes part in the steps (attribute != -1) */
__global__ void k_mark_active(int n, const unsigned int *__restrict__ attr, unsigned int *__restrict__ keep) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d < n) keep[d] = attr[d] != 0xffffffffu ? 1u : 0u;
}

/* stable partition, active slots first: perm[new slot] = old slot, from the
 * exclusive scan of the keep flags (scan[n] = the active count) */
__global__ void k_partition_perm(int n, const unsigned int *__restrict__ scan, unsigned int *__restrict__ perm) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    const unsigned int s = scan[d], keep = scan[d + 1] - s, nk = scan[n];
    perm[keep ? s : nk + ((unsigned int)d - s)] = (unsigned int)d;
}

/* rows of k4 float4 per slot: dst[d] = src[perm[d]] */
__global__ void k_gather_rows(int n, const unsigned int *__restrict__ perm, const float4 *__restrict__ src,
                              float4 *__restrict__ dst, int k4) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n * k4) return;
    const long long d = t / k4, c = t % k4;
    dst[t] = src[(long long)perm[d] * k4 + c];
}

/* ======================================================================== */
/* density on a lattice (for meshing)                                       */
/* ======================================================================== */

/* The density field at the nodes of an nx x ny x nz lattice (i fastest),
 * node (i, j, k) at minp + (i, j, k) d: 0 outside [lo, hi], else
 * sum_j m W(r_j) over the particles with fl32(|x - x_j|^2) <= fl32(h h),
 * r_j = fl32(sqrt(Dist2)), the terms W in more than single precision and the
 * sum in float, as rxPBDSPH::CalColorField (rx_sph_pbd.cpp:2075-2108, the CPU
 * form of pbdsphCalDensityInGrid, rx_pbdsph_kernel.cu:1220-1299).
 *
 * The reference's terms are doubles.  This GPU runs 2 FP64 lanes a clock and
 * SM, and a warp whose nodes meet their neighbours at different steps of the
 * walk ran the 22 FP64 instructions of a term at nearly every one of its 290
 * steps: 1,492 us for 0.31 M nodes.  The whole call went from 1,662 to 255 us,
 * to 185 without building neighbour lists that the nodes never read, and to 121
 * with the bricks below.  Here
 *  - a thread first collects its candidates by the single-precision test (a
 *    1e-4 band around h^2), then evaluates them together with the others of
 *    its warp (about 35 terms, all lanes busy); a warp is a brick of nodes, so
 *    its lanes walk the same cells;
 *  - the terms are sums and products of split floats (48 bits: relative errors
 *    of 1e-14 where the sum that takes them is rounded to 6e-8), about 105
 *    single-precision instructions;
 *  - lengths are scaled by a power of two (len.sc, exact) so that h lies in
 *    [1, 2): no step leaves the range of floats for any h. */
struct LatticeLen {
    float sc;        /* the power of two */
    float h2;        /* fl32(h h) sc^2 */
    Split hh;        /* h^2 sc^2 */
    Split c;         /* m aw / sc^6 */
};
/* A node's sum. */
struct LatticeNode {
    Split x, y, z; /* its position */
    float acc = 0.0f;
    /* ((a - x) sc)^2 */
    __device__ __forceinline__ static Split square(Split a, float x, float sc) {
        const Split e = two_diff(a.h, x);
        const Split t = renorm(e.h, __fadd_rn(e.l, a.l));
        const float h = __fmul_rn(t.h, sc), l = __fmul_rn(t.l, sc);
        Split q = two_prod(h, h);
        q.l = __fmaf_rn(__fadd_rn(h, h), l, q.l);
        return q;
    }
    __device__ __forceinline__ void add(const LatticeLen &len, const float4 &xq) {
        const Split a = square(x, xq.x, len.sc), b = square(y, xq.y, len.sc), d = square(z, xq.z, len.sc);
        const Split ab = two_sum(a.h, b.h), abd = two_sum(ab.h, d.h);
        const float d2 =
            __fadd_rn(abd.h, __fadd_rn(__fadd_rn(__fadd_rn(a.l, b.l), d.l), __fadd_rn(ab.l, abd.l)));
        if (!(d2 <= len.h2)) return;
        const float r = __fsqrt_rn(d2);
        const Split rr = two_prod(r, r);
        const Split dq = two_diff(len.hh.h, rr.h);
        const Split q = renorm(dq.h, __fsub_rn(__fadd_rn(dq.l, len.hh.l), rr.l)); /* h^2 - r^2 */
        Split q2 = two_prod(q.h, q.h);
        q2.l = __fmaf_rn(__fadd_rn(q.h, q.h), q.l, q2.l);
        Split q3 = two_prod(q2.h, q.h);
        q3.l = __fmaf_rn(q2.l, q.h, __fmaf_rn(q2.h, q.l, q3.l));
        Split w = two_prod(len.c.h, q3.h);
        w.l = __fmaf_rn(len.c.l, q3.h, __fmaf_rn(len.c.h, q3.l, w.l));
        const Split sum = two_sum(acc, w.h);
        acc = __fadd_rn(sum.h, __fadd_rn(sum.l, w.l));
    }
};
constexpr int kLatBlock = 128, kLatMax = 48; /* threads a block; candidates collected before they are evaluated */
__global__ void __launch_bounds__(kLatBlock) k_density_grid(DevParams p, const unsigned int *__restrict__ cell_start,
                                                            const float4 *__restrict__ pos, int nx, int ny, int nz,
                                                            int3 lb, LatticeLen len, double3 minp, double3 dd,
                                                            double3 lo, double3 hi, float *__restrict__ out) {
    __shared__ unsigned int s_j[kLatMax][kLatBlock];
    /* a warp's brick of 2^lb.x x 2^lb.y x 2^lb.z nodes */
    const int lane = threadIdx.x & 31;
    const int bx = (nx + (1 << lb.x) - 1) >> lb.x, by = (ny + (1 << lb.y) - 1) >> lb.y;
    const long long brick = (long long)blockIdx.x * (kLatBlock / 32) + (threadIdx.x >> 5);
    const long long i = ((brick % bx) << lb.x) + (lane & ((1 << lb.x) - 1));
    const long long j = (((brick / bx) % by) << lb.y) + ((lane >> lb.x) & ((1 << lb.y) - 1));
    const long long k = ((brick / ((long long)bx * by)) << lb.z) + (lane >> (lb.x + lb.y));
    if (i >= nx || j >= ny || k >= nz) return;
    /* minp + Vec3(i, j, k) * d, each product and sum rounded in double */
    const double X = __dadd_rn(minp.x, __dmul_rn((double)i, dd.x));
    const double Y = __dadd_rn(minp.y, __dmul_rn((double)j, dd.y));
    const double Z = __dadd_rn(minp.z, __dmul_rn((double)k, dd.z));
    LatticeNode node{split_of(X), split_of(Y), split_of(Z)};
    if (X >= lo.x && X <= hi.x && Y >= lo.y && Y <= hi.y && Z >= lo.z && Z <= hi.z) {
        const float3 xf = make_float3(node.x.h, node.y.h, node.z.h);
        const int3 c = cell_of(xf, p);
        const float band = p.h2 * (1.0f + 1e-4f);
        int m = 0;
        auto evaluate = [&]() {
            for (int t = 0; t < m; ++t) node.add(len, __ldg(pos + s_j[t][threadIdx.x]));
            m = 0;
        };
        for (int dz = -1; dz <= 1; ++dz)
            for (int dy = -1; dy <= 1; ++dy) {
                unsigned int s, e;
                row_range(cell_start, c, dy, dz, p, s, e);
                for (unsigned int q0 = s; q0 < e; q0 += 4) { /* four loads in flight */
                    float4 xq[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) xq[u] = __ldg(pos + min(q0 + u, e - 1));
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float3 df = xf - f3(xq[u]);
                        if (q0 + u >= e || dot3(df, df) > band) continue;
                        if (m == kLatMax) evaluate();
                        s_j[m++][threadIdx.x] = q0 + u;
                    }
                }
            }
        evaluate();
    }
    out[(k * ny + j) * nx + i] = node.acc;
}

/* The same for bricks that are small against h (launch_density_grid): their nodes
 * share most of their candidates.  The warp gathers the particles within h of the
 * brick's box, 32 loads side by side, into shared memory, each lane tests them (8
 * instructions, one broadcast for the warp) into a mask and evaluates what passed,
 * in slot order as above.  0.31 M nodes h / 2 apart 88 us instead of 148, in which
 * each lane walked its own 27 cells. */
constexpr int kLatNear = 256; /* particles gathered before they are tested */
__global__ void __launch_bounds__(kLatBlock) k_density_brick(DevParams p, const unsigned int *__restrict__ cell_start,
                                                             const float4 *__restrict__ pos, int nx, int ny, int nz,
                                                             int3 lb, LatticeLen len, double3 minp, double3 dd,
                                                             double3 lo, double3 hi, float *__restrict__ out) {
    __shared__ float4 s_near[kLatBlock / 32][kLatNear];
    __shared__ unsigned int s_mask[kLatBlock / 32][kLatNear / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4 *const near = s_near[warp];
    const int bx = (nx + (1 << lb.x) - 1) >> lb.x, by = (ny + (1 << lb.y) - 1) >> lb.y;
    const long long brick = (long long)blockIdx.x * (kLatBlock / 32) + warp;
    const long long i = ((brick % bx) << lb.x) + (lane & ((1 << lb.x) - 1));
    const long long j = (((brick / bx) % by) << lb.y) + ((lane >> lb.x) & ((1 << lb.y) - 1));
    const long long k = ((brick / ((long long)bx * by)) << lb.z) + (lane >> (lb.x + lb.y));
    const bool mine = i < nx && j < ny && k < nz;
    const double X = __dadd_rn(minp.x, __dmul_rn((double)i, dd.x));
    const double Y = __dadd_rn(minp.y, __dmul_rn((double)j, dd.y));
    const double Z = __dadd_rn(minp.z, __dmul_rn((double)k, dd.z));
    const bool live = mine && X >= lo.x && X <= hi.x && Y >= lo.y && Y <= hi.y && Z >= lo.z && Z <= hi.z;
    LatticeNode node{split_of(X), split_of(Y), split_of(Z)};
    if (__any_sync(0xffffffffu, live)) {
        const float3 xf = make_float3(node.x.h, node.y.h, node.z.h);
        const float big = 3e38f;
        const float3 b0 = make_float3(-warp_max(live ? -xf.x : -big), -warp_max(live ? -xf.y : -big),
                                      -warp_max(live ? -xf.z : -big));
        const float3 b1 = make_float3(warp_max(live ? xf.x : -big), warp_max(live ? xf.y : -big),
                                      warp_max(live ? xf.z : -big));
        const int3 c0 = cell_of(b0, p), c1 = cell_of(b1, p);
        const float band = p.h2 * (1.0f + 1e-4f);
        int n = 0;
        auto evaluate = [&]() {
            __syncwarp();
            unsigned int some = 0u;
            for (int w = 0; 32 * w < n; ++w) {
                unsigned int m = 0u;
#pragma unroll 8
                for (int b = 0; b < 32; ++b) {
                    const float3 d = xf - f3(near[32 * w + b]);
                    m = __funnelshift_l(__float_as_uint(fmaf(d.z, d.z, fmaf(d.y, d.y, fmaf(d.x, d.x, -band)))), m, 1);
                }
                if (n < 32 * w + 32) m &= 0xffffffffu << (32 * w + 32 - n); /* what lies past the last */
                s_mask[warp][w][lane] = m;
                if (m) some |= 0x80000000u >> w;
            }
            if (!live) some = 0u;
            unsigned int m = 0u;
            int w = 0;
            while (m || some) {
                if (!m) {
                    w = __clz((int)some);
                    some &= ~(0x80000000u >> w);
                    m = s_mask[warp][w][lane];
                }
                const int b = __clz((int)m);
                m &= ~(0x80000000u >> b);
                node.add(len, near[32 * w + b]);
            }
            __syncwarp();
            n = 0;
        };
        for (int z = c0.z - 1; z <= c1.z + 1; ++z)
            for (int y = c0.y - 1; y <= c1.y + 1; ++y) {
                const unsigned int f = cell_index(make_int3(c0.x, y, z), p), l = cell_index(make_int3(c1.x, y, z), p);
                if (!cell_row_ok(p, f) || !cell_row_ok(p, l)) continue;
                const unsigned int s = __ldg(cell_start + f - 1);
                const unsigned int e = bounded(p, __ldg(cell_start + l + 2), (unsigned int)p.n + 1u, kBoundSlot);
                for (unsigned int q0 = s; q0 < e; q0 += 32) {
                    const float4 x = __ldg(pos + min(q0 + lane, e - 1));
                    const float dx = fmaxf(fmaxf(b0.x - x.x, x.x - b1.x), 0.0f);
                    const float dy = fmaxf(fmaxf(b0.y - x.y, x.y - b1.y), 0.0f);
                    const float dz = fmaxf(fmaxf(b0.z - x.z, x.z - b1.z), 0.0f);
                    const bool in = q0 + lane < e && dx * dx + dy * dy + dz * dz <= band;
                    const unsigned int hit = __ballot_sync(0xffffffffu, in);
                    if (n + __popc(hit) > kLatNear) evaluate();
                    if (in) near[n + __popc(hit & ((1u << lane) - 1u))] = x;
                    n += __popc(hit);
                }
            }
        evaluate();
    }
    if (mine) out[(k * ny + j) * nx + i] = node.acc;
}

/* ======================================================================== */
/* order conversion                                                         */
/* ======================================================================== */

__global__ void k_unsort4(int n, const unsigned int *__restrict__ id, const float4 *__restrict__ src,
                          float4 *__restrict__ dst, int zero_w) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    float4 v = src[d];
    if (zero_w) v.w = 0.0f;
    dst[id[d]] = v;
}
__global__ void k_unsort1(int n, const unsigned int *__restrict__ id, const unsigned int *__restrict__ src,
                          unsigned int *__restrict__ dst) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    dst[id[d]] = src[d];
}
__global__ void k_unsort_w(int n, const unsigned int *__restrict__ id, const float4 *__restrict__ src,
                           float *__restrict__ dst) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    dst[id[d]] = src[d].w;
}
__global__ void k_unsort_rows(int n, const unsigned int *__restrict__ id, const float4 *__restrict__ src,
                              float4 *__restrict__ dst, int k4) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * k4) return;
    int d = e / k4, q = e % k4;
    dst[(size_t)id[d] * k4 + q] = src[e];
}
void launch_unsort_rows(int n, const unsigned int *id, const float4 *src, float4 *dst, int k4, cudaStream_t s) {
    k_unsort_rows<<<blocks_for((long long)n * k4), kBlock, 0, s>>>(n, id, src, dst, k4);
}
__global__ void k_iota(int n, unsigned int *dst) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d < n) dst[d] = (unsigned int)d;
}
/* The caller's vectors a (and b), checked and, where dst is given, copied on
 * the way.  *bad lies in pinned host memory: the host clears it, waits for the
 * stream and reads it, so no memset and no copy go with a check.  A frame that
 * writes positions and velocities and reads three arrays on the device spent
 * 100 us outside its step, whatever its size below 262 k particles, in copies,
 * memsets and launches around five waits; with the copies done by this kernel
 * and the reordering ones it spends 60 us (WCSPH, 32 k: 157 -> 119 us). */
__global__ void k_check_finite(int n, const float4 *__restrict__ a, const float4 *__restrict__ b,
                               float4 *__restrict__ dst_a, float4 *__restrict__ dst_b, unsigned int *bad) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    float4 x = a[d];
    if (dst_a) dst_a[d] = x;
    bool ok = isfinite(x.x) && isfinite(x.y) && isfinite(x.z);
    if (b) {
        float4 v = b[d];
        if (dst_b) dst_b[d] = v;
        ok = ok && isfinite(v.x) && isfinite(v.y) && isfinite(v.z);
    }
    if (!ok) *bad = 1u;
}
void launch_check_finite(int n, const float4 *a, const float4 *b, unsigned int *bad, cudaStream_t s, float4 *dst_a,
                         float4 *dst_b) {
    k_check_finite<<<blocks_for(n), kBlock, 0, s>>>(n, a, b, dst_a, dst_b, bad);
}
__global__ void k_pack_w(int n, float4 *dst, const float *w) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d < n) dst[d].w = w[d];
}

/* ======================================================================== */
/* launchers                                                                */
/* ======================================================================== */

void launch_predict_hash(const DevParams &p, const float4 *pos, const float4 *vel, const float4 *acc,
                         float4 *ppos_out, unsigned int *key, unsigned int *rank, unsigned int *count,
                         const float4 *dwarm, float4 *xpred_out, cudaStream_t s) {
    k_predict_hash<<<blocks_for(p.n), kBlock, 0, s>>>(p, pos, vel, acc, ppos_out, key, rank, count, dwarm,
                                                      xpred_out);
}
void launch_hash(const DevParams &p, const float4 *x, unsigned int *key, unsigned int *rank, unsigned int *count,
                 cudaStream_t s) {
    k_hash<<<blocks_for(p.n), kBlock, 0, s>>>(p, x, key, rank, count);
}
void launch_scan(unsigned int *count, unsigned int *cell_start, unsigned int *block_sums, unsigned int ncells,
                 cudaStream_t s) {
    const unsigned int nb = scan_blocks(ncells);
    k_scan_local<<<nb, kScanBlock, 0, s>>>(count, cell_start, block_sums, ncells);
    if (nb == 1) return;
    /* Up to kScanSum tiles every block of the last phase sums the totals before
     * it itself (at most kScanSum / kScanBlock loads a thread) instead of a phase of
     * one block between the two: a launch less, about 4 us of each grid build.
     * Past it those loads (nb^2 / 2 words in all) cost more than the launch. */
    if (nb <= kScanSum) {
        k_scan_add<true><<<nb, kScanBlock, 0, s>>>(cell_start, block_sums, ncells);
    } else {
        k_scan_top<<<1, 1024, 0, s>>>(block_sums, nb, cell_start, ncells);
        k_scan_add<false><<<nb, kScanBlock, 0, s>>>(cell_start, block_sums, ncells);
    }
}
bool launch_small_grid(const DevParams &p, unsigned int ncells, const float4 *x4, float4 *x_out, unsigned int *order,
                       unsigned int *cell_start, cudaStream_t s) {
    /* up to kSmallGrid particles (8 a thread) whose table fits beside them in
     * shared memory: 8,000 particles take 27 us with the pass behind, 8,400 in
     * five launches 36 */
    constexpr size_t most = 200 * 1024;
    const size_t bytes = ((size_t)ncells + 1 + (size_t)p.n) * sizeof(unsigned int);
    if (p.n > kSmallGrid || bytes > most) return false;
    static PerDevice limit;
    if (!raise_shared_limit(limit, (const void *)k_small_grid, most)) return false;
    k_small_grid<<<1, 1024, bytes, s>>>(p, ncells, x4, x_out, order, cell_start);
    return true;
}
CellOrder launch_scatter(const DevParams &p, const unsigned int *key, const unsigned int *rank,
                         const unsigned int *cell_start, unsigned int *perm, cudaStream_t s) {
    k_scatter<<<blocks_for(p.n), kBlock, 0, s>>>(p.n, key, rank, cell_start, perm);
    CellOrder o;
    o.perm = perm;
    o.key = key;
    o.cell_start = cell_start;
    return o;
}
void launch_gather(int n, const CellOrder &o, const Gather &g, DevCtl *count_build, cudaStream_t s) {
    k_gather<<<blocks_for(n), kBlock, 0, s>>>(n, o, g, count_build);
}
void launch_hash_parity(const DevParams &p, const float4 *ppos0, const float4 *ppos1, const DevCtl *ctl,
                        unsigned int *key, unsigned int *rank, unsigned int *count, cudaStream_t s) {
    k_hash_parity<<<blocks_for(p.n), kBlock, 0, s>>>(p, ppos0, ppos1, ctl, key, rank, count);
}
void launch_rebuild_gather(int n, const CellOrder &o, const DevCtl *ctl, const float4 *pos, const float4 *ppos0,
                           const float4 *ppos1, const unsigned int *id, const unsigned int *attr, const float *dens,
                           float4 *t_pos, float4 *t_x, unsigned int *t_id, unsigned int *t_attr, float *t_dens,
                           const unsigned int *key, unsigned int *cellb, const float4 *xpred, float4 *t_xpred,
                           float *t_lam, cudaStream_t s) {
    k_rebuild_gather<<<blocks_for(n), kBlock, 0, s>>>(n, o, ctl, pos, ppos0, ppos1, id, attr, dens, t_pos, t_x,
                                                      t_id, t_attr, t_dens, key, cellb, xpred, t_xpred, t_lam);
}
void launch_rebuild_copy(int n, DevCtl *ctl, const float4 *t_pos, const float4 *t_x, const unsigned int *t_id,
                         const unsigned int *t_attr, const float *t_dens, float4 *pos, float4 *ppos0, float4 *ppos1,
                         float4 *xb, unsigned int *id, unsigned int *attr, float *dens, const float4 *t_xpred,
                         float4 *xpred, const float *t_lam, cudaStream_t s) {
    k_rebuild_copy<<<blocks_for(n), kBlock, 0, s>>>(n, ctl, t_pos, t_x, t_id, t_attr, t_dens, pos, ppos0, ppos1, xb,
                                                    id, attr, dens, t_xpred, xpred, t_lam);
}
void launch_pbf_density(const DevParams &p, const unsigned int *cell_start, const float4 *pos, float *dens,
                        cudaStream_t s) {
    k_pbf_density<<<blocks_for(p.n), kBlock, 0, s>>>(p, cell_start, pos, dens);
}
void launch_pbf_visc(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const float4 *vel,
                     const float *dens, float4 *acc, cudaStream_t s) {
    k_pbf_visc<<<blocks_for(p.n), kBlock, 0, s>>>(p, cell_start, pos, vel, dens, acc);
}
/* resident blocks of the persistent lambda pass, looked up once per kernel
 * (contexts may step from several host threads) */
static unsigned int resident_blocks(const void *kernel) {
    static std::mutex mu;
    static const void *known[2] = {nullptr, nullptr};
    static int resident[2] = {0, 0};
    std::lock_guard<std::mutex> lock(mu);
    const int k = !known[0] || known[0] == kernel ? 0 : 1;
    if (known[k] != kernel) {
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kPassBlock, 0);
        resident[k] = std::max(1, sms * std::max(per, 1));
        known[k] = kernel;
    }
    return (unsigned int)resident[k];
}

/* the passes' shape by size (kDeepMax in fsph_kernels.cuh) */
static bool deep_pass(const DevParams &p) { return p.n <= kDeepMax && p.use_lists; }
static bool deep_constraint(const DevParams &p) {
    return p.n <= (p.nb ? kDeepMaxBoundary : kDeepMax) && p.use_lists;
}

void launch_lambda(const DevParams &p, const unsigned int *cell_start, float4 *ppos0, float4 *ppos1, float *dens,
                   DevCtl *ctl, ErrPartial *part, unsigned long long while_handle, int use_graph,
                   const NbrLists &nl, cudaStream_t s) {
    const bool deep = deep_constraint(p);
    auto k = deep ? (p.compensated ? k_lambda<true, true> : k_lambda<false, true>)
                  : (p.compensated ? k_lambda<true, false> : k_lambda<false, false>);
    const unsigned int blocks = deep ? blocks_for(p.n, kDeepBlock)
                                     : std::min(blocks_for(p.n, kPassBlock), resident_blocks((const void *)k));
    k<<<blocks, deep ? kDeepBlock : kPassBlock, 0, s>>>(p, cell_start, ppos0, ppos1, dens, ctl, part,
                                                        (cudaGraphConditionalHandle)while_handle, use_graph,
                                                        p.use_lists ? nl.list : nullptr, nl.cnt);
}
/* The list build: four warps / one warp for 32 slots take, in us, 10.3 / 16.4 at
 * 6,912 slots, 12.3 / 15.8 at 16,384, 16.5 / 20.5 at 32,000, 19.5 / 17.2 at 42,592,
 * 23.0 / 18.5 at 62,500 (two 18.5 at 32,000, eight 20.5). */
constexpr int kListSplitMax = 1 << 15;
void launch_build_list(const DevParams &p, const unsigned int *cell_start, const float4 *xb, const NbrLists &nl,
                       cudaStream_t s) {
    if (!p.use_lists) return;
    if (p.n <= kListSplitMax)
        k_build_list<4><<<blocks_for(p.n, 32), 128, 0, s>>>(p, cell_start, xb, nl.cellb, nl.list, nl.cnt);
    else
        k_build_list<1><<<blocks_for(p.n, kListBlock), kListBlock, 0, s>>>(p, cell_start, xb, nl.cellb, nl.list, nl.cnt);
}
void launch_correction(const DevParams &p, const unsigned int *cell_start, float4 *ppos0, float4 *ppos1,
                       const float4 *xb, DevCtl *ctl, float *part, unsigned long long if_handle,
                       unsigned long long if_handle2, int use_graph, float4 *dp_out, const NbrLists &nl,
                       cudaStream_t s) {
    const bool deep = deep_constraint(p);
    auto k = deep ? k_correction<true> : k_correction<false>;
    const int block = deep ? kDeepBlock : kPassBlock;
    k<<<blocks_for(p.n, block), block, 0, s>>>(p, cell_start, ppos0, ppos1, xb, ctl, part,
                                               (cudaGraphConditionalHandle)if_handle,
                                               (cudaGraphConditionalHandle)if_handle2, use_graph, dp_out,
                                               p.use_lists ? nl.list : nullptr, nl.cnt);
}
void launch_finalize(const DevParams &p, const float4 *pos_b, const float4 *ppos0, const float4 *ppos1,
                     const DevCtl *ctl, const unsigned int *id_b, const unsigned int *attr_b, float4 *pos_a,
                     float4 *vel_a, unsigned int *id_a, unsigned int *attr_a, const float4 *xpred, float4 *dstep,
                     cudaStream_t s, const float *dens, float4 *xm) {
    k_finalize<<<blocks_for(p.n), kBlock, 0, s>>>(p, pos_b, ppos0, ppos1, ctl, id_b, attr_b, pos_a, vel_a, id_a,
                                                  attr_a, xpred, dstep, dens, xm);
}
void launch_xsph_vort(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const float4 *vel,
                      const float *dens, float4 *vel_out, float4 *vort, const FeatureOut &fo, const NbrLists &nl,
                      cudaStream_t s, float *mag) {
    /* the neighbour means cost a gather per pair: only when they are used */
    const bool deep = mag && deep_pass(p), nbr = fo.nbr != 0;
    auto k = !mag      ? k_xsph_vort<false, false, false, false>
             : fo.feat ? (deep ? (nbr ? k_xsph_vort<true, true, true, true> : k_xsph_vort<true, false, true, true>)
                               : (nbr ? k_xsph_vort<true, true, true, false> : k_xsph_vort<true, false, true, false>))
                       : (deep ? k_xsph_vort<false, false, true, true> : k_xsph_vort<false, false, true, false>);
    const int block = deep ? kDeepBlock : kPostBlock;
    k<<<blocks_for(p.n, block), block, 0, s>>>(p, cell_start, pos, vel, dens, vel_out, vort, fo,
                                               p.use_lists ? nl.list : nullptr, nl.cnt, mag);
}
void launch_vort_apply(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const float4 *vort,
                       const float *dens, const float4 *vel_in, float4 *vel_out, const NbrLists &nl, cudaStream_t s,
                       const float *mag) {
    const bool deep = mag && deep_pass(p);
    auto k = deep ? k_vort_apply<true, true> : mag ? k_vort_apply<true, false> : k_vort_apply<false, false>;
    const int block = deep ? kDeepBlock : kPostBlock;
    k<<<blocks_for(p.n, block), block, 0, s>>>(p, cell_start, pos, vort, dens, vel_in, vel_out,
                                               p.use_lists ? nl.list : nullptr, nl.cnt, mag);
}
/* lanes per particle (a power of two, at most `most`): enough that the launch
 * holds about as many threads as the GPU keeps resident (1536 per SM) */
static int lanes_to_fill(int n, int most) {
    static const int resident = [] { /* initialised once, thread-safely */
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        return std::max(sms, 1) * 1536;
    }();
    int lanes = 1;
    while (lanes < most && (long long)n * lanes < (long long)resident) lanes *= 2;
    return lanes;
}
static int sph_force_lanes(int n) { return lanes_to_fill(n, 8); }
/* The density pass by size, us at 8,000 / 15,625 / 32,768 / 64,000 / 125,000 /
 * 262,144 slots: a warp a particle 10.9 / 16.3 / 22.7 / 51.3 / - / -, four warps
 * for the tile of 32 slots 14.4 / 14.3 / 16.4 / 28.2 / 45.5 / 84.5, one warp 20.5 /
 * 22.5 / 22.8 / 28.8 / 36.9 / 59.6; at 4,096 a warp a particle takes 8.7 (eight
 * lanes 16.4). */
constexpr int kSphTileMin = 12288, kSphSplitMax = 1 << 16;
void launch_sph_density(const DevParams &p, const unsigned int *cell_start, float4 *pos, float4 *vel, float *dens,
                        float *pres, const NbrLists &nl, cudaStream_t s) {
    ListEntry *l = p.use_lists ? nl.list : nullptr;
    if (p.n > kSphSplitMax) {
        k_sph_density<1><<<blocks_for(p.n, kListBlock), kListBlock, 0, s>>>(p, cell_start, pos, vel, dens, pres, l, nl.cnt);
        return;
    }
    if (p.n >= kSphTileMin) {
        k_sph_density<4><<<blocks_for(p.n, 32), 128, 0, s>>>(p, cell_start, pos, vel, dens, pres, l, nl.cnt);
        return;
    }
    k_sph_density_lanes<<<blocks_for((long long)p.n * 32), kBlock, 0, s>>>(p, cell_start, pos, vel, dens, pres, l, nl.cnt);
}
void launch_lambda_walk(const DevParams &p, const unsigned int *cell_start, const float4 *x, const unsigned int *order,
                        float *dens, float *lambda, cudaStream_t s) {
    const int lanes = lanes_to_fill(p.n, 32);
    auto k = p.compensated ? (lanes >= 32   ? k_lambda_walk<32, true>
                              : lanes >= 16 ? k_lambda_walk<16, true>
                              : lanes >= 8  ? k_lambda_walk<8, true>
                                            : k_lambda_walk<4, true>)
                           : (lanes >= 32   ? k_lambda_walk<32, false>
                              : lanes >= 16 ? k_lambda_walk<16, false>
                              : lanes >= 8  ? k_lambda_walk<8, false>
                                            : k_lambda_walk<4, false>);
    const int lpp = lanes >= 4 ? lanes : 4;
    k<<<blocks_for((long long)p.n * lpp), kBlock, 0, s>>>(p, cell_start, x, order, dens, lambda);
}
void launch_sph_force(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const float4 *vel,
                      float4 *acc, const NbrLists &nl, cudaStream_t s) {
    const ListEntry *l = p.use_lists ? nl.list : nullptr;
    const int lanes = sph_force_lanes(p.n);
    const unsigned int g = blocks_for((long long)p.n * lanes);
    switch (lanes) {
    case 1: k_sph_force<1><<<g, kBlock, 0, s>>>(p, cell_start, pos, vel, acc, l, nl.cnt); break;
    case 2: k_sph_force<2><<<g, kBlock, 0, s>>>(p, cell_start, pos, vel, acc, l, nl.cnt); break;
    case 4: k_sph_force<4><<<g, kBlock, 0, s>>>(p, cell_start, pos, vel, acc, l, nl.cnt); break;
    default: k_sph_force<8><<<g, kBlock, 0, s>>>(p, cell_start, pos, vel, acc, l, nl.cnt); break;
    }
}
void launch_sph_integrate(const DevParams &p, const float4 *pos_b, const float4 *vel_b, const float4 *acc,
                          const unsigned int *id_b, const unsigned int *attr_b, float4 *pos_a, float4 *vel_a,
                          unsigned int *id_a, unsigned int *attr_a, cudaStream_t s) {
    k_sph_integrate<<<blocks_for(p.n), kBlock, 0, s>>>(p, pos_b, vel_b, acc, id_b, attr_b, pos_a, vel_a, id_a,
                                                       attr_a);
}
void launch_nb_count(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const unsigned int *id,
                     unsigned int *cnt_p, unsigned long long *total, const NbrLists &nl, cudaStream_t s) {
    k_nb_count<<<blocks_for(p.n, kListBlock), kListBlock, 0, s>>>(p, cell_start, pos, id, cnt_p, total, nl.list,
                                                                  nl.cnt);
}
void launch_nb_rows(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const unsigned int *id,
                    const unsigned int *offsets, const NbrLists &nl, int *out, float *d2out, cudaStream_t s) {
    k_nb_rows<<<blocks_for((long long)p.n * 32), kBlock, 0, s>>>(p, cell_start, pos, id, offsets, nl.list, nl.cnt, out,
                                                                 d2out);
}
void launch_delete_regions(int n, float4 *pos, float4 *vel, unsigned int *attr, const float4 *reg, int nreg,
                           cudaStream_t s) {
    if (n > 0 && nreg > 0) k_delete_regions<<<blocks_for(n), kBlock, 0, s>>>(n, pos, vel, attr, reg, nreg);
}
void launch_mark_active(int n, const unsigned int *attr, unsigned int *keep, cudaStream_t s) {
    if (n > 0) k_mark_active<<<blocks_for(n), kBlock, 0, s>>>(n, attr, keep);
}
void launch_partition_perm(int n, const unsigned int *scan, unsigned int *perm, cudaStream_t s) {
    if (n > 0) k_partition_perm<<<blocks_for(n), kBlock, 0, s>>>(n, scan, perm);
}
void launch_gather_rows(int n, const unsigned int *perm, const float4 *src, float4 *dst, int k4, cudaStream_t s) {
    if (n > 0) k_gather_rows<<<blocks_for((long long)n * k4), kBlock, 0, s>>>(n, perm, src, dst, k4);
}
constexpr double kLatShare = 130.0;
void launch_density_grid(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const int nn[3],
                         const double minp[3], const double d[3], const double lo[3], const double hi[3], float *out,
                         cudaStream_t s) {
    /* bricks of 4 x 4 x 2 nodes; an axis with fewer nodes gives its share to the others */
    int most[3], lb[3] = {2, 2, 1};
    for (int a = 0; a < 3; ++a) {
        most[a] = 0;
        while (most[a] < 5 && (1ll << most[a]) < nn[a]) ++most[a];
        lb[a] = std::min(lb[a], most[a]);
    }
    for (int a = 0; a < 3; ++a)
        while (lb[0] + lb[1] + lb[2] < 5 && lb[a] < most[a]) ++lb[a];
    lb[0] += 5 - (lb[0] + lb[1] + lb[2]); /* fewer than 32 nodes in all */
    long long bricks = 1;
    for (int a = 0; a < 3; ++a) bricks *= ((long long)nn[a] + (1 << lb[a]) - 1) >> lb[a];
    auto split = [](double v) {
        const float h = (float)v;
        return Split{h, (float)(v - (double)h)};
    };
    int ex = 0;
    std::frexp((double)p.h, &ex); /* h = f 2^ex, f in [1/2, 1) */
    const double sc = std::ldexp(1.0, 1 - ex), hs = (double)p.h * sc;
    LatticeLen len;
    len.sc = (float)sc;
    len.h2 = (float)((double)p.h2 * sc * sc);
    len.hh = split(hs * hs);
    len.c = split((double)p.mass * p.aw_d * std::ldexp(1.0, 6 * (ex - 1)));
    /* a brick's lanes share a gathered set while the box within h of the brick is
     * below kLatShare h^3 (a lane's own 27 cells are 36).  Calls over 1 M particles
     * with nodes 1.3 h apart (115 h^3) take 132 us so and 142 the other way, 1.6 h
     * (166 h^3) 142 and 126, h / 2 (35 h^3) 330 and 497 */
    double near = 1.0;
    for (int a = 0; a < 3; ++a) near *= ((1 << lb[a]) - 1) * std::fabs(d[a]) / (double)p.h + 2.0;
    auto kernel = near <= kLatShare ? k_density_brick : k_density_grid;
    kernel<<<blocks_for(bricks, kLatBlock / 32), kLatBlock, 0, s>>>(
        p, cell_start, pos, nn[0], nn[1], nn[2], make_int3(lb[0], lb[1], lb[2]), len,
        make_double3(minp[0], minp[1], minp[2]), make_double3(d[0], d[1], d[2]), make_double3(lo[0], lo[1], lo[2]),
        make_double3(hi[0], hi[1], hi[2]), out);
}
/* The reference's cell hash of each position (z Gy Gx + y Gx + x):
 * rule 0 = its CPU grid (rxNNGrid::CalGridHash(Vec3), rx_nnsearch.h:590-599:
 * (p - min) / cw in double, truncated to int, clamped to [0, G-1]);
 * rule 1 = its GPU grid (calcGridPos / calcGridHash, rx_cu_common.cu:121-144:
 * floor((p - origin) / cw) in float, clamped). */
__global__ void __launch_bounds__(kBlock) k_reference_cells(int n, const float4 *__restrict__ pos, int rule,
                                                            double3 org, double cw, int gx, int gy, int gz,
                                                            unsigned int *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 x = pos[i];
    int c[3];
    const int g[3] = {gx, gy, gz};
    const float xf[3] = {x.x, x.y, x.z};
    const double o[3] = {org.x, org.y, org.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int k;
        if (rule == 0) {
            k = (int)__ddiv_rn((double)xf[a] - o[a], cw);
        } else {
            k = (int)floorf(__fdiv_rn(__fsub_rn(xf[a], (float)o[a]), (float)cw));
        }
        c[a] = k < 0 ? 0 : (k >= g[a] ? g[a] - 1 : k);
    }
    out[i] = ((unsigned int)c[2] * (unsigned int)gy + (unsigned int)c[1]) * (unsigned int)gx + (unsigned int)c[0];
}

/* The triangle-mesh collision alone, for parity: x1 and v updated in place
 * from the segments x0 -> x1. */
__global__ void __launch_bounds__(kBlock) k_polygon_collide(DevParams p, int n, const float4 *__restrict__ x0,
                                                            float4 *__restrict__ x1, float4 *__restrict__ v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float3 x = f3(x1[i]), vv = f3(v[i]);
    polygon_collide(f3(x0[i]), x, vv, p.dt, p);
    x1[i] = make_float4(x.x, x.y, x.z, x1[i].w);
    v[i] = make_float4(vv.x, vv.y, vv.z, v[i].w);
}
void launch_polygon_collide(const DevParams &p, int n, const float4 *x0, float4 *x1, float4 *v, cudaStream_t s) {
    if (n > 0 && p.ntri) k_polygon_collide<<<blocks_for(n), kBlock, 0, s>>>(p, n, x0, x1, v);
}

void launch_reference_cells(int n, const float4 *pos, int rule, const double org[3], double cw, const int g[3],
                            unsigned int *out, cudaStream_t s) {
    if (n > 0)
        k_reference_cells<<<blocks_for(n), kBlock, 0, s>>>(n, pos, rule, make_double3(org[0], org[1], org[2]), cw,
                                                          g[0], g[1], g[2], out);
}

void launch_unsort4(int n, const unsigned int *id, const float4 *src, float4 *dst, int zero_w, cudaStream_t s) {
    k_unsort4<<<blocks_for(n), kBlock, 0, s>>>(n, id, src, dst, zero_w);
}
void launch_unsort1(int n, const unsigned int *id, const unsigned int *src, unsigned int *dst, cudaStream_t s) {
    k_unsort1<<<blocks_for(n), kBlock, 0, s>>>(n, id, src, dst);
}
void launch_unsort_w(int n, const unsigned int *id, const float4 *src, float *dst, cudaStream_t s) {
    k_unsort_w<<<blocks_for(n), kBlock, 0, s>>>(n, id, src, dst);
}
void launch_iota(int n, unsigned int *dst, cudaStream_t s) { k_iota<<<blocks_for(n), kBlock, 0, s>>>(n, dst); }
void launch_pack_w(int n, float4 *dst, const float *w, cudaStream_t s) {
    k_pack_w<<<blocks_for(n), kBlock, 0, s>>>(n, dst, w);
}

}  // namespace fsph

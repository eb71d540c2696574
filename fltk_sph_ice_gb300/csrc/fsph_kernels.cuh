/*
 * fsph_kernels.cuh -- host-callable launchers of the fluid-step kernels
 * (defined in fsph_kernels.cu).  Every launcher enqueues on `s` and returns
 * without synchronising.
 */
#pragma once
#include "fsph_internal.cuh"
#include "fsph_per_device.h"

namespace fsph {

/* raises a kernel's dynamic shared-memory limit on the current device, once for
 * each (done: the kernel's own); false, with no error left pending, when it cannot */
inline bool raise_shared_limit(PerDevice &done, const void *kernel, size_t bytes) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return done.once(dev, [&] {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess)
            return true;
        cudaGetLastError();
        return false;
    });
}

constexpr int kBlock = 256;
/* threads per block of the two constraint passes (k_lambda, k_correction);
 * measured at 1 M particles against 256: 128 +6 %, 64 +38 %, 512 -0.8 %
 * per warm step */
#ifndef FSPH_PASS_BLOCK
#define FSPH_PASS_BLOCK 512
#endif
constexpr int kPassBlock = FSPH_PASS_BLOCK;
/* up to kDeepMax particles the list passes run in blocks of 64 with eight
 * candidates in flight (for_each_candidate's DEEP; 12 blocks an SM, 72
 * registers): 14 blocks of 512 left 138 SMs idle at 6,912 particles.  A lambda
 * and a correction pass together: 31.0 -> 22.6 us at 6,912, 33.0 -> 27.7 at
 * 32,000, 43.1 -> 42.0 at 131,072, 71.4 -> 81.6 at 294,912 */
constexpr int kDeepBlock = 64, kDeepMinB = 12, kDeepMax = 65536;
/* Beside a boundary a pass waits for the few warps at its shell, and which form is
 * the faster depends on where they land, which a particle count does not tell.
 * Drops of 20^3 to 40^3 particles, 3 to 10 iterations, two skins, deep against
 * plain: always the faster up to 13,824 (3 to 8 %), from 12 % faster to 12 % slower
 * up to 54,872 (46,656 the slower, 1,301 against 1,171 us; 54,872 the faster, 988
 * against 1,139), up to 22 % slower at 59,319 and from 6 % faster to 13 % slower at
 * 64,000.  The line only keeps the worst of it out. */
constexpr int kDeepMaxBoundary = 57344;
/* The XSPH and vorticity passes of larger scenes: a step of 1 M particles with two
 * iterations took 852 us in blocks of 128, 857 of 256, 865 of 512, 878 with eight
 * candidates in flight; with registers for five or six blocks of 256 per SM 867
 * and 914. */
constexpr int kPostBlock = 128;
constexpr int kListBlock = 128; /* threads per block of the list build: four warps with a tile of 8.8 KB each */
constexpr int kBlockMax = 512;  /* largest block of the batched persistent kernels */
constexpr int kScanTile = 4096, kScanBlock = 256; /* cells and threads per block of the first scan phase */
constexpr unsigned int kScanSum = 2048; /* tiles up to which the scan runs in two phases */

inline unsigned int blocks_for(long long n, int b = kBlock) { return (unsigned int)((n + b - 1) / b); }
inline unsigned int scan_blocks(unsigned int ncells) { return (ncells + kScanTile - 1) / kScanTile; }

/* ---- grid build: counting sort on the 64-bit key (cell << 32 | previous slot) ---- */
/* x* = walls(x + dt (v + dt a)), a = gravity when acc == NULL; then key + rank.
 * xpred_out (optional) keeps that prediction; dwarm (optional) is a warm-start
 * correction: the iterations then start from walls(x* + dwarm). */
void launch_predict_hash(const DevParams &p, const float4 *pos, const float4 *vel, const float4 *acc,
                         float4 *ppos_out, unsigned int *key, unsigned int *rank, unsigned int *count,
                         const float4 *dwarm, float4 *xpred_out, cudaStream_t s);
void launch_hash(const DevParams &p, const float4 *x, unsigned int *key, unsigned int *rank, unsigned int *count,
                 cudaStream_t s);
/* exclusive scan of count[C] into cell_start[C+1]; zeroes count for the next build */
void launch_scan(unsigned int *count, unsigned int *cell_start, unsigned int *block_sums, unsigned int ncells,
                 cudaStream_t s);
/* The order of a grid build.  key == NULL: perm[d] = the previous slot of slot
 * d.  Else perm holds each cell's previous slots in the arbitrary order of the
 * atomic ranks, and the kernel that moves the particles ranks them on the way
 * (ranked_slot in fsph_kernels.cu); sorted (optional) then receives the order
 * itself, for callers that need it afterwards. */
struct CellOrder {
    const unsigned int *perm = nullptr, *key = nullptr, *cell_start = nullptr;
    unsigned int *sorted = nullptr;
};
/* perm[cell_start[key] + rank] = slot; returns the order it stands for */
CellOrder launch_scatter(const DevParams &p, const unsigned int *key, const unsigned int *rank,
                         const unsigned int *cell_start, unsigned int *perm, cudaStream_t s);

/* the whole build of a small cloud (hash, scan, order, x4 into x_out, order[slot]
 * = particle) in one launch; false (nothing launched) when it is too large */
constexpr int kSmallGrid = 8192;
bool launch_small_grid(const DevParams &p, unsigned int ncells, const float4 *x4, float4 *x_out, unsigned int *order,
                       unsigned int *cell_start, cudaStream_t s);

/* dst[d] = src[previous slot of d] for up to 6 float4 and 4 u32 streams */
struct Gather {
    const float4 *src4[6];
    float4 *dst4[6];
    const unsigned int *src1[4];
    unsigned int *dst1[4];
    int n4, n1;
};
void launch_gather(int n, const CellOrder &o, const Gather &g, DevCtl *count_build, cudaStream_t s);

/* in-loop rebuild (the current x* buffer is chosen on the device by ctl->parity) */
void launch_hash_parity(const DevParams &p, const float4 *ppos0, const float4 *ppos1, const DevCtl *ctl,
                        unsigned int *key, unsigned int *rank, unsigned int *count, cudaStream_t s);
void launch_rebuild_gather(int n, const CellOrder &o, const DevCtl *ctl, const float4 *pos, const float4 *ppos0,
                           const float4 *ppos1, const unsigned int *id, const unsigned int *attr, const float *dens,
                           float4 *t_pos, float4 *t_x, unsigned int *t_id, unsigned int *t_attr, float *t_dens,
                           const unsigned int *key, unsigned int *cellb, const float4 *xpred, float4 *t_xpred,
                           float *t_lam, cudaStream_t s);

/* neighbour lists (see fsph_internal.cuh) */
struct NbrLists {
    ListEntry *list = nullptr;       /* [kListMax][n] */
    unsigned char *cnt = nullptr;    /* [n], kListOverflow = use the cell walk */
    unsigned int *cellb = nullptr;   /* [n] build cell of each slot */
};
/* lists of every slot from the build positions xb (a no-op when p.use_lists == 0) */
void launch_build_list(const DevParams &p, const unsigned int *cell_start, const float4 *xb, const NbrLists &nl,
                       cudaStream_t s);
void launch_rebuild_copy(int n, DevCtl *ctl, const float4 *t_pos, const float4 *t_x, const unsigned int *t_id,
                         const unsigned int *t_attr, const float *t_dens, float4 *pos, float4 *ppos0, float4 *ppos1,
                         float4 *xb, unsigned int *id, unsigned int *attr, float *dens, const float4 *t_xpred,
                         float4 *xpred, const float *t_lam, cudaStream_t s);

/* ---- PBF ---- */
void launch_pbf_density(const DevParams &p, const unsigned int *cell_start, const float4 *pos, float *dens,
                        cudaStream_t s);
void launch_pbf_visc(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const float4 *vel,
                     const float *dens, float4 *acc, cudaStream_t s);
void launch_lambda(const DevParams &p, const unsigned int *cell_start, float4 *ppos0, float4 *ppos1, float *dens,
                   DevCtl *ctl, ErrPartial *part, unsigned long long while_handle, int use_graph,
                   const NbrLists &nl, cudaStream_t s);
/* The whole constraint loop in one cooperative kernel (fsph_loop.cu): iterations
 * until the loop ends or a grid rebuild is due, then the three conditions are set
 * (use_graph: 1, with the third 3, outside a graph 0).  loop_fits: lists are on, there is no boundary (its
 * lambda is a kernel of its own between the passes) and every block is resident at
 * once.  Up to kLoopMax particles each has a thread of its own.  polls: before a
 * block gives a barrier up (0: the default). */
constexpr int kLoopMax = 65536;
bool loop_fits(const DevParams &p);
cudaError_t launch_pbf_loop(const DevParams &p, const unsigned int *cell_start, float4 *ppos0, float4 *ppos1,
                            float *dens, const float4 *xb, DevCtl *ctl, LoopCtl *lc, unsigned long long while_handle,
                            unsigned long long if_handle, unsigned long long if_handle2, int use_graph,
                            unsigned long long polls, const NbrLists &nl, cudaStream_t s);
/* density and lambda of x (slot order) at order[slot], walking the cells */
void launch_lambda_walk(const DevParams &p, const unsigned int *cell_start, const float4 *x, const unsigned int *order,
                        float *dens, float *lambda, cudaStream_t s);
void launch_correction(const DevParams &p, const unsigned int *cell_start, float4 *ppos0, float4 *ppos1,
                       const float4 *xb, DevCtl *ctl, float *part, unsigned long long if_handle,
                       unsigned long long if_handle2, int use_graph, float4 *dp_out, const NbrLists &nl,
                       cudaStream_t s);
void launch_finalize(const DevParams &p, const float4 *pos_b, const float4 *ppos0, const float4 *ppos1,
                     const DevCtl *ctl, const unsigned int *id_b, const unsigned int *attr_b, float4 *pos_a,
                     float4 *vel_a, unsigned int *id_a, unsigned int *attr_a, const float4 *xpred, float4 *dstep,
                     cudaStream_t s, const float *dens = nullptr, float4 *xm = nullptr);
/* XSPH + vorticity (omega) pass; with fo.feat (and mag) also the warm-start
 * features.  With mag, pos is launch_finalize's xm: the pass takes m / rho_j from
 * pos[j].w instead of dividing per pair and leaves |omega| in mag, which
 * launch_vort_apply then gathers with xm in place of vort and dens. */
void launch_xsph_vort(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const float4 *vel,
                      const float *dens, float4 *vel_out, float4 *vort, const FeatureOut &fo, const NbrLists &nl,
                      cudaStream_t s, float *mag = nullptr);
void launch_vort_apply(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const float4 *vort,
                       const float *dens, const float4 *vel_in, float4 *vel_out, const NbrLists &nl, cudaStream_t s,
                       const float *mag = nullptr);

/* ---- static boundary particles (p.bpos / p.bcell / p.bnear of the sorted boundary) ---- */
/* bscale[b] = rho0 psi_b / m with psi_b = m / sum_b' m W(r_bb') (rx_sph_pbd.cpp:1061-1090) */
void launch_boundary_volume(const DevParams &p, float *bscale, cudaStream_t s);
/* bstat[b] = (sum_b' rho0 psi_b' W, sum_b' |(rho0 psi_b' / m) grad W / rho0|^2): the static
 * boundary-boundary parts of lambda_b */
void launch_boundary_static(const DevParams &p, float2 *bstat, cudaStream_t s);
/* bnear[c] = 1 when any boundary slot lies in the 27 cells around cell c */
void launch_boundary_near(const DevParams &p, unsigned int ncells, unsigned char *bnear, cudaStream_t s);
/* lambda_b of every boundary particle from the fluid x* of the current parity (rx_sph_pbd.cpp:825-913) */
void launch_boundary_lambda(const DevParams &p, const unsigned int *cell_start, const float4 *ppos0,
                            const float4 *ppos1, const DevCtl *ctl, const float2 *bstat, float *blam, cudaStream_t s);

/* ---- WCSPH ---- */
/* density + pressure of the sorted positions, the force pass's neighbour
 * lists (nl.list / nl.cnt, when p.use_lists) and its per-neighbour factors
 * in pos.w = p / rho^2 and vel.w = 1 / rho */
void launch_sph_density(const DevParams &p, const unsigned int *cell_start, float4 *pos, float4 *vel, float *dens,
                        float *pres, const NbrLists &nl, cudaStream_t s);
/* acceleration from the lists and .w factors of launch_sph_density */
void launch_sph_force(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const float4 *vel,
                      float4 *acc, const NbrLists &nl, cudaStream_t s);
void launch_sph_integrate(const DevParams &p, const float4 *pos_b, const float4 *vel_b, const float4 *acc,
                          const unsigned int *id_b, const unsigned int *attr_b, float4 *pos_a, float4 *vel_a,
                          unsigned int *id_a, unsigned int *attr_a, cudaStream_t s);

/* ---- neighbour sets under the reference criterion ---- */
void launch_nb_count(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const unsigned int *id,
                     unsigned int *cnt_p, unsigned long long *total, const NbrLists &nl, cudaStream_t s);
void launch_nb_rows(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const unsigned int *id,
                    const unsigned int *offsets, const NbrLists &nl, int *out, float *d2out, cudaStream_t s);

/* ---- deletion regions and the active / parked partition ---- */
/* reg: nreg pairs (lo, hi) of float4 */
void launch_delete_regions(int n, float4 *pos, float4 *vel, unsigned int *attr, const float4 *reg, int nreg,
                           cudaStream_t s);
void launch_mark_active(int n, const unsigned int *attr, unsigned int *keep, cudaStream_t s);
void launch_partition_perm(int n, const unsigned int *scan, unsigned int *perm, cudaStream_t s);
void launch_gather_rows(int n, const unsigned int *perm, const float4 *src, float4 *dst, int k4, cudaStream_t s);

/* ---- density on a lattice (CalImplicitField) ---- */
void launch_density_grid(const DevParams &p, const unsigned int *cell_start, const float4 *pos, const int nn[3],
                         const double minp[3], const double d[3], const double lo[3], const double hi[3], float *out,
                         cudaStream_t s);

/* ---- grid sort as an LSD radix sort of (cell << 32 | slot) keys ---- */
struct RadixBufs {
    unsigned long long *k0 = nullptr, *k1 = nullptr; /* n keys each (ping-pong) */
    unsigned int *hist = nullptr, *offs = nullptr;   /* 256 x tiles (offs: + 1 for the scan's total) */
    unsigned int *bsum = nullptr;                    /* scan_blocks(256 x tiles) */
};
unsigned int radix_tiles(int n);
int radix_passes(unsigned int ncells);
/* perm[d] = the previous slot of the d-th key in (cell, slot) order */
void launch_radix_sort_cells(int n, const unsigned int *cell, unsigned int ncells, const RadixBufs &b,
                             unsigned int *perm, cudaStream_t s);

/* ---- triangle-mesh collision of given segments (parity) ---- */
void launch_polygon_collide(const DevParams &p, int n, const float4 *x0, float4 *x1, float4 *v, cudaStream_t s);

/* ---- the reference's cell hash (rule 0: its CPU grid, 1: its GPU grid) ---- */
void launch_reference_cells(int n, const float4 *pos, int rule, const double org[3], double cw, const int g[3],
                            unsigned int *out, cudaStream_t s);

/* ---- particle order <-> device order ---- */
void launch_unsort4(int n, const unsigned int *id, const float4 *src, float4 *dst, int zero_w, cudaStream_t s);
void launch_unsort1(int n, const unsigned int *id, const unsigned int *src, unsigned int *dst, cudaStream_t s);
void launch_unsort_w(int n, const unsigned int *id, const float4 *src, float *dst, cudaStream_t s);
void launch_iota(int n, unsigned int *dst, cudaStream_t s);
/* rows of k4 float4 per slot: dst[id[d]] = src[d] */
void launch_unsort_rows(int n, const unsigned int *id, const float4 *src, float4 *dst, int k4, cudaStream_t s);
void launch_pack_w(int n, float4 *dst, const float *w, cudaStream_t s);
/* *flag |= 1 when any x/y/z of a (or b, if given) is not finite */
/* *bad = 1 (pinned host memory) when a component of a or b (optional) is not
 * finite; dst_a / dst_b (optional) receive copies */
void launch_check_finite(int n, const float4 *a, const float4 *b, unsigned int *bad, cudaStream_t s,
                         float4 *dst_a = nullptr, float4 *dst_b = nullptr);
/* [p, p + bytes) lies in one allocation of the current device and p is aligned
 * to `align`: a kernel may then read or write the caller's memory itself.
 * Anything else (host or managed memory, another device, a range that leaves
 * its allocation) takes a copy call, which reports what is wrong with it. */
bool device_span(const void *p, size_t bytes, size_t align);

}  // namespace fsph

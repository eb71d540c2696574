/*
 * fsph_loop.cu -- the constraint iterations of a PBF step in one cooperative
 * kernel, in two forms.
 *
 * A scene of up to kLoopMax particles leaves most of the GPU idle in a lambda
 * or correction launch: what an iteration costs is the chain of dependent
 * accesses of each launch (the loop state, the counts, list group after list
 * group and the positions behind each, the block partials and their last
 * block) and the launches themselves.  k_pbf_loop keeps every particle on
 * its own thread for all iterations: its position and lambda stay in
 * registers, its list in shared memory (16-bit slots), so a pass is a few rounds
 * of gathers and a barrier over the grid.  Measured,
 * an iteration of 6,912 particles takes 10.7 us instead of 23.5 (31 before the
 * passes had their form for few warps), of 32,000 13.3 instead of 27.3.
 *
 * From there on a launch of its own still costs each pass about 8 us (launch, a
 * first round of loads with nothing to hide it, the last block's reduction).
 * k_pbf_sweep runs the same passes from the lists in memory, over the slots
 * that fit the GPU's threads at once and then the rest, with a barrier between
 * them.  Measured, an iteration takes, in us, launches / sweep: 69,632
 * particles 29.8 / 21.4, 131,072 35.8 / 24.9, 221,184 46.3 / 35.0, 262,144
 * 55.7 / 49.6, 524,288 88.1 / 78.9, 1,048,576 148.7 / 137.5, 8,192,000 1010 /
 * 998.  What bounds the passes is in fsph_passes.cuh: the L1 wavefronts of the
 * gathers.
 *
 * The pair terms, their order and the order-free error sums are those of
 * k_lambda and k_correction (fsph_passes.cuh): the results are the same bit
 * for bit.
 */
#include <algorithm>
#include <mutex>

#include "fsph_kernels.cuh"
#include "fsph_passes.cuh"

namespace fsph {

namespace {

/* polls before a block gives the barrier up, where the caller sets no limit: about
 * two seconds, and as much again for each 65,536 particles (a co-resident grid needs
 * a few; a scene that has collapsed into one cell may take long over a pass) */
constexpr unsigned long long kLoopPolls = 1ull << 21;

/* The grid barrier in two halves, so that what need not be done before the
 * other blocks go on is done while waiting for them.  Writes of the block
 * before grid_arrive are visible to every block after its grid_wait(want),
 * want = the arrivals since the kernel began.  grid_wait is false, for every
 * thread of the block alike, when `polls` polls did not see them all. */
__device__ __forceinline__ void grid_arrive(LoopCtl *lc) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&lc->arrived, 1u);
    }
}
__device__ __forceinline__ bool grid_wait(LoopCtl *lc, unsigned int want, unsigned long long polls, int &s_ok) {
    if (threadIdx.x == 0) {
        unsigned int seen;
        while (true) {
            /* relaxed, and with a pause: an acquire would empty the SM's L1 at every
             * poll, under the blocks that are still in their pass */
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&lc->arrived) : "memory");
            if ((int)(seen - want) >= 0 || --polls == 0ull) break; /* the counter may wrap */
            __nanosleep(64);
        }
        __threadfence();
        s_ok = (int)(seen - want) >= 0 ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
}

/* One particle's candidates from its list in shared memory (two 16-bit slots a
 * word, word w of a thread at [w * BLOCK]); an overflowed list walks the cells.
 * Blocks of 64 threads are up to two per SM, with registers to spare and no other
 * warp to hide a load: 24 gathers leave together, two rounds for most particles.
 * In larger blocks the next eight are in flight while eight are evaluated.  An
 * iteration of 6,912 particles takes 12.3 us by eights, 11.5 with 16 together, 10.7
 * with 24, 12.3 with 28, 14.0 with 40, its lists of about 33 entries; with 37 (a
 * stirred state) 13.5 by eights, 12.9 with 16, 13.1 with 24, 14.6 with 32, and so in
 * proportion from 1,000 to 19,456 particles.  Past 64 entries the walks of the
 * overflowed lists are what counts (55 us).  32,000 particles (blocks of 128) 13.6
 * by eights and 14.2 with 24. */
constexpr int kTogether = 24;
template <int BLOCK, class Load, class F>
__device__ __forceinline__ void for_each_kept(const DevParams &p, const unsigned int *__restrict__ cell_start,
                                              const unsigned int *kept, int k, int i, float3 xi, Load &&load, F &&f) {
    if (k == (int)kListOverflow) {
        for_each_candidate<1>(p, cell_start, nullptr, nullptr, i, xi, 0, load, f);
        return;
    }
    /* groups past the list's end hold its last entry again or the rest of the
     * last group: real slots, fetched and not used */
    auto fetch = [&](int t0, float4(&xj)[8], unsigned int(&j)[8]) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned int v = kept[min((t0 >> 1) + u, (k - 1) >> 1) * BLOCK];
            j[2 * u] = v & 0xffffu;
            j[2 * u + 1] = v >> 16;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) xj[u] = load(j[u]);
    };
    if (k == 0) return;
    if (BLOCK == 64) {
        for (int t0 = 0; t0 < k; t0 += kTogether) {
            unsigned int v[kTogether / 2];
            float4 xj[kTogether];
#pragma unroll
            for (int u = 0; u < kTogether / 2; ++u) v[u] = kept[min((t0 >> 1) + u, (k - 1) >> 1) * BLOCK];
#pragma unroll
            for (int u = 0; u < kTogether; ++u) xj[u] = load(u & 1 ? v[u / 2] >> 16 : v[u / 2] & 0xffffu);
#pragma unroll
            for (int u = 0; u < kTogether; ++u)
                if (t0 + u < k) f(u & 1 ? v[u / 2] >> 16 : v[u / 2] & 0xffffu, xj[u]);
        }
        return;
    }
    float4 xa[8], xb[8];
    unsigned int ja[8], jb[8];
    fetch(0, xa, ja);
    for (int t0 = 0; t0 < k; t0 += 16) {
        fetch(t0 + 8, xb, jb);
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (t0 + u < k) f(ja[u], xa[u]);
        if (t0 + 8 >= k) break;
        fetch(t0 + 16, xa, ja);
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (t0 + 8 + u < k) f(jb[u], xb[u]);
    }
}

/* One block's state of a launch, the same in every block (thread 0 decides for
 * the block from sums that nobody writes any more). */
struct LoopState {
    unsigned int par, iter, cont, rebuild, at;
    float md;
};
/* the next iteration's sums: last read before the barrier that ended the iteration
 * before, next written after this one's first */
__device__ __forceinline__ void loop_clear(LoopCtl *lc, unsigned int nx) {
    lc->e1[nx] = lc->e2[nx] = 0ull;
    lc->em[nx] = lc->disp[nx] = lc->nan[nx] = lc->grab[nx] = lc->grab2[nx] = 0u;
}
__device__ __forceinline__ void loop_add(LoopCtl *lc, unsigned int at, unsigned long long q1, unsigned long long q2,
                                         float qm, float disp2) {
    atomicAdd(&lc->e1[at], q1);
    atomicAdd(&lc->e2[at], q2);
    atomicMax(&lc->em[at], __float_as_uint(qm)); /* |C| >= 0: the bits order as the values */
    atomicMax(&lc->disp[at], __float_as_uint(disp2));
}
/* continue (cont) and rebuild first (rebuild) after the iteration that s.iter
 * counts up to; true: another iteration follows in this launch */
__device__ __forceinline__ bool loop_decide(const DevParams &p, const LoopCtl *lc, LoopState &s) {
    const unsigned long long e = __ldcg(p.error_mode ? &lc->e2[s.at] : &lc->e1[s.at]);
    s.md = __uint_as_float(__ldcg(&lc->disp[s.at]));
    const unsigned int bad = __ldcg(&lc->nan[s.at]);
    const int it = (int)s.iter + 1, minit = p.min_iter > 1 ? p.min_iter : 1;
    s.cont = it < p.max_iter && !bad;
    if (s.cont && it >= minit) /* the mean in double, as lambda_tail_fix (two slow divisions: only when it decides) */
        s.cont = !((float)((double)e * 0x1p-32 / (double)p.n) <= p.eta);
    s.rebuild = (s.md > p.skin2 || !(s.md == s.md)) ? 1u : 0u;
    return s.cont && !s.rebuild;
}
/* thread 0 of each block, last: the last block out leaves the step's loop state,
 * and the counters for another launch */
__device__ __forceinline__ void loop_leave(const DevParams &p, DevCtl *ctl, LoopCtl *lc, const LoopState &s, bool ok,
                                           cudaGraphConditionalHandle hwhile, cudaGraphConditionalHandle hif,
                                           cudaGraphConditionalHandle hif2, int use_graph) {
    if (!ok) ctl->wait_err = 1u;
    __threadfence();
    if (atomicAdd(&lc->left, 1u) != gridDim.x - 1u) return;
    __threadfence();
    ctl->err1 = (float)((double)__ldcg(&lc->e1[s.at]) * 0x1p-32 / (double)p.n);
    ctl->err2 = (float)((double)__ldcg(&lc->e2[s.at]) * 0x1p-32 / (double)p.n);
    ctl->errmax = __uint_as_float(__ldcg(&lc->em[s.at]));
    ctl->iter = s.iter;
    ctl->done = s.cont ? 0u : 1u;
    ctl->disp2_bits = __float_as_uint(s.md);
    ctl->rebuild = s.rebuild;
    ctl->parity = s.par;
    ctl->loops += 1u;
    lc->arrived = 0u;
    lc->left = 0u;
    for (unsigned int k = 0; k < 3u; ++k) loop_clear(lc, k);
    const unsigned int cont = __ldcg(&ctl->wait_err) ? 0u : s.cont; /* a wait ran out: the step ends and reports it */
    /* a correction that was not a number also asks for a rebuild: the launch after
     * it stops at its first errors, as k_lambda does */
    if (cont && __ldcg(&ctl->nan_flag)) lc->nan[0] = 1u;
    if (use_graph & 1) {
        cudaGraphSetConditional(hwhile, cont);
        cudaGraphSetConditional(hif, cont & s.rebuild);
        if (use_graph & 2) cudaGraphSetConditional(hif2, s.rebuild);
    }
}

template <bool KAHAN, int BLOCK>
__global__ void __launch_bounds__(BLOCK, BLOCK == 64 ? 4 : 512 / BLOCK)
    k_pbf_loop(DevParams p, const unsigned int *__restrict__ cell_start, float4 *ppos0, float4 *ppos1,
               float *__restrict__ dens, const float4 *__restrict__ xb, DevCtl *ctl, LoopCtl *lc,
               cudaGraphConditionalHandle hwhile, cudaGraphConditionalHandle hif, cudaGraphConditionalHandle hif2,
               int use_graph, unsigned long long polls, const ListEntry *__restrict__ list,
               const unsigned char *__restrict__ cnt) {
    __shared__ unsigned int s_kept[(kListMax / 2) * BLOCK];
    __shared__ unsigned long long s_e1[BLOCK / 32], s_e2[BLOCK / 32];
    __shared__ float s_em[BLOCK / 32], s_d[BLOCK / 32];
    __shared__ int s_ok, s_go;
    const int i = blockIdx.x * BLOCK + (int)threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool valid = i < p.n;
    LoopState st{*((volatile unsigned int *)&ctl->parity), *((volatile unsigned int *)&ctl->iter), 1u, 0u, 0u, 0.f};
    unsigned int *kept = s_kept + threadIdx.x;
    float3 xi = make_float3(0.f, 0.f, 0.f), xbi = xi;
    int k = 0;
    if (valid) {
        k = (int)cnt[i];
        xi = f3((st.par ? ppos1 : ppos0)[i]);
        xbi = f3(xb[i]);
        if (k != (int)kListOverflow) {
            const uint4 *lg = reinterpret_cast<const uint4 *>(list) + i;
            for (int g = 0; 4 * g < k; ++g) {
                const uint4 e = __ldg(lg + (size_t)g * (size_t)p.n);
                const unsigned int n = (unsigned int)p.n;
                const unsigned int a = bounded(p, e.x, n, kBoundSlot), b = bounded(p, e.y, n, kBoundSlot),
                                   c = bounded(p, e.z, n, kBoundSlot), d = bounded(p, e.w, n, kBoundSlot);
                kept[(2 * g) * BLOCK] = a | b << 16;
                kept[(2 * g + 1) * BLOCK] = c | d << 16;
            }
        }
    }
    const unsigned int nb = gridDim.x;
    unsigned int want = 0u;
    float rho = 0.f;
    bool ok = true;
    while (true) {
        float4 *pp = st.par ? ppos1 : ppos0, *dst = st.par ? ppos0 : ppos1;
        const unsigned int at = st.at, nx = at == 2u ? 0u : at + 1u;
        if (blockIdx.x == 0 && threadIdx.x == 0) loop_clear(lc, nx);
        /* lambda of every particle, its error terms */
        float li = 0.f;
        unsigned long long q1 = 0ull, q2 = 0ull;
        float qm = 0.f;
        if (valid) {
            const float C = lambda_terms<1, KAHAN>(
                p, pp, xi,
                [&](auto &&load, auto &&f) { for_each_kept<BLOCK>(p, cell_start, kept, k, i, xi, load, f); }, rho, li);
            reinterpret_cast<float *>(pp + i)[3] = li;
            if (!(rho == rho)) {
                ctl->nan_flag = 1u;
                lc->nan[at] = 1u;
            }
            q1 = err_fix(C > 0.0f ? C : 0.0f);
            q2 = err_fix(fabsf(C));
            qm = fmaxf(qm, fabsf(C)); /* a C that is not a number is left out, as in k_lambda */
        }
        grid_arrive(lc);
        /* the error sums are needed only by the barrier after the corrections */
        q1 = warp_sum_u64(q1);
        q2 = warp_sum_u64(q2);
        qm = warp_max(qm);
        if (lane == 0) { s_e1[warp] = q1; s_e2[warp] = q2; s_em[warp] = qm; }
        want += nb;
        if (!(ok = grid_wait(lc, want, polls, s_ok))) break;
        /* corrections from every particle's lambda */
        float disp2 = 0.f;
        if (valid) {
            const float3 dp = correction_terms<1>(p, pp, xi, li, [&](auto &&load, auto &&f) {
                for_each_kept<BLOCK>(p, cell_start, kept, k, i, xi, load, f);
            });
            const float3 xn = solid_project(xi + dp, p);
            dst[i] = make_float4(xn.x, xn.y, xn.z, 0.0f);
            if (!(xn.x == xn.x && xn.y == xn.y && xn.z == xn.z)) {
                ctl->nan_flag = 1u;
                lc->nan[nx] = 1u; /* stops the loop at the next errors, as k_lambda does */
            }
            const float3 dd = xn - xbi;
            disp2 = fmaxf(disp2, dot3(dd, dd));
            xi = xn;
        }
        disp2 = warp_max(disp2);
        if (lane == 0) s_d[warp] = disp2;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < BLOCK / 32; ++w) {
                q1 += s_e1[w];
                q2 += s_e2[w];
                qm = fmaxf(qm, s_em[w]);
                disp2 = fmaxf(disp2, s_d[w]);
            }
            loop_add(lc, at, q1, q2, qm, disp2);
        }
        grid_arrive(lc);
        want += nb;
        if (!(ok = grid_wait(lc, want, polls, s_ok))) break;
        if (threadIdx.x == 0) s_go = loop_decide(p, lc, st);
        __syncthreads();
        ++st.iter;
        st.par ^= 1u;
        if (!s_go) break;
        st.at = nx;
    }
    if (valid) dens[i] = rho;
    if (threadIdx.x == 0) loop_leave(p, ctl, lc, st, ok, hwhile, hif, hif2, use_graph);
}

/* The same loop from the lists in memory, for scenes that do not fit k_pbf_loop:
 * two blocks per SM of as many warps as there are chunks of 32 slots for, at most
 * 24 (40 registers a thread).  A warp takes whole rounds in turn and the last two
 * on demand, as k_lambda does.  Two large blocks, because each block's arrival and
 * polls cost the barrier: an iteration at 1,048,576 particles took 150.4 us in
 * blocks of 256, 142.4 of 512 and 138.2 of 768 (137.3 with the pause between
 * polls), and with the same 768 threads at 131,072 particles, where 171 blocks
 * leave the SMs uneven, 33.9 instead of 24.9. */
constexpr int kSweepBlock = 768;
template <bool KAHAN>
__global__ void __launch_bounds__(kSweepBlock, 2)
    k_pbf_sweep(DevParams p, const unsigned int *__restrict__ cell_start, float4 *ppos0, float4 *ppos1,
                float *__restrict__ dens, const float4 *__restrict__ xb, DevCtl *ctl, LoopCtl *lc,
                cudaGraphConditionalHandle hwhile, cudaGraphConditionalHandle hif, cudaGraphConditionalHandle hif2,
                int use_graph, unsigned long long polls, const ListEntry *__restrict__ list,
                const unsigned char *__restrict__ cnt) {
    __shared__ unsigned long long s_e1[kSweepBlock / 32], s_e2[kSweepBlock / 32];
    __shared__ float s_em[kSweepBlock / 32], s_d[kSweepBlock / 32];
    __shared__ int s_ok, s_go;
    __shared__ LoopState st;
    const int lane = threadIdx.x & 31, nchunks = (p.n + 31) >> 5;
    const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), nw = (int)((gridDim.x * blockDim.x) >> 5);
    const int stat = max(nchunks / nw - 1, 1) * nw;
    if (threadIdx.x == 0)
        st = LoopState{*((volatile unsigned int *)&ctl->parity), *((volatile unsigned int *)&ctl->iter), 1u, 0u, 0u, 0.f};
    __syncthreads();
    unsigned int want = 0u;
    bool ok = true;
    while (true) {
        {
            float4 *pp = st.par ? ppos1 : ppos0;
            const unsigned int at = st.at;
            if (blockIdx.x == 0 && threadIdx.x == 0) loop_clear(lc, at == 2u ? 0u : at + 1u);
            unsigned long long q1 = 0ull, q2 = 0ull;
            float qm = 0.f;
            for (int c = warp; c < nchunks;
                 c = stat >= nchunks ? nchunks : next_chunk(c, nw, stat, &lc->grab[at], lane)) {
                const int i = c * 32 + lane;
                if (i < p.n) {
                    const float3 xi = f3(pp[i]);
                    float rho, li;
                    const float C = lambda_terms<1, KAHAN>(
                        p, pp, xi,
                        [&](auto &&load, auto &&f) {
                            for_each_candidate<1>(p, cell_start, list, cnt, i, xi, 0, load, f);
                        },
                        rho, li);
                    reinterpret_cast<float *>(pp + i)[3] = li;
                    dens[i] = rho;
                    if (!(rho == rho)) {
                        ctl->nan_flag = 1u;
                        lc->nan[at] = 1u;
                    }
                    q1 += err_fix(C > 0.0f ? C : 0.0f);
                    q2 += err_fix(fabsf(C));
                    qm = fmaxf(qm, fabsf(C));
                }
            }
            q1 = warp_sum_u64(q1);
            q2 = warp_sum_u64(q2);
            qm = warp_max(qm);
            if (lane == 0) { s_e1[threadIdx.x >> 5] = q1; s_e2[threadIdx.x >> 5] = q2; s_em[threadIdx.x >> 5] = qm; }
        }
        grid_arrive(lc);
        want += gridDim.x;
        if (!(ok = grid_wait(lc, want, polls, s_ok))) break;
        {
            const float4 *src = st.par ? ppos1 : ppos0;
            float4 *dst = st.par ? ppos0 : ppos1;
            const unsigned int at = st.at;
            float disp2 = 0.f;
            for (int c = warp; c < nchunks;
                 c = stat >= nchunks ? nchunks : next_chunk(c, nw, stat, &lc->grab2[at], lane)) {
                const int i = c * 32 + lane;
                if (i < p.n) {
                    const float4 xi4 = src[i];
                    const float3 xi = f3(xi4);
                    const float3 dp = correction_terms<1>(p, src, xi, xi4.w, [&](auto &&load, auto &&f) {
                        for_each_candidate<1>(p, cell_start, list, cnt, i, xi, 0, load, f);
                    });
                    const float3 xn = solid_project(xi + dp, p);
                    dst[i] = make_float4(xn.x, xn.y, xn.z, 0.0f);
                    if (!(xn.x == xn.x && xn.y == xn.y && xn.z == xn.z)) {
                        ctl->nan_flag = 1u;
                        lc->nan[at == 2u ? 0u : at + 1u] = 1u; /* stops the loop at the next errors, as k_lambda does */
                    }
                    const float3 dd = xn - f3(xb[i]);
                    disp2 = fmaxf(disp2, dot3(dd, dd));
                }
            }
            disp2 = warp_max(disp2);
            if (lane == 0) s_d[threadIdx.x >> 5] = disp2;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long q1 = 0ull, q2 = 0ull;
            float qm = 0.f, disp2 = 0.f;
            for (unsigned int w = 0; w < blockDim.x >> 5; ++w) {
                q1 += s_e1[w];
                q2 += s_e2[w];
                qm = fmaxf(qm, s_em[w]);
                disp2 = fmaxf(disp2, s_d[w]);
            }
            loop_add(lc, st.at, q1, q2, qm, disp2);
        }
        grid_arrive(lc);
        want += gridDim.x;
        if (!(ok = grid_wait(lc, want, polls, s_ok))) break;
        if (threadIdx.x == 0) {
            s_go = loop_decide(p, lc, st);
            ++st.iter;
            st.par ^= 1u;
            if (s_go) st.at = st.at == 2u ? 0u : st.at + 1u;
        }
        __syncthreads();
        if (!s_go) break;
    }
    if (threadIdx.x == 0) loop_leave(p, ctl, lc, st, ok, hwhile, hif, hif2, use_graph);
}

typedef void (*LoopKernel)(DevParams, const unsigned int *, float4 *, float4 *, float *, const float4 *, DevCtl *,
                           LoopCtl *, cudaGraphConditionalHandle, cudaGraphConditionalHandle,
                           cudaGraphConditionalHandle, int, unsigned long long, const ListEntry *,
                           const unsigned char *);

template <int BLOCK>
LoopKernel loop_kernel(bool kahan) {
    return kahan ? k_pbf_loop<true, BLOCK> : k_pbf_loop<false, BLOCK>;
}

struct LoopShape {
    LoopKernel kernel;
    int block;
};
/* a block of 64 threads up to two per SM, then 128 and 256: the barrier's cost
 * is its arrivals, the passes' the warps that share an SM */
LoopShape loop_shape(const DevParams &p, int sms) {
    const bool kahan = p.compensated != 0;
    if (p.n <= 2 * sms * 64) return LoopShape{loop_kernel<64>(kahan), 64};
    if (p.n <= 2 * sms * 128) return LoopShape{loop_kernel<128>(kahan), 128};
    if (p.n <= kLoopMax) return LoopShape{loop_kernel<256>(kahan), 256};
    /* two blocks per SM, as many warps in each as there are chunks for */
    const int warps = blocks_for(p.n, 2 * sms * 32);
    return LoopShape{kahan ? k_pbf_sweep<true> : k_pbf_sweep<false>, std::min(32 * warps, kSweepBlock)};
}

}  // namespace

/* the launch's blocks, every one resident at once; 0: it cannot be launched so */
static unsigned int loop_blocks(const DevParams &p, LoopShape &sh) {
    int dev = 0, sms = 0, coop = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
        return 0u;
    sh = loop_shape(p, sms);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void *)sh.kernel, sh.block, 0) != cudaSuccess)
        return 0u;
    const unsigned int all = blocks_for(p.n, sh.block), room = (unsigned int)(per * sms);
    if (p.n > kLoopMax) return std::min(all, std::min(room, 2u * (unsigned int)sms));
    return all <= room ? all : 0u;
}

bool loop_fits(const DevParams &p) {
    LoopShape sh;
    return p.n > 0 && p.use_lists && !p.nb && loop_blocks(p, sh) > 0u;
}

cudaError_t launch_pbf_loop(const DevParams &p, const unsigned int *cell_start, float4 *ppos0, float4 *ppos1,
                            float *dens, const float4 *xb, DevCtl *ctl, LoopCtl *lc, unsigned long long while_handle,
                            unsigned long long if_handle, unsigned long long if_handle2, int use_graph,
                            unsigned long long polls, const NbrLists &nl, cudaStream_t s) {
    LoopShape sh;
    const unsigned int blocks = loop_blocks(p, sh);
    if (!blocks) return cudaErrorCooperativeLaunchTooLarge;
    DevParams q = p;
    cudaGraphConditionalHandle hw = while_handle, h1 = if_handle, h2 = if_handle2;
    const ListEntry *list = nl.list;
    const unsigned char *cnt = nl.cnt;
    if (!polls) polls = kLoopPolls * (1ull + ((unsigned int)p.n >> 16));
    void *args[] = {&q, &cell_start, &ppos0, &ppos1, &dens, &xb, &ctl, &lc, &hw, &h1, &h2, &use_graph, &polls,
                    &list, &cnt};
    return cudaLaunchCooperativeKernel((const void *)sh.kernel, dim3(blocks), dim3(sh.block), args, 0, s);
}

}  // namespace fsph

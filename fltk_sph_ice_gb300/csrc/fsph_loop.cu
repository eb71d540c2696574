/*
 * fsph_loop.cu -- the constraint iterations of a small PBF scene in one
 * cooperative kernel.
 *
 * A scene of up to kLoopMax particles leaves most of the GPU idle in a lambda
 * or correction launch: what an iteration costs is the chain of dependent
 * accesses of each launch (the loop state, the counts, list group after list
 * group and the positions behind each, the block partials and their last
 * block) and the launches themselves.  Here one launch keeps every particle on
 * its own thread for all iterations: its position and lambda stay in
 * registers, its list in shared memory (16-bit slots), so a pass is one round
 * of gathers, up to sixteen in flight, and a barrier over the grid.  Measured,
 * an iteration of 6,912 particles takes 12 us instead of 23.5 (31 before the
 * passes had their form for few warps), of 32,000 13.5 instead of 27.3; the
 * whole step of 6,912 (10 iterations, results read back) 360 -> 272 us.
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

/* polls before a block gives the barrier up (about a second; a co-resident
 * grid needs a few) */
constexpr unsigned int kLoopPolls = 1u << 21;

/* The grid barrier in two halves, so that what need not be done before the
 * other blocks go on is done while waiting for them.  Writes of the block
 * before grid_arrive are visible to every block after its grid_wait(want),
 * want = the arrivals since the kernel began.  grid_wait is false, for every
 * thread of the block alike, when the wait ran out. */
__device__ __forceinline__ void grid_arrive(LoopCtl *lc) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&lc->arrived, 1u);
    }
}
__device__ __forceinline__ bool grid_wait(LoopCtl *lc, unsigned int want, int &s_ok) {
    if (threadIdx.x == 0) {
        unsigned int seen = 0u, polls = 0u;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&lc->arrived) : "memory");
        } while (seen < want && ++polls < kLoopPolls);
        __threadfence();
        s_ok = seen >= want ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
}

/* One particle's candidates from its list in shared memory (two 16-bit slots a
 * word, word w of a thread at [w * BLOCK]), the next eight gathers in flight while
 * eight are evaluated; an overflowed list walks the cells. */
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

template <bool KAHAN, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 512 / BLOCK)
    k_pbf_loop(DevParams p, const unsigned int *__restrict__ cell_start, float4 *ppos0, float4 *ppos1,
               float *__restrict__ dens, const float4 *__restrict__ xb, DevCtl *ctl, LoopCtl *lc,
               cudaGraphConditionalHandle hwhile, cudaGraphConditionalHandle hif, cudaGraphConditionalHandle hif2,
               int post, const ListEntry *__restrict__ list, const unsigned char *__restrict__ cnt) {
    __shared__ unsigned int s_kept[(kListMax / 2) * BLOCK];
    __shared__ unsigned long long s_e1[BLOCK / 32], s_e2[BLOCK / 32];
    __shared__ float s_em[BLOCK / 32], s_d[BLOCK / 32];
    __shared__ int s_ok, s_go;
    const int i = blockIdx.x * BLOCK + (int)threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool valid = i < p.n;
    unsigned int par = *((volatile unsigned int *)&ctl->parity), iter = *((volatile unsigned int *)&ctl->iter);
    unsigned int *kept = s_kept + threadIdx.x;
    float3 xi = make_float3(0.f, 0.f, 0.f), xbi = xi;
    int k = 0;
    if (valid) {
        k = (int)cnt[i];
        xi = f3((par ? ppos1 : ppos0)[i]);
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
    unsigned int want = 0u, cont = 1u, rebuild = 0u, at = 0u;
    float md = 0.f, rho = 0.f;
    bool ok = true;
    while (true) {
        float4 *pp = par ? ppos1 : ppos0, *dst = par ? ppos0 : ppos1;
        const unsigned int nx = at == 2u ? 0u : at + 1u;
        /* lambda of every particle, its error terms */
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            /* the next iteration's sums: last read before the barrier that ended the
             * iteration before, next written after this one's first */
            lc->e1[nx] = lc->e2[nx] = 0ull;
            lc->em[nx] = lc->disp[nx] = lc->nan[nx] = 0u;
        }
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
            qm = fabsf(C);
        }
        grid_arrive(lc);
        /* the error sums are needed only by the barrier after the corrections */
        q1 = warp_sum_u64(q1);
        q2 = warp_sum_u64(q2);
        qm = warp_max(qm);
        if (lane == 0) { s_e1[warp] = q1; s_e2[warp] = q2; s_em[warp] = qm; }
        want += nb;
        if (!(ok = grid_wait(lc, want, s_ok))) break;
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
            disp2 = dot3(dd, dd);
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
            atomicAdd(&lc->e1[at], q1);
            atomicAdd(&lc->e2[at], q2);
            atomicMax(&lc->em[at], __float_as_uint(qm)); /* |C| >= 0: the bits order as the values */
            atomicMax(&lc->disp[at], __float_as_uint(disp2));
        }
        grid_arrive(lc);
        want += nb;
        if (!(ok = grid_wait(lc, want, s_ok))) break;
        /* the loop's decisions, from the same numbers in every block (the sums and
         * flags of this iteration, which nobody writes any more) */
        if (threadIdx.x == 0) {
            const unsigned long long e = __ldcg(p.error_mode ? &lc->e2[at] : &lc->e1[at]);
            md = __uint_as_float(__ldcg(&lc->disp[at]));
            const unsigned int bad = __ldcg(&lc->nan[at]);
            const int it = (int)iter + 1, minit = p.min_iter > 1 ? p.min_iter : 1;
            cont = it < p.max_iter && !bad;
            if (cont && it >= minit) /* the mean in double, as lambda_tail_fix (two slow divisions: only when it decides) */
                cont = !((float)((double)e * 0x1p-32 / (double)p.n) <= p.eta);
            rebuild = (md > p.skin2 || !(md == md)) ? 1u : 0u;
            s_go = cont && !rebuild;
        }
        __syncthreads();
        ++iter;
        par ^= 1u;
        if (!s_go) break;
        at = nx;
    }
    if (valid) dens[i] = rho;
    if (threadIdx.x != 0) return;
    if (!ok) ctl->wait_err = 1u;
    __threadfence();
    if (atomicAdd(&lc->left, 1u) != nb - 1u) return;
    /* the last block out: the step's loop state, and the counters for another launch */
    __threadfence();
    ctl->err1 = (float)((double)__ldcg(&lc->e1[at]) * 0x1p-32 / (double)p.n);
    ctl->err2 = (float)((double)__ldcg(&lc->e2[at]) * 0x1p-32 / (double)p.n);
    ctl->errmax = __uint_as_float(__ldcg(&lc->em[at]));
    ctl->iter = iter;
    ctl->done = cont ? 0u : 1u;
    ctl->disp2_bits = __float_as_uint(md);
    ctl->rebuild = rebuild;
    ctl->parity = par;
    ctl->loops += 1u;
    lc->arrived = 0u;
    lc->left = 0u;
    for (int s = 0; s < 3; ++s) {
        lc->e1[s] = lc->e2[s] = 0ull;
        lc->em[s] = lc->disp[s] = lc->nan[s] = 0u;
    }
    if (__ldcg(&ctl->wait_err)) cont = 0u; /* a wait ran out: the step ends and reports it */
    cudaGraphSetConditional(hwhile, cont);
    cudaGraphSetConditional(hif, cont & rebuild);
    if (post) cudaGraphSetConditional(hif2, rebuild);
}

typedef void (*LoopKernel)(DevParams, const unsigned int *, float4 *, float4 *, float *, const float4 *, DevCtl *,
                           LoopCtl *, cudaGraphConditionalHandle, cudaGraphConditionalHandle,
                           cudaGraphConditionalHandle, int, const ListEntry *, const unsigned char *);

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
    return LoopShape{loop_kernel<256>(kahan), 256};
}

}  // namespace

bool loop_fits(const DevParams &p) {
    if (p.n <= 0 || p.n > kLoopMax || !p.use_lists || p.nb) return false;
    int dev = 0, sms = 0, coop = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
        return false;
    const LoopShape sh = loop_shape(p, sms);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void *)sh.kernel, sh.block, 0) != cudaSuccess)
        return false;
    return (long long)per * sms * sh.block >= (long long)p.n; /* every block resident at once */
}

cudaError_t launch_pbf_loop(const DevParams &p, const unsigned int *cell_start, float4 *ppos0, float4 *ppos1,
                            float *dens, const float4 *xb, DevCtl *ctl, LoopCtl *lc, unsigned long long while_handle,
                            unsigned long long if_handle, unsigned long long if_handle2, int post, const NbrLists &nl,
                            cudaStream_t s) {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const LoopShape sh = loop_shape(p, sms);
    DevParams q = p;
    cudaGraphConditionalHandle hw = while_handle, h1 = if_handle, h2 = if_handle2;
    const ListEntry *list = nl.list;
    const unsigned char *cnt = nl.cnt;
    void *args[] = {&q, &cell_start, &ppos0, &ppos1, &dens, &xb, &ctl, &lc, &hw, &h1, &h2, &post, &list, &cnt};
    return cudaLaunchCooperativeKernel((const void *)sh.kernel, dim3(blocks_for(p.n, sh.block)), dim3(sh.block), args,
                                       0, s);
}

}  // namespace fsph

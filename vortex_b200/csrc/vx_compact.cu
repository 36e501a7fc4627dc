// vx_compact.cu — removal of vortices with |G| < drop_eps, reproducing the
// reference's serial swap-with-last permutation exactly, in parallel.
//
// Reference: sort_Kernel src/kernel.cu:1159-1178 (one thread walks i upward
// and swaps every dead element with the current last one).  Closed form of
// its result, with m = number of live elements among [0, n0), scan[p] = live
// elements before p, H = dead elements below m (= live elements at or above m):
//  * live elements below m stay;
//  * the t-th dead position below m (ascending) receives the live element
//    that is t-th from the top among positions >= m;
//  * each tail position e in [m, n0) gets G = 0 and the position of
//      - the hole it was swapped with, when e is the first slot of its run
//        (e = n0-1, or e+1 holds a live element); the hole of the run with
//        k live elements above e is the k-th hole, or m itself once all
//        holes are filled,
//      - otherwise the element that was at e+1.
// Everything outside [0, n0) is untouched.
//
// The dead ones are marked in a bitmap, from which one block finds all places
// (vx_cmp_block).  Where few are dead, as after a step's convection, that
// block makes the moves too, and the two launches after it (gather into
// scratch, scatter back) return at once.
#include "vx_compact.cuh"

constexpr int CMP_T = 1024;
// Most dead vortices the marking kernel's last block removes by itself.
constexpr long long CMP_FEW = 8192;

// Marks the dead; the block that finishes last goes on (vx_cmp_block).  A
// warp takes whole words of the bitmap, four at a time, and writes those that
// are not zero (the bitmap is zero between compactions).  Bound: the read of
// the strengths, and the last block's latency.  count_step: this compaction
// closes a whole step, which it counts (no kernel after it in the step reads
// the step index).
// With the two launches after it, each timed by itself: 23 / 33 / 46 us at
// 2e4 / 1e6 / 3e6 vortices; as counts, classification, gather and scatter
// over all of them 32 / 39 / 50.
VX_DEVK void k_cmp_mark_body(VxBlkB<CMP_T, 0> vb, const VxView &v, VxScalars *S, double eps, const VxCompact &c,
                             int count_step) {
    constexpr int U = 4;
    const long long n0 = S->n;
    const int lane = threadIdx.x & 31;
    for (long long base = (vb.x * (long long)CMP_T + (threadIdx.x & ~31)) * U; base < n0;
         base += (long long)vb.n * CMP_T * U) {
        bool dead[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long p = base + u * 32 + lane;
            dead[u] = p < n0 && !vx_live(v, p, eps);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned w = __ballot_sync(0xffffffffu, dead[u]);
            if (w != 0 && lane == 0) c.bits[(base >> 5) + u] = w;
        }
    }
    if (!vx_last_block(&S->sync_ctr, vb.n)) return;
    if (threadIdx.x == 0) {
        if (count_step) S->step += 1;
        S->c_n0 = S->c_m = n0;   // nothing left for the next two launches
        S->c_H = 0;
    }
    __syncthreads();
    vx_cmp_block<CMP_T>(v, S, c, n0, CMP_FEW, true, nullptr, nullptr);
}
__global__ void __launch_bounds__(CMP_T) k_cmp_mark(VxView v, VxScalars *S, double eps, VxCompact c, int count_step) {
    VX_PDL_WAIT();
    k_cmp_mark_body(VxBlkB<CMP_T, 0>{blockIdx.x, gridDim.x}, v, S, eps, c, count_step);
}

VX_DEVK void k_cmp_gather_body(VxBlkB<0, 0> vb, const VxView &v, const VxScalars *S, const VxCompact &c) {
    const long long n0 = S->c_n0, m = S->c_m, H = S->c_H;
    if (m == n0) return;
    vx_cmp_gather<1>(v, c, H, H + n0 - m, vb.x * (long long)blockDim.x + threadIdx.x, (long long)vb.n * blockDim.x);
}
__global__ void k_cmp_gather(VxView v, const VxScalars *S, VxCompact c) {
    VX_PDL_WAIT();
    k_cmp_gather_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, v, S, c);
}

VX_DEVK void k_cmp_scatter_body(VxBlkB<0, 0> vb, const VxView &v, VxScalars *S, const VxCompact &c) {
    const long long n0 = S->c_n0, m = S->c_m, H = S->c_H;
    if (m == n0) return;
    vx_cmp_scatter<1>(v, c, m, H, H + n0 - m, vb.x * (long long)blockDim.x + threadIdx.x,
                      (long long)vb.n * blockDim.x, nullptr, nullptr);
    if (vb.x == 0 && threadIdx.x == 0) S->n = m;
}
__global__ void k_cmp_scatter(VxView v, VxScalars *S, VxCompact c) {
    VX_PDL_WAIT();
    k_cmp_scatter_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, v, S, c);
}

cudaError_t vx_launch_compact(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S,
                              VxWork &w, bool count_step) {
    vx_launch<k_cmp_mark, k_cmp_mark_body>(L, L.num_sms * 2, CMP_T, 0, v, S, p.drop_eps, w.cmp, count_step ? 1 : 0);
    vx_launch<k_cmp_gather, k_cmp_gather_body>(L, L.num_sms * 4, VX_THREADS, 0, v, S, w.cmp);
    vx_launch<k_cmp_scatter, k_cmp_scatter_body>(L, L.num_sms * 4, VX_THREADS, 0, v, S, w.cmp);
    return cudaGetLastError();
}

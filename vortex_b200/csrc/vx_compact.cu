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
// block makes the moves too; else the three launches after it (lists, gather
// into scratch, scatter back) do, which return at once otherwise.
#include "vx_compact.cuh"

constexpr int CMP_T = 1024;

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
        S->cmp_many = 0;
    }
    __syncthreads();
    vx_cmp_block<CMP_T>(v, S, c, n0, VX_CMP_FEW, true, nullptr, nullptr);
}
__global__ void __launch_bounds__(CMP_T) k_cmp_mark(VxView v, VxScalars *S, double eps, VxCompact c, int count_step) {
    VX_PDL_WAIT();
    k_cmp_mark_body(VxBlkB<CMP_T, 0>{blockIdx.x, gridDim.x}, v, S, eps, c, count_step);
}

// Lists of the holes, of what fills them and of the tail's sources, a warp to
// 128 vortices; then the moves.  All bits stay until the last launch.
VX_DEVK void k_cmp_list_body(VxBlkB<0, 0> vb, VxScalars *S, const VxCompact &c) {
    if (!S->cmp_many) return;
    const long long n0 = S->c_n0, m = S->c_m, n4 = (n0 + 127) / 128, m4 = m >> 7;
    const int lane = threadIdx.x & 31;
    int below = c.pre[m4];   // dead below m: the holes
    for (int u = 0; u < 4; ++u) {
        const long long w = m4 * 4 + u;
        if (w * 32 + 32 <= m) below += __popc(c.bits[w]);
        else if (w * 32 < m) below += __popc(c.bits[w] & ((1u << (m & 31)) - 1u));
    }
    const int H = below;
    if (vb.x == 0 && threadIdx.x == 0) S->c_H = H;
    for (long long q = (vb.x * (long long)blockDim.x + threadIdx.x) >> 5; q < n4; q += ((long long)vb.n * blockDim.x) >> 5) {
        int before = c.pre[q];   // dead before the word
        for (int u = 0; u < 4; ++u) {
            const long long w = q * 4 + u, p = w * 32 + lane;
            const unsigned dead = c.bits[w], next = c.bits[w + 1];
            const int k = before + __popc(dead & ((1u << lane) - 1u));
            const bool dd = dead >> lane & 1;
            if (p < m) {
                if (dd) c.hole_pos[k] = (int)p;
            } else if (p < n0) {
                const int r = (int)(p - m) - (k - H);   // live ones in [m, p)
                if (!dd) c.hole_src[H - 1 - r] = (int)p;
                const bool next_live = p + 1 < n0 && !((lane < 31 ? dead >> (lane + 1) : next) & 1u);
                const int grp = H - r - (dd ? 0 : 1);   // live ones in (p, n0)
                c.tail_src[p - m] = p == n0 - 1 || next_live ? (grp < H ? -(grp + 1) : (int)m) : (int)(p + 1);
            }
            before += __popc(dead);
        }
    }
}
__global__ void k_cmp_list(VxScalars *S, VxCompact c) {
    VX_PDL_WAIT();
    k_cmp_list_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, S, c);
}

VX_DEVK void k_cmp_gather_body(VxBlkB<0, 0> vb, const VxView &v, const VxScalars *S, const VxCompact &c) {
    if (!S->cmp_many) return;
    const long long n0 = S->c_n0, m = S->c_m, H = S->c_H;
    vx_cmp_gather<1>(v, c, H, H + n0 - m, vb.x * (long long)blockDim.x + threadIdx.x, (long long)vb.n * blockDim.x);
}
__global__ void k_cmp_gather(VxView v, const VxScalars *S, VxCompact c) {
    VX_PDL_WAIT();
    k_cmp_gather_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, v, S, c);
}

VX_DEVK void k_cmp_scatter_body(VxBlkB<0, 0> vb, const VxView &v, VxScalars *S, const VxCompact &c, const int *slot,
                                long long *rec_i) {
    if (!S->cmp_many) return;
    const long long n0 = S->c_n0, m = S->c_m, H = S->c_H;
    const long long first = vb.x * (long long)blockDim.x + threadIdx.x, stride = (long long)vb.n * blockDim.x;
    vx_cmp_scatter<1>(v, c, m, H, H + n0 - m, first, stride, slot, rec_i);
    for (long long w = first; w < (n0 + 31) / 32; w += stride) c.bits[w] = 0;
    if (first == 0) S->n = m;
}
__global__ void k_cmp_scatter(VxView v, VxScalars *S, VxCompact c, const int *slot, long long *rec_i) {
    VX_PDL_WAIT();
    k_cmp_scatter_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, v, S, c, slot, rec_i);
}

// The moves of a compaction that found more dead than one block should make.
cudaError_t vx_launch_moves(const VxLaunch &L, const VxView &v, VxScalars *S, VxWork &w, const int *slot,
                            long long *rec_i) {
    vx_launch<k_cmp_list, k_cmp_list_body>(L, L.num_sms * 4, VX_THREADS, 0, S, w.cmp);
    vx_launch<k_cmp_gather, k_cmp_gather_body>(L, L.num_sms * 4, VX_THREADS, 0, v, S, w.cmp);
    vx_launch<k_cmp_scatter, k_cmp_scatter_body>(L, L.num_sms * 4, VX_THREADS, 0, v, S, w.cmp, slot, rec_i);
    return cudaGetLastError();
}

cudaError_t vx_launch_compact(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S,
                              VxWork &w, bool count_step) {
    vx_launch<k_cmp_mark, k_cmp_mark_body>(L, L.num_sms * 2, CMP_T, 0, v, S, p.drop_eps, w.cmp, count_step ? 1 : 0);
    return vx_launch_moves(L, v, S, w, nullptr, nullptr);
}

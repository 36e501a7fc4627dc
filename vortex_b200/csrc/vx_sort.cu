// vx_sort.cu — the stable bucket order of the particle grids (cells of the
// diffusion grid, leaves of the quadtree): particle indices arranged by
// bucket, each bucket's particles in index order, from per-bucket counts and
// their exclusive scan (which the grids compute anyway), without a radix sort.
// Equal keys keep their input order, so sorting particle indices by cell gives
// a deterministic order inside every cell.
#include <climits>
#include <vector>

#include "vx_internal.cuh"

// Stable order by bucket, for keys whose buckets have starts (an exclusive
// scan of their counts) and whose elements have ranks (what counting them
// returned, in no fixed order): every element takes the slot of its rank, and
// a copy of what the grids keep per slot with it; then each slot's element
// counts those of its bucket with a lower index and moves to that place, the
// one a stable sort by bucket gives.
//
// Bound: the scattered writes of the first launch (its reads are in element
// order), so a slot's element, bucket and copy are one record, a whole DRAM
// sector (three arrays: twice the time at 3e6 vortices); then the latency of
// a few dependent reads, neighbouring threads reading the same bucket.
// Gathering each slot's element after the order was known read three or four
// sectors a vortex at random, and a thread, warp or block per bucket by its
// size needed a third launch: place and order of both grids 59 / 131 / 370 us
// at 2e4 / 1e6 / 3e6 vortices, now 29 / 66 / 195.
VX_DEVK void k_bk_place_body(VxBlkB<0, 0> vb, const long long *d_n, const unsigned *key, const int *rank,
                             const int *start, VxOrderRec *rec, const VxGather &gt) {
    const long long n = *d_n;
    for (long long i = vb.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)vb.n * blockDim.x) {
        const unsigned c = key[i];
        const int pos = start[c] + rank[i];
        const float4 q = gt.mode ? vx_gather(gt, i, c) : make_float4(0.f, 0.f, 0.f, 0.f);
        VxOrderRec *r = rec + pos;
        r->val = q;
        *reinterpret_cast<int4 *>(&r->key) = make_int4((int)c, (int)i, 0, 0);
    }
}
__global__ void k_bk_place(const long long *d_n, const unsigned *key, const int *rank, const int *start,
                           VxOrderRec *rec, VxGather gt) {
    VX_PDL_WAIT();
    k_bk_place_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, d_n, key, rank, start, rec, gt);
}

VX_DEVK void k_bk_order_body(VxBlkB<0, 0> vb, const long long *d_n, const VxOrderRec *rec, const int *start,
                             unsigned *okey, int *oval, float4 *srt, const VxScalars *born_of, int *born) {
    const long long n = *d_n;
    const long long b0 = born ? born_of->n0 : 0, b1 = born ? born_of->n : 0;
    for (long long p = vb.x * (long long)blockDim.x + threadIdx.x; p < n;
         p += (long long)vb.n * blockDim.x) {
        const int2 ki = *reinterpret_cast<const int2 *>(&rec[p].key);
        const unsigned c = (unsigned)ki.x;
        const int i = ki.y, a = start[c], e = start[c + 1];
        float4 q;
        if (srt) q = rec[p].val;
        int to = a;
#pragma unroll 4
        for (int k = a; k < e; ++k) to += rec[k].idx < i;
        okey[p] = c;
        oval[to] = i;
        if (srt) srt[to] = q;
        if (i >= b0 && i < b1) born[i - b0] = to;
    }
}
__global__ void k_bk_order(const long long *d_n, const VxOrderRec *rec, const int *start, unsigned *okey, int *oval,
                           float4 *srt, const VxScalars *born_of, int *born) {
    VX_PDL_WAIT();
    k_bk_order_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, d_n, rec, start, okey, oval, srt, born_of, born);
}

cudaError_t vx_bucket_order(const VxLaunch &L, const long long *d_n, const unsigned *key, const int *rank,
                            const int *start, unsigned *okey, int *oval, VxOrderRec *rec, const VxGather &gt) {
    const int grid = L.num_sms * 8;
    vx_launch<k_bk_place, k_bk_place_body>(L, grid, 256, 0, d_n, key, rank, start, rec, gt);
    VxLaunch next = L;
    next.pdl = true;
    vx_launch<k_bk_order, k_bk_order_body>(next, grid, 256, 0, d_n, (const VxOrderRec *)rec, start, okey, oval, gt.mode ? gt.srt : nullptr, gt.S, gt.born);
    return cudaGetLastError();
}

// Validation hook: the bucket order of n keys (device array, each below nb)
// into `order` (device array of n element indices), with starts and ranks
// computed on the host (the ranks against index order).  Allocates its own scratch; not for the step path.
extern "C" vx_status vx_eval_bucket_order(const unsigned *key, int64_t n, int64_t nb, int *order) {
    if (n < 0 || nb < 1 || n > INT_MAX || (n > 0 && (!key || !order))) return VX_ERR_ARG;
    if (n == 0) return VX_OK;
    std::vector<unsigned> hk((size_t)n);
    if (cudaMemcpy(hk.data(), key, sizeof(unsigned) * n, cudaMemcpyDeviceToHost) != cudaSuccess) return VX_ERR_CUDA;
    std::vector<int> cnt((size_t)nb, 0), start((size_t)nb + 1, 0);
    for (unsigned k : hk) {
        if ((int64_t)k >= nb) return VX_ERR_ARG;
        ++cnt[k];
    }
    for (int64_t b = 0; b < nb; ++b) start[b + 1] = start[b] + cnt[b];
    std::vector<int> rank((size_t)n), left(cnt);
    for (int64_t i = 0; i < n; ++i) rank[i] = --left[hk[i]];
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    void *mem[5] = {};
    const size_t sz[5] = {sizeof(long long), sizeof(int) * (nb + 1), sizeof(int) * n, sizeof(unsigned) * n,
                          sizeof(VxOrderRec) * n};
    vx_status st = VX_OK;
    for (int q = 0; q < 5 && st == VX_OK; ++q)
        if (cudaMalloc(&mem[q], sz[q]) != cudaSuccess) st = VX_ERR_NOMEM;
    if (st == VX_OK) {
        long long *dn = (long long *)mem[0];
        const long long hn = (long long)n;
        int *dstart = (int *)mem[1], *drank = (int *)mem[2];
        bool ok = cudaMemcpy(dn, &hn, sizeof(hn), cudaMemcpyHostToDevice) == cudaSuccess &&
                  cudaMemcpy(dstart, start.data(), sizeof(int) * (nb + 1), cudaMemcpyHostToDevice) == cudaSuccess &&
                  cudaMemcpy(drank, rank.data(), sizeof(int) * n, cudaMemcpyHostToDevice) == cudaSuccess;
        if (ok) {
            VxLaunch L;
            L.stream = 0;
            L.launches = nullptr;
            L.num_sms = sms;
            ok = vx_bucket_order(L, dn, key, drank, dstart, (unsigned *)mem[3], order,
                                 (VxOrderRec *)mem[4]) == cudaSuccess &&
                 cudaDeviceSynchronize() == cudaSuccess;
        }
        if (!ok) st = VX_ERR_CUDA;
    }
    for (void *p : mem) if (p) cudaFree(p);
    return st;
}

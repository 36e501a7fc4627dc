// vx_fmm.cu — bulk-form Biot-Savart velocity by a quadtree fast multipole
// method, with the mean 3-nearest distance from the near field.
//
// Replaces, for the bulk form, the direct O(N^2) sum of the reference's
// shared_Kernel (src/kernel.cu:875-983); the reference's own tree
// (src/kernel.cu:78-763, src/unit_1.cu:686-960) is off in every shipped
// configuration, so the direct sum is the parity target.
//
// With z = x + i y, the conjugate velocity induced by vortices j is
//   u - i v = 1/(2 pi i) sum_j G_j / (z - z_j)         (|z - z_j| >= eps)
// and the core smoothing max(r^2, eps^2) only acts closer than eps.  The
// leaves are at least eps wide, so every pair that goes through expansions
// is farther apart than eps and sees the plain Cauchy kernel.
//
// Tree: uniform levels 0..L over the particles' square bounding box, dense
// row-major cell arrays per level.  Expansions in FP64, scaled by the cell
// side s (w = (z - c)/s keeps every coefficient O(1)) and by factorials:
//   multipole  B_k  = (1/k!) sum_j G_j w_j^k               (P2M)
//   field      f(z) = sum_k k! B_k s^k (z - c)^-(k+1)
//   local      f(z) = sum_l A_l u^l / l!,  u = (z - c)/s      (M2L, L2L, L2P)
// M2L between two cells of one level with integer offset t = (c_T - c_S)/s
// is then a Hankel product (no binomials):
//   A_l += ((-1)^l / s) sum_k B_k H_{k+l},  H_j = j! t^-(j+1),
// and the shifts M2M / L2L use E_p = d^p / p! for the child offset d:
//   B_k(parent) = sum_m E_{k-m} 2^-m B_m(child),
//   A_l(child)  = 2^-l sum_{j>=l} E_{j-l} A_j(parent).
// Interaction list: children of the parent's 3x3 neighbours that are not
// neighbours of the cell.  Near field: the 3x3 leaves around a target's leaf,
// direct FP32 with the core smoothing; the 3 nearest come from there and are
// exact when the third distance is below the leaf side (nothing outside the
// 3x3 block can be closer); the few targets that fail the test are redone by
// a search over squares of leaves.
#include <algorithm>

#include "vx_internal.cuh"

// Expansion terms P: a template parameter of the kernels that hold
// expansions, one of VX_FMM_ORDERS (run-time choice, VxParams::fmm_p).
constexpr int FMM_PMAX = 20;
constexpr int FMM_T = 256;
constexpr int FMM_W = 32;        // targets per near-field work item (one warp)

struct cplx {
    double r, i;
};
__device__ __forceinline__ cplx cmul(cplx a, cplx b) { return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
__device__ __forceinline__ cplx cadd(cplx a, cplx b) { return {a.r + b.r, a.i + b.i}; }
__device__ __forceinline__ cplx cscale(cplx a, double s) { return {a.r * s, a.i * s}; }
__device__ __forceinline__ cplx cinv(cplx a) {
    const double d = a.r * a.r + a.i * a.i;
    return {a.r / d, -a.i / d};
}

__host__ __device__ inline long long fmm_level_off(int l) { return ((1LL << (2 * l)) - 1) / 3; }

// 1/k for k = 1..FMM_PMAX (folded at compile time)
__constant__ double c_fmm_inv[FMM_PMAX + 1] = {0.0,      1.0,      1.0 / 2,  1.0 / 3,  1.0 / 4,  1.0 / 5,
                                               1.0 / 6,  1.0 / 7,  1.0 / 8,  1.0 / 9,  1.0 / 10, 1.0 / 11,
                                               1.0 / 12, 1.0 / 13, 1.0 / 14, 1.0 / 15, 1.0 / 16, 1.0 / 17,
                                               1.0 / 18, 1.0 / 19, 1.0 / 20};
// M2L blocks stage their tables in dynamic shared memory (over 48 KB at P = 20)
extern __shared__ __align__(16) unsigned char vx_fmm_dyn[];

// ---------------------------------------------------------------------------
// Start of the velocity stage, one launch: the count arrays zeroed to their
// capacity, the bounding box (per-block keys into part[], combined by the
// last block), then, in the last block, the stage's counters and the tree:
// square box, depth L = ceil(log4(n / leaf)) within [2, Lmax], deepened while
// the leaf occupancy a vortex sees would reach 2 leaf, reduced until the leaf
// side is at least eps.  The occupancy a vortex sees is sum(c^2) / n over the
// cells; the last build measured it over its quarter-leaf cells (k_fmm_leafid),
// and at the density it implies, a leaf of side a holds rho a^2.  A clustered
// cloud (a dense wall layer, a Gaussian core) then gets the depth its dense
// part needs rather than the one its bounding box implies; a uniform one
// keeps ceil(log4(n / leaf)).  The first build of a body (no measurement yet)
// uses the box rule alone.  Deepening stops one level above a build whose
// 3-nearest pass left more than 0.5 % of its targets to the exact search.
VX_DEVK void k_fmm_prep_body(VxBlkB<FMM_T, 0> vb, const VxView &v, VxScalars *S, double eps, int Lmax, int leaf, int *cnt,
                             long long ncnt, int *subcnt, long long nsub, unsigned long long *part) {
    const long long n = S->n;
    for (long long c = vb.x * (long long)blockDim.x + threadIdx.x; c < ncnt + nsub;
         c += (long long)vb.n * blockDim.x) {
        if (c < ncnt) cnt[c] = 0;
        else subcnt[c - ncnt] = 0;
    }
    unsigned long long k[4] = {~0ull, ~0ull, ~0ull, ~0ull};
    for (long long i = vb.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)vb.n * blockDim.x) {
        const double x = v.x[i * v.ps], y = v.y[i * v.ps];
        k[0] = min(k[0], vx_dkey(x)); k[1] = min(k[1], vx_dkey(-x));
        k[2] = min(k[2], vx_dkey(y)); k[3] = min(k[3], vx_dkey(-y));
    }
    vx_block_min4<FMM_T / 32>(k);
    if (threadIdx.x == 0)
        for (int q = 0; q < 4; ++q) part[4 * vb.x + q] = k[q];
    if (!vx_last_block(&S->sync_side, vb.n)) return;
    for (int q = 0; q < 4; ++q) k[q] = ~0ull;
    for (unsigned b = threadIdx.x; b < vb.n; b += blockDim.x)
        for (int q = 0; q < 4; ++q) k[q] = min(k[q], __ldcg(&part[4 * b + q]));
    vx_block_min4<FMM_T / 32>(k);
    if (threadIdx.x != 0) return;
    // the last build's quarter-cell occupancy, sources, box, depth and the
    // targets its 3-nearest pass left to the exact search
    const unsigned long long q2 = S->fsq;
    const long long s_prev = S->fs;
    const double side_prev = S->fside;
    const int L_prev = S->fL;
    const long long flags_prev = S->fnflag;
    S->fsq = 0;
    S->fnflag = 0;
    S->fnbrute = 0;
    const double x0 = vx_dunkey(k[0]), x1 = -vx_dunkey(k[1]);
    const double y0 = vx_dunkey(k[2]), y1 = -vx_dunkey(k[3]);
    double side = fmax(x1 - x0, y1 - y0);
    side = side * (1.0 + 1e-9) + 1e-12;
    // the depth's ceiling follows the count, not the store's capacity (the
    // arrays are sized for the capacity's ceiling, which is never lower), so
    // the tree does not depend on when the store grew
    int Lc = 2;
    while (Lc < 10 && (double)(1LL << (2 * Lc)) * 8.0 < (double)vx_round32(n)) ++Lc;
    Lmax = min(Lmax, Lc);
    int L = 2;
    while (L < Lmax && (double)(1LL << (2 * L)) * (double)leaf < (double)n) ++L;
    // a tree deep enough for a dense region leaves the sparse rest of the
    // cloud with quarters too small for their 3 nearest: once a build left
    // more than 0.5 % of its targets to the exact search, the depth rule
    // deepens no further than one level above that build, from then on
    if (q2 > 0 && s_prev > 0 && L_prev >= 3 && flags_prev * 200 > s_prev)
        S->fLcap = S->fLcap > 0 ? min(S->fLcap, L_prev - 1) : L_prev - 1;
    const int Ldeep = S->fLcap > 0 ? max(L, min(Lmax, S->fLcap)) : Lmax;
    if (q2 > 0 && s_prev > 0 && side_prev > 0.0 && L_prev >= 1) {
        const double qa = side_prev / (double)(2LL << L_prev);                      // quarter side then
        const double rho = (double)q2 / (double)s_prev / (qa * qa) * ((double)vx_round32(n) / (double)s_prev);
        while (L < Ldeep) {
            const double a = side / (double)(1LL << L);
            if (rho * a * a < 2.0 * (double)leaf) break;
            ++L;
        }
    }
    while (L > 2 && side / (double)(1LL << L) < eps) --L;
    // a box smaller than 4 eps: no pair may use an expansion, all near field
    if (side / 4.0 < eps) L = 1;
    S->fx0 = 0.5 * (x0 + x1) - 0.5 * side;
    S->fy0 = 0.5 * (y0 + y1) - 0.5 * side;
    S->fside = side;
    S->fL = L;
    S->fcnt_off = fmm_level_off(L);
    S->fnleaves = 1LL << (2 * L);
    S->fnsub = 4 * S->fnleaves;
    S->fs = vx_round32(n);   // sources include the round-32 padding (3-nearest)
}
__global__ void __launch_bounds__(FMM_T) k_fmm_prep(VxView v, VxScalars *S, double eps, int Lmax, int leaf, int *cnt,
                                                    long long ncnt, int *subcnt, long long nsub,
                                                    unsigned long long *part) {
    VX_PDL_WAIT();
    k_fmm_prep_body(VxBlkB<FMM_T, 0>{blockIdx.x, gridDim.x}, v, S, eps, Lmax, leaf, cnt, ncnt, subcnt, nsub, part);
}

__device__ __forceinline__ long long fmm_leaf(const VxScalars *S, double x, double y) {
    const long long m = 1LL << S->fL;
    const double h = S->fside / (double)m;
    long long ix = (long long)floor((x - S->fx0) / h), iy = (long long)floor((y - S->fy0) / h);
    ix = ix < 0 ? 0 : (ix >= m ? m - 1 : ix);
    iy = iy < 0 ? 0 : (iy >= m ? m - 1 : iy);
    return iy * m + ix;
}

// Cell of the level below the leaves of every source slot [0, s), as the
// key 4 leaf + child (child = 2 (row & 1) + (column & 1) at that level), so
// that sorting by it keeps each leaf's sources contiguous, its four quarters
// one after the other; counts per key.  The leaf of the key is the one
// fmm_leaf gives (x / (h/2) is exactly 2 (x / h)).
__device__ __forceinline__ unsigned fmm_subkey(const VxScalars *S, double x, double y) {
    const long long m2 = 2LL << S->fL;
    const double h2 = 0.5 * (S->fside / (double)(m2 >> 1));
    long long ix = (long long)floor((x - S->fx0) / h2), iy = (long long)floor((y - S->fy0) / h2);
    ix = ix < 0 ? 0 : (ix >= m2 ? m2 - 1 : ix);
    iy = iy < 0 ? 0 : (iy >= m2 ? m2 - 1 : iy);
    const long long leaf = (iy >> 1) * (m2 >> 1) + (ix >> 1);
    return (unsigned)(4 * leaf + 2 * (iy & 1) + (ix & 1));
}

// The sum of count^2 over the cells (the next build's depth rule) comes from
// the same increments: a cell's count going from c to c + 1 adds 2 c + 1.
VX_DEVK void k_fmm_leafid_body(VxBlkB<0, 0> vb, const VxView &v, VxScalars *S, unsigned *key, int *rank, int *subcnt) {
    const long long s = S->fs;
    unsigned long long sq = 0;
    for (long long j = vb.x * (long long)blockDim.x + threadIdx.x; j < s;
         j += (long long)vb.n * blockDim.x) {
        const unsigned k = fmm_subkey(S, v.x[j * v.ps], v.y[j * v.ps]);
        const int r = atomicAdd(&subcnt[k], 1);
        key[j] = k;
        rank[j] = r;
        sq += 2ull * (unsigned)r + 1ull;
    }
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0 && sq) atomicAdd(&S->fsq, sq);
}
__global__ void k_fmm_leafid(VxView v, VxScalars *S, unsigned *key, int *rank, int *subcnt) {
    VX_PDL_WAIT();
    k_fmm_leafid_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, v, S, key, rank, subcnt);
}

constexpr int FMM_SCAN_PER = 8;
// Starts of the quarters (one-pass scan of their counts), and with them the
// leaf counts (the tree's leaf level: the sum of a leaf's four quarters) and
// the leaf starts (its first quarter's); both end with the sources' total.
VX_DEVK void k_fmm_scan_body(VxBlkB<VX_SCAN_T, 0> vb, VxScalars *S, int *subcnt, int *substart, int *cnt,
                             int *start, unsigned long long *tiles) {
    constexpr int PER = FMM_SCAN_PER;   // a multiple of 4: a thread holds whole leaves
    const long long len = S->fnsub, nl = S->fnleaves;
    int *leafcnt = cnt + fmm_level_off(S->fL);
    vx_scan_lookback<PER>(
        vb.n, len, S, tiles, [&](long long i0, unsigned (&val)[PER]) { vx_scan_load<false>(subcnt, i0, len, val); },
        [&](long long i0, const unsigned (&val)[PER], long long run) {
            vx_scan_store(substart, i0, len, val, run);
#pragma unroll
            for (int q = 0; q < PER; q += 4) {
                if (i0 + q >= len) break;
                const long long leaf = (i0 + q) >> 2;
                const int c = (int)(val[q] + val[q + 1] + val[q + 2] + val[q + 3]);
                leafcnt[leaf] = c;
                start[leaf] = (int)run;
                run += c;
            }
        },
        [&](long long) {
            substart[len] = (int)S->fs;
            start[nl] = (int)S->fs;
        });
}
__global__ void __launch_bounds__(VX_SCAN_T) k_fmm_scan(VxScalars *S, int *subcnt, int *substart, int *cnt, int *start,
                                                        unsigned long long *tiles) {
    VX_PDL_WAIT();
    k_fmm_scan_body(VxBlkB<VX_SCAN_T, 0>{blockIdx.x, gridDim.x}, S, subcnt, substart, cnt, start, tiles);
}

// Shift table shared by M2M and L2L, built per block in shared memory:
// E[q][p] = d_q^p / p! for the child offsets d_q = (+-1 +- i)/4 (in units of
// the parent side), q = (dy > 0) * 2 + (dx > 0).
template <int P>
__device__ __forceinline__ void fmm_shift_table(cplx (*se)[P]) {
    if (threadIdx.x < 4) {
        const int q = threadIdx.x;
        const cplx dd = {(q & 1) ? 0.25 : -0.25, (q >> 1) ? 0.25 : -0.25};
        cplx pw = {1.0, 0.0};
        for (int p = 0; p < P; ++p) { se[q][p] = pw; pw = cscale(cmul(pw, dd), c_fmm_inv[p + 1]); }
    }
}

// The upward pass.  A warp takes a cell of level L - 1: P2M of its four
// leaves (8 lanes each, a lane every eighth vortex of the leaf, FP64
// positions), then M2M of the cell from the coefficients just summed, in
// shared memory; a block's four warps are the children of a cell of level
// L - 2, which its first warp sums last.  Eight lanes a leaf keep the sum over
// the lanes short (28 shuffles for four leaves; a warp a leaf, 31 each, spent
// most of its time on them) and a block's chain is two levels whatever the
// depth: 4^(L-2) blocks instead of 4^(L-3), with one leaf after another a
// quarter as long.  Upward pass (this kernel and k_fmm_up_top, event times) at
// 2e4 vortices 87 -> 26 us, at 1e6 131 -> 68, at 3e6 370 -> 192; bound by the
// gathers of the positions and the levels' latency.
//
// Expansions of empty cells are not written: nothing reads them (the counts
// of all levels start at zero).  Levels 1 and 0 have no interactions and are
// not summed beyond what a block of a shallow tree writes on its way.
constexpr int FMM_TOP = 3;  // levels below this one are left to the last block of the upward pass
constexpr int UP_W = 4;     // warps of a block of k_fmm_up

__device__ __forceinline__ double fmm_pow2n(int k) {   // 2^-k
    return __longlong_as_double((long long)(1023 - k) << 52);
}

// M2M of one cell by one warp, coefficients of the children q = 0..3 in
// src[q][m], already scaled by 2^-m: lane (k, q) sums the terms of
// coefficient k from child q, four lanes add up (all get the sum).
template <int P>
__device__ __forceinline__ cplx fmm_m2m_terms(const cplx (*se)[P], const cplx (*src)[P], int k, int q) {
    cplx b = {0.0, 0.0};
#pragma unroll
    for (int m = 0; m < P; ++m)
        if (m <= k) {
            const cplx e = se[q][k - m], t = src[q][m];
            b.r = fma(e.r, t.r, fma(-e.i, t.i, b.r));
            b.i = fma(e.r, t.i, fma(e.i, t.r, b.i));
        }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        b.r += __shfl_xor_sync(0xffffffffu, b.r, o);
        b.i += __shfl_xor_sync(0xffffffffu, b.i, o);
    }
    return b;
}

template <int P>
VX_DEVK void k_fmm_up_body(VxBlkB<32 * UP_W, 4> vb, const VxView &v, const VxScalars *S, const int *start,
                           const int *sorted, int *cnt, cplx *M) {
    constexpr int V = 2 * P / 8;   // values a lane keeps of its leaf's 2 P
    __shared__ cplx se[4][P];
    __shared__ double sf[P];                // 1 / k!
    __shared__ cplx sb[UP_W][4][P];         // the leaves' coefficients times 2^-k
    __shared__ cplx sp[4][P];               // and those of level L - 1
    __shared__ int sn[UP_W];
    const int L = S->fL;
    if (L < 2) return;   // no expansions
    const long long m = 1LL << L, n = S->n;
    const double h = S->fside / (double)m, ih = 1.0 / h, fx0 = S->fx0, fy0 = S->fy0;
    cplx *ML = M + fmm_level_off(L) * P, *M1 = M + fmm_level_off(L - 1) * P, *M2 = M + fmm_level_off(L - 2) * P;
    int *cnt1 = cnt + fmm_level_off(L - 1), *cnt2 = cnt + fmm_level_off(L - 2);
    fmm_shift_table<P>(se);
    if (threadIdx.x == 0) {
        double f = 1.0;
        for (int k = 0; k < P; ++k) { sf[k] = f; f *= c_fmm_inv[k + 1]; }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = lane >> 3, l8 = lane & 7;
    const long long m2 = m >> 2;
    for (long long r = vb.x; r < m2 * m2; r += vb.n) {
        const long long px = 2 * (r % m2) + (warp & 1), py = 2 * (r / m2) + (warp >> 1);   // level L - 1
        const long long ix = 2 * px + (q & 1), iy = 2 * py + (q >> 1), c = iy * m + ix;
        const int j0 = start[c], j1 = start[c + 1];
        const int np = __reduce_add_sync(0xffffffffu, l8 == 0 ? j1 - j0 : 0);
        if (np > 0) {
            double acc[2 * P];
#pragma unroll
            for (int k = 0; k < 2 * P; ++k) acc[k] = 0.0;
            const double cx = fx0 + ((double)ix + 0.5) * h, cy = fy0 + ((double)iy + 0.5) * h;
            long long jn = j0 + l8 < j1 ? sorted[j0 + l8] : n;
            for (int t = j0 + l8; t < j1; t += 8) {
                const long long j = jn;   // the next vortex's index is loaded before this one is expanded
                jn = t + 8 < j1 ? sorted[t + 8] : n;
                if (j >= n) continue;
                const double wr = (v.x[j * v.ps] - cx) * ih, wi = (v.y[j * v.ps] - cy) * ih;
                double pr = v.g[j * v.ps], pi = 0.0;   // G w^k
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    acc[2 * k] += pr;
                    acc[2 * k + 1] += pi;
                    const double nr = fma(pr, wr, -(pi * wi));
                    pi = fma(pr, wi, pi * wr);
                    pr = nr;
                }
            }
            __syncwarp();
            // reduce-scatter over the leaf's eight lanes: at each halving a
            // lane keeps the half its lane bit selects and adds the partner's
            // copy of it; lane l8 ends with values V l8 ..
#pragma unroll
            for (int half = P, o = 4; o > 0; half >>= 1, o >>= 1) {
                const bool up = (l8 & o) != 0;
#pragma unroll
                for (int i = 0; i < half; ++i) {
                    const double send = up ? acc[i] : acc[i + half];
                    const double keep = up ? acc[i + half] : acc[i];
                    acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const int e = V * l8 + i, k = e >> 1;
                const double b = acc[i] * sf[k];
                if (j1 > j0) reinterpret_cast<double *>(ML + c * P)[e] = b;
                reinterpret_cast<double *>(sb[warp][q])[e] = b * fmm_pow2n(k);
            }
            __syncwarp();
        }
        if (np > 0) {
            const long long c1 = py * (m >> 1) + px;
            if (lane == 0) cnt1[c1] = np;
#pragma unroll
            for (int k0 = 0; k0 < P; k0 += 8) {
                const int k = k0 + (lane >> 2);
                const cplx b = fmm_m2m_terms<P>(se, sb[warp], k < P ? k : P - 1, lane & 3);
                if ((lane & 3) == 0 && k < P) {
                    M1[c1 * P + k] = b;
                    sp[warp][k] = cscale(b, fmm_pow2n(k));
                }
            }
        } else {
            for (int k = lane; k < P; k += 32) sp[warp][k] = cplx{0.0, 0.0};
        }
        if (lane == 0) sn[warp] = np;
        __syncthreads();
        const int np2 = sn[0] + sn[1] + sn[2] + sn[3];
        if (warp == 0 && np2 > 0) {
            if (lane == 0) cnt2[r] = np2;
#pragma unroll
            for (int k0 = 0; k0 < P; k0 += 8) {
                const int k = k0 + (lane >> 2);
                const cplx b = fmm_m2m_terms<P>(se, sp, k < P ? k : P - 1, lane & 3);
                if ((lane & 3) == 0 && k < P) M2[r * P + k] = b;
            }
        }
        __syncthreads();
    }
}
template <int P>
__global__ void __launch_bounds__(32 * UP_W, 4) k_fmm_up(VxView v, const VxScalars *S, const int *start,
                                                         const int *sorted, int *cnt, cplx *M) {
    VX_PDL_WAIT();
    k_fmm_up_body<P>(VxBlkB<32 * UP_W, 4>{blockIdx.x, gridDim.x}, v, S, start, sorted, cnt, M);
}

// M2M of the cells of level l below cell r of level lo, a warp per cell.
// Children are read through L2: another block of the same launch may have
// written them.
template <int P>
__device__ __forceinline__ void fmm_m2m_level(const cplx (*se)[P], cplx (*src)[P], int *cnt, cplx *M, int lo, int l,
                                              long long r) {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const long long m = 1LL << l, m2 = 2 * m, mlo = 1LL << lo, sl = 1LL << (l - lo);
    const int *cc = cnt + fmm_level_off(l + 1);
    const cplx *Mc = M + fmm_level_off(l + 1) * P;
    for (long long e = threadIdx.x >> 5; e < sl * sl; e += nw) {
        const long long ix = (r % mlo) * sl + e % sl, iy = (r / mlo) * sl + e / sl;
        // a child's count and coefficients are loaded side by side (an empty
        // child's are whatever was there, and dropped)
        int np = 0;
#pragma unroll
        for (int w0 = 0; w0 < 4 * P; w0 += 32) {
            const int w = w0 + lane, q = min(w / P, 3), k = w % P;
            const long long child = (2 * iy + (q >> 1)) * m2 + 2 * ix + (q & 1);
            const int nq = __ldcg(&cc[child]);
            const double2 t = __ldcg(reinterpret_cast<const double2 *>(&Mc[child * P + k]));
            np += __reduce_add_sync(0xffffffffu, w < 4 * P && k == 0 ? nq : 0);
            if (w < 4 * P) src[q][k] = nq > 0 ? cscale(cplx{t.x, t.y}, fmm_pow2n(k)) : cplx{0.0, 0.0};
        }
        __syncwarp();
        if (np == 0) continue;
        const long long c = iy * m + ix;
        if (lane == 0) (cnt + fmm_level_off(l))[c] = np;
#pragma unroll
        for (int k0 = 0; k0 < P; k0 += 8) {
            const int k = k0 + (lane >> 2);
            const cplx b = fmm_m2m_terms<P>(se, src, k < P ? k : P - 1, lane & 3);
            if ((lane & 3) == 0 && k < P) M[(fmm_level_off(l) + c) * P + k] = b;
        }
        __syncwarp();
    }
}

// The rest of the upward pass: levels L - 3 up to 3, a block per cell of
// level 3, then level 2 by the block that finishes last.
constexpr int TOP_W = 16;
template <int P>
VX_DEVK void k_fmm_up_top_body(VxBlkB<32 * TOP_W, 0> vb, VxScalars *S, int *cnt, cplx *M) {
    __shared__ cplx se[4][P];
    __shared__ cplx src[TOP_W][4][P];
    const int hi = S->fL - 2;
    if (hi < FMM_TOP) return;
    fmm_shift_table<P>(se);
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    for (long long r = vb.x; r < (1LL << (2 * FMM_TOP)); r += vb.n)
        for (int l = hi - 1; l >= FMM_TOP; --l) {
            fmm_m2m_level<P>(se, src[warp], cnt, M, FMM_TOP, l, r);
            __syncthreads();
        }
    if (!vx_last_block(&S->sync_ctr, vb.n)) return;
    fmm_m2m_level<P>(se, src[warp], cnt, M, 0, FMM_TOP - 1, 0);
}
template <int P>
__global__ void __launch_bounds__(32 * TOP_W) k_fmm_up_top(VxScalars *S, int *cnt, cplx *M) {
    VX_PDL_WAIT();
    k_fmm_up_top_body<P>(VxBlkB<32 * TOP_W, 0>{blockIdx.x, gridDim.x}, S, cnt, M);
}

// M2L at level l (2 <= l <= L) plus L2L from level l-1.  A block takes a
// 4 x 4 tile of target cells (two parents wide); the interaction lists of the
// tile draw on the 8 x 8 source cells around it (children of the parents'
// neighbours), whose multipoles are staged once in shared memory.  The
// Hankel entries H_j = j! t^-(j+1) of the integer offsets t are tabulated
// per block.
//
// H_j(-t) = (-1)^(j+1) H_j(t) and H_j(conj t) = conj H_j(t), so the sources B1
// .. B4 of a cell at t, -t, conj t and -conj t share one Hankel product: with
// sigma = (-1)^(k+l+1), U = B1 + sigma B2 and W = B3 + sigma B4,
//   Re: (U.r + W.r) h.r - (U.i - W.i) h.i,
//   Im: (U.r - W.r) h.i + (U.i + W.i) h.r
// are the four sources' term of (k, l): 4 FP64 FMAs for four sources (and 16
// additions a k for both signs, shared by the l) instead of 16.  The 27
// sources of an interaction list, offsets [-2, 3]^2 (mirrored by the cell's
// place in its parent) without [-1, 1]^2, fall into 12 such sets:
//   (2,1) (1,2) (2,2) with all four; (3,1) (3,2) with their conjugates;
//   (1,3) (2,3) with their negative conjugates; (2,0) (0,2) with their
//   negatives; (3,0) (0,3) (3,3) alone.
// Thread (cell, coefficient group cg, part pt) sums the G coefficients G cg ..
// G cg + G - 1 (G = 8 where it divides the order, else 4) over three of them,
// one of each kind of code (a missing source is a row of zeros), so that the
// parts of a warp run together.  A ring of G Hankel entries stays in
// registers.  The four parts (adjacent lanes) are then reduce-scattered in a
// fixed tree, so part pt ends with coefficients G cg + (G / 4) pt onwards.
// All levels at 1e6 vortices (event times) 171 -> 130 us, at 3e6 521 -> 364, against
// a product per source with unpadded rows (4-way bank conflicts).
//
// The levels up to M2L_SMALL have few cells each: their M2L parts are
// independent of one another and run in one launch over all their tiles
// (k_fmm_m2l_small), then their L2L level by level (k_fmm_l2l_small); deeper
// levels take one launch each (k_fmm_m2l_l2l), M2L and L2L together.
constexpr int M2L_TILE = 4;
constexpr int M2L_SRC = 2 * M2L_TILE;   // 8 x 8 staged source cells
constexpr int M2L_SMALL = 6;
template <int P> __host__ __device__ constexpr int m2l_group() { return P % 8 == 0 ? 8 : 4; }   // coefficients a thread sums
template <int P> __host__ __device__ constexpr int m2l_threads() { return M2L_TILE * M2L_TILE * 4 * (P / m2l_group<P>()); }
#ifndef VX_M2L_MINB
#define VX_M2L_MINB 0   // minimum resident blocks per SM requested for the M2L kernels (0: none)
#endif

template <int P>
struct M2LShared {
    // rows of 16 (odd) bytes, so that the rows of a warp's lanes fall into
    // different banks
    cplx sh[49][2 * P + 1];   // offset (dx, dy) in [-3, 3]^2 at (dy+3)*7 + dx+3
    cplx se[4][P];
    cplx sm[M2L_SRC * M2L_SRC + 1][P + 1];   // the last row: zeros
    int sc[M2L_SRC * M2L_SRC];
};

template <int P>
__device__ void m2l_tables(M2LShared<P> &T) {
    fmm_shift_table<P>(T.se);
    for (int q = threadIdx.x; q < 49; q += blockDim.x) {
        const int dx = q % 7 - 3, dy = q / 7 - 3;
        if (abs(dx) <= 1 && abs(dy) <= 1) continue;   // neighbours: never an interaction
        const cplx ti = cinv(cplx{(double)dx, (double)dy});
        cplx tp = ti;
        double fact = 1.0;   // j!
        for (int j = 0; j < 2 * P - 1; ++j) {
            T.sh[q][j] = cscale(tp, fact);
            tp = cmul(tp, ti);
            fact *= (double)(j + 1);
        }
        T.sh[q][2 * P - 1] = T.sh[q][2 * P] = cplx{0.0, 0.0};   // loaded ahead, not used
    }
    for (int k = threadIdx.x; k <= P; k += blockDim.x) T.sm[M2L_SRC * M2L_SRC][k] = cplx{0.0, 0.0};
}

// One set of sources (b2, b3, b4 at the negative, the conjugate, the negative
// conjugate of b1's offset; MASK bits 2, 4, 8: which of them the code has)
// into the G coefficients of v.  H: the offset's entries from G cg on.
template <int P, int MASK>
__device__ __forceinline__ void m2l_set(double (&v)[2 * m2l_group<P>()], const cplx *H, const cplx *b1, const cplx *b2,
                                        const cplx *b3, const cplx *b4) {
    constexpr int G = m2l_group<P>();
    cplx h[G];   // H_{k + j} at (k + j) % G
#pragma unroll
    for (int j = 0; j < G; ++j) h[j] = H[j];
#pragma unroll 1
    for (int k0 = 0; k0 < P; k0 += G) {
#pragma unroll
        for (int kk = 0; kk < G; ++kk) {
            const int k = k0 + kk;
            // [0]: k + l even (sigma -1), [1]: odd (sigma +1)
            cplx U[2], W[2];
            U[0] = U[1] = b1[k];
            W[0] = W[1] = cplx{0.0, 0.0};
            if (MASK & 2) {
                const cplx c = b2[k];
                U[0] = cplx{U[0].r - c.r, U[0].i - c.i};
                U[1] = cplx{U[1].r + c.r, U[1].i + c.i};
            }
            if (MASK & 4) W[0] = W[1] = b3[k];
            if (MASK & 8) {
                const cplx c = b4[k];
                W[0] = cplx{W[0].r - c.r, W[0].i - c.i};
                W[1] = cplx{W[1].r + c.r, W[1].i + c.i};
            }
            double pr[2], qi[2], ri[2], sr[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (MASK & 12) {
                    pr[e] = U[e].r + W[e].r; qi[e] = U[e].i - W[e].i;
                    ri[e] = U[e].r - W[e].r; sr[e] = U[e].i + W[e].i;
                } else {
                    pr[e] = ri[e] = U[e].r;
                    qi[e] = sr[e] = U[e].i;
                }
            }
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const cplx t = h[(kk + j) % G];
                const int e = (kk + j) & 1;
                v[2 * j] = fma(pr[e], t.r, fma(-qi[e], t.i, v[2 * j]));
                v[2 * j + 1] = fma(ri[e], t.i, fma(sr[e], t.r, v[2 * j + 1]));
            }
            h[kk] = H[k + G];
        }
    }
}

// M2L of tile t of level l for this thread's (cell, lc); the block's threads
// all take part.  Returns whether the cell exists; *c its index, *busy
// whether it holds vortices, *a its scaled M2L coefficient lc.
template <int P>
__device__ bool m2l_tile(const VxScalars *S, const int *cnt, const cplx *M, int l, long long t, M2LShared<P> &T,
                         long long &c, bool &busy, int &lc0, cplx (&a)[2]) {
    constexpr int G = m2l_group<P>(), NC = G / 4, TPC = 4 * (P / G);   // threads per cell
    const long long m = 1LL << l;
    const long long tiles1 = vx_ceil_div(m, (long long)M2L_TILE);
    const double s = S->fside / (double)m;
    const cplx *Ml = M + fmm_level_off(l) * P;
    const int *cl = cnt + fmm_level_off(l);
    const int cell = threadIdx.x / TPC;
    const int cg = (threadIdx.x % TPC) >> 2, pt = threadIdx.x & 3;
    lc0 = G * cg + NC * pt;
    const long long tx0 = (t % tiles1) * M2L_TILE, ty0 = (t / tiles1) * M2L_TILE;
    const long long sx0 = tx0 - 2, sy0 = ty0 - 2;   // staged region origin
    const long long ix = tx0 + cell % M2L_TILE, iy = ty0 + cell / M2L_TILE;
    const bool live = ix < m && iy < m;
    c = live ? iy * m + ix : 0;
    // the barrier: the previous tile is done with sm / sc, tables are built;
    // a tile with no vortex under any of its cells is skipped (an empty
    // cell's local expansion is never read: L2L and L2P read busy cells only)
    if (!__syncthreads_or(live && cl[c] > 0)) {
        busy = false;
        return false;
    }
    for (int e = threadIdx.x; e < M2L_SRC * M2L_SRC * P; e += blockDim.x) {
        const int q = e / P, k = e % P;
        const long long qx = sx0 + q % M2L_SRC, qy = sy0 + q / M2L_SRC;
        const bool in = qx >= 0 && qx < m && qy >= 0 && qy < m;
        const long long src = qy * m + qx;
        const int n = in ? cl[src] : 0;
        if (k == 0) T.sc[q] = n;
        T.sm[q][k] = n > 0 ? Ml[src * P + k] : cplx{0.0, 0.0};
    }
    __syncthreads();
    busy = live && cl[c] > 0;
    double v[2 * G];   // (re, im) of coefficients G cg + j
#pragma unroll
    for (int j = 0; j < 2 * G; ++j) v[j] = 0.0;
    if (__any_sync(0xffffffffu, busy)) {
        constexpr int NONE = M2L_SRC * M2L_SRC;
        // the source fa right and fb up of the cell, mirrored by its place in
        // its parent: its row of sm, the row of zeros if it is empty or not
        // wanted (all lie in the staged region)
        const int fx = (ix & 1) ? -1 : 1, fy = (iy & 1) ? -1 : 1;
        const int here = (int)(iy - sy0) * M2L_SRC + (int)(ix - sx0);
        const auto at = [&](int fa, int fb, bool want = true) {
            const int q = here + fy * fb * M2L_SRC + fx * fa;
            return want && T.sc[q] > 0 ? q : NONE;
        };
        const auto hank = [&](int fa, int fb) { return T.sh[(3 - fy * fb) * 7 + 3 - fx * fa] + G * cg; };
        {   // (2,1) (1,2) (2,2) with all four, (2,0) with its negative
            const int fa = pt == 1 ? 1 : 2, fb = pt == 0 ? 1 : (pt == 3 ? 0 : 2);
            const int q1 = at(fa, fb), q2 = at(-fa, -fb), q3 = at(fa, -fb, pt != 3), q4 = at(-fa, fb, pt != 3);
            if (__any_sync(0xffffffffu, min(min(q1, q2), min(q3, q4)) < NONE))
                m2l_set<P, 15>(v, hank(fa, fb), T.sm[q1], T.sm[q2], T.sm[q3], T.sm[q4]);
        }
        {   // (3,1) (3,2) with their conjugates, (1,3) (2,3) with their negative conjugates
            const int fa = pt < 2 ? 3 : pt - 1, fb = pt < 2 ? pt + 1 : 3;
            const int q1 = at(fa, fb), q3 = at(fa, pt < 2 ? -fb : fb, pt < 2), q4 = at(pt < 2 ? fa : -fa, fb, pt >= 2);
            if (__any_sync(0xffffffffu, min(q1, min(q3, q4)) < NONE))
                m2l_set<P, 13>(v, hank(fa, fb), T.sm[q1], nullptr, T.sm[q3], T.sm[q4]);
        }
        {   // (3,0) (0,3) (3,3) alone, (0,2) with its negative
            const int fa = pt == 0 || pt == 2 ? 3 : 0, fb = pt == 0 ? 0 : (pt == 3 ? 2 : 3);
            const int q1 = at(fa, fb), q2 = at(0, pt == 3 ? -2 : 0, pt == 3);
            if (__any_sync(0xffffffffu, min(q1, q2) < NONE))
                m2l_set<P, 3>(v, hank(fa, fb), T.sm[q1], T.sm[q2], nullptr, nullptr);
        }
    }
    // reduce-scatter over the four parts (all lanes take part): first with
    // the part two lanes away (halves of the G coefficients), then with the
    // neighbouring part (halves of those): (p0 + p2) + (p1 + p3) for each
#pragma unroll
    for (int lvl = 0; lvl < 2; ++lvl) {
        const int half = G >> lvl, x = 2 >> lvl;
        const bool up = (pt & x) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const double send = up ? v[i] : v[i + half];
            const double keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, x);
        }
    }
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        a[i] = {v[2 * i], v[2 * i + 1]};
        if (busy) a[i] = cscale(a[i], (((lc0 + i) & 1) ? -1.0 : 1.0) / s);
    }
    return live;
}

// L2L of coefficient lc of cell (ix, iy) of level l from its parent's local
// expansion Lp (level l-1).
template <int P>
__device__ __forceinline__ cplx l2l_term(const cplx *Lp, const cplx (*se)[P], long long m, long long ix,
                                         long long iy, int lc) {
    const long long parent = (iy >> 1) * (m >> 1) + (ix >> 1);
    const int q = (int)((iy & 1) * 2 + (ix & 1));
    cplx acc = {0.0, 0.0};
#pragma unroll
    for (int j = 0; j < P; ++j)   // unrolled, the terms below lc predicated off: the loads issue together
        if (j >= lc) acc = cadd(acc, cmul(Lp[parent * P + j], se[q][j - lc]));
    return cscale(acc, ldexp(1.0, -lc));
}

template <int P>
VX_DEVK void k_fmm_m2l_l2l_body(VxBlkB<m2l_threads<P>(), 0> vb, const VxScalars *S, const int *cnt, const cplx *M,
                                cplx *Loc, int l) {
    constexpr int NC = m2l_group<P>() / 4;
    M2LShared<P> &T = *reinterpret_cast<M2LShared<P> *>(vx_fmm_dyn);
    if (l > S->fL) return;
    m2l_tables<P>(T);
    const long long m = 1LL << l;
    const long long tiles1 = vx_ceil_div(m, (long long)M2L_TILE);
    cplx *Ll = Loc + fmm_level_off(l) * P;
    const cplx *Lp = Loc + fmm_level_off(l - 1) * P;
    for (long long t = vb.x; t < tiles1 * tiles1; t += vb.n) {
        long long c;
        bool busy;
        int lc0;
        cplx a[2];
        if (!m2l_tile<P>(S, cnt, M, l, t, T, c, busy, lc0, a)) continue;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            if (busy && l > 2) a[i] = cadd(a[i], l2l_term<P>(Lp, T.se, m, c % m, c / m, lc0 + i));
            Ll[c * P + lc0 + i] = a[i];
        }
    }
}
template <int P>
__global__ void __launch_bounds__(m2l_threads<P>(), VX_M2L_MINB) k_fmm_m2l_l2l(const VxScalars *S, const int *cnt, const cplx *M,
                                                       cplx *Loc, int l) {
    VX_PDL_WAIT();
    k_fmm_m2l_l2l_body<P>(VxBlkB<m2l_threads<P>(), 0>{blockIdx.x, gridDim.x}, S, cnt, M, Loc, l);
}

// M2L (without L2L) of levels 2 .. min(M2L_SMALL, L): blocks over the tiles
// of all of them.
template <int P>
VX_DEVK void k_fmm_m2l_small_body(VxBlkB<m2l_threads<P>(), 0> vb, const VxScalars *S, const int *cnt, const cplx *M,
                                  cplx *Loc) {
    constexpr int NC = m2l_group<P>() / 4;
    M2LShared<P> &T = *reinterpret_cast<M2LShared<P> *>(vx_fmm_dyn);
    const int hi = min(S->fL, M2L_SMALL);
    if (hi < 2) return;
    m2l_tables<P>(T);
    long long total = 0;
    for (int l = 2; l <= hi; ++l) total += vx_ceil_div(1LL << (2 * l), (long long)(M2L_TILE * M2L_TILE));
    for (long long b = vb.x; b < total; b += vb.n) {
        int l = 2;
        long long t = b;
        while (t >= vx_ceil_div(1LL << (2 * l), (long long)(M2L_TILE * M2L_TILE))) {
            t -= vx_ceil_div(1LL << (2 * l), (long long)(M2L_TILE * M2L_TILE));
            ++l;
        }
        long long c;
        bool busy;
        int lc0;
        cplx a[2];
        if (!m2l_tile<P>(S, cnt, M, l, t, T, c, busy, lc0, a)) continue;
#pragma unroll
        for (int i = 0; i < NC; ++i) Loc[(fmm_level_off(l) + c) * P + lc0 + i] = a[i];
    }
}
template <int P>
__global__ void __launch_bounds__(m2l_threads<P>(), VX_M2L_MINB) k_fmm_m2l_small(const VxScalars *S, const int *cnt, const cplx *M,
                                                         cplx *Loc) {
    VX_PDL_WAIT();
    k_fmm_m2l_small_body<P>(VxBlkB<m2l_threads<P>(), 0>{blockIdx.x, gridDim.x}, S, cnt, M, Loc);
}

// L2L into levels 3 .. min(M2L_SMALL, L), one launch: a block takes a cell
// of level 3 and walks down its subtree level by level (a barrier between
// levels), one thread per (cell, coefficient).
template <int P>
VX_DEVK void k_fmm_l2l_small_body(VxBlkB<256, 0> vb, const VxScalars *S, const int *cnt, cplx *Loc) {
    __shared__ cplx se[4][P];
    const int hi = min(S->fL, M2L_SMALL);
    if (hi < 3) return;
    fmm_shift_table<P>(se);
    __syncthreads();
    for (long long r = vb.x; r < 64; r += vb.n) {
        const long long rx = r % 8, ry = r / 8;
        for (int l = 3; l <= hi; ++l) {
            const long long sl = 1LL << (l - 3), m = 1LL << l;
            const int *cl = cnt + fmm_level_off(l);
            cplx *Ll = Loc + fmm_level_off(l) * P;
            const cplx *Lp = Loc + fmm_level_off(l - 1) * P;
            for (long long e = threadIdx.x; e < sl * sl * P; e += blockDim.x) {
                const long long q = e / P;
                const int lc = (int)(e % P);
                const long long c = (ry * sl + q / sl) * m + rx * sl + q % sl;
                if (cl[c] > 0) Ll[c * P + lc] = cadd(Ll[c * P + lc], l2l_term<P>(Lp, se, m, c % m, c / m, lc));
            }
            __syncthreads();
        }
    }
}
template <int P>
__global__ void __launch_bounds__(256) k_fmm_l2l_small(const VxScalars *S, const int *cnt, cplx *Loc) {
    VX_PDL_WAIT();
    k_fmm_l2l_small_body<P>(VxBlkB<256, 0>{blockIdx.x, gridDim.x}, S, cnt, Loc);
}

// Near field (FP32, core smoothing) + far field (L2P, FP64): one warp per
// work item of up to FMM_W targets of one leaf.  All of them share the 3 x 3
// leaves around it, whose sources the warp stages 32 at a time (three
// contiguous runs of the leaf-sorted array), coordinates relative to the
// item's leaf centre.  The 3 nearest come from their own pass
// (k_fmm_nn3_sub) over the finer grid of quarter leaves.
__device__ __forceinline__ float vx_rcp_approx2(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Two near-field pairs (one target, sources a and b of a staged slot) in
// packed FP32: core-smoothed Biot-Savart terms.  The target's own slot adds
// 0 (dx = dy = 0), so no pair is skipped.  One reciprocal serves both pairs:
// 1/a = b (1/(a b)), 1/b = a (1/(a b)) (a b stays within FP32 range: padding
// sources sit 1e12 away, and both padded gives 1/inf = 0, G = 0).
__device__ __forceinline__ void near_pair2(f2 SX, f2 SYs, f2 G, f2 TX, f2 TY, float eps2, f2 &SY, f2 &SXN) {
    const f2 DX = f2_sub(TX, SX), DY = f2_sub(TY, SYs);
    const f2 R2 = f2_fma(DX, DX, f2_mul(DY, DY));
    float r2a, r2b;
    f2_unpack(R2, r2a, r2b);
    const float ra = fmaxf(r2a, eps2), rb = fmaxf(r2b, eps2);
    const float q = vx_rcp_approx2(ra * rb);
    const f2 MM = f2_mul(G, f2_mul(f2_pack(rb, ra), f2_pack(q, q)));
    SY = f2_fma(MM, DX, SY);
    SXN = f2_fma(MM, DY, SXN);   // sum of +mm dy: negated by the caller
}

#ifndef VX_NEAR_MINB
#define VX_NEAR_MINB 2   // minimum resident blocks per SM requested for k_fmm_near (at most 128 registers)
#endif
// The sources of an item: the 3 x 3 leaves around its own are three
// contiguous runs (rows row-1..row+1 of columns c0..c1), walked as one stream
// in chunks of 32 sources, so only the stream's last chunk is padded.
struct NearRows {
    int j0[3], pre[4];
    float oy[3];   // y offset of the run's row
};
constexpr int NEAR_STRIDE = 36;   // floats a staged chunk: the groups' chunks lie on different banks

// Velocity sums of a warp's targets over the stream.  GF groups of 32 / GF
// lanes hold the same targets and take every GF-th chunk; their sums, FP64
// between chunks, are added at the end (in every lane).  wx, wy, wg: the
// warp's staging rows, a chunk's x, y, G each in NEAR_STRIDE floats, so that
// one 16-byte shared load brings four sources' x (or y, or G).
template <int GF>
__device__ __forceinline__ void near_stream(const float4 *srt, const NearRows &r, f2 TX, f2 TY, float eps2, float hf,
                                            float colf, float *wx, float *wy, float *wg, int lane, double &ax,
                                            double &ay) {
    const int total = r.pre[3];
    // source f of the stream: its slot in the leaf-sorted array and the
    // y offset of its row; the x offset of its column, (column - col) h
    // with the difference -1, 0 or 1, is exact in FP32
    auto src_of = [&](int f, float &oy) {
        const bool in0 = f < r.pre[1], in1 = f < r.pre[2];
        oy = in0 ? r.oy[0] : (in1 ? r.oy[1] : r.oy[2]);
        return in0 ? r.j0[0] + f : (in1 ? r.j0[1] + (f - r.pre[1]) : r.j0[2] + (f - r.pre[2]));
    };
    const int own = GF == 1 ? 0 : lane / (32 / GF) * (NEAR_STRIDE / 4);
    const float4 *cx = reinterpret_cast<const float4 *>(wx) + own, *cy = reinterpret_cast<const float4 *>(wy) + own,
                 *cg = reinterpret_cast<const float4 *>(wg) + own;
    // the next chunks' sources are loaded before the current ones' pairs run
    float4 qn[GF];
    float oyn[GF];
#pragma unroll
    for (int k = 0; k < GF; ++k)
        if (32 * k + lane < total) qn[k] = srt[src_of(32 * k + lane, oyn[k])];
    for (int jt = 0; jt < total; jt += 32 * GF) {
#pragma unroll
        for (int k = 0; k < GF; ++k) {
            // padding: G = 0 sources far away add exactly 0
            const int f = jt + 32 * k + lane;
            float x = 1e12f, y = 1e12f, g = 0.f;
            if (f < total) {
                x = qn[k].x + (qn[k].w - colf) * hf;
                y = qn[k].y + oyn[k];
                g = qn[k].z;
            }
            if (f + 32 * GF < total) qn[k] = srt[src_of(f + 32 * GF, oyn[k])];
            wx[k * NEAR_STRIDE + lane] = x;
            wy[k * NEAR_STRIDE + lane] = y;
            wg[k * NEAR_STRIDE + lane] = g;
        }
        __syncwarp();
        f2 SY = 0ull, SXN = 0ull;   // +0.0f in both halves
#pragma unroll
        for (int q4 = 0; q4 < 8; ++q4) {   // sources 2q, 2q + 1 a pair step, in index order
            const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(cx + q4);
            const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(cy + q4);
            const ulonglong2 G = *reinterpret_cast<const ulonglong2 *>(cg + q4);
            near_pair2(X.x, Y.x, G.x, TX, TY, eps2, SY, SXN);
            near_pair2(X.y, Y.y, G.y, TX, TY, eps2, SY, SXN);
        }
        __syncwarp();
        float a, b;   // the two halves are added in FP32, then carried in FP64
        f2_unpack(SXN, a, b); ax -= (double)(a + b);
        f2_unpack(SY, a, b); ay += (double)(a + b);
    }
#pragma unroll
    for (int o = 32 / GF; o < 32; o <<= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
    }
}

// Near field and the far field's evaluation, one warp per item (up to 32
// targets of one leaf).  Bound: the FMA pipe's nine packed instructions per
// two pairs, and the lanes without a target: a leaf's last item holds any
// number of them, so with at most 16 (8) the warp's halves (quarters) take
// the same targets and every second (fourth) chunk of sources.
// A warp of up to 32 lanes for each item: 262 us at 1e6 vortices, 840 at 3e6; so
// 252 and 667.
template <int P>
VX_DEVK void k_fmm_near_body(VxBlkB<FMM_T, VX_NEAR_MINB> vb, const VxParams &p, const VxView &v, VxScalars *S, const float4 *srt,
                             const int *sorted, const int *start, const int2 *items, const cplx *Loc) {
    __shared__ __align__(16) float stage[FMM_T / 32][3][4 * NEAR_STRIDE];
    const int lane = threadIdx.x & 31;
    float *wx = stage[threadIdx.x >> 5][0], *wy = stage[threadIdx.x >> 5][1], *wg = stage[threadIdx.x >> 5][2];
    const long long n = S->n;
    const int L = S->fL;
    const long long m = 1LL << L;
    const double h = S->fside / (double)m;
    const float eps2 = (float)p.eps2;
    const long long nitems = S->fnitems;
    const cplx *LL = Loc + fmm_level_off(L) * P;
    const long long wpb = FMM_T / 32;
    for (long long it = vb.x * wpb + (threadIdx.x >> 5); it < nitems; it += vb.n * wpb) {
        const int2 item = items[it];
        const long long leaf = item.x;
        const long long row = leaf / m, col = leaf % m;
        const int nt = min(FMM_W, start[leaf + 1] - item.y);   // targets
        const int GF = nt > 16 ? 1 : (nt > 8 ? 2 : 4);
        const int slot = lane & (32 / GF - 1);
        const long long t = item.y + slot;
        const bool valid = slot < nt;
        const float4 me = valid ? srt[t] : make_float4(0.f, 0.f, 0.f, 0.f);   // relative to the leaf centre
        const long long j_self = valid && slot == lane ? sorted[t] : n;
        const long long c0 = max(col - 1, 0LL), c1 = min(col + 1, m - 1);
        const f2 TX = f2_pack(me.x, me.x), TY = f2_pack(me.y, me.y);
        double ax = 0.0, ay = 0.0;
        const long long r_lo = max(row - 1, 0LL), r_hi = min(row + 1, m - 1);
        NearRows rows;
        rows.pre[0] = 0;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const long long rr = r_lo + r;
            int len = 0;
            rows.j0[r] = 0;
            rows.oy[r] = 0.f;
            if (rr <= r_hi) {
                rows.j0[r] = start[rr * m + c0];
                len = start[rr * m + c1 + 1] - rows.j0[r];
                rows.oy[r] = (float)((double)(rr - row) * h);
            }
            rows.pre[r + 1] = rows.pre[r] + len;
        }
        const float hf = (float)h, colf = (float)col;
        if (GF == 1) near_stream<1>(srt, rows, TX, TY, eps2, hf, colf, wx, wy, wg, lane, ax, ay);
        else if (GF == 2) near_stream<2>(srt, rows, TX, TY, eps2, hf, colf, wx, wy, wg, lane, ax, ay);
        else near_stream<4>(srt, rows, TX, TY, eps2, hf, colf, wx, wy, wg, lane, ax, ay);
        // executed near-field pairs: every target of the item sees the same 3x3 leaves
        if (lane == 0) atomicAdd(&S->pairs_bs, (unsigned long long)rows.pre[3] * (unsigned long long)nt);
        if (j_self < n) {
            // far field: f(z) = sum a_l u^l at the target's leaf (none below depth 2)
            cplx f = {0.0, 0.0};
            if (L >= 2) {
                const double xd = v.x[j_self * v.ps], yd = v.y[j_self * v.ps];
                const cplx u = {(xd - (S->fx0 + ((double)col + 0.5) * h)) / h,
                                (yd - (S->fy0 + ((double)row + 0.5) * h)) / h};
                // f = sum_l A_l u^l / l!, nested as A_0 + (u/1)(A_1 + (u/2)(A_2 + ...))
                f = LL[leaf * P + P - 1];
                for (int l = P - 2; l >= 0; --l)
                    f = cadd(cmul(f, cscale(u, c_fmm_inv[l + 1])), LL[leaf * P + l]);
            }
            // u - i v = f / (2 pi i): vx = Im f / 2pi, vy = Re f / 2pi
            v.vx[j_self * v.vs] = (ax + f.i) / VX_TWO_PI + S->vinf[0];
            v.vy[j_self * v.vs] = (ay + f.r) / VX_TWO_PI + S->vinf[1];
        }
    }
}
template <int P>
__global__ void __launch_bounds__(FMM_T, VX_NEAR_MINB) k_fmm_near(VxParams p, VxView v, VxScalars *S, const float4 *srt,
                                                   const int *sorted, const int *start, const int2 *items,
                                                   const cplx *Loc) {
    VX_PDL_WAIT();
    k_fmm_near_body<P>(VxBlkB<FMM_T, VX_NEAR_MINB>{blockIdx.x, gridDim.x}, p, v, S, srt, sorted, start, items, Loc);
}

// The 3 nearest sources of every live target (the reference's padded
// launch: sources include the round-32 slots after the live ones; the
// target itself excluded) over the 3 x 3 quarter leaves around its own
// quarter (each quarter a contiguous run of the sorted sources; coordinates
// relative to the target's leaf centre, computed as the near field computes
// them).  Exact when the third distance is below the quarter's side (every
// source outside the 3 x 3 block is farther); the others go to the search over
// squares of leaves (k_fmm_nn3_fix).
//
// Bound: issue slots.  A lane takes its target's own quarter first, which
// usually settles the three.  A quarter around it whose box lies farther than
// the third distance found so far (with a margin over FP32 rounding) cannot
// hold one of them; a target needs about one of the four edge neighbours
// still, few a corner.  Walked by each lane for its own target, these
// left 12 of 32 lanes active; so the warp lists the (target, quarter) pairs
// that are left, edges, then corners, and deals them out, a pair a lane.  The
// three smallest of several lists do not depend on the order.  2e4 / 1e6 / 3e6
// vortices: 29 -> 15, 144 -> 83, 349 -> 203 us.
VX_DEVK void k_fmm_nn3_sub_body(VxBlkB<FMM_T, 0> vb, const VxView &v, VxScalars *S, const float4 *srt, const unsigned *skey,
                                const int *sorted, const int *substart, int *flag_list) {
    __shared__ unsigned char pair_of[FMM_T / 32][4 * 32];   // lane | neighbour << 5
    const long long s = S->fs, n = S->n;
    const int L = S->fL, m = 1 << L;
    const int lane = threadIdx.x & 31;
    const unsigned before = (1u << lane) - 1u;
    unsigned char *pairs = pair_of[threadIdx.x >> 5];
    const double h = S->fside / (double)m;
    const float sq2 = (float)(0.25 * h * h);   // (quarter side)^2
    // a source's offset to the target's leaf centre: (its leaf's column -
    // col) h and (its leaf's row - row) h, differences of -1, 0 or 1, so
    // exact in FP32 and the same for every source of a quarter
    const float hf = (float)h, hq = 0.5f * hf;
    for (long long t0 = vb.x * (long long)blockDim.x + (threadIdx.x & ~31); t0 < s; t0 += (long long)vb.n * blockDim.x) {
        const long long t = t0 + lane;
        const int j = t < s ? sorted[t] : INT_MAX;
        const bool valid = j < n;
        const unsigned key = valid ? skey[t] : 0u;
        const float4 me = valid ? srt[t] : make_float4(0.f, 0.f, 0.f, 0.f);
        // the quarter's column and row inside its leaf's row of quarters are
        // 2 col + bit 0 and 2 row + bit 1 of the key
        const int col = (int)(key >> 2) & (m - 1), row = (int)(key >> 2) >> L;
        float d1 = 1e5f, d2 = 1e5f, d3 = 1e5f;
        if (valid) {
            const int q1 = substart[key + 1];
#pragma unroll 2
            for (int qq = substart[key]; qq < q1; ++qq) {
                const float2 q = *reinterpret_cast<const float2 *>(srt + qq);   // x, y of the source
                const float dx = me.x - q.x, dy = me.y - q.y;
                vx_nn3_insert_bf(d1, d2, d3, qq == t ? 1e5f : fmaf(dx, dx, dy * dy));
            }
        }
#pragma unroll
        for (int ring = 0; ring < 2; ++ring) {   // the edge neighbours, then the corners
            unsigned want[4];
            int off[4], count = 0;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int ddx = ring ? (e & 1 ? 1 : -1) : (e == 0 ? -1 : (e == 1 ? 1 : 0));
                const int ddy = ring ? (e & 2 ? 1 : -1) : (e == 2 ? -1 : (e == 3 ? 1 : 0));
                // in quarters of the leaf frame: a quarter X of it spans
                // [(X - 1) hq, X hq]
                const int X = (int)(key & 1) + ddx, Y = (int)((key >> 1) & 1) + ddy;
                const float gx = fmaxf(fmaxf((float)(X - 1) * hq - me.x, me.x - (float)X * hq), 0.0f);
                const float gy = fmaxf(fmaxf((float)(Y - 1) * hq - me.y, me.y - (float)Y * hq), 0.0f);
                const bool need = valid && 2 * col + X >= 0 && 2 * col + X < 2 * m && 2 * row + Y >= 0 &&
                                  2 * row + Y < 2 * m && !(fmaf(gx, gx, gy * gy) > 1.0001f * d3);
                want[e] = __ballot_sync(0xffffffffu, need);
                off[e] = count + __popc(want[e] & before);
                count += __popc(want[e]);
                if (need) pairs[off[e]] = (unsigned char)(lane | e << 5);
            }
            __syncwarp();
            for (int base = 0; base < count; base += 32) {
                const bool mine = base + lane < count;
                const int pr = mine ? pairs[base + lane] : 0, src = pr & 31, e = pr >> 5;
                const float tx = __shfl_sync(0xffffffffu, me.x, src), ty = __shfl_sync(0xffffffffu, me.y, src);
                const unsigned tk = __shfl_sync(0xffffffffu, key, src);
                float f1 = 1e5f, f2 = 1e5f, f3 = 1e5f;
                if (mine) {
                    const int ddx = ring ? (e & 1 ? 1 : -1) : (e == 0 ? -1 : (e == 1 ? 1 : 0));
                    const int ddy = ring ? (e & 2 ? 1 : -1) : (e == 2 ? -1 : (e == 3 ? 1 : 0));
                    const int X = (int)(tk & 1) + ddx, Y = (int)((tk >> 1) & 1) + ddy;   // -1 .. 2
                    const int lx = X >> 1, ly = Y >> 1;                                  // leaves off: -1, 0, 1
                    const float ox = (float)lx * hf, oy = (float)ly * hf;
                    const int k = 4 * ((int)(tk >> 2) + ly * m + lx) + 2 * (Y & 1) + (X & 1);
                    const int q1 = substart[k + 1];
#pragma unroll 2
                    for (int qq = substart[k]; qq < q1; ++qq) {
                        const float2 q = *reinterpret_cast<const float2 *>(srt + qq);
                        const float dx = tx - (q.x + ox), dy = ty - (q.y + oy);
                        vx_nn3_insert_bf(f1, f2, f3, fmaf(dx, dx, dy * dy));
                    }
                }
#pragma unroll
                for (int o = 0; o < 4; ++o) {
                    if (want[o] == 0u) continue;
                    const int from = off[o] - base;
                    const float e1 = __shfl_sync(0xffffffffu, f1, from & 31);
                    const float e2 = __shfl_sync(0xffffffffu, f2, from & 31);
                    const float e3 = __shfl_sync(0xffffffffu, f3, from & 31);
                    if ((want[o] >> lane & 1u) && from >= 0 && from < 32) {
                        vx_nn3_insert_bf(d1, d2, d3, e1);
                        vx_nn3_insert_bf(d1, d2, d3, e2);
                        vx_nn3_insert_bf(d1, d2, d3, e3);
                    }
                }
            }
            __syncwarp();
        }
        if (!valid) continue;
        v.d[j] = (double)((sqrtf(d1) + sqrtf(d2) + sqrtf(d3)) / 3);
        if (!(d3 < sq2)) {   // a closer source could lie outside the 3x3 quarters
            const int slot = atomicAdd(&S->fnflag, 1);
            flag_list[slot] = (int)t;
        }
    }
}
__global__ void __launch_bounds__(FMM_T) k_fmm_nn3_sub(VxView v, VxScalars *S, const float4 *srt, const unsigned *skey,
                                                      const int *sorted, const int *substart, int *flag_list) {
    VX_PDL_WAIT();
    k_fmm_nn3_sub_body(VxBlkB<FMM_T, 0>{blockIdx.x, gridDim.x}, v, S, srt, skey, sorted, substart, flag_list);
}

// Targets whose third-nearest distance reached the quarter's side: exact 3
// nearest by a search over the leaves (one warp per target) in the squares of
// leaves within 1, 3 and 6 of the target's.  Every source outside the square
// of half-width k lies at least k h from the target (a source clamped into an
// edge leaf lies farther out than that leaf), so the search stops once the
// third distance is below (k h)^2 or the square covers the grid.  A square's
// rows are contiguous runs of the leaf-sorted sources; the lanes take the
// concatenated runs 32 sources at a time (a lane per leaf, each walking its
// own leaf's sources, left a dense cloud's edge to a few lanes: 48 us in a
// batch of 16 bodies).  Coordinates are relative to the target's leaf
// centre, as in the near field.  An isolated vortex (one flung out of the
// wake) would need rows over much of the grid; it is left to the last block's
// scan of every source.
constexpr int NN3_HALF = 6;                      // half-width of the largest square
constexpr int NN3_ROWS = 2 * NN3_HALF + 1;
struct Nn3Row {
    int j0, pre;   // first source of the row's run, sources of the rows before it
    float oy;      // row offset
};

// The targets that search left over, by one block: each scans every
// source slot (FP64 differences, as the direct pass).
__device__ void fmm_nn3_brute_block(VxView v, VxScalars *S, const int *brute_list) {
    __shared__ float sd[3][FMM_T / 32];
    const int nb = __ldcg(&S->fnbrute);
    const long long fs = S->fs;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int b = 0; b < nb; ++b) {
        const long long i = __ldcg(&brute_list[b]);
        const double xi = v.x[i * v.ps], yi = v.y[i * v.ps];
        float d1 = 1e5f, d2 = 1e5f, d3 = 1e5f;
        for (long long j = threadIdx.x; j < fs; j += blockDim.x) {
            if (j == i) continue;
            const double dx = xi - v.x[j * v.ps], dy = yi - v.y[j * v.ps];
            vx_nn3_insert_bf(d1, d2, d3, (float)fma(dx, dx, dy * dy));
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float e1 = __shfl_xor_sync(0xffffffffu, d1, o);
            const float e2 = __shfl_xor_sync(0xffffffffu, d2, o);
            const float e3 = __shfl_xor_sync(0xffffffffu, d3, o);
            vx_nn3_insert_bf(d1, d2, d3, e1);
            vx_nn3_insert_bf(d1, d2, d3, e2);
            vx_nn3_insert_bf(d1, d2, d3, e3);
        }
        if (lane == 0) { sd[0][warp] = d1; sd[1][warp] = d2; sd[2][warp] = d3; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < FMM_T / 32; ++w) {
                vx_nn3_insert_bf(d1, d2, d3, sd[0][w]);
                vx_nn3_insert_bf(d1, d2, d3, sd[1][w]);
                vx_nn3_insert_bf(d1, d2, d3, sd[2][w]);
            }
            v.d[i] = (double)((sqrtf(d1) + sqrtf(d2) + sqrtf(d3)) / 3);
        }
        __syncthreads();
    }
}

VX_DEVK void k_fmm_nn3_fix_body(VxBlkB<FMM_T, 0> vb, const VxView &v, VxScalars *S, const float4 *srt, const int *sorted,
                                const int *start, const int *flag_list, int *brute_list) {
    __shared__ Nn3Row stab[FMM_T / 32][NN3_ROWS + 1];
    const int nf = S->fnflag;
    const long long m = 1LL << S->fL;
    const double h = S->fside / (double)m;
    const int lane = threadIdx.x & 31;
    Nn3Row *rows = stab[threadIdx.x >> 5];
    const int warps = (vb.n * blockDim.x) >> 5;
    for (int f = (vb.x * blockDim.x + threadIdx.x) >> 5; f < nf; f += warps) {
        const long long t = flag_list[f];
        const long long i = sorted[t];
        const long long leaf = fmm_leaf(S, v.x[i * v.ps], v.y[i * v.ps]);
        const int cx = (int)(leaf % m), cy = (int)(leaf / m);
        const float4 me = srt[t];
        const int kmax = max(max(cx, (int)m - 1 - cx), max(cy, (int)m - 1 - cy));
        float d1 = 1e5f, d2 = 1e5f, d3 = 1e5f;
        bool found = false;
        for (int k = 1; k <= NN3_HALF; k = k == 1 ? 3 : (k == 3 ? NN3_HALF : NN3_HALF + 1)) {
            const int c0 = max(cx - k, 0), c1 = min(cx + k, (int)m - 1), nr = 2 * k + 1;
            int j0 = 0, len = 0;
            const int rr = cy - k + lane;
            if (lane < nr && rr >= 0 && rr < m) {
                j0 = start[rr * m + c0];
                len = start[rr * m + c1 + 1] - j0;
            }
            int inc = len;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += u;
            }
            const int total = __shfl_sync(0xffffffffu, inc, 31);
            if (lane < nr) rows[lane] = Nn3Row{j0, inc - len, (float)((double)(lane - k) * h)};
            if (lane == 0) rows[nr].pre = total;
            __syncwarp();
            d1 = d2 = d3 = 1e5f;
            int rc = 0;
            for (int e = lane; e < total; e += 32) {
                while (rows[rc + 1].pre <= e) ++rc;   // the entry after the last row (the total) stops it
                const Nn3Row r = rows[rc];
                const int j = r.j0 + (e - r.pre);
                if (j == t) continue;
                const float4 q = srt[j];
                // the source's column less the target's, times h
                const float ox = (float)((double)(q.w - (float)cx) * h);
                const float dx = me.x - (q.x + ox), dy = me.y - (q.y + r.oy);
                vx_nn3_insert_bf(d1, d2, d3, fmaf(dx, dx, dy * dy));
            }
            __syncwarp();   // the rows are rewritten by the next square
            for (int o = 16; o > 0; o >>= 1) {
                const float e1 = __shfl_xor_sync(0xffffffffu, d1, o);
                const float e2 = __shfl_xor_sync(0xffffffffu, d2, o);
                const float e3 = __shfl_xor_sync(0xffffffffu, d3, o);
                vx_nn3_insert_bf(d1, d2, d3, e1);
                vx_nn3_insert_bf(d1, d2, d3, e2);
                vx_nn3_insert_bf(d1, d2, d3, e3);
            }
            const float kh = (float)((double)k * h);
            if (d3 < kh * kh || k >= kmax) { found = true; break; }
        }
        if (lane == 0) {
            if (found) v.d[i] = (double)((sqrtf(d1) + sqrtf(d2) + sqrtf(d3)) / 3);
            else brute_list[atomicAdd(&S->fnbrute, 1)] = (int)i;
        }
    }
    // the rare targets no square settled: the block that finishes last scans
    // every source for them
    if (vx_last_block(&S->sync_side, vb.n)) fmm_nn3_brute_block(v, S, brute_list);
}
__global__ void __launch_bounds__(FMM_T) k_fmm_nn3_fix(VxView v, VxScalars *S, const float4 *srt, const int *sorted,
                              const int *start, const int *flag_list, int *brute_list) {
    VX_PDL_WAIT();
    k_fmm_nn3_fix_body(VxBlkB<FMM_T, 0>{blockIdx.x, gridDim.x}, v, S, srt, sorted, start, flag_list, brute_list);
}

// Near-field work items: every leaf's targets in chunks of FMM_W, leaves in
// index order (row-major), as (leaf, first target slot); one-pass scan of
// the leaves' item counts, each thread writing its leaves' items.
VX_DEVK void k_fmm_items_body(VxBlkB<VX_SCAN_T, 0> vb, VxScalars *S, const int *start, int2 *items,
                              long long items_cap, unsigned long long *tiles) {
    constexpr int PER = 4;
    const long long nl = S->fnleaves;
    vx_scan_lookback<PER>(
        vb.n, nl, S, tiles,
        [&](long long c0, unsigned (&val)[PER]) {
#pragma unroll
            for (int q = 0; q < PER; ++q)
                val[q] = c0 + q < nl ? (unsigned)(start[c0 + q + 1] - start[c0 + q] + FMM_W - 1) / FMM_W : 0u;
        },
        [&](long long c0, const unsigned (&val)[PER], long long run) {
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const long long c = c0 + q;
                if (c >= nl) break;
                const int j0 = start[c];
                for (unsigned k = 0; k < val[q]; ++k, ++run)
                    if (run < items_cap) items[run] = make_int2((int)c, j0 + (int)k * FMM_W);
            }
        },
        [&](long long tot) {
            // the item buffer holds s/32 + cells items, so this never truncates
            if (tot > items_cap) S->err |= VX_DERR_GRID;
            S->fnitems = tot <= items_cap ? tot : items_cap;
        });
}
__global__ void __launch_bounds__(VX_SCAN_T) k_fmm_items(VxScalars *S, const int *start, int2 *items,
                                                         long long items_cap, unsigned long long *tiles) {
    VX_PDL_WAIT();
    k_fmm_items_body(VxBlkB<VX_SCAN_T, 0>{blockIdx.x, gridDim.x}, S, start, items, items_cap, tiles);
}

long long vx_fmm_cells(int lmax) { return fmm_level_off(lmax + 1); }

int vx_fmm_max_level(long long cap) {
    int L = 2;
    while (L < 10 && (double)(1LL << (2 * L)) * 8.0 < (double)cap) ++L;
    return L;
}

cudaError_t vx_launch_fmm_tree(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S, VxWork &w,
                               bool early) {
    const int grid = L.num_sms * 4;
    const int Lmax = w.fmm_lmax;
    const int pgrid = std::min(grid, VX_RED_BLOCKS);   // 4 box keys per block
    vx_launch<k_fmm_prep, k_fmm_prep_body>(early ? vx_full_dependency(L) : L, pgrid, FMM_T, 0, v, S, p.eps, Lmax, p.fmm_leaf > 0 ? p.fmm_leaf : 32,
                                           w.fmm_cnt, vx_fmm_cells(Lmax), w.fmm_sub_cnt, 1LL << (2 * (Lmax + 1)),
                                           w.box);
    vx_launch<k_fmm_leafid, k_fmm_leafid_body>(L, grid, FMM_T, 0, v, S, w.key0, w.val0, w.fmm_sub_cnt);
    vx_launch<k_fmm_scan, k_fmm_scan_body>(L, grid, VX_SCAN_T, 0, S, w.fmm_sub_cnt, w.fmm_sub_start,
                                           w.fmm_cnt, w.fmm_start, w.scan_tiles);
    // source order: by quarter-leaf, each quarter's sources in index order
    // (a stable sort by the key 4 leaf + child; each leaf stays contiguous),
    // the FP32 sources gathered at their slots on the way
    VxGather gt;
    gt.mode = 1;
    gt.v = v;
    gt.S = S;
    gt.srt = w.srt;
    gt.born = early ? w.born : nullptr;
    vx_bucket_order(L, &S->fs, w.key0, w.val0, w.fmm_sub_start, w.key1, w.val1, vx_order_rec(w), gt);
    vx_launch<k_fmm_items, k_fmm_items_body>(L, grid, VX_SCAN_T, 0, S, w.fmm_start, w.fitems, w.fitems_cap, w.scan_tiles);
    return cudaGetLastError();
}

cudaError_t vx_launch_fmm_nn3(const VxLaunch &L, const VxView &v, VxScalars *S, VxWork &w) {
    const int grid = L.num_sms * 4;
    vx_launch<k_fmm_nn3_sub, k_fmm_nn3_sub_body>(L, grid * 2, FMM_T, 0, v, S, w.srt, w.key1, w.val1,
                                                 (const int *)w.fmm_sub_start, w.fmm_flags);
    VxLaunch next = L;
    next.pdl = true;
    vx_launch<k_fmm_nn3_fix, k_fmm_nn3_fix_body>(next, grid, FMM_T, 0, v, S, w.srt, w.val1, w.fmm_start, w.fmm_flags, w.fmm_brute);
    return cudaGetLastError();
}

// The new vortices' strengths in the quadtree's order, once they are known.
VX_DEVK void k_fmm_born_body(VxBlkB<0, 0> vb, const VxView &v, const VxScalars *S, const int *born, float4 *srt) {
    const long long n0 = S->n0, m = S->n - n0;
    for (long long i = vb.x * (long long)blockDim.x + threadIdx.x; i < m; i += (long long)vb.n * blockDim.x)
        srt[born[i]].z = (float)v.g[(n0 + i) * v.ps];
}
__global__ void k_fmm_born(VxView v, const VxScalars *S, const int *born, float4 *srt) {
    VX_PDL_WAIT();
    k_fmm_born_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, v, S, born, srt);
}

template <int P>
static cudaError_t velocity_fmm(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S, VxWork &w,
                                bool built) {
    constexpr int M2L_T = m2l_threads<P>();
    constexpr size_t M2L_SMEM = sizeof(M2LShared<P>);
    // over 48 KB of shared memory (P = 20); asked for each time, as a device
    // that was reset has forgotten it
    if (M2L_SMEM > 48 * 1024 && !L.rec) {
        cudaFuncSetAttribute(k_fmm_m2l_l2l<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)M2L_SMEM);
        cudaFuncSetAttribute(k_fmm_m2l_small<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)M2L_SMEM);
    }
    const int grid = L.num_sms * 4;
    const int Lmax = w.fmm_lmax;
    const int *sorted = w.val1;
    // The 3 nearest (and, in a step, the diffusion grid's build after them)
    // share nothing with the expansions and the near field but what is built
    // above, so they run beside them where the body has a side stream: they
    // are short launches, bound by latency, that fill what the others leave.
    // One after the other, velocity and diffusion of 1000 / 30 000 vortices
    // took 148 / 257 us, a step of 2e4 / 1e6 290 / 2260; so 127 / 229, 257 / 2215.
    if (!built) {
        vx_launch_fmm_tree(L, p, v, S, w, false);
        const VxLaunch B = vx_fork(L);
        vx_launch_fmm_nn3(vx_full_dependency(B), v, S, w);
    } else {
        vx_await(L, VX_EVT_TREE);
        vx_launch<k_fmm_born, k_fmm_born_body>(vx_full_dependency(L), (int)vx_ceil_div(p.P, 256), 256, 0, v, S, (const int *)w.born, w.srt);
    }
    // upward pass: P2M + M2M of the 2 levels above the leaves, then the
    // levels above those (two launches whatever the depth)
    const int gup = (int)std::min<long long>(grid * 4, 1LL << (2 * std::max(Lmax - 2, 0)));
    vx_launch<k_fmm_up<P>, k_fmm_up_body<P>>(L, gup, 32 * UP_W, 0, v, S, w.fmm_start, sorted, w.fmm_cnt, (cplx *)w.fmm_M);
    vx_launch<k_fmm_up_top<P>, k_fmm_up_top_body<P>>(L, Lmax - 2 > FMM_TOP ? 1 << (2 * FMM_TOP) : 1, 32 * TOP_W, 0, S, w.fmm_cnt, (cplx *)w.fmm_M);
    {
        long long tiles = 0;
        for (int l = 2; l <= std::min(Lmax, M2L_SMALL); ++l) tiles += vx_ceil_div(1LL << (2 * l), 16LL);
        if (tiles > 0) {
            vx_launch<k_fmm_m2l_small<P>, k_fmm_m2l_small_body<P>>(L, (int)std::min<long long>(grid * 2, tiles), M2L_T, M2L_SMEM, S, w.fmm_cnt, (const cplx *)w.fmm_M, (cplx *)w.fmm_L);
            vx_launch<k_fmm_l2l_small<P>, k_fmm_l2l_small_body<P>>(L, 64, 256, 0, S, w.fmm_cnt, (cplx *)w.fmm_L);
        }
    }
    for (int l = M2L_SMALL + 1; l <= Lmax; ++l) {
        const long long t1 = vx_ceil_div(1LL << l, (long long)M2L_TILE);
        const int g = (int)std::min<long long>(grid * 2, t1 * t1);
        vx_launch<k_fmm_m2l_l2l<P>, k_fmm_m2l_l2l_body<P>>(L, g, M2L_T, M2L_SMEM, S, w.fmm_cnt, (const cplx *)w.fmm_M, (cplx *)w.fmm_L, l);

    }
    VX_EV(L, 0);
    vx_launch<k_fmm_near<P>, k_fmm_near_body<P>>(L, L.num_sms * 8, FMM_T, 0, p, v, S, w.srt, sorted, w.fmm_start,
                                                 w.fitems, (const cplx *)w.fmm_L);
    VX_EV(L, 1);
    return cudaGetLastError();
}

cudaError_t vx_launch_velocity_fmm(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S,
                                   VxWork &w, bool built) {
    switch (p.fmm_p) {
    case 8: return velocity_fmm<8>(L, p, v, S, w, built);
    case 12: return velocity_fmm<12>(L, p, v, S, w, built);
    case 20: return velocity_fmm<20>(L, p, v, S, w, built);
    default: return velocity_fmm<16>(L, p, v, S, w, built);
    }
}

// vx_gj.cu — the panel system's inverse by the reference's Gauss-Jordan
// elimination (src/unit_1.cu:115-227: its pivot rule, or partial pivoting),
// in blocks of GJ_B columns.
//
// Every entry of the augmented matrix goes through the operations of the
// column-by-column elimination in their order: a <- a - c_k * (row k), a
// multiplication and a subtraction each, for k = 0, 1, ...  The updates of an
// entry by the GJ_B steps of a block are only put off until the block's
// multipliers are known, so the result is the column-by-column one bit for
// bit while the matrix is read and written once per GJ_B steps instead of
// once per step.  2 (P+1) launches that each swept it took 16 of the 20 ms a
// body of 1000 panels took to create (of 212 ms at 2576 panels); the blocks
// take 2.6 of 6.6 (16 of 20).
//
//   k_gj_panel   one cluster factorises the block's columns, a matrix row
//                per thread, its GJ_B + 1 entries in registers (the rule
//                looks one column ahead).  Rows stay where they are and
//                carry their position, so a row swap exchanges two numbers;
//                a step costs one barrier: before it each warp publishes its
//                pivot candidate and the pivot row's thread its row, to
//                every block of the cluster.  Bound by the steps' serial
//                chain, 1.4 us each (23 us a block at 1000 panels).
//   k_gj_apply   a block per strip of 8 columns: the block's row moves, the
//                pivot rows' values at their own steps (a triangular solve
//                of GJ_B rows), then every row's GJ_B updates.
//   k_gj_finish  the last step's elimination and the division by the
//                diagonal, written in the inverse's column order.
//
// The right half (the inverse being built) is held by pivot position: the
// column of position q is the unit vector e_q until step q uses it, so only
// the columns of steps already taken are stored; orig[q] is the column of
// the inverse it belongs to.  The eliminated columns left of the block hold
// rounding residuals that later steps still subtract from the diagonal the
// rows are divided by at the end: they are carried below the block and on
// the diagonal, where those steps read them.
#include <algorithm>
#include <climits>

#include <cooperative_groups.h>

#include "vx_internal.cuh"

namespace cg = cooperative_groups;

constexpr int GJ_B = 16;        // steps of a block: 17 + 16 register doubles a row
constexpr int GJ_T = 512;       // most rows of one block of the panel cluster
constexpr long long GJ_ROWS_MIN = 128;   // and the rows that make a further block worth it
constexpr int GJ_MAXC = 8;      // blocks of a portable cluster
constexpr int GJ_STRIP = 8;     // columns of a strip: 64 bytes a row
constexpr int GJ_AT = 256;
constexpr int GJ_U = 4;                                  // rows of a thread at a time
constexpr int GJ_ROWS = GJ_U * (GJ_AT / GJ_STRIP);       // and of the block
constexpr int GJ_MOVES = 2 * GJ_B + 8;   // rows a block's swaps can move (2 a step, 2 for the first column)
constexpr double GJ_DELT = 1e-12;

struct GjPart {
    unsigned hi, lo;   // |value|'s words; the lowest position that holds it
    int pos;
};

// Largest value (lowest position on a tie) over the warp.
__device__ __forceinline__ GjPart gj_warp_best(bool ok, GjPart v) {
    GjPart b;
    b.hi = __reduce_max_sync(0xffffffffu, ok ? v.hi : 0u);
    ok = ok && v.hi == b.hi;
    b.lo = __reduce_max_sync(0xffffffffu, ok ? v.lo : 0u);
    ok = ok && v.lo == b.lo;
    b.pos = __reduce_min_sync(0xffffffffu, ok ? v.pos : INT_MAX);
    return b;
}

template <bool ROBUST>
__global__ void __launch_bounds__(GJ_T) k_gj_panel(double *A, long long ld, int S, int k0, int kb, double *C, int *orig,
                                                   int2 *moved, int *nmoved, int *flag) {
    VX_PDL_WAIT();
    __shared__ GjPart parts[2][GJ_MAXC * GJ_T / 32];
    __shared__ double prow[2][GJ_B + 1];
    extern __shared__ __align__(16) double gj_dyn[];
    double (*Cs)[GJ_B + 1] = reinterpret_cast<double (*)[GJ_B + 1]>(gj_dyn);   // the rows' multipliers
    cg::cluster_group cl = cg::this_cluster();
    const int nc = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (*flag) return;   // set by an earlier launch: the same for every block
    const int row = rank * blockDim.x + threadIdx.x;
    const bool act = row < S;
    int pos = act ? row : INT_MAX;
    const int myorig = act ? orig[row] : 0;
    // the row, rotated by one entry a step: a[0] is the step's column, a[1]
    // the next one (one loop body for all steps: unrolled, its 16 copies ran
    // once each at the speed of instruction fetch)
    double a[GJ_B + 1];
#pragma unroll
    for (int j = 0; j <= GJ_B; ++j) a[j] = act && j <= kb ? A[row * ld + k0 + j] : 0.0;

    auto barrier = [&]() {
        if (nc > 1) cl.sync();
        else __syncthreads();
    };
    // this warp's best |v| among the rows at positions >= lo
    auto publish = [&](double v, int lo, int buf) {
        const bool ok = act && pos >= lo && !isnan(v);
        const unsigned long long key = (unsigned long long)__double_as_longlong(fabs(v));
        const GjPart b = gj_warp_best(ok, GjPart{(unsigned)(key >> 32), (unsigned)key, pos});
        if (lane < nc) *cl.map_shared_rank(&parts[buf][rank * nw + warp], lane) = b;
    };
    auto best_of = [&](int buf, int &line) {
        GjPart m = {0u, 0u, INT_MAX};
        for (int e = lane; e < nc * nw; e += 32) {
            const GjPart q = parts[buf][e];
            if (q.pos != INT_MAX && (m.pos == INT_MAX || q.hi > m.hi || (q.hi == m.hi && (q.lo > m.lo || (q.lo == m.lo && q.pos < m.pos)))))
                m = q;
        }
        m = gj_warp_best(m.pos != INT_MAX, m);
        line = m.pos;
        return m.pos == INT_MAX ? -1.0 : __longlong_as_double((long long)(((unsigned long long)m.hi << 32) | m.lo));
    };
    auto send_row = [&](int k, int buf) {   // the row at position k, to every block
        if (!__any_sync(0xffffffffu, pos == k)) return;
        if (pos == k) {
#pragma unroll
            for (int j = 0; j <= GJ_B; ++j) prow[buf][j] = a[j];
        }
        if (nc > 1) {
            __syncwarp();
            const double v = prow[buf][min(lane, GJ_B)];
            for (int b = 0; b < nc; ++b)
                if (b != rank && lane <= GJ_B) *cl.map_shared_rank(&prow[buf][lane], b) = v;
        }
    };
    auto swap_pos = [&](int p, int q) {
        if (pos == p) pos = q;
        else if (pos == q) pos = p;
    };

    int line;
    barrier();   // every block of the cluster runs before its memory is written
    if (!ROBUST && k0 == 0) {   // a first pivot below the threshold is exchanged
        publish(a[0], 1, 1);
        send_row(0, 1);
        barrier();
        const double best = best_of(1, line), first = fabs(prow[1][0]);
        if (first < GJ_DELT && best > first) swap_pos(0, line);
    }
#pragma unroll 1
    for (int kk = 0; kk < kb; ++kk) {
        const int k = k0 + kk, buf = kk & 1;
        if (ROBUST) {
            publish(a[0], k, buf);
            barrier();
            const double best = best_of(buf, line);
            if (best < GJ_DELT) {
                if (row == 0) *flag = 1;
                return;
            }
            swap_pos(k, line);
            send_row(k, buf);
            barrier();
        } else {
            publish(a[1], k + 1, buf);
            send_row(k, buf);
            barrier();
            const double best = best_of(buf, line);
            if (fabs(prow[buf][0]) < GJ_DELT || best < GJ_DELT) {
                if (row == 0) *flag = 1;
                return;
            }
            swap_pos(k + 1, line);
        }
        double m = 0.0, first = a[0];
        if (pos != k) {
            m = a[0] / prow[buf][0];
            first = a[0] - m * prow[buf][0];
#pragma unroll
            for (int j = 0; j < GJ_B; ++j) a[j] = a[j + 1] - m * prow[buf][j + 1];
        } else {
#pragma unroll
            for (int j = 0; j < GJ_B; ++j) a[j] = a[j + 1];
        }
        a[GJ_B] = first;
        if (act) Cs[threadIdx.x][kk] = m;
    }
    if (!act) return;
    // kb rotations of GJ_B + 1 entries: a[j] is column (j + kb) % (GJ_B + 1)
#pragma unroll
    for (int j = 0; j <= GJ_B; ++j) {
        const int q = j + kb <= GJ_B ? j + kb : j + kb - GJ_B - 1;
        if (q <= kb) A[pos * ld + k0 + q] = a[j];
    }
#pragma unroll
    for (int j = 0; j < GJ_B; ++j) C[(long long)pos * GJ_B + j] = j < kb ? Cs[threadIdx.x][j] : 0.0;
    orig[pos] = myorig;
    if (pos != row) moved[atomicAdd(nmoved, 1)] = make_int2(row, pos);
}

// Strips of 8 columns: first the nR strips right of the panel (columns from
// k0 + kb + 1), then the nG eliminated ones left of it, then the stored
// columns [0, k0 + kb) of the right half W.  128 rows of a strip at a time,
// four entries a thread (four chains of dependent updates); the strip's pivot
// rows stay in registers, the rows' multipliers come through shared memory,
// where the 8 threads of a row read them.  Bound by FP64 issue
// (2 instructions an update) while the matrix fits in L2, by HBM beyond.
__global__ void __launch_bounds__(GJ_AT) k_gj_apply(double *A, double *W, long long ld, int S, int k0, int kb,
                                                    const double *C, const int2 *moved, const int *nmoved,
                                                    const int *flag, int nR, int nG) {
    VX_PDL_WAIT();
    __shared__ double sT[GJ_B][GJ_STRIP], sC[GJ_B][GJ_B], sM[GJ_MOVES][GJ_STRIP];
    __shared__ int2 sl[GJ_MOVES];
    __shared__ double2 sR2[2][GJ_ROWS][GJ_B / 2 + 1];   // multipliers, a row padded by 16 bytes: no bank conflicts
    double (*sR)[GJ_ROWS][GJ_B + 2] = reinterpret_cast<double (*)[GJ_ROWS][GJ_B + 2]>(sR2);
    if (*flag) return;
    const int strip = blockIdx.x;
    const bool right = strip < nR, left = !right && strip < nR + nG;
    double *M = right || left ? A : W;
    const int j0 = right ? k0 + kb + 1 + strip * GJ_STRIP : (strip - nR - (left ? 0 : nG)) * GJ_STRIP;
    const int jend = right ? S : (left ? k0 : k0 + kb);
    const bool fresh = !right && !left && j0 >= k0;   // unit vectors until now
    const int cl = threadIdx.x % GJ_STRIP, rg = threadIdx.x / GJ_STRIP;
    const int j = j0 + cl;
    const bool in = j < jend;
    const int nm = min(*nmoved, GJ_MOVES);
    if (!fresh) {
        for (int e = rg; e < nm; e += GJ_AT / GJ_STRIP) {
            const int2 mv = moved[e];
            if (cl == 0) sl[e] = mv;
            sM[e][cl] = in ? M[mv.x * ld + j] : 0.0;
        }
        __syncthreads();
        for (int e = rg; e < nm; e += GJ_AT / GJ_STRIP)
            if (in) M[sl[e].y * ld + j] = sM[e][cl];
        __syncthreads();
    }
    for (int e = threadIdx.x; e < GJ_B * GJ_B; e += GJ_AT)
        sC[e / GJ_B][e % GJ_B] = e / GJ_B < kb ? C[(long long)(k0 + e / GJ_B) * GJ_B + e % GJ_B] : 0.0;
    if (rg < GJ_B) sT[rg][cl] = !in || rg >= kb ? 0.0 : (fresh ? (k0 + rg == j ? 1.0 : 0.0) : M[(k0 + rg) * ld + j]);
    for (int q = 0; q + 1 < kb; ++q) {
        __syncthreads();
        if (rg > q && rg < kb) sT[rg][cl] = sT[rg][cl] - sC[rg][q] * sT[q][cl];
    }
    __syncthreads();
    double t[GJ_B];
#pragma unroll
    for (int q = 0; q < GJ_B; ++q) t[q] = sT[q][cl];
    if (in && !left && rg < kb) {   // the pivot rows: their later steps
        double v = t[0];
#pragma unroll
        for (int q = 1; q < GJ_B; ++q) v = q == rg ? t[q] : v;
#pragma unroll
        for (int q = 0; q < GJ_B; ++q)
            if (q > rg && q < kb) v = v - sC[rg][q] * t[q];
        M[(k0 + rg) * ld + j] = v;
    }
    if (in && left && rg < GJ_STRIP) {   // the diagonal
        double v = M[(j0 + rg) * ld + j];
#pragma unroll
        for (int q = 0; q < GJ_B; ++q) v = v - C[(long long)(j0 + rg) * GJ_B + q] * t[q];
        M[(j0 + rg) * ld + j] = v;
    }
    // the other rows, GJ_ROWS at a time: the next rows' entries and
    // multipliers are on their way while these are updated
    const int i0 = left ? k0 + kb : 0, nch = (S - i0 + GJ_ROWS - 1) / GJ_ROWS;
    double v[GJ_U];
    const auto fetch = [&](int ch) {
        const int b = i0 + ch * GJ_ROWS;
#pragma unroll
        for (int e = 0; e < GJ_ROWS * GJ_B / 2 / GJ_AT; ++e) {
            const int w = e * GJ_AT + threadIdx.x, r = w / (GJ_B / 2), q = w % (GJ_B / 2);
            if (b + r < S)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 (unsigned)__cvta_generic_to_shared(&sR[ch & 1][r][2 * q])),
                             "l"(C + (long long)(b + r) * GJ_B + 2 * q));
        }
        asm volatile("cp.async.commit_group;");
#pragma unroll
        for (int u = 0; u < GJ_U; ++u) {
            const int i = b + rg + u * (GJ_AT / GJ_STRIP);
            v[u] = in && i < S && !fresh ? M[i * ld + j] : 0.0;
        }
    };
    if (nch > 0) fetch(0);
    for (int ch = 0; ch < nch; ++ch) {
        double w[GJ_U];
#pragma unroll
        for (int u = 0; u < GJ_U; ++u) w[u] = v[u];
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // this chunk's multipliers are here, the other buffer's are used up
        if (ch + 1 < nch) fetch(ch + 1);
#pragma unroll
        for (int q = 0; q < GJ_B; q += 2)
#pragma unroll
            for (int u = 0; u < GJ_U; ++u) {
                const double2 m = *reinterpret_cast<const double2 *>(&sR[ch & 1][rg + u * (GJ_AT / GJ_STRIP)][q]);
                w[u] = w[u] - m.x * t[q];
                w[u] = w[u] - m.y * t[q + 1];
            }
#pragma unroll
        for (int u = 0; u < GJ_U; ++u) {
            const int i = i0 + ch * GJ_ROWS + rg + u * (GJ_AT / GJ_STRIP);
            if (in && i < S && (i < k0 || i >= k0 + kb)) M[i * ld + j] = w[u];
        }
    }
}

__global__ void k_gj_begin(int *orig, int S, int *nmoved, int nblk) {
    VX_PDL_WAIT();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S; i += gridDim.x * blockDim.x) {
        orig[i] = i;
        if (i < nblk) nmoved[i] = 0;
    }
}

// The last step (row S - 1 from the others; its column of the right half is
// still the unit vector) and the division by the diagonal.
__global__ void k_gj_finish(const double *A, const double *W, long long ld, int S, const int *orig, double *Inv,
                            int *flag) {
    VX_PDL_WAIT();
    if (*flag) return;
    const int l = S - 1;
    const double piv = A[l * ld + l];
    if (fabs(piv) < GJ_DELT) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *flag = 2;
        return;
    }
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)S * S;
         e += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(e / S), q = (int)(e % S);
        double w = q < l ? W[i * ld + q] : (i == l ? 1.0 : 0.0);
        if (i < l) {
            const double c = A[i * ld + l] / piv;
            w = w - c * (q < l ? W[l * ld + q] : 1.0);
        }
        Inv[(long long)i * S + orig[q]] = w / A[i * ld + i];
    }
}

static int gj_blocks(long long S) { return (int)vx_ceil_div(S, GJ_B); }
static long long gj_ld(long long S) { return vx_ceil_div(S, GJ_STRIP) * GJ_STRIP; }

// Over 48 KB of shared memory from 362 rows a block on.  Asked for each time (a
// device that was reset has forgotten it), always for the most a block takes
// (bodies may be created from several threads).
static cudaError_t gj_shared(int robust) {
    constexpr int most = (int)sizeof(double) * (GJ_B + 1) * GJ_T;
    return robust ? cudaFuncSetAttribute(k_gj_panel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most)
                  : cudaFuncSetAttribute(k_gj_panel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}

bool vx_gj_fits(long long S) { return S <= (long long)GJ_MAXC * GJ_T; }
long long vx_gj_stride(long long S) { return gj_ld(S); }
long long vx_gj_work(long long S) {   // doubles: A, W, C, then the integer lists
    return 2 * S * gj_ld(S) + S * GJ_B + vx_ceil_div(S + gj_blocks(S) * (2 * GJ_MOVES + 1) + 2, 2);
}

// A: S x S with row stride vx_gj_stride(S), at the start of vx_gj_work(S)
// doubles; Inv: S x S.  robust: partial pivoting instead of the reference's
// rule.
cudaError_t vx_invert_gj(const VxLaunch &L, double *A, double *Inv, long long S, int *flag, int robust) {
    const long long ld = gj_ld(S);
    const int n = (int)S, nblk = gj_blocks(S);
    double *W = A + S * ld, *C = W + S * ld;
    int2 *moved = reinterpret_cast<int2 *>(C + S * GJ_B);
    int *nmoved = reinterpret_cast<int *>(moved + (long long)nblk * GJ_MOVES), *orig = nmoved + nblk;
    // blocks of the panel cluster: 128 rows each (one warp a scheduler; a
    // step is a chain of instructions the warps of a scheduler take turns
    // at) up to 8 blocks, more rows beyond.  Body creation with 128 / 256 /
    // 512 rows a block: 4.2 / 4.5 / 4.8 ms at 400 panels, 6.6 / 7.1 / 8.4 at 1000.
    const unsigned nc = (unsigned)std::min<long long>(GJ_MAXC, vx_ceil_div(S, GJ_ROWS_MIN));
    const unsigned nt = (unsigned)vx_round32(vx_ceil_div(S, (long long)nc));
    VX_COUNT(L);
    cudaError_t e = vx_launch_pdl(k_gj_begin, (unsigned)vx_ceil_div(S, 256LL), 256, 0, L.stream, orig, n, nmoved, nblk);
    if (e == cudaSuccess) e = gj_shared(robust);
    for (int k0 = 0; k0 < n - 1 && e == cudaSuccess; k0 += GJ_B) {
        const int kb = std::min(GJ_B, n - 1 - k0), b = k0 / GJ_B;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(nc);
        cfg.blockDim = dim3(nt);
        cfg.dynamicSmemBytes = sizeof(double) * (GJ_B + 1) * nt;
        cfg.stream = L.stream;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = nc;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 2;
        VX_COUNT(L);
        int2 *mv = moved + (long long)b * GJ_MOVES;
        e = robust ? cudaLaunchKernelEx(&cfg, k_gj_panel<true>, A, ld, n, k0, kb, C, orig, mv, nmoved + b, flag)
                   : cudaLaunchKernelEx(&cfg, k_gj_panel<false>, A, ld, n, k0, kb, C, orig, mv, nmoved + b, flag);
        if (e != cudaSuccess) break;
        const int nR = (int)vx_ceil_div(n - (k0 + kb + 1), GJ_STRIP), nG = k0 / GJ_STRIP;
        const int nW = (int)vx_ceil_div(k0 + kb, GJ_STRIP);
        VX_COUNT(L);
        e = vx_launch_pdl(k_gj_apply, (unsigned)(nR + nG + nW), GJ_AT, 0, L.stream, A, W, ld, n, k0, kb,
                          (const double *)C, (const int2 *)mv, (const int *)(nmoved + b), (const int *)flag, nR, nG);
    }
    if (e != cudaSuccess) return e;
    VX_COUNT(L);
    return vx_launch_pdl(k_gj_finish, (unsigned)std::min(vx_ceil_div(S * S, 256LL), 16LL * L.num_sms), 256, 0, L.stream,
                         (const double *)A, (const double *)W, ld, n, (const int *)orig, Inv, flag);
}

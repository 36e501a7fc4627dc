// vx_collapse.cu — merging of close vortex pairs, two passes (opposite signs,
// then same sign), each repeated up to n_col times while the count changes.
//
// Reference: first_setka_Kernel/second_setka_Kernel src/kernel.cu:1180-1235
// (COL[i] = smallest j > i that qualifies, an O(N^2) scan per thread),
// first_collapse_Kernel/second_collapse_Kernel src/kernel.cu:1237-1271 (one
// thread merges in index order), pass loop src/unit_1.cu:1137-1216.
//
// Here:
//  * COL comes from a uniform cell grid with cells no smaller than the merge
//    radius (counting sort into cells, 3x3 neighbourhood query).  The distance
//    test is the same FP64 expression as the oracle's, so COL is identical.
//  * The serial merge is resolved in parallel.  Candidate i (COL[i] >= 0) is
//    applied iff no applied candidate points at i; rounds decide every
//    candidate whose in-pointing candidates are all decided.  An applied i
//    merges with the original j only if it is the smallest applied candidate
//    pointing at j; later ones merge with (0, 1e10) as the serial loop does,
//    which re-rounds their position.
//  * Compaction then runs as after convection.
// The first round is six launches: prep (box, bookkeeping and grid in one, the
// last block finishing), count, a one-pass scan of the cell counts, scatter,
// query, and settle (resolution, merge, write-back and compaction in one
// block: the settle knows which vortices its merges removed).
//
// The second round takes the first one's grid.  A pair that qualifies in it
// holds a vortex the first round moved (two unmoved ones that qualify would
// have made the first of them a candidate, and every candidate is merged or
// consumed), so only the moved ones look for partners (k_col_query_moved).
// The settle keeps the cell-sorted copy in step: a merged vortex's slot gets
// its new place, a consumed one's strength 0, and the compaction renames the
// ones it moves into holes.  A merged vortex lies between the two it came
// from, closer than a cell side, so its slot is at most one cell off and
// the query looks two cells around.  Second round's kernels before its
// compaction at 1e6 / 3e6 vortices, each timed by itself: 150 / 406 us ->
// 23 / 31.  A third round and later ones build their grid again.
//
// col, in_cnt and first_app are all zero between rounds: the settle clears the
// entries its candidates used.  col holds INT_MAX - j, first_app
// INT_MAX - i (atomicMax keeps the smallest index, 0 is none).
#include <limits.h>

#include "vx_compact.cuh"

// Start of a round: the bounding box (per-block keys into part[], combined
// by the last block), the round's bookkeeping and the cell grid.  A round
// after one that removed nothing (or after a failed one) does nothing: the
// pass has converged (col_done, set by the compaction that removed nothing).  Cell side h = r (1 + 1e-6): any pair closer than r is
// in neighbouring cells; when the box would need more than cells_cap cells,
// h grows.
VX_DEVK void k_col_prep_body(VxBlkB<VX_THREADS, 0> vb, const VxView &v, VxScalars *S, int reset, double r2,
                             long long cells_cap, unsigned long long *part) {
    if (!reset && S->col_done) return;
    const long long n = S->n;
    unsigned long long k[4] = {~0ull, ~0ull, ~0ull, ~0ull};
    for (long long i = vb.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)vb.n * blockDim.x) {
        const double x = v.x[i * v.ps], y = v.y[i * v.ps];
        k[0] = min(k[0], vx_dkey(x));
        k[1] = min(k[1], vx_dkey(-x));
        k[2] = min(k[2], vx_dkey(y));
        k[3] = min(k[3], vx_dkey(-y));
    }
    vx_block_min4<VX_THREADS / 32>(k);
    if (threadIdx.x == 0)
        for (int q = 0; q < 4; ++q) part[4 * vb.x + q] = k[q];
    if (!vx_last_block(&S->sync_ctr, vb.n)) return;
    for (int q = 0; q < 4; ++q) k[q] = ~0ull;
    for (unsigned b = threadIdx.x; b < vb.n; b += blockDim.x)
        for (int q = 0; q < 4; ++q) k[q] = min(k[q], __ldcg(&part[4 * b + q]));
    vx_block_min4<VX_THREADS / 32>(k);
    if (threadIdx.x != 0) return;
    S->col_done = 0;
    S->ncand = 0;
    S->nmoved = 0;
    if (n == 0) { S->gncells = 0; S->gnx = S->gny = 0; return; }
    const double x0 = vx_dunkey(k[0]), x1 = -vx_dunkey(k[1]);
    const double y0 = vx_dunkey(k[2]), y1 = -vx_dunkey(k[3]);
    // side = the collapse radius: the 3 x 3 search is exact and sees the
    // fewest candidates (a side at the mean spacing, with a quarter of the
    // cells to count and scan, was measured slower: the query dominates)
    double h = sqrt(r2) * (1.0 + 1e-6);
    long long nx = -1, ny = -1;
    for (int it = 0; it < 200; ++it) {
        double fx = floor((x1 - x0) / h) + 1.0, fy = floor((y1 - y0) / h) + 1.0;
        if (fx * fy <= (double)cells_cap) { nx = (long long)fx; ny = (long long)fy; break; }
        h *= 1.25;
    }
    if (nx < 0) { S->err |= VX_DERR_GRID; S->gncells = 0; S->col_done = 1; return; }
    S->gx0 = x0; S->gy0 = y0; S->gh = h;
    S->gnx = nx; S->gny = ny; S->gncells = nx * ny;
}
__global__ void __launch_bounds__(VX_THREADS) k_col_prep(VxView v, VxScalars *S, int reset, double r2,
                                                         long long cells_cap, unsigned long long *part) {
    VX_PDL_WAIT();
    k_col_prep_body(VxBlkB<VX_THREADS, 0>{blockIdx.x, gridDim.x}, v, S, reset, r2, cells_cap, part);
}

__device__ __forceinline__ void vx_cell_of(const VxScalars *S, double x, double y, long long &cx,
                                           long long &cy) {
    cx = (long long)floor((x - S->gx0) / S->gh);
    cy = (long long)floor((y - S->gy0) / S->gh);
    cx = cx < 0 ? 0 : (cx >= S->gnx ? S->gnx - 1 : cx);
    cy = cy < 0 ? 0 : (cy >= S->gny ? S->gny - 1 : cy);
}

// Counts per cell (zero between rounds: the scan zeroes them behind it) and
// each vortex's rank in its cell.
VX_DEVK void k_col_count_body(VxBlkB<0, 0> vb, const VxView &v, const VxScalars *S, int *rank, int *cnt) {
    if (S->col_done) return;
    const long long n = S->n;
    for (long long i = vb.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)vb.n * blockDim.x) {
        long long cx, cy;
        vx_cell_of(S, v.x[i * v.ps], v.y[i * v.ps], cx, cy);
        rank[i] = atomicAdd(&cnt[cy * S->gnx + cx], 1);
    }
}
__global__ void k_col_count(VxView v, const VxScalars *S, int *rank, int *cnt) {
    VX_PDL_WAIT();
    k_col_count_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, v, S, rank, cnt);
}

// Cell starts: exclusive scan of the counts in one pass, start[gncells] = n.
constexpr int COL_SCAN_PER = 16;
VX_DEVK void k_col_scan_body(VxBlkB<VX_SCAN_T, 0> vb, VxScalars *S, int *cnt, int *start, unsigned long long *tiles) {
    if (S->col_done) return;
    const long long nc = S->gncells;
    vx_scan_lookback<COL_SCAN_PER>(
        vb.n, nc, S, tiles,
        [&](long long i0, unsigned (&val)[COL_SCAN_PER]) { vx_scan_load<true>(cnt, i0, nc, val); },
        [&](long long i0, const unsigned (&val)[COL_SCAN_PER], long long run) { vx_scan_store(start, i0, nc, val, run); },
        [&](long long tot) { start[nc] = (int)tot; });
}
__global__ void __launch_bounds__(VX_SCAN_T) k_col_scan(VxScalars *S, int *cnt, int *start, unsigned long long *tiles) {
    VX_PDL_WAIT();
    k_col_scan_body(VxBlkB<VX_SCAN_T, 0>{blockIdx.x, gridDim.x}, S, cnt, start, tiles);
}

// A slot of the cell-sorted copy: position, strength and index of the vortex
// (32 bytes, one DRAM sector, written by one thread).
struct __align__(32) ColRec {
    double x, y, g;
    long long i;
};

// Each vortex's slot from its cell's start and its rank (which becomes its
// slot); the slot gets a copy of the vortex (ColRec), so that the query reads
// its candidates as contiguous runs.  A vortex too weak to stay (there is none
// after a compaction) is marked for the round's own.
VX_DEVK void k_col_scatter_body(VxBlkB<0, 0> vb, const VxView &v, const VxScalars *S, const int *start, int *slot,
                                ColRec *rec, double drop_eps, unsigned *dead) {
    if (S->col_done) return;
    const long long n = S->n;
    for (long long i = vb.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)vb.n * blockDim.x) {
        const double x = v.x[i * v.ps], y = v.y[i * v.ps];
        long long cx, cy;
        vx_cell_of(S, x, y, cx, cy);
        const int k = start[cy * S->gnx + cx] + slot[i];
        slot[i] = k;
        double2 *r = reinterpret_cast<double2 *>(rec + k);
        r[0] = make_double2(x, y);
        const double g = v.g[i * v.ps];
        r[1] = make_double2(g, __longlong_as_double(i));
        if (!(fabs(g) >= drop_eps)) vx_set_dead(dead, i);
    }
}
__global__ void k_col_scatter(VxView v, const VxScalars *S, const int *start, int *slot, ColRec *rec, double drop_eps,
                              unsigned *dead) {
    VX_PDL_WAIT();
    k_col_scatter_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, v, S, start, slot, rec, drop_eps, dead);
}

// Whether a pair qualifies in a pass.
template <int PASS>
__device__ __forceinline__ bool vx_col_pair(const VxParams &p, double xi, double yi, double gi, double xj, double yj,
                                            double gj) {
    const double dx = xi - xj, dy = yi - yj;
    const double r2 = fma(dx, dx, dy * dy);
    if (PASS == 1) return (gi * gj < 0) && (r2 < p.r_diff2);
    return (gi * gj > 0) && (r2 < p.r_same2) && (fabs(gi + gj) < p.max_ve_g);
}

// COL[i] = smallest j > i in the 3x3 cell neighbourhood that qualifies.  The
// targets are taken in cell order (slot k0 of the cell-sorted copy), so
// neighbouring threads read the same cells and sources, all as contiguous
// runs of the copy (a row's three cells are one run); each target's answer
// does not depend on the order.  The target's cell is recomputed from its
// position by the count's expression.
template <int PASS>
VX_DEVK void k_col_query_body(VxBlkB<VX_THREADS, 4> vb, const VxParams &p, VxScalars *S, const int *start, const ColRec *rec,
                              int *col, int *cand, int *cstate, int *in_cnt) {
    if (S->col_done) return;
    const long long n = S->n;
    const long long gnx = S->gnx, gny = S->gny;
    for (long long k0 = vb.x * (long long)blockDim.x + threadIdx.x; k0 < n;
         k0 += (long long)vb.n * blockDim.x) {
        const double2 m0 = reinterpret_cast<const double2 *>(rec + k0)[0];
        const double2 m1 = reinterpret_cast<const double2 *>(rec + k0)[1];
        const double xi = m0.x, yi = m0.y, gi = m1.x;
        const long long i = __double_as_longlong(m1.y);
        long long cx, cy;
        vx_cell_of(S, xi, yi, cx, cy);
        int best = INT_MAX;
        for (long long yy = max(cy - 1, 0LL); yy <= min(cy + 1, gny - 1); ++yy) {
            const long long r0 = yy * gnx;
            const int k1 = start[r0 + min(cx + 1, gnx - 1) + 1];
            for (int k = start[r0 + max(cx - 1, 0LL)]; k < k1; ++k) {
                const double2 q1 = reinterpret_cast<const double2 *>(rec + k)[1];
                const int j = (int)__double_as_longlong(q1.y);
                if (j <= i || j >= best) continue;
                const double2 q0 = reinterpret_cast<const double2 *>(rec + k)[0];
                if (vx_col_pair<PASS>(p, xi, yi, gi, q0.x, q0.y, q1.x)) best = j;
            }
        }
        if (best != INT_MAX) {
            const int c = atomicAdd(&S->ncand, 1);
            col[i] = INT_MAX - best;
            cand[c] = (int)i;
            cstate[c] = 0;
            atomicAdd(&in_cnt[best], 1);
        }
    }
}
template <int PASS>
__global__ void k_col_query(VxParams p, VxScalars *S, const int *start, const ColRec *rec, int *col, int *cand,
                            int *cstate, int *in_cnt) {
    VX_PDL_WAIT();
    k_col_query_body<PASS>(VxBlkB<VX_THREADS, 4>{blockIdx.x, gridDim.x}, p, S, start, rec, col, cand, cstate, in_cnt);
}

// Second round: the partners of the vortices the first one moved (their slots
// in moved[]), a lane per row of cells, eight lanes a vortex; a pair of two
// moved ones is met from both sides.
template <int PASS>
VX_DEVK void k_col_query_moved_body(VxBlkB<VX_THREADS, 0> vb, const VxParams &p, VxScalars *S, const int *start,
                                    const ColRec *rec, const int *moved, int *col, int *cand, int *cstate) {
    if (S->col_done) return;
    const int nm = S->nmoved;
    const long long gnx = S->gnx, gny = S->gny;
    const int row = (threadIdx.x & 7) - 2;
    if (row > 2) return;
    for (int e = (vb.x * blockDim.x + threadIdx.x) >> 3; e < nm; e += (vb.n * blockDim.x) >> 3) {
        const int k0 = moved[e];
        const double2 m0 = reinterpret_cast<const double2 *>(rec + k0)[0];
        const double2 m1 = reinterpret_cast<const double2 *>(rec + k0)[1];
        const int i = (int)__double_as_longlong(m1.y);
        long long cx, cy;
        vx_cell_of(S, m0.x, m0.y, cx, cy);
        if (cy + row < 0 || cy + row >= gny) continue;
        const long long r0 = (cy + row) * gnx;
        const int k1 = start[r0 + min(cx + 2, gnx - 1) + 1];
        for (int k = start[r0 + max(cx - 2, 0LL)]; k < k1; ++k) {
            if (k == k0) continue;
            const double2 q0 = reinterpret_cast<const double2 *>(rec + k)[0];
            const double2 q1 = reinterpret_cast<const double2 *>(rec + k)[1];
            if (!(fabs(q1.x) >= p.drop_eps)) continue;   // removed after the first round
            if (!vx_col_pair<PASS>(p, m0.x, m0.y, m1.x, q0.x, q0.y, q1.x)) continue;
            const int j = (int)__double_as_longlong(q1.y), lo = min(i, j);
            if (atomicMax(&col[lo], INT_MAX - max(i, j)) == 0) {
                const int c = atomicAdd(&S->ncand, 1);
                cand[c] = lo;
                cstate[c] = 0;
            }
        }
    }
}
template <int PASS>
__global__ void __launch_bounds__(VX_THREADS) k_col_query_moved(VxParams p, VxScalars *S, const int *start,
                                                                const ColRec *rec, const int *moved, int *col,
                                                                int *cand, int *cstate) {
    VX_PDL_WAIT();
    k_col_query_moved_body<PASS>(VxBlkB<VX_THREADS, 0>{blockIdx.x, gridDim.x}, p, S, start, rec, moved, col, cand, cstate);
}

// One round over the candidate list, by one block: those whose turn it is are
// decided.  U candidates of a thread at a time, all loads of a kind before the
// next: the time of a long list is their latency.
template <int U>
__device__ __forceinline__ void col_decide(int nc, const int *cand, const int *col, int *in_cnt, int *first_app,
                                           int *cstate, int *cdec, int &undecided) {
    const int T = blockDim.x;
    for (int k0 = threadIdx.x; k0 < nc; k0 += U * T) {
        int i[U], taken[U], before[U];
        bool open[U];
#pragma unroll
        for (int u = 0; u < U; ++u) open[u] = k0 + u * T < nc && cstate[k0 + u * T] == 0;
#pragma unroll
        for (int u = 0; u < U; ++u) i[u] = open[u] ? cand[k0 + u * T] : 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            taken[u] = open[u] ? first_app[i[u]] : 0;   // by an applied candidate before it
            before[u] = open[u] ? in_cnt[i[u]] : 0;     // undecided ones before it
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (open[u]) cdec[k0 + u * T] = taken[u] ? 2 : (before[u] == 0 ? 1 : 0);
    }
    if (threadIdx.x == 0) undecided = 0;
    __syncthreads();
    for (int k0 = threadIdx.x; k0 < nc; k0 += U * T) {
        int i[U], j[U], d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) d[u] = k0 + u * T < nc && cstate[k0 + u * T] == 0 ? cdec[k0 + u * T] : -1;
#pragma unroll
        for (int u = 0; u < U; ++u) i[u] = d[u] > 0 ? cand[k0 + u * T] : 0;
#pragma unroll
        for (int u = 0; u < U; ++u) j[u] = d[u] > 0 ? INT_MAX - col[i[u]] : 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (d[u] == 0) undecided = 1;
            if (d[u] <= 0) continue;
            cstate[k0 + u * T] = d[u];
            atomicSub(&in_cnt[j[u]], 1);
            if (d[u] == 1) atomicMax(&first_app[j[u]], INT_MAX - i[u]);
        }
    }
}

// Settles the candidates in one block: rounds over the candidate list decide
// each one (cstate: 0 undecided, 1 applied, 2 consumed before its turn), then
// every applied candidate's merged vortex is written.  An applied candidate is
// nobody's partner, and of those that share a partner the first alone reads
// it and removes it, so no merge reads what another writes.
// counted: in_cnt holds the candidates that point at each vortex (the second
// round's partners are settled only when its query is done).
// track: the cell-sorted copy is kept in step for the second round, and the
// slots of the moved vortices are listed (in cdec, done with by then).
// The round's compaction follows in the same block (vx_cmp_block): what the
// merges removed is marked as they are written.  It adds 8 / 16 / 20 us at
// 2e4 / 1e6 / 3e6 vortices; as four launches over all of them (count,
// classify, gather, scatter) it took 32 / 39 / 50.
// A whole pass of two rounds (vx_stage) with 460 / 44,000 / 406,000 merges of 1e6
// vortices takes 188 / 965 / 9560 us, with 630 / 5300 of 2e4 90 / 200.  With the merged
// values kept between two passes over the list, a second flag per vortex and
// four entries of each candidate cleared, 190 / 1250 / 13,300 and 94 / 236.
template <int PASS>
VX_DEVK void k_col_settle_body(VxBlkB<1024, 0> vb, const VxView &v, VxScalars *S, const int *cand, int *col,
                               int *in_cnt, int *first_app, int *cstate, int *cdec, const int *slot, ColRec *rec,
                               double drop_eps, int track, int counted, const VxCompact &cmp, long long limit) {
    if (threadIdx.x == 0) S->cmp_many = 0;
    if (S->col_done) return;
    __shared__ int undecided, listed;
    const int nc = S->ncand;
    if (threadIdx.x == 0) listed = 0;
    if (!counted)
        for (int k = threadIdx.x; k < nc; k += blockDim.x) atomicAdd(&in_cnt[INT_MAX - col[cand[k]]], 1);
    __syncthreads();
    const int max_rounds = nc + 2;
    int round = 0;
    for (; round < max_rounds; ++round) {
        if (nc > (int)blockDim.x) col_decide<4>(nc, cand, col, in_cnt, first_app, cstate, cdec, undecided);
        else col_decide<1>(nc, cand, col, in_cnt, first_app, cstate, cdec, undecided);
        __syncthreads();
        if (undecided == 0) break;
        __syncthreads();
    }
    const bool failed = round >= max_rounds;
    for (int k0 = 0; k0 < nc; k0 += blockDim.x) {
        const int k = k0 + threadIdx.x;
        int moved = -1;   // slot of a vortex the second round starts from
        if (k < nc) {
            const long long i = cand[k], j = INT_MAX - col[i];
            if (!failed && cstate[k] == 1) {
                const double xi = v.x[i * v.ps], yi = v.y[i * v.ps], gi = v.g[i * v.ps];
                const bool first = first_app[j] == (int)(INT_MAX - i);
                double xj = 1e10, yj = 1e10, gj = 0.0, x, y, g;
                if (first) { xj = v.x[j * v.ps]; yj = v.y[j * v.ps]; gj = v.g[j * v.ps]; }
                if (PASS == 1) {
                    const double ai = fabs(gi), aj = fabs(gj);
                    const double mn = ai + aj;
                    x = (xi * ai + xj * aj) / fabs(mn);
                    y = (yi * ai + yj * aj) / fabs(mn);
                    g = gi + gj;
                } else {
                    g = gi + gj;
                    x = (xi * gi + xj * gj) / g;
                    y = (yi * gi + yj * gj) / g;
                }
                v.x[i * v.ps] = x; v.y[i * v.ps] = y; v.g[i * v.ps] = g;
                const bool left = fabs(g) >= drop_eps;   // else the compaction removes it
                if (!left) vx_set_dead(cmp.bits, i);
                else if (!(fabs(gi) >= drop_eps)) atomicAnd(&cmp.bits[i >> 5], ~(1u << (i & 31)));   // marked by the scatter
                if (track) {
                    const int si = slot[i];
                    ColRec *r = rec + si;
                    r->x = x; r->y = y; r->g = left ? g : 0.0;
                    if (left) moved = si;
                }
                if (first) {
                    v.x[j * v.ps] = 1e10; v.y[j * v.ps] = 1e10; v.g[j * v.ps] = 0.0;
                    if (!(0.0 >= drop_eps)) vx_set_dead(cmp.bits, j);
                    if (track) rec[slot[j]].g = 0.0;
                    first_app[j] = 0;
                }
            }
            // the next round finds the entries clear (every decision took its
            // candidate off in_cnt)
            col[i] = 0;
            if (failed) in_cnt[j] = first_app[j] = 0;
        }
        if (track) {
            const unsigned w = __ballot_sync(0xffffffffu, moved >= 0);
            int at = 0;
            if ((threadIdx.x & 31) == 0 && w) at = atomicAdd(&listed, __popc(w));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(w & ((1u << (threadIdx.x & 31)) - 1u));
            if (moved >= 0) cdec[at] = moved;
        }
    }
    __syncthreads();
    // the round's compaction (none after a failed one); one that removes
    // nothing ends the pass
    const long long n0 = S->n;
    const long long removed = vx_cmp_block<1024>(v, S, cmp, n0, limit, !failed, slot, track ? &rec[0].i : nullptr);
    if (threadIdx.x == 0) {
        S->ncand = 0;
        S->nmoved = listed;
        if (failed) S->err |= VX_DERR_RESOLVE;
        if (failed || removed == 0) S->col_done = 1;
    }
}
template <int PASS>
__global__ void __launch_bounds__(1024) k_col_settle(VxView v, VxScalars *S, const int *cand, int *col,
                                                     int *in_cnt, int *first_app, int *cstate, int *cdec,
                                                     const int *slot, ColRec *rec, double drop_eps, int track,
                                                     int counted, VxCompact cmp, long long limit) {
    VX_PDL_WAIT();
    k_col_settle_body<PASS>(VxBlkB<1024, 0>{blockIdx.x, gridDim.x}, v, S, cand, col, in_cnt, first_app,
                            cstate, cdec, slot, rec, drop_eps, track, counted, cmp, limit);
}

template <int PASS>
static cudaError_t collapse_pass(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S, VxWork &w,
                                 int n_col) {
    const double r2 = PASS == 1 ? p.r_diff2 : p.r_same2;
    const int grid = std::min(L.num_sms * 4, VX_RED_BLOCKS);   // 4 box keys per block
    // the cell-sorted copy (32 bytes a vortex) lives in the pair kernels'
    // partial-sum buffer, unused by collapse (at least 5 doubles a slot)
    ColRec *rec = reinterpret_cast<ColRec *>(w.part);
    const bool small = w.cap <= VX_CMP_SMALL;
    for (int cc = 0; cc < n_col; ++cc) {
        const int track = cc == 0 && n_col > 1;
        if (cc == 1) {
            vx_launch<k_col_query_moved<PASS>, k_col_query_moved_body<PASS>>(L, grid, VX_THREADS, 0, p, S, w.cell_start, (const ColRec *)rec, (const int *)w.cdec, w.col, w.cand, w.cstate);
        } else {
            vx_launch<k_col_prep, k_col_prep_body>(L, grid, VX_THREADS, 0, v, S, cc == 0, r2, w.cells_cap, w.box);
            vx_launch<k_col_count, k_col_count_body>(L, grid, VX_THREADS, 0, v, S, w.cellid, w.cell_cnt);
            vx_launch<k_col_scan, k_col_scan_body>(L, grid, VX_SCAN_T, 0, S, w.cell_cnt, w.cell_start, w.scan_tiles);
            vx_launch<k_col_scatter, k_col_scatter_body>(L, grid, VX_THREADS, 0, v, S, w.cell_start, w.cellid, rec, p.drop_eps, w.cmp.bits);
            vx_launch<k_col_query<PASS>, k_col_query_body<PASS>>(L, grid, VX_THREADS, 0, p, S, w.cell_start, (const ColRec *)rec, w.col, w.cand, w.cstate, w.in_cnt);
        }
        vx_launch<k_col_settle<PASS>, k_col_settle_body<PASS>>(L, 1, 1024, 0, v, S, w.cand, w.col, w.in_cnt, w.first_app, w.cstate, w.cdec, w.cellid, rec, p.drop_eps, track, cc != 1, w.cmp, small ? w.cap : VX_CMP_FEW);
        if (!small) vx_launch_moves(L, v, S, w, w.cellid, track ? &rec[0].i : nullptr);
    }
    return cudaGetLastError();
}

cudaError_t vx_launch_collapse(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S,
                               VxWork &w, int pass, int n_col) {
    const double r2 = pass == 1 ? p.r_diff2 : p.r_same2;
    if (!(r2 > 0.0) || n_col <= 0) return cudaSuccess;   // no pair can qualify
    return pass == 1 ? collapse_pass<1>(L, p, v, S, w, n_col) : collapse_pass<2>(L, p, v, S, w, n_col);
}

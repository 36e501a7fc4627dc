// vx_compact.cuh — the compaction's work from the bits of dead vortices, as
// one block does it (vx_compact.cu describes the permutation it makes).
#pragma once
#include "vx_internal.cuh"

__device__ __forceinline__ bool vx_live(const VxView &v, long long p, double eps) {
    return fabs(v.g[p * v.ps]) >= eps;
}

__device__ __forceinline__ void vx_set_dead(unsigned *bits, long long p) {
    atomicOr(&bits[p >> 5], 1u << (p & 31));
}

// A compaction's moves e, e + stride, ... (U at a time, so that as many
// loads are in flight) below `moves` = H + the dead ones: the first H fill
// the holes, the others are the tail's.  Gather into scratch:
template <int U>
__device__ __forceinline__ void vx_cmp_gather(const VxView &v, const VxCompact &c, long long H, long long moves,
                                              long long first, long long stride) {
    for (long long e0 = first; e0 < moves; e0 += U * stride) {
        long long s[U];
        double x[U], y[U], g[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long e = e0 + u * stride;
            s[u] = e >= moves ? -1 : (e < H ? c.hole_src[e] : c.tail_src[e - H]);
            if (s[u] < 0 && e < moves) s[u] = c.hole_pos[-s[u] - 1];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (s[u] < 0) continue;
            x[u] = v.x[s[u] * v.ps]; y[u] = v.y[s[u] * v.ps]; g[u] = v.g[s[u] * v.ps];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long e = e0 + u * stride;
            if (s[u] < 0) continue;
            if (e < H) { c.hx[e] = x[u]; c.hy[e] = y[u]; c.hg[e] = g[u]; }
            else { c.tx[e - H] = x[u]; c.ty[e - H] = y[u]; }
        }
    }
}
// ... and scatter back.  With rec_i, a vortex moved into a hole gets its new
// index in the collapse's cell-sorted copy (rec_i: the copy's index fields,
// 4 apart; slot: each vortex's slot, by its index before).
template <int U>
__device__ __forceinline__ void vx_cmp_scatter(const VxView &v, const VxCompact &c, long long m, long long H,
                                               long long moves, long long first, long long stride, const int *slot,
                                               long long *rec_i) {
    for (long long e0 = first; e0 < moves; e0 += U * stride) {
        long long d[U];
        double x[U], y[U], g[U];
        int k[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long e = e0 + u * stride;
            d[u] = -1;
            if (e >= moves) continue;
            const bool hole = e < H;
            d[u] = hole ? c.hole_pos[e] : m + e - H;
            x[u] = hole ? c.hx[e] : c.tx[e - H];
            y[u] = hole ? c.hy[e] : c.ty[e - H];
            g[u] = hole ? c.hg[e] : 0.0;
            k[u] = hole && rec_i ? c.hole_src[e] : -1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (d[u] >= 0 && k[u] >= 0) k[u] = slot[k[u]];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (d[u] < 0) continue;
            v.x[d[u] * v.ps] = x[u]; v.y[d[u] * v.ps] = y[u]; v.g[d[u] * v.ps] = g[u];
            if (k[u] >= 0) rec_i[4LL * k[u]] = d[u];
        }
    }
}

// Compaction of [0, n0) from the dead bits, by one block of T threads, which
// leaves the bits at zero.  Returns the dead vortices found.  With up to
// `limit` of them the moves are made and the count S->n set here; with more,
// S->cmp_many is set and the bits, the dead before each 16 bytes of them
// (c.pre) and S->c_* are left for the three launches of vx_launch_moves.
// apply = false: only the bits are cleared.
//
// Bound: the latency of a few dependent passes.  The bits are read twice (31
// KB each 250,000 vortices), a run of them to a warp and four 16-byte loads a
// lane at a time, so that one block-wide scan gives every hole its place (a run
// to a thread, read sector by sector: 37 us a call at 1e6 vortices, not 16);
// the tail's words go the same way.  No list is sorted and nothing of the
// size of the state but the bits is read.
template <int T>
__device__ long long vx_cmp_block(const VxView &v, VxScalars *S, const VxCompact &c, long long n0, long long limit,
                                  bool apply, const int *slot, long long *rec_i) {
    constexpr int NW = T / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int4 *b4 = reinterpret_cast<int4 *>(c.bits);
    const long long n4 = (n0 + 127) / 128, run4 = (n4 + T - 1) / T * 32;
    const long long a = min(n4, warp * run4), b = min(n4, a + run4);
    // the lane's four loads of a round, from q
    auto load = [&](int4 (&w)[4], long long q) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            w[u] = q + u * 32 + lane < b ? __ldcg(&b4[q + u * 32 + lane]) : make_int4(0, 0, 0, 0);
    };
    auto dead_in = [](const int4 &w) { return __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w); };
    int mine = 0, total;
    for (long long q = a; q < b; q += 128) {
        int4 w[4];
        load(w, q);
#pragma unroll
        for (int u = 0; u < 4; ++u) mine += dead_in(w[u]);
    }
    // dead ones before the warp's (its lanes' counts stand in order)
    int rank = __shfl_sync(0xffffffffu, vx_block_scan<NW>(mine, total), 0);
    if (total == 0) return 0;
    const long long m = n0 - total;
    if (!apply) {
        for (long long q = a + lane; q < b; q += 32) b4[q] = make_int4(0, 0, 0, 0);
    } else {
        const bool many = total > limit;
        if (many || __any_sync(0xffffffffu, mine != 0))
            for (long long q = a; q < b; q += 128) {
                int4 w4[4];
                load(w4, q);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int k = dead_in(w4[u]);
                    const long long q4 = q + u * 32 + lane;
                    if (!__any_sync(0xffffffffu, k != 0)) {
                        if (many && q4 < b) c.pre[q4] = rank;
                        continue;
                    }
                    int inc = k;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, inc, o);
                        if (lane >= o) inc += t;
                    }
                    int h = rank + inc - k;
                    rank += __shfl_sync(0xffffffffu, inc, 31);
                    if (many) {
                        if (q4 < b) c.pre[q4] = h;
                        continue;
                    }
                    const unsigned w[4] = {(unsigned)w4[u].x, (unsigned)w4[u].y, (unsigned)w4[u].z, (unsigned)w4[u].w};
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        for (unsigned x = w[s]; x; x &= x - 1) {
                            const long long p = q4 * 128 + s * 32 + __ffs(x) - 1;
                            if (p < m) c.hole_pos[h++] = (int)p;
                        }
                }
            }
        if (many) {
            if (tid == 0) {
                S->cmp_many = 1;
                S->c_n0 = n0;
                S->c_m = m;
            }
            return total;
        }
        // the tail [m, n0): live ones fill the holes, from the top
        const long long w0 = m >> 5, nt = ((n0 - 1) >> 5) - w0 + 1, per = (nt + NW - 1) / NW;
        const long long wa = w0 + min(nt, warp * per), wb = w0 + min(nt, (warp + 1) * per);
        auto live_of = [&](long long w, unsigned dead) {
            unsigned x = ~dead;
            if (w == w0) x &= ~0u << (m & 31);
            if (w == (n0 - 1) >> 5) x &= ~0u >> (31 - ((n0 - 1) & 31));
            return x;
        };
        int k = 0, H;
        for (long long w = wa + lane; w < wb; w += 32) k += __popc(live_of(w, __ldcg(&c.bits[w])));
        // a warp's live ones before it (its lanes' counts stand in order)
        const int before = vx_block_scan<NW>(k, H);
        int run = __shfl_sync(0xffffffffu, before, 0);
        for (long long w = wa; w < wb; ++w) {
            const unsigned dead = __ldcg(&c.bits[w]), next = __ldcg(&c.bits[w + 1]), live = live_of(w, dead);
            const long long p = w * 32 + lane;
            if (p >= m && p < n0) {
                const bool lv = live >> lane & 1;
                const int r = run + __popc(live & ((1u << lane) - 1u));
                if (lv) c.hole_src[H - 1 - r] = (int)p;
                const bool next_live = p + 1 < n0 && !((lane < 31 ? dead >> (lane + 1) : next) & 1u);
                const int grp = H - r - (lv ? 1 : 0);   // live elements in (p, n0)
                c.tail_src[p - m] = p == n0 - 1 || next_live ? (grp < H ? -(grp + 1) : (int)m) : (int)(p + 1);
            }
            run += __popc(live);
        }
        __syncthreads();
        for (int e = tid; e < H; e += T) c.bits[c.hole_pos[e] >> 5] = 0;
        for (long long w = w0 + tid; w < w0 + nt; w += T) c.bits[w] = 0;
        const long long moves = H + (long long)total;
        vx_cmp_gather<4>(v, c, H, moves, tid, T);
        __syncthreads();
        vx_cmp_scatter<4>(v, c, m, H, moves, tid, T, slot, rec_i);
        if (tid == 0) S->n = m;
    }
    return total;
}

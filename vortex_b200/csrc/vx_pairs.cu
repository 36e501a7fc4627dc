// vx_pairs.cu — direct pair sums: convective (Biot-Savart) velocity with the
// mean distance to the 3 nearest particles, vortex-vortex diffusive velocity,
// and the probe velocity.
//
// Reference: shared_Kernel src/kernel.cu:875-983, diffusion_Kernel
// src/kernel.cu:985-1029, velocity_control_Kernel src/kernel.cu:1434-1475.
//
// Work decomposition: a target tile (2 or 4 targets per thread, 256 threads)
// x a source chunk is one work item; persistent CTAs walk the items, which
// fill them a whole number of times.  Sources are staged through shared
// memory 256 at a time and read as warp-wide broadcasts.  Each item writes partial sums; a combine kernel adds the chunks in a fixed
// order, so results are deterministic for a given split.
//
// Precision: FP64 (plain form) computes every pair in double and adds each
// 256-source tile's sum to the chunk's.  FP32 (bulk
// form) computes pairs in float and accumulates each 256-source tile in
// float, adding tile sums into a double accumulator (blocked compensation).
#include <algorithm>

#include "vx_internal.cuh"

constexpr int PT = 256;       // threads per block = sources per shared tile
// Resident blocks per SM the pair kernels are compiled for (at most 128
// registers a thread; the FP32 sum without the 3 nearest needs fewer).
constexpr int PAIR_MINB = 2;
constexpr int PROBE32_MINB = 4;

// Source split of the pair kernels: K source chunks; the partial sums of
// target i and chunk sc sit at part[(sc nout + q) tstride + i], tstride =
// cap / (nout K).  K > 0: the caller's split (probe points); K == 0: from the
// body's own count on the device (vx_pair_split), so a step's sums never
// depend on the host's running bound.
struct VxSplit {
    long long cap;
    int K, slots, tile, nout, rounds;
};
__device__ __forceinline__ void vx_split_of(const VxScalars *S, const VxSplit &sp, int &K, long long &tstride) {
    K = sp.K > 0 ? sp.K : vx_pair_split(S->n, S->n, sp.tile, sp.slots, sp.rounds);
    tstride = sp.cap / ((long long)sp.nout * K);
}
// Sources of one chunk: equal chunks, rounded up to whole warps of sources.
__device__ __forceinline__ long long vx_split_chunk(long long sources, int K) {
    return (vx_ceil_div(sources, (long long)K) + 31) / 32 * 32;
}


// ---------------------------------------------------------------------------
// Packed FP32 sources for the bulk form: (x, y, G, 0), G masked to 0 beyond n.
VX_DEVK void k_pack32_body(VxBlkB<0, 0> vb, const VxView &v, const VxScalars *S, float4 *src, long long upto) {
    const long long n = S->n;
    const long long s = vx_round32(n);
    for (long long j = vb.x * (long long)blockDim.x + threadIdx.x; j < s;
         j += (long long)vb.n * blockDim.x) {
        if (j >= upto) break;
        src[j] = make_float4((float)v.x[j * v.ps], (float)v.y[j * v.ps],
                             j < n ? (float)v.g[j * v.ps] : 0.0f, 0.0f);
    }
}
__global__ void k_pack32(VxView v, const VxScalars *S, float4 *src, long long upto) {
    VX_PDL_WAIT();
    k_pack32_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, v, S, src, upto);
}

// Sources of one shared tile.
template <typename T>
struct SrcTile {
    T x[PT], y[PT], g[PT];
};

template <typename T>
__device__ __forceinline__ void load_src(SrcTile<T> &t, const VxView &v, const float4 *src32,
                                         long long j, long long jend, long long nvel) {
    if (j < jend) {
        if (src32) {
            float4 q = src32[j];
            t.x[threadIdx.x] = (T)q.x; t.y[threadIdx.x] = (T)q.y; t.g[threadIdx.x] = (T)q.z;
        } else {
            t.x[threadIdx.x] = (T)v.x[j * v.ps];
            t.y[threadIdx.x] = (T)v.y[j * v.ps];
            t.g[threadIdx.x] = j < nvel ? (T)v.g[j * v.ps] : (T)0;
        }
    }
}

// 1/x and 1/sqrt(x) in FP64 from the hardware's approximations (about 20
// bits) and one third-order step each: with e the residual of the seed y,
// 1/x = y (1 + e + e^2), 1/sqrt(x) = y (1 + e/2 + 3 e^2/8), the next terms
// below 2^-60.  3 and 5 FP64 instructions, within an ulp or so; the correctly
// rounded division and square root take about 8 and 10.
__device__ __forceinline__ double vx_rcp64(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double vx_rsqrt64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(e * y, fma(e, 0.375, 0.5), y);
}
__device__ __forceinline__ unsigned vx_hi(double v) { return (unsigned)__double2hiint(v); }

// ---------------------------------------------------------------------------
// Plain-form Biot-Savart (+ 3 nearest when NN3), FP64.  Targets: particles
// (nt < 0 -> n) or probe points (tx/ty with stride tstr).  Partials:
// [sc][NOUT][tstride].
//
// Bound by issue: 12 FP64 instructions a pair (two cycles a warp each, three
// with three register operands) and about as many others.  The 3-nearest
// test compares the high words as integers, off the FP64 pipe, and only a
// warp with a candidate takes the exact FP64 insertion (a vote and a branch;
// predicated, it ran for every pair); with the sources in chunks every chunk
// starts its own three, so the chunks are as few as fill the GPU
// (vx_pair_split).  16 365 vortices: 757 -> 443 us with the correctly rounded
// division, 37 chunks and the predicated insertion before; 60 000: 4.2 ms.
constexpr int BS64_TPT = 2;
template <bool NN3>
VX_DEVK void k_bs64_partial_body(VxBlkB<PT, PAIR_MINB> vb, const VxParams &p, const VxView &v, const VxScalars *S,
                                 const double *tx, const double *ty, long long tstr, long long nt_in, double *part,
                                 VxSplit sp) {
    int K;
    long long tstride;
    vx_split_of(S, sp, K, tstride);
    constexpr int TPT = BS64_TPT;
    constexpr int NOUT = NN3 ? 5 : 2;
    __shared__ SrcTile<double> st;
    const long long n = S->n;
    const long long nt = nt_in < 0 ? n : nt_in;
    const long long srange = NN3 ? vx_round32(n) : n;
    const long long tile = (long long)PT * TPT;
    const long long tiles = vx_ceil_div(nt, tile);
    const long long cs = vx_split_chunk(srange, K);
    const long long items = tiles * K;
    const double eps2 = p.eps2;
    for (long long it = vb.x; it < items; it += vb.n) {
        const long long tt = it % tiles, sc = it / tiles;
        double ax[TPT], ay[TPT], sx[TPT], sy[TPT], d1[TPT], d2[TPT], d3[TPT];
        int ti[TPT];
#pragma unroll
        for (int k = 0; k < TPT; ++k) {
            ti[k] = (int)(tt * tile) + k * PT + threadIdx.x;
            const long long i = ti[k] < nt ? ti[k] : 0;
            ax[k] = tx[i * tstr];
            ay[k] = ty[i * tstr];
            sx[k] = sy[k] = 0.0;
            d1[k] = d2[k] = d3[k] = 1e5;
        }
        const long long j0 = min(sc * cs, srange), j1 = min(srange, j0 + cs);
        for (long long jt = j0; jt < j1; jt += PT) {
            __syncthreads();
            load_src<double>(st, v, nullptr, jt + threadIdx.x, j1, n);
            __syncthreads();
            const int cnt = (int)min((long long)PT, j1 - jt);
            double px[TPT], py[TPT];   // the tile's sums
#pragma unroll
            for (int k = 0; k < TPT; ++k) px[k] = py[k] = 0.0;
            int self[TPT];
#pragma unroll
            for (int k = 0; k < TPT; ++k) self[k] = ti[k] - (int)jt;
#pragma unroll 2
            for (int q = 0; q < cnt; ++q) {
                const double bx = st.x[q], by = st.y[q], bg = st.g[q];
                double dx[TPT], dy[TPT], r2[TPT];
                bool near = false;
#pragma unroll
                for (int k = 0; k < TPT; ++k) {
                    dx[k] = ax[k] - bx;
                    dy[k] = ay[k] - by;
                    r2[k] = fma(dx[k], dx[k], dy[k] * dy[k]);
                    near = near || vx_hi(r2[k]) <= vx_hi(d3[k]);
                }
                if (NN3 && __any_sync(0xffffffffu, near)) {   // a branch: predicated, it would run for every pair
#pragma unroll
                    for (int k = 0; k < TPT; ++k)
                        vx_nn3_insert<double>(d1[k], d2[k], d3[k], q == self[k] ? INFINITY : r2[k]);
                }
#pragma unroll
                for (int k = 0; k < TPT; ++k) {
                    const double rm = fmax(r2[k], eps2);
                    // an infinite r2 (a pair out of range) weighs 0, as 1/inf does
                    const double m = bg * vx_rcp64(__hiloint2double(min(__double2hiint(rm), 0x7fefffff), __double2loint(rm)));
                    py[k] = fma(m, dx[k], py[k]);
                    px[k] = fma(-m, dy[k], px[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < TPT; ++k) { sx[k] += px[k]; sy[k] += py[k]; }
        }
#pragma unroll
        for (int k = 0; k < TPT; ++k) {
            if (ti[k] < nt) {
                double *o = part + (long long)sc * NOUT * tstride + ti[k];
                o[0] = sx[k];
                o[tstride] = sy[k];
                if (NN3) {
                    o[2 * tstride] = d1[k];
                    o[3 * tstride] = d2[k];
                    o[4 * tstride] = d3[k];
                }
            }
        }
    }
}
template <bool NN3>
__global__ void __launch_bounds__(PT, PAIR_MINB) k_bs64_partial(VxParams p, VxView v, const VxScalars *S,
                                                                const double *tx, const double *ty, long long tstr,
                                                                long long nt_in, double *part, VxSplit sp) {
    VX_PDL_WAIT();
    k_bs64_partial_body<NN3>(VxBlkB<PT, PAIR_MINB>{blockIdx.x, gridDim.x}, p, v, S, tx, ty, tstr, nt_in, part, sp);
}

// ---------------------------------------------------------------------------
// Bulk-form Biot-Savart + 3 nearest, FP32.  Same decomposition as above, with
// the inner loop cut to the arithmetic: sources come from shared memory as
// one float4 broadcast each, the loop runs unrolled over full tiles, the
// reciprocal is the hardware approximation (rcp.approx, 1 ulp), and the
// self pair is excluded only in the one tile per target that can contain it
// (a uniform branch per tile), so the hot loop has no index compare.
__device__ __forceinline__ float vx_rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

constexpr int BS32_TPT = 4;

template <bool CHECK_SELF>
__device__ __forceinline__ void bs32_tile(const float4 *sm, int cnt, int jbase, const int *ti,
                                          const float *ax, const float *ay, float eps2, float *sx,
                                          float *sy, float *d1, float *d2, float *d3) {
#pragma unroll 4
    for (int q = 0; q < cnt; ++q) {
        const float4 s = sm[q];
#pragma unroll
        for (int k = 0; k < BS32_TPT; ++k) {
            const float dx = ax[k] - s.x, dy = ay[k] - s.y;
            const float r2 = fmaf(dx, dx, dy * dy);
            if (r2 < d3[k] && (!CHECK_SELF || jbase + q != ti[k])) {
                d3[k] = r2;
                float t = fminf(d3[k], d2[k]); d3[k] = fmaxf(d3[k], d2[k]); d2[k] = t;
                t = fminf(d1[k], d2[k]); d2[k] = fmaxf(d1[k], d2[k]); d1[k] = t;
            }
            const float m = s.z * vx_rcp_approx(fmaxf(r2, eps2));
            sy[k] = fmaf(m, dx, sy[k]);
            sx[k] = fmaf(-m, dy, sx[k]);
        }
    }
}

VX_DEVK void k_bs32_partial_body(VxBlkB<PT, PAIR_MINB> vb, const VxParams &p, const VxScalars *S, const float4 *src32,
                                 const double *tx, const double *ty, long long tstr, double *part, VxSplit sp) {
    int K;
    long long tstride;
    vx_split_of(S, sp, K, tstride);
    __shared__ float4 sm[PT];
    const long long n = S->n;
    const long long srange = vx_round32(n);
    const long long tile = (long long)PT * BS32_TPT;
    const long long tiles = vx_ceil_div(n, tile);
    const long long cs = vx_split_chunk(srange, K);
    const long long items = tiles * K;
    const float eps2 = (float)p.eps2;
    for (long long it = vb.x; it < items; it += vb.n) {
        const long long tt = it % tiles, sc = it / tiles;
        const long long tlo = tt * tile, thi = min(n, tlo + tile);
        float ax[BS32_TPT], ay[BS32_TPT], d1[BS32_TPT], d2[BS32_TPT], d3[BS32_TPT];
        int ti[BS32_TPT];
        double vxa[BS32_TPT], vya[BS32_TPT];
#pragma unroll
        for (int k = 0; k < BS32_TPT; ++k) {
            const long long t = tlo + (long long)k * PT + threadIdx.x;
            ti[k] = (int)t;
            const long long i = t < n ? t : 0;
            ax[k] = (float)tx[i * tstr];
            ay[k] = (float)ty[i * tstr];
            vxa[k] = 0.0; vya[k] = 0.0;
            d1[k] = d2[k] = d3[k] = 1e5f;
        }
        const long long j0 = min(sc * cs, srange), j1 = min(srange, j0 + cs);
        for (long long jt = j0; jt < j1; jt += PT) {
            __syncthreads();
            if (jt + threadIdx.x < j1) sm[threadIdx.x] = src32[jt + threadIdx.x];
            __syncthreads();
            const int cnt = (int)min((long long)PT, j1 - jt);
            float sx[BS32_TPT], sy[BS32_TPT];
#pragma unroll
            for (int k = 0; k < BS32_TPT; ++k) { sx[k] = 0.0f; sy[k] = 0.0f; }
            const bool self = jt < thi && jt + cnt > tlo;   // uniform per block
            if (self)
                bs32_tile<true>(sm, cnt, (int)jt, ti, ax, ay, eps2, sx, sy, d1, d2, d3);
            else
                bs32_tile<false>(sm, cnt, (int)jt, ti, ax, ay, eps2, sx, sy, d1, d2, d3);
#pragma unroll
            for (int k = 0; k < BS32_TPT; ++k) { vxa[k] += (double)sx[k]; vya[k] += (double)sy[k]; }
        }
#pragma unroll
        for (int k = 0; k < BS32_TPT; ++k) {
            if (ti[k] < n) {
                double *o = part + (long long)sc * 5 * tstride + ti[k];
                o[0] = vxa[k];
                o[tstride] = vya[k];
                o[2 * tstride] = (double)d1[k];
                o[3 * tstride] = (double)d2[k];
                o[4 * tstride] = (double)d3[k];
            }
        }
    }
}
__global__ void __launch_bounds__(PT, PAIR_MINB) k_bs32_partial(VxParams p, const VxScalars *S, const float4 *src32,
                                                                const double *tx, const double *ty, long long tstr,
                                                                double *part, VxSplit sp) {
    VX_PDL_WAIT();
    k_bs32_partial_body(VxBlkB<PT, PAIR_MINB>{blockIdx.x, gridDim.x}, p, S, src32, tx, ty, tstr, part, sp);
}

// Bulk-form probe points: the same sums without the 3 nearest, two targets in
// one packed FP32 operation (sources staged as pairs of equal values), so the
// special-function pipe's reciprocal a pair is what bounds it (16 a clock and
// SM) and not issue.  A probe call of 4096 points over 1e6 vortices: 1.50 ms
// with one target an operation -> 1.30.  Four targets a thread, two where all
// points fit a tile of 512.
template <int PROBE_TPT>
VX_DEVK void k_probe32_partial_body(VxBlkB<PT, PROBE32_MINB> vb, const VxParams &p, const VxScalars *S,
                                    const float4 *src32, const double *tx, const double *ty, long long tstr,
                                    long long nt, double *part, VxSplit sp) {
    int K;
    long long tstride;
    vx_split_of(S, sp, K, tstride);
    __shared__ ulonglong2 sxy[PT];   // (x, x), (y, y)
    __shared__ f2 sg[PT];            // (G, G)
    const long long n = S->n;
    const long long tile = (long long)PT * PROBE_TPT;
    const long long tiles = vx_ceil_div(nt, tile);
    const long long cs = vx_split_chunk(n, K);
    const long long items = tiles * K;
    const float eps2 = (float)p.eps2;
    for (long long it = vb.x; it < items; it += vb.n) {
        const long long tt = it % tiles, sc = it / tiles;
        f2 ax[PROBE_TPT / 2], ay[PROBE_TPT / 2];
        double vxa[PROBE_TPT], vya[PROBE_TPT];
#pragma unroll
        for (int k = 0; k < PROBE_TPT; k += 2) {
            float x[2], y[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const long long t = tt * tile + (long long)(k + h) * PT + threadIdx.x, i = t < nt ? t : 0;
                x[h] = (float)tx[i * tstr];
                y[h] = (float)ty[i * tstr];
                vxa[k + h] = vya[k + h] = 0.0;
            }
            ax[k / 2] = f2_pack(x[0], x[1]);
            ay[k / 2] = f2_pack(y[0], y[1]);
        }
        const long long j0 = min(sc * cs, n), j1 = min(n, j0 + cs);
        for (long long jt = j0; jt < j1; jt += PT) {
            __syncthreads();
            if (jt + threadIdx.x < j1) {
                const float4 q = src32[jt + threadIdx.x];
                sxy[threadIdx.x] = make_ulonglong2(f2_pack(q.x, q.x), f2_pack(q.y, q.y));
                sg[threadIdx.x] = f2_pack(q.z, q.z);
            }
            __syncthreads();
            const int cnt = (int)min((long long)PT, j1 - jt);
            f2 sx[PROBE_TPT / 2], sy[PROBE_TPT / 2];
#pragma unroll
            for (int k = 0; k < PROBE_TPT / 2; ++k) sx[k] = sy[k] = 0ull;   // +0.0f in both halves
#pragma unroll 4
            for (int q = 0; q < cnt; ++q) {
                const ulonglong2 c = sxy[q];
                const f2 g = sg[q];
#pragma unroll
                for (int k = 0; k < PROBE_TPT / 2; ++k) {
                    const f2 dx = f2_sub(ax[k], c.x), dy = f2_sub(ay[k], c.y);
                    float ra, rb;
                    f2_unpack(f2_fma(dx, dx, f2_mul(dy, dy)), ra, rb);
                    const f2 m = f2_mul(g, f2_pack(vx_rcp_approx(fmaxf(ra, eps2)), vx_rcp_approx(fmaxf(rb, eps2))));
                    sy[k] = f2_fma(m, dx, sy[k]);
                    sx[k] = f2_fma(m, dy, sx[k]);   // sum of +m dy: negated below
                }
            }
#pragma unroll
            for (int k = 0; k < PROBE_TPT / 2; ++k) {
                float a, b;
                f2_unpack(sx[k], a, b); vxa[2 * k] -= (double)a; vxa[2 * k + 1] -= (double)b;
                f2_unpack(sy[k], a, b); vya[2 * k] += (double)a; vya[2 * k + 1] += (double)b;
            }
        }
#pragma unroll
        for (int k = 0; k < PROBE_TPT; ++k) {
            const long long t = tt * tile + (long long)k * PT + threadIdx.x;
            if (t < nt) {
                double *o = part + (long long)sc * 2 * tstride + t;
                o[0] = vxa[k];
                o[tstride] = vya[k];
            }
        }
    }
}
template <int TPT>
__global__ void __launch_bounds__(PT, PROBE32_MINB) k_probe32_partial(VxParams p, const VxScalars *S,
                                                                      const float4 *src32, const double *tx,
                                                                      const double *ty, long long tstr, long long nt,
                                                                      double *part, VxSplit sp) {
    VX_PDL_WAIT();
    k_probe32_partial_body<TPT>(VxBlkB<PT, PROBE32_MINB>{blockIdx.x, gridDim.x}, p, S, src32, tx, ty, tstr, nt, part, sp);
}

// Combine: V = sum/(2 pi) + V_inf, d = mean of the 3 nearest distances.  A
// block takes 64 targets, its four slices of 64 threads a quarter of the
// chunks each (every fourth), the slices' sums and nearest three added in
// order.
constexpr int CMB_T = 64, CMB_S = 4;
template <bool FP32>
VX_DEVK void k_bs_combine_body(VxBlkB<CMB_T * CMB_S, 0> vb, const VxView &v, const VxScalars *S, const double *part,
                               VxSplit sp) {
    __shared__ double sh[CMB_S - 1][5][CMB_T];
    int K;
    long long tstride;
    vx_split_of(S, sp, K, tstride);
    const long long n = S->n;
    const int col = threadIdx.x % CMB_T, slice = threadIdx.x / CMB_T;
    for (long long b = vb.x; b * CMB_T < n; b += vb.n) {
        const long long i = b * CMB_T + col;
        double sx = 0.0, sy = 0.0;
        double d1 = 1e5, d2 = 1e5, d3 = 1e5;
        if (i < n) {
#pragma unroll 2
            for (int sc = slice; sc < K; sc += CMB_S) {
                const double *o = part + (long long)sc * 5 * tstride + i;
                const double u = o[0], w = o[tstride], e1 = o[2 * tstride], e2 = o[3 * tstride], e3 = o[4 * tstride];
                sx += u;
                sy += w;
                vx_nn3_insert<double>(d1, d2, d3, e1);
                vx_nn3_insert<double>(d1, d2, d3, e2);
                vx_nn3_insert<double>(d1, d2, d3, e3);
            }
        }
        if (slice > 0) {
            double (*o)[CMB_T] = sh[slice - 1];
            o[0][col] = sx; o[1][col] = sy; o[2][col] = d1; o[3][col] = d2; o[4][col] = d3;
        }
        __syncthreads();
        if (slice == 0 && i < n) {
            for (int q = 0; q < CMB_S - 1; ++q) {
                sx += sh[q][0][col];
                sy += sh[q][1][col];
                for (int e = 2; e < 5; ++e) vx_nn3_insert<double>(d1, d2, d3, sh[q][e][col]);
            }
            if (FP32)
                v.d[i] = (double)((sqrtf((float)d1) + sqrtf((float)d2) + sqrtf((float)d3)) / 3);
            else
                v.d[i] = (sqrt(d1) + sqrt(d2) + sqrt(d3)) / 3;
            v.vx[i * v.vs] = sx / VX_TWO_PI + S->vinf[0];
            v.vy[i * v.vs] = sy / VX_TWO_PI + S->vinf[1];
        }
        __syncthreads();
    }
}
template <bool FP32>
__global__ void __launch_bounds__(CMB_T * CMB_S) k_bs_combine(VxView v, const VxScalars *S, const double *part,
                                                              VxSplit sp) {
    VX_PDL_WAIT();
    k_bs_combine_body<FP32>(VxBlkB<CMB_T * CMB_S, 0>{blockIdx.x, gridDim.x}, v, S, part, sp);
}

// 32 points a block, its eight warps an eighth of the chunks each.
VX_DEVK void k_probe_combine_body(VxBlkB<256, 0> vb, const VxScalars *S, const double *part, VxSplit sp,
                                  long long np, double *ovx, double *ovy, long long ostride) {
    __shared__ double sh[2][8][32];
    int K;
    long long tstride;
    vx_split_of(S, sp, K, tstride);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long b = vb.x; b * 32 < np; b += vb.n) {
        const long long i = b * 32 + lane;
        double sx = 0.0, sy = 0.0;
        if (i < np) {
#pragma unroll 8
            for (int sc = warp; sc < K; sc += 8) {
                const double *o = part + (long long)sc * 2 * tstride + i;
                sx += o[0];
                sy += o[tstride];
            }
        }
        sh[0][warp][lane] = sx;
        sh[1][warp][lane] = sy;
        __syncthreads();
        if (warp < 2 && i < np) {
            double t = 0.0;
            for (int w = 0; w < 8; ++w) t += sh[warp][w][lane];
            (warp ? ovy : ovx)[i * ostride] = t / VX_TWO_PI + S->vinf[warp];
        }
        __syncthreads();
    }
}
__global__ void __launch_bounds__(256) k_probe_combine(const VxScalars *S, const double *part, VxSplit sp,
                                                       long long np, double *ovx, double *ovy, long long ostride) {
    VX_PDL_WAIT();
    k_probe_combine_body(VxBlkB<256, 0>{blockIdx.x, gridDim.x}, S, part, sp, np, ovx, ovy, ostride);
}

// ---------------------------------------------------------------------------
// Vortex-vortex diffusion (src/kernel.cu:985-1029).  Partials [sc][3][tstride].
// Plain form, FP64: 1/r from vx_rsqrt64, r = r2 (1/r) with one correction,
// and e^(-r/d) by the table method (P.T.P. Tang, Table-driven implementation
// of the exponential function in IEEE floating-point arithmetic, 1989) from
// y = -(32 / ln2) r / d: with n the integer nearest to y and f = y - n
// (exact), e^(-r/d) = 2^(n / 32) 2^(f / 32), the second factor by its Taylor
// polynomial to f^6 (remainder below 2^-57).  Lane j of a warp holds 2^(j /
// 32) and a lane takes its entry by shuffle (random reads of a table in
// shared memory conflict).  28 FP64 instructions a pair, which bound it (62 %
// of the pipe's cycles; the library's square root, division and exp took
// about 50): 16 365 vortices 1133 -> 749 us, 60 000: 8.8 ms.
constexpr double EXP_SCALE = 46.16624130844683;   // 32 / ln2
__device__ const double c_exp_table[32] = {
    0x1.0000000000000p+0, 0x1.059b0d3158574p+0, 0x1.0b5586cf9890fp+0, 0x1.11301d0125b51p+0,
    0x1.172b83c7d517bp+0, 0x1.1d4873168b9aap+0, 0x1.2387a6e756238p+0, 0x1.29e9df51fdee1p+0,
    0x1.306fe0a31b715p+0, 0x1.371a7373aa9cbp+0, 0x1.3dea64c123422p+0, 0x1.44e086061892dp+0,
    0x1.4bfdad5362a27p+0, 0x1.5342b569d4f82p+0, 0x1.5ab07dd485429p+0, 0x1.6247eb03a5585p+0,
    0x1.6a09e667f3bcdp+0, 0x1.71f75e8ec5f74p+0, 0x1.7a11473eb0187p+0, 0x1.82589994cce13p+0,
    0x1.8ace5422aa0dbp+0, 0x1.93737b0cdc5e5p+0, 0x1.9c49182a3f090p+0, 0x1.a5503b23e255dp+0,
    0x1.ae89f995ad3adp+0, 0x1.b7f76f2fb5e47p+0, 0x1.c199bdd85529cp+0, 0x1.cb720dcef9069p+0,
    0x1.d5818dcfba487p+0, 0x1.dfc97337b9b5fp+0, 0x1.ea4afa2a490dap+0, 0x1.f50765b6e4540p+0,
};
__device__ __forceinline__ double vx_exp2_32(double y, double tab) {   // 2^(y / 32), -32 1021 <= y <= 0, by whole warps
    const double MAGIC = 6755399441055744.0;   // 1.5 2^52: the sum's low word is the rounded integer
    const double t = y + MAGIC;
    const double f = y - (t - MAGIC);
    const int n = __double2loint(t);
    const double w = __shfl_sync(0xffffffffu, tab, n & 31);
    double q = fma(f, 1.4345655584131934e-13, 3.973709984549416e-11);
    q = fma(q, f, 9.172562701824643e-09);
    q = fma(q, f, 1.693850972437182e-06);
    q = fma(q, f, 0.0002345961982022468);
    q = fma(q, f, 0.02166084939249829);
    const double e = fma(w * f, q, w);
    return __hiloint2double(__double2hiint(e) + ((n >> 5) << 20), __double2loint(e));
}

VX_DEVK void k_diff64_partial_body(VxBlkB<PT, PAIR_MINB> vb, const VxParams &p, const VxView &v,
                                   const VxScalars *S, double *part, VxSplit sp) {
    int K;
    long long tstride;
    vx_split_of(S, sp, K, tstride);
    constexpr int TPT = BS64_TPT;
    __shared__ SrcTile<double> st;
    const double tab = c_exp_table[threadIdx.x & 31];
    const long long n = S->n;
    const long long tile = (long long)PT * TPT;
    const long long tiles = vx_ceil_div(n, tile);
    const long long cs = vx_split_chunk(n, K);
    const long long items = tiles * K;
    const long long thr2 = __double_as_longlong((0.001 * p.eps) * (0.001 * p.eps));
    const int thr_hi = (int)(thr2 >> 32);
    for (long long it = vb.x; it < items; it += vb.n) {
        const long long tt = it % tiles, sc = it / tiles;
        double ax[TPT], ay[TPT], ndd[TPT], a2x[TPT], a2y[TPT], a1[TPT];
        int ti[TPT];
#pragma unroll
        for (int k = 0; k < TPT; ++k) {
            ti[k] = (int)(tt * tile) + k * PT + threadIdx.x;
            const long long i = ti[k] < n ? ti[k] : 0;
            ax[k] = v.x[i * v.ps];
            ay[k] = v.y[i * v.ps];
            ndd[k] = -EXP_SCALE / v.d[i];
            a2x[k] = a2y[k] = a1[k] = 0.0;
        }
        const long long j0 = min(sc * cs, n), j1 = min(n, j0 + cs);
        for (long long jt = j0; jt < j1; jt += PT) {
            __syncthreads();
            load_src<double>(st, v, nullptr, jt + threadIdx.x, j1, n);
            __syncthreads();
            const int cnt = (int)min((long long)PT, j1 - jt);
            double s2x[TPT], s2y[TPT], s1[TPT];   // the tile's sums
#pragma unroll
            for (int k = 0; k < TPT; ++k) s2x[k] = s2y[k] = s1[k] = 0.0;
#pragma unroll 1
            for (int q = 0; q < cnt; ++q) {
                const double bx = st.x[q], by = st.y[q], bg = st.g[q];
#pragma unroll
                for (int k = 0; k < TPT; ++k) {
                    const double dx = ax[k] - bx, dy = ay[k] - by;
                    const double r2 = fma(dx, dx, dy * dy);
                    // 1/r stays finite, above 0, where the pair is left out below
                    const double rc = __hiloint2double(min(max(__double2hiint(r2), thr_hi), 0x7fefffff),
                                                       __double2loint(r2));
                    const double rd = vx_rsqrt64(rc);
                    double dist = rc * rd;
                    dist = fma(fma(-dist, dist, rc), 0.5 * rd, dist);
                    const double y = dist * ndd[k];
                    // not the pair itself (r > 0.001 eps, compared as integers)
                    // nor one whose exponential is below the normal range
                    // (y <= -32 1021, its high word)
                    const bool use = __double_as_longlong(r2) > thr2 && (vx_hi(y) ^ 0x80000000u) < 0x40dfe800u;
                    const double e = vx_exp2_32(y, tab);
                    const double ge = use ? bg * e : 0.0;
                    const double me = ge * rd;
                    s2x[k] = fma(-me, dx, s2x[k]);
                    s2y[k] = fma(-me, dy, s2y[k]);
                    s1[k] += ge;
                }
            }
#pragma unroll
            for (int k = 0; k < TPT; ++k) { a2x[k] += s2x[k]; a2y[k] += s2y[k]; a1[k] += s1[k]; }
        }
#pragma unroll
        for (int k = 0; k < TPT; ++k) {
            if (ti[k] < n) {
                double *o = part + (long long)sc * 3 * tstride + ti[k];
                o[0] = a2x[k];
                o[tstride] = a2y[k];
                o[2 * tstride] = a1[k];
            }
        }
    }
}
__global__ void __launch_bounds__(PT, PAIR_MINB) k_diff64_partial(VxParams p, VxView v, const VxScalars *S,
                                                                    double *part, VxSplit sp) {
    VX_PDL_WAIT();
    k_diff64_partial_body(VxBlkB<PT, PAIR_MINB>{blockIdx.x, gridDim.x}, p, v, S, part, sp);
}

// FP32 without a cut-off (diff_cutoff <= 0): direct sums, tile sums in FP32
// carried in FP64.
VX_DEVK void k_diff32_partial_body(VxBlkB<PT, PAIR_MINB> vb, const VxParams &p, const VxView &v, const VxScalars *S,
                                   const float4 *src32, double *part, VxSplit sp) {
    int K;
    long long tstride;
    vx_split_of(S, sp, K, tstride);
    constexpr int TPT = 4;
    __shared__ SrcTile<float> st;
    const long long n = S->n;
    const long long tile = (long long)PT * TPT;
    const long long tiles = vx_ceil_div(n, tile);
    const long long cs = vx_split_chunk(n, K);
    const long long items = tiles * K;
    const float thr = (float)(0.001 * p.eps);
    const float thr2 = thr * thr;
    for (long long it = vb.x; it < items; it += vb.n) {
        const long long tt = it % tiles, sc = it / tiles;
        float ax[TPT], ay[TPT], ndd[TPT];
        long long ti[TPT];
        double a2x[TPT], a2y[TPT], a1[TPT];
#pragma unroll
        for (int k = 0; k < TPT; ++k) {
            ti[k] = tt * tile + (long long)k * PT + threadIdx.x;
            const long long i = ti[k] < n ? ti[k] : 0;
            ax[k] = (float)v.x[i * v.ps];
            ay[k] = (float)v.y[i * v.ps];
            ndd[k] = -1.0f / (float)v.d[i];
            a2x[k] = a2y[k] = a1[k] = 0.0;
        }
        const long long j0 = min(sc * cs, n), j1 = min(n, j0 + cs);
        for (long long jt = j0; jt < j1; jt += PT) {
            __syncthreads();
            load_src<float>(st, v, src32, jt + threadIdx.x, j1, n);
            __syncthreads();
            const int cnt = (int)min((long long)PT, j1 - jt);
            float s2x[TPT], s2y[TPT], s1[TPT];
#pragma unroll
            for (int k = 0; k < TPT; ++k) { s2x[k] = 0; s2y[k] = 0; s1[k] = 0; }
            for (int q = 0; q < cnt; ++q) {
                const float bx = st.x[q], by = st.y[q], bg = st.g[q];
#pragma unroll
                for (int k = 0; k < TPT; ++k) {
                    const float dx = ax[k] - bx, dy = ay[k] - by;
                    const float r2 = fmaf(dx, dx, dy * dy);
                    const float rd = rsqrtf(r2);
                    const float e = __expf(r2 * rd * ndd[k]);
                    const bool use = r2 > thr2;
                    const float ge = use ? bg * e : 0.0f;
                    const float me = use ? ge * rd : 0.0f;   // r = 0 would give 0 * inf
                    s2x[k] = fmaf(-me, dx, s2x[k]);
                    s2y[k] = fmaf(-me, dy, s2y[k]);
                    s1[k] += ge;
                }
            }
#pragma unroll
            for (int k = 0; k < TPT; ++k) {
                a2x[k] += (double)s2x[k]; a2y[k] += (double)s2y[k]; a1[k] += (double)s1[k];
            }
        }
#pragma unroll
        for (int k = 0; k < TPT; ++k) {
            if (ti[k] < n) {
                double *o = part + (long long)sc * 3 * tstride + ti[k];
                o[0] = a2x[k];
                o[tstride] = a2y[k];
                o[2 * tstride] = a1[k];
            }
        }
    }
}
__global__ void __launch_bounds__(PT, PAIR_MINB) k_diff32_partial(VxParams p, VxView v, const VxScalars *S, const float4 *src32,
                                                       double *part, VxSplit sp) {
    VX_PDL_WAIT();
    k_diff32_partial_body(VxBlkB<PT, PAIR_MINB>{blockIdx.x, gridDim.x}, p, v, S, src32, part, sp);
}

VX_DEVK void k_diff_combine_body(VxBlkB<0, 0> vb, const VxParams &p, const VxView &v, const VxScalars *S, const double *part,
                                 VxSplit sp) {
    int K;
    long long tstride;
    vx_split_of(S, sp, K, tstride);
    const long long n = S->n;
    for (long long i = vb.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)vb.n * blockDim.x) {
        double I2x = 0.0, I2y = 0.0, I1 = 0.0;
#pragma unroll 8
        for (int sc = 0; sc < K; ++sc) {
            const double *o = part + (long long)sc * 3 * tstride + i;
            I2x += o[0];
            I2y += o[tstride];
            I1 += o[2 * tstride];
        }
        if (fabs(I1) > 1e-5) {
            const double dd = v.d[i];
            v.vx[i * v.vs] += -p.nu * I2x / (I1 * dd);
            v.vy[i * v.vs] += -p.nu * I2y / (I1 * dd);
        }
    }
}
__global__ void k_diff_combine(VxParams p, VxView v, const VxScalars *S, const double *part,
                               VxSplit sp) {
    VX_PDL_WAIT();
    k_diff_combine_body(VxBlkB<0, 0>{blockIdx.x, gridDim.x}, p, v, S, part, sp);
}

// ---------------------------------------------------------------------------
// Resident blocks of a pair kernel: its grid, and what the split fills.
static int pair_slots(const VxLaunch &L, const VxParams &p, bool probe = false) {
    return vx_full_sms(L) * (probe && p.prec == VX_PREC_FP32 ? PROBE32_MINB : PAIR_MINB);
}
static int pair_tile(const VxParams &p) { return PT * (p.prec == VX_PREC_FP32 ? BS32_TPT : BS64_TPT); }

static cudaError_t maybe_pack(const VxLaunch &L, const VxParams &p, const VxView &v,
                              VxScalars *S, VxWork &w) {
    if (p.prec != VX_PREC_FP32) return cudaSuccess;
    vx_launch<k_pack32, k_pack32_body>(L, L.num_sms * 4, 256, 0, v, S, w.src32, w.cap);

    return cudaGetLastError();
}

// K: 0 for a step's sums (derived on the device from the body's own count).
static VxSplit pair_split(const VxLaunch &L, const VxParams &p, const VxWork &w, int nout, int K) {
    VxSplit sp;
    sp.cap = w.part_cap;
    sp.K = K;
    sp.slots = pair_slots(L, p, K > 0);
    sp.tile = pair_tile(p);
    sp.nout = nout;
    // within the partial-sum buffer (5 (8 SMs 1024 + capacity) doubles)
    sp.rounds = 4;
    return sp;
}

cudaError_t vx_launch_velocity(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S,
                               VxWork &w) {
    const VxSplit sp = pair_split(L, p, w, 5, 0);
    const int grid = pair_slots(L, p);
    if (maybe_pack(L, p, v, S, w) != cudaSuccess) return cudaGetLastError();
    if (p.prec == VX_PREC_FP32) {
        VX_EV(L, 0);
        vx_launch<k_bs32_partial, k_bs32_partial_body>(L, grid, PT, 0, p, S, w.src32, v.x, v.y, v.ps, w.part, sp);
        VX_EV(L, 1);

        vx_launch<k_bs_combine<true>, k_bs_combine_body<true>>(L, L.num_sms * 16, CMB_T * CMB_S, 0, v, S, w.part, sp);
    } else {
        VX_EV(L, 0);
        vx_launch<k_bs64_partial<true>, k_bs64_partial_body<true>>(L, grid, PT, 0, p, v, S, v.x, v.y, v.ps, -1, w.part, sp);
        VX_EV(L, 1);

        vx_launch<k_bs_combine<false>, k_bs_combine_body<false>>(L, L.num_sms * 16, CMB_T * CMB_S, 0, v, S, w.part, sp);
    }

    return cudaGetLastError();
}

cudaError_t vx_launch_diffusion(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S,
                                VxWork &w, bool packed) {
    // bulk form: neighbour lists within diff_cutoff * d_i (vx_cells.cu)
    if (p.prec == VX_PREC_FP32 && p.diff_cutoff > 0.0) return vx_launch_diffusion_cells(L, p, v, S, w);
    if (!packed && maybe_pack(L, p, v, S, w) != cudaSuccess) return cudaGetLastError();
    const VxSplit sp = pair_split(L, p, w, 3, 0);
    const int grid = pair_slots(L, p);
    VX_EV(L, 2);
    if (p.prec == VX_PREC_FP32) {
        vx_launch<k_diff32_partial, k_diff32_partial_body>(L, grid, PT, 0, p, v, S, w.src32, w.part, sp);
    } else {
        vx_launch<k_diff64_partial, k_diff64_partial_body>(L, grid, PT, 0, p, v, S, w.part, sp);
    }
    VX_EV(L, 3);

    vx_launch<k_diff_combine, k_diff_combine_body>(L, L.num_sms * 4, 256, 0, p, v, S, w.part, sp);

    return cudaGetLastError();
}

// Probe points: one round of resident blocks (their number is the caller's,
// so the split may follow it on the host; the sources' is on the device).
cudaError_t vx_launch_probe(const VxLaunch &L, const VxParams &p, const VxView &v, VxScalars *S,
                            VxWork &w, const double *px, const double *py, long long pstride,
                            long long np, double *ovx, double *ovy, long long ostride) {
    const bool few = p.prec == VX_PREC_FP32 && np <= 2 * PT;   // two targets a thread
    const int tile = few ? 2 * PT : pair_tile(p);
    const VxSplit sp = pair_split(L, p, w, 2, vx_pair_split(np, 1LL << 30, tile, pair_slots(L, p, true), 1));
    const int grid = pair_slots(L, p, true);
    if (w.part_cap / (2LL * sp.K) < np) return cudaErrorInvalidValue;
    if (maybe_pack(L, p, v, S, w) != cudaSuccess) return cudaGetLastError();
    if (few)
        vx_launch<k_probe32_partial<2>, k_probe32_partial_body<2>>(L, grid, PT, 0, p, S, w.src32, px, py, pstride, np, w.part, sp);
    else if (p.prec == VX_PREC_FP32)
        vx_launch<k_probe32_partial<4>, k_probe32_partial_body<4>>(L, grid, PT, 0, p, S, w.src32, px, py, pstride, np, w.part, sp);
    else
        vx_launch<k_bs64_partial<false>, k_bs64_partial_body<false>>(L, grid, PT, 0, p, v, S, px, py, pstride, np, w.part, sp);

    vx_launch<k_probe_combine, k_probe_combine_body>(L, (int)std::min(vx_ceil_div(np, 32), 4096LL), 256, 0, S, w.part, sp, np, ovx, ovy, ostride);

    return cudaGetLastError();
}

// Validation hook: one of the plain sums' own FP64 functions at n points.
__global__ void __launch_bounds__(PT) k_eval_fp64(int which, const double *x, double *out, long long n) {
    const double tab = c_exp_table[threadIdx.x & 31];
    for (long long b = blockIdx.x * (long long)PT; b < n; b += (long long)gridDim.x * PT) {   // whole warps
        const long long i = b + threadIdx.x;
        const double v = i < n ? x[i] : 0.0;
        const double r = which == 0 ? vx_rcp64(v) : (which == 1 ? vx_rsqrt64(v) : vx_exp2_32(v, tab));
        if (i < n) out[i] = r;
    }
}
extern "C" vx_status vx_eval_fp64(int which, const double *x, double *out, int64_t n) {
    if (which < 0 || which > 2 || n < 0 || (n > 0 && (!x || !out))) return VX_ERR_ARG;
    if (n == 0) return VX_OK;
    k_eval_fp64<<<(unsigned)std::min<long long>(vx_ceil_div(n, (long long)PT), 1024), PT>>>(which, x, out, n);
    return cudaDeviceSynchronize() == cudaSuccess ? VX_OK : VX_ERR_CUDA;
}

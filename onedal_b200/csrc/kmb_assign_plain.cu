// Plain-form assignment: fused x.c contraction + per-row argmin (FP32 / FP64 FMA).
//
// Replaces, for every row block, DAAL's
//   buf = clSq - X_b * C^T  (xxgemm, α = -1, β = 1) followed by a strict-'<'
//   argmin scan over clusters
// (cpp/daal/src/algorithms/kmeans/kmeans_lloyd_impl.i:174-216 in the update loop and
//  cpp/daal/src/algorithms/kmeans/kmeans_lloyd_postprocessing.h:95-130 for the final
//  responses). The n x k score matrix is never materialised: every kernel here streams
// clusters past its rows and keeps a running best (with a recheck queue: best, second and
// third) per row in registers.
//
//   assign_small_kernel     k <= 32 and d <= 64: a row per thread
//   assign_f64_kernel       other double rows: FP64 on the tensor pipe
//   assign_resident_kernel  float rows, many of them, clusters a multiple of 256 that fit
//                           shared memory
//   assign_few_kernel       all other float rows
//
// Scores are h_j - x.c_j with h_j = 0.5 ||c_j||^2 (the DAAL form); ties resolve to
// the lowest cluster index. Rows whose best/second gap lies inside the derived
// rounding bound are queued for an FP64 recheck when a queue is given.
#include "kmb_internal.cuh"

#include <float.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>

namespace kmb {
namespace {

constexpr int BM = 128;  // rows per CTA (FP64)
constexpr int BK = 8;    // columns that C^T's rows are padded to; the FP64 contraction chunk
constexpr int NT = 256;  // threads (FP64)

template <typename F> struct Vec4;
template <> struct Vec4<float> { using T = float4; };
template <> struct Vec4<double> { using T = double4; };

template <typename F> __device__ __forceinline__ F f_inf();
template <> __device__ __forceinline__ float f_inf<float>() { return __int_as_float(0x7f800000); }
template <> __device__ __forceinline__ double f_inf<double>() { return __longlong_as_double(0x7ff0000000000000LL); }

template <typename F> __device__ __forceinline__ double unit_roundoff();
template <> __device__ __forceinline__ double unit_roundoff<float>() { return 5.9604644775390625e-8; }   // 2^-24
template <> __device__ __forceinline__ double unit_roundoff<double>() { return 1.1102230246251565e-16; } // 2^-53

// (value, index) lexicographic "less".
template <typename F>
__device__ __forceinline__ bool lex_less(F a, int ia, F b, int ib) {
    return a < b || (a == b && ia < ib);
}

template <typename F>
struct RowTop {
    F b, s, t;   // best, second, third score
    int ib, is;  // best / second cluster index
};

template <typename F>
__device__ __forceinline__ void top_push(RowTop<F> &r, F v, int c) {
    // Columns arrive in increasing order within a thread, so strict '<' keeps
    // the lowest index on ties.
    if (v < r.b) {
        r.t = r.s;
        r.s = r.b;
        r.is = r.ib;
        r.b = v;
        r.ib = c;
    } else if (v < r.s) {
        r.t = r.s;
        r.s = v;
        r.is = c;
    } else if (v < r.t) {
        r.t = v;
    }
}

// top_push with selects instead of branches (the same result).
template <typename F>
__device__ __forceinline__ void top_push_sel(RowTop<F> &r, F v, int c) {
    const bool lb = v < r.b, ls = v < r.s, lt = v < r.t;
    r.t = ls ? r.s : (lt ? v : r.t);
    r.s = lb ? r.b : (ls ? v : r.s);
    r.is = lb ? r.ib : (ls ? c : r.is);
    r.b = lb ? v : r.b;
    r.ib = lb ? c : r.ib;
}

// Merge of two sorted triples in (value, index) order, by selects; indices are kept for
// the first two places only.
template <typename F>
__device__ __forceinline__ RowTop<F> top_merge_sel(const RowTop<F> &x, const RowTop<F> &y) {
    constexpr int kNone = 0x7fffffff;  // index of a third place
    const bool c0 = lex_less(x.b, x.ib, y.b, y.ib);
    // second place: the heads of both lists after the first output
    const F xa = c0 ? x.s : x.b, ya = c0 ? y.b : y.s;
    const int xai = c0 ? x.is : x.ib, yai = c0 ? y.ib : y.is;
    const bool c1 = lex_less(xa, xai, ya, yai);
    // third place: x took both (x.t vs y.b), y took both (x.b vs y.t), or one each (x.s vs y.s)
    const bool xx = c0 && c1, yy = !c0 && !c1;
    const F xh = xx ? x.t : (yy ? x.b : x.s), yh = xx ? y.b : (yy ? y.t : y.s);
    const int xhi = xx ? kNone : (yy ? x.ib : x.is), yhi = xx ? y.ib : (yy ? kNone : y.is);
    const bool c2 = lex_less(xh, xhi, yh, yhi);
    RowTop<F> r;
    r.b = c0 ? x.b : y.b;
    r.ib = c0 ? x.ib : y.ib;
    r.s = c1 ? xa : ya;
    r.is = c1 ? xai : yai;
    r.t = c2 ? xh : yh;
    return r;
}

template <typename F>
__device__ __forceinline__ RowTop<F> shfl_top(const RowTop<F> &x, int mask) {
    RowTop<F> y;
    y.b = __shfl_xor_sync(0xffffffffu, x.b, mask);
    y.s = __shfl_xor_sync(0xffffffffu, x.s, mask);
    y.t = __shfl_xor_sync(0xffffffffu, x.t, mask);
    y.ib = __shfl_xor_sync(0xffffffffu, x.ib, mask);
    y.is = __shfl_xor_sync(0xffffffffu, x.is, mask);
    return y;
}

// Keeps the rows of one half of `t` (hi: the upper half) and merges in the
// partner lane's triples of the same rows.
template <int R>
__device__ __forceinline__ void res_exchange(RowTop<float> (&t)[8], int mask, bool hi) {
#pragma unroll
    for (int q = 0; q < R / 2; ++q) {
        const RowTop<float> keep = hi ? t[R / 2 + q] : t[q];
        const RowTop<float> send = hi ? t[q] : t[R / 2 + q];
        t[q] = top_merge_sel(keep, shfl_top(send, mask));
    }
}

// The best alone (value, lowest index): the same exchange.
struct RowBest {
    float b;
    int ib;
};
__device__ __forceinline__ RowBest best_of(const RowBest &x, const RowBest &y) {
    const bool c = lex_less(x.b, x.ib, y.b, y.ib);
    return RowBest{c ? x.b : y.b, c ? x.ib : y.ib};
}
__device__ __forceinline__ RowBest shfl_best(const RowBest &x, int mask) {
    return RowBest{__shfl_xor_sync(0xffffffffu, x.b, mask), __shfl_xor_sync(0xffffffffu, x.ib, mask)};
}
template <int R>
__device__ __forceinline__ void best_exchange(RowBest (&t)[8], int mask, bool hi) {
#pragma unroll
    for (int q = 0; q < R / 2; ++q) {
        const RowBest keep = hi ? t[R / 2 + q] : t[q];
        const RowBest send = hi ? t[q] : t[R / 2 + q];
        t[q] = best_of(keep, shfl_best(send, mask));
    }
}

__device__ __forceinline__ void cp_async_zfill(void *smem, const void *gmem, int bytes, bool ok) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    if (bytes == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s), "l"(gmem), "r"(ok ? 4 : 0) : "memory");
    else if (bytes == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(s), "l"(gmem), "r"(ok ? 8 : 0) : "memory");
    else
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(ok ? 16 : 0) : "memory");
}

// ---- float rows --------------------------------------------------------------
// 32 rows per CTA (so a few thousand rows already cover the SMs): 4 warps of 8 rows, a
// lane the clusters 4l .. 4l+3 and 128+4l .. of each 256-cluster pass (the first four alone
// where a pass holds 128); row values are shared-memory broadcasts, centroid chunks of 16
// columns come by cp.async in a ring of two. Dot products add x_t * c_t in ascending t with
// FMAs from zero: the scores, and the labels, distances and recheck entries, are those of
// the other float kernels. Without a queue only a row's best is kept (a compare and two
// selects per score instead of ten instructions). Bound by the operands' way from shared
// memory into registers, one byte per FMA. Per launch, against the kernels used before (128
// x 128 tiles per CTA; 64-row tiles with resident centroids):
//   4097 x 64, k = 300 40 -> 11.6 us; 76,000 x 64, k = 300 173 -> 105; 300,000 x 128, k =
//   1000 2018 -> 1724; 1M x 37, k = 300 1295 -> 979; 50,000 x 1000, k = 500 1855 -> 1150
constexpr int kFewRows = 32, kFewPass = 256, kFewK = 16, kFewThreads = 128, kFewR = 8;

template <bool VEC, bool TOP3>
__global__ void __launch_bounds__(kFewThreads, 3)
assign_few_kernel(const float *__restrict__ X, int64_t n, int d, const float *__restrict__ Ct,
                  const float *__restrict__ h, int k, int kpad, const float *__restrict__ xnorm,
                  const double *__restrict__ cnorm_max, int32_t *__restrict__ labels, float *__restrict__ d2,
                  RecheckEntry *__restrict__ queue, LoopState *__restrict__ st) {
    if (st && st->done) return;
    __shared__ __align__(16) float Xs[2][kFewRows][kFewK];
    __shared__ __align__(16) float Cs[2][kFewK][kFewPass];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t row0 = (int64_t)blockIdx.x * kFewRows;
    const int dpad = (d + BK - 1) / BK * BK;           // rows of Ct
    const int nk = (d + kFewK - 1) / kFewK;
    const int npass = (kpad + kFewPass - 1) / kFewPass;
    const int steps = nk * npass;
    auto issue = [&](int step) {
        if (step < steps) {
            const int ps = step / nk, kb = (step - ps * nk) * kFewK, buf = step & 1;
            if (tid < kFewRows * kFewK / 4) {  // a row's four columns a thread
                const int r = tid / (kFewK / 4), c = 4 * (tid % (kFewK / 4));
                const float *src = X + (row0 + r < n ? row0 + r : 0) * d + kb + c;
                if (VEC) {  // d % 4 == 0 at a 16-byte aligned base
                    const bool ok = row0 + r < n && kb + c < d;
                    cp_async_zfill(&Xs[buf][r][c], ok ? src : X, 16, ok);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool ok = row0 + r < n && kb + c + i < d;
                        cp_async_zfill(&Xs[buf][r][c + i], ok ? src + i : X, 4, ok);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < kFewK * kFewPass / 4 / kFewThreads; ++i) {
                const int e = tid + i * kFewThreads, r = e / (kFewPass / 4), c = 4 * (e % (kFewPass / 4));
                const bool ok = kb + r < dpad && ps * kFewPass + c < kpad;
                cp_async_zfill(&Cs[buf][r][c], ok ? Ct + (int64_t)(kb + r) * kpad + ps * kFewPass + c : Ct, 16, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    RowTop<float> top[TOP3 ? kFewR : 1];  // TOP3: for the recheck queue; else the best alone
    RowBest best[TOP3 ? 1 : kFewR];
    float2 acc[kFewR][4];  // acc[i][q]: clusters 2q, 2q + 1 of this lane's eight
#pragma unroll
    for (int i = 0; i < kFewR; ++i) {
        if constexpr (TOP3) {
            top[i].b = top[i].s = top[i].t = f_inf<float>();
            top[i].ib = top[i].is = 0;
        } else {
            best[i] = RowBest{f_inf<float>(), 0};
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = make_float2(0.f, 0.f);
    }
    issue(0);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the step's chunks are visible, and every warp is done with the other buffer
        issue(step + 1);
        const int buf = step & 1, ps = step / nk;
        auto contract = [&](auto q_tag) {  // Q pairs of this lane's clusters
            constexpr int Q = decltype(q_tag)::value;
#pragma unroll
            for (int t = 0; t < kFewK; t += 2) {
                float2 a[kFewR];
#pragma unroll
                for (int i = 0; i < kFewR; ++i) a[i] = *reinterpret_cast<const float2 *>(&Xs[buf][kFewR * warp + i][t]);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float4 b0 = *reinterpret_cast<const float4 *>(&Cs[buf][t + u][4 * lane]);
                    float2 b[Q];
                    b[0] = make_float2(b0.x, b0.y);
                    b[1] = make_float2(b0.z, b0.w);
                    if constexpr (Q == 4) {
                        const float4 b1 = *reinterpret_cast<const float4 *>(&Cs[buf][t + u][128 + 4 * lane]);
                        b[2] = make_float2(b1.x, b1.y);
                        b[3] = make_float2(b1.z, b1.w);
                    }
#pragma unroll
                    for (int i = 0; i < kFewR; ++i) {
                        const float x = u ? a[i].y : a[i].x;
#pragma unroll
                        for (int q = 0; q < Q; ++q) acc[i][q] = __ffma2_rn(make_float2(x, x), b[q], acc[i][q]);
                    }
                }
            }
        };
        const bool narrow = ps * kFewPass + 128 >= kpad;
        if (narrow) contract(std::integral_constant<int, 2>());
        else contract(std::integral_constant<int, 4>());
        if (step - ps * nk == nk - 1) {  // the pass's scores, this lane's clusters in ascending order
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q >= 2 && narrow) break;
                const int col = ps * kFewPass + (q < 2 ? 4 * lane + 2 * q : 124 + 4 * lane + 2 * q);
                const float h0 = col < kpad ? h[col] : f_inf<float>(), h1 = col + 1 < kpad ? h[col + 1] : f_inf<float>();
#pragma unroll
                for (int i = 0; i < kFewR; ++i) {
                    const float v0 = h0 - acc[i][q].x, v1 = h1 - acc[i][q].y;
                    if constexpr (TOP3) {
                        top_push_sel(top[i], v0, col);
                        top_push_sel(top[i], v1, col + 1);
                    } else {
                        best[i].ib = v0 < best[i].b ? col : best[i].ib;
                        best[i].b = v0 < best[i].b ? v0 : best[i].b;
                        best[i].ib = v1 < best[i].b ? col + 1 : best[i].ib;
                        best[i].b = v1 < best[i].b ? v1 : best[i].b;
                    }
                    acc[i][q] = make_float2(0.f, 0.f);
                }
            }
        }
    }
    // lanes exchange halves of their rows; row `own` ends in four lanes
    const bool h16 = (lane >> 4) & 1, h8 = (lane >> 3) & 1, h4 = (lane >> 2) & 1;
    const int own = 4 * h16 + 2 * h8 + h4;
    if constexpr (TOP3) {
        res_exchange<8>(top, 16, h16);
        res_exchange<4>(top, 8, h8);
        res_exchange<2>(top, 4, h4);
        top[0] = top_merge_sel(top[0], shfl_top(top[0], 2));
        top[0] = top_merge_sel(top[0], shfl_top(top[0], 1));
    } else {
        best_exchange<8>(best, 16, h16);
        best_exchange<4>(best, 8, h8);
        best_exchange<2>(best, 4, h4);
        best[0] = best_of(best[0], shfl_best(best[0], 2));
        best[0] = best_of(best[0], shfl_best(best[0], 1));
    }
    if ((lane & 3) == 0) {
        RowTop<float> t = {};
        if constexpr (TOP3) {
            t = top[0];
        } else {
            t.b = best[0].b;
            t.ib = best[0].ib;
        }
        const int64_t r = row0 + kFewR * warp + own;
        if (r < n) {
            labels[r] = t.ib;
            const float xn = xnorm[r];
            d2[r] = 2.0f * t.b + xn;
            if (TOP3 && queue) {
                const double cmax = cnorm_max ? *cnorm_max : 0.0;
                const double xl = sqrt(fmax((double)xn, 0.0));
                const double e = 1.0625 * unit_roundoff<float>() * (cmax * cmax + (double)(d + 2) * xl * cmax);
                const double band = 2.0 * e;
                if ((double)t.s - (double)t.b <= band)
                    enqueue_recheck(queue, n, st, (int)r, t.ib, t.is, (double)t.t - (double)t.b <= band);
            }
        }
    }
}

// ---- FP64 on the tensor pipe --------------------------------------------------
// Double rows: a CTA of 8 warps (4 x 2) scores 128 rows against tiles of BN clusters with
// mma.sync m8n8k4.f64, whose products and sums are FP64 FMAs (the FP64 rate of the tensor
// pipe is that of the FMA pipe here, but a warp's 32 x BN/2 tile takes 12 operand values
// from shared memory for 256 FMAs per lane where the 8 x 8 tile per thread took 16 for 64:
// its shared-memory reads bounded it). Row and centroid chunks of 8 columns arrive by
// cp.async in a ring of three; the pitches (12 and BN + 4 doubles) keep the 8-byte fragment
// reads free of bank conflicts. BN = 64 where it pads k less than 128 does. TOP3: the
// running third place is kept for the recheck queue; else the best alone.
// Per launch: 300,007 x 37, k = 101 349 -> 179 us; 500,000 x 128, k = 1024 8.18 -> 5.03 ms
// (26 TFLOP/s).
constexpr int kDP = BK + 4;  // row pitch of the staged X chunk, in doubles
constexpr int kDStages = 3;

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

template <int BNT>
constexpr size_t f64_smem_bytes() { return sizeof(double) * kDStages * (BM * kDP + BK * (BNT + 4)); }

template <int BNT, bool TOP3>
__global__ void __launch_bounds__(NT, 1)
assign_f64_kernel(const double *__restrict__ X, int64_t n, int d, const double *__restrict__ Ct,
                  const double *__restrict__ h, int k, int kpad, const double *__restrict__ xnorm,
                  const double *__restrict__ cnorm_max, int32_t *__restrict__ labels, double *__restrict__ d2,
                  RecheckEntry *__restrict__ queue, LoopState *__restrict__ st) {
    if (st && st->done) return;
    constexpr int CP = BNT + 4;     // pitch of the staged centroid chunk
    constexpr int NTL = BNT / 16;   // 8-cluster tiles of a warp
    extern __shared__ __align__(16) double f64_smem[];
    double *Xs = f64_smem, *Cs = f64_smem + kDStages * BM * kDP;
    __shared__ RowTop<double> s_top[BM];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = warp & 3, wc = warp >> 2;  // rows 32 wr .., clusters BNT/2 wc ..
    const int g = lane >> 2, q4 = lane & 3;
    const int64_t row0 = (int64_t)blockIdx.x * BM;
    const int nk = (d + BK - 1) / BK;
    const int ntiles = (k + BNT - 1) / BNT;  // (tiles of padding alone are left out)
    const int steps = nk * ntiles;
    auto issue = [&](int step) {
        if (step < steps) {
            const int nt = step / nk, kb = (step - nt * nk) * BK, stage = step % kDStages;
            double *xd = Xs + stage * BM * kDP, *cd = Cs + stage * BK * CP;
#pragma unroll
            for (int i = 0; i < BM * BK / NT; ++i) {
                const int e = tid + i * NT, r = e / BK, c = e % BK;
                const bool ok = row0 + r < n && kb + c < d;
                cp_async_zfill(xd + r * kDP + c, ok ? X + (row0 + r) * d + kb + c : X, 8, ok);
            }
#pragma unroll
            for (int i = 0; i < BK * BNT / 2 / NT; ++i) {  // Ct has nk * BK rows, kpad columns (a multiple of 128)
                const int e = tid + i * NT, r = e / (BNT / 2), c = 2 * (e % (BNT / 2));
                cp_async_zfill(cd + r * CP + c, Ct + (int64_t)(kb + r) * kpad + nt * BNT + c, 16, true);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    RowTop<double> top[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        top[i].b = top[i].s = top[i].t = f_inf<double>();
        top[i].ib = top[i].is = 0;
    }
    double acc[4][NTL][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NTL; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    for (int p = 0; p < kDStages - 1; ++p) issue(p);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kDStages - 2) : "memory");
        __syncthreads();  // the step's chunks are visible, and every warp is done with the oldest stage
        issue(step + kDStages - 1);
        const int stage = step % kDStages;
        const double *xs = Xs + stage * BM * kDP + (32 * wr + g) * kDP + q4;
        const double *cs = Cs + stage * BK * CP + q4 * CP + wc * (BNT / 2) + g;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            double a[4], b[NTL];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[8 * i * kDP + kk];
#pragma unroll
            for (int j = 0; j < NTL; ++j) b[j] = cs[kk * CP + 8 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < NTL; ++j) dmma(acc[i][j], a[i], b[j]);
        }
        const int nt = step / nk;
        if (step - nt * nk == nk - 1) {  // the tile's scores h_j - x.c_j into the running places
            const int col0 = nt * BNT + wc * (BNT / 2) + 2 * q4;
#pragma unroll
            for (int j = 0; j < NTL; ++j) {
                const int col = col0 + 8 * j;
                const double h0 = h[col], h1 = h[col + 1];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const double v0 = h0 - acc[i][j][0], v1 = h1 - acc[i][j][1];
                    acc[i][j][0] = acc[i][j][1] = 0.0;
                    if constexpr (TOP3) {
                        top_push_sel(top[i], v0, col);
                        top_push_sel(top[i], v1, col + 1);
                    } else {
                        if (v0 < top[i].b) {
                            top[i].b = v0;
                            top[i].ib = col;
                        }
                        if (v1 < top[i].b) {
                            top[i].b = v1;
                            top[i].ib = col + 1;
                        }
                    }
                }
            }
        }
    }
    // a row's places from its four lanes, then from the two warps that share it
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        top[i] = top_merge_sel(top[i], shfl_top(top[i], 1));
        top[i] = top_merge_sel(top[i], shfl_top(top[i], 2));
        if (wc == 1 && q4 == 0) s_top[32 * wr + 8 * i + g] = top[i];
    }
    __syncthreads();
    if (wc == 0 && q4 == 0) {
        const double u = unit_roundoff<double>();
        const double cmax = cnorm_max ? *cnorm_max : 0.0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t r = row0 + 32 * wr + 8 * i + g;
            if (r >= n) continue;
            const RowTop<double> t = top_merge_sel(top[i], s_top[32 * wr + 8 * i + g]);
            labels[r] = t.ib;
            const double xn = xnorm[r];
            d2[r] = 2.0 * t.b + xn;
            if (TOP3 && queue) {
                // |computed - exact| per score <= u*cmax^2 + (d+2)*u*||x||*cmax (+ slack), in any
                // order of the FMAs; two scores further apart than twice that are in order
                const double xl = sqrt(fmax(xn, 0.0));
                const double e = 1.0625 * u * (cmax * cmax + (double)(d + 2) * xl * cmax);
                const double band = 2.0 * e;
                if (t.s - t.b <= band) enqueue_recheck(queue, n, st, (int)r, t.ib, t.is, t.t - t.b <= band);
            }
        }
    }
}

// Per-iteration centroid preparation: Ct (dpad x kpad, zero padded), h (kpad,
// +inf padding), max ||c|| (double).
template <typename F>
__global__ void prep_centroids_kernel(const F *__restrict__ C, int k, int d, int dpad, int kpad, F *__restrict__ Ct,
                                      F *__restrict__ h, double *__restrict__ cnorm_max, const LoopState *st) {
    if (st && st->done) return;
    __shared__ double red[32];
    const int j = blockIdx.x;  // one block per (padded) cluster
    double s = 0.0;
    for (int t = threadIdx.x; t < dpad; t += blockDim.x) {
        F v = (j < k && t < d) ? C[(int64_t)j * d + t] : F(0);
        Ct[(int64_t)t * kpad + j] = v;
        s += (double)v * (double)v;
    }
    for (int m = 16; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
        h[j] = (j < k) ? F(0.5 * tot) : f_inf<F>();
        if (j < k) {
            // max of non-negative doubles via the ordered integer view
            atomicMax(reinterpret_cast<unsigned long long *>(cnorm_max),
                      (unsigned long long)__double_as_longlong(sqrt(tot)));
        }
    }
}

// ||x||^2 per row: FP64 sum of squares (lane t, t+32, ...; then a butterfly), rounded to F.
// R rows a warp at a time, so that R loads are in flight; the lanes halve the rows they hold
// at each exchange, which adds the same pairs as a butterfly per row does.
template <typename F, int R>
__global__ void __launch_bounds__(256) row_norms_kernel(const F *__restrict__ X, int64_t n, int d,
                                                        F *__restrict__ xnorm) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t row = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * R; row < n; row += warps * R) {
        double v[R];
        const F *x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            v[i] = 0.0;
            x[i] = X + min(row + i, n - 1) * d;
        }
        for (int t = lane; t < d; t += 32) {
            F xt[R];
#pragma unroll
            for (int i = 0; i < R; ++i) xt[i] = x[i][t];
#pragma unroll
            for (int i = 0; i < R; ++i) v[i] += (double)xt[i] * (double)xt[i];
        }
        int mine = 0;
#pragma unroll
        for (int m = 16, held = R; m >= 1; m >>= 1) {
            if (held > 1) {
                held >>= 1;
                const bool upper = lane & m;
#pragma unroll
                for (int i = 0; i < R / 2; ++i)
                    if (i < held) {
                        const double keep = upper ? v[i + held] : v[i], send = upper ? v[i] : v[i + held];
                        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                    }
                if (upper) mine += held;
            } else {
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
            }
        }
        if (lane % (32 / R) == 0 && row + mine < n) xnorm[row + mine] = F(v[0]);
    }
}

constexpr int kSmallK = 32;        // clusters handled by assign_small_kernel
constexpr int kSmallThreads = 128;

// Few clusters (k <= 32, d <= 64): one row per thread, its d values in registers,
// all centroids in shared memory (read as broadcasts). The contraction of row and
// cluster accumulates x_t * c_t in ascending t, as the other kernels do, so the
// scores -- and the labels, distances and recheck entries -- are the same; only
// the 128-cluster tile padding and the tile epilogue are gone.
// d > 32: bound by the rows' bytes, and a thread that reads its own row straight from memory
// touches 32 lines a load (9M x 64 floats 2436 us, 0.95 TB/s; 9.6M x 64 doubles 2948 us). Each
// warp copies its 32 rows side by side into an odd-strided tile, moves them to registers and
// has the next rows on their way while it works, four clusters at a time since one dot
// product is a chain of d FMAs: 841 and 1608 us. Shorter rows stay in L1 between a thread's
// loads and are read directly (5M x 17, k = 31 floats: 410 us, through the tile 501 us).
template <typename F, int DMAX>
__global__ void __launch_bounds__(kSmallThreads)
assign_small_kernel(const F *__restrict__ X, int64_t n, int d, const F *__restrict__ Ct, const F *__restrict__ h,
                    int k, int kpad, const F *__restrict__ xnorm, const double *__restrict__ cnorm_max,
                    int32_t *__restrict__ labels, F *__restrict__ d2, RecheckEntry *__restrict__ queue,
                    LoopState *__restrict__ st) {
    if (st && st->done) return;
    __shared__ __align__(16) F Cs[kSmallK][DMAX];
    __shared__ F hs[kSmallK];
    extern __shared__ __align__(16) unsigned char small_rows[];
    constexpr bool kTile = DMAX > 32;
    constexpr int QN = kTile ? 4 : 1;  // clusters at a time
    for (int i = threadIdx.x; i < kSmallK * DMAX; i += blockDim.x) {
        const int j = i / DMAX, t = i % DMAX;
        Cs[j][t] = (j < k && t < d) ? Ct[(int64_t)t * kpad + j] : F(0);
    }
    for (int j = threadIdx.x; j < kSmallK; j += blockDim.x) hs[j] = j < k ? h[j] : f_inf<F>();
    __syncthreads();
    const double u = unit_roundoff<F>();
    const double cmax = cnorm_max ? *cnorm_max : 0.0;
    const int lane = threadIdx.x & 31, ld = d | 1;
    F *tile = reinterpret_cast<F *>(small_rows) + (threadIdx.x >> 5) * 32 * ld;
    const int64_t step = (int64_t)gridDim.x * kSmallThreads;
    auto copy_rows = [&](int64_t first) {  // rows [first, first + 32) below n: one run of memory
        const int total = first < n ? (int)min((int64_t)32, n - first) * d : 0;
        const F *src = X + first * d;
        for (int i = lane, r = 0, t = lane; i < total; i += 32, t += 32) {
            if (t >= d) {  // d > 32: one row on at most
                t -= d;
                ++r;
            }
            cp_async_zfill(&tile[r * ld + t], src + i, (int)sizeof(F), true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // The warp's first row, or the thread's own where it reads directly.
    int64_t first = (int64_t)blockIdx.x * kSmallThreads + (kTile ? threadIdx.x & ~31 : threadIdx.x);
    if (kTile) copy_rows(first);
    for (; first < n; first += step) {
        const int64_t r = first + (kTile ? lane : 0);
        F x[DMAX];
        if constexpr (kTile) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();
#pragma unroll
            for (int t = 0; t < DMAX; ++t) x[t] = t < d ? tile[lane * ld + t] : F(0);
            __syncwarp();
            copy_rows(first + step);
            if (r >= n) continue;
        } else {
            const F *xr = X + r * (int64_t)d;
#pragma unroll
            for (int t = 0; t < DMAX; ++t) x[t] = t < d ? xr[t] : F(0);
        }
        RowTop<F> top;
        top.b = top.s = top.t = f_inf<F>();
        top.ib = top.is = 0;
        for (int j = 0; j < k; j += QN) {
            F dot[QN];
#pragma unroll
            for (int q = 0; q < QN; ++q) dot[q] = F(0);
#pragma unroll
            for (int t = 0; t < DMAX; t += 4) {
#pragma unroll
                for (int q = 0; q < QN; ++q) {
                    const typename Vec4<F>::T c = *reinterpret_cast<const typename Vec4<F>::T *>(&Cs[j + q][t]);
                    dot[q] = fma(x[t], c.x, dot[q]);
                    dot[q] = fma(x[t + 1], c.y, dot[q]);
                    dot[q] = fma(x[t + 2], c.z, dot[q]);
                    dot[q] = fma(x[t + 3], c.w, dot[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < QN; ++q)
                if (j + q < k) top_push(top, hs[j + q] - dot[q], j + q);
        }
        labels[r] = top.ib;
        const F xn = xnorm[r];
        d2[r] = F(2) * top.b + xn;
        if (queue) {
            const double xl = sqrt(fmax((double)xn, 0.0));
            const double e = 1.0625 * u * (cmax * cmax + (double)(d + 2) * xl * cmax);
            const double band = 2.0 * e;
            if ((double)top.s - (double)top.b <= band)
                enqueue_recheck(queue, n, st, (int)r, top.ib, top.is, (double)top.t - (double)top.b <= band);
        }
    }
    if (kTile) asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---- FP32, centroids resident in shared memory ------------------------------
// When all (padded) centroids fit in shared memory next to the row stages, one
// persistent CTA per SM keeps C^T and the half norms resident and streams 64-row
// tiles of X through TMA, so no centroid byte is re-read per row tile. 16 warps in two groups of 8; each group owns every other
// 64-row tile (group g of CTA b takes tiles 2(b + i·grid) + g) and one or two TMA
// stages. In a group, warp w owns rows 8w..8w+7 of the tile, lane l the clusters
// 4l..4l+3 and 128+4l..128+4l+3 of each 256-cluster pass: the row values are
// shared-memory broadcasts and the centroid reads are conflict-free 16-byte
// loads. Per (row, cluster) the contraction accumulates x_t * c_t in ascending
// t with FMAs from zero, as the other float kernels do, so the scores -- and the
// labels, distances and recheck entries -- are the same. After each pass a
// lane holds the top-3 (the best alone without a recheck queue: 10M x 64, k = 256 8.62 ms
// a launch with the top-3, 7.34 ms with the best) of its 8 clusters for its warp's 8 rows; five exchange
// rounds halve the rows a lane keeps while merging in the partner's (value,
// index) triples, leaving each row's top-3 in four lanes; with more than one
// pass the row's owner lane merges it into the running top-3 in shared memory.
//
// Ping-pong: the two groups take turns at the FMA pipe. A group runs a pass's
// contraction only in its turn and hands the turn over (named barriers 1 and 2)
// before its top-3 epilogue, so one group's epilogue (compares, selects,
// shuffles) issues beside the other group's FMAs instead of every warp of the SM
// reaching its epilogue at once and leaving the FMA pipe idle. Both groups take
// the same number of turns (a group without a tile left takes empty turns), so
// every barrier completes. With two stages per group the next tile's load is
// issued at the start of a tile's first turn (the turn barriers order the
// stage's last reads before it); with one stage, after the tile's last
// contraction, once the group's warps have met at named barrier 3 + g.
constexpr int kResThreads = 512;
constexpr int kResGroupThreads = 256;
constexpr int kResRows = 64;    // rows per tile (one group's)
constexpr int kResCtaRows = 128;  // rows per CTA step (both groups)
constexpr int kResPass = 256;
constexpr long long kResTimeout = 4000000000ll;  // ~2 s of SM clocks per wait

struct ResBarriers {
    uint64_t full[4];  // [group][stage]
    int abort;
    int issued[4];  // loads issued into each stage (the group's thread 0)
};

__device__ __forceinline__ uint32_t res_su32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool res_try_wait(uint64_t *b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(res_su32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: false after ~2 s (recorded in abort) or when another thread aborted.
__device__ __forceinline__ bool res_wait(uint64_t *b, uint32_t parity, volatile int *abort) {
    if (res_try_wait(b, parity)) return true;
    const long long t0 = clock64();
    while (!res_try_wait(b, parity)) {
        if (*abort) return false;
        if (clock64() - t0 > kResTimeout) {
            *abort = 1;
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void res_load_tile(float *dst, const CUtensorMap *tm, uint64_t *bar, int row0,
                                              uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(res_su32(bar)), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            res_su32(dst)),
        "l"(tm), "r"(res_su32(bar)), "r"(0), "r"(row0)
        : "memory");
}

// Named barriers of the turn protocol: the waiting group's 256 threads sync, the
// other group's 256 arrive.
__device__ __forceinline__ void res_turn_wait(int id) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(kResThreads) : "memory");
}
__device__ __forceinline__ void res_turn_give(int id) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(kResThreads) : "memory");
}

// DPADT > 0 fixes the padded row width at compile time (row and centroid offsets
// become immediates); 0 reads it from dpad. STAGES: TMA stages per group (1 or 2).
// kres: the clusters, padded to 256.
template <int DPADT, int STAGES, bool TOP3>
__global__ void __launch_bounds__(kResThreads, 1)
assign_resident_kernel(const __grid_constant__ CUtensorMap tmX, int64_t n, int d, int dpad_rt, const float *__restrict__ Ct,
                       const float *__restrict__ h, int k, int kpad, int kres,
                       const float *__restrict__ xnorm, const double *__restrict__ cnorm_max,
                       int32_t *__restrict__ labels, float *__restrict__ d2, RecheckEntry *__restrict__ queue,
                       LoopState *__restrict__ st) {
    __shared__ int s_skip;
    if (threadIdx.x == 0) s_skip = st ? st->done : 0;
    __syncthreads();
    if (s_skip) return;
    const int dpad = DPADT > 0 ? DPADT : dpad_rt;
    extern __shared__ uint8_t res_smem_raw[];
    uint8_t *sm = (uint8_t *)(((uintptr_t)res_smem_raw + 127) & ~(uintptr_t)127);
    const int tile_floats = kResRows * dpad;
    float *Xs = (float *)sm;                        // [group][stage][64][dpad]
    float *Cs = Xs + 2 * STAGES * tile_floats;      // [kres / 256][dpad][256]: pass-major blocks
    float *hs = Cs + (size_t)dpad * kres;           // [kres]
    RowTop<float> *run = (RowTop<float> *)(hs + kres);  // [group][64] running top-3
    ResBarriers *bar = (ResBarriers *)(run + 2 * kResRows);
    volatile int *abort = &bar->abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = warp >> 3, gw = warp & 7, gtid = tid & (kResGroupThreads - 1);
    // tiles of group g: 2 (b + i·grid) + g for i = 0 .. my_tiles - 1
    const int64_t n_tiles = (n + kResRows - 1) / kResRows;
    const int64_t par_tiles = (n_tiles - g + 1) / 2;     // tiles of parity g
    const int64_t par_tiles0 = (n_tiles + 1) / 2;        // of parity 0 (the most)
    const int grid = (int)gridDim.x, b = (int)blockIdx.x;
    const int my_tiles = par_tiles > b ? (int)((par_tiles - b + grid - 1) / grid) : 0;
    const int steps = par_tiles0 > b ? (int)((par_tiles0 - b + grid - 1) / grid) : 0;  // group 0's count
    const uint32_t tile_bytes = (uint32_t)tile_floats * 4u;
    float *Xg = Xs + STAGES * g * tile_floats;  // this group's stages
    uint64_t *full = &bar->full[2 * g];
    int *issued = &bar->issued[2 * g];
    if (tid == 0) {
        for (int i = 0; i < 4; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(res_su32(&bar->full[i])) : "memory");
            bar->issued[i] = 0;
        }
        bar->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (gtid == 0 && my_tiles > 0) {
        res_load_tile(Xg, &tmX, &full[0], (int)((2 * (int64_t)b + g) * kResRows), tile_bytes);
        issued[0] = 1;
    }
    // Resident centroids: C^T in 256-column blocks, one per pass, so a pass reads rows 256
    // floats apart (zero columns past kpad), and the half norms (+inf past kpad).
    const int kq = kres / 4;
    for (int i = tid; i < dpad * kq; i += kResThreads) {
        const int t = i / kq, c = 4 * (i - t * kq);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < kpad) v = *reinterpret_cast<const float4 *>(Ct + (size_t)t * kpad + c);
        *reinterpret_cast<float4 *>(Cs + ((size_t)(c / kResPass) * dpad + t) * kResPass + (c % kResPass)) = v;
    }
    for (int j = tid; j < kres; j += kResThreads) hs[j] = j < kpad ? h[j] : f_inf<float>();
    __syncthreads();

    const double u = 5.9604644775390625e-8;  // 2^-24
    const double cmax = cnorm_max ? *cnorm_max : 0.0;
    const int total_turns = steps * (kres / kResPass);  // the same for both groups
    // the row of the tile whose final top-3 this lane holds after the exchange
    const int own = 8 * gw + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    bool ok = true;
    int turn = 0;
    const int passes = kres / kResPass;
    RowTop<float> *grun = run + g * kResRows;
    for (int lt = 0; lt < steps; ++lt) {
        const bool has = lt < my_tiles;
        const bool nxt_has = has && lt + 1 < my_tiles;
        const auto row_of = [&](int i) { return (2 * ((int64_t)b + (int64_t)i * grid) + g) * kResRows; };
        // this tile's stage and load parity (the group's tiles are loaded in order)
        const int stage = lt % STAGES;
        const uint32_t parity = (uint32_t)(lt / STAGES) & 1u;
        for (int pass = 0; pass < passes; ++pass, ++turn) {
            // wait for this group's turn at the FMA pipe: group 0 goes first
            if (g == 0) {
                if (turn > 0) res_turn_wait(1);
            } else {
                res_turn_wait(2);
            }
            if (pass == 0 && has) {
                // Two stages: the next tile goes into the other stage, whose last
                // reads (the previous tile's contractions) came before this group
                // handed over its previous turn.
                if (STAGES == 2 && gtid == 0 && ok && nxt_has) {
                    const int s2 = (lt + 1) % STAGES;
                    res_load_tile(Xg + s2 * tile_floats, &tmX, &full[s2], (int)row_of(lt + 1), tile_bytes);
                    issued[s2] += 1;
                }
                if (ok && !__all_sync(0xffffffffu, res_wait(&full[stage], parity, abort))) ok = false;
            }
            const bool work = has && ok;
            // Packed FP32 FMAs (fma.rn.f32x2: two correctly rounded FMAs, the same
            // results as fmaf): each pair holds two of this lane's clusters for one
            // row, with the row's value duplicated; one issue slot per two FMAs.
            float2 acc2[8][4];  // acc2[i][q] = clusters 2q, 2q + 1 of this lane's eight
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int q2 = 0; q2 < 4; ++q2) acc2[i][q2] = make_float2(0.f, 0.f);
            if (work) {
                const float *xa = Xg + stage * tile_floats + (8 * gw) * dpad;
                const float *cb = Cs + (size_t)pass * dpad * kResPass + 4 * lane;
#pragma unroll 1
                for (int t = 0; t < dpad; t += 2) {
                    float2 a[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float2 *>(xa + i * dpad + t);
                    const float4 b00 = *reinterpret_cast<const float4 *>(cb + t * kResPass);
                    const float4 b01 = *reinterpret_cast<const float4 *>(cb + t * kResPass + 128);
                    const float4 b10 = *reinterpret_cast<const float4 *>(cb + (t + 1) * kResPass);
                    const float4 b11 = *reinterpret_cast<const float4 *>(cb + (t + 1) * kResPass + 128);
                    const float2 bx[4] = {make_float2(b00.x, b00.y), make_float2(b00.z, b00.w),
                                          make_float2(b01.x, b01.y), make_float2(b01.z, b01.w)};
                    const float2 by[4] = {make_float2(b10.x, b10.y), make_float2(b10.z, b10.w),
                                          make_float2(b11.x, b11.y), make_float2(b11.z, b11.w)};
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float2 ax = make_float2(a[i].x, a[i].x);
#pragma unroll
                        for (int q2 = 0; q2 < 4; ++q2) acc2[i][q2] = __ffma2_rn(ax, bx[q2], acc2[i][q2]);
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float2 ay = make_float2(a[i].y, a[i].y);
#pragma unroll
                        for (int q2 = 0; q2 < 4; ++q2) acc2[i][q2] = __ffma2_rn(ay, by[q2], acc2[i][q2]);
                    }
                }
            }
            const bool last_pass = pass + 1 == passes;
            // One stage: the group's warps meet once the tile's last contraction is
            // done (warp 0 waits, the others arrive), before the turn goes over.
            if (STAGES == 1 && last_pass) {
                if (gw == 0) asm volatile("bar.sync %0, %1;" ::"r"(3 + g), "r"(kResGroupThreads) : "memory");
                else asm volatile("bar.arrive %0, %1;" ::"r"(3 + g), "r"(kResGroupThreads) : "memory");
            }
            // hand the FMA pipe to the other group (group 1's last turn has no taker)
            if (g == 0) {
                res_turn_give(2);
            } else if (turn + 1 < total_turns) {
                res_turn_give(1);
            }
            if (STAGES == 1 && last_pass && gtid == 0 && ok && nxt_has) {
                res_load_tile(Xg, &tmX, &full[0], (int)row_of(lt + 1), tile_bytes);
                issued[0] += 1;
            }
            if (!work) continue;
            float acc[8][8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int q2 = 0; q2 < 4; ++q2) {
                    acc[i][2 * q2] = acc2[i][q2].x;
                    acc[i][2 * q2 + 1] = acc2[i][q2].y;
                }
            // this lane's clusters in ascending order: strict '<' keeps the lowest index
            // on ties; row by row, so a row's scores are dead once its top-3 is built
            float hv[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) hv[j] = hs[pass * kResPass + (j < 4 ? 4 * lane + j : 128 + 4 * lane + (j - 4))];
            const int col0 = pass * kResPass + 4 * lane;
            RowTop<float> r = {};  // row `own`'s places, in four lanes after the exchange
            if constexpr (TOP3) {
                RowTop<float> top[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float v0 = hv[0] - acc[i][0];
                    const bool l0 = v0 < f_inf<float>();  // a push into an empty triple
                    top[i].b = l0 ? v0 : f_inf<float>();
                    top[i].ib = l0 ? col0 : 0;
                    top[i].s = top[i].t = f_inf<float>();
                    top[i].is = 0;
#pragma unroll
                    for (int j = 1; j < 8; ++j) top_push_sel(top[i], hv[j] - acc[i][j], col0 + (j < 4 ? j : 124 + j));
                }
                res_exchange<8>(top, 16, (lane >> 4) & 1);
                res_exchange<4>(top, 8, (lane >> 3) & 1);
                res_exchange<2>(top, 4, (lane >> 2) & 1);
                top[0] = top_merge_sel(top[0], shfl_top(top[0], 2));
                top[0] = top_merge_sel(top[0], shfl_top(top[0], 1));
                r = top[0];
            } else {
                RowBest best[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    best[i] = RowBest{f_inf<float>(), 0};
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float v = hv[j] - acc[i][j];
                        const bool l = v < best[i].b;
                        best[i].ib = l ? col0 + (j < 4 ? j : 124 + j) : best[i].ib;
                        best[i].b = l ? v : best[i].b;
                    }
                }
                best_exchange<8>(best, 16, (lane >> 4) & 1);
                best_exchange<4>(best, 8, (lane >> 3) & 1);
                best_exchange<2>(best, 4, (lane >> 2) & 1);
                best[0] = best_of(best[0], shfl_best(best[0], 2));
                best[0] = best_of(best[0], shfl_best(best[0], 1));
                r.b = best[0].b;
                r.ib = best[0].ib;
            }
            if ((lane & 3) == 0) {
                if (pass > 0) {
                    if constexpr (TOP3) {
                        r = top_merge_sel(grun[own], r);
                    } else {
                        const RowBest m = best_of(RowBest{grun[own].b, grun[own].ib}, RowBest{r.b, r.ib});
                        r.b = m.b;
                        r.ib = m.ib;
                    }
                }
                if (!last_pass) {
                    grun[own] = r;
                } else {
                    const int64_t row = row_of(lt) + own;
                    if (row < n) {
                        labels[row] = r.ib;
                        const float xn = xnorm[row];
                        d2[row] = 2.0f * r.b + xn;
                        if (TOP3 && queue) {
                            const double xl = sqrt(fmax((double)xn, 0.0));
                            const double e = 1.0625 * u * (cmax * cmax + (double)(d + 2) * xl * cmax);
                            const double band = 2.0 * e;
                            if ((double)r.s - (double)r.b <= band)
                                enqueue_recheck(queue, n, st, (int)row, r.ib, r.is,
                                                (double)r.t - (double)r.b <= band);
                        }
                    }
                }
            }
        }
    }
    __syncthreads();  // every wait of both groups has ended before abort is read
    if (gtid == 0) {
        if (*abort) {
            // leave no bulk copy landing in shared memory behind: wait (bounded) for
            // the last load this group issued into each of its stages
            for (int s2 = 0; s2 < STAGES; ++s2) {
                const int iss = issued[s2];
                if (!iss) continue;
                const long long t0 = clock64();
                while (!res_try_wait(&full[s2], (uint32_t)((iss - 1) & 1)) && clock64() - t0 < kResTimeout) {
                }
            }
            if (st) {
                st->error = KMB_ETIMEDOUT;
                st->done = 1;
            }
        }
    }
}

// Shared memory of assign_resident_kernel for dpad features, kres resident clusters and
// STAGES stages per group.
size_t resident_smem_bytes(int dpad, int kres, int stages) {
    return 128 + (size_t)2 * stages * kResRows * dpad * 4 + (size_t)dpad * kres * 4 + (size_t)kres * 4 +
           (size_t)2 * kResRows * sizeof(RowTop<float>) + sizeof(ResBarriers);
}

}  // namespace

template <typename F>
void launch_prep_centroids(const F *C, int64_t k, int64_t d, int64_t kpad, F *Ct, F *h, double *cnorm_max,
                           const LoopState *st, cudaStream_t s) {
    const int dpad = (int)((d + BK - 1) / BK * BK);
    prep_centroids_kernel<F><<<(unsigned)kpad, 128, 0, s>>>(C, (int)k, (int)d, dpad, (int)kpad, Ct, h, cnorm_max, st);
    KMB_LAUNCHED();
}

template <typename F>
void launch_row_norms(const F *X, int64_t n, int64_t d, F *xnorm, cudaStream_t s) {
    if (n == 0) return;
    // Eight rows a warp where that still gives every SM its warps and a row alone is few loads
    // (9M x 64 floats 1184 -> 632 us, 9.6M x 64 doubles 1278 -> 907 us; 4M x 128 doubles 592 us
    // one by one, 621 us by eight).
    if (n >= 148 * 64 * 8 && d * (int64_t)sizeof(F) <= 512) {
        const int64_t blocks = std::min<int64_t>((n + 63) / 64, 148 * 16);
        row_norms_kernel<F, 8><<<(unsigned)blocks, 256, 0, s>>>(X, n, (int)d, xnorm);
    } else {
        const int64_t blocks = std::min<int64_t>((n + 7) / 8, 148 * 16);
        row_norms_kernel<F, 1><<<(unsigned)blocks, 256, 0, s>>>(X, n, (int)d, xnorm);
    }
    KMB_LAUNCHED();
}

template <typename F, int DMAX>
void launch_small(const F *X, int64_t n, int64_t d, const F *Ct, const F *h, int64_t k, int64_t kpad, const F *xnorm,
                  const double *cnorm_max, int32_t *labels, F *d2, RecheckEntry *queue, LoopState *st,
                  cudaStream_t s) {
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((n + kSmallThreads - 1) / kSmallThreads, 148 * 16));
    size_t smem = 0;
    if (DMAX > 32) {  // the tiles; the limit is the largest d's in every call, as threads set it side by side
        smem = sizeof(F) * kSmallThreads * (d | 1);
        cudaFuncSetAttribute(assign_small_kernel<F, DMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(sizeof(F) * kSmallThreads * (DMAX | 1)));
    }
    assign_small_kernel<F, DMAX><<<(unsigned)blocks, kSmallThreads, smem, s>>>(X, n, (int)d, Ct, h, (int)k, (int)kpad,
                                                                              xnorm, cnorm_max, labels, d2, queue, st);
    KMB_LAUNCHED();
}

// FP32 rows whose centroids fit in shared memory (d a multiple of 4 and at most 256,
// 16-byte aligned rows): the resident kernel. False when it does not apply.
template <typename F>
bool launch_resident(const F *, int64_t, int64_t, const F *, const F *, int64_t, int64_t, const F *, const double *,
                     int32_t *, F *, RecheckEntry *, LoopState *, cudaStream_t) {
    return false;
}
template <>
bool launch_resident<float>(const float *X, int64_t n, int64_t d, const float *Ct, const float *h, int64_t k,
                            int64_t kpad, const float *xnorm, const double *cnorm_max, int32_t *labels, float *d2,
                            RecheckEntry *queue, LoopState *st, cudaStream_t s) {
    if (d % 4 != 0 || d > 256 || (reinterpret_cast<uintptr_t>(X) % 16) != 0 || n > INT32_MAX - 2 * kResCtaRows)
        return false;
    // KMB_PLAIN_RESIDENT: 0 never, 1 wherever it applies (tests compare the two); else the
    // size rule below
    const char *e = getenv("KMB_PLAIN_RESIDENT");
    if (e && e[0] == '0') return false;
    const bool forced = e && e[0] == '1';
    // The better one for many rows and whole 256-cluster passes: 300,000 x 64, k = 256 241 us
    // against 246, 3M 2236 against 2313 (76,000: 78 against 68; 3M x 64, k = 300, whose
    // second pass is mostly padding here, 4422 against 3652)
    if (!forced && (n < (1 << 18) || kpad % kResPass != 0)) return false;
    const int dpad = (int)((d + BK - 1) / BK * BK);  // the rows of Ct
    const int kres = (int)((kpad + kResPass - 1) / kResPass * kResPass);
    int dev = 0, optin = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // Two stages per group; one where two do not fit beside 256 clusters (112 to 144 columns:
    // 3M x 128, k = 256 with a recheck queue, 3 iterations 21.6 ms against 22.4).
    const int stages = resident_smem_bytes(dpad, kres, 2) <= (size_t)optin ? 2 : 1;
    const size_t smem = resident_smem_bytes(dpad, kres, stages);
    if (smem + 64 > (size_t)optin || (stages == 1 && kres > kResPass)) return false;  // (64: static)
    CUtensorMap tm;
    // box: 64 rows x dpad columns (columns past d read as zeros)
    if (!encode_tensor_map_2d(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, X, (uint64_t)d, (uint64_t)n, (uint64_t)d * 4,
                              (uint32_t)dpad, (uint32_t)kResRows, CU_TENSOR_MAP_SWIZZLE_NONE))
        return false;
    // without a recheck queue only the best cluster of a row is kept
    auto pick = [&](auto top3) {
        constexpr bool T3 = decltype(top3)::value;
        auto by_d = [&](auto k32, auto k64, auto k128, auto k0) { return dpad == 32 ? k32 : dpad == 64 ? k64 : dpad == 128 ? k128 : k0; };
        return stages == 2 ? by_d(assign_resident_kernel<32, 2, T3>, assign_resident_kernel<64, 2, T3>,
                                  assign_resident_kernel<128, 2, T3>, assign_resident_kernel<0, 2, T3>)
                           : dpad == 128 ? assign_resident_kernel<128, 1, T3> : assign_resident_kernel<0, 1, T3>;
    };
    auto kern = queue ? pick(std::true_type()) : pick(std::false_type());
    if (allow_smem((const void *)kern) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const int64_t n_steps = (n + kResCtaRows - 1) / kResCtaRows;  // 128-row steps: two tiles, one per group
    const int grid = (int)std::min<int64_t>(n_steps, sms);
    kern<<<grid, kResThreads, smem, s>>>(tm, n, (int)d, dpad, Ct, h, (int)k, (int)kpad, kres, xnorm, cnorm_max, labels, d2, queue, st);
    KMB_LAUNCHED();
    return true;
}

static void launch_f64(unsigned blocks, const double *X, int64_t n, int64_t d, const double *Ct, const double *h,
                       int64_t k, int64_t kpad, const double *xnorm, const double *cnorm_max, int32_t *labels,
                       double *d2, RecheckEntry *queue, LoopState *st, cudaStream_t s) {
    // 64-cluster tiles where they pad k to fewer clusters
    const bool narrow = (k + 63) / 64 * 64 < (k + 127) / 128 * 128;
    auto kern = narrow ? (queue ? assign_f64_kernel<64, true> : assign_f64_kernel<64, false>)
                       : (queue ? assign_f64_kernel<128, true> : assign_f64_kernel<128, false>);
    const int smem = (int)(narrow ? f64_smem_bytes<64>() : f64_smem_bytes<128>());
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return;
    kern<<<blocks, NT, smem, s>>>(X, n, (int)d, Ct, h, (int)k, (int)kpad, xnorm, cnorm_max, labels, d2, queue, st);
    KMB_LAUNCHED();
}

template <typename F>
void launch_assign_plain(const F *X, int64_t n, int64_t d, const F *Ct, const F *h, int64_t k, int64_t kpad,
                         const F *xnorm, const double *cnorm_max, int32_t *labels, F *d2, RecheckEntry *queue,
                         LoopState *st, cudaStream_t s) {
    if (n == 0) return;
    if (k <= kSmallK && d <= 64) {  // few clusters: row per thread, centroids in shared memory
        if (d <= 16) launch_small<F, 16>(X, n, d, Ct, h, k, kpad, xnorm, cnorm_max, labels, d2, queue, st, s);
        else if (d <= 32) launch_small<F, 32>(X, n, d, Ct, h, k, kpad, xnorm, cnorm_max, labels, d2, queue, st, s);
        else launch_small<F, 64>(X, n, d, Ct, h, k, kpad, xnorm, cnorm_max, labels, d2, queue, st, s);
        return;
    }
    if constexpr (sizeof(F) == 8) {
        launch_f64((unsigned)((n + BM - 1) / BM), X, n, d, Ct, h, k, kpad, xnorm, cnorm_max, labels, d2, queue, st, s);
    } else {
        if (launch_resident(X, n, d, Ct, h, k, kpad, xnorm, cnorm_max, labels, d2, queue, st, s)) return;
        const bool vec = d % 4 == 0 && (reinterpret_cast<uintptr_t>(X) % 16) == 0;
        auto kern = vec ? (queue ? assign_few_kernel<true, true> : assign_few_kernel<true, false>)
                        : (queue ? assign_few_kernel<false, true> : assign_few_kernel<false, false>);
        kern<<<(unsigned)((n + kFewRows - 1) / kFewRows), kFewThreads, 0, s>>>(X, n, (int)d, Ct, h, (int)k, (int)kpad,
                                                                              xnorm, cnorm_max, labels, d2, queue, st);
        KMB_LAUNCHED();
    }
}

#define KMB_INST(F)                                                                                                \
    template void launch_prep_centroids<F>(const F *, int64_t, int64_t, int64_t, F *, F *, double *,            \
                                           const LoopState *, cudaStream_t);                                     \
    template void launch_row_norms<F>(const F *, int64_t, int64_t, F *, cudaStream_t);                                            \
    template void launch_assign_plain<F>(const F *, int64_t, int64_t, const F *, const F *, int64_t, int64_t,    \
                                         const F *, const double *, int32_t *, F *, RecheckEntry *, LoopState *, \
                                         cudaStream_t);
KMB_INST(float)
KMB_INST(double)
#undef KMB_INST

}  // namespace kmb

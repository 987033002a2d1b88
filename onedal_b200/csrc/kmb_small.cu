// Lloyd training of small dense problems in one cooperative launch (plain form).
//
// A small problem's iteration is a few microseconds of work; as separate kernels it is
// bound by the launches (14 per iteration, 1.3-2.3 us each). Here the whole train call --
// the Lloyd loop with its empty-cluster reseeding and stop test, the responses under the
// final centroids and the exact objective
// (cpp/daal/src/algorithms/kmeans/kmeans_lloyd_batch_impl.i:117-234) -- is one persistent
// kernel: at most one CTA per SM, each with a contiguous block of rows kept in shared
// memory for the whole call (X is read once from HBM), and two grid barriers per
// iteration.
//
//   assign      one row per thread, the row's values in registers, the centroids broadcast
//               from shared memory; the dot products add x_t * c_t in ascending t from
//               zero with FMAs, norms and half norms are summed in the order of the
//               separate kernels: for floats, and for doubles with k <= 32, the same
//               scores, labels and distances bit for bit (wider double problems are
//               scored on the tensor pipe there, in its own order)
//   accumulate  the CTA's rows are listed by label (stable); a thread per (segment of the
//               list, column) sums its runs of equal labels, and a cluster's runs are
//               added in order: float values as the exact integers of the exact update,
//               double values in FP64 in a fixed order
//   barrier
//   finalize    as many lanes per (cluster, column) as CTAs, over the grid: their sums in a fixed
//               order, the new centroid value and its part of the shift
//   barrier
//   decide      every CTA reads the new centroids, counts and shift parts and takes the
//               same decisions; with empty clusters the farthest rows are selected first
//               (two more barriers)
//
// Float centroids equal the general path's bit for bit (exact integers); double sums are
// added in another fixed order. Measured (whole train call, separate kernels -> here): 100 x
// 3, k = 3, double 347 -> 60 us; 100,000 x 20, k = 20, 50 iterations: float 3.4 -> 0.94 ms,
// double 5.8 -> 0.89 ms. There an iteration takes 35,000 cycles: assign 6,700 (float) or
// 12,000 (double), accumulate 14,000 or 9,300, the barriers with their waits 7,000, the
// finalize and the reading back 6,000.
#include "kmb_internal.cuh"

#include <algorithm>
#include <cfloat>
#include <type_traits>

namespace kmb {
namespace {

constexpr int kNT = 512;
constexpr int kNW = kNT / 32;
static_assert(kSmallTrainMaxK <= kNT, "a thread per cluster");

template <typename F> __device__ __forceinline__ F inf_of();
template <> __device__ __forceinline__ float inf_of<float>() { return __int_as_float(0x7f800000); }
template <> __device__ __forceinline__ double inf_of<double>() { return __longlong_as_double(0x7ff0000000000000LL); }

template <typename F> struct Acc;  // a cluster-column sum
template <> struct Acc<float> {
    long long v[3];
};
template <> struct Acc<double> {
    double v[1];
};
template <typename F> constexpr int planes_of() { return (int)(sizeof(Acc<F>) / 8); }

struct SmallCand {
    unsigned long long key;
    long long row;
};

template <typename F>
struct SmallArgs {
    const F *X, *C0;
    F *C_out;          // k x d
    int32_t *labels;
    int64_t n;
    int d, k;
    int rows;          // rows per CTA
    int64_t T;         // iterations at most
    double eps;
    int runs;          // the runs of equal labels fit shared memory
    int final_pass;    // responses under the final centroids and the objective
    SmallOut *out;     // cleared before the launch, as is colbits
    unsigned *colbits; // d (float): column maxima as float bits
    unsigned long long *part;  // [plane][cell][CTA] limb sums or doubles
    int *part_cnt;     // [cluster][CTA]
    F *C_new;          // k x d
    double *dshift;    // k x d
    int *counts;       // k
    SmallCand *cand;   // [CTA][k]
    long long *sel;    // k
    double *obj_part;  // CTA
    long long wait;    // cycles, of every barrier
};

// Segments of the accumulation's row list: a thread per (segment, column).
__host__ __device__ constexpr int small_segments(int d) { return kNT / d < 128 ? kNT / d : 128; }
constexpr size_t kMaxRunBytes = 48 * 1024;

// Shared memory of one CTA, in bytes from the base.
struct SmallLayout {
    int ds, dp;  // row pitch of X (odd), of the centroids (16-byte multiple)
    size_t xs, cs, hs, xn, d2, lab, order, seg, start, red, runs, total;
};

template <typename F>
__host__ __device__ inline SmallLayout small_layout(int rows, int d, int k, int dmax) {
    SmallLayout L;
    L.ds = d | 1;
    L.dp = dmax;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 15) / 16 * 16;
        return at;
    };
    L.cs = take(sizeof(F) * (size_t)((k + 3) / 4 * 4) * dmax);
    L.hs = take(sizeof(F) * (size_t)((k + 3) / 4 * 4));
    L.xs = take(sizeof(F) * (size_t)rows * L.ds);
    L.xn = take(sizeof(F) * (size_t)rows);
    L.d2 = take(sizeof(F) * (size_t)rows);
    L.lab = take(sizeof(int) * (size_t)((rows + 3) / 4 * 4 + 4));
    L.order = take(sizeof(unsigned short) * (size_t)rows);
    L.seg = take(sizeof(int) * kNT);
    L.start = take(sizeof(int) * (size_t)(k + 1));
    L.runs = sizeof(Acc<F>) * (size_t)(small_segments(d) + k) * d;
    L.red = take(L.runs <= kMaxRunBytes ? L.runs : 0);
    L.total = o;
    return L;
}

// Sum over the CTA, the same in every thread.
__device__ __forceinline__ double cta_sum(double v, double *red) {
    for (int m = 16; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double tot = 0.0;
    for (int w = 0; w < kNW; ++w) tot += red[w];
    return tot;
}

// h_j = 0.5 ||c_j||^2 of the centroids in shared memory, one warp per cluster: the sum
// of prep_centroids_kernel (a butterfly per 32 columns, then the groups in order).
template <typename F, int DMAX>
__device__ __forceinline__ void half_norms(const F *Cs, F *hs, int d, int k) {
    const int lane = threadIdx.x & 31;
    for (int j = threadIdx.x >> 5; j < k; j += kNW) {
        double tot = 0.0;
#pragma unroll
        for (int b = 0; b < DMAX; b += 32) {
            const F v = b + lane < d ? Cs[j * DMAX + b + lane] : F(0);
            double s = (double)v * (double)v;
            for (int m = 16; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
            tot += s;
        }
        if (lane == 0) hs[j] = F(0.5 * tot);
    }
}

// Labels and squared distances of the CTA's rows. Bound by the centroid values' way from
// shared memory into registers (128 bytes a cycle and SM, broadcast or not), so a thread
// takes RT = 2 rows where their values fit its registers beside the accumulators and the
// CTA has more rows than threads.
template <typename F, int DMAX>
constexpr int rows_per_thread() { return (int)sizeof(F) * DMAX <= 192 ? 2 : 1; }

template <typename F, int DMAX, int RT>
__device__ __forceinline__ void assign_rows_of(const F *Xs, int ds, const F *Cs, const F *hs, const F *xn, int rows, int d,
                                            int k, int *lab, F *d2) {
    constexpr int V = 16 / (int)sizeof(F);
    constexpr int kBytes = (int)sizeof(F) * DMAX;
    constexpr bool kRegs = kBytes <= 256;                  // wider rows: read from shared memory
    constexpr int Q = sizeof(F) == 8 && RT == 2 ? 2 : 4;   // clusters at a time (independent chains)
    const int step = (rows + RT - 1) / RT;                 // row i of a thread: its first + i * step
    for (int r0 = threadIdx.x; r0 < step; r0 += kNT) {
        F x[RT][kRegs ? DMAX : 1];
        F best[RT];
        int bi[RT], row[RT];
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            row[i] = min(r0 + i * step, rows - 1);  // (a row past the end repeats the last one)
            best[i] = inf_of<F>();
            bi[i] = 0;
            if constexpr (kRegs) {
#pragma unroll
                for (int t = 0; t < DMAX; ++t) x[i][t] = t < d ? Xs[row[i] * ds + t] : F(0);
            }
        }
        for (int j = 0; j < k; j += Q) {  // (clusters past k: zero rows, not used)
            F a[RT][Q];
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int q = 0; q < Q; ++q) a[i][q] = F(0);
#pragma unroll
            for (int t = 0; t < DMAX; t += V) {
                F c[Q][V];
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const F *p = Cs + (size_t)(j + q) * DMAX + t;
                    if constexpr (sizeof(F) == 4) {
                        const float4 u = *reinterpret_cast<const float4 *>(p);
                        c[q][0] = u.x, c[q][1] = u.y, c[q][2] = u.z, c[q][3] = u.w;
                    } else {
                        const double2 u = *reinterpret_cast<const double2 *>(p);
                        c[q][0] = u.x, c[q][1] = u.y;
                    }
                }
#pragma unroll
                for (int v = 0; v < V; ++v)
#pragma unroll
                    for (int i = 0; i < RT; ++i) {
                        F xv;
                        if constexpr (kRegs) xv = x[i][t + v];
                        else xv = t + v < d ? Xs[row[i] * ds + t + v] : F(0);
#pragma unroll
                        for (int q = 0; q < Q; ++q) a[i][q] = fma(xv, c[q][v], a[i][q]);
                    }
            }
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const F v = hs[j + q] - a[i][q];
                    if (j + q < k && v < best[i]) {
                        best[i] = v;
                        bi[i] = j + q;
                    }
                }
        }
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            lab[row[i]] = bi[i];
            d2[row[i]] = F(2) * best[i] + xn[row[i]];
        }
    }
}

template <typename F, int DMAX>
__device__ __forceinline__ void assign_rows(const F *Xs, int ds, const F *Cs, const F *hs, const F *xn, int rows, int d,
                                            int k, int *lab, F *d2) {
    if (rows_per_thread<F, DMAX>() == 2 && rows > kNT)
        assign_rows_of<F, DMAX, rows_per_thread<F, DMAX>()>(Xs, ds, Cs, hs, xn, rows, d, k, lab, d2);
    else
        assign_rows_of<F, DMAX, 1>(Xs, ds, Cs, hs, xn, rows, d, k, lab, d2);
}

// order[start[j] .. start[j + 1]): the CTA's rows with label j, ascending.
__device__ __forceinline__ void list_rows(const int *lab, int rows, int k, unsigned short *order, int *seg, int *start) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int nseg = min(32, kNT / k);  // k <= kSmallTrainMaxK <= kNT
    const int L = ((rows + nseg - 1) / nseg + 3) & ~3;  // rows per segment, whole int4s
    // thread (segment s, cluster j) counts, then lists, its segment's rows of j
    const int j = tid % k, s = tid / k, e = min(rows, (s + 1) * L);
    const bool user = tid < k * nseg;
    if (user) {
        int c = 0;
        for (int r = s * L; r < e; r += 4) {
            const int4 q = *reinterpret_cast<const int4 *>(lab + r);  // (entries past rows are -1)
            c += (q.x == j) + (q.y == j) + (q.z == j) + (q.w == j);
        }
        seg[s * k + j] = c;
    }
    __syncthreads();
    if (tid < 32) {  // start: exclusive scan of the clusters' totals, one warp
        int run = 0;
        for (int j0 = 0; j0 < k; j0 += 32) {
            const int jj = j0 + lane;
            int c = 0;
            if (jj < k)
                for (int s2 = 0; s2 < nseg; ++s2) c += seg[s2 * k + jj];
            int inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
            if (jj < k) start[jj] = run + inc - c;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) start[k] = run;
    }
    __syncthreads();
    if (user) {
        int at = start[j];
        for (int s2 = 0; s2 < s; ++s2) at += seg[s2 * k + j];
        for (int r = s * L; r < e; r += 4) {
            const int4 q = *reinterpret_cast<const int4 *>(lab + r);
            if (q.x == j) order[at++] = (unsigned short)r;
            if (q.y == j) order[at++] = (unsigned short)(r + 1);
            if (q.z == j) order[at++] = (unsigned short)(r + 2);
            if (q.w == j) order[at++] = (unsigned short)(r + 3);
        }
    }
    __syncthreads();
}

// out[0, have): the CTA's rows with the largest d2, in (d2 descending, row ascending) order;
// 1 <= have <= min(rows, k). A radix select of the have-th row, eight bits a round over the
// distance's ordered key and then over the row (it ends once a whole bin is taken), the
// chosen rows listed in any order, and a rank of each in that list. Bound by the reads of d2,
// a few a row. Comparing every row with every other took 8.2 ms at 12,000 rows a CTA and 3.2 ms at
// 7,400 (148 CTAs), one empty cluster; 13 and 10 us here. `seg`: kNT ints of scratch.
template <typename F>
__device__ void farthest_rows(const F *d2, int rows, int have, int64_t row0, int *seg, SmallCand *out) {
    static_assert(kNT >= 256 + kSmallTrainMaxK, "bins and chosen rows");
    int *bins = seg, *chosen = seg + 256;
    __shared__ int s_bin, s_need, s_all, s_at;
    constexpr int KD = (int)sizeof(F);  // digits of the key; two more of the row
    const int tid = threadIdx.x, lane = tid & 31;
    const int rounds = (rows + kNT - 1) / kNT * kNT;  // (whole warps stay together)
    unsigned long long key_low = 0;  // the smallest key that can still be the have-th row's
    unsigned row_low = 0;            // and, at that key, the smallest 0xffff - row
    int need = have;
    for (int q = 0; q < KD + 2; ++q) {
        const int ks = 8 * (KD - 1 - q), rs = 8 * (KD + 1 - q);  // this digit's place in the key, in the row
        for (int i = tid; i < 256; i += kNT) bins[i] = 0;
        __syncthreads();
        for (int r = tid; r < rounds; r += kNT) {
            bool in = r < rows;
            unsigned digit = 0;
            if (in) {
                const unsigned long long key = order_key(d2[r]);
                const unsigned inv = 0xffffu - (unsigned)r;
                if (q < KD) {
                    in = ((key ^ key_low) >> ks) >> 8 == 0;
                    digit = (unsigned)(key >> ks) & 0xffu;
                } else {
                    in = key == key_low && ((inv ^ row_low) >> rs) >> 8 == 0;
                    digit = (inv >> rs) & 0xffu;
                }
            }
            const unsigned votes = __ballot_sync(0xffffffffu, in);
            if (votes == 0) continue;
            const unsigned first = __shfl_sync(0xffffffffu, digit, __ffs(votes) - 1);
            if (__all_sync(0xffffffffu, !in || digit == first)) {  // (the leading digits mostly agree)
                if (lane == 0) atomicAdd(&bins[first], __popc(votes));
            } else if (in) {
                atomicAdd(&bins[digit], 1);
            }
        }
        __syncthreads();
        if (tid < 32) {  // the bin of the need-th row: eight bins a lane, the highest first
            int c[8], sum = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) sum += c[i] = bins[255 - 8 * lane - i];
            int before = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += t;
            }
            before -= sum;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (before < need && before + c[i] >= need) {
                    s_bin = 255 - 8 * lane - i;
                    s_need = need - before;
                    s_all = c[i] == need - before;
                }
                before += c[i];
            }
            if (lane == 0) s_at = 0;
        }
        __syncthreads();
        need = s_need;
        if (q < KD) key_low |= (unsigned long long)s_bin << ks;
        else row_low |= (unsigned)s_bin << rs;
        if (s_all) break;  // (uniform; the next writes of s_* lie behind a barrier)
    }
    for (int r = tid; r < rows; r += kNT) {
        const unsigned long long key = order_key(d2[r]);
        if (key > key_low || (key == key_low && 0xffffu - (unsigned)r >= row_low)) chosen[atomicAdd(&s_at, 1)] = r;
    }
    __syncthreads();
    for (int e = tid; e < have; e += kNT) {
        const int r = chosen[e];
        const unsigned long long key = order_key(d2[r]);
        int rank = 0;
        for (int i = 0; i < have; ++i) {
            const int o = chosen[i];
            const unsigned long long ok = order_key(d2[o]);
            rank += ok > key || (ok == key && o < r);
        }
        out[rank] = SmallCand{key, (long long)(row0 + r)};
    }
}

__device__ __forceinline__ void acc_add(Acc<float> &a, float x, int e) {
    const Limbs L = fixed_of(x, e);
    a.v[0] += L.l0;
    a.v[1] += L.l1;
    a.v[2] += L.l2;
}
__device__ __forceinline__ void acc_add(Acc<double> &a, double x, int) { a.v[0] += x; }

// The centroid value of summed parts.
__device__ __forceinline__ float centroid_of(const Acc<float> &a, int e, int count) {
    const __int128 S = ((__int128)a.v[2] << 64) + ((__int128)a.v[1] << 32) + (__int128)a.v[0];
    const double Sd = S < 0 ? -u128_to_double((unsigned __int128)(-S)) : u128_to_double((unsigned __int128)S);
    return (float)(ldexp(Sd, -e) / (double)count);
}
__device__ __forceinline__ double centroid_of(const Acc<double> &a, int, int count) {
    return a.v[0] / (double)count;
}

template <typename F, int DMAX>
__global__ void __launch_bounds__(kNT, 1) small_train_kernel(const SmallArgs<F> a) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    constexpr int NP = planes_of<F>();
    const int d = a.d, k = a.k;
    const SmallLayout L = small_layout<F>(a.rows, d, k, DMAX);
    F *Cs = (F *)(small_smem + L.cs), *hs = (F *)(small_smem + L.hs), *Xs = (F *)(small_smem + L.xs);
    F *xn = (F *)(small_smem + L.xn), *d2 = (F *)(small_smem + L.d2);
    int *lab = (int *)(small_smem + L.lab), *seg = (int *)(small_smem + L.seg), *start = (int *)(small_smem + L.start);
    unsigned short *order = (unsigned short *)(small_smem + L.order);
    Acc<F> *red = (Acc<F> *)(small_smem + L.red);
    __shared__ double s_red[kNW];
    __shared__ int s_exp[DMAX];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = gridDim.x, b = blockIdx.x;
    const int ds = L.ds, cells = k * d;
    const int64_t row0 = (int64_t)b * a.rows;
    const int rows = (int)max((int64_t)0, min((int64_t)a.rows, a.n - row0));
    const int k4 = (k + 3) / 4 * 4;

    // the CTA's rows and the initial centroids into shared memory
    int infinite = 0;
    for (int64_t i = tid; i < (int64_t)rows * d; i += kNT) {
        const int r = (int)(i / d), t = (int)(i - (int64_t)r * d);
        const F x = a.X[row0 * d + i];
        Xs[r * ds + t] = x;
        infinite |= !isfinite(x);
    }
    // (the bins take finite values of a finite column, e != 0; fixed_of takes the others)
    const bool finite = __syncthreads_or(infinite) == 0;
    for (int i = tid; i < k4 * DMAX; i += kNT) {
        const int j = i / DMAX, t = i % DMAX;
        Cs[i] = (j < k && t < d) ? a.C0[j * d + t] : F(0);
    }
    for (int j = k + tid; j < k4; j += kNT) hs[j] = F(0);
    for (int r = rows + tid; r < (a.rows + 3) / 4 * 4 + 4; r += kNT) lab[r] = -1;
    __syncthreads();
    for (int r = warp; r < rows; r += kNW) {  // ||x||^2 in the order of row_norms_kernel
        double s = 0.0;
        for (int t = lane; t < d; t += 32) {
            const double v = (double)Xs[r * ds + t];
            s += v * v;
        }
        for (int m = 16; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
        if (lane == 0) xn[r] = F(s);
    }
    GridSync *sync = &a.out->sync;
    unsigned arrived = 0;
    bool ok = true;
    if (sizeof(F) == 4 && a.T > 0) {  // column exponents of the exact sums
        for (int t = warp; t < d; t += kNW) {
            float m = 0.f;
            for (int r = lane; r < rows; r += 32) {
                const float v = fabsf((float)Xs[r * ds + t]);
                if (v > m) m = v;
            }
            for (int o = 16; o >= 1; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane == 0 && m > 0.f) atomicMax(&a.colbits[t], __float_as_uint(m));
        }
        ok = grid_sync(sync, arrived, a.wait);
        for (int t = tid; t < d; t += kNT) {
            const unsigned bits = __ldcg(a.colbits + t);
            const float m = __uint_as_float(bits);
            int e = 0;
            if (bits != 0u && isfinite(m)) {
                int ex;
                frexpf(m, &ex);  // m < 2^ex
                e = kExactMaxBits - ex;
            }
            s_exp[t] = e;
        }
    }
    half_norms<F, DMAX>(Cs, hs, d, k);
    __syncthreads();

    int64_t iterations = 0, events = 0;
    double shift = 0.0;
    int n_empty = 0;
    bool done = false;
    // Sums by runs: the listed rows are cut into nseg equal segments, a thread per (segment,
    // column) sums the runs of equal labels in its segment, and a cluster's runs are added
    // in order. Run (segment p, cluster j) has the number p + j: both only grow along the
    // list, so the numbers are distinct. Without room for the runs, a thread per (cluster,
    // column) sums the whole list (a large cluster's list is then one thread's).
    const int nseg = small_segments(d);
    const int seg_rows = (rows + nseg - 1) / nseg;
    const bool runs = a.runs != 0;
    // the finalize takes 2^lg lanes a cell: as many as there are CTAs, a warp at most
    int lg = 0;
    while (lg < 5 && 1 << lg < G) ++lg;
    while (ok && !done && iterations < a.T) {
        assign_rows<F, DMAX>(Xs, ds, Cs, hs, xn, rows, d, k, lab, d2);
        __syncthreads();
        list_rows(lab, rows, k, order, seg, start);
        auto sum_span = [&](int i, int hi, int t) {  // listed rows [i, hi) of column t
            Acc<F> v = {};
            const int e = sizeof(F) == 4 ? s_exp[t] : 0;
            if constexpr (sizeof(F) == 4) {
                if (finite && e != 0) {
                    const Bins::Magic mg(e);
                    Bins bins;
                    for (; i + 4 <= hi; i += 4) {
                        F x[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) x[q] = Xs[order[i + q] * ds + t];
#pragma unroll
                        for (int q = 0; q < 4; ++q) bins.add(x[q], mg);
                    }
                    for (; i < hi; ++i) bins.add(Xs[order[i] * ds + t], mg);
                    const Limbs l = bins.limbs(e);
                    return Acc<float>{{l.l0, l.l1, l.l2}};
                }
            }
            for (; i + 4 <= hi; i += 4) {
                F x[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) x[q] = Xs[order[i + q] * ds + t];
#pragma unroll
                for (int q = 0; q < 4; ++q) acc_add(v, x[q], e);
            }
            for (; i < hi; ++i) acc_add(v, Xs[order[i] * ds + t], e);
            return v;
        };
        if (runs) {
            if (tid < nseg * d) {
                const int p = tid / d, t = tid - p * d;
                int i = p * seg_rows;
                const int hi = min(rows, i + seg_rows);
                int j = 0, up = k;  // the cluster of list position i: start[j] <= i < start[j + 1]
                while (up - j > 1) {
                    const int mid = (j + up) >> 1;
                    if (start[mid] <= i) j = mid;
                    else up = mid;
                }
                while (i < hi) {
                    const int end = min(hi, start[j + 1]);
                    if (end > i) red[(p + j) * d + t] = sum_span(i, end, t);
                    i = end;
                    ++j;
                }
            }
            __syncthreads();
        }
        for (int cell = tid; cell < cells; cell += kNT) {
            const int j = cell / d, t = cell - j * d;
            Acc<F> s = {};
            if (runs) {
                if (start[j + 1] > start[j]) {
                    const int p1 = (start[j + 1] - 1) / seg_rows;
                    for (int p = start[j] / seg_rows; p <= p1; ++p)
#pragma unroll
                        for (int l = 0; l < NP; ++l) s.v[l] += red[(p + j) * d + t].v[l];
                }
            } else {
                s = sum_span(start[j], start[j + 1], t);
            }
#pragma unroll
            for (int l = 0; l < NP; ++l)
                a.part[((size_t)l * cells + cell) * G + b] = *reinterpret_cast<unsigned long long *>(&s.v[l]);
        }
        for (int j = tid; j < k; j += kNT) a.part_cnt[(size_t)j * G + b] = start[j + 1] - start[j];
        if (!(ok = grid_sync(sync, arrived, a.wait))) break;
        // finalize over the grid (256 x 64, k = 256, one CTA: 1460 us a train with a warp per
        // cell, 235 us with a thread)
        auto finalize = [&](auto whole) {  // whole: a warp a cell, known at compile time
            constexpr bool W = decltype(whole)::value;
            const int per = W ? 1 : 32 >> lg, sub = W ? lane : lane & ((1 << lg) - 1);
            for (int first = (b * kNW + warp) * per; first < cells; first += G * kNW * per) {
                const int cell = W ? first : first + (lane >> lg);
                const bool in = W || cell < cells;
                const int j = in ? cell / d : 0, t = in ? cell - j * d : 0;
                Acc<F> s = {};
                int cnt = 0;
                for (int c0 = sub; c0 < G; c0 += 5 * 32) {  // five CTAs' loads in flight per lane
                    unsigned long long v[5][NP];
                    int n5[5];
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        const int c = c0 + 32 * q;
                        n5[q] = in && c < G ? __ldcg(a.part_cnt + (size_t)j * G + c) : 0;
#pragma unroll
                        for (int l = 0; l < NP; ++l)
                            v[q][l] = in && c < G ? __ldcg(a.part + ((size_t)l * cells + cell) * G + c) : 0ull;  // (0.0 too)
                    }
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        cnt += n5[q];
#pragma unroll
                        for (int l = 0; l < NP; ++l) s.v[l] += *reinterpret_cast<const decltype(s.v[0] + 0) *>(&v[q][l]);
                    }
                }
#pragma unroll
                for (int m = 16; m >= 1; m >>= 1) {
                    if (!W && m >> lg) continue;
#pragma unroll
                    for (int l = 0; l < NP; ++l) s.v[l] += __shfl_xor_sync(0xffffffffu, s.v[l], m);
                    cnt += __shfl_xor_sync(0xffffffffu, cnt, m);
                }
                if (in && sub == 0) {
                    const F old = Cs[j * DMAX + t];
                    const F c = cnt > 0 ? centroid_of(s, sizeof(F) == 4 ? s_exp[t] : 0, cnt) : old;
                    const double df = (double)old - (double)c;
                    a.C_new[cell] = c;
                    a.dshift[cell] = cnt > 0 ? df * df : 0.0;
                    if (t == 0) a.counts[j] = cnt;
                }
            }
        };
        if (lg == 5) finalize(std::true_type());
        else finalize(std::false_type());
        if (!(ok = grid_sync(sync, arrived, a.wait))) break;
        // every CTA: the new centroids, the shift, the empty clusters
        double part = 0.0;
        for (int i = tid; i < cells; i += kNT) {
            const int j = i / d, t = i - j * d;
            Cs[j * DMAX + t] = __ldcg(a.C_new + i);
            part += __ldcg(a.dshift + i);
        }
        shift = cta_sum(part, s_red);
        const int ne = __syncthreads_count(tid < k && __ldcg(a.counts + tid) == 0);
        n_empty = ne;
        if (ne > 0) {
            // this CTA's farthest rows in order, then the grid's, by a rank over the CTAs' lists
            const int have = min(ne, rows);
            SmallCand *mine = a.cand + (size_t)b * k;
            farthest_rows(d2, rows, have, row0, seg, mine);
            if (!(ok = grid_sync(sync, arrived, a.wait))) break;
            for (int e = warp; e < have; e += kNW) {
                const unsigned long long key = __ldcg(&mine[e].key);
                const long long row = __ldcg(&mine[e].row);
                int before = 0;
                for (int c = lane; c < G; c += 32) {
                    const int64_t crows = min((int64_t)a.rows, a.n - (int64_t)c * a.rows);
                    const SmallCand *list = a.cand + (size_t)c * k;
                    int lo = 0, hi = (int)max((int64_t)0, min((int64_t)ne, crows));  // entries before (key, row)
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        const unsigned long long o = __ldcg(&list[mid].key);
                        if (o > key || (o == key && __ldcg(&list[mid].row) < row))
                            lo = mid + 1;
                        else
                            hi = mid;
                    }
                    before += lo;
                }
                before = __reduce_add_sync(0xffffffffu, before);
                if (lane == 0 && before < ne) a.sel[before] = row;
            }
            if (!(ok = grid_sync(sync, arrived, a.wait))) break;
            if (warp == 0) {  // the empty clusters' ids, ascending, in seg
                int base = 0;
                for (int j0 = 0; j0 < k; j0 += 32) {
                    const int j = j0 + lane;
                    const bool em = j < k && __ldcg(a.counts + j) == 0;
                    const unsigned votes = __ballot_sync(0xffffffffu, em);
                    if (em) seg[base + __popc(votes & ((1u << lane) - 1u))] = j;
                    base += __popc(votes);
                }
            }
            __syncthreads();
            part = 0.0;
            for (int i = tid; i < ne * d; i += kNT) {
                const int e = i / d, t = i - e * d, id = seg[e];
                const F x = a.X[__ldcg(a.sel + e) * d + t];
                const double df = (double)Cs[id * DMAX + t] - (double)x;
                part += df * df;
                Cs[id * DMAX + t] = x;
            }
            shift += cta_sum(part, s_red);
            events += ne;
        }
        __syncthreads();
        half_norms<F, DMAX>(Cs, hs, d, k);
        __syncthreads();
        ++iterations;
        done = shift <= a.eps;
    }
    double objective = 0.0;
    if (ok && a.final_pass) {
        assign_rows<F, DMAX>(Xs, ds, Cs, hs, xn, rows, d, k, lab, d2);
        __syncthreads();
        double s = 0.0;
        for (int r = tid; r < rows; r += kNT) {
            const F *c = Cs + lab[r] * DMAX;
            for (int t = 0; t < d; ++t) {
                const double df = (double)Xs[r * ds + t] - (double)c[t];
                s += df * df;
            }
        }
        s = cta_sum(s, s_red);
        if (tid == 0) a.obj_part[b] = s;
        ok = grid_sync(sync, arrived, a.wait);
        if (ok && b == 0) {
            double v = 0.0;
            for (int c = tid; c < G; c += kNT) v += __ldcg(a.obj_part + c);
            objective = cta_sum(v, s_red);
        }
    }
    if (ok && a.labels && (a.final_pass || iterations > 0))
        for (int r = tid; r < rows; r += kNT) a.labels[row0 + r] = lab[r];
    if (b == 0) {
        if (ok)
            for (int i = tid; i < cells; i += kNT) a.C_out[i] = Cs[i / d * DMAX + i % d];
        if (tid == 0) {
            LoopState z = {};
            z.done = done;
            z.iterations = (int)iterations;
            z.n_empty = n_empty;
            z.empty_events = events;
            z.shift = shift;
            z.eps = a.eps;
            z.objective = objective;
            a.out->st = z;
        }
    }
}

int dmax_of(int64_t d) {
    for (int m : {4, 8, 16, 24, 32, 48, 64})
        if (d <= m) return m;
    return 0;
}

template <typename F>
const void *kernel_of(int dmax) {
    switch (dmax) {
        case 4: return (const void *)small_train_kernel<F, 4>;
        case 8: return (const void *)small_train_kernel<F, 8>;
        case 16: return (const void *)small_train_kernel<F, 16>;
        case 24: return (const void *)small_train_kernel<F, 24>;
        case 32: return (const void *)small_train_kernel<F, 32>;
        case 48: return (const void *)small_train_kernel<F, 48>;
        default: return (const void *)small_train_kernel<F, 64>;
    }
}

}  // namespace

template <typename F>
SmallPlan make_small_plan(int64_t n, int64_t d, int64_t k, int sms) {
    SmallPlan p;
    const int dmax = dmax_of(d);
    if (dmax == 0 || k > kSmallTrainMaxK || n > INT32_MAX || n * k * d > kSmallTrainMacs) return p;
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    optin -= 2048;  // static shared memory
    // A row's k * d products are one thread's work, so a wide problem of few rows leaves most of
    // the chip idle here, and the general path is the better one (train of 10 iterations there
    // and here, us): floats and doubles of d <= 32, whose row is in registers, 1000 x 64, k = 256
    // 519 and 820, 4000 x 64, k = 256 502 and 490, 1000 x 64, k = 160 460 and 448; wider doubles
    // 4000 x 48, k = 128 503 and 399, 4000 x 64, k = 128 565 and 638, k = 256 570 and 982.
    const int64_t kd = k * d;
    if (sizeof(F) * dmax <= 256 ? kd > 10240 && n < 4096 : kd > 6144) return p;
    // One CTA of at most a row per thread while it does an iteration's work in about the time
    // that barriers and the exchange take (300 x 1, k = 3 113 us, in two CTAs 125; 400 x 64,
    // k = 10 149 and 126). Else blocks of 256 rows over the SMs, or, up to 125 CTAs, of fewer
    // rows, 2^19 multiply-adds an iteration but 64 rows at least (3000 x 60, k = 100 361 us by
    // 256 rows, 287 by 87; past 125 the exchange outweighs: 8000 x 64, k = 256 460 us in 125
    // CTAs, 496 in 148; and 32,000 x 64, k = 256 1140 us in 125, 1340 in 128, whose strides of
    // 1 KB fall on few L2 slices).
    const int64_t light = std::max<int64_t>(64, (1 << 19) / kd);
    int64_t ctas = 1;
    if (n > kNT || n * kd > 1 << 17)
        ctas = std::min<int64_t>(sms, std::max((n + 255) / 256, std::min<int64_t>(125, (n + light - 1) / light)));
    for (;;) {
        const int64_t rows = (n + ctas - 1) / ctas;
        if (rows <= 65535 && small_layout<F>((int)rows, (int)d, (int)k, dmax).total <= (size_t)optin) {
            p.rows = (int)rows;
            p.ctas = (int)((n + rows - 1) / rows);
            return p;
        }
        if (ctas == sms) return p;  // the rows do not fit the chip's shared memory
        ctas = std::min<int64_t>(sms, ctas * 2);
    }
}

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Scratch: the results, the barrier and the column maxima first (cleared before every launch).
static size_t small_head(int64_t d) { return align256(sizeof(SmallOut)) + align256(sizeof(unsigned) * d); }

template <typename F>
size_t small_scratch_bytes(const SmallPlan &p, int64_t d, int64_t k) {
    const size_t cells = (size_t)k * d, G = p.ctas;
    return small_head(d) + align256(sizeof(Acc<F>) * cells * G) + align256(sizeof(int) * k * G) +
           align256(sizeof(F) * cells) + align256(sizeof(double) * cells) + align256(sizeof(int) * k) +
           align256(sizeof(SmallCand) * k * G) + align256(sizeof(long long) * k) + align256(sizeof(double) * G);
}

template <typename F>
cudaError_t launch_small_train(const SmallPlan &p, const F *X, int64_t n, int64_t d, const F *C0, int64_t k, int64_t T,
                               double eps, bool final_pass, F *C_out, int32_t *labels, void *scratch, cudaStream_t s) {
    const int dmax = dmax_of(d);
    const size_t cells = (size_t)k * d, G = p.ctas;
    unsigned char *q = (unsigned char *)scratch;
    auto take = [&](size_t bytes) {
        unsigned char *at = q;
        q += align256(bytes);
        return (void *)at;
    };
    SmallArgs<F> a;
    a.X = X;
    a.C0 = C0;
    a.C_out = C_out;
    a.labels = labels;
    a.n = n;
    a.d = (int)d;
    a.k = (int)k;
    a.rows = p.rows;
    a.T = T;
    a.eps = eps;
    a.runs = small_layout<F>(p.rows, (int)d, (int)k, dmax).runs <= kMaxRunBytes;
    a.final_pass = final_pass ? 1 : 0;
    a.out = (SmallOut *)take(sizeof(SmallOut));
    a.colbits = (unsigned *)take(sizeof(unsigned) * d);
    a.part = (unsigned long long *)take(sizeof(Acc<F>) * cells * G);
    a.part_cnt = (int *)take(sizeof(int) * k * G);
    a.C_new = (F *)take(sizeof(F) * cells);
    a.dshift = (double *)take(sizeof(double) * cells);
    a.counts = (int *)take(sizeof(int) * k);
    a.cand = (SmallCand *)take(sizeof(SmallCand) * k * G);
    a.sel = (long long *)take(sizeof(long long) * k);
    a.obj_part = (double *)take(sizeof(double) * G);
    a.wait = grid_wait_cycles();
    cudaError_t e = cudaMemsetAsync(scratch, 0, small_head(d), s);
    if (e != cudaSuccess) return e;
    const size_t smem = small_layout<F>(p.rows, (int)d, (int)k, dmax).total;
    const void *kern = kernel_of<F>(dmax);
    if ((e = allow_smem(kern)) != cudaSuccess) return e;
    void *args[] = {&a};
    e = cudaLaunchCooperativeKernel(kern, dim3((unsigned)p.ctas), dim3(kNT), args, smem, s);
    if (e == cudaSuccess) KMB_LAUNCHED();
    return e;
}

#define KMB_SMALL_INST(F)                                                                                             \
    template SmallPlan make_small_plan<F>(int64_t, int64_t, int64_t, int);                                               \
    template size_t small_scratch_bytes<F>(const SmallPlan &, int64_t, int64_t);                                      \
    template cudaError_t launch_small_train<F>(const SmallPlan &, const F *, int64_t, int64_t, const F *, int64_t,    \
                                               int64_t, double, bool, F *, int32_t *, void *, cudaStream_t);
KMB_SMALL_INST(float)
KMB_SMALL_INST(double)
#undef KMB_SMALL_INST

}  // namespace kmb

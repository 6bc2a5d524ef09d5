// ensemble.cu — per-node statistics of an ensemble of realizations, on the
// device: mean, variance, empirical cdf / ccdf at thresholds and quantiles.
//
// Replaces the reference's Ensemble statistics (src/ensembles.jl:42-52,
// reduced per node by ereduce, :76-85): mean, var (Statistics.var, corrected:
// divides by R - 1), cdf(e, x) = count(<= x) / R, ccdf(e, x) = count(> x) / R,
// quantile(e, p) = Statistics.quantile of the node's R values (the default
// definition: linear interpolation between order statistics, h = (R - 1) p,
// x[floor h] + (h - floor h) (x[floor h + 1] - x[floor h]) on the sorted
// values).  The realizations stay in HBM: the values are the node-major rows
// sgs_plan_simulate_device / sgs_batch_simulate_device write (row of R
// values, row stride >= R, float or double, centred), and `offset` (the
// process mean) is added to every value.
//
// FP64 values: one warp per node, sums in FP64, quantiles by a sort in shared
// memory (bitonic, R <= 1024).  Rows of float, which the FP32 sweep writes,
// have forms of their own below that keep off the FP64 pipe (a warp FP64
// instruction holds its scheduler for 64 cycles): exact sums in integers,
// sorting networks in registers, thresholds moved to the floats between which
// they fall.  1M nodes x 100 float values, one GB300: mean and variance 4.57
// -> 0.23 ms, 3 quantiles 4.36 -> 0.30, 3 thresholds 1.79 -> 0.11 (0.06 each
// to read).  Nothing is allocated: the threshold and probability lists (at
// most 32 per launch) travel in the kernel parameters, and the host wrapper
// launches once per 32 of them.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

#include "common.cuh"

namespace sgs {

constexpr int ENS_WARPS = 8;
constexpr int ENS_LIST = 32;
constexpr int ENS_RMAX = 1024;

struct EnsArgs {
    const void* vals;
    int fp64;          // 1: double values, 0: float
    int64_t N;
    int R;
    int stride;        // row stride (elements)
    double offset;
    int nlist;         // entries of `list` used
    int list_stride;   // output row length (all entries of the full list)
    int list0;         // first output column of this launch
    double list[ENS_LIST];   // thresholds or probabilities; float rows' quantiles: the
                             // weight of the upper order statistic, whose lower one is lo
    float tf[ENS_LIST];      // float rows: thresholds as floats
    int lo[ENS_LIST];
};

__device__ __forceinline__ double ens_val(const EnsArgs& a, int64_t g, int r) {
    const int64_t i = g * a.stride + r;
    return (a.fp64 ? reinterpret_cast<const double*>(a.vals)[i] : (double)reinterpret_cast<const float*>(a.vals)[i]) +
           a.offset;
}

__device__ __forceinline__ double ens_warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

__global__ void __launch_bounds__(ENS_WARPS * 32) ens_stats_kernel(const EnsArgs a, double* mean, double* var) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * ENS_WARPS;
    for (int64_t g = (int64_t)blockIdx.x * ENS_WARPS + (threadIdx.x >> 5); g < a.N; g += nw) {
        double s = 0.0;
        for (int r = lane; r < a.R; r += 32) s += ens_val(a, g, r);
        const double m = ens_warp_sum(s) / a.R;
        double q = 0.0;
        for (int r = lane; r < a.R; r += 32) {
            const double d = ens_val(a, g, r) - m;
            q += d * d;
        }
        q = ens_warp_sum(q);
        if (lane == 0) {
            if (mean) mean[g] = m;
            if (var) var[g] = a.R > 1 ? q / (a.R - 1) : nan("");
        }
    }
}

// cdf (complement = 0: count(v <= x) / R) or ccdf (1: count(v > x) / R)
__global__ void __launch_bounds__(ENS_WARPS * 32) ens_cdf_kernel(const EnsArgs a, int complement, double* out) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * ENS_WARPS;
    for (int64_t g = (int64_t)blockIdx.x * ENS_WARPS + (threadIdx.x >> 5); g < a.N; g += nw) {
        int cnt[ENS_LIST];
#pragma unroll
        for (int i = 0; i < ENS_LIST; ++i) cnt[i] = 0;
        for (int r0 = 0; r0 < a.R; r0 += 32) {
            const int r = r0 + lane;
            const bool in = r < a.R;
            const double v = in ? ens_val(a, g, r) : 0.0;
#pragma unroll
            for (int i = 0; i < ENS_LIST; ++i)
                if (i < a.nlist) {
                    const bool c = in && (complement ? v > a.list[i] : v <= a.list[i]);
                    cnt[i] += __popc(__ballot_sync(FULL_MASK, c));
                }
        }
        for (int i = lane; i < a.nlist; i += 32) {
            int c = 0;
#pragma unroll
            for (int j = 0; j < ENS_LIST; ++j)
                if (j == i) c = cnt[j];
            out[g * a.list_stride + a.list0 + i] = (double)c / a.R;
        }
    }
}

// quantiles: the row sorted in shared memory, then linear interpolation
__global__ void __launch_bounds__(ENS_WARPS * 32) ens_quantile_kernel(const EnsArgs a, double* out) {
    extern __shared__ double s_rows[];
    const int lane = threadIdx.x & 31;
    int P = 1;
    while (P < a.R) P <<= 1;
    double* x = s_rows + (size_t)(threadIdx.x >> 5) * P;
    const int64_t nw = (int64_t)gridDim.x * ENS_WARPS;
    for (int64_t g = (int64_t)blockIdx.x * ENS_WARPS + (threadIdx.x >> 5); g < a.N; g += nw) {
        for (int r = lane; r < P; r += 32) x[r] = r < a.R ? ens_val(a, g, r) : INFINITY;
        __syncwarp();
        for (int size = 2; size <= P; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int t = lane; t < (P >> 1); t += 32) {
                    const int i = (t / stride) * stride * 2 + (t % stride);
                    const int j = i + stride;
                    const bool asc = (i & size) == 0;
                    const double xi = x[i], xj = x[j];
                    if ((xi > xj) == asc) {
                        x[i] = xj;
                        x[j] = xi;
                    }
                }
                __syncwarp();
            }
        for (int i = lane; i < a.nlist; i += 32) {
            const double h = (a.R - 1) * a.list[i];
            const double fl = floor(h);
            const int lo = min(max((int)fl, 0), a.R - 1);
            const int hi = min(lo + 1, a.R - 1);
            out[g * a.list_stride + a.list0 + i] = x[lo] + (h - fl) * (x[hi] - x[lo]);
        }
        __syncwarp();
    }
}

// ---- rows of float ----
// LPN lanes per node (8, or 32 for long rows), 32 / LPN nodes per warp; lane q
// holds the values q, q + LPN, ... of the row, V of them at most.
template <int LPN, int V>
__device__ __forceinline__ void ens_load(const float* __restrict__ row, int R, int q, bool in, float pad, float (&x)[V]) {
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] = in && i * LPN + q < R ? row[i * LPN + q] : pad;
}

template <int LPN>
__device__ __forceinline__ long long ens_group_sum(long long v) {
#pragma unroll
    for (int o = LPN / 2; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

template <int LPN>
__device__ __forceinline__ double ens_group_sum(double v) {
#pragma unroll
    for (int o = LPN / 2; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

// What a node's sums are, until 32 nodes are finished together.
struct EnsSums {
    long long s, c, hh, hl, ll;
    int e;  // ENS_DONE: s and hh hold the mean and the sum of squares (FP64)
};
constexpr int ENS_DONE = INT_MIN;
constexpr int ENS_FIXED_MAX = 512;  // values of a row in the integer form

// Mean and variance in integers.  With |x| < 2^e over a row, X = x 2^(51 - e)
// is an integer where no value but 0 is below 2^(e - 28) (whose last bit is
// 2^(e - 51)); sums of at most 512 of them are exact, and so are the three
// partial sums of the squares of X - M, M an integer near the mean, taken as
// 26-bit halves: sum (X - M)^2 = hh 2^52 + 2 hl 2^26 + ll.  The variance is
// the sum less (sum (X - M))^2 / R.  FP64 is left to the last dozen
// operations, for 32 nodes at a time.  Rows with smaller values, infinities, NaN or magnitudes
// beyond 2^60 or below 2^-60 are summed in FP64.
template <int LPN, int V>
__global__ void __launch_bounds__(ENS_WARPS * 32) ens_stats_fixed_kernel(const EnsArgs a, int rounds, double* mean,
                                                                         double* var) {
    __shared__ EnsSums s_sum[ENS_WARPS][32];
    EnsSums* sum = s_sum[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, grp = lane / LPN, q = lane % LPN;
    constexpr int NPW = 32 / LPN;
    const float* vals = reinterpret_cast<const float*>(a.vals);
    const int span = rounds * NPW;  // nodes a warp finishes together
    const int64_t step = (int64_t)gridDim.x * ENS_WARPS * span;
    const float rinv = 1.0f / (float)a.R;
    for (int64_t g0 = ((int64_t)blockIdx.x * ENS_WARPS + (threadIdx.x >> 5)) * span; g0 < a.N; g0 += step) {
        for (int it = 0; it < rounds; ++it) {
            const int64_t g = g0 + it * NPW + grp;
            const float* row = vals + g * a.stride;
            float x[V];
            ens_load<LPN, V>(row, a.R, q, g < a.N, 0.0f, x);
            unsigned mx = 0, mn = ~0u;  // of the magnitudes; the smallest less 1, zeros left out
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const unsigned v = __float_as_uint(x[i]) & 0x7fffffffu;
                mx = max(mx, v);
                mn = min(mn, v - 1);
            }
#pragma unroll
            for (int o = LPN / 2; o > 0; o >>= 1) {
                mx = max(mx, __shfl_xor_sync(FULL_MASK, mx, o));
                mn = min(mn, __shfl_xor_sync(FULL_MASK, mn, o));
            }
            const int e = mx ? (int)(mx >> 23) - 126 : 0;
            // 27 binades below the largest one's at most
            const bool fixed = e >= -60 && e <= 60 && ((mn + 1) >> 23) + 27 >= mx >> 23;
            const float sc = __uint_as_float((unsigned)(127 + 25 - (fixed ? e : 0)) << 23);
            long long X[V], s = 0;
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const float y = __fmul_rn(x[i], sc);
                const int h = __float2int_rn(y);
                const int l = __float2int_rn(__fmul_rn(__fadd_rn(y, -__int2float_rn(h)), 67108864.0f));
                X[i] = (long long)h * (1 << 26) + l;
                s += X[i];
            }
            s = ens_group_sum<LPN>(s);
            const long long M = __float2ll_rn(__fmul_rn((float)s, rinv));
            long long hh = 0, hl = 0, ll = 0;
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const long long d = i * LPN + q < a.R ? X[i] - M : 0;
                const int dh = (int)(d >> 26), dl = (int)d & ((1 << 26) - 1);
                hh += (long long)dh * dh;
                hl += (long long)dh * dl;
                ll += (long long)dl * dl;
            }
            hh = ens_group_sum<LPN>(hh);
            hl = ens_group_sum<LPN>(hl);
            ll = ens_group_sum<LPN>(ll);
            if (q == 0) sum[it * NPW + grp] = {s, s - a.R * M, hh, hl, ll, e};
            if (__any_sync(FULL_MASK, !fixed)) {
                double t = 0.0;
#pragma unroll 1
                for (int r = q; r < a.R && g < a.N; r += LPN) t += ens_val(a, g, r);
                const double m = ens_group_sum<LPN>(t) / a.R;
                t = 0.0;
#pragma unroll 1
                for (int r = q; r < a.R && g < a.N; r += LPN) {
                    const double d = ens_val(a, g, r) - m;
                    t += d * d;
                }
                t = ens_group_sum<LPN>(t);
                if (!fixed && q == 0)
                    sum[it * NPW + grp] = {__double_as_longlong(m), 0, __double_as_longlong(t), 0, 0, ENS_DONE};
            }
        }
        __syncwarp();
        const int64_t g = g0 + lane;
        if (lane < span && g < a.N) {
            const EnsSums v = sum[lane];
            double m, t;
            if (v.e == ENS_DONE) {
                m = __longlong_as_double(v.s);
                t = __longlong_as_double(v.hh);
            } else {
                const double u = __hiloint2double((1023 + v.e - 51) << 20, 0);
                m = (double)v.s / a.R * u + a.offset;
                t = fma((double)v.hh, 4503599627370496.0, fma((double)v.hl, 134217728.0, (double)v.ll));
                const double c = (double)v.c;
                t = fmax(t - c * c / a.R, 0.0) * (u * u);
            }
            if (mean) mean[g] = m;
            if (var) var[g] = a.R > 1 ? t / (a.R - 1) : nan("");
        }
        __syncwarp();
    }
}

// count(x <= t) or, complement, count(x > t) of the floats t in tf: the
// largest for which t + offset <= threshold still holds.
template <int LPN, int LIST>
__global__ void __launch_bounds__(ENS_WARPS * 32) ens_cdf_float_kernel(const __grid_constant__ EnsArgs a, int complement,
                                                                       double* out) {
    extern __shared__ double s_frac[];  // c / R
    for (int c = threadIdx.x; c <= a.R; c += ENS_WARPS * 32) s_frac[c] = (double)c / a.R;
    __syncthreads();
    const int lane = threadIdx.x & 31, grp = lane / LPN, q = lane % LPN;
    constexpr int NPW = 32 / LPN;
    const float* vals = reinterpret_cast<const float*>(a.vals);
    float tf[LIST];
#pragma unroll
    for (int i = 0; i < LIST; ++i) tf[i] = a.tf[i];
    const int64_t step = (int64_t)gridDim.x * ENS_WARPS * NPW;
    for (int64_t g0 = ((int64_t)blockIdx.x * ENS_WARPS + (threadIdx.x >> 5)) * NPW; g0 < a.N; g0 += step) {
        const int64_t g = g0 + grp;
        const float* row = vals + g * a.stride;
        int cnt[LIST];
#pragma unroll
        for (int i = 0; i < LIST; ++i) cnt[i] = 0;
        if (g < a.N)
#pragma unroll 4
            for (int r = q; r < a.R; r += LPN) {
                const float x = row[r];
#pragma unroll
                for (int i = 0; i < LIST; ++i) cnt[i] += complement ? x > tf[i] : x <= tf[i];
            }
#pragma unroll
        for (int o = LPN / 2; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < LIST; ++i) cnt[i] += __shfl_xor_sync(FULL_MASK, cnt[i], o);
        if (g < a.N)
            for (int i = q; i < a.nlist; i += LPN) {
                int c = 0;
#pragma unroll
                for (int j = 0; j < LIST; ++j)
                    if (j == i) c = cnt[j];
                out[g * a.list_stride + a.list0 + i] = s_frac[c];
            }
    }
}

// order-preserving integer of a float (NaN with a clear sign last) and back
__device__ __forceinline__ int ens_key(float x) {
    const int b = __float_as_int(x);
    return b ^ ((b >> 31) & 0x7fffffff);
}

// Quantiles: each row sorted in registers, V keys a lane, by merges that
// compare i with its mirror image in the merged run first (so that every
// comparison keeps the smaller key at the smaller index) and then at halved
// distances; only the last log2(LPN) distances of a merge cross lanes.
template <int LPN, int V>
__global__ void __launch_bounds__(ENS_WARPS * 32) ens_quantile_float_kernel(const __grid_constant__ EnsArgs a,
                                                                            double* out) {
    extern __shared__ int s_keys[];
    const int lane = threadIdx.x & 31, grp = lane / LPN, q = lane % LPN;
    constexpr int NPW = 32 / LPN, P = LPN * V;
    int* sorted = s_keys + (size_t)(threadIdx.x >> 5) * (NPW * (P + 4));
    const float* vals = reinterpret_cast<const float*>(a.vals);
    const int64_t step = (int64_t)gridDim.x * ENS_WARPS * NPW;
    for (int64_t g0 = ((int64_t)blockIdx.x * ENS_WARPS + (threadIdx.x >> 5)) * NPW; g0 < a.N; g0 += step) {
        const int64_t g = g0 + grp;
        float x[V];
        ens_load<LPN, V>(vals + g * a.stride, a.R, q, g < a.N, 0.0f, x);
        int key[V];
#pragma unroll
        for (int i = 0; i < V; ++i) key[i] = i * LPN + q < a.R ? ens_key(x[i]) : INT_MAX;
        auto order = [&](int i, int j) {
            const int lo = min(key[i], key[j]), hi = max(key[i], key[j]);
            key[i] = lo;
            key[j] = hi;
        };
        // runs within a lane
#pragma unroll
        for (int size = 2; size <= V; size <<= 1) {
#pragma unroll
            for (int i = 0; i < V; ++i)
                if ((i & (size / 2)) == 0) order(i, i ^ (size - 1));
#pragma unroll
            for (int d = size / 4; d > 0; d >>= 1)
#pragma unroll
                for (int i = 0; i < V; ++i)
                    if ((i & d) == 0) order(i, i ^ d);
        }
        // runs across lanes
#pragma unroll
        for (int size = 2; size <= LPN; size <<= 1) {  // lanes merged
            {
                const bool low = (q & (size / 2)) == 0;
                int y[V];
#pragma unroll
                for (int i = 0; i < V; ++i) y[i] = __shfl_xor_sync(FULL_MASK, key[V - 1 - i], size - 1);
#pragma unroll
                for (int i = 0; i < V; ++i) key[i] = (y[i] < key[i]) == low ? y[i] : key[i];
            }
#pragma unroll
            for (int d = size / 4; d > 0; d >>= 1) {
                const bool low = (q & d) == 0;
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const int y = __shfl_xor_sync(FULL_MASK, key[i], d);
                    key[i] = (y < key[i]) == low ? y : key[i];
                }
            }
#pragma unroll
            for (int d = V / 2; d > 0; d >>= 1)
#pragma unroll
                for (int i = 0; i < V; ++i)
                    if ((i & d) == 0) order(i, i ^ d);
        }
#pragma unroll
        for (int i = 0; i < V; i += 4)
            *reinterpret_cast<int4*>(sorted + grp * (P + 4) + q * V + i) = make_int4(key[i], key[i + 1], key[i + 2], key[i + 3]);
        __syncwarp();
        for (int t = lane; t < NPW * a.nlist; t += 32) {
            const int gi = t / a.nlist, i = t - gi * a.nlist;
            if (g0 + gi < a.N) {
                const int* srt = sorted + gi * (P + 4);
                const int lo = a.lo[i], hi = min(lo + 1, a.R - 1);
                auto value = [&](int p) {
                    const int b = srt[p];
                    return (double)__int_as_float(b ^ ((b >> 31) & 0x7fffffff)) + a.offset;
                };
                const double vl = value(lo);
                out[(g0 + gi) * a.list_stride + a.list0 + i] = vl + a.list[i] * (value(hi) - vl);
            }
        }
        __syncwarp();
    }
}

}  // namespace sgs

using namespace sgs;

namespace {

int ens_fail(int code, const char* msg) {
    sgs::set_thread_error(msg);
    return code;
}

int ens_args(EnsArgs& a, const void* vals, int32_t precision, int64_t N, int32_t R, int32_t stride, double offset) {
    if (!vals || N < 0 || R < 1 || stride < R) return ens_fail(SGS_ERR_ARG, "invalid ensemble array");
    if (precision != SGS_PREC_FP64 && precision != SGS_PREC_FP32_REFINE) return ens_fail(SGS_ERR_ARG, "unknown precision");
    a = EnsArgs{};
    a.vals = vals;
    a.fp64 = precision == SGS_PREC_FP64;
    a.N = N;
    a.R = R;
    a.stride = stride;
    a.offset = offset;
    return SGS_OK;
}

int ens_grid(int64_t N) {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int64_t want = (N + ENS_WARPS - 1) / ENS_WARPS;
    const int64_t cap = (int64_t)(nsm > 0 ? nsm : 1) * 16;
    return (int)std::max<int64_t>(1, std::min(want, cap));
}

// nodes one warp finishes together (in rounds of npw), fewer where that would
// leave warps without work
int ens_rounds(int64_t N, int lpn) {
    const int npw = 32 / lpn;
    const int64_t warps = (int64_t)ens_grid(INT64_MAX / 2) * ENS_WARPS;
    return (int)std::max<int64_t>(1, std::min<int64_t>(lpn, N / (npw * warps)));
}

// The largest float t with (double)t + offset <= x: (double)t + offset does
// not decrease with t, so x <= threshold can be decided on floats.  NaN where
// nothing compares (x is NaN).
float ens_threshold(double x, double offset) {
    if (std::isnan(x)) return NAN;
    auto value = [](int64_t k) {  // k-th float from -inf = 0 upward
        int32_t b = (int32_t)(k - 0x7f800000);
        b = b < 0 ? (int32_t)(0x80000000u | (uint32_t)-(int64_t)b) : b;
        float f;
        std::memcpy(&f, &b, sizeof(f));
        return f;
    };
    int64_t lo = 0, hi = 2 * (int64_t)0x7f800000;  // -inf + offset <= x always holds
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) / 2;
        if ((double)value(mid) + offset <= x) lo = mid;
        else hi = mid - 1;
    }
    return value(lo);
}

int ens_done(cudaError_t e, const char* where) {
    if (e != cudaSuccess) {
        sgs::set_thread_error(std::string(where) + ": " + cudaGetErrorString(e));
        return SGS_ERR_CUDA;
    }
    return SGS_OK;
}

}  // namespace

extern "C" int sgs_ensemble_stats(const void* vals, int32_t precision, int64_t nnodes, int32_t nreals,
                                  int32_t row_stride, double offset, double* mean, double* var, void* stream) {
    EnsArgs a;
    int rc = ens_args(a, vals, precision, nnodes, nreals, row_stride, offset);
    if (rc) return rc;
    if (!mean && !var) return ens_fail(SGS_ERR_ARG, "no output");
    if (nnodes == 0) return SGS_OK;
    const cudaStream_t st = (cudaStream_t)stream;
    if (!a.fp64 && nreals <= ENS_FIXED_MAX && std::isfinite(offset)) {
        const int lpn = nreals <= 128 ? 8 : 32;
        const int rounds = ens_rounds(nnodes, lpn);
        const int grid = ens_grid((nnodes + rounds * (32 / lpn) - 1) / (rounds * (32 / lpn)));
        if (nreals <= 32) ens_stats_fixed_kernel<8, 4><<<grid, ENS_WARPS * 32, 0, st>>>(a, rounds, mean, var);
        else if (nreals <= 128) ens_stats_fixed_kernel<8, 16><<<grid, ENS_WARPS * 32, 0, st>>>(a, rounds, mean, var);
        else ens_stats_fixed_kernel<32, 16><<<grid, ENS_WARPS * 32, 0, st>>>(a, rounds, mean, var);
    } else {
        ens_stats_kernel<<<ens_grid(nnodes), ENS_WARPS * 32, 0, st>>>(a, mean, var);
    }
    return ens_done(cudaGetLastError(), "sgs_ensemble_stats");
}

extern "C" int sgs_ensemble_cdf(const void* vals, int32_t precision, int64_t nnodes, int32_t nreals,
                                int32_t row_stride, double offset, const double* x, int32_t nx, int32_t complement,
                                double* out, void* stream) {
    EnsArgs a;
    int rc = ens_args(a, vals, precision, nnodes, nreals, row_stride, offset);
    if (rc) return rc;
    if (!x || nx < 1 || !out) return ens_fail(SGS_ERR_ARG, "invalid thresholds or output");
    if (nnodes == 0) return SGS_OK;
    a.list_stride = nx;
    for (int i0 = 0; i0 < nx; i0 += ENS_LIST) {
        a.list0 = i0;
        a.nlist = std::min(ENS_LIST, nx - i0);
        for (int i = 0; i < a.nlist; ++i) a.list[i] = x[i0 + i];
        const cudaStream_t st = (cudaStream_t)stream;
        if (!a.fp64 && nreals <= ENS_RMAX && std::isfinite(offset)) {
            for (int i = 0; i < ENS_LIST; ++i) a.tf[i] = i < a.nlist ? ens_threshold(a.list[i], offset) : 0.0f;
            const size_t smem = (size_t)(nreals + 1) * sizeof(double);
            const int lpn = nreals <= 128 ? 8 : 32;
            const int grid = ens_grid((nnodes + 32 / lpn - 1) / (32 / lpn)), c = complement ? 1 : 0;
            if (lpn == 8 && a.nlist <= 4) ens_cdf_float_kernel<8, 4><<<grid, ENS_WARPS * 32, smem, st>>>(a, c, out);
            else if (lpn == 8) ens_cdf_float_kernel<8, ENS_LIST><<<grid, ENS_WARPS * 32, smem, st>>>(a, c, out);
            else if (a.nlist <= 4) ens_cdf_float_kernel<32, 4><<<grid, ENS_WARPS * 32, smem, st>>>(a, c, out);
            else ens_cdf_float_kernel<32, ENS_LIST><<<grid, ENS_WARPS * 32, smem, st>>>(a, c, out);
        } else {
            ens_cdf_kernel<<<ens_grid(nnodes), ENS_WARPS * 32, 0, st>>>(a, complement ? 1 : 0, out);
        }
        if ((rc = ens_done(cudaGetLastError(), "sgs_ensemble_cdf"))) return rc;
    }
    return SGS_OK;
}

extern "C" int sgs_ensemble_quantile(const void* vals, int32_t precision, int64_t nnodes, int32_t nreals,
                                     int32_t row_stride, double offset, const double* p, int32_t np, double* out,
                                     void* stream) {
    EnsArgs a;
    int rc = ens_args(a, vals, precision, nnodes, nreals, row_stride, offset);
    if (rc) return rc;
    if (!p || np < 1 || !out) return ens_fail(SGS_ERR_ARG, "invalid probabilities or output");
    if (nreals > ENS_RMAX) return ens_fail(SGS_ERR_ARG, "quantiles take at most 1024 realizations");
    for (int i = 0; i < np; ++i)
        if (!(p[i] >= 0.0 && p[i] <= 1.0)) return ens_fail(SGS_ERR_ARG, "probabilities must be in [0, 1]");
    if (nnodes == 0) return SGS_OK;
    a.list_stride = np;
    const cudaStream_t st = (cudaStream_t)stream;
    int P = 1;
    while (P < nreals) P <<= 1;
    for (int i0 = 0; i0 < np; i0 += ENS_LIST) {
        a.list0 = i0;
        a.nlist = std::min(ENS_LIST, np - i0);
        for (int i = 0; i < a.nlist; ++i) a.list[i] = p[i0 + i];
        if (a.fp64) {
            const size_t smem = (size_t)ENS_WARPS * P * sizeof(double);
            // the limit for the longest rows: it is one for all threads of the process
            constexpr int most = ENS_WARPS * ENS_RMAX * (int)sizeof(double);
            if ((rc = ens_done(cudaFuncSetAttribute(ens_quantile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most),
                               "sgs_ensemble_quantile")))
                return rc;
            ens_quantile_kernel<<<ens_grid(nnodes), ENS_WARPS * 32, smem, st>>>(a, out);
        } else {
            for (int i = 0; i < a.nlist; ++i) {
                const double h = (a.R - 1) * a.list[i], fl = std::floor(h);
                a.lo[i] = std::min(std::max((int)fl, 0), a.R - 1);
                a.list[i] = h - fl;
            }
            auto launch = [&](auto kernel, int lpn, int v) {
                const int npw = 32 / lpn;
                const size_t smem = (size_t)ENS_WARPS * npw * (lpn * v + 4) * sizeof(int);
                kernel<<<ens_grid((nnodes + npw - 1) / npw), ENS_WARPS * 32, smem, st>>>(a, out);
            };
            if (nreals <= 32) launch(ens_quantile_float_kernel<8, 4>, 8, 4);
            else if (nreals <= 64) launch(ens_quantile_float_kernel<8, 8>, 8, 8);
            else if (nreals <= 128) launch(ens_quantile_float_kernel<8, 16>, 8, 16);
            else if (nreals <= 256) launch(ens_quantile_float_kernel<32, 8>, 32, 8);
            else if (nreals <= 512) launch(ens_quantile_float_kernel<32, 16>, 32, 16);
            else launch(ens_quantile_float_kernel<32, 32>, 32, 32);
        }
        if ((rc = ens_done(cudaGetLastError(), "sgs_ensemble_quantile"))) return rc;
    }
    return SGS_OK;
}

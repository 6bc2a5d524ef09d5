// sweep.cu — kernel (c): the level-scheduled value sweep over all
// realizations, and the layout conversions around it.
//
// Replaces the draw of randsingle's loop, v = mu_hat + sigma_hat * z
// (src/simulation/field/seqsim.jl:132,335-340, prior :109-111), for every
// realization at once.  Values are centred (v - mu) and node-major,
// V[node][Rp] with realizations contiguous, so one node's update reads each
// grid neighbour's row of realizations with coalesced vector loads:
//   V[g][r] = b0 + sum_j w_j V[nb_j][r] + sigma * z[g][r]
// All nodes of one dependency level are independent.  The default sweep is
// one persistent dataflow launch (sweep_flow_kernel) in which each node waits
// only for its own neighbours; per-level launches and a cooperative launch
// with grid barriers between levels are the alternatives.  The data's fixed
// values enter through b0 (computed by the solve).
#include <algorithm>

#include <cooperative_groups.h>

#include "common.cuh"
#include "flow.cuh"

namespace cg = cooperative_groups;

namespace sgs {

template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
    __device__ static float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
    __device__ static void store(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
};

__device__ __forceinline__ D4 load_d4(const double* p) {
    const double2 a = reinterpret_cast<const double2*>(p)[0];
    const double2 b = reinterpret_cast<const double2*>(p)[1];
    return {a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void store_d4(double* p, D4 v) {
    reinterpret_cast<double2*>(p)[0] = make_double2(settle(v.x), settle(v.y));
    reinterpret_cast<double2*>(p)[1] = make_double2(settle(v.z), settle(v.w));
}

// Compensated dot product in FP32 (Dot2: Ogita, Rump & Oishi 2005, "Accurate
// sum and dot product"): the product w*x is split exactly into p + pe with an
// FMA, p is added to the running sum s with TwoSum (Knuth), and every
// rounding error, plus the low part of the weight, goes into the correction
// c.  s + c carries the dot product to about twice FP32 precision; only the
// final rounding to the stored FP32 value remains.
struct Dot2 {
    float s, c;
    __device__ __forceinline__ void init(float hi, float lo) {
        s = hi;
        c = lo;
    }
    __device__ __forceinline__ void add(float wh, float wl, float x) {
        const float p = __fmul_rn(wh, x);
        const float pe = __fmaf_rn(wh, x, -p);
        const float t = __fadd_rn(s, p);
        const float bp = __fsub_rn(t, s);
        const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(p, bp));
        s = t;
        c = __fadd_rn(c, __fadd_rn(e, __fmaf_rn(wl, x, pe)));
    }
    __device__ __forceinline__ float value() const { return __fadd_rn(s, c); }
};

// Adds another compensated sum (s2, c2) to a (TwoSum of the leading parts).
__device__ __forceinline__ void dot2_merge(Dot2& a, float s2, float c2) {
    const DF t = df_two_sum(a.s, s2);
    a.s = t.hi;
    a.c = __fadd_rn(a.c, __fadd_rn(c2, t.lo));
}

// Update one node's chunk of 4 realizations (FP32 values, compensated sum).
__device__ __forceinline__ void sweep_item_fp32(const SweepTables<float>& t, int k, int64_t pos, int ch, int Rp,
                                                const float* __restrict__ z, uint64_t seed, float* __restrict__ V) {
    const int g = t.node[pos];
    const int m = t.m[pos];
    const float2 b0 = reinterpret_cast<const float2*>(t.b0)[pos];
    Dot2 a0, a1, a2, a3;
    a0.init(b0.x, b0.y);
    a1.init(b0.x, b0.y);
    a2.init(b0.x, b0.y);
    a3.init(b0.x, b0.y);
    const int32_t* idx = t.idx + pos * k;
    const float2* w = reinterpret_cast<const float2*>(t.w) + pos * k;
#pragma unroll 4
    for (int j = 0; j < m; ++j) {
        const float4 v = Vec4<float>::load(V + (int64_t)idx[j] * Rp + 4 * ch);
        const float2 wj = w[j];
        a0.add(wj.x, wj.y, v.x);
        a1.add(wj.x, wj.y, v.y);
        a2.add(wj.x, wj.y, v.z);
        a3.add(wj.x, wj.y, v.w);
    }
    const float4 zz = z ? Vec4<float>::load(z + (int64_t)g * Rp + 4 * ch) : normals4(seed, g, ch);
    const float2 sg = reinterpret_cast<const float2*>(t.sigma)[pos];
    a0.add(sg.x, sg.y, zz.x);
    a1.add(sg.x, sg.y, zz.y);
    a2.add(sg.x, sg.y, zz.z);
    a3.add(sg.x, sg.y, zz.w);
    Vec4<float>::store(V + (int64_t)g * Rp + 4 * ch, make_float4(a0.value(), a1.value(), a2.value(), a3.value()));
}

// Update one node's chunk of 4 realizations (FP64 values).
__device__ __forceinline__ void sweep_item_fp64(const SweepTables<double>& t, int k, int64_t pos, int ch, int Rp,
                                                const double* __restrict__ z, uint64_t seed, double* __restrict__ V) {
    const int g = t.node[pos];
    const int m = t.m[pos];
    const double b0 = t.b0[pos];
    D4 acc = {b0, b0, b0, b0};
    const int32_t* idx = t.idx + pos * k;
    const double* w = t.w + pos * k;
#pragma unroll 4
    for (int j = 0; j < m; ++j) {
        const D4 v = load_d4(V + (int64_t)idx[j] * Rp + 4 * ch);
        const double wj = w[j];
        acc.x = fma(wj, v.x, acc.x);
        acc.y = fma(wj, v.y, acc.y);
        acc.z = fma(wj, v.z, acc.z);
        acc.w = fma(wj, v.w, acc.w);
    }
    D4 zz;
    if (z) {
        zz = load_d4(z + (int64_t)g * Rp + 4 * ch);
    } else {
        const float4 f = normals4(seed, g, ch);
        zz = {(double)f.x, (double)f.y, (double)f.z, (double)f.w};
    }
    const double s = t.sigma[pos];
    acc.x = fma(s, zz.x, acc.x);
    acc.y = fma(s, zz.y, acc.y);
    acc.z = fma(s, zz.z, acc.z);
    acc.w = fma(s, zz.w, acc.w);
    store_d4(V + (int64_t)g * Rp + 4 * ch, acc);
}

// CH consecutive chunks of 4 realizations (ch .. ch + CH - 1 < cpn) of one
// node, FP32: CH independent row loads per neighbour in flight per thread.
template <int CH>
__device__ __forceinline__ void sweep_itemN_fp32(const SweepTables<float>& t, int k, int64_t pos, int ch, int Rp,
                                                 const float* __restrict__ z, uint64_t seed, float* __restrict__ V) {
    const int g = t.node[pos];
    const int m = t.m[pos];
    const float2 b0 = reinterpret_cast<const float2*>(t.b0)[pos];
    Dot2 a[4 * CH];
#pragma unroll
    for (int q = 0; q < 4 * CH; ++q) a[q].init(b0.x, b0.y);
    const int32_t* idx = t.idx + pos * k;
    const float2* w = reinterpret_cast<const float2*>(t.w) + pos * k;
#pragma unroll 4
    for (int j = 0; j < m; ++j) {
        const float* row = V + (int64_t)idx[j] * Rp + 4 * ch;
        float4 v[CH];
#pragma unroll
        for (int h = 0; h < CH; ++h) v[h] = Vec4<float>::load(row + 4 * h);
        const float2 wj = w[j];
#pragma unroll
        for (int h = 0; h < CH; ++h) {
            a[4 * h + 0].add(wj.x, wj.y, v[h].x);
            a[4 * h + 1].add(wj.x, wj.y, v[h].y);
            a[4 * h + 2].add(wj.x, wj.y, v[h].z);
            a[4 * h + 3].add(wj.x, wj.y, v[h].w);
        }
    }
    const float2 sg = reinterpret_cast<const float2*>(t.sigma)[pos];
#pragma unroll
    for (int h = 0; h < CH; ++h) {
        const float4 zz = z ? Vec4<float>::load(z + (int64_t)g * Rp + 4 * (ch + h)) : normals4(seed, g, ch + h);
        a[4 * h + 0].add(sg.x, sg.y, zz.x);
        a[4 * h + 1].add(sg.x, sg.y, zz.y);
        a[4 * h + 2].add(sg.x, sg.y, zz.z);
        a[4 * h + 3].add(sg.x, sg.y, zz.w);
        Vec4<float>::store(V + (int64_t)g * Rp + 4 * (ch + h),
                           make_float4(a[4 * h].value(), a[4 * h + 1].value(), a[4 * h + 2].value(), a[4 * h + 3].value()));
    }
}

// One level per launch, FP32, rows of a multiple of CH chunks: one thread
// per (node, CH consecutive chunks).
template <int CH>
__global__ void __launch_bounds__(256) sweep_levelN_kernel(const SweepTables<float> t, int k, int64_t p0, int64_t p1,
                                                           int Rp, const float* __restrict__ z, uint64_t seed,
                                                           float* __restrict__ V) {
    const int cpg = Rp / (4 * CH);  // chunk groups per node
    const int64_t total = (p1 - p0) * cpg;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x)
        sweep_itemN_fp32<CH>(t, k, p0 + i / cpg, CH * (int)(i % cpg), Rp, z, seed, V);
}

// One level per launch for levels of few nodes (FP32, rows of a multiple of
// 8 realizations): one block per node, its SPLIT_WARPS warps splitting the
// node's neighbour list (warp s takes every SPLIT_WARPS-th neighbour from
// s), each lane 2 chunks of 4 realizations (64 chunks per pass over the
// row), so each thread's chain of dependent row loads is SPLIT_WARPS times
// shorter; warp 0 merges the warps' compensated partial sums (error-free
// TwoSum merges) from shared memory, adds b0 and sigma z and stores.
constexpr int SPLIT_WARPS = 8;

__global__ void __launch_bounds__(SPLIT_WARPS * 32) sweep_split_kernel(const SweepTables<float> t, int k, int64_t p0,
                                                                       int64_t p1, int Rp, const float* __restrict__ z,
                                                                       uint64_t seed, float* __restrict__ V) {
    __shared__ float2 part[SPLIT_WARPS - 1][8][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int cpn = Rp >> 2;
    for (int64_t pos = p0 + blockIdx.x; pos < p1; pos += gridDim.x) {
        const int g = t.node[pos];
        const int m = t.m[pos];
        const int32_t* idx = t.idx + pos * k;
        const float2* w = reinterpret_cast<const float2*>(t.w) + pos * k;
        for (int c0 = 0; c0 < cpn; c0 += 64) {
            const int ch = c0 + 2 * lane;  // chunks ch and ch + 1 (cpn is even)
            const bool act = ch < cpn;
            Dot2 a[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) a[q].init(0.f, 0.f);
            if (act) {
#pragma unroll 2
                for (int j = wid; j < m; j += SPLIT_WARPS) {
                    const float* row = V + (int64_t)idx[j] * Rp + 4 * ch;
                    const float4 v0 = Vec4<float>::load(row);
                    const float4 v1 = Vec4<float>::load(row + 4);
                    const float2 wj = w[j];
                    a[0].add(wj.x, wj.y, v0.x);
                    a[1].add(wj.x, wj.y, v0.y);
                    a[2].add(wj.x, wj.y, v0.z);
                    a[3].add(wj.x, wj.y, v0.w);
                    a[4].add(wj.x, wj.y, v1.x);
                    a[5].add(wj.x, wj.y, v1.y);
                    a[6].add(wj.x, wj.y, v1.z);
                    a[7].add(wj.x, wj.y, v1.w);
                }
            }
            if (wid > 0)
#pragma unroll
                for (int q = 0; q < 8; ++q) part[wid - 1][q][lane] = make_float2(a[q].s, a[q].c);
            __syncthreads();
            if (wid == 0 && act) {
#pragma unroll 1
                for (int s = 0; s < SPLIT_WARPS - 1; ++s)
#pragma unroll
                    for (int q = 0; q < 8; ++q) dot2_merge(a[q], part[s][q][lane].x, part[s][q][lane].y);
                const float2 b0 = reinterpret_cast<const float2*>(t.b0)[pos];
                const float2 sg = reinterpret_cast<const float2*>(t.sigma)[pos];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 zz =
                        z ? Vec4<float>::load(z + (int64_t)g * Rp + 4 * (ch + h)) : normals4(seed, g, ch + h);
#pragma unroll
                    for (int q = 0; q < 4; ++q) dot2_merge(a[4 * h + q], b0.x, b0.y);
                    a[4 * h + 0].add(sg.x, sg.y, zz.x);
                    a[4 * h + 1].add(sg.x, sg.y, zz.y);
                    a[4 * h + 2].add(sg.x, sg.y, zz.z);
                    a[4 * h + 3].add(sg.x, sg.y, zz.w);
                    Vec4<float>::store(V + (int64_t)g * Rp + 4 * (ch + h),
                                       make_float4(a[4 * h].value(), a[4 * h + 1].value(), a[4 * h + 2].value(),
                                                   a[4 * h + 3].value()));
                }
            }
            __syncthreads();
        }
    }
}

// One level per launch: one thread per (node, chunk of 4 realizations).
template <typename T>
__global__ void __launch_bounds__(256) sweep_level_kernel(const SweepTables<T> t, int k, int64_t p0, int64_t p1, int Rp,
                                                          const T* __restrict__ z, uint64_t seed, T* __restrict__ V) {
    const int cpn = Rp >> 2;
    const int64_t total = (p1 - p0) * cpn;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        if constexpr (sizeof(T) == 4) sweep_item_fp32(t, k, p0 + i / cpn, (int)(i % cpn), Rp, z, seed, V);
        else sweep_item_fp64(t, k, p0 + i / cpn, (int)(i % cpn), Rp, z, seed, V);
    }
}

// All levels in one cooperative launch: the grid walks level after level and
// synchronizes between them (cooperative_groups grid barrier; every block of
// a cooperative launch is resident, so the barrier always completes).  This
// removes the per-level launch gaps that dominate sweeps with many small
// levels.
template <typename T>
__global__ void __launch_bounds__(256) sweep_all_kernel(const SweepTables<T> t, int k, const int32_t* __restrict__ loff,
                                                        int nlevels, int Rp, const T* __restrict__ z, uint64_t seed,
                                                        T* __restrict__ V) {
    cg::grid_group grid = cg::this_grid();
    const int cpn = Rp >> 2;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int l = 0; l < nlevels; ++l) {
        const int64_t p0 = loff[l], p1 = loff[l + 1];
        const int64_t total = (p1 - p0) * cpn;
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += stride) {
            if constexpr (sizeof(T) == 4) sweep_item_fp32(t, k, p0 + i / cpn, (int)(i % cpn), Rp, z, seed, V);
            else sweep_item_fp64(t, k, p0 + i / cpn, (int)(i % cpn), Rp, z, seed, V);
        }
        grid.sync();
    }
}

// One warp per node for rows of at most 32 chunks (R <= 128): lane = s * cpn +
// ch, where ch is the realization chunk and s one of S = 32 / cpn slices of
// the neighbour list.  Each lane accumulates every S-th neighbour, so the
// chain of dependent loads per lane is S times shorter than one thread per
// chunk walking all neighbours (the small levels are latency-bound); the S
// partial sums are then combined across lanes (error-free for the
// compensated FP32 sums).

template <typename T>
__global__ void __launch_bounds__(256) sweep_warp_kernel(const SweepTables<T> t, int k, int64_t p0, int64_t p1, int Rp,
                                                         int cpn, const T* __restrict__ z, uint64_t seed,
                                                         T* __restrict__ V) {
    const int lane = threadIdx.x & 31;
    const int ch = lane % cpn, s = lane / cpn, S = 32 / cpn;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t pos = p0 + (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); pos < p1; pos += nw) {
        const int g = t.node[pos];
        const int m = t.m[pos];
        const int32_t* idx = t.idx + pos * k;
        if constexpr (sizeof(T) == 4) {
            Dot2 a0, a1, a2, a3;
            a0.init(0.f, 0.f);
            a1.init(0.f, 0.f);
            a2.init(0.f, 0.f);
            a3.init(0.f, 0.f);
            const float2* w = reinterpret_cast<const float2*>(t.w) + pos * k;
            for (int j = s; j < m; j += S) {
                const float4 v = Vec4<float>::load(V + (int64_t)idx[j] * Rp + 4 * ch);
                const float2 wj = w[j];
                a0.add(wj.x, wj.y, v.x);
                a1.add(wj.x, wj.y, v.y);
                a2.add(wj.x, wj.y, v.z);
                a3.add(wj.x, wj.y, v.w);
            }
            for (int o = cpn; o < 32; o <<= 1) {
                dot2_merge(a0, __shfl_xor_sync(FULL_MASK, a0.s, o), __shfl_xor_sync(FULL_MASK, a0.c, o));
                dot2_merge(a1, __shfl_xor_sync(FULL_MASK, a1.s, o), __shfl_xor_sync(FULL_MASK, a1.c, o));
                dot2_merge(a2, __shfl_xor_sync(FULL_MASK, a2.s, o), __shfl_xor_sync(FULL_MASK, a2.c, o));
                dot2_merge(a3, __shfl_xor_sync(FULL_MASK, a3.s, o), __shfl_xor_sync(FULL_MASK, a3.c, o));
            }
            if (s == 0) {
                const float2 b0 = reinterpret_cast<const float2*>(t.b0)[pos];
                dot2_merge(a0, b0.x, b0.y);
                dot2_merge(a1, b0.x, b0.y);
                dot2_merge(a2, b0.x, b0.y);
                dot2_merge(a3, b0.x, b0.y);
                const float4 zz = z ? Vec4<float>::load(z + (int64_t)g * Rp + 4 * ch) : normals4(seed, g, ch);
                const float2 sg = reinterpret_cast<const float2*>(t.sigma)[pos];
                a0.add(sg.x, sg.y, zz.x);
                a1.add(sg.x, sg.y, zz.y);
                a2.add(sg.x, sg.y, zz.z);
                a3.add(sg.x, sg.y, zz.w);
                Vec4<float>::store(V + (int64_t)g * Rp + 4 * ch,
                                   make_float4(a0.value(), a1.value(), a2.value(), a3.value()));
            }
        } else {
            D4 acc = {0.0, 0.0, 0.0, 0.0};
            const double* w = t.w + pos * k;
            for (int j = s; j < m; j += S) {
                const D4 v = load_d4(V + (int64_t)idx[j] * Rp + 4 * ch);
                const double wj = w[j];
                acc.x = fma(wj, v.x, acc.x);
                acc.y = fma(wj, v.y, acc.y);
                acc.z = fma(wj, v.z, acc.z);
                acc.w = fma(wj, v.w, acc.w);
            }
            for (int o = cpn; o < 32; o <<= 1) {
                acc.x += __shfl_xor_sync(FULL_MASK, acc.x, o);
                acc.y += __shfl_xor_sync(FULL_MASK, acc.y, o);
                acc.z += __shfl_xor_sync(FULL_MASK, acc.z, o);
                acc.w += __shfl_xor_sync(FULL_MASK, acc.w, o);
            }
            if (s == 0) {
                const double b0 = t.b0[pos];
                D4 zz;
                if (z) {
                    zz = load_d4(z + (int64_t)g * Rp + 4 * ch);
                } else {
                    const float4 f = normals4(seed, g, ch);
                    zz = {(double)f.x, (double)f.y, (double)f.z, (double)f.w};
                }
                const double sg = t.sigma[pos];
                acc.x = fma(sg, zz.x, acc.x + b0);
                acc.y = fma(sg, zz.y, acc.y + b0);
                acc.z = fma(sg, zz.z, acc.z + b0);
                acc.w = fma(sg, zz.w, acc.w + b0);
                store_d4(V + (int64_t)g * Rp + 4 * ch, acc);
            }
        }
    }
}

static int sweep_blocks(int64_t total) {
    int64_t b = (total + 255) / 256;
    if (b > (1 << 20)) b = 1 << 20;
    return (int)(b < 1 ? 1 : b);
}

// warp-per-node variant when a row has a power-of-two number of chunks <= 16
static bool use_warp_sweep(int Rp) {
    const int cpn = Rp / 4;
    return cpn <= 16 && (cpn & (cpn - 1)) == 0;
}

template <typename T>
static cudaError_t sweep_level(const SweepTables<T>& t, int k, int64_t p0, int64_t p1, int Rp, const T* z,
                               uint64_t seed, T* V, cudaStream_t s) {
    if (p1 <= p0) return cudaSuccess;
    if (use_warp_sweep(Rp)) {
        const int64_t nodes = p1 - p0;
        int64_t blocks = (nodes + 7) / 8;
        if (blocks > (1 << 20)) blocks = 1 << 20;
        sweep_warp_kernel<T><<<(int)blocks, 256, 0, s>>>(t, k, p0, p1, Rp, Rp / 4, z, seed, V);
    } else {
        sweep_level_kernel<T><<<sweep_blocks((p1 - p0) * (Rp / 4)), 256, 0, s>>>(t, k, p0, p1, Rp, z, seed, V);
    }
    return cudaGetLastError();
}

cudaError_t launch_sweep_fp32(const SweepTables<float>& t, int k, int64_t p0, int64_t p1, int Rp, const float* z,
                              uint64_t seed, float* V, cudaStream_t s, int pairs, int split) {
    // pairs: chunks of 4 realizations per thread (1, 2 or 4); split: one
    // block per node with the neighbour list split over its warps
    if (split && Rp % 8 == 0) {
        if (p1 <= p0) return cudaSuccess;
        const int64_t nodes = p1 - p0;
        sweep_split_kernel<<<(unsigned)std::min<int64_t>(nodes, 1 << 20), SPLIT_WARPS * 32, 0, s>>>(t, k, p0, p1, Rp,
                                                                                                   z, seed, V);
        return cudaGetLastError();
    }
    if ((pairs == 2 || pairs == 4) && Rp % (4 * pairs) == 0 && !use_warp_sweep(Rp)) {
        if (p1 <= p0) return cudaSuccess;
        if (pairs == 2)
            sweep_levelN_kernel<2><<<sweep_blocks((p1 - p0) * (Rp / 8)), 256, 0, s>>>(t, k, p0, p1, Rp, z, seed, V);
        else
            sweep_levelN_kernel<4><<<sweep_blocks((p1 - p0) * (Rp / 16)), 256, 0, s>>>(t, k, p0, p1, Rp, z, seed, V);
        return cudaGetLastError();
    }
    return sweep_level<float>(t, k, p0, p1, Rp, z, seed, V, s);
}

cudaError_t launch_sweep_fp64(const SweepTables<double>& t, int k, int64_t p0, int64_t p1, int Rp, const double* z,
                              uint64_t seed, double* V, cudaStream_t s) {
    return sweep_level<double>(t, k, p0, p1, Rp, z, seed, V, s);
}

template <typename T>
static cudaError_t sweep_all(const SweepTables<T>& t, int k, const int32_t* loff, int nlevels, int Rp, const T* z,
                             uint64_t seed, T* V, cudaStream_t s) {
    int dev = 0, nsm = 0, coop = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return cudaErrorNotSupported;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sweep_all_kernel<T>, 256, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorNotSupported;
    dim3 grid(nsm * per_sm), block(256);
    void* args[] = {(void*)&t, (void*)&k, (void*)&loff, (void*)&nlevels, (void*)&Rp, (void*)&z, (void*)&seed, (void*)&V};
    return cudaLaunchCooperativeKernel((const void*)sweep_all_kernel<T>, grid, block, args, 0, s);
}

cudaError_t launch_sweep_all_fp32(const SweepTables<float>& t, int k, const int32_t* loff, int nlevels, int Rp,
                                  const float* z, uint64_t seed, float* V, cudaStream_t s) {
    return sweep_all<float>(t, k, loff, nlevels, Rp, z, seed, V, s);
}

cudaError_t launch_sweep_all_fp64(const SweepTables<double>& t, int k, const int32_t* loff, int nlevels, int Rp,
                                  const double* z, uint64_t seed, double* V, cudaStream_t s) {
    return sweep_all<double>(t, k, loff, nlevels, Rp, z, seed, V, s);
}

// ---------------------------------------------------------------------------
// Dataflow sweep: the dependency levels in one persistent launch, with no
// barrier between levels.  Realizations are independent, so a node's row is
// cut into H pieces of P4 chunks of 4 realizations, and every (node, piece)
// is a work item.  Items are numbered position-major (item = pos * H + q,
// positions in level order) and warps take `chunk` consecutive items per
// ticket, the next ticket while the current one is worked on.  A dependency
// always has a smaller item number (strictly lower level, same piece), and
// item numbers are taken in increasing order by warps that are running, so
// every wait ends: the smallest unfinished item can always proceed.
//
// The values are their own flags.  Before the launch every word of the rows it
// writes holds a bit pattern no stored value has (all ones, a NaN that
// arithmetic does not produce; settle() replaces it should one come in with
// the draws).  A reader loads a neighbour's chunk past L1 and, word by word,
// either has the value or loads again; nothing is ordered by it but the value
// itself, so there are no fences and no flag reads.  With a flag per (node,
// piece), a release fence and acquire polls, one dependent step took 2.6 us
// (a chain of 2,125 levels: 5.6 ms) instead of 0.74.  Waits are bounded
// (wait_ns of wall-clock time, or a count of polls reached no earlier); a
// warp that gives up sets err and stores NaN, and no warp takes new tickets
// once err is set.
//
// What bounds it: the neighbours' rows, gathered from anywhere in the values
// (no reuse once they exceed L2), or on narrow levels the step above.  4M
// nodes x 48 neighbours x 256 FP32 values: 32.4 ms, 65 with flags, 37.6 by
// per-level launches; 16.8M nodes x 64 values 27.2, 59 and 36.3; 1.2M x 100
// 3.2, 6.8 and 5.9.
//
// Lane layout inside a warp: W lanes per slice of the neighbour list (a
// power of two), S = 32 / W slices, each lane G chunks of the piece
// (P4 = W * G); the S partial sums are combined across lanes at the end.
// The sums of one chunk (4 realizations): FP32 values with (hi, lo) weights
// and compensated sums, FP64 values with plain FMA sums.
template <typename T>
struct FlowSum;
template <>
struct FlowSum<float> {
    using Weight = float2;
    using Value = float4;
    // Dot2 of two realizations at a time, the same operations on register
    // pairs (f32x2): half the instructions to issue
    // (4M nodes x 48 neighbours x 256 values 40.8 -> 35.5 ms)
    F2 s[2], c[2];
    __device__ __forceinline__ void init(Weight) { s[0] = s[1] = c[0] = c[1] = 0; }  // b0 is merged in the end
    __device__ static Weight entry(const float* p, int64_t i, int) { return reinterpret_cast<const float2*>(p)[i]; }
    __device__ static Weight shfl(Weight w, int l) {
        return make_float2(__shfl_sync(FULL_MASK, w.x, l), __shfl_sync(FULL_MASK, w.y, l));
    }
    __device__ static Value draws(const float* z, uint64_t seed, int g, int64_t row, int ch) {
        return z ? *reinterpret_cast<const float4*>(z + row + 4 * ch) : normals4(seed, g, ch);
    }
    // s becomes s + p, the rounding error is returned
    __device__ static F2 two_sum(F2& s, F2 p) {
        const F2 t = f2_add(s, p), bp = f2_sub(t, s);
        const F2 e = f2_add(f2_sub(s, f2_sub(t, bp)), f2_sub(p, bp));
        s = t;
        return e;
    }
    __device__ __forceinline__ void add(Weight w, const Value& v) {
        const F2 wh = f2_pack(w.x, w.x), wl = f2_pack(w.y, w.y);
        const F2 x[2] = {f2_pack(v.x, v.y), f2_pack(v.z, v.w)};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const F2 p = f2_mul(wh, x[q]);
            const F2 pe = f2_fma(wh, x[q], f2_mul(p, 0xbf800000bf800000ull));
            const F2 e = two_sum(s[q], p);
            c[q] = f2_add(c[q], f2_add(e, f2_fma(wl, x[q], pe)));
        }
    }
    __device__ __forceinline__ void merge(int q, F2 s2, F2 c2) {
        const F2 e = two_sum(s[q], s2);
        c[q] = f2_add(c[q], f2_add(c2, e));
    }
    __device__ __forceinline__ void across(int o) {
#pragma unroll
        for (int q = 0; q < 2; ++q)
            merge(q, __shfl_xor_sync(FULL_MASK, s[q], o), __shfl_xor_sync(FULL_MASK, c[q], o));
    }
    __device__ __forceinline__ Value finish(Weight b0, Weight sg, const Value& z) {
#pragma unroll
        for (int q = 0; q < 2; ++q) merge(q, f2_pack(b0.x, b0.x), f2_pack(b0.y, b0.y));
        add(sg, z);
        const F2 r0 = f2_add(s[0], c[0]), r1 = f2_add(s[1], c[1]);
        return make_float4(f2_lo(r0), f2_hi(r0), f2_lo(r1), f2_hi(r1));
    }
};
template <>
struct FlowSum<double> {
    using Weight = double;
    using Value = D4;
    D4 a;
    __device__ __forceinline__ void init(Weight b0) { a = {b0, b0, b0, b0}; }
    // pairs: each 8-byte table entry holds an FP32 (hi, lo) pair
    __device__ static Weight entry(const double* p, int64_t i, int pairs) {
        if (pairs) {
            const float2 v = reinterpret_cast<const float2*>(p)[i];
            return (double)v.x + (double)v.y;
        }
        return p[i];
    }
    __device__ static Weight shfl(Weight w, int l) { return __shfl_sync(FULL_MASK, w, l); }
    __device__ static Value draws(const double* z, uint64_t seed, int g, int64_t row, int ch) {
        if (z) return load_d4(z + row + 4 * ch);
        const float4 n4 = normals4(seed, g, ch);
        return {(double)n4.x, (double)n4.y, (double)n4.z, (double)n4.w};
    }
    __device__ __forceinline__ void add(Weight w, const Value& v) {
        a.x = fma(w, v.x, a.x);
        a.y = fma(w, v.y, a.y);
        a.z = fma(w, v.z, a.z);
        a.w = fma(w, v.w, a.w);
    }
    __device__ __forceinline__ void across(int o) {
        a.x += __shfl_xor_sync(FULL_MASK, a.x, o);
        a.y += __shfl_xor_sync(FULL_MASK, a.y, o);
        a.z += __shfl_xor_sync(FULL_MASK, a.z, o);
        a.w += __shfl_xor_sync(FULL_MASK, a.w, o);
    }
    __device__ __forceinline__ Value finish(Weight, Weight sg, const Value& z) {
        return {fma(sg, z.x, a.x), fma(sg, z.y, a.y), fma(sg, z.z, a.z), fma(sg, z.w, a.w)};
    }
};

// CSR: packed tables (t.off rows) and the seed read from f.seed_dev, the form
// used by batches of domains.
//
// A warp has three items under way: the ticket of the one after next, the
// table rows of the next one (a neighbour per lane, handed round by shuffles),
// and AHEAD neighbours' values of the current one, loaded before the first
// of them is looked at.
template <typename T, int G, int AHEAD, int MINB, bool CSR>
__global__ void __launch_bounds__(256, MINB) sweep_flow_kernel(const SweepTables<T> t, int k, int Rp, int W,
                                                               const T* __restrict__ z, uint64_t seed, T* V,
                                                               const __grid_constant__ FlowArgs f) {
    using Sum = FlowSum<T>;
    using Weight = typename Sum::Weight;
    using Value = typename Sum::Value;
    const int lane = threadIdx.x & 31;
    const int S = 32 / W, s = lane / W, cl = lane % W, cpn = Rp >> 2;
    const int64_t Rs = f.row_stride ? f.row_stride : Rp;
    const int pairs = CSR && sizeof(T) == 8 ? f.pairs : 0;
    const uint32_t stride16 = (uint32_t)(Rs * sizeof(T) / 16);  // a row, in 16 bytes: 32 x 32 bit products
    if (CSR && f.seed_dev) seed = *f.seed_dev;
    FlowItems next(f);
    // the next item's tables
    int64_t nrow = 0;
    int ng = 0, nm = 0, nidx = 0;
    Weight nw{};
    auto tables = [&]() {
        if (!next.live()) return;
        const int64_t pos = next.position();
        ng = t.node[pos];
        nm = t.m[pos];
        nrow = CSR ? t.off[pos] : pos * (int64_t)k;
        if (lane < (CSR ? nm : k)) {
            nidx = t.idx[nrow + lane];
            nw = Sum::entry(t.w, nrow + lane, pairs);
        }
    };
    tables();
    while (next.live()) {
        const int64_t pos = next.position();
        const int c0 = (int)(next.it - pos * f.H) * (W * G);
        const int64_t row = nrow;
        const int g = ng, m = nm;
        int idx = nidx;
        Weight w = nw;
        next.step();
        tables();
        if (CSR && f.node_class && f.node_class[g] != f.cls) continue;  // the other launch's node
        // rows of up to 8 realizations (W <= 2, the kernels with AHEAD = 2): the
        // sums over 16 or 32 slices are reduced with one realization left per
        // lane, and the first four slices finish one each
        constexpr bool spread = G == 1 && AHEAD == 2;
        // the draws and the node's own terms: nothing of them waits
        Value zz[G];
        if (spread) zz[0] = Value{};
        Weight b0{}, sg{};
        if (s < (spread ? 4 : 1)) {
            b0 = Sum::entry(t.b0, pos, pairs);
            sg = Sum::entry(t.sigma, pos, pairs);
#pragma unroll
            for (int gi = 0; gi < G; ++gi) {
                const int ch = c0 + cl + gi * W;
                if (ch < cpn) zz[gi] = Sum::draws(z, seed, g, (int64_t)g * Rs, ch);
            }
        }
        bool stuck = false;
        const uint4* Vl = reinterpret_cast<const uint4*>(V + 4 * (c0 + cl));
        Sum a[G];
#pragma unroll
        for (int gi = 0; gi < G; ++gi) a[gi].init(s == 0 ? b0 : Weight{});
        for (int jb = 0; jb < m; jb += 32) {
            if (jb && jb + lane < m) {
                idx = t.idx[row + jb + lane];
                w = Sum::entry(t.w, row + jb + lane, pairs);
            }
            const int mm = min(32, m - jb);
            for (int j0 = 0; j0 < mm; j0 += AHEAD * S) {
                Value v[AHEAD][G];
                auto wanted = [&](int h, int gi) { return j0 + h * S + s < mm && c0 + cl + gi * W < cpn; };
                auto chunk = [&](int h) {
                    const uint32_t i = __shfl_sync(FULL_MASK, idx, (j0 + h * S + s) & 31);
                    return reinterpret_cast<const T*>(Vl + (uint64_t)i * stride16);
                };
#pragma unroll
                for (int h = 0; h < AHEAD; ++h) {
                    const T* p = chunk(h);
#pragma unroll
                    for (int gi = 0; gi < G; ++gi) {
                        v[h][gi] = Value{};
                        if (wanted(h, gi)) v[h][gi] = ld_value4(p + 4 * gi * W);
                    }
                }
                // whatever is not stored yet is loaded again
                FlowBound bound;
                for (;;) {
                    bool miss = false;
#pragma unroll
                    for (int h = 0; h < AHEAD; ++h)
#pragma unroll
                        for (int gi = 0; gi < G; ++gi) miss |= missing4(v[h][gi]);
                    if (!__any_sync(FULL_MASK, miss) || stuck) break;
                    stuck = !bound.more(f.err, f.wait_ns);
                    stuck = __any_sync(FULL_MASK, stuck);
#pragma unroll
                    for (int h = 0; h < AHEAD; ++h) {
                        const T* p = chunk(h);
#pragma unroll
                        for (int gi = 0; gi < G; ++gi)
                            if (wanted(h, gi) && missing4(v[h][gi])) v[h][gi] = ld_value4(p + 4 * gi * W);
                    }
                }
#pragma unroll
                for (int h = 0; h < AHEAD; ++h) {
                    // for no lane of the warp: an FP64 instruction without any costs
                    // as much.  With b0 as the sum's start instead of an addition
                    // at its end, 1M nodes of 20 neighbours x 32 values 3.12 ->
                    // 2.14 ms, x 64 3.74 -> 2.98 (with flags 2.64, 3.28)
                    if (sizeof(T) == 8 && j0 + h * S >= mm) break;
                    const Weight wj = Sum::shfl(w, (j0 + h * S + s) & 31);
#pragma unroll
                    for (int gi = 0; gi < G; ++gi)
                        if (wanted(h, gi)) a[gi].add(wj, v[h][gi]);
                }
            }
        }
        if constexpr (spread) {
            // the additions of the tree below, each done once: 6 FP64
            // instructions for 32 slices instead of 20, and 2 to finish
            // instead of 8 (122 levels of 82 nodes, 4 realizations: 0.27 ->
            // 0.15 ms; FP32, 2,125 levels: 1.92 -> 1.56, 5.45M rows of 8
            // 4.9 -> 4.4)
            const bool up = s & 1, up2 = s & 2;
            const int ch = c0 + cl;
            const T zc = up ? (up2 ? zz[0].w : zz[0].z) : (up2 ? zz[0].y : zz[0].x);
            T r;
            if constexpr (sizeof(T) == 8) {
                const D4 v = a[0].a;
                const double k0 = (up ? v.z : v.x) + __shfl_xor_sync(FULL_MASK, up ? v.x : v.z, W);
                const double k1 = (up ? v.w : v.y) + __shfl_xor_sync(FULL_MASK, up ? v.y : v.w, W);
                double k = (up2 ? k1 : k0) + __shfl_xor_sync(FULL_MASK, up2 ? k0 : k1, 2 * W);
                for (int o = 4 * W; o < 32; o <<= 1) k += __shfl_xor_sync(FULL_MASK, k, o);
                r = fma(sg, zc, k);
            } else {
                F2 ks = up ? a[0].s[1] : a[0].s[0], kc = up ? a[0].c[1] : a[0].c[0];
                const F2 os = __shfl_xor_sync(FULL_MASK, up ? a[0].s[0] : a[0].s[1], W);
                const F2 oc = __shfl_xor_sync(FULL_MASK, up ? a[0].c[0] : a[0].c[1], W);
                const F2 e = Sum::two_sum(ks, os);
                kc = f2_add(kc, f2_add(oc, e));
                Dot2 d{up2 ? f2_hi(ks) : f2_lo(ks), up2 ? f2_hi(kc) : f2_lo(kc)};
                dot2_merge(d, __shfl_xor_sync(FULL_MASK, up2 ? f2_lo(ks) : f2_hi(ks), 2 * W),
                           __shfl_xor_sync(FULL_MASK, up2 ? f2_lo(kc) : f2_hi(kc), 2 * W));
                for (int o = 4 * W; o < 32; o <<= 1)
                    dot2_merge(d, __shfl_xor_sync(FULL_MASK, d.s, o), __shfl_xor_sync(FULL_MASK, d.c, o));
                dot2_merge(d, b0.x, b0.y);
                d.add(sg.x, sg.y, zc);
                r = d.value();
            }
            if (s < 4 && ch < cpn)
                st_value(V + (int64_t)g * Rs + 4 * ch + 2 * (s & 1) + (s >> 1), stuck ? settle(unstored<T>()) : r);
            continue;
        }
        for (int o = W; o < 32; o <<= 1)
#pragma unroll
            for (int gi = 0; gi < G; ++gi) a[gi].across(o);
        if (s == 0) {
#pragma unroll
            for (int gi = 0; gi < G; ++gi) {
                const int ch = c0 + cl + gi * W;
                if (ch < cpn) {
                    Value r = a[gi].finish(b0, sg, zz[gi]);
                    if (stuck) r.x = r.y = r.z = r.w = settle(unstored<T>());
                    st_value4(V + (int64_t)g * Rs + 4 * ch, r);
                }
            }
        }
    }
}

// Self-test of the dataflow wait: one warp waits, with the sweep's own
// bound, on a row that nothing stores; the wait must give up after
// f.wait_ns and report it in *f.err, leaving the context usable.
__global__ void flow_wait_selftest_kernel(const float* row, const __grid_constant__ FlowArgs f) {
    FlowBound bound;
    while (missing4(ld_value4(row)))
        if (!bound.more(f.err, f.wait_ns)) return;
}

cudaError_t launch_flow_wait_selftest(const float* row, const FlowArgs& f, cudaStream_t s) {
    flow_wait_selftest_kernel<<<1, 32, 0, s>>>(row, f);
    return cudaGetLastError();
}

// Rows of the positions [p0, p1) set to the pattern that stands for "not yet
// stored" (row_bytes a multiple of 16).
__global__ void flow_clear_kernel(const int32_t* __restrict__ node, int64_t p0, int64_t p1, int row16,
                                  uint4* __restrict__ V) {
    const int64_t n = (p1 - p0) * row16;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = i / row16;
        V[(int64_t)node[p0 + p] * row16 + (i - p * row16)] = make_uint4(~0u, ~0u, ~0u, ~0u);
    }
}

cudaError_t launch_flow_clear(const int32_t* node, int64_t p0, int64_t p1, int64_t N, size_t row_bytes, void* V,
                              cudaStream_t s) {
    if (p1 <= p0) return cudaSuccess;
    if (p0 == 0 && p1 == N) return cudaMemsetAsync(V, 0xff, (size_t)N * row_bytes, s);
    const int64_t n = (p1 - p0) * (int64_t)(row_bytes / 16);
    const int blocks = (int)std::min<int64_t>((n + 255) / 256, 1 << 14);
    flow_clear_kernel<<<blocks, 256, 0, s>>>(node, p0, p1, (int)(row_bytes / 16), reinterpret_cast<uint4*>(V));
    return cudaGetLastError();
}

// Posterior mean and variance from the tables of a plan whose neighbours are
// data only: its data terms and conditional deviations, node by node.
template <typename T>
__global__ void krige_moments_kernel(const SweepTables<T> t, const int8_t* __restrict__ status, double mean, int64_t N,
                                     double* __restrict__ m, double* __restrict__ v) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x) {
        double b0, sd;
        if constexpr (sizeof(T) == 8) {
            b0 = t.b0[p];
            sd = t.sigma[p];
        } else {
            b0 = (double)t.b0[2 * p] + (double)t.b0[2 * p + 1];
            sd = (double)t.sigma[2 * p] + (double)t.sigma[2 * p + 1];
        }
        const int32_t g = t.node[p];
        const bool ok = status[g] == SGS_NODE_KRIGED_;
        m[g] = ok ? mean + b0 : nan("");
        v[g] = ok ? sd * sd : nan("");
    }
}

template <typename T>
cudaError_t launch_krige_moments(const SweepTables<T>& t, const int8_t* status, double mean, int64_t N, double* m,
                                 double* v, cudaStream_t s) {
    krige_moments_kernel<T><<<(int)std::min<int64_t>((N + 255) / 256, 1 << 14), 256, 0, s>>>(t, status, mean, N, m, v);
    return cudaGetLastError();
}
template cudaError_t launch_krige_moments<float>(const SweepTables<float>&, const int8_t*, double, int64_t, double*,
                                                 double*, cudaStream_t);
template cudaError_t launch_krige_moments<double>(const SweepTables<double>&, const int8_t*, double, int64_t, double*,
                                                  double*, cudaStream_t);

// Lane layout for a row of cpn chunks: W lanes per slice (0 = automatic),
// G chunks per lane; returns the pieces per row.
int flow_layout(int Rp, int& W, int& G) {
    const int cpn = Rp / 4;
    int p2 = 1;
    while (p2 < cpn && p2 < 32) p2 <<= 1;
    if (W <= 0 || W > p2) W = p2;
    if (G != 2) G = 1;
    if (W * G > cpn && G == 2) G = 1;
    return (cpn + W * G - 1) / (W * G);
}

template <typename T, bool CSR>
using FlowKernel = void (*)(const SweepTables<T>, int, int, int, const T*, uint64_t, T*, const FlowArgs);

// The kernel for G chunks per lane and W lanes per slice.  A lane has 4 loads
// in flight; 2 where 16 or 32 slices cover a neighbour list with that many
// (W <= 2: with 4, the empty ones cost 8 % on batches of 8 realizations).
template <typename T, bool CSR>
static FlowKernel<T, CSR> flow_kernel(int G, int W, bool tight) {
    constexpr bool F = sizeof(T) == 4;
    if (G == 2) return tight ? sweep_flow_kernel<T, 2, 2, F ? 3 : 2, CSR> : sweep_flow_kernel<T, 2, 2, F ? 2 : 1, CSR>;
    if (W <= 2) return tight ? sweep_flow_kernel<T, 1, 2, F ? 4 : 3, CSR> : sweep_flow_kernel<T, 1, 2, 2, CSR>;
    return tight ? sweep_flow_kernel<T, 1, 4, F ? 4 : 3, CSR> : sweep_flow_kernel<T, 1, 4, 2, CSR>;
}

template <typename T, bool CSR>
static cudaError_t flow_launch(const SweepTables<T>& t, int k, int Rp, int W, int G, const T* z, uint64_t seed, T* V,
                               const FlowArgs& f, int nsm, cudaStream_t s) {
    const FlowKernel<T, CSR> kernel = flow_kernel<T, CSR>(G, W, f.tight);
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * FLOW_CLASSES, 0);
    if (e != cudaSuccess) return e;
    if (f.blocks_per_sm > 0 && f.blocks_per_sm < per_sm) per_sm = f.blocks_per_sm;
    if (per_sm < 1) per_sm = 1;
    const int64_t items = (f.item1 - f.item0 + f.chunk - 1) / f.chunk;
    int64_t blocks = std::min<int64_t>((int64_t)nsm * per_sm, (items + FLOW_CLASSES - 1) / FLOW_CLASSES);
    if (blocks < 1) blocks = 1;
    kernel<<<(int)blocks, 32 * FLOW_CLASSES, 0, s>>>(t, k, Rp, W, z, seed, V, f);
    return cudaGetLastError();
}

template <typename T>
static cudaError_t sweep_flow(const SweepTables<T>& t, int k, int Rp, int W, int G, const T* z, uint64_t seed, T* V,
                              FlowArgs f, int nsm, cudaStream_t s) {
    if (f.item1 <= f.item0) return cudaSuccess;
    f.rec = f.H > 1 ? ~0ull / (uint64_t)f.H + 1 : 0;
    return t.off ? flow_launch<T, true>(t, k, Rp, W, G, z, seed, V, f, nsm, s)
                 : flow_launch<T, false>(t, k, Rp, W, G, z, seed, V, f, nsm, s);
}

cudaError_t launch_sweep_flow_fp32(const SweepTables<float>& t, int k, int Rp, int W, int G, const float* z,
                                   uint64_t seed, float* V, const FlowArgs& f, int nsm, cudaStream_t s) {
    return sweep_flow<float>(t, k, Rp, W, G, z, seed, V, f, nsm, s);
}

cudaError_t launch_sweep_flow_fp64(const SweepTables<double>& t, int k, int Rp, int W, int G, const double* z,
                                   uint64_t seed, double* V, const FlowArgs& f, int nsm, cudaStream_t s) {
    return sweep_flow<double>(t, k, Rp, W, G, z, seed, V, f, nsm, s);
}

// ---------------------------------------------------------------------------
// Tiled transposes between the caller's realization-major [R][N] double
// arrays and the node-major [N][Rp] rows (32x32 tiles through shared memory).
template <typename T>
__global__ void z_to_rows_kernel(const double* __restrict__ zin, int64_t N, int R, int Rp, T* __restrict__ z) {
    __shared__ double tile[32][33];
    const int64_t g0 = (int64_t)blockIdx.x * 32;
    const int r0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int r = r0 + j;
        const int64_t g = g0 + threadIdx.x;
        tile[j][threadIdx.x] = (r < R && g < N) ? zin[(int64_t)r * N + g] : 0.0;
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int64_t g = g0 + j;
        const int r = r0 + threadIdx.x;
        if (g < N && r < Rp) z[g * Rp + r] = (T)tile[threadIdx.x][j];
    }
}

template <typename T>
__global__ void rows_to_out_kernel(const T* __restrict__ V, int64_t N, int R, int Rp, double mu,
                                   double* __restrict__ out) {
    __shared__ double tile[32][33];
    const int64_t g0 = (int64_t)blockIdx.x * 32;
    const int r0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int64_t g = g0 + j;
        const int r = r0 + threadIdx.x;
        tile[j][threadIdx.x] = (g < N && r < R) ? (double)V[g * Rp + r] : 0.0;
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int r = r0 + j;
        const int64_t g = g0 + threadIdx.x;
        if (r < R && g < N) out[(int64_t)r * N + g] = tile[threadIdx.x][j] + mu;
    }
}

template <typename T>
static cudaError_t z_rows(const double* zin, int64_t N, int R, int Rp, T* z, cudaStream_t s) {
    dim3 grid((unsigned)((N + 31) / 32), (unsigned)((Rp + 31) / 32));
    z_to_rows_kernel<T><<<grid, dim3(32, 8), 0, s>>>(zin, N, R, Rp, z);
    return cudaGetLastError();
}

template <typename T>
static cudaError_t rows_out(const T* V, int64_t N, int R, int Rp, double mu, double* out, cudaStream_t s) {
    dim3 grid((unsigned)((N + 31) / 32), (unsigned)((R + 31) / 32));
    rows_to_out_kernel<T><<<grid, dim3(32, 8), 0, s>>>(V, N, R, Rp, mu, out);
    return cudaGetLastError();
}

cudaError_t launch_z_to_rows_fp32(const double* zin, int64_t N, int R, int Rp, float* z, cudaStream_t s) {
    return z_rows<float>(zin, N, R, Rp, z, s);
}
cudaError_t launch_z_to_rows_fp64(const double* zin, int64_t N, int R, int Rp, double* z, cudaStream_t s) {
    return z_rows<double>(zin, N, R, Rp, z, s);
}
cudaError_t launch_rows_to_out_fp32(const float* V, int64_t N, int R, int Rp, double mu, double* out, cudaStream_t s) {
    return rows_out<float>(V, N, R, Rp, mu, out, s);
}
cudaError_t launch_rows_to_out_fp64(const double* V, int64_t N, int R, int Rp, double mu, double* out, cudaStream_t s) {
    return rows_out<double>(V, N, R, Rp, mu, out, s);
}

}  // namespace sgs

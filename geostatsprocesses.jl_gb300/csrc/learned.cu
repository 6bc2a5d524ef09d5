// learned.cu — the kriging-weight network used as a learned warm start:
// features, forward (inference), backward (gradients) and Adam kernels.
//
// The network is permutation invariant over a system's neighbours (a
// DeepSets form): for neighbour i with features f_i
//     h_i = relu(W1 f_i + b1)                    (H = 32)
//     g   = mean_i h_i
//     q_i = relu(W2a h_i + W2b g + b2)
//     y_i = w3 . q_i + b3                        (predicted weight of i)
// Features (F = 8): the lag from the neighbour to the node in the
// variogram's normalized frame u = diag(1/ranges) R^T (x0 - x_i) (3), |u|,
// the covariance C(x_i, x0) / sill, nugget / sill, and the variogram family
// (exponential, gaussian flags; spherical is neither).  Training minimizes
// the mean squared error of y against the weights the method's own solver
// produced.  One warp per system throughout; parameters live in shared
// memory.
#include <algorithm>

#include "common.cuh"

namespace sgs {

constexpr int NNF = 8;
constexpr int NNH = 32;
constexpr int NN_W1 = 0;                       // [H][F]
constexpr int NN_B1 = NN_W1 + NNH * NNF;       // [H]
constexpr int NN_W2A = NN_B1 + NNH;            // [H][H]
constexpr int NN_W2B = NN_W2A + NNH * NNH;     // [H][H]
constexpr int NN_B2 = NN_W2B + NNH * NNH;      // [H]
constexpr int NN_W3 = NN_B2 + NNH;             // [H]
constexpr int NN_B3 = NN_W3 + NNH;             // scalar
constexpr int NN_PARAMS = NN_B3 + 1;           // 2401
constexpr int NN_WARPS = 4;
constexpr int NN_LD = NNH + 1;                 // padded row of per-neighbour vectors

// Features of neighbour q of a system (see the file comment).
__device__ void nn_features(const GridDev& G, const VarioDev& v, const int* cq, const double* xq, bool qdata,
                            const int* cp, float* f) {
    double h[3] = {0.0, 0.0, 0.0};
    for (int j = 0; j < G.dim; ++j) {
        if (qdata) h[j] = centroid(G, j, cp[j]) - xq[j];
        else h[j] = (double)(cp[j] - cq[j]) * G.spacing[j];
    }
    float u[3] = {0.f, 0.f, 0.f};
    double s = 0.0;
    for (int j = 0; j < G.dim; ++j) {
        double t = v.R[0 + 3 * j] * h[0] + v.R[1 + 3 * j] * h[1];
        if (G.dim == 3) t += v.R[2 + 3 * j] * h[2];
        t *= v.inv_range[j];
        u[j] = (float)t;
        s += t * t;
    }
    f[0] = u[0];
    f[1] = u[1];
    f[2] = u[2];
    f[3] = (float)sqrt(s);
    f[4] = (float)(cov_fp64(v, G.dim, h[0], h[1], h[2]) / v.sill);
    f[5] = (float)(v.nugget / v.sill);
    f[6] = v.type == 2 ? 1.0f : 0.0f;
    f[7] = v.type == 3 ? 1.0f : 0.0f;
}

__global__ void nn_features_kernel(const GridDev G, const VarioDev v, const int32_t* nbr, const int32_t* cnt, int k,
                                   const double* data_xyz, float* feat) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t g = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); g < G.N; g += nw) {
        int cp[3];
        cell_of(G, (int)g, cp[0], cp[1], cp[2]);
        const int n = cnt[g];
        for (int q = lane; q < k; q += 32) {
            float f[NNF] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (q < n) {
                const int id = nbr[g * k + q];
                int cq[3] = {0, 0, 0};
                double xq[3] = {0, 0, 0};
                const bool isdata = id >= G.N;
                if (isdata) {
                    for (int j = 0; j < 3; ++j) xq[j] = data_xyz[3 * (int64_t)(id - G.N) + j];
                } else {
                    cell_of(G, id, cq[0], cq[1], cq[2]);
                }
                nn_features(G, v, cq, xq, isdata, cp, f);
            }
            float* o = feat + (g * k + q) * NNF;
#pragma unroll
            for (int j = 0; j < NNF; ++j) o[j] = f[j];
        }
    }
}

cudaError_t launch_nn_features(const GridDev& G, const VarioDev& v, const int32_t* nbr, const int32_t* cnt, int k,
                               const double* data_xyz, float* feat, cudaStream_t s) {
    int64_t blocks = (G.N + 7) / 8;
    if (blocks > 65535 * 8) blocks = 65535 * 8;
    nn_features_kernel<<<(int)blocks, 256, 0, s>>>(G, v, nbr, cnt, k, data_xyz, feat);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Forward pass of one system by one warp.  P: parameters (shared memory),
// f: features [n][F] (global), Hs/Qs: per-warp [64][NN_LD] scratch, gs/us:
// [H].  Leaves h_i in Hs, q_i in Qs (both post-activation), g in gs and
// W2b g + b2 in us; returns y for the lane's neighbours (i = lane, lane + 32).
__device__ void nn_forward_warp(const float* P, const float* f, int n, float* Hs, float* Qs, float* gs, float* us,
                                int lane, float y[2]) {
    for (int t = 0; t < 2; ++t) {
        const int i = lane + 32 * t;
        if (i < n) {
            float fi[NNF];
#pragma unroll
            for (int j = 0; j < NNF; ++j) fi[j] = f[i * NNF + j];
#pragma unroll 8
            for (int a = 0; a < NNH; ++a) {
                float z = P[NN_B1 + a];
#pragma unroll
                for (int j = 0; j < NNF; ++j) z = fmaf(P[NN_W1 + a * NNF + j], fi[j], z);
                Hs[i * NN_LD + a] = fmaxf(z, 0.0f);
            }
        }
    }
    __syncwarp();
    {
        float s = 0.0f;
        for (int i = 0; i < n; ++i) s += Hs[i * NN_LD + lane];
        gs[lane] = n > 0 ? s / (float)n : 0.0f;
    }
    __syncwarp();
    {
        float z = P[NN_B2 + lane];
        for (int b = 0; b < NNH; ++b) z = fmaf(P[NN_W2B + lane * NNH + b], gs[b], z);
        us[lane] = z;
    }
    __syncwarp();
    for (int t = 0; t < 2; ++t) {
        const int i = lane + 32 * t;
        y[t] = 0.0f;
        if (i < n) {
            float out = P[NN_B3];
#pragma unroll 4
            for (int a = 0; a < NNH; ++a) {
                float z = us[a];
                for (int b = 0; b < NNH; ++b) z = fmaf(P[NN_W2A + a * NNH + b], Hs[i * NN_LD + b], z);
                z = fmaxf(z, 0.0f);
                Qs[i * NN_LD + a] = z;
                out = fmaf(P[NN_W3 + a], z, out);
            }
            y[t] = out;
        }
    }
    __syncwarp();
}

struct NNSmem {
    float P[NN_PARAMS];
    float Hs[NN_WARPS][64 * NN_LD];
    float Qs[NN_WARPS][64 * NN_LD];
    float gs[NN_WARPS][NNH];
    float us[NN_WARPS][NNH];
};

__global__ void __launch_bounds__(NN_WARPS * 32) nn_forward_kernel(const float* __restrict__ params,
                                                                   const float* __restrict__ feat,
                                                                   const int32_t* __restrict__ count, int64_t nsys,
                                                                   int k, float* __restrict__ pred) {
    extern __shared__ __align__(16) unsigned char raw[];
    NNSmem& S = *reinterpret_cast<NNSmem*>(raw);
    for (int i = threadIdx.x; i < NN_PARAMS; i += blockDim.x) S.P[i] = params[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t nw = (int64_t)gridDim.x * NN_WARPS;
    for (int64_t s = (int64_t)blockIdx.x * NN_WARPS + wib; s < nsys; s += nw) {
        const int n = min(count[s], k);
        float y[2];
        nn_forward_warp(S.P, feat + s * k * NNF, n, S.Hs[wib], S.Qs[wib], S.gs[wib], S.us[wib], lane, y);
        for (int t = 0; t < 2; ++t) {
            const int i = lane + 32 * t;
            if (i < k) pred[s * k + i] = i < n ? y[t] : 0.0f;
        }
    }
}

// Loss and gradients of a batch: every system adds its mean squared error
// to *loss and its gradient to grad.
//
// One warp per system, its neighbours in chunks of 32 rows.  All products are
// 32 x 32 (or x 8) tiles of the warp, 4 x 8 of them per lane, one step of the
// inner dimension taking 3 shared-memory loads for 32 FP32 multiply-adds (16
// instructions): H = F W1', Z = H W2a', dW2a = dZ' H, dH = dZ W2a, dW1 = dZ1'
// F.  The matrices a step reads along both dimensions are kept in both orders.
// The gradients of the weights stay in registers over all systems of a warp,
// are added up per block in shared memory and once per block in global
// memory.  Bound: FP32 issue and shared-memory loads of 12 warps per SM (what
// shared memory holds).  Shared-memory sums with one neighbour per lane, 32
// lanes adding to one bank, took 16,384 systems of 32 neighbours 0.66 ms; this
// 0.13.
constexpr int NN_LDT = 36;               // tile row: 16-byte aligned, 8 rows of 4 on different banks
constexpr int NN_TILE = 32 * NN_LDT;

template <int NC>  // chunks of 32 neighbours
struct NNTiles {
    static constexpr int WARPS = 12 / NC;
    struct alignas(16) Warp {
        float H[NC][NN_TILE];    // h, [neighbour][unit]
        float T[NC][NN_TILE];    // h, then dz2, [unit][neighbour]
        float Z[NC][NN_TILE];    // dz2, then dz1, [neighbour][unit]
        float F[NC][32 * NNF];   // features, [neighbour][feature]
        float FT[NNF * NN_LDT];  // of one chunk, [feature][neighbour]
        float g[32], u[32], sz[32], dg[32];
    };
    float W1T[NNF * NN_LDT], W2A[NN_TILE], W2AT[NN_TILE], W2B[NN_TILE], W2BT[NN_TILE];
    float b1[32], b2[32], w3[32], b3[4], warp_loss[16];
    Warp warp[WARPS];
    static_assert(sizeof(Warp) % 16 == 0 && NN_TILE % 4 == 0 && WARPS <= 16, "16-byte loads");
};

// acc[r][p] += A[r] B[2p, 2p + 1], r < 4, p < 4
__device__ __forceinline__ void nn_step(F2 (&acc)[4][4], const float* A, const float* B) {
    const float4 a = *reinterpret_cast<const float4*>(A);
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(B), y = *reinterpret_cast<const ulonglong2*>(B + 4);
    const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const F2 s = f2_pack(av[r], av[r]);
        acc[r][0] = f2_fma(s, x.x, acc[r][0]);
        acc[r][1] = f2_fma(s, x.y, acc[r][1]);
        acc[r][2] = f2_fma(s, y.x, acc[r][2]);
        acc[r][3] = f2_fma(s, y.y, acc[r][3]);
    }
}

__device__ __forceinline__ void nn_load8(const float* p, F2 (&v)[4]) {
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(p), y = *reinterpret_cast<const ulonglong2*>(p + 4);
    v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
}

__device__ __forceinline__ void nn_store8(float* p, const F2 (&v)[4]) {
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v[0], v[1]);
    *reinterpret_cast<ulonglong2*>(p + 4) = make_ulonglong2(v[2], v[3]);
}

// the lane's tile by columns: X[unit][neighbours]
__device__ __forceinline__ void nn_store_t(float* X, const F2 (&t)[4][4]) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        *reinterpret_cast<float4*>(X + (2 * p) * NN_LDT) = make_float4(f2_lo(t[0][p]), f2_lo(t[1][p]), f2_lo(t[2][p]), f2_lo(t[3][p]));
        *reinterpret_cast<float4*>(X + (2 * p + 1) * NN_LDT) =
            make_float4(f2_hi(t[0][p]), f2_hi(t[1][p]), f2_hi(t[2][p]), f2_hi(t[3][p]));
    }
}

// sums over the 8 lanes that hold the same units
__device__ __forceinline__ void nn_sum_rows(F2 (&v)[4]) {
    const F2 one = f2_pack(1.0f, 1.0f);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1)
#pragma unroll
        for (int p = 0; p < 4; ++p) v[p] = f2_fma(one, __shfl_xor_sync(FULL_MASK, v[p], o), v[p]);
}

template <int NC>
__global__ void __launch_bounds__(NNTiles<NC>::WARPS * 32, 1)
nn_backward_kernel(const float* __restrict__ params, const float* __restrict__ feat, const int32_t* __restrict__ count,
                   const float* __restrict__ target, int64_t nsys, int k, float* grad, float* loss) {
    extern __shared__ __align__(16) unsigned char raw[];
    using S = NNTiles<NC>;
    S& sh = *reinterpret_cast<S*>(raw);
    const int lane = threadIdx.x & 31, ri = lane >> 2, ui = lane & 3;
    typename S::Warp& w = sh.warp[threadIdx.x >> 5];
    for (int i = threadIdx.x; i < NNH * NNH; i += S::WARPS * 32) {
        const int a = i / NNH, b = i % NNH;
        sh.W2A[a * NN_LDT + b] = sh.W2AT[b * NN_LDT + a] = params[NN_W2A + i];
        sh.W2B[a * NN_LDT + b] = sh.W2BT[b * NN_LDT + a] = params[NN_W2B + i];
        if (i < NNH * NNF) sh.W1T[(i % NNF) * NN_LDT + i / NNF] = params[NN_W1 + i];
        if (i < NNH) {
            sh.b1[i] = params[NN_B1 + i];
            sh.b2[i] = params[NN_B2 + i];
            sh.w3[i] = params[NN_W3 + i];
        }
        if (i == 0) sh.b3[0] = params[NN_B3];
    }
    __syncthreads();
    const bool vec = (reinterpret_cast<uintptr_t>(feat) & 15) == 0;
    const F2 one = f2_pack(1.0f, 1.0f);
    F2 dw2a[4][4], dw2b[4][4], dw1[4], dw3[4], db1[4], db2[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
        for (int p = 0; p < 4; ++p) dw2a[r][p] = dw2b[r][p] = 0;
        dw1[r] = dw3[r] = db1[r] = db2[r] = 0;
    }
    float db3 = 0.0f, total = 0.0f;
    const int64_t nw = (int64_t)gridDim.x * S::WARPS;
    for (int64_t s = (int64_t)blockIdx.x * S::WARPS + (threadIdx.x >> 5); s < nsys; s += nw) {
        const int n = min(count[s], k);
        if (n <= 0) continue;
        const float inv_n = 1.0f / (float)n;
        // ---- h = relu(W1 f + b1), its mean ----
        F2 sum[4] = {0, 0, 0, 0};
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (32 * c >= n) break;
            const int i = 32 * c + lane;
            float f[NNF];
#pragma unroll
            for (int j = 0; j < NNF; ++j) f[j] = 0.0f;
            if (i < n) {
                const float* fp = feat + (s * k + i) * NNF;
                if (vec) {
                    const float4 x = reinterpret_cast<const float4*>(fp)[0], y = reinterpret_cast<const float4*>(fp)[1];
                    f[0] = x.x, f[1] = x.y, f[2] = x.z, f[3] = x.w, f[4] = y.x, f[5] = y.y, f[6] = y.z, f[7] = y.w;
                } else {
#pragma unroll
                    for (int j = 0; j < NNF; ++j) f[j] = fp[j];
                }
            }
            *reinterpret_cast<float4*>(&w.F[c][lane * NNF]) = make_float4(f[0], f[1], f[2], f[3]);
            *reinterpret_cast<float4*>(&w.F[c][lane * NNF + 4]) = make_float4(f[4], f[5], f[6], f[7]);
#pragma unroll
            for (int j = 0; j < NNF; ++j) w.FT[j * NN_LDT + lane] = f[j];
            __syncwarp();
            F2 h[4][4];
            nn_load8(sh.b1 + 8 * ui, h[0]);
#pragma unroll
            for (int p = 0; p < 4; ++p) h[1][p] = h[2][p] = h[3][p] = h[0][p];
#pragma unroll
            for (int j = 0; j < NNF; ++j) nn_step(h, w.FT + j * NN_LDT + 4 * ri, sh.W1T + j * NN_LDT + 8 * ui);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const bool in = 32 * c + 4 * ri + r < n;
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    h[r][p] = in ? f2_pack(fmaxf(f2_lo(h[r][p]), 0.0f), fmaxf(f2_hi(h[r][p]), 0.0f)) : 0;
                    sum[p] = f2_fma(one, h[r][p], sum[p]);
                }
                nn_store8(&w.H[c][(4 * ri + r) * NN_LDT + 8 * ui], h[r]);
            }
            nn_store_t(&w.T[c][8 * ui * NN_LDT + 4 * ri], h);
            __syncwarp();
        }
        nn_sum_rows(sum);
        if (ri == 0) nn_store8(w.g + 8 * ui, sum);
        __syncwarp();
        w.g[lane] /= (float)n;
        __syncwarp();
        {
            float z = sh.b2[lane];
#pragma unroll
            for (int b = 0; b < NNH; ++b) z = fmaf(sh.W2BT[b * NN_LDT + lane], w.g[b], z);
            w.u[lane] = z;
        }
        __syncwarp();
        // ---- q = relu(W2a h + u), y = w3 q + b3; dz2 = dL/dy w3 (q > 0) ----
#pragma unroll
        for (int p = 0; p < 4; ++p) sum[p] = 0;
        float l2 = 0.0f;
        F2 w3[4];
        nn_load8(sh.w3 + 8 * ui, w3);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (32 * c >= n) break;
            float t[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = 32 * c + 4 * ri + r;
                t[r] = i < n ? target[s * k + i] : 0.0f;
            }
            F2 z[4][4];
            nn_load8(w.u + 8 * ui, z[0]);
#pragma unroll
            for (int p = 0; p < 4; ++p) z[1][p] = z[2][p] = z[3][p] = z[0][p];
#pragma unroll 8
            for (int b = 0; b < NNH; ++b) nn_step(z, w.T[c] + b * NN_LDT + 4 * ri, sh.W2AT + b * NN_LDT + 8 * ui);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                F2 y2 = 0;
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    z[r][p] = f2_pack(fmaxf(f2_lo(z[r][p]), 0.0f), fmaxf(f2_hi(z[r][p]), 0.0f));
                    y2 = f2_fma(w3[p], z[r][p], y2);
                }
                float y = f2_lo(y2) + f2_hi(y2);
                y += __shfl_xor_sync(FULL_MASK, y, 1);
                y += __shfl_xor_sync(FULL_MASK, y, 2);
                const bool in = 32 * c + 4 * ri + r < n;
                const float e = in ? y + sh.b3[0] - t[r] : 0.0f;
                const float dy = 2.0f * e / (float)n;
                if (ui == 0) {
                    l2 += e * e;
                    db3 += dy;
                }
                const F2 d2 = f2_pack(dy, dy);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    dw3[p] = f2_fma(d2, z[r][p], dw3[p]);
                    const float wl = f2_lo(w3[p]) * dy, wh = f2_hi(w3[p]) * dy;
                    z[r][p] = f2_pack(f2_lo(z[r][p]) > 0.0f ? wl : 0.0f, f2_hi(z[r][p]) > 0.0f ? wh : 0.0f);
                    sum[p] = f2_fma(one, z[r][p], sum[p]);
                }
                nn_store8(&w.Z[c][(4 * ri + r) * NN_LDT + 8 * ui], z[r]);
            }
            __syncwarp();  // T has been read
            nn_store_t(&w.T[c][8 * ui * NN_LDT + 4 * ri], z);
        }
        total += l2 * inv_n;
#pragma unroll
        for (int p = 0; p < 4; ++p) db2[p] = f2_fma(one, sum[p], db2[p]);
        nn_sum_rows(sum);
        if (ri == 0) nn_store8(w.sz + 8 * ui, sum);
        __syncwarp();
        // ---- dW2a = dz2' h, dW2b = (sum dz2)' g, dg = W2b' sum dz2 / n ----
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int rows = min(32, n - 32 * c);
#pragma unroll 4
            for (int i = 0; i < rows; ++i) nn_step(dw2a, w.Z[c] + i * NN_LDT + 4 * ri, w.H[c] + i * NN_LDT + 8 * ui);
        }
        nn_step(dw2b, w.sz + 4 * ri, w.g + 8 * ui);
        {
            float d = 0.0f;
#pragma unroll
            for (int a = 0; a < NNH; ++a) d = fmaf(sh.W2B[a * NN_LDT + lane], w.sz[a], d);
            w.dg[lane] = d * inv_n;
        }
        __syncwarp();
        // ---- dz1 = (W2a' dz2 + dg) (h > 0), dW1 = dz1' f ----
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (32 * c >= n) break;
            F2 d[4][4];
            nn_load8(w.dg + 8 * ui, d[0]);
#pragma unroll
            for (int p = 0; p < 4; ++p) d[1][p] = d[2][p] = d[3][p] = d[0][p];
#pragma unroll 8
            for (int a = 0; a < NNH; ++a) nn_step(d, w.T[c] + a * NN_LDT + 4 * ri, sh.W2A + a * NN_LDT + 8 * ui);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                F2 h[4];
                nn_load8(&w.H[c][(4 * ri + r) * NN_LDT + 8 * ui], h);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    d[r][p] = f2_pack(f2_lo(h[p]) > 0.0f ? f2_lo(d[r][p]) : 0.0f, f2_hi(h[p]) > 0.0f ? f2_hi(d[r][p]) : 0.0f);
                    db1[p] = f2_fma(one, d[r][p], db1[p]);
                }
                nn_store8(&w.Z[c][(4 * ri + r) * NN_LDT + 8 * ui], d[r]);
            }
            __syncwarp();
            const int rows = min(32, n - 32 * c);
#pragma unroll 4
            for (int i = 0; i < rows; ++i) {  // units 4 ri .., features 2 ui ..
                const float4 x = *reinterpret_cast<const float4*>(&w.Z[c][i * NN_LDT + 4 * ri]);
                const F2 f = *reinterpret_cast<const F2*>(&w.F[c][i * NNF + 2 * ui]);
                dw1[0] = f2_fma(f2_pack(x.x, x.x), f, dw1[0]);
                dw1[1] = f2_fma(f2_pack(x.y, x.y), f, dw1[1]);
                dw1[2] = f2_fma(f2_pack(x.z, x.z), f, dw1[2]);
                dw1[3] = f2_fma(f2_pack(x.w, x.w), f, dw1[3]);
            }
            __syncwarp();
        }
    }
    // ---- the block's gradient, over the tiles' memory ----
    __syncthreads();
    float* G = reinterpret_cast<float*>(&sh.warp[0]);
    static_assert(sizeof(sh.warp) >= NN_PARAMS * sizeof(float), "room for the gradient");
    for (int i = threadIdx.x; i < NN_PARAMS; i += S::WARPS * 32) G[i] = 0.0f;
    __syncthreads();
    auto add = [&](int i, F2 v) {
        atomicAdd(&G[i], f2_lo(v));
        atomicAdd(&G[i + 1], f2_hi(v));
    };
    nn_sum_rows(dw3);
    nn_sum_rows(db1);
    nn_sum_rows(db2);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int at = (4 * ri + r) * NNH + 8 * ui + 2 * p;
            add(NN_W2A + at, dw2a[r][p]);
            add(NN_W2B + at, dw2b[r][p]);
        }
        add(NN_W1 + (4 * ri + p) * NNF + 2 * ui, dw1[p]);
        if (ri == 0) {
            add(NN_W3 + 8 * ui + 2 * p, dw3[p]);
            add(NN_B1 + 8 * ui + 2 * p, db1[p]);
            add(NN_B2 + 8 * ui + 2 * p, db2[p]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        db3 += __shfl_xor_sync(FULL_MASK, db3, o);
        total += __shfl_xor_sync(FULL_MASK, total, o);
    }
    if (lane == 0) {
        atomicAdd(&G[NN_B3], db3);
        sh.warp_loss[threadIdx.x >> 5] = total;
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // once per block: fewer roundings of the whole sum
        double t = 0.0;
        for (int i = 0; i < S::WARPS; ++i) t += (double)sh.warp_loss[i];
        atomicAdd(loss, (float)t);
    }
    for (int i = threadIdx.x; i < NN_PARAMS; i += S::WARPS * 32) atomicAdd(&grad[i], G[i]);
}

// Warm-start predictions for every node of a plan: features computed in
// shared memory, then the forward pass; out is node-indexed [N][k].
__global__ void __launch_bounds__(NN_WARPS * 32) nn_predict_plan_kernel(const GridDev G, const VarioDev v,
                                                                        const int32_t* __restrict__ nbr,
                                                                        const int32_t* __restrict__ cnt, int k,
                                                                        const double* __restrict__ data_xyz,
                                                                        const float* __restrict__ params,
                                                                        float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char raw[];
    NNSmem& S = *reinterpret_cast<NNSmem*>(raw);
    float* F = reinterpret_cast<float*>(raw + sizeof(NNSmem));  // [NN_WARPS][64][NNF]
    for (int i = threadIdx.x; i < NN_PARAMS; i += blockDim.x) S.P[i] = params[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    float* f = F + wib * 64 * NNF;
    const int64_t nw = (int64_t)gridDim.x * NN_WARPS;
    for (int64_t g = (int64_t)blockIdx.x * NN_WARPS + wib; g < G.N; g += nw) {
        int cp[3];
        cell_of(G, (int)g, cp[0], cp[1], cp[2]);
        const int n = min(cnt[g], k);
        for (int q = lane; q < n; q += 32) {
            const int id = nbr[g * k + q];
            int cq[3] = {0, 0, 0};
            double xq[3] = {0, 0, 0};
            const bool isdata = id >= G.N;
            if (isdata) {
                for (int j = 0; j < 3; ++j) xq[j] = data_xyz[3 * (int64_t)(id - G.N) + j];
            } else {
                cell_of(G, id, cq[0], cq[1], cq[2]);
            }
            nn_features(G, v, cq, xq, isdata, cp, f + q * NNF);
        }
        __syncwarp();
        float y[2];
        nn_forward_warp(S.P, f, n, S.Hs[wib], S.Qs[wib], S.gs[wib], S.us[wib], lane, y);
        for (int t = 0; t < 2; ++t) {
            const int i = lane + 32 * t;
            if (i < k) out[g * k + i] = i < n ? y[t] : 0.0f;
        }
    }
}

static int nn_blocks(int64_t nsys);

cudaError_t launch_nn_predict_plan(const GridDev& G, const VarioDev& v, const int32_t* nbr, const int32_t* cnt, int k,
                                   const double* data_xyz, const float* params, float* out, cudaStream_t s) {
    const size_t smem = sizeof(NNSmem) + (size_t)NN_WARPS * 64 * NNF * sizeof(float);
    cudaError_t e =
        cudaFuncSetAttribute(nn_predict_plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    nn_predict_plan_kernel<<<nn_blocks(G.N), NN_WARPS * 32, smem, s>>>(G, v, nbr, cnt, k, data_xyz, params, out);
    return cudaGetLastError();
}

__global__ void nn_adam_kernel(float* p, const float* g, float* m, float* v, int step, float lr, float scale) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NN_PARAMS) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float gi = g[i] * scale;
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / (1.0f - powf(b1, (float)step));
    const float vh = vi / (1.0f - powf(b2, (float)step));
    p[i] -= lr * mh / (sqrtf(vh) + eps);
}

static int nn_blocks(int64_t nsys) {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    int64_t b = (nsys + NN_WARPS - 1) / NN_WARPS;
    const int64_t cap = (int64_t)nsm * 4;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

cudaError_t launch_nn_forward(const float* params, const float* feat, const int32_t* count, int64_t nsys, int k,
                              float* pred, cudaStream_t s) {
    const size_t smem = sizeof(NNSmem);
    cudaError_t e = cudaFuncSetAttribute(nn_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    nn_forward_kernel<<<nn_blocks(nsys), NN_WARPS * 32, smem, s>>>(params, feat, count, nsys, k, pred);
    return cudaGetLastError();
}

template <int NC>
static cudaError_t nn_backward(const float* params, const float* feat, const int32_t* count, const float* target,
                               int64_t nsys, int k, float* grad, float* loss, cudaStream_t s) {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = sizeof(NNTiles<NC>);
    cudaError_t e = cudaFuncSetAttribute(nn_backward_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    constexpr int W = NNTiles<NC>::WARPS;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(nsm, (nsys + W - 1) / W));
    nn_backward_kernel<NC><<<blocks, W * 32, smem, s>>>(params, feat, count, target, nsys, k, grad, loss);
    return cudaGetLastError();
}

cudaError_t launch_nn_backward(const float* params, const float* feat, const int32_t* count, const float* target,
                               int64_t nsys, int k, float* grad, float* loss, cudaStream_t s) {
    return k <= 32 ? nn_backward<1>(params, feat, count, target, nsys, k, grad, loss, s)
                   : nn_backward<2>(params, feat, count, target, nsys, k, grad, loss, s);
}

cudaError_t launch_nn_adam(float* p, const float* g, float* m, float* v, int step, float lr, float scale,
                           cudaStream_t s) {
    nn_adam_kernel<<<(NN_PARAMS + 255) / 256, 256, 0, s>>>(p, g, m, v, step, lr, scale);
    return cudaGetLastError();
}

}  // namespace sgs

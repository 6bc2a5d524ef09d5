// indicator.cu — sequential indicator simulation (SIS): the categorical
// counterpart of the sweep for an IndicatorProcess simulated with SEQSIM
// (src/simulation/field/seqsim.jl:247-261 one-hot transform, :292-310
// Kriging(func, prob) with a Categorical prior and conditional, :342-347
// categorical draw).
//
// For a separable (intrinsic) indicator covariance C_ab(h) = A_ab rho(h) —
// which includes the proportional transiogram t_ab(h) = p_b + (delta_ab -
// p_b) rho(h), where A = diag(p) - p p' — simple cokriging of isotopic
// indicators gives every category the same weights: those of simple kriging
// with rho (the weights of the plan's solve), so
//   p_l = prob_l + sum_i w_i (I_l(x_i) - prob_l)
//       = prob_l (1 - W) + sum_{grid nbrs of category l} w_j + D_l
// with W the sum of all weights and D_l the weights of data of category l
// (both written by the solve).  The conditional is Categorical(normalize(
// clamp(p, 0, 1), 1)); a node without a kriging system (fewer than
// minneighbors neighbours, or singular) has W = D = 0, i.e. the prior.
// The draw is the inverse cdf at a uniform u: the first category whose
// cumulative probability exceeds u.
//
// Categories are bytes, node-major [N][Rp].
// Per-category sums are compensated FP32 sums of (hi, lo) weights (about
// 1e-12), so the category decision equals an FP64 evaluation except at
// exact ties.
#include <algorithm>

#include "common.cuh"
#include "flow.cuh"

namespace sgs {

// four uniforms in (0, 1) of node g, realizations 4q..4q+3: (2m+1)/2^24 on
// the top 23 bits m of the Philox4x32-10 output words (counter: node,
// realization / 4, 0x5349), exact in FP32 and FP64
__device__ __forceinline__ float4 uniforms4(uint64_t seed, int64_t g, int q) {
    uint4 c = philox10(make_uint4((uint32_t)g, (uint32_t)((uint64_t)g >> 32), (uint32_t)q, 0x5349u),
                       (uint32_t)seed, (uint32_t)(seed >> 32));
    const float sc = 1.0f / 16777216.0f;
    return make_float4((float)((c.x >> 9) * 2u + 1u) * sc, (float)((c.y >> 9) * 2u + 1u) * sc,
                       (float)((c.z >> 9) * 2u + 1u) * sc, (float)((c.w >> 9) * 2u + 1u) * sc);
}

__device__ __forceinline__ int draw_category(const IndArgs& ia, const double* p, double u) {
    double q[IND_MAX_CAT];
    double s = 0.0;
#pragma unroll
    for (int l = 0; l < IND_MAX_CAT; ++l) {
        q[l] = l < ia.ncat ? fmin(fmax(p[l], 0.0), 1.0) : 0.0;
        s += q[l];
    }
    if (!(s > 0.0)) {  // every kriged probability clamped to 0: the prior
#pragma unroll
        for (int l = 0; l < IND_MAX_CAT; ++l) q[l] = l < ia.ncat ? ia.prob[l] : 0.0;
        s = 1.0;
    }
    double cum = 0.0;
#pragma unroll
    for (int l = 0; l < IND_MAX_CAT - 1; ++l) {
        if (l < ia.ncat - 1) {
            cum += q[l] / s;
            if (u < cum) return l;
        }
    }
    return ia.ncat - 1;
}

// The sweeps below are dataflow launches (sweep.cu): an item is a node and up
// to 32 of its realizations, W lanes one realization each and 32 / W slices of
// the neighbour list.  A lane loads its realization's category of 4 neighbours
// (the multivariate sweep: its LM variables of 8 / LM neighbours) and adds
// them once they are stored; with 8, 16 or 24 it is slower.  One launch per
// level, with the categories of 4 realizations and up to 28 FP64 divisions to
// a thread, took 48 us for a level (174 levels of 256 x 256 nodes x 32: 8.3
// ms); this takes 2.4 (0.42 ms; 0.70 with a branch on the category instead of
// adding zero to the others).
constexpr int IND_AHEAD = 4;

// The category drawn at u for probabilities proportional to base + sum,
// clamped: in FP32 where that decides it.  The FP32 sums differ from exact ones
// by less than 2^-19 (1 + A), A the sum of the terms' magnitudes; where u falls
// within twice that of a boundary, or nothing is left after clamping, the FP64
// evaluation decides.
template <int LM, class Sum, class Exact>
__device__ __forceinline__ int draw_category32(const IndArgs& ia, const float (&base)[LM], Sum sum, Exact exact,
                                               double u) {
    float q[LM], s = 0.0f, A = 1.0f;
#pragma unroll
    for (int l = 0; l < LM; ++l) {
        q[l] = 0.0f;
        if (l < ia.ncat) {
            const float b = base[l], g = sum(l);
            A += fabsf(b) + fabsf(g);
            q[l] = fminf(fmaxf(b + g, 0.0f), 1.0f);
            s += q[l];
        }
    }
    const float margin = A * 3.8e-6f, us = (float)u * s;
    bool near = !(s > margin);
    float cum = 0.0f;
    int cat = ia.ncat - 1;
#pragma unroll
    for (int l = 0; l < LM - 1; ++l)
        if (l < ia.ncat - 1) {
            cum += q[l];
            near = near || !(fabsf(us - cum) > margin);
            if (us < cum && cat == ia.ncat - 1) cat = l;
        }
    if (near) {
        double p[IND_MAX_CAT];
#pragma unroll
        for (int l = 0; l < IND_MAX_CAT; ++l) p[l] = 0.0;
#pragma unroll
        for (int l = 0; l < LM; ++l)
            if (l < ia.ncat) p[l] = exact(l);
        cat = draw_category(ia, p, u);
    }
    return cat;
}

// uniform (given or seeded) of a node's realization
__device__ __forceinline__ double uniform_of(const double* __restrict__ u, uint64_t seed, int64_t g, int Rp, int r) {
    if (u) return u[g * Rp + r];
    const float4 f = uniforms4(seed, g, r >> 2);
    return (double)((r & 2) ? ((r & 1) ? f.w : f.z) : ((r & 1) ? f.y : f.x));
}

// Categories of neighbours j + h S, h < IND_AHEAD, of one realization (C: its
// column) once they are stored, IND_NONE where there is none; false where the
// wait was given up.
constexpr uint32_t IND_NONE = 0xfe;
__device__ __forceinline__ bool flow_categories(const int32_t* idx, int m, int j, int S, bool on, const uint8_t* C, int Rp,
                                                const FlowArgs& f, uint32_t (&cat)[IND_AHEAD]) {
    int g[IND_AHEAD];
#pragma unroll
    for (int h = 0; h < IND_AHEAD; ++h) g[h] = on && j + h * S < m ? idx[j + h * S] : -1;
#pragma unroll
    for (int h = 0; h < IND_AHEAD; ++h) cat[h] = g[h] >= 0 ? ld_category(C + (int64_t)g[h] * Rp) : IND_NONE;
    FlowBound bound;
    for (;;) {
        bool miss = false;
#pragma unroll
        for (int h = 0; h < IND_AHEAD; ++h) miss |= cat[h] == 0xff;
        if (!miss) return true;
        if (!bound.more(f.err, f.wait_ns)) return false;
#pragma unroll
        for (int h = 0; h < IND_AHEAD; ++h)
            if (cat[h] == 0xff) cat[h] = ld_category(C + (int64_t)g[h] * Rp);
    }
}

template <typename T, int LM>
__global__ void __launch_bounds__(256) sis_flow_kernel(const SweepTables<T> t, int k, int Rp, const IndArgs ia,
                                                       const double* __restrict__ u, uint64_t seed, uint8_t* C,
                                                       const __grid_constant__ FlowArgs f, int W) {
    const int lane = threadIdx.x & 31, S = 32 / W, s = lane / W;
    bool ok = true;
    for (FlowItems next(f); next.live(); next.step()) {
        const int64_t pos = next.position();
        const int r = (int)(next.it - pos * f.H) * W + lane % W;
        const bool on = r < Rp;
        const int g = t.node[pos];
        const int m = t.m[pos];
        const int32_t* idx = t.idx + pos * k;
        // weights: (hi, lo) pairs, or the two words of a double
        const float2* tw = reinterpret_cast<const float2*>(t.w) + pos * k;
        float2 w0 = make_float2(0.f, 0.f), w1 = w0;
        if (lane < m) w0 = tw[lane];
        if (lane + 32 < m) w1 = tw[lane + 32];
        const double W1 = 1.0 - ia.wsum[pos];
        const double* D = ia.dsum + pos * ia.ncat;
        float b0[LM];
#pragma unroll
        for (int l = 0; l < LM; ++l) b0[l] = l < ia.ncat ? (float)(ia.prob[l] * W1 + D[l]) : 0.f;
        const double ur = on ? uniform_of(u, seed, g, Rp, r) : 0.0;
        // per category: the weights of grid neighbours of that category
        // (compensated FP32 sums, or FP64 for FP64 tables)
        float sh[LM], sc[LM];
        double sd[LM];
#pragma unroll
        for (int l = 0; l < LM; ++l) {
            sh[l] = sc[l] = 0.f;
            sd[l] = 0.0;
        }
        for (int j0 = 0; j0 < m; j0 += IND_AHEAD * S) {
            uint32_t cat[IND_AHEAD];
            ok = flow_categories(idx, ok ? m : 0, j0 + s, S, on, C + r, Rp, f, cat) && ok;
#pragma unroll
            for (int h = 0; h < IND_AHEAD; ++h) {
                const int j = j0 + h * S + s;
                const float hi0 = __shfl_sync(FULL_MASK, w0.x, j & 31), lo0 = __shfl_sync(FULL_MASK, w0.y, j & 31);
                float2 wj = make_float2(hi0, lo0);
                if (m > 32) {
                    const float hi1 = __shfl_sync(FULL_MASK, w1.x, j & 31), lo1 = __shfl_sync(FULL_MASK, w1.y, j & 31);
                    if (j >= 32) wj = make_float2(hi1, lo1);
                }
                if constexpr (sizeof(T) == 4) {
#pragma unroll
                    for (int l = 0; l < LM; ++l) {  // zeros for the other categories
                        const bool own = l == (int)cat[h];
                        const DF ts = df_two_sum(sh[l], own ? wj.x : 0.f);
                        sh[l] = ts.hi;
                        sc[l] = __fadd_rn(sc[l], __fadd_rn(ts.lo, own ? wj.y : 0.f));
                    }
                } else {
                    const double wd = __hiloint2double(__float_as_int(wj.y), __float_as_int(wj.x));
#pragma unroll
                    for (int l = 0; l < LM; ++l) sd[l] += l == (int)cat[h] ? wd : 0.0;
                }
            }
        }
        for (int o = W; o < 32; o <<= 1)
#pragma unroll
            for (int l = 0; l < LM; ++l) {
                if constexpr (sizeof(T) == 4) {
                    const DF ts = df_two_sum(sh[l], __shfl_xor_sync(FULL_MASK, sh[l], o));
                    sc[l] = __fadd_rn(sc[l], __shfl_xor_sync(FULL_MASK, sc[l], o));
                    sh[l] = ts.hi;
                    sc[l] = __fadd_rn(sc[l], ts.lo);
                } else {
                    sd[l] += __shfl_xor_sync(FULL_MASK, sd[l], o);
                }
            }
        if (s == 0 && on) {
            const int cat = draw_category32<LM>(
                ia, b0, [&](int l) { return sizeof(T) == 4 ? sh[l] + sc[l] : (float)sd[l]; },
                [&](int l) {
                    return ia.prob[l] * W1 + (sizeof(T) == 4 ? (double)sh[l] + (double)sc[l] : sd[l]) + D[l];
                },
                ur);
            st_category(C + (int64_t)g * Rp + r, ok ? cat : 0);
        }
    }
}

// the items and pieces of a dataflow launch over all N positions, values
// cleared to the unstored pattern
template <class K, class... A>
static cudaError_t ind_flow(K kernel, FlowArgs f, int64_t N, int Rp, void* V, size_t bytes, cudaStream_t s, A... args) {
    int W = 1;
    while (W < Rp && W < 32) W <<= 1;
    f.H = (Rp + W - 1) / W;
    f.rec = f.H > 1 ? ~0ull / (uint64_t)f.H + 1 : 0;
    f.item0 = 0;
    f.item1 = N * f.H;
    f.chunk = 1;
    cudaError_t e = cudaMemsetAsync(V, 0xff, bytes, s);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * FLOW_CLASSES, 0);
    if (e != cudaSuccess) return e;
    const int64_t full = (int64_t)nsm * std::max(per_sm, 1);
    const int blocks = (int)std::max<int64_t>(1, std::min(full, (f.item1 + FLOW_CLASSES - 1) / FLOW_CLASSES));
    kernel<<<blocks, 32 * FLOW_CLASSES, 0, s>>>(args..., f, W);
    return cudaGetLastError();
}

cudaError_t launch_sis_flow_fp32(const SweepTables<float>& t, int k, int64_t N, int Rp, const IndArgs& ia,
                                 const double* u, uint64_t seed, uint8_t* C, const FlowArgs& f, cudaStream_t s) {
    const size_t bytes = (size_t)N * Rp;
    if (ia.ncat <= 2) return ind_flow(sis_flow_kernel<float, 2>, f, N, Rp, C, bytes, s, t, k, Rp, ia, u, seed, C);
    if (ia.ncat <= 4) return ind_flow(sis_flow_kernel<float, 4>, f, N, Rp, C, bytes, s, t, k, Rp, ia, u, seed, C);
    return ind_flow(sis_flow_kernel<float, 8>, f, N, Rp, C, bytes, s, t, k, Rp, ia, u, seed, C);
}

cudaError_t launch_sis_flow_fp64(const SweepTables<double>& t, int k, int64_t N, int Rp, const IndArgs& ia,
                                 const double* u, uint64_t seed, uint8_t* C, const FlowArgs& f, cudaStream_t s) {
    const size_t bytes = (size_t)N * Rp;
    if (ia.ncat <= 2) return ind_flow(sis_flow_kernel<double, 2>, f, N, Rp, C, bytes, s, t, k, Rp, ia, u, seed, C);
    if (ia.ncat <= 4) return ind_flow(sis_flow_kernel<double, 4>, f, N, Rp, C, bytes, s, t, k, Rp, ia, u, seed, C);
    return ind_flow(sis_flow_kernel<double, 8>, f, N, Rp, C, bytes, s, t, k, Rp, ia, u, seed, C);
}

// ---------------------------------------------------------------------------
// Full simple cokriging (SIS with a non-separable indicator covariance, e.g.
// structures of different ranges with their own coregionalization matrices):
// the reference's Kriging(f, prob) with a multivariate f solves, per node,
// one system over the n neighbours' L indicators (seqsim.jl:292-310).  LHS
// (nL x nL) blocks C(x_i - x_j), right-hand sides (nL x L) blocks
// C(x_i - x_0), C_ab(h) = sum_s coef[s][a][b] (sill_s - gamma_s(h)); FP64
// Cholesky by one warp with the canonical singular rule; then
//   p_t = prob_t + sum_i sum_a Lambda[(i, a), t] (I_a(x_i) - prob_a)
//       = cst_t + sum_{grid nbrs j} w[j][cat_j][t],
// the data's terms and every prob term folded into cst.
//
// Multivariate Gaussian simulation (GAUSS: a GaussianProcess whose function
// is such a model, seqsim.jl:277-290 Kriging(f, mu) with an MvNormal prior,
// predictprob's MvNormal conditional) solves the same systems with the L
// variables' values in place of indicators:
//   mu^_t = mu_t + sum_i sum_a Lambda[(i, a), t] (v_a(x_i) - mu_a)
//   S^    = C(0) - c' Lambda          (c: the right-hand sides, nL x L)
// and stores the lower Cholesky factor F of S^ (of C(0) for a node drawn from
// the prior): v = mu^ + F z.  F's rule: a pivot not above tau contributes
// nothing (its column of F is zero), so a conditional covariance that is zero
// up to rounding (a node on a datum) draws no noise.
constexpr int COK_WARPS = 4;

// K, L right-hand sides and C(0) below it; two vectors; neighbour cells / data
// ids; for up to n neighbours
__host__ __device__ constexpr int cok_rows(int n, int L) { return n * L + L; }
__host__ __device__ constexpr size_t cok_smem_per_warp(int n, int L) {
    const int M = cok_rows(n, L);
    return (size_t)(M * ldl_stride(M) + 2 * ((M + 1) / 2 * 2)) * sizeof(double) + (size_t)n * 4 * sizeof(int);
}

// the largest of any call (a kernel's limit is one for all threads of the process)
constexpr int cok_smem_max() {
    size_t m = 0;
    for (int L = 1; L <= IND_MAX_CAT; ++L) {
        const size_t s = cok_smem_per_warp(COK_MAX / L, L);
        m = s > m ? s : m;
    }
    return (int)(m * COK_WARPS);
}

// lower Cholesky factor of the L x L symmetric matrix S (lower triangle,
// row-major) into F (full L x L, zero above the diagonal); pivots not above
// tau give zero columns
__device__ __forceinline__ void mv_factor(const double* S, int L, double tau, double* F) {
    for (int i = 0; i < L * L; ++i) F[i] = 0.0;
    for (int j = 0; j < L; ++j) {
        double d = S[j * L + j];
        for (int l = 0; l < j; ++l) d -= F[j * L + l] * F[j * L + l];
        if (!(d > tau)) continue;
        const double fjj = sqrt(d);
        F[j * L + j] = fjj;
        for (int i = j + 1; i < L; ++i) {
            double t = S[i * L + j];
            for (int l = 0; l < j; ++l) t -= F[i * L + l] * F[j * L + l];
            F[i * L + j] = t / fjj;
        }
    }
}

__device__ __forceinline__ double structure_cov(const VarioStructDev& v, int dim, double h0, double h1, double h2) {
    if (h0 == 0.0 && h1 == 0.0 && (dim == 2 || h2 == 0.0)) return v.sill;
    return structure_cov_nonzero(v, dim, h0, h1, h2);
}

// lag between two points of the augmented set (grid cells or data), as the
// plain solve evaluates it
__device__ __forceinline__ void cok_lag(const SolveArgs& a, const int* ca, const int* cb, double* h) {
    const GridDev& G = a.grid;
    if (ca[3] < 0 && cb[3] < 0) {
        for (int j = 0; j < 3; ++j) h[j] = j < G.dim ? dmul((double)(cb[j] - ca[j]), G.spacing[j]) : 0.0;
        return;
    }
    double xa[3], xb[3];
    for (int j = 0; j < 3; ++j) {
        xa[j] = ca[3] < 0 ? (j < G.dim ? centroid(G, j, ca[j]) : 0.0) : a.data_xyz[3 * (int64_t)ca[3] + j];
        xb[j] = cb[3] < 0 ? (j < G.dim ? centroid(G, j, cb[j]) : 0.0) : a.data_xyz[3 * (int64_t)cb[3] + j];
        h[j] = dsub(xb[j], xa[j]);
    }
}

// C_s(h) of every structure: from the lag table, or evaluated
__device__ __forceinline__ void cok_cov(const SolveArgs& a, const CokArgs& c, const int* ca, const int* cb, double* cs) {
    const int S = a.vario.ns;
    if (c.lut && ca[3] < 0 && cb[3] < 0) {
        const CovLut& t = a.lut;
        const int l0 = cb[0] - ca[0], l1 = cb[1] - ca[1], l2 = cb[2] - ca[2];
        if (abs(l0) <= t.e[0] && abs(l1) <= t.e[1] && abs(l2) <= t.e[2]) {
            const double* e = c.lut + ((l0 + t.e[0]) + t.w[0] * ((l1 + t.e[1]) + t.w[1] * (l2 + t.e[2])));
            const int64_t total = (int64_t)t.w[0] * t.w[1] * t.w[2];
            for (int s = 0; s < S; ++s) cs[s] = e[s * total];
            return;
        }
    }
    double h[3];
    cok_lag(a, ca, cb, h);
    for (int s = 0; s < S; ++s) cs[s] = structure_cov(a.vario.st[s], a.grid.dim, h[0], h[1], h[2]);
}

__global__ void cok_lut_kernel(const GridDev G, const VarioDev v, const CovLut t, int64_t total, double* out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int L0 = (int)(i % t.w[0]) - t.e[0];
        const int64_t r = i / t.w[0];
        const int L1 = (int)(r % t.w[1]) - t.e[1];
        const int L2 = (int)(r / t.w[1]) - t.e[2];
        for (int s = 0; s < v.ns; ++s)
            out[s * total + i] = structure_cov(v.st[s], G.dim, dmul((double)L0, G.spacing[0]), dmul((double)L1, G.spacing[1]),
                                               G.dim == 3 ? dmul((double)L2, G.spacing[2]) : 0.0);
    }
}

cudaError_t launch_cok_lut(const GridDev& g, const VarioDev& v, const CovLut& lut, double* out, cudaStream_t s) {
    const int64_t total = (int64_t)lut.w[0] * lut.w[1] * lut.w[2];
    cok_lut_kernel<<<(int)std::min<int64_t>((total + 127) / 128, 65535), 128, 0, s>>>(g, v, lut, total, out);
    return cudaGetLastError();
}

// One warp per system: its n L equations, L right-hand sides and C(0) in
// shared memory, eliminated together (warp_ldl), which leaves C(0) - c'
// Lambda.  FP64 instructions bound it.  25.6k systems of 16 neighbours x 2
// variables took 5.9 ms with covariances evaluated pair by pair, a Cholesky
// factorization, two substitutions with divisions per variable and shared
// memory for 64 equations whatever their number; 1.5 so.
template <bool GAUSS>
__global__ void __launch_bounds__(COK_WARPS * 32) cok_solve_kernel(const __grid_constant__ SolveArgs a, const CokArgs c) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const GridDev& G = a.grid;
    const int L = c.ncat, k = a.k, S = a.vario.ns, Mk = cok_rows(k, L), ld = ldl_stride(Mk);
    double* A = reinterpret_cast<double*>(smem + (size_t)wib * cok_smem_per_warp(k, L));
    double* av = A + Mk * ld;
    double* fv = av + (Mk + 1) / 2 * 2;
    int* cell = reinterpret_cast<int*>(fv + (Mk + 1) / 2 * 2);  // [n][4]: c0, c1, c2, data id (-1: grid)
    const int nwarps = gridDim.x * COK_WARPS;
    for (int64_t pos = (int64_t)blockIdx.x * COK_WARPS + wib; pos < a.P; pos += nwarps) {
        const int g = a.order[pos];
        const int n = a.cnt[g];
        const int m = n * L;
        int self[4];
        cell_of(G, g, self[0], self[1], self[2]);
        self[3] = -1;
        bool kriged = n >= a.nmin;
        double* rhs = A + m * ld;  // row t: right-hand side t, then the weights Lambda[(i, a), t]
        // C(0) beside the right-hand sides
        for (int e = lane; e < L * L; e += 32) {
            const int t = e / L, u = e - t * L;
            double v = 0.0;
            for (int s = 0; s < S; ++s) v += c.coef[(s * L + t) * L + u] * a.vario.st[s].sill;
            rhs[t * ld + m + u] = v;
        }
        if (kriged) {
            for (int q = lane; q < n; q += 32) {
                const int id = a.nbr[(int64_t)g * k + q];
                int* cq = cell + 4 * q;
                if (id < G.N) {
                    cell_of(G, id, cq[0], cq[1], cq[2]);
                    cq[3] = -1;
                } else {
                    cq[0] = cq[1] = cq[2] = 0;
                    cq[3] = id - (int)G.N;
                }
            }
            __syncwarp();
            // lower triangle of the LHS, one neighbour pair (i >= j) per lane
            for (int item = lane; item < n * (n + 1) / 2; item += 32) {
                int i = (int)((sqrtf(8.0f * (float)item + 1.0f) - 1.0f) * 0.5f);
                while (i * (i + 1) / 2 > item) --i;
                while ((i + 1) * (i + 2) / 2 <= item) ++i;
                const int j = item - i * (i + 1) / 2;
                double cs[SGS_MAX_STRUCTURES];
                cok_cov(a, c, cell + 4 * j, cell + 4 * i, cs);
                for (int ai = 0; ai < L; ++ai)
                    for (int b = 0; b < L; ++b) {
                        const int r = i * L + ai, q = j * L + b;
                        if (q > r) continue;
                        double v = 0.0;
                        for (int s = 0; s < S; ++s) v += c.coef[(s * L + ai) * L + b] * cs[s];
                        A[r * ld + q] = v;
                    }
            }
            for (int i = lane; i < n; i += 32) {
                double cs[SGS_MAX_STRUCTURES];
                cok_cov(a, c, self, cell + 4 * i, cs);
                for (int ai = 0; ai < L; ++ai)
                    for (int t = 0; t < L; ++t) {
                        double v = 0.0;
                        for (int s = 0; s < S; ++s) v += c.coef[(s * L + ai) * L + t] * cs[s];
                        rhs[t * ld + i * L + ai] = v;
                    }
            }
            __syncwarp();
            kriged = warp_ldl(A, ld, m, m + L, c.tau, av, fv, lane);
        }
        if (kriged)
            for (int t = 0; t < L; ++t) warp_ldl_solve(A, ld, m, m + t, lane);
        __syncwarp();
        if constexpr (GAUSS) {
            // the factor of the conditional covariance (the prior's C(0) for
            // a node without a system)
            if (lane == 0) {
                double C0[IND_MAX_CAT * IND_MAX_CAT], F[IND_MAX_CAT * IND_MAX_CAT];
                for (int t = 0; t < L; ++t)
                    for (int u = 0; u <= t; ++u) {
                        double v = 0.0;
                        if (kriged) {
                            v = rhs[t * ld + m + u];
                        } else {  // a factorization may have stopped halfway
                            for (int s = 0; s < S; ++s) v += c.coef[(s * L + t) * L + u] * a.vario.st[s].sill;
                        }
                        C0[t * L + u] = v;
                    }
                mv_factor(C0, L, c.tau, F);
                for (int i = 0; i < L * L; ++i) c.fac[pos * L * L + i] = F[i] * c.unit;
            }
            __syncwarp();
        }
        // outputs: grid neighbours compacted in neighbour order, prob and
        // data terms folded into cst
        int mg = 0;
        double cst[IND_MAX_CAT];
        for (int t = 0; t < IND_MAX_CAT; ++t) cst[t] = 0.0;
        if (kriged) {
            for (int b0 = 0; b0 < n; b0 += 32) {
                const int i = b0 + lane;
                const bool isgrid = i < n && cell[4 * i + 3] < 0;
                const unsigned bal = __ballot_sync(FULL_MASK, isgrid);
                if (i < n) {
                    if constexpr (GAUSS) {
                        const int d = isgrid ? -1 : cell[4 * i + 3];
                        for (int t = 0; t < L; ++t) {
                            double v = 0.0;
                            for (int ai = 0; ai < L; ++ai) {
                                const double lam = rhs[t * ld + i * L + ai];
                                v -= lam * c.prob[ai];
                                if (d >= 0) v += lam * c.data_val[(int64_t)d * L + ai];
                            }
                            cst[t] += v;
                        }
                    } else {
                        const int dcat = isgrid ? -1 : c.data_cat[cell[4 * i + 3]];
                        for (int t = 0; t < L; ++t) {
                            double v = 0.0;
                            for (int ai = 0; ai < L; ++ai) {
                                const double lam = rhs[t * ld + i * L + ai];
                                v -= lam * c.prob[ai];
                                if (ai == dcat) v += lam;
                            }
                            cst[t] += v;
                        }
                    }
                    if (isgrid) {
                        const int jj = mg + __popc(bal & lanemask_lt());
                        const int64_t e = pos * k + jj;
                        c.idx[e] = a.nbr[(int64_t)g * k + i];
                        for (int b = 0; b < L; ++b)
                            for (int t = 0; t < L; ++t)
                                c.w[(e * L + b) * L + t] = rhs[t * ld + i * L + b];
                    }
                }
                mg += __popc(bal);
            }
        }
        for (int t = 0; t < L; ++t) {
            double v = cst[t];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
            if (lane == 0) c.cst[pos * L + t] = c.prob[t] + v;
        }
        if (lane == 0) {
            c.m[pos] = mg;
            a.status[g] = (int8_t)(n < a.nmin ? SGS_NODE_PRIOR_NMIN_ : (kriged ? SGS_NODE_KRIGED_ : SGS_NODE_PRIOR_SINGULAR_));
        }
        __syncwarp();
    }
}

template <bool GAUSS>
static cudaError_t cok_solve(const SolveArgs& a, const CokArgs& c, cudaStream_t s) {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = cok_smem_per_warp(a.k, c.ncat) * COK_WARPS;
    cudaError_t e =
        cudaFuncSetAttribute(cok_solve_kernel<GAUSS>, cudaFuncAttributeMaxDynamicSharedMemorySize, cok_smem_max());
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cok_solve_kernel<GAUSS>, COK_WARPS * 32, smem);
    if (per_sm < 1) per_sm = 1;
    const int64_t want = (a.P + COK_WARPS - 1) / COK_WARPS;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)nsm * per_sm));
    cok_solve_kernel<GAUSS><<<blocks, COK_WARPS * 32, smem, s>>>(a, c);
    return cudaGetLastError();
}

cudaError_t launch_cok_solve(const SolveArgs& a, const CokArgs& c, bool gaussian, cudaStream_t s) {
    return gaussian ? cok_solve<true>(a, c, s) : cok_solve<false>(a, c, s);
}

template <int LM>
__global__ void __launch_bounds__(256) cok_flow_kernel(const CokArgs c, const int32_t* __restrict__ node, int k, int Rp,
                                                       const double* __restrict__ u, uint64_t seed, uint8_t* C,
                                                       const __grid_constant__ FlowArgs f, int W) {
    const int lane = threadIdx.x & 31, S = 32 / W, s = lane / W, L = c.ncat;
    IndArgs ia{};
    ia.ncat = L;
    for (int l = 0; l < IND_MAX_CAT; ++l) ia.prob[l] = c.prob[l];
    bool ok = true;
    for (FlowItems next(f); next.live(); next.step()) {
        const int64_t pos = next.position();
        const int r = (int)(next.it - pos * f.H) * W + lane % W;
        const bool on = r < Rp;
        const int g = node[pos];
        const int m = c.m[pos];
        const double* w = c.w + pos * k * L * L;
        for (int b = lane * 16; b < m * L * L; b += 512) asm volatile("prefetch.global.L1 [%0];" ::"l"(w + b));
        float b0[LM];
        double p[LM];
#pragma unroll
        for (int t = 0; t < LM; ++t) {
            b0[t] = t < L ? (float)c.cst[pos * L + t] : 0.f;
            p[t] = 0.0;
        }
        const double ur = on ? uniform_of(u, seed, g, Rp, r) : 0.0;
        for (int j0 = 0; j0 < m; j0 += IND_AHEAD * S) {
            uint32_t cat[IND_AHEAD];
            ok = flow_categories(c.idx + pos * k, ok ? m : 0, j0 + s, S, on, C + r, Rp, f, cat) && ok;
#pragma unroll
            for (int h = 0; h < IND_AHEAD; ++h)
                if (cat[h] < IND_MAX_CAT) {
                    const double* wr = w + ((j0 + h * S + s) * L + cat[h]) * L;
#pragma unroll
                    for (int t = 0; t < LM; ++t)
                        if (t < L) p[t] += wr[t];
                }
        }
        __syncwarp();
        for (int o = W; o < 32; o <<= 1)
#pragma unroll
            for (int t = 0; t < LM; ++t)
                if (t < L) p[t] += __shfl_xor_sync(FULL_MASK, p[t], o);
        if (s == 0 && on) {
            const int cat = draw_category32<LM>(
                ia, b0, [&](int l) { return (float)p[l]; }, [&](int l) { return c.cst[pos * L + l] + p[l]; }, ur);
            st_category(C + (int64_t)g * Rp + r, ok ? cat : 0);
        }
    }
}

cudaError_t launch_cok_flow(const CokArgs& c, const int32_t* node, int k, int64_t N, int Rp, const double* u,
                            uint64_t seed, uint8_t* C, const FlowArgs& f, cudaStream_t s) {
    const size_t bytes = (size_t)N * Rp;
    if (c.ncat <= 2) return ind_flow(cok_flow_kernel<2>, f, N, Rp, C, bytes, s, c, node, k, Rp, u, seed, C);
    if (c.ncat <= 4) return ind_flow(cok_flow_kernel<4>, f, N, Rp, C, bytes, s, c, node, k, Rp, u, seed, C);
    return ind_flow(cok_flow_kernel<8>, f, N, Rp, C, bytes, s, c, node, k, Rp, u, seed, C);
}

// The multivariate Gaussian sweep: mu^_t = cst_t + sum_j sum_b w[j][b][t]
// v_b(x_j) over the system's grid neighbours, then v = mu^ + F z with z the
// given normals or the seeded ones of pseudo-node a*N + g (variable a of node
// g).  LM: the variables' bound (2, 4, 8), 8 / LM neighbours at a time.  136
// levels of 160 x 160 nodes, two variables x 16: 8.9 ms by level launches,
// 0.44 so.
template <int LM>
__global__ void __launch_bounds__(256) mv_flow_kernel(const CokArgs c, const int32_t* __restrict__ node, int k, int64_t N,
                                                      int Rp, const double* __restrict__ z, uint64_t seed, double* V,
                                                      const __grid_constant__ FlowArgs f, int W) {
    constexpr int AHEAD = 8 / LM;
    const int lane = threadIdx.x & 31, S = 32 / W, s = lane / W, L = c.ncat;
    bool ok = true;
    for (FlowItems next(f); next.live(); next.step()) {
        const int64_t pos = next.position();
        const int r = (int)(next.it - pos * f.H) * W + lane % W;
        const bool on = r < Rp;
        const int64_t g = node[pos];
        const int m = c.m[pos];
        // what nothing has to wait for: the noise F z and the constant
        double mu[LM], out[LM];
#pragma unroll
        for (int t = 0; t < LM; ++t) mu[t] = out[t] = 0.0;
        if (s == 0 && on) {
            const double* F = c.fac + pos * L * L;
#pragma unroll
            for (int b = 0; b < LM; ++b)
                if (b < L) {
                    double zb;
                    if (z) {
                        zb = z[((int64_t)b * N + g) * Rp + r];
                    } else {
                        const float4 n4 = normals4(seed, (int64_t)b * N + g, r >> 2);
                        zb = (double)((r & 2) ? ((r & 1) ? n4.w : n4.z) : ((r & 1) ? n4.y : n4.x));
                    }
#pragma unroll
                    for (int t = b; t < LM; ++t)
                        if (t < L) out[t] += F[t * L + b] * zb;
                }
#pragma unroll
            for (int t = 0; t < LM; ++t)
                if (t < L) mu[t] = c.cst[pos * L + t];
        }
        // the weights are on their way to L1 while the values are waited for
        const double* w = c.w + pos * k * L * L;
        for (int b = lane * 16; b < m * L * L; b += 512)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(w + b));
        for (int j0 = 0; j0 < m; j0 += AHEAD * S) {
            const double* p[AHEAD];
            double v[AHEAD][LM];
#pragma unroll
            for (int h = 0; h < AHEAD; ++h) {
                const int j = j0 + h * S + s;
                p[h] = ok && on && j < m ? V + (int64_t)c.idx[pos * k + j] * Rp + r : nullptr;
#pragma unroll
                for (int b = 0; b < LM; ++b)
                    if (p[h] && b < L) v[h][b] = ld_value(p[h] + b * N * Rp);
            }
            FlowBound bound;
            while (ok) {
                bool miss = false;
#pragma unroll
                for (int h = 0; h < AHEAD; ++h)
#pragma unroll
                    for (int b = 0; b < LM; ++b) miss |= p[h] && b < L && missing(v[h][b]);
                if (!miss) break;
                ok = bound.more(f.err, f.wait_ns);
#pragma unroll
                for (int h = 0; h < AHEAD; ++h)
#pragma unroll
                    for (int b = 0; b < LM; ++b)
                        if (p[h] && b < L && missing(v[h][b])) v[h][b] = ld_value(p[h] + b * N * Rp);
            }
#pragma unroll
            for (int h = 0; h < AHEAD; ++h)
                if (p[h]) {
#pragma unroll
                    for (int b = 0; b < LM; ++b)
                        if (b < L) {
                            const double* wr = w + ((j0 + h * S + s) * L + b) * L;
#pragma unroll
                            for (int t = 0; t < LM; ++t)
                                if (t < L) mu[t] += wr[t] * v[h][b];
                        }
                }
        }
        __syncwarp();
        for (int o = W; o < 32; o <<= 1)
#pragma unroll
            for (int t = 0; t < LM; ++t)
                if (t < L) mu[t] += __shfl_xor_sync(FULL_MASK, mu[t], o);
        if (s == 0 && on)
#pragma unroll
            for (int t = 0; t < LM; ++t)
                if (t < L) st_value(V + ((int64_t)t * N + g) * Rp + r, ok ? mu[t] + out[t] : settle(unstored<double>()));
    }
}

cudaError_t launch_mv_flow(const CokArgs& c, const int32_t* node, int k, int64_t N, int Rp, const double* z,
                           uint64_t seed, double* V, const FlowArgs& f, cudaStream_t s) {
    const size_t bytes = (size_t)N * c.ncat * Rp * sizeof(double);
    if (c.ncat <= 2) return ind_flow(mv_flow_kernel<2>, f, N, Rp, V, bytes, s, c, node, k, N, Rp, z, seed, V);
    if (c.ncat <= 4) return ind_flow(mv_flow_kernel<4>, f, N, Rp, V, bytes, s, c, node, k, N, Rp, z, seed, V);
    return ind_flow(mv_flow_kernel<8>, f, N, Rp, V, bytes, s, c, node, k, N, Rp, z, seed, V);
}

// node-major category bytes [N][Rp] -> realization-major int32 [R][N]
__global__ void cats_to_out_kernel(const uint8_t* __restrict__ C, int64_t N, int R, int Rp, int32_t* __restrict__ out) {
    const int64_t total = N * R;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / N);
        const int64_t g = i - (int64_t)r * N;
        out[i] = C[g * Rp + r];
    }
}

cudaError_t launch_cats_to_out(const uint8_t* C, int64_t N, int R, int Rp, int32_t* out, cudaStream_t s) {
    const int64_t total = N * R;
    int64_t blocks = (total + 255) / 256;
    if (blocks > (1 << 20)) blocks = 1 << 20;
    if (blocks < 1) blocks = 1;
    cats_to_out_kernel<<<(int)blocks, 256, 0, s>>>(C, N, R, Rp, out);
    return cudaGetLastError();
}

}  // namespace sgs

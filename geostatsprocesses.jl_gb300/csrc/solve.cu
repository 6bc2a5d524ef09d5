// solve.cu — kernel (b): batched simple-kriging build + solve for every node.
//
// Replaces GeoStatsModels.fit(Kriging(f, mu), neighbourhood) + status +
// predictprob (src/simulation/field/seqsim.jl:124-131,302-304): the LHS
// C_ab = sill - gamma(x_a, x_b) (src/utils.jl:50-62), its Cholesky factor,
// the weights w = C^-1 c, the conditional variance sigma^2 = C(0) - w'c, and
// the prior fallback when the factorization fails or the node has fewer
// than minneighbors neighbours (seqsim.jl:109-111,127-131).
//
// Grid-grid covariances come from a table over integer lags (every neighbour
// of a node is a cell offset inside the search template, so pairwise lags are
// bounded); lags involving data points are evaluated directly in FP64.
//
// Precision modes:
//   FP64          FP64 LHS, L D L' and weights: several systems of up to 16
//                 neighbours per warp in registers, or one warp per system in
//                 shared memory (the plain path; also re-solves queued systems)
//   FP32+refine   half a warp per system: register-resident L D L' of the
//                 FP32 LHS with L^-1 carried in place, refinement against the
//                 LHS in fixed point with exact residuals, double-FP32
//                 variance (solve_fp32_kernel below)
// Results are written in level order (the sweep's layout): the grid
// neighbours with their weights, and the data neighbours folded into the
// constant b0 = sum_data w_i (d_i - mu).
#include <algorithm>
#include <cmath>
#include <utility>

#include "common.cuh"

namespace sgs {

constexpr int SOLVE_WARPS = 4;

struct NbInfo {
    int c0, c1, c2;  // cell (grid neighbour or query)
    int did;         // data id, -1 for a grid node
};

__device__ __forceinline__ double lut_or_cov(const SolveArgs& a, int L0, int L1, int L2) {
    const CovLut& t = a.lut;
    if (t.c64 != nullptr && L0 >= -t.e[0] && L0 <= t.e[0] && L1 >= -t.e[1] && L1 <= t.e[1] &&
        L2 >= -t.e[2] && L2 <= t.e[2]) {
        return t.c64[(L0 + t.e[0]) + t.w[0] * ((L1 + t.e[1]) + t.w[1] * (L2 + t.e[2]))];
    }
    const GridDev& G = a.grid;
    return cov_fp64(a.vario, G.dim, dmul((double)L0, G.spacing[0]), dmul((double)L1, G.spacing[1]),
                    G.dim == 3 ? dmul((double)L2, G.spacing[2]) : 0.0);
}

__device__ __forceinline__ void point_of(const SolveArgs& a, const NbInfo& p, double* x) {
    const GridDev& G = a.grid;
    if (p.did < 0) {
        x[0] = centroid(G, 0, p.c0);
        x[1] = centroid(G, 1, p.c1);
        x[2] = G.dim == 3 ? centroid(G, 2, p.c2) : 0.0;
    } else {
        x[0] = a.data_xyz[3 * (int64_t)p.did + 0];
        x[1] = a.data_xyz[3 * (int64_t)p.did + 1];
        x[2] = a.data_xyz[3 * (int64_t)p.did + 2];
    }
}

// FP64 covariance between two points of the augmented set
__device__ __forceinline__ double kcov(const SolveArgs& a, const NbInfo& p, const NbInfo& q) {
    if (p.did < 0 && q.did < 0) return lut_or_cov(a, q.c0 - p.c0, q.c1 - p.c1, q.c2 - p.c2);
    double xp[3], xq[3];
    point_of(a, p, xp);
    point_of(a, q, xq);
    return cov_fp64(a.vario, a.grid.dim, dsub(xq[0], xp[0]), dsub(xq[1], xp[1]), dsub(xq[2], xp[2]));
}

// Indices of the neighbours that are data points, in order, into dl; returns
// their number (warp-uniform).
__device__ __forceinline__ int collect_data(const NbInfo* info, int n, int* dl, int lane) {
    int nd = 0;
    for (int b = 0; b < n; b += 32) {
        const int q = b + lane;
        const bool isdata = q < n && info[q].did >= 0;
        const unsigned bal = __ballot_sync(FULL_MASK, isdata);
        if (isdata) dl[nd + __popc(bal & lanemask_lt())] = q;
        nd += __popc(bal);
    }
    __syncwarp();
    return nd;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

__host__ __device__ constexpr size_t warp_smem_bytes(int k) {
    // K and the right-hand side's row, two vectors of scratch, neighbour info
    return (size_t)((k + 1) * ldl_stride(k + 1) + 2 * ((k + 2) / 2 * 2)) * sizeof(double) + (size_t)k * sizeof(NbInfo);
}

// A kernel's shared-memory limit is one for all threads of the process: it is set
// to the largest that any call needs, not to a call's own.
constexpr int kSolveSmemMax = (int)(warp_smem_bytes(KMAX) * SOLVE_WARPS);

// Indicator sums of one system (SolveArgs::ind_*): w holds the weights of the
// system's n neighbours (FP64 values `wq(q)`), kriged = false for a prior
// node (all sums zero).
template <typename WF>
__device__ __forceinline__ void write_indicator_sums(const SolveArgs& a, int64_t pos, int n, const NbInfo* info,
                                                     bool kriged, WF wq, int lane) {
    double ws = 0.0;
    double ds[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) ds[l] = 0.0;
    if (kriged)
        for (int q = lane; q < n; q += 32) {
            const double v = wq(q);
            ws += v;
            if (info[q].did >= 0) {
                const int c = a.ind_cat[info[q].did];
#pragma unroll
                for (int l = 0; l < 8; ++l)
                    if (l == c) ds[l] += v;
            }
        }
    ws = warp_sum(ws);
    if (lane == 0) a.ind_wsum[pos] = ws;
#pragma unroll
    for (int l = 0; l < 8; ++l)
        if (l < a.ncat) {
            const double v = warp_sum(ds[l]);
            if (lane == 0) a.ind_dsum[pos * a.ncat + l] = v;
        }
}

// Store an FP64 value into a table entry: as is, or as an FP32 (hi, lo) pair.
__device__ __forceinline__ void put(double* t, int64_t i, double v) { t[i] = v; }
__device__ __forceinline__ void put(float* t, int64_t i, double v) {
    const float hi = (float)v;
    t[2 * i] = hi;
    t[2 * i + 1] = (float)(v - (double)hi);
}

// Write one position's sweep-table row (and the optional node-indexed export).
template <typename O>
__device__ void write_row(const SolveArgs& a, const SweepTables<O>& tab, int64_t pos, int g, int n,
                          const NbInfo* info, const double* w, double sigma, int status, int lane) {
    const int k = a.k;
    const int64_t row = table_row(tab, pos, k);
    int m = 0;
    double b0 = 0.0, l1 = 0.0;
    if (status == SGS_NODE_KRIGED_) {
        for (int base = 0; base < n; base += 32) {
            const int q = base + lane;
            const bool isgrid = q < n && info[q].did < 0;
            const unsigned b = __ballot_sync(FULL_MASK, isgrid);
            if (isgrid) {
                const int j = m + __popc(b & lanemask_lt());
                tab.idx[row + j] = a.nbr[(int64_t)g * k + q] + (int32_t)a.node0;
                put(tab.w, row + j, w[q]);
                l1 += fabs(w[q]);
            } else if (q < n) {
                b0 += w[q] * (a.data_val[info[q].did] - a.mu);
            }
            m += __popc(b);
        }
        b0 = warp_sum(b0);
        if (a.wl1_max) {
            l1 = warp_sum(l1);
            if (lane == 0) atomicMax(a.wl1_max, __float_as_uint((float)l1));
        }
    }
    if (a.ind_wsum)
        write_indicator_sums(a, pos, n, info, status == SGS_NODE_KRIGED_, [&](int q) { return w[q]; }, lane);
    if (lane == 0) {
        if (a.sum_m) atomicAdd(a.sum_m, (unsigned long long)m);
        tab.node[pos] = g + (int32_t)a.node0;
        tab.m[pos] = m;
        put(tab.b0, pos, b0);
        put(tab.sigma, pos, sigma);
        a.status[g] = (int8_t)status;
    }
    if (a.w_full) {
        for (int q = lane; q < k; q += 32)
            a.w_full[(int64_t)g * k + q] = (status == SGS_NODE_KRIGED_ && q < n) ? w[q] : 0.0;
        if (lane == 0) a.sigma_full[g] = sigma;
    }
}

// One system (node g, sweep-table row pos) of the problem `a`, in this warp's
// shared-memory slot `base` laid out for up to kl neighbours (kl >= a.k, or
// >= the node's neighbour count).
template <typename O>
__device__ __forceinline__ void solve_system(const SolveArgs& a, const SweepTables<O>& tab, int64_t pos, int g,
                                             unsigned char* base, int kl, int lane) {
    const int k = a.k;
    const int ld = ldl_stride(kl + 1);
    double* A = reinterpret_cast<double*>(base);
    double* av = A + (kl + 1) * ld;
    double* fv = av + (kl + 2) / 2 * 2;
    NbInfo* info = reinterpret_cast<NbInfo*>(fv + (kl + 2) / 2 * 2);
    const GridDev& G = a.grid;
    const double sill = a.vario.sill;
    const double prior_sd = sqrt(sill) * a.vario.unit;
    {
        const int n = a.cnt[g];
        double* c = A + n * ld;  // the right-hand side, then the weights
        if (n < a.nmin) {
            write_row<O>(a, tab, pos, g, n, info, c, prior_sd, SGS_NODE_PRIOR_NMIN_, lane);
            return;
        }
        NbInfo self;
        cell_of(G, g, self.c0, self.c1, self.c2);
        self.did = -1;
        for (int q = lane; q < n; q += 32) {
            const int id = a.nbr[(int64_t)g * k + q];
            NbInfo in;
            if (id < G.N) {
                cell_of(G, id, in.c0, in.c1, in.c2);
                in.did = -1;
            } else {
                in.c0 = in.c1 = in.c2 = 0;
                in.did = id - (int)G.N;
            }
            info[q] = in;
        }
        __syncwarp();
        for (int q = lane; q < n; q += 32) c[q] = kcov(a, info[q], self);
        if (lane == 0) c[n] = sill;
        for (int r = 0; r < n; ++r) {
            const NbInfo ir = info[r];
            if (ir.did >= 0) continue;
            for (int q = lane; q <= r; q += 32) {
                const NbInfo iq = info[q];
                if (iq.did < 0) A[r * ld + q] = kcov(a, iq, ir);
            }
        }
        {
            int* dl = reinterpret_cast<int*>(av);
            const int nd = collect_data(info, n, dl, lane);
            for (int item = lane; item < nd * n; item += 32) {
                const int da = dl[item / n], q = item % n;
                const NbInfo iq = info[q];
                if (iq.did >= 0 && q > da) continue;
                A[(da >= q ? da : q) * ld + (da >= q ? q : da)] = kcov(a, iq, info[da]);
            }
        }
        __syncwarp();

        if (!warp_ldl(A, ld, n, n + 1, a.tau, av, fv, lane)) {
            write_row<O>(a, tab, pos, g, n, info, c, prior_sd, SGS_NODE_PRIOR_SINGULAR_, lane);
            return;
        }
        const double var = c[n];  // sill - c' K^-1 c
        warp_ldl_solve(A, ld, n, n, lane);
        write_row<O>(a, tab, pos, g, n, info, c, sqrt(var > 0.0 ? var : 0.0) * a.vario.unit, SGS_NODE_KRIGED_, lane);
        __syncwarp();
    }
}

// The plain FP64 path: FP64 LHS, L D L' and weights.  O is the
// table type: double for the FP64 path, float (hi, lo pairs) when it re-solves
// the systems the FP32 path queued.  With a.list set, solves only the queued
// positions.
template <typename O>
__global__ void __launch_bounds__(SOLVE_WARPS * 32) solve_kernel(const SolveArgs a, const SweepTables<O> tab) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    unsigned char* base = smem + (size_t)wib * warp_smem_bytes(a.k);
    const int64_t count = a.list ? (int64_t)*a.nfallback : a.P;
    const int64_t nwarps = (int64_t)gridDim.x * SOLVE_WARPS;
    for (int64_t it = (int64_t)blockIdx.x * SOLVE_WARPS + wib; it < count; it += nwarps) {
        const int64_t pos = a.list ? (int64_t)a.list[it] : it;
        solve_system<O>(a, tab, pos, a.order[pos], base, a.k, lane);
    }
}

// Batch form: desc[0] positions list[desc[1] ...] of the level-ordered
// global node list `order`, each solved with its domain's descriptor (domain
// d owns global node ids [noff[d], noff[d+1])); shared memory laid out for kl
// neighbours.
template <typename O>
__global__ void __launch_bounds__(SOLVE_WARPS * 32)
solve_batch_kernel(const SolveArgs* __restrict__ doms, const int64_t* __restrict__ noff, int ndom,
                   const int32_t* __restrict__ order, const int32_t* __restrict__ list,
                   const int32_t* __restrict__ desc, int kl, const SweepTables<O> tab) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SolveArgs s_dom[SOLVE_WARPS];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    unsigned char* base = smem + (size_t)wib * warp_smem_bytes(kl);
    const int64_t n = desc[0];
    const int32_t* lst = list + desc[1];
    const int64_t nwarps = (int64_t)gridDim.x * SOLVE_WARPS;
    int64_t lo = 0, hi = 0;
    for (int64_t it = (int64_t)blockIdx.x * SOLVE_WARPS + wib; it < n; it += nwarps) {
        const int64_t pos = lst[it];
        const int64_t gg = order[pos];
        if (gg < lo || gg >= hi) {
            const int d = find_domain(noff, ndom, gg);
            lo = noff[d];
            hi = noff[d + 1];
            __syncwarp();
            warp_copy_struct(&s_dom[wib], &doms[d], lane);
            __syncwarp();
        }
        solve_system<O>(s_dom[wib], tab, pos, (int)(gg - lo), base, kl, lane);
    }
}

// The plain FP64 path for at most 16 neighbours: GS lanes per system (8, 10 or
// 16, one per neighbour), 32 / GS systems per warp.  A warp FP64 instruction
// holds its scheduler for 64 cycles whatever its lanes do, so what counts is
// the number of instructions and the systems that share them.  Pairs with a
// datum, the only ones evaluated, are queued and taken 32 at a time; lane i
// then holds row i of the LHS in registers, and L D L' is eliminated with the
// right-hand side (the k-th pivot is the one Cholesky's square root would be
// taken of) by one reciprocal a column and rows broadcast by shuffles, in
// chunks of 4 entries up to the longest system of the warp.  One warp per
// system with a Cholesky factorization in shared memory and a division per
// row in each substitution took 250k systems of 10 data 8.9 ms, this 1.4 (1.9 with
// 16 lanes each: 10 neighbours are kriging's default).
template <int GS>
struct Sys64 {
    static constexpr int SYS = 32 / GS;
    static constexpr int LD = GS + 1;
    double K[SYS][(GS + 1) * LD];  // row GS: the right-hand side
    NbInfo info[SYS][GS + 1];      // [n]: the node itself
    unsigned short queue[64];      // pairs with a datum: is the node's, system, row, column
};

__device__ __noinline__ double kcov_pair(const SolveArgs& a, const NbInfo& p, const NbInfo& q) { return kcov(a, p, q); }

template <int GS, typename O>
__global__ void __launch_bounds__(SOLVE_WARPS * 32, 4) solve64_kernel(const __grid_constant__ SolveArgs a,
                                                                      const SweepTables<O> tab) {
    using S = Sys64<GS>;
    constexpr int LD = S::LD;
    extern __shared__ __align__(16) unsigned char smem[];
    S& sh = reinterpret_cast<S*>(smem)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, grp = lane / GS, q = lane % GS, l0g = grp * GS;
    const int k = a.k;
    const GridDev& G = a.grid;
    const double sill = a.vario.sill;
    const int64_t count = a.list ? (int64_t)*a.nfallback : a.P;
    const int64_t rounds = (count + S::SYS - 1) / S::SYS;
    const int64_t nwarps = (int64_t)gridDim.x * SOLVE_WARPS;
    unsigned long long msum = 0;
    float l1max = 0.0f;
    for (int64_t it = (int64_t)blockIdx.x * SOLVE_WARPS + (threadIdx.x >> 5); it < rounds; it += nwarps) {
        const int64_t item = it * S::SYS + grp;
        const bool have = grp < S::SYS && item < count;  // lanes past the last group are idle
        const int64_t pos = have ? (a.list ? (int64_t)a.list[item] : item) : 0;
        const int g = have ? a.order[pos] : 0;
        const int cnt = have ? a.cnt[g] : 0;
        const int n = have && cnt >= a.nmin ? cnt : 0;  // systems to solve (0: none, or the prior)
        NbInfo in{0, 0, 0, -1};
        int id = 0;
        if (q < n) {
            id = a.nbr[(int64_t)g * k + q];
            if (id < G.N) cell_of(G, id, in.c0, in.c1, in.c2);
            else in.did = id - (int)G.N;
            sh.info[grp][q] = in;
        }
        if (q == 0 && grp < S::SYS) {
            NbInfo self{0, 0, 0, -1};
            cell_of(G, g, self.c0, self.c1, self.c2);
            sh.info[grp][n] = self;
        }
        __syncwarp();
        const int nmax = (int)__reduce_max_sync(FULL_MASK, (unsigned)n);

        // ---- covariances of the pairs among the neighbours and the node ----
        int nq = 0;
        auto evaluate = [&](int c) {
            if (lane < c) {
                const unsigned e = sh.queue[lane];
                const int sg = (e >> 12) & 3, i = (e >> 6) & 63, j = e & 63;
                const double v = kcov_pair(a, sh.info[sg][j], sh.info[sg][i]);
                const int row = e >> 14 ? GS : i;  // the node's own
                sh.K[sg][row * LD + j] = v;
                if (row < GS) sh.K[sg][j * LD + i] = v;
            }
        };
        const int pairs = n * (n + 1) / 2, pmax = nmax * (nmax + 1) / 2;
        for (int p0 = 0; p0 < pmax; p0 += GS) {
            const int p = p0 + q;
            // p = i (i - 1) / 2 + j, j < i, i in 1 .. n (n: the node)
            int i = (int)((1.0f + sqrtf(8.0f * (float)p + 1.0f)) * 0.5f);
            if (i * (i - 1) / 2 > p) --i;
            if (i * (i + 1) / 2 <= p) ++i;
            const int j = p - i * (i - 1) / 2;
            bool queued = false;
            // the node's own row is kept as row GS
            const int row = i == n ? GS : i;
            if (p < pairs) {
                const NbInfo pj = sh.info[grp][j], pi = sh.info[grp][i];
                queued = pj.did >= 0 || pi.did >= 0;
                if (!queued) {
                    const double v = lut_or_cov(a, pi.c0 - pj.c0, pi.c1 - pj.c1, pi.c2 - pj.c2);
                    sh.K[grp][row * LD + j] = v;
                    if (i < n) sh.K[grp][j * LD + i] = v;
                }
            }
            const unsigned b = __ballot_sync(FULL_MASK, queued);
            if (queued) sh.queue[nq + __popc(b & lanemask_lt())] = (unsigned short)((i == n) << 14 | grp << 12 | i << 6 | j);
            nq += __popc(b);
            __syncwarp();
            if (nq >= 32) {
                evaluate(32);
                __syncwarp();
                const unsigned short rest = lane + 32 < nq ? sh.queue[lane + 32] : 0;
                __syncwarp();
                sh.queue[lane] = rest;
                __syncwarp();
                nq -= 32;
            }
        }
        evaluate(nq);
        __syncwarp();

        // ---- L D L' of the rows in registers, with the right-hand side ----
        double A[GS];
#pragma unroll
        for (int l = 0; l < GS; ++l)
            A[l] = q < n && l < n && l != q ? sh.K[grp][q * LD + l] : (l == q ? (q < n ? sill : 1.0) : 0.0);
        const double c = q < n ? sh.K[grp][GS * LD + q] : 0.0;
        double y = c, dinv = 1.0;
        bool ok = true;
#pragma unroll
        for (int j = 0; j < GS; ++j) {
            if (j < nmax) {
                const double d = __shfl_sync(FULL_MASK, A[j], l0g + j);
                ok = ok && (j >= n || d > a.tau);
                const double inv = reciprocal(d);
                if (q == j) dinv = inv;
                const double f = q > j ? -A[j] * inv : 0.0;
                y = fma(f, __shfl_sync(FULL_MASK, y, l0g + j), y);
#pragma unroll
                for (int l0 = 0; l0 < GS; l0 += 4)
                    if (l0 + 3 > j && l0 < nmax) {
#pragma unroll
                        for (int l = l0; l < l0 + 4 && l < GS; ++l)
                            if (l > j) A[l] = fma(f, __shfl_sync(FULL_MASK, A[l], l0g + j), A[l]);
                    }
            }
        }
        // summed below: c' K^-1 c by terms of one sign.  As w'c the deviations of
        // systems of 4 neighbours were off by 1.7e-16, with Cholesky's weights by
        // 1.35e-16, so by 1.0e-16 (root mean square, spherical model)
        double wc = q < n ? y * (y * dinv) : 0.0;
        double w = 0.0;
#pragma unroll
        for (int j = GS - 1; j >= 0; --j) {
            if (j < nmax) {
                const double t = y * dinv;
                if (q == j) w = t;
                const double wj = __shfl_sync(FULL_MASK, t, l0g + j);
                if (q < j) y = fma(-A[j], wj, y);
            }
        }
        if (q >= n) w = 0.0;

        // ---- the sweep-table row ----
        const bool kriged = n > 0 && ok;
        const bool isgrid = kriged && q < n && in.did < 0;
        double b0 = kriged && q < n && in.did >= 0 ? w * (a.data_val[in.did] - a.mu) : 0.0;
        float l1 = isgrid ? (float)fabs(w) : 0.0f;
        // sums over the group, in its first lane
#pragma unroll
        for (int o = GS > 8 ? 8 : 4; o > 0; o >>= 1) {
            const double tw = __shfl_down_sync(FULL_MASK, wc, o), tb = __shfl_down_sync(FULL_MASK, b0, o);
            const float tl = __shfl_down_sync(FULL_MASK, l1, o);
            if (q + o < GS) {
                wc += tw;
                b0 += tb;
                l1 += tl;
            }
        }
        const double var = kriged ? sill - wc : sill;
        const double sigma = sqrt(var > 0.0 ? var : 0.0) * a.vario.unit;
        const unsigned gb = (__ballot_sync(FULL_MASK, isgrid) >> l0g) & (0xffffffffu >> (32 - GS));
        const int m = __popc(gb);
        if (have) {
            const int64_t row = table_row(tab, pos, k);
            if (isgrid) {
                const int j = __popc(gb & ((1u << q) - 1));
                tab.idx[row + j] = id + (int32_t)a.node0;
                put(tab.w, row + j, w);
            }
            if (q == 0) {
                msum += m;
                l1max = fmaxf(l1max, l1);
                tab.node[pos] = g + (int32_t)a.node0;
                tab.m[pos] = m;
                put(tab.b0, pos, b0);
                put(tab.sigma, pos, sigma);
                a.status[g] = (int8_t)(n == 0 ? SGS_NODE_PRIOR_NMIN_ : (ok ? SGS_NODE_KRIGED_ : SGS_NODE_PRIOR_SINGULAR_));
            }
            if (a.w_full) {
                for (int l = q; l < k; l += GS) a.w_full[(int64_t)g * k + l] = l == q && kriged && q < n ? w : 0.0;
                if (q == 0) a.sigma_full[g] = sigma;
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        msum += __shfl_xor_sync(FULL_MASK, msum, o);
        l1max = fmaxf(l1max, __shfl_xor_sync(FULL_MASK, l1max, o));
    }
    if (lane == 0) {
        if (a.sum_m && msum) atomicAdd(a.sum_m, msum);
        if (a.wl1_max && l1max > 0.0f) atomicMax(a.wl1_max, __float_as_uint(l1max));
    }
}

template <int GS, typename O>
static cudaError_t launch_solve64(const SolveArgs& a, const SweepTables<O>& t, cudaStream_t s) {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = sizeof(Sys64<GS>) * SOLVE_WARPS;
    cudaError_t e = cudaFuncSetAttribute(solve64_kernel<GS, O>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, solve64_kernel<GS, O>, SOLVE_WARPS * 32, smem);
    if (e != cudaSuccess) return e;
    const int64_t full = (int64_t)nsm * std::max(per_sm, 1);
    const int64_t per_block = SOLVE_WARPS * Sys64<GS>::SYS;
    const int64_t want = a.list ? full : (a.P + per_block - 1) / per_block;
    const int blocks = (int)std::max<int64_t>(1, std::min(want, full));
    solve64_kernel<GS, O><<<blocks, SOLVE_WARPS * 32, smem, s>>>(a, t);
    return cudaGetLastError();
}

template <typename O>
static cudaError_t launch_solve(const SolveArgs& a, const SweepTables<O>& t, cudaStream_t s) {
    // several systems share a warp, and no category sums are wanted (a lone
    // system of 32 gains nothing from that form; 90k of 18 neighbours take
    // 1.38 ms in the other, 4.1 with a Cholesky factorization)
    if (a.k <= 16 && !a.ind_wsum)
        return a.k <= 8 ? launch_solve64<8, O>(a, t, s)
                        : (a.k <= 10 ? launch_solve64<10, O>(a, t, s) : launch_solve64<16, O>(a, t, s));
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = warp_smem_bytes(a.k) * SOLVE_WARPS;
    cudaError_t e = cudaFuncSetAttribute(solve_kernel<O>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSolveSmemMax);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, solve_kernel<O>, SOLVE_WARPS * 32, smem);
    if (per_sm < 1) per_sm = 1;
    int64_t want = a.list ? (int64_t)nsm * per_sm : (a.P + SOLVE_WARPS - 1) / SOLVE_WARPS;
    int blocks = (int)(want < (int64_t)nsm * per_sm ? want : (int64_t)nsm * per_sm);
    if (blocks < 1) blocks = 1;
    solve_kernel<O><<<blocks, SOLVE_WARPS * 32, smem, s>>>(a, t);
    return cudaGetLastError();
}

cudaError_t launch_solve_fp64(const SolveArgs& a, const SweepTables<double>& t, cudaStream_t s) {
    return launch_solve<double>(a, t, s);
}

// ---------------------------------------------------------------------------
// FP32 path.  Half a warp (16 lanes) per system, two systems per warp.  Lane
// (r, c) of the half's 4 x 4 lane grid owns the entries (r + 4a, c + 4b),
// b <= a, of the LHS's lower triangle in registers: the triangle's storage is
// near n^2 / 2 and its updates near n^3 / 3, where one row per lane holds and
// updates the whole square.  The LHS is normalized by the sill (a correlation
// matrix: pivots in (0, 1], weights unchanged).
//
// Shared memory keeps each entry as K = hi 2^-28 + lo, hi a 32-bit integer and
// lo the FP32 remainder (about 2^-53), in 4 x 4 blocks of the lower triangle
// (diagonal blocks whole), so that a lane's own entries lie at its constant
// offset in every block.  Grid pairs come from the lag table, pairs with a
// datum from one FP64 evaluation each, spread over the block's threads.
//
// The FP32 copy in registers becomes M = L^-1 and D of K = L D L' by one
// Gauss elimination that carries the inverse in place (no pivoting, which is
// stable for symmetric positive definite matrices; the k-th pivot is the
// Schur complement a Cholesky factorization would test).  A solve is then
// two triangular matrix-vector products, M' D^-1 M x, without sequential
// substitution.  The weights are refined against the stored K: the iterate
// is rounded to a multiple of 2^-24 (and a second multiple of 2^-48 after the
// first correction), so every product hi W is an integer and the residual
// c - K w is summed exactly in 64-bit integers, one multiply-add each; only
// the remainders' products are FP32.  That is more accurate than a
// compensated FP32 sum of (hi, lo) pairs and takes 2 instructions a term
// instead of 13.  Weights, sigma^2 = sill (1 - w'c) and b0 are double-FP32 and
// are written as (hi, lo) pairs for the compensated sweep.  A system with a
// pivot below 1e-3 (near-singular: the canonical 1e-10 decision needs FP64;
// a datum on another neighbour's point is singular without one: 27.8k such of
// 250k systems of 32 went through FP64 in 1.3 ms), a weight of 32 or more (the integer sums' range) or whose refinement does
// not contract is queued for the FP64 kernel.
//
// Bound: latency and issue slots of 6 (above 48 neighbours) to 24 warps per SM
// (shared memory and registers hold the systems; counters of the 32-neighbour form: issue slots 49 % used, L1's
// data pipe 73 % before the table gathers were put in lag order), and the
// FP64 pipe where many pairs involve data.  Measured against one warp per
// system with a full Gauss-Jordan inverse (CUDA events, one GB300): 2 M
// systems of 48 neighbours 37.3 -> 20.4 ms (30.8 -> 14.2 ms without data),
// 4.2 M of 32 23.5 -> 12.6 ms, 1.2 M of 24 6.7 -> 3.6 ms, 1.2 M of 16 4.1 ->
// 1.7 ms, 1.2 M of 60 35.4 -> 22.2 ms.
constexpr float KFIX = 268435456.0f;          // 2^28: units of an entry's integer part
constexpr float WFIX = 16777216.0f;           // 2^24: units of a weight's first integer part
constexpr float WFIX2 = 281474976710656.0f;   // 2^48: and of its second
constexpr float WLIM = 32.0f;                 // 64 entries x 2^28 x (32 x 2^24) < 2^63
// Warps per block and resident blocks per SM.  The warps of a block go through
// a round's phases together (they share the FP64 evaluations and the
// instruction cache lines of code that each runs once a round).  As many
// warps as registers allow without spills, two per scheduler at 48
// neighbours: what shared memory they leave is L1 for the lag table (2 M
// systems of 48: 4 x 2 blocks 20.4 ms, 5 x 2 22.8, 2 x 5 23.8, 1 x 8 24.6;
// 4.2 M of 32: 4 x 4 12.6 ms, 2 x 9 14.0, 8 x 2 13.5).
constexpr int solve32_warps(int nmax) { return nmax > 48 ? 3 : (nmax > 16 ? 4 : 2); }
constexpr int solve32_blocks(int nmax) { return nmax > 32 ? 2 : (nmax > 16 ? 4 : 12); }

struct KF {
    int hi;
    float lo;
};

template <int NMAX>
struct Sys32 {
    static constexpr int NP = NMAX / 4;            // block rows
    static constexpr int NR = NP / 4;              // rows a lane holds of a vector
    static constexpr int NB = NP * (NP + 1) / 2;   // blocks of the lower triangle
    static constexpr int K = NB * 128;             // 16 entries of 8 bytes a block
    static constexpr int C = NMAX * (int)sizeof(KF);
    static constexpr int V = NMAX * 4;             // one vector
    // K, c, three vector buffers, 1 / D; an odd multiple of 64 bytes puts the
    // two systems of a warp on different banks (where it fits)
    static constexpr int raw = K + C + 3 * V + V;
    static constexpr int bytes = raw % 128 == 0 && NMAX < 64 ? raw + 64 : raw;
    static_assert(NMAX % 16 == 0 && bytes % 16 == 0, "16-byte aligned layout");
    // byte offset of entry (i, j) inside a 4 x 4 block (a, b): its 16-byte
    // pieces are permuted by the lane groups that read the block's rows and
    // columns together, so that those reads use different banks
    __device__ static __forceinline__ int swz(int a, int b) { return (((a / NR) & 1) << 4) ^ (((b / NR) & 3) << 5); }
    __device__ static __forceinline__ int block(int a, int b) { return (a * (a + 1) / 2 + b) * 128; }
    __device__ static __forceinline__ int at(int i, int j) {  // i / 4 >= j / 4
        return block(i >> 2, j >> 2) + ((((i & 3) << 5) + ((j & 3) << 3)) ^ swz(i >> 2, j >> 2));
    }
    // a block's systems, then what it shares for the pairs with data
    static constexpr int WARPS = solve32_warps(NMAX);
    static constexpr int SYS = 2 * WARPS;
    static constexpr int CHUNK = 4 * WARPS;  // data rows evaluated at a time
    struct Shared {
        double u[CHUNK][3];       // a datum's lag to its system's node, in the model's frame
        unsigned long long mask[SYS];  // the systems' neighbours that are data
        int n[SYS], g[SYS], dom[SYS];
        unsigned short row[CHUNK];     // system << 6 | neighbour
        unsigned short first[2][CHUNK];  // their pairs' numbers: with the grid and the node, with earlier data
        unsigned char place[SYS][NMAX];  // row of the matrix a neighbour stands in
        unsigned char order[SYS][NMAX];  // the grid neighbours, then the data
        unsigned char same[SYS];  // 1: a datum and another neighbour are one point
        unsigned short total[2];
    };
    static constexpr int block_bytes = SYS * bytes + (int)sizeof(Shared);
};

__device__ __forceinline__ KF kf_from_double(double v) {
    const double shift = 1.5 * 16777216.0;  // 1.5 x 2^24: the sum's low word is v in units of 2^-28
    const double t = v + shift;
    return {__double2loint(t), (float)(v - (t - shift))};
}

// the entry as a double-FP32 value (exact up to the second float's rounding)
__device__ __forceinline__ DF kf_df(KF v) {
    const float f = __int2float_rn(v.hi);
    const float rest = __fmaf_rn(__int2float_rn(v.hi - __float2int_rn(f)), 1.0f / KFIX, v.lo);
    return df_fast_two_sum(__fmul_rn(f, 1.0f / KFIX), rest);
}

// w / 2^24 of an integer weight as a double-FP32 value (exact)
__device__ __forceinline__ DF wfix_df(int w) {
    const float f = __int2float_rn(w);
    return {__fmul_rn(f, 1.0f / WFIX), __fmul_rn(__int2float_rn(w - __float2int_rn(f)), 1.0f / WFIX)};
}

__device__ __forceinline__ NbInfo nb_of(const SolveArgs& a, int id) {
    NbInfo in;
    if (id < a.grid.N) {
        cell_of(a.grid, id, in.c0, in.c1, in.c2);
        in.did = -1;
    } else {
        in.c0 = in.c1 = in.c2 = 0;
        in.did = id - (int)a.grid.N;
    }
    return in;
}

// normalized covariance between two points of the augmented set in FP64: a
// call, so that its code stays out of the solve's own
__device__ __noinline__ KF kcov64n(const SolveArgs& a, NbInfo p, NbInfo q) {
    return kf_from_double(kcov(a, p, q) * a.inv_sill);
}

// lag of datum d to the centroid of cell (c0, c1, c2) in the frame of the
// model's first structure, diag(1 / ranges) R' h
__device__ __noinline__ void datum_lag(const SolveArgs& a, int d, int c0, int c1, int c2, double* u) {
    const GridDev& G = a.grid;
    const double h0 = a.data_xyz[3 * (int64_t)d] - centroid(G, 0, c0);
    const double h1 = a.data_xyz[3 * (int64_t)d + 1] - centroid(G, 1, c1);
    const double h2 = G.dim == 3 ? a.data_xyz[3 * (int64_t)d + 2] - centroid(G, 2, c2) : 0.0;
    const double* W = a.vario.st[0].W;
#pragma unroll
    for (int j = 0; j < 3; ++j) u[j] = W[j] * h0 + W[3 + j] * h1 + W[6 + j] * h2;
}

// normalized covariance of a datum whose lag to the node is u (datum_lag) with
// the grid point d0, d1, d2 cells from the node, for a model of one structure;
// hit = false where the lag is too short to tell it from zero this way
__device__ __noinline__ KF datum_cov(const SolveArgs& a, const double* u, int d0, int d1, int d2, bool& hit) {
    const VarioStructDev& v = a.vario.st[0];
    const double x0 = (double)d0, x1 = (double)d1;
    double s = 0.0;
    if (a.grid.dim == 3) {
        const double x2 = (double)d2;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double t = fma(-v.E[j], x0, fma(-v.E[3 + j], x1, fma(-v.E[6 + j], x2, u[j])));
            s = fma(t, t, s);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const double t = fma(-v.E[j], x0, fma(-v.E[3 + j], x1, u[j]));
            s = fma(t, t, s);
        }
    }
    hit = __double2hiint(s) > a.s_near;
    const unsigned long long x = __umul64hi(shape_fixed(v.type, s), a.ratio63);  // 2^-61
    const int hi = (int)((x + (1ull << 32)) >> 33);
    return {hi, __fmul_rn(__ll2float_rn((long long)(x - ((unsigned long long)hi << 33))), 4.3368086899420177e-19f)};
}

// the same, from the lag table where it holds the pair
__device__ __forceinline__ KF kcovn(const SolveArgs& a, const NbInfo& p, const NbInfo& q) {
    if (p.did < 0 && q.did < 0) {
        const CovLut& t = a.lut;
        const int L0 = q.c0 - p.c0, L1 = q.c1 - p.c1, L2 = q.c2 - p.c2;
        if (t.cn != nullptr && L0 >= -t.e[0] && L0 <= t.e[0] && L1 >= -t.e[1] && L1 <= t.e[1] && L2 >= -t.e[2] &&
            L2 <= t.e[2]) {
            const int2 v = t.cn[(L0 + t.e[0]) + t.w[0] * ((L1 + t.e[1]) + t.w[1] * (L2 + t.e[2]))];
            return {v.x, __int_as_float(v.y)};
        }
    }
    return kcov64n(a, p, q);
}

__device__ __forceinline__ DF df_mul(DF a, DF b) {
    const float p = __fmul_rn(a.hi, b.hi);
    const float e = __fmaf_rn(a.hi, b.hi, -p);
    return df_fast_two_sum(p, __fadd_rn(e, __fmaf_rn(a.hi, b.lo, __fmul_rn(a.lo, b.hi))));
}

// reductions over the 16 lanes of a half warp
__device__ __forceinline__ float half_max(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(FULL_MASK, v, o));
    return v;
}
__device__ __forceinline__ double half_sum(double v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}
__device__ __forceinline__ DF half_sum_df(DF v) {
#pragma unroll 1
    for (int o = 8; o > 0; o >>= 1) v = df_add(v, shfl_xor_df(v, o));
    return v;
}

// Sums a lane keeps over the systems its half warp solves, added to the
// problem's counters when the half leaves the problem.
struct SolveTally {
    uint32_t m = 0, warm = 0;
    float l1 = 0.0f;
    __device__ __forceinline__ void flush(const SolveArgs& a, int l16) {
        if (l16 == 0) {
            if (a.sum_m && m) atomicAdd(a.sum_m, (unsigned long long)m);
            if (a.n_warm && warm) atomicAdd(a.n_warm, (unsigned long long)warm);
            if (a.wl1_max && l1 > 0.0f) atomicMax(a.wl1_max, __float_as_uint(l1));
        }
        m = warm = 0;
        l1 = 0.0f;
    }
};

// f(0), f(1), .. f(N - 1) with constant indices: every use of a register array
// inside is resolved before the compiler decides where the array lives (the
// large triangular loops below stay in local memory under #pragma unroll)
template <class F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
    static_for_impl(f, std::make_integer_sequence<int, N>{});
}

// registers of the lower triangle's rows, two entries each: row i holds
// entries 0 .. i (and one unused past an even i) from register tri2(i)
__host__ __device__ constexpr int tri2(int i) { return (i / 2) * (i / 2 + 1) + (i & 1) * (i / 2 + 1); }

// vector of NP floats (a lane group's entries) from shared memory, in pairs
template <int NP>
__device__ __forceinline__ void load_vec(const float* p, F2 (&v)[NP / 2]) {
#pragma unroll
    for (int i = 0; i < NP / 4; ++i) {
        const ulonglong2 q = reinterpret_cast<const ulonglong2*>(p)[i];
        v[2 * i] = q.x;
        v[2 * i + 1] = q.y;
    }
}

// four entries of a system's row from one 4 x 4 block in shared memory: a row
// of the block (two 16-byte reads) or a column (four reads of 8), chosen per
// lane by predicates, so that lanes on both sides of the diagonal stay together
template <int OROW, int OCOL>
__device__ __forceinline__ void lds_block(bool row, uint32_t pr0, uint32_t pr1, uint32_t pc0, uint32_t pc1, uint32_t pc2,
                                          uint32_t pc3, int2 (&e)[4]) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.s32 p, %14, 0;\n\t"
        "@p ld.shared.v4.b32 {%0, %1, %2, %3}, [%8 + %15];\n\t"
        "@p ld.shared.v4.b32 {%4, %5, %6, %7}, [%9 + %15];\n\t"
        "@!p ld.shared.v2.b32 {%0, %1}, [%10 + %16];\n\t"
        "@!p ld.shared.v2.b32 {%2, %3}, [%11 + %16];\n\t"
        "@!p ld.shared.v2.b32 {%4, %5}, [%12 + %16];\n\t"
        "@!p ld.shared.v2.b32 {%6, %7}, [%13 + %16];\n\t}"
        : "=&r"(e[0].x), "=&r"(e[0].y), "=&r"(e[1].x), "=&r"(e[1].y), "=&r"(e[2].x), "=&r"(e[2].y), "=&r"(e[3].x),
          "=&r"(e[3].y)
        : "r"(pr0), "r"(pr1), "r"(pc0), "r"(pc1), "r"(pc2), "r"(pc3), "r"((int)row), "n"(OROW), "n"(OCOL)
        : "memory");
}

// One system per half warp: node g (live: this half has one) of the problem
// `a` with n_all neighbours, ids nid (lane l of the half holds neighbours l +
// 16 s), table row pos; a0 / a1 and base0: the two halves' problems and the
// first half's shared-memory slot (the FP64 evaluations of both systems share
// the warp).
template <int NMAX, bool BATCH>
__device__ __forceinline__ void solve32_pair(const SolveArgs& a, const SolveArgs* __restrict__ doms, int dom,
                                             const SweepTables<float>& tab, int64_t pos, int g, bool live, int n_all,
                                             const int (&nid)[NMAX / 16], unsigned char* smem, SolveTally& tl) {
    using S = Sys32<NMAX>;
    constexpr int NP = S::NP, NR = S::NR;
    const int lane = threadIdx.x & 31, half = lane >> 4, l16 = lane & 15, r = l16 >> 2, c = l16 & 3;
    const int sys = threadIdx.x >> 4;  // of the block's systems
    unsigned char* base = smem + sys * S::bytes;
    typename S::Shared& sh = *reinterpret_cast<typename S::Shared*>(smem + S::SYS * S::bytes);
    auto problem = [&](int es) -> const SolveArgs& {  // of the block's system es
        if constexpr (BATCH) return doms[sh.dom[es]];
        else return a;
    };
    unsigned char* Kb = base;
    KF* C = reinterpret_cast<KF*>(base + S::K);
    float* v0 = reinterpret_cast<float*>(base + S::K + S::C);
    float* v1 = v0 + NMAX;
    float* v2 = v1 + NMAX;
    float* dinv = v2 + NMAX;
    const int k = a.k;
    const bool prior = n_all < a.nmin;        // fewer than minneighbors (or no system)
    int n = prior ? 0 : n_all;
    const int nw = max(n, __shfl_xor_sync(FULL_MASK, n, 16));  // warp-uniform
    int status = prior ? SGS_NODE_PRIOR_NMIN_ : SGS_NODE_KRIGED_;
    DF sigma = {a.sd_sill[0], a.sd_sill[1]};
    bool accept = true;
    unsigned char* place = sh.place[sys];
    const int32_t* __restrict__ nrow = a.nbr + (int64_t)g * k;
    // vectors are stored as [index % 4][index / 4]; this lane holds entries
    // c + 4 (NR r + s), s < NR, of the vectors the solves produce
    const int own = c * NP + NR * r;
    DF w[NR];
#pragma unroll
    for (int s = 0; s < NR; ++s) w[s] = {0.0f, 0.0f};
    if (__syncthreads_or(nw > 0)) {  // block-uniform; the block's warps stay in step
        // ---- neighbours, their lag-table offsets and c ----
        unsigned long long dmask = 0;  // neighbours that are data, in order
        bool fits = true;  // every grid neighbour within half the table's extents
        {
            const CovLut& T = a.lut;
            const int lw0 = T.w[0], lw1 = T.w[1];
            const int lcentre = T.e[0] + lw0 * (T.e[1] + lw1 * T.e[2]);
            NbInfo self = {0, 0, 0, -1};
            if (n > 0) cell_of(a.grid, g, self.c0, self.c1, self.c2);
            int* lin = reinterpret_cast<int*>(v0);
            // Order of the matrix: grid neighbours by their linear table
            // offset (z, then y, then x), data last.  The table index of a
            // pair is the difference of its offsets, so the 16 pairs of a 4 x
            // 4 block then read 4 to 5 lines of the table instead of 10 or 11
            // (distance order), and L1 serves a gather line by line.
            int key[NMAX / 16], off[NMAX / 16];
            int* keys = reinterpret_cast<int*>(v1);
#pragma unroll
            for (int s = 0; s < NMAX / 16; ++s) {
                const int q = l16 + 16 * s;
                off[s] = 0;
                key[s] = (1 << 30) + NMAX + q;  // past the system
                if (q < n) {
                    const NbInfo in = nb_of(a, nid[s]);
                    if (in.did < 0) {
                        const int d0 = in.c0 - self.c0, d1 = in.c1 - self.c1, d2 = in.c2 - self.c2;
                        fits = fits && 2 * abs(d0) <= T.e[0] && 2 * abs(d1) <= T.e[1] && 2 * abs(d2) <= T.e[2];
                        key[s] = off[s] = d0 + lw0 * (d1 + lw1 * d2);
                    } else {
                        key[s] = (1 << 30) + q;
                    }
                }
                keys[q] = key[s];
                const unsigned bal = __ballot_sync(FULL_MASK, key[s] >= (1 << 30) && q < n);
                dmask |= (unsigned long long)((bal >> (16 * half)) & 0xffffu) << (16 * s);
            }
            // without a table the offsets may collide: neighbour order then
            const unsigned fo = __ballot_sync(FULL_MASK, fits);
            const bool ordered = T.cn != nullptr && ((fo >> (16 * half)) & 0xffffu) == 0xffffu;
            __syncwarp();
            int pl[NMAX / 16];
#pragma unroll
            for (int s = 0; s < NMAX / 16; ++s) pl[s] = 0;
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                const int4 kj = reinterpret_cast<const int4*>(keys)[j];
#pragma unroll
                for (int s = 0; s < NMAX / 16; ++s)
                    pl[s] += (kj.x < key[s]) + (kj.y < key[s]) + (kj.z < key[s]) + (kj.w < key[s]);
            }
#pragma unroll
            for (int s = 0; s < NMAX / 16; ++s) {
                const int q = l16 + 16 * s;
                if (!ordered) pl[s] = q;
                place[q] = (unsigned char)pl[s];
                lin[(pl[s] & 3) * NP + (pl[s] >> 2)] = off[s];
            }
            fits = ordered;
            __syncwarp();
            if (fits) {
                // Lags of grid pairs: table index centre + lin[i] - lin[j].
                // Every neighbour's lag fits half the extents, so every pair's
                // index is inside the table; data and padding take the
                // query's own cell (lin = 0), are read like the others and
                // then overwritten (data) or never used (padding).
                const int2* __restrict__ lut = T.cn + lcentre;
                int lc[NP];
#pragma unroll
                for (int i = 0; i < NP / 4; ++i) {
                    const int4 y = reinterpret_cast<const int4*>(lin + c * NP)[i];
                    lc[4 * i] = y.x, lc[4 * i + 1] = y.y, lc[4 * i + 2] = y.z, lc[4 * i + 3] = y.w;
                }
#pragma unroll
                for (int s = 0; s < NMAX / 16; ++s) {
                    const int q = l16 + 16 * s;
                    const int2 x = lut[-lin[(q & 3) * NP + (q >> 2)]];
                    C[q] = {x.x, __int_as_float(x.y)};
                }
                // two block rows at a time: their gathers are all issued
                // before the first is stored
                const int l8 = l16 * 8;
                static_for<NP / 2>([&](auto im) {
                    constexpr int m = 2 * im;
                    if (4 * m < nw) {
                        const int2 *lr0 = lut + lin[r * NP + m], *lr1 = lut + lin[r * NP + m + 1];
                        int2 e0[m + 1], e1[m + 2];
                        static_for<m + 1>([&](auto ib) { e0[ib] = __ldg(lr0 - lc[ib]); });
                        static_for<m + 2>([&](auto ib) { e1[ib] = __ldg(lr1 - lc[ib]); });
                        static_for<m + 1>([&](auto ib) {
                            *reinterpret_cast<int2*>(Kb + S::block(m, ib) + (l8 ^ S::swz(m, ib))) = e0[ib];
                        });
                        static_for<m + 2>([&](auto ib) {
                            *reinterpret_cast<int2*>(Kb + S::block(m + 1, ib) + (l8 ^ S::swz(m + 1, ib))) = e1[ib];
                        });
                    }
                });
            } else {
                // no table, or a neighbour outside it (a batch's capped
                // table): every grid pair by itself
#pragma unroll 1
                for (int e = l16; e < S::K / 8; e += 16) reinterpret_cast<KF*>(Kb)[e] = {0, 0.0f};
#pragma unroll 1
                for (int q = l16; q < NMAX; q += 16) {
                    C[q] = {0, 0.0f};
                    if (q < n && nrow[q] < a.grid.N) C[q] = kcovn(a, nb_of(a, nrow[q]), self);
                }
            }
            __syncwarp();
            if (!fits)
#pragma unroll 1
                for (int i = 0; i < n; ++i) {
                    const NbInfo ni = nb_of(a, nrow[i]);
                    if (ni.did >= 0) continue;
#pragma unroll 1
                    for (int j = l16; j <= i; j += 16) {
                        const NbInfo nj = nb_of(a, nrow[j]);
                        if (nj.did >= 0) continue;
                        const KF x = kcovn(a, nj, ni);
                        *reinterpret_cast<KF*>(Kb + S::at(i, j)) = x;
                        if ((i >> 2) == (j >> 2)) *reinterpret_cast<KF*>(Kb + S::at(j, i)) = x;
                    }
                }
            __syncwarp();
        }
        // ---- pairs with a datum: FP64, over the whole block ----
#pragma unroll
        for (int s = 0; s < NMAX / 16; ++s) {
            const int q = l16 + 16 * s;
            const unsigned long long lower = (1ull << q) - 1;
            const int nd = __popcll(dmask & lower);
            if (q < n) sh.order[sys][(dmask >> q) & 1 ? n - __popcll(dmask) + nd : q - nd] = (unsigned char)q;
        }
        if (l16 == 0) {
            sh.mask[sys] = dmask;
            sh.same[sys] = 0;
            sh.n[sys] = n;
            sh.g[sys] = g;
            sh.dom[sys] = dom;
        }
        const int rows = __syncthreads_or(dmask != 0) ? -1 : 0;  // unknown number, or none
#pragma unroll 1
        for (int r0 = 0, left = rows; left != 0; r0 += S::CHUNK) {  // block-uniform
            // the r0-th and later data rows of the block's systems
            int total = 0;
            for (int e = 0; e < S::SYS; ++e) total += __popcll(sh.mask[e]);
            const int nr = min(total - r0, S::CHUNK);
            left = total - r0 - nr;
            int counts[2] = {0, 0};  // pairs of each kind in the chunk
            if (threadIdx.x < 32) {
                if (lane < nr) {
                    int t = r0 + lane, es = 0;
                    while (t >= __popcll(sh.mask[es])) t -= __popcll(sh.mask[es++]);
                    const int ng = sh.n[es] - __popcll(sh.mask[es]), da = sh.order[es][ng + t];
                    sh.row[lane] = (unsigned short)(es << 6 | da);
                    counts[0] = ng + 1;
                    counts[1] = t;
                    const SolveArgs& ah = problem(es);
                    if (ah.vario.ns == 1) {
                        int c0, c1, c2;
                        cell_of(ah.grid, sh.g[es], c0, c1, c2);
                        datum_lag(ah, ah.nbr[(int64_t)sh.g[es] * ah.k + da] - (int)ah.grid.N, c0, c1, c2, sh.u[lane]);
                    }
                }
                __syncwarp();
#pragma unroll
                for (int kind = 0; kind < 2; ++kind) {
                    int end = counts[kind];
#pragma unroll
                    for (int o = 1; o < S::CHUNK; o <<= 1) {
                        const int y = __shfl_up_sync(FULL_MASK, end, o);
                        if (lane >= o) end += y;
                    }
                    if (lane < S::CHUNK) sh.first[kind][lane] = (unsigned short)(end - counts[kind]);
                    if (lane == S::CHUNK - 1) sh.total[kind] = (unsigned short)end;
                }
            }
            __syncthreads();
            // A pair to a thread, none of them idle: first the rows' pairs with
            // grid neighbours and the node, then those with earlier data, so that a
            // warp takes one kind.  With a slot for every pair of a row and the
            // system's largest size, two thirds of them empty, 40k systems of
            // 40 data (spherical) took 6.5 ms, more than one warp per system
            // had (4.9); this takes 3.0, and systems of 20 0.76 (1.93, 1.35).
#pragma unroll 1
            for (int kind = 0; kind < 2; ++kind) {
                const int pairs = sh.total[kind];
#pragma unroll 1
                for (int item = threadIdx.x; item < pairs; item += 32 * S::WARPS) {
                    int ei = 0;
#pragma unroll
                    for (int step = 8; step > 0; step >>= 1)
                        if (ei + step < nr && sh.first[kind][ei + step] <= item) ei += step;
                    const int e = sh.row[ei], es = e >> 6, da = e & 63, j = item - sh.first[kind][ei];
                    const SolveArgs& ah = problem(es);
                    unsigned char* bh = smem + es * S::bytes;
                    const int gh = sh.g[es], ng = sh.n[es] - __popcll(sh.mask[es]);
                    const int32_t* rowh = ah.nbr + (int64_t)gh * ah.k;
                    const bool own = kind == 0 && j == ng;  // the pair with the node (its own diagonal is 1)
                    const int q = own ? da : sh.order[es][kind ? ng + j : j];
                    const NbInfo nq = nb_of(ah, own ? gh : rowh[q]);
                    KF x;
                    bool hit = false;
                    if (kind == 0 && ah.vario.ns == 1) {
                        int c0, c1, c2;
                        cell_of(ah.grid, gh, c0, c1, c2);
                        x = datum_cov(ah, sh.u[ei], nq.c0 - c0, nq.c1 - c1, nq.c2 - c2, hit);
                    }
                    if (!hit) x = kcov64n(ah, nq, nb_of(ah, rowh[da]));
                    const int pd = sh.place[es][da];
                    if (own) {
                        reinterpret_cast<KF*>(bh + S::K)[pd] = x;
                        *reinterpret_cast<KF*>(bh + S::at(pd, pd)) = {(int)KFIX, 0.0f};
                    } else {
                        // Correlation 1: the variance of their difference, 2 (1 - K), bounds the
                        // later one's pivot, which is then far below the singular rule's 1e-10.
                        if (x.hi == (int)KFIX && fabsf(x.lo) <= 1e-12f) sh.same[es] = 1;
                        const int pq = sh.place[es][q], i = max(pq, pd), jj = min(pq, pd);
                        *reinterpret_cast<KF*>(bh + S::at(i, jj)) = x;
                        if ((i >> 2) == (jj >> 2)) *reinterpret_cast<KF*>(bh + S::at(jj, i)) = x;
                    }
                }
            }
            __syncthreads();
        }
        const bool singular = sh.same[sys];
        // ---- the FP32 LHS into registers (identity past the system) ----
        F2 A[tri2(NP)];
#define SLOT(a_, b_) (((b_) & 1) ? f2_hi(A[tri2(a_) + (b_) / 2]) : f2_lo(A[tri2(a_) + (b_) / 2]))
        static_for<NP>([&](auto ia) {
            constexpr int ba = ia;
            const bool in = r + 4 * ba < n;
            const float sc = in ? 1.0f / KFIX : 0.0f;
            auto entry = [&](int bb) {
                const float v = __fmul_rn(
                    __int2float_rn(*reinterpret_cast<const int*>(Kb + S::block(ba, bb) + ((l16 * 8) ^ S::swz(ba, bb)))), sc);
                return bb == ba && !in && r == c ? 1.0f : v;
            };
            static_for<ba / 2 + 1>([&](auto ib) {
                constexpr int bb = 2 * ib;
                A[tri2(ba) + ib] = f2_pack(entry(bb), bb + 1 <= ba ? entry(bb + 1) : 0.0f);
            });
        });
        // ---- elimination: A -> M = L^-1 (below the diagonal) and D ----
        // Step kk = 4p + t: v_j is row kk of M for j < kk and column kk of the
        // Schur complement for j > kk; every row i > kk takes -l_i v_j with
        // l_i = a_i,kk / d, and v_kk = d + 1 turns its own a_i,kk into -l_i.
        // Lane (r, c) needs v at its rows r + 4a and its columns c + 4b: both
        // come by shuffles from the lanes that hold them (no shared memory,
        // no divergence).  The steps of a block column run in a rolled loop
        // (every register index is static); rows above the pivot are
        // finished, so block rows < p are left out.
        bool ok = true;
        static_for<NP>([&](auto ip) {
            constexpr int p = ip;
            if (4 * p < nw) {
#pragma unroll 1
                for (int t = 0; t < 4; ++t) {
                    const int h16 = lane & 16;
                    const int src_r = h16 | (r << 2) | t;  // column kk in row r (block rows >= p)
                    const int src_c = h16 | (c << 2) | t;  // column kk in row c
                    const int src_m = h16 | (t << 2) | c;  // row kk, column c (block columns < p)
                    const float d = __shfl_sync(FULL_MASK, SLOT(p, p), h16 | (t << 2) | t);
                    float u[NP], vcs[NP];
                    static_for<NP>([&](auto ij) {
                        constexpr int j = ij;
                        if constexpr (j < p) vcs[j] = __shfl_sync(FULL_MASK, SLOT(p, j), src_m);
                        else if constexpr (j == p) vcs[j] = __shfl_sync(FULL_MASK, SLOT(p, p), c > t ? src_c : src_m);
                        else vcs[j] = __shfl_sync(FULL_MASK, SLOT(j, p), src_c);
                    });
                    static_for<NP - p>([&](auto ii) {
                        constexpr int i = p + ii;
                        u[i] = __shfl_sync(FULL_MASK, SLOT(i, p), src_r);
                    });
                    // the inverse is a preconditioner only: the approximate
                    // reciprocal (pivots lie in (1e-3, 1], no denormals) is enough
                    float inv;
                    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(d));
                    ok = ok && d > 1e-3f;
                    if (l16 == 0) dinv[t * NP + p] = inv;
                    if (c == t) vcs[p] = __fadd_rn(d, 1.0f);
                    F2 vc[NP / 2];
                    static_for<NP / 2>([&](auto ij) { vc[ij] = f2_pack(vcs[2 * ij], vcs[2 * ij + 1]); });
                    static_for<NP - p>([&](auto ii) {
                        constexpr int i = p + ii;
                        float ui = __fmul_rn(u[i], -inv);
                        if (i == p && r <= t) ui = 0.0f;
                        const F2 uu = f2_pack(ui, ui);
                        static_for<i / 2 + 1>([&](auto ij) {
                            constexpr int j = ij;
                            A[tri2(i) + j] = f2_fma(uu, vc[j], A[tri2(i) + j]);
                        });
                    });
                }
            }
        });
        accept = ok;
        // unit diagonal of M, nothing above it
        static_for<NP>([&](auto ii) {
            constexpr int i = ii;
            const float dg = r > c ? SLOT(i, i) : (r == c ? 1.0f : 0.0f);
            A[tri2(i) + i / 2] = (i & 1) ? f2_pack(SLOT(i, i - 1), dg) : f2_pack(dg, 0.0f);
        });
        __syncwarp();
        // ---- weights: w = M' D^-1 M c (or the network's prediction), then
        // corrections from the exact residual ----
        const int steps = a.refine_steps;
        const bool warm = a.w_init != nullptr;
        float prev = 0.0f, last = 0.0f, wmax = 0.0f;
        // the residual of the last iterate w and the correction it gave (the
        // weights are w + sd)
        float sr[NR], sd[NR];
#pragma unroll
        for (int s = 0; s < NR; ++s) sr[s] = sd[s] = 0.0f;
        bool early = false, done = n == 0 || singular;  // half-uniform
        float x[NR];
        if (warm) {
#pragma unroll
            for (int s = 0; s < NMAX / 16; ++s) {
                const int q = l16 + 16 * s;
                v2[place[q]] = q < n ? a.w_init[(int64_t)g * k + q] : 0.0f;
            }
            __syncwarp();
#pragma unroll
            for (int s = 0; s < NR; ++s) w[s] = {v2[c + 4 * (NR * r + s)], 0.0f};
            __syncwarp();
        }
        for (int it = warm ? 0 : -1;; ++it) {  // block-uniform (only plans are warm-started)
            if (__syncthreads_and(done)) break;
            if (__all_sync(FULL_MASK, done)) continue;  // this warp waits for the others
            if (it >= 0) {
                if (it > 0 && !done)
#pragma unroll
                    for (int s = 0; s < NR; ++s) w[s] = df_add(w[s], {sd[s], 0.0f});
                // the iterate as integers: W1 2^-24 (+ W2 2^-48 after a correction)
                float wm = 0.0f;
                auto first = [](const DF& v) { return __float2int_rn(__fmul_rn(v.hi, WFIX)); };  // W1
                auto second = [&](const DF& v) {                                                 // W2
                    const DF q = wfix_df(first(v));
                    const float rest = __fadd_rn(__fsub_rn(__fsub_rn(v.hi, q.hi), q.lo), v.lo);
                    return __float2int_rn(__fmul_rn(rest, WFIX2));
                };
#pragma unroll
                for (int s = 0; s < NR; ++s) {
                    const int i = c + 4 * (NR * r + s);
                    if (!done) {
                        const DF q = wfix_df(first(w[s]));
                        const DF y = df_two_sum(q.hi, it > 0 ? __fmul_rn(__int2float_rn(second(w[s])), 1.0f / WFIX2) : 0.0f);
                        w[s] = df_fast_two_sum(y.hi, __fadd_rn(y.lo, q.lo));
                    }
                    wm = fmaxf(wm, fabsf(w[s].hi));
                    const int W1 = first(w[s]);
                    reinterpret_cast<int*>(v1)[i] = -W1;
                    v2[i] = -wfix_df(W1).hi;
                }
                wm = half_max(wm);
                if (it == 0) wmax = wm;
                if (!done && !(wm < WLIM)) accept = false;
                __syncwarp();
                // residual c - K w of the own entries, the two parts of the
                // weights one after the other
#pragma unroll 1
                for (int part = 0;; ++part) {  // warp-uniform
                    long long acc[NR];
                    float accf[NR];
                    uint32_t rowp[NR];  // block row I of the triangle
                    const uint32_t kaddr = (uint32_t)__cvta_generic_to_shared(Kb);
#pragma unroll
                    for (int s = 0; s < NR; ++s) {
                        const int I = NR * r + s;
                        const KF ci = C[c + 4 * I];
                        acc[s] = part ? 0 : (long long)ci.hi << 24;
                        accf[s] = part ? 0.0f : ci.lo;
                        rowp[s] = kaddr + S::block(I, 0);
                    }
                    // Entry (i, 4J + j) lies in row c of block (I, J) up to the
                    // diagonal and in column c of block (J, I) past it (a
                    // rolled loop: 80 of the registers hold M).
                    uint32_t colp = kaddr + NR * r * 128;  // block row J, from column NR r
#pragma unroll 1
                    for (int J = 0; 4 * J < nw; ++J) {
                        const int4 W = reinterpret_cast<const int4*>(v1)[J];
                        const float4 F = reinterpret_cast<const float4*>(v2)[J];
                        const int G = J / NR;
                        const uint32_t xr = ((c << 5) | ((r & 1) << 4)) ^ (G << 5);
                        const uint32_t pc = colp + ((c << 3) ^ ((G & 1) << 4));
                        static_for<NR>([&](auto is) {
                            constexpr int s = is;
                            int2 e[4];
                            lds_block<0, s * 128>(J <= NR * r + s, rowp[s] + xr, rowp[s] + (xr ^ 16), pc + (r << 5),
                                                  pc + ((r ^ 1) << 5), pc + ((r ^ 2) << 5), pc + ((r ^ 3) << 5), e);
                            acc[s] += (long long)e[0].x * W.x;
                            acc[s] += (long long)e[1].x * W.y;
                            acc[s] += (long long)e[2].x * W.z;
                            acc[s] += (long long)e[3].x * W.w;
                            accf[s] = __fmaf_rn(__int_as_float(e[0].y), F.x, accf[s]);
                            accf[s] = __fmaf_rn(__int_as_float(e[1].y), F.y, accf[s]);
                            accf[s] = __fmaf_rn(__int_as_float(e[2].y), F.z, accf[s]);
                            accf[s] = __fmaf_rn(__int_as_float(e[3].y), F.w, accf[s]);
                            rowp[s] += 128;
                        });
                        colp += (J + 1) * 128;
                    }
                    const float unit = part ? 1.0f / (KFIX * WFIX2) : 1.0f / (KFIX * WFIX);
#pragma unroll
                    for (int s = 0; s < NR; ++s) {
                        const float f = __fadd_rn(__fmul_rn(__ll2float_rn(acc[s]), unit), accf[s]);
                        x[s] = part ? __fadd_rn(x[s], f) : f;
                    }
                    __syncwarp();
                    if (part == 1 || it == 0) break;
#pragma unroll
                    for (int s = 0; s < NR; ++s) {
                        const int i = c + 4 * (NR * r + s);
                        reinterpret_cast<int*>(v1)[i] = -second(w[s]);
                        v2[i] = 0.0f;
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int s = 0; s < NR; ++s) {
                    if (c + 4 * (NR * r + s) >= n) x[s] = 0.0f;
                    if (!done) {
                        sr[s] = x[s];
                        sd[s] = 0.0f;
                    }
                }
                if (it >= steps) done = true;  // steps == 0: no correction
            } else {
#pragma unroll
                for (int s = 0; s < NR; ++s) {
                    const int i = c + 4 * (NR * r + s);
                    x[s] = i < n ? __fmul_rn(__int2float_rn(C[i].hi), 1.0f / KFIX) : 0.0f;
                }
            }
            if (__all_sync(FULL_MASK, done)) continue;
            // ---- x -> M' D^-1 M x ----
#pragma unroll
            for (int s = 0; s < NR; ++s) v0[own + s] = x[s];
            __syncwarp();
            {
                F2 xc[NP / 2];
                float tv[NP], h[NP / 2];
                load_vec<NP>(v0 + c * NP, xc);
                static_for<NP>([&](auto ii) {
                    constexpr int i = ii;
                    F2 t2 = f2_pack(0.0f, 0.0f);
                    static_for<i / 2 + 1>([&](auto ij) {
                        constexpr int j = ij;
                        t2 = f2_fma(A[tri2(i) + j], xc[j], t2);
                    });
                    tv[i] = __fadd_rn(f2_lo(t2), f2_hi(t2));
                });
                // sums over the four lanes of a row, each lane keeping NR of them
#pragma unroll
                for (int i = 0; i < NP / 2; ++i) {
                    const float keep = (c & 2) ? tv[NP / 2 + i] : tv[i], send = (c & 2) ? tv[i] : tv[NP / 2 + i];
                    h[i] = __fadd_rn(keep, __shfl_xor_sync(FULL_MASK, send, 2));
                }
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const float keep = (c & 1) ? h[NR + i] : h[i], send = (c & 1) ? h[i] : h[NR + i];
                    const float y = __fadd_rn(keep, __shfl_xor_sync(FULL_MASK, send, 1));
                    const int e = r * NP + NR * c + i;
                    v1[e] = r + 4 * (NR * c + i) < n ? __fmul_rn(y, dinv[e]) : 0.0f;
                }
                __syncwarp();
                load_vec<NP>(v1 + r * NP, xc);
                F2 z2[NP / 2];
#pragma unroll
                for (int j = 0; j < NP / 2; ++j) z2[j] = f2_pack(0.0f, 0.0f);
                static_for<NP>([&](auto ii) {
                    constexpr int i = ii;
                    const float yi = (i & 1) ? f2_hi(xc[i / 2]) : f2_lo(xc[i / 2]);
                    const F2 yy = f2_pack(yi, yi);
                    static_for<i / 2 + 1>([&](auto ij) {
                        constexpr int j = ij;
                        z2[j] = f2_fma(A[tri2(i) + j], yy, z2[j]);
                    });
                });
#pragma unroll
                for (int j = 0; j < NP / 2; ++j) {
                    tv[2 * j] = f2_lo(z2[j]);
                    tv[2 * j + 1] = f2_hi(z2[j]);
                }
#pragma unroll
                for (int i = 0; i < NP / 2; ++i) {
                    const float keep = (r & 2) ? tv[NP / 2 + i] : tv[i], send = (r & 2) ? tv[i] : tv[NP / 2 + i];
                    h[i] = __fadd_rn(keep, __shfl_xor_sync(FULL_MASK, send, 8));
                }
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const float keep = (r & 1) ? h[NR + i] : h[i], send = (r & 1) ? h[i] : h[NR + i];
                    x[i] = __fadd_rn(keep, __shfl_xor_sync(FULL_MASK, send, 4));
                    if (c + 4 * (NR * r + i) >= n) x[i] = 0.0f;
                }
                __syncwarp();  // the vectors' buffers are rewritten by the next pass
            }
            if (it < 0) {
                if (!warm)
#pragma unroll
                    for (int s = 0; s < NR; ++s) w[s] = {x[s], 0.0f};
                continue;
            }
            float dmax = 0.0f;
#pragma unroll
            for (int s = 0; s < NR; ++s) dmax = fmaxf(dmax, fabsf(x[s]));
            bool finite = true;
#pragma unroll
            for (int s = 0; s < NR; ++s) finite = finite && isfinite(x[s]);
            dmax = half_max(dmax);
            const unsigned fin = __ballot_sync(FULL_MASK, finite);
            if (((fin >> (16 * half)) & 0xffffu) != 0xffffu) dmax = INFINITY;
            if (!done) {
#pragma unroll
                for (int s = 0; s < NR; ++s) {
                    sd[s] = x[s];
                }
                prev = last;
                last = dmax;
                if (it + 1 == steps) {
                    done = true;  // the final weights need no residual
                } else if (it == 0 && !warm && last * last <= 1e-10f * wmax && isfinite(last)) {
                    // One correction is enough when the start was already
                    // good: the start's error is about |d| and the
                    // contraction factor of the FP32 factors about |d| / |w|,
                    // so the corrected weights are off by about |d|^2 / |w|
                    // (measured on the 200x200x100 anisotropic systems:
                    // within a factor 4 of the true error, which is ~1e-12).
                    early = done = true;
                } else if (it >= 1 && prev > 0.0f && last < 0.5f * prev && (last / prev) * last <= 1e-9f &&
                           isfinite(last)) {
                    // Later corrections: stop as soon as the contraction test
                    // passes (a warm start from a prediction needs two).
                    early = done = true;
                }
            }
        }
#undef SLOT
        // the remaining error is about the contraction factor times the last
        // correction
        if (accept && !early && n > 0) {
            if (steps >= 2) {
                const float rho = prev > 0.0f ? last / prev : 0.0f;
                accept = rho < 0.5f && rho * last <= 1e-9f && isfinite(last);
            } else {
                accept = isfinite(last);
            }
        }
        // sigma^2 = sill S(w), S(w) = 1 - w'c - w'r with r = c - K w: equal to
        // 1 - w'c at the exact weights, but stationary there (its error is
        // (w - w*)' K (w - w*)), so it stays accurate where the variance
        // cancels to ~0 (a node on a datum), where sqrt would magnify any
        // error.  It is taken at the final weights w + d: S(w + d) = S(w) -
        // 2 d'r + d' K d, and K d = r up to the inverse's error, so S(w + d) =
        // S(w) - d'r with an error of order |d| |r| x that error.
        DFAcc acc;
        acc.init({0.0f, 0.0f});
#pragma unroll
        for (int s = 0; s < NR; ++s) {
            const int i = c + 4 * (NR * r + s);
            if (i < n) {
                acc.add_prod(w[s], df_add(kf_df(C[i]), {sr[s], 0.0f}));
                acc.add_prod({sd[s], 0.0f}, {sr[s], 0.0f});
                w[s] = df_add(w[s], {sd[s], 0.0f});
            }
        }
        const DF wc = half_sum_df(acc.value());
        if (singular) {
            accept = true;
            status = SGS_NODE_PRIOR_SINGULAR_;
            n = 0;
        }
        if (n > 0) sigma = df_mul(sigma, df_sqrt(df_add({1.0f, 0.0f}, df_neg(wc))));
        __syncwarp();
        if (live && !accept && l16 == 0) a.fallback[atomicAdd(a.nfallback, 1)] = (int32_t)pos;
    }
    __syncthreads();
    // ---- table row: grid neighbours with (hi, lo) weights, data folded into b0
    DF* ws = reinterpret_cast<DF*>(v0);  // the weights in neighbour order (v0, v1)
#pragma unroll
    for (int s = 0; s < NR; ++s) ws[c + 4 * (NR * r + s)] = w[s];
    __syncwarp();
    const bool wr = live && accept;
    int m = 0;
    const int64_t row = wr ? table_row(tab, pos, k) : 0;
    DFAcc b0acc;
    b0acc.init({0.0f, 0.0f});
    float l1 = 0.0f;
#pragma unroll 1
    for (int s = 0; s < NMAX / 16; ++s) {
        const int q = l16 + 16 * s;
        const bool in = wr && q < n;
        const int id = in ? nrow[q] : 0;
        const bool isgrid = in && id < a.grid.N;
        const unsigned bal = (__ballot_sync(FULL_MASK, isgrid) >> (16 * half)) & 0xffffu;
        if (in) {
            const DF wq = ws[place[q]];
            if (isgrid) {
                const int j = m + __popc(bal & ((1u << l16) - 1u));
                tab.idx[row + j] = id + (int32_t)a.node0;
                reinterpret_cast<float2*>(tab.w)[row + j] = make_float2(wq.hi, wq.lo);
                l1 += fabsf(wq.hi);
            } else {
                b0acc.add_prod(wq, df_from_double(a.data_val[id - a.grid.N] - a.mu));
            }
        }
        m += __popc(bal);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) l1 += __shfl_xor_sync(FULL_MASK, l1, o);
    const DF b0 = half_sum_df(b0acc.value());
    if (wr) {
        tl.m += m;
        tl.l1 = fmaxf(tl.l1, l1);
        if (a.w_init && n > 0) tl.warm += 1;
        if (l16 == 0) {
            tab.node[pos] = g + (int32_t)a.node0;
            tab.m[pos] = m;
            reinterpret_cast<float2*>(tab.b0)[pos] = make_float2(b0.hi, b0.lo);
            reinterpret_cast<float2*>(tab.sigma)[pos] = make_float2(sigma.hi, sigma.lo);
            a.status[g] = (int8_t)status;
        }
    }
    if (a.ind_wsum) {  // plans only: both halves have the same problem
        double wsum = 0.0, ds[8];
#pragma unroll
        for (int l = 0; l < 8; ++l) ds[l] = 0.0;
        if (wr)
#pragma unroll 1
            for (int q = l16; q < n; q += 16) {
                const double v = (double)ws[place[q]].hi + (double)ws[place[q]].lo;
                wsum += v;
                if (nrow[q] >= a.grid.N) {
                    const int cat = a.ind_cat[nrow[q] - a.grid.N];
#pragma unroll
                    for (int l = 0; l < 8; ++l)
                        if (l == cat) ds[l] += v;
                }
            }
        wsum = half_sum(wsum);
        if (wr && l16 == 0) a.ind_wsum[pos] = wsum;
#pragma unroll
        for (int l = 0; l < 8; ++l)
            if (l < a.ncat) {
                const double v = half_sum(ds[l]);
                if (wr && l16 == 0) a.ind_dsum[pos * a.ncat + l] = v;
            }
    }
    if (a.w_full && wr) {
#pragma unroll 1
        for (int q = l16; q < k; q += 16) {  // k may be above NMAX in a batch
            const DF wq = ws[q < n ? place[q] : 0];
            a.w_full[(int64_t)g * k + q] = q < n ? (double)wq.hi + (double)wq.lo : 0.0;
        }
        if (l16 == 0) a.sigma_full[g] = (double)sigma.hi + (double)sigma.lo;
    }
    __syncwarp();
}

// neighbour count and ids of node g (g < 0: none) for solve32_pair
template <int NMAX>
__device__ __forceinline__ void read_row(const SolveArgs& a, int g, int l16, int& n, int (&nid)[NMAX / 16]) {
    n = g >= 0 ? a.cnt[g] : 0;
#pragma unroll
    for (int s = 0; s < NMAX / 16; ++s) {
        const int q = l16 + 16 * s;
        nid[s] = g >= 0 && q < a.k ? a.nbr[(int64_t)g * a.k + q] : -1;
    }
}

template <int NMAX>
__global__ void __launch_bounds__(solve32_warps(NMAX) * 32, solve32_blocks(NMAX))
solve_fp32_kernel(const __grid_constant__ SolveArgs a, const SweepTables<float> tab) {
    using S = Sys32<NMAX>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int l16 = threadIdx.x & 15;
    const int64_t nsys = (int64_t)gridDim.x * S::SYS;  // systems of the grid per round
    SolveTally tl;
    // the next round's neighbours are read while this one is solved (a chain
    // of two dependent reads; the node ids one round further ahead)
    const int64_t pos0 = (int64_t)blockIdx.x * S::SYS + (threadIdx.x >> 4);
    auto node_at = [&](int64_t p) { return p < a.P ? a.order[p] : -1; };
    int g = node_at(pos0), g1 = node_at(pos0 + nsys);
    int n, nid[NMAX / 16];
    read_row<NMAX>(a, g, l16, n, nid);
    for (int64_t b0 = (int64_t)blockIdx.x * S::SYS, pos = pos0; b0 < a.P; b0 += nsys, pos += nsys) {  // block-uniform
        const int g2 = node_at(pos + 2 * nsys);
        int n1, nid1[NMAX / 16];
        read_row<NMAX>(a, g1, l16, n1, nid1);
        solve32_pair<NMAX, false>(a, nullptr, 0, tab, pos, max(g, 0), g >= 0, n, nid, smem, tl);
        g = g1;
        g1 = g2;
        n = n1;
#pragma unroll
        for (int s = 0; s < NMAX / 16; ++s) nid[s] = nid1[s];
    }
    tl.flush(a, l16);
}

// Batch form of solve_fp32_kernel: desc[0] positions list[desc[1] ...]
// (systems with at most NMAX neighbours, from any domain), each solved with
// its domain's descriptor.
template <int NMAX>
__global__ void __launch_bounds__(solve32_warps(NMAX) * 32, solve32_blocks(NMAX))
solve_fp32_batch_kernel(const SolveArgs* __restrict__ doms, const int64_t* __restrict__ noff, int ndom,
                        const int32_t* __restrict__ order, const int32_t* __restrict__ list,
                        const int32_t* __restrict__ desc, const SweepTables<float> tab) {
    using S = Sys32<NMAX>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int l16 = threadIdx.x & 15;
    const int64_t n = desc[0];
    const int32_t* lst = list + desc[1];
    const int64_t nsys = (int64_t)gridDim.x * S::SYS;
    int64_t lo = 0, hi = 0;
    int d = 0;
    SolveTally tl;
    for (int64_t b0 = (int64_t)blockIdx.x * S::SYS; b0 < n; b0 += nsys) {  // block-uniform
        const int64_t i = b0 + (threadIdx.x >> 4);
        const bool live = i < n;
        const int64_t pos = lst[live ? i : b0];
        const int64_t gg = order[pos];
        if (gg < lo || gg >= hi) {  // half-uniform
            if (hi > 0) tl.flush(doms[d], l16);
            d = find_domain(noff, ndom, gg);
            lo = noff[d];
            hi = noff[d + 1];
        }
        __syncwarp();
        int nn, nid[NMAX / 16];
        read_row<NMAX>(doms[d], live ? (int)(gg - lo) : -1, l16, nn, nid);
        solve32_pair<NMAX, true>(doms[d], doms, d, tab, pos, (int)(gg - lo), live, nn, nid, smem, tl);
    }
    if (hi > 0) tl.flush(doms[d], l16);
}

template <int NMAX>
static cudaError_t launch_solve32(const SolveArgs& a, const SweepTables<float>& t, cudaStream_t s) {
    using S = Sys32<NMAX>;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e =
        cudaFuncSetAttribute(solve_fp32_kernel<NMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::block_bytes);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, solve_fp32_kernel<NMAX>, S::WARPS * 32, S::block_bytes);
    if (per_sm < 1) per_sm = 1;
    int64_t want = (a.P + S::SYS - 1) / S::SYS;
    int blocks = (int)(want < (int64_t)nsm * per_sm ? want : (int64_t)nsm * per_sm);
    if (blocks < 1) blocks = 1;
    solve_fp32_kernel<NMAX><<<blocks, S::WARPS * 32, S::block_bytes, s>>>(a, t);
    return cudaGetLastError();
}

cudaError_t launch_solve_fp32(const SolveArgs& a, const SweepTables<float>& t, cudaStream_t s) {
    if (a.k <= 16) return launch_solve32<16>(a, t, s);
    if (a.k <= 32) return launch_solve32<32>(a, t, s);
    if (a.k <= 48) return launch_solve32<48>(a, t, s);
    return launch_solve32<64>(a, t, s);
}

cudaError_t launch_solve_fp64_into_fp32(const SolveArgs& a, const SweepTables<float>& t, cudaStream_t s) {
    return launch_solve<float>(a, t, s);
}

// ---------------------------------------------------------------------------
// Batches of domains.  Persistent grids (as many blocks as fit on the SMs)
// walk a device-resident list whose length is read on the device, so the
// launches need nothing from the host and can be captured in a graph.
template <int NMAX>
static cudaError_t launch_solve32_batch(const SolveArgs* doms, const int64_t* noff, int ndom, const int32_t* order,
                                        const int32_t* list, const int32_t* desc, const SweepTables<float>& t,
                                        int nsm, cudaStream_t s) {
    using S = Sys32<NMAX>;
    cudaError_t e =
        cudaFuncSetAttribute(solve_fp32_batch_kernel<NMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::block_bytes);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, solve_fp32_batch_kernel<NMAX>, S::WARPS * 32, S::block_bytes);
    if (per_sm < 1) per_sm = 1;
    solve_fp32_batch_kernel<NMAX><<<nsm * per_sm, S::WARPS * 32, S::block_bytes, s>>>(doms, noff, ndom, order, list, desc, t);
    return cudaGetLastError();
}

cudaError_t launch_solve_fp32_batch(int nmax, const SolveArgs* doms, const int64_t* noff, int ndom,
                                    const int32_t* order, const int32_t* list, const int32_t* desc,
                                    const SweepTables<float>& t, int nsm, cudaStream_t s) {
    switch (nmax) {
        case 8:
        case 16: return launch_solve32_batch<16>(doms, noff, ndom, order, list, desc, t, nsm, s);
        case 32: return launch_solve32_batch<32>(doms, noff, ndom, order, list, desc, t, nsm, s);
        case 48: return launch_solve32_batch<48>(doms, noff, ndom, order, list, desc, t, nsm, s);
        case 64: return launch_solve32_batch<64>(doms, noff, ndom, order, list, desc, t, nsm, s);
        default: return cudaErrorInvalidValue;
    }
}

template <typename O>
static cudaError_t launch_solve64_batch(int kl, const SolveArgs* doms, const int64_t* noff, int ndom,
                                        const int32_t* order, const int32_t* list, const int32_t* desc,
                                        const SweepTables<O>& t, int nsm, cudaStream_t s) {
    if (kl < 1 || kl > KMAX) return cudaErrorInvalidValue;
    const size_t smem = warp_smem_bytes(kl) * SOLVE_WARPS;
    cudaError_t e = cudaFuncSetAttribute(solve_batch_kernel<O>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kSolveSmemMax);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, solve_batch_kernel<O>, SOLVE_WARPS * 32, smem);
    if (per_sm < 1) per_sm = 1;
    solve_batch_kernel<O><<<nsm * per_sm, SOLVE_WARPS * 32, smem, s>>>(doms, noff, ndom, order, list, desc, kl, t);
    return cudaGetLastError();
}

cudaError_t launch_solve_fp64_batch(int kl, const SolveArgs* doms, const int64_t* noff, int ndom,
                                    const int32_t* order, const int32_t* list, const int32_t* desc,
                                    const SweepTables<double>& t, int nsm, cudaStream_t s) {
    return launch_solve64_batch<double>(kl, doms, noff, ndom, order, list, desc, t, nsm, s);
}

cudaError_t launch_solve_fp64_into_fp32_batch(int kl, const SolveArgs* doms, const int64_t* noff, int ndom,
                                              const int32_t* order, const int32_t* list, const int32_t* desc,
                                              const SweepTables<float>& t, int nsm, cudaStream_t s) {
    return launch_solve64_batch<float>(kl, doms, noff, ndom, order, list, desc, t, nsm, s);
}

// ---------------------------------------------------------------------------
__global__ void tables_to_fp64_kernel(const SweepTables<float> src, SweepTables<double> dst, int64_t P,
                                      int64_t entries) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < entries; i += stride)
        dst.w[i] = (double)src.w[2 * i] + (double)src.w[2 * i + 1];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < P; i += stride) {
        dst.b0[i] = (double)src.b0[2 * i] + (double)src.b0[2 * i + 1];
        dst.sigma[i] = (double)src.sigma[2 * i] + (double)src.sigma[2 * i + 1];
    }
}

cudaError_t launch_tables_to_fp64(const SweepTables<float>& src, SweepTables<double>& dst, int64_t P, int64_t entries,
                                  cudaStream_t s) {
    dst.node = src.node;
    dst.m = src.m;
    dst.idx = src.idx;
    dst.off = src.off;
    const int64_t n = entries > P ? entries : P;
    int blocks = (int)((n + 255) / 256);
    if (blocks > 65535) blocks = 65535;
    if (blocks < 1) blocks = 1;
    tables_to_fp64_kernel<<<blocks, 256, 0, s>>>(src, dst, P, entries);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
__global__ void fill_lut_kernel(const GridDev G, const VarioDev v, const CovLut t, double* c64, int2* cn,
                                int64_t total) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int L0 = (int)(i % t.w[0]) - t.e[0];
        const int64_t r = i / t.w[0];
        const int L1 = (int)(r % t.w[1]) - t.e[1];
        const int L2 = (int)(r / t.w[1]) - t.e[2];
        const double c = cov_fp64(v, G.dim, dmul((double)L0, G.spacing[0]), dmul((double)L1, G.spacing[1]),
                                  G.dim == 3 ? dmul((double)L2, G.spacing[2]) : 0.0);
        if (c64) c64[i] = c;
        if (cn) {  // normalized by the sill, in the FP32 path's (hi, lo) form
            const KF x = kf_from_double(c / v.sill);
            cn[i] = make_int2(x.hi, __float_as_int(x.lo));
        }
    }
}

cudaError_t launch_fill_cov_lut(const GridDev& g, const VarioDev& v, CovLut lut, double* c64, int2* cn,
                                cudaStream_t s) {
    const int64_t total = (int64_t)lut.w[0] * lut.w[1] * lut.w[2];
    int blocks = (int)((total + 255) / 256);
    if (blocks > 65535) blocks = 65535;
    fill_lut_kernel<<<blocks, 256, 0, s>>>(g, v, lut, c64, cn, total);
    return cudaGetLastError();
}

}  // namespace sgs

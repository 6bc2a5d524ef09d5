// internal.h — structures and launch wrappers shared by the host side of
// libgeosgs (api.cu) and the kernel files (search.cu, solve.cu, sweep.cu).
// Not part of the public ABI (include/geosgs.h is).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>
#include <cuda_runtime.h>

#include "../../include/geosgs.h"

namespace sgs {

constexpr int KMAX = 64;           // largest maxneighbors on the GPU
constexpr int METRIC_ISO = 0;
constexpr int METRIC_ELLIPSOID = 1;
constexpr int METRIC_NEAREST = 2;
constexpr int SGS_NODE_KRIGED_ = 0;          // mirrors SGS_NODE_* of geosgs.h
constexpr int SGS_NODE_PRIOR_NMIN_ = 1;
constexpr int SGS_NODE_PRIOR_SINGULAR_ = 2;

struct GridDev {
    int dim;
    int n[3];
    double origin[3];
    double spacing[3];
    int64_t N;
    uint32_t magic[2];  // node / n[j] = umulhi(node, magic[j]) >> shift[j] (n[j] > 1)
    int shift[2];
};

struct MetricDev {
    int kind;
    double rr;          // r*r (iso)
    double radii[3];
    double inv[3];      // 1 / radii, rounded once
    double R[9];        // column-major, leading dimension 3
    double ext[3];      // bounding-box half extents (physical units)
    float Rf[9];        // FP32 copies for the conservative prefilter
    float invf[3];
    float bound_f;      // FP32 prefilter bound: (1 + 1e-3) * (r*r or 1) + slack_f
                        // (+infinity for the unbounded nearest-neighbour metric)
    float slack_f;      // FP32 rounding allowance of the screen near the boundary
    float dh_f;         // bound on the FP32 rounding of an origin-relative coordinate
};

// One structure of a (nested) variogram model.
struct VarioStructDev {
    int type;
    double sill, nugget;
    double inv_range[3];
    double R[9];
    // lag -> normalized lag, diag(1 / ranges) R': component j of lag h is
    // sum_i W[3 i + j] h_i, and of a lag of d cells sum_i E[3 i + j] d_i
    double W[9], E[9];
    double psill62;  // (sill - nugget) 2^-62
};

// The process's variogram: ns structures summed (GeoStatsFunctions'
// NestedVariogram; ns = 1 for a single variogram).  type, inv_range and R
// repeat the first structure (the learned warm start's frame); sill and
// nugget are the model's, the structures' summed.  Sills whose systems would
// meet FP64's smallest or largest numbers are kept divided by unit^2, a power
// of four: weights do not depend on it, and deviations are `unit` times theirs.
struct VarioDev {
    int type;
    double sill, nugget;
    double unit;
    double inv_range[3];
    double R[9];
    int ns;
    VarioStructDev st[SGS_MAX_STRUCTURES];
};

// Covariance lookup table over integer grid lags L in [-e, e] per axis:
// entry (L0+e0) + w0*((L1+e1) + w1*(L2+e2)), w = 2e+1.
struct CovLut {
    const double* c64;  // nullptr when absent
    const int2* cn;     // the covariances / sill as integer multiples of 2^-28 (x) and
                        // the FP32 bits of the remainder (y)
    int e[3];
    int w[3];
};

// Offset template entry: cell offset and linear offset of a grid candidate.
struct TmplEntry {
    int dx, dy, dz, dlin;
};

struct SearchArgs {
    GridDev grid;
    MetricDev metric;
    int k;
    int T;                       // template entries
    const TmplEntry* tmpl;
    const double* tmpl_d2;
    const int32_t* path;
    const int32_t* rank;
    int64_t D;
    const double* dxyz;          // data coords, bucket order, D x 3
    const float4* dxyz_f;        // the same relative to the grid origin, FP32 (screen)
    const int32_t* did;          // data id of each bucket-ordered entry
    const int32_t* bstart;       // bucket start offsets (nb+1)
    int nb[3];
    int ring0;                   // buckets on each side of a node's own to start with
                                 // when its k nearest data are looked for (search_ring0)
    double bw[3];                // bucket widths (physical)
    float inv_bw_f[3];           // FP32 1 / bucket width, for the bucket range
    float ext_f[3];              // FP32 bounding-box half extents
    float spacing_f[3];
    int32_t* nbr;                // N x k, node-indexed
    int32_t* cnt;                // N
    int32_t* ngrid;              // N: grid neighbours among them
    int data_only;               // 1: data candidates only (kriging from the data)
    // optional [2] (single-problem search only): candidates examined (grid:
    // earlier path nodes tested by the early ranks and template entries
    // inside the grid, each one path rank read; data: bucket entries
    // screened), summed once per warp
    unsigned long long* scanned;
    unsigned long long* ticket;  // hands out the nodes (single-problem search)
};

// The ring whose box of buckets holds 1.5 k of D evenly spread data.
inline int search_ring0(int k, int64_t D, int dim, const int* nb) {
    const double side = std::pow(1.5 * k * nb[0] * nb[1] * nb[2] / (double)std::max<int64_t>(D, 1), 1.0 / dim);
    return (int)std::min(std::max(0.0, std::floor(0.5 * (side - 1.0))), 1e6);
}

// Longest wait of the dependency-level kernels for one neighbour's level.
// Their waits end by construction (a neighbour's path rank is smaller, and
// ranks are taken in increasing order by running warps), and the longest
// level computation measured (354 M nodes in one batch) takes 0.6 s in total,
// so a wait of 2 s only happens on a table that breaks the path order.
constexpr uint64_t LEVEL_WAIT_NS = 2000000000ull;

// Blocks of 8 warps per SM of the dependency-level kernels.  Warps beyond what
// throughput needs only wait, and their polls slow the chain of the early
// ranks: 250 k nodes take 0.39 ms with one block per SM and 0.53 with two,
// 4 M 1.75 and 1.58 ms, 16.8 M 5.3 and 4.0 ms (four and eight are no faster).
inline int level_blocks_per_sm(int64_t nodes) { return nodes >= ((int64_t)1 << 21) ? 2 : 1; }

struct LevelArgs {
    int64_t N;
    int k;
    const int32_t* path;
    const int32_t* nbr;
    const int32_t* cnt;
    int path_linear;             // 1: the path visits the nodes in id order
    int32_t* level;              // N, -1 = not yet known
    int32_t* ticket;             // 1 counter
    int32_t* maxlevel;           // 1 counter
    int32_t* err;                // 1 flag
    uint64_t wait_ns;            // longest wait for one neighbour's level
};

// Sweep tables, indexed by position in level order.  For T = double one
// value per entry; for T = float every weight, b0 and sigma is stored as an
// unevaluated FP32 pair (hi, lo) with hi + lo equal to the FP64 value to
// about 2^-48 relative, consumed by the compensated (Dot2) FP32 sweep.
template <typename T>
struct SweepTables {
    static constexpr int S = sizeof(T) == 4 ? 2 : 1;  // entries per value
    int32_t* node;               // P -> node id
    int32_t* m;                  // grid neighbours used
    int32_t* idx;                // P x k grid neighbour node ids
    T* w;                        // P x k x S weights of those
    T* b0;                       // P x S: data term sum_i w_i (d_i - mu)
    T* sigma;                    // P x S: conditional std (sqrt(sill) for the prior)
    const int64_t* off;          // nullptr: row p starts at p * k; else CSR row starts
                                 // (P + 1), used by batches of domains
};

// Item counters of a dataflow launch: one per warp of a block (class), each in
// its own 256 bytes; class c takes the items c, c + 8, c + 16, ... (in chunks).
// One counter for all hands out an item every 2.3 ns, which bounded wide
// launches (5.45 million rows of 8 values: 12.3 ms).
constexpr int FLOW_CLASSES = 8;
constexpr int FLOW_TICKET_STRIDE = 32;  // words
constexpr int FLOW_TICKETS = FLOW_CLASSES * FLOW_TICKET_STRIDE;
constexpr int FLOW_WORDS = FLOW_TICKET_STRIDE + 2 * FLOW_TICKETS;  // error flag, the counters of two launches

// More warps than a level has items only poll: the kernels compiled for
// higher residency run from levels of 16 items per SM (the other form's
// warps) on.  A mean of 4,096 items in a level: 3.24 ms with it, 3.97
// without; of 905: 1.10 and 0.81.
inline int flow_tight(int64_t items, int levels, int nsm) { return items >= (int64_t)levels * 16 * nsm; }

// Dataflow sweep state: warps take items (position in level order x piece of
// the row) from `ticket` and wait, per value, until a neighbour's row holds
// something else than the pattern it was cleared to (launch_flow_clear).
struct FlowArgs {
    int64_t item0;               // first item of this launch (earlier ones are done)
    int64_t item1;               // one past the last item of this launch
    int H;                       // pieces per row
    uint64_t rec;                // its reciprocal (set by the launch)
    unsigned long long* ticket;  // FLOW_TICKETS words, zero at launch
    int32_t* err;                // 1 flag, zero at launch
    int chunk;                   // consecutive items taken per ticket
    int blocks_per_sm;           // resident blocks per SM to launch (<= occupancy)
    int tight;                   // 1: kernel compiled for higher residency (register cap)
    uint64_t wait_ns;            // longest wait for one value before giving up
    const uint64_t* seed_dev;    // nullptr, or the draw seed in device memory (read at
                                 // launch; lets a captured graph take a new seed)
    int pairs;                   // FP64 values, packed tables: every 8-byte weight, b0
                                 // and sigma entry is an FP32 (hi, lo) pair
    int64_t row_stride;          // values between consecutive nodes' rows (0: Rp)
    const uint8_t* node_class;   // nullptr, or a class (0/1) per node: this launch
    int cls;                     // sweeps only the nodes of class cls, and another
                                 // launch the rest (their dependencies never cross)
};

struct SolveArgs {
    GridDev grid;
    VarioDev vario;
    CovLut lut;
    int k;
    int nmin;
    double mu;
    double tau;                  // singular pivot threshold (absolute)
    unsigned long long ratio63;  // (sill - nugget) / sill of the first structure, 2^-63
    double inv_sill;             // 1 / sill (the FP32 path works on the correlation matrix)
    float sd_sill[2];            // sqrt(sill) as an FP32 (hi, lo) pair
    int s_near;                  // high word of the squared normalized lag up to which a lag
                                 // computed from rounded parts may stand for zero
    int refine_steps;
    int64_t P;                   // positions to solve
    const int32_t* order;        // P -> node
    const int32_t* nbr;
    const int32_t* cnt;
    int64_t N;
    const double* data_xyz;      // D x 3, data id order
    const double* data_val;
    int8_t* status;              // node-indexed
    double* w_full;              // optional N x k export of all weights (node-indexed)
    double* sigma_full;          // optional N
    int32_t* fallback;           // FP32 path: list of positions that need FP64
    int32_t* nfallback;
    const int32_t* list;         // FP64 re-solve: positions to solve (nullptr = all)
    unsigned long long* sum_m;   // accumulates the grid neighbours written to the tables
    const float* w_init;         // optional node-indexed [N][k] warm-start weights (FP32 path)
    unsigned long long* n_warm;  // counts systems accepted from the warm start
    int64_t node0;               // added to node ids written to the sweep tables (the
                                 // domain's first global id in a batch; 0 for a plan)
    // indicator simulation (nullptr otherwise): per position, the sum of all
    // weights and, per category, the sum of the weights of data of that
    // category (zero for prior nodes)
    const int32_t* ind_cat;      // D data categories, 0 .. ncat-1
    int ncat;
    double* ind_wsum;            // [P]
    double* ind_dsum;            // [P][ncat]
    unsigned int* wl1_max;       // optional: FP32 bit pattern of the largest sum of
                                 // |weights| of grid neighbours over the systems
};

// Sequential indicator simulation (indicator.cu).
constexpr int IND_MAX_CAT = 8;
struct IndArgs {
    int ncat;
    double prob[IND_MAX_CAT];    // prior probabilities (normalized)
    const double* wsum;          // [P] sum of a system's weights (0 for the prior)
    const double* dsum;          // [P][ncat] weights of data of each category
};
// dataflow launches over all positions; f: error flag, tickets and wait_ns
cudaError_t launch_sis_flow_fp32(const SweepTables<float>& t, int k, int64_t N, int Rp, const IndArgs& ia,
                                 const double* u, uint64_t seed, uint8_t* C, const FlowArgs& f, cudaStream_t s);
cudaError_t launch_sis_flow_fp64(const SweepTables<double>& t, int k, int64_t N, int Rp, const IndArgs& ia,
                                 const double* u, uint64_t seed, uint8_t* C, const FlowArgs& f, cudaStream_t s);
cudaError_t launch_cats_to_out(const uint8_t* C, int64_t N, int R, int Rp, int32_t* out, cudaStream_t s);

// Full simple cokriging of the indicators (indicator.cu) for a linear model
// of coregionalization C_ab(h) = sum_s coef[s][a][b] C_s(h) over the
// structures of the plan's variogram.  Unknowns per system: n x L <= COK_MAX.
// The same systems serve multivariate Gaussian simulation (a GaussianProcess
// whose function is such a model): there L is the number of variables,
// `prob` holds their means, the data's L values replace their categories and
// the solve also factors each node's conditional covariance.
constexpr int COK_MAX = 64;
struct CokArgs {
    int ncat;                    // L
    double prob[IND_MAX_CAT];    // prior probabilities (normalized); Gaussian: the means
    const double* coef;          // [S][L][L]
    const int32_t* data_cat;     // [D] data categories (indicator)
    const double* data_val;      // [D][L] data values (Gaussian)
    double tau;                  // singular pivot threshold (absolute)
    double unit;                 // factor of the deviations (VarioDev::unit, and the same of coef)
    int32_t* m;                  // [P] grid neighbours of the position's system
    int32_t* idx;                // [P][k] their node ids
    double* w;                   // [P][k][L][L] weight of (grid neighbour j, its category b) for category t
    double* cst;                 // [P][L] prior term and the data's contribution
    const double* lut;           // nullptr, or C_s by lag, [S][lags of SolveArgs::lut]
    double* fac;                 // [P][L][L] Gaussian: lower Cholesky factor of the conditional
                                 // covariance (of the prior's for prior nodes), row-major
};
// systems of every position (a: geometry, neighbours, order, status; the
// status of each node is overwritten with its cokriging status)
// C_s of every structure s over the lags of `lut` (out: [S][lags])
cudaError_t launch_cok_lut(const GridDev& g, const VarioDev& v, const CovLut& lut, double* out, cudaStream_t s);
cudaError_t launch_cok_solve(const SolveArgs& a, const CokArgs& c, bool gaussian, cudaStream_t s);
cudaError_t launch_cok_flow(const CokArgs& c, const int32_t* node, int k, int64_t N, int Rp, const double* u,
                            uint64_t seed, uint8_t* C, const FlowArgs& f, cudaStream_t s);
// The multivariate Gaussian sweep.  V: values [L][N][Rp] (variable-major rows
// of Rp realizations); z: the normals in the same layout, or null for the
// seeded normals of pseudo-node a*N + g.
cudaError_t launch_mv_flow(const CokArgs& c, const int32_t* node, int k, int64_t N, int Rp, const double* z,
                           uint64_t seed, double* V, const FlowArgs& f, cudaStream_t s);

// The power of two u for which variances of size v are kept as v / u^2: 1
// within 2^-900 .. 2^900, where pivots down to 1e-10 v, their reciprocals and
// products keep all their bits.
inline double variance_unit(double v) {
    int e = 0;
    std::frexp(v, &e);
    return e > 900 || e < -900 ? std::ldexp(1.0, e / 2) : 1.0;
}

// Host-side description of one problem (api.cu: host_domain): everything
// sgs_plan_create derives on the host before uploading.
struct HostDomain {
    GridDev grid{};
    MetricDev metric{};
    VarioDev vario{};
    double mean = 0.0;
    int k = 0, nmin = 1;
    int64_t N = 0, D = 0;
    std::vector<TmplEntry> tmpl;          // offsets sorted by (d2, linear offset)
    std::vector<double> tmpl_d2;
    int tmpl_ext[3] = {0, 0, 0};          // largest |offset| per axis
    std::vector<double> xyz, val;         // data, id order (xyz: D x 3)
    std::vector<double> xyz_b;            // data, bucket order
    std::vector<int32_t> did, bstart;     // data id per bucket entry; bucket starts
    std::vector<float4> xf;               // FP32 origin-relative coordinates, bucket order
    int nb[3] = {1, 1, 1};
    double bw[3] = {1, 1, 1};
    int s_near = 0;                       // SolveArgs::s_near
};
// Validates *pr and fills H; SGS_OK or SGS_ERR_ARG with err set.  The path
// is left to the caller: plans and batches build and check its ranks on the
// device (launch_path_ranks, launch_batch_path_ranks).
// grid_neighbors: false for kriging from the data alone, whose search has no
// template (none is built; neighbourhoods too large for one stay refused)
int host_domain(const sgs_problem* pr, HostDomain& H, std::string& err, bool grid_neighbors = true);
// rank[path[t]] = t for a path of N nodes on the device (path NULL: the
// linear path, written into path_out), checking that the path is a
// permutation of [0, N): *err (zeroed by the caller) is set otherwise.
// path_out may equal path.
cudaError_t launch_path_ranks(const int32_t* path, int64_t N, int32_t* path_out, int32_t* rank, int32_t* err,
                              int nsm, cudaStream_t s);
// The same over a batch's path arena (local ids per domain, domains by the
// offsets off[0..nd]); *bad_domain (preset to nd) takes the smallest domain
// whose path is not a permutation.
cudaError_t launch_batch_path_ranks(const int32_t* path, const int64_t* off, int nd, int64_t total, int32_t* rank,
                                    int32_t* bad_domain, int nsm, cudaStream_t s);
// The geometry fields of a domain's SearchArgs (device pointers left as they are).
void search_args_of(const HostDomain& H, SearchArgs& sa);

// Device address of a page-locked host buffer (cudaHostAlloc'd or
// registered), or nullptr for any other pointer (pageable memory is never
// handed to a kernel).
inline double* pinned_device_view(double* host) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (a.type != cudaMemoryTypeHost || a.devicePointer == nullptr) return nullptr;
    return static_cast<double*>(a.devicePointer);
}

// Message returned by sgs_last_error(NULL) on this host thread.
// Device memory of plans and batches comes from one stream-ordered pool per
// device that keeps freed memory for the next plan instead of returning it
// (sgs_trim_memory returns it).  pool_alloc: usable on every stream when it
// returns; pool_free: ordered after the work already queued on `stream`.
cudaError_t pool_alloc(void** ptr, size_t bytes, int device);
cudaError_t pool_free(void* ptr, cudaStream_t stream);

void set_thread_error(const char* msg);
inline void set_thread_error(const std::string& msg) { set_thread_error(msg.c_str()); }

// ---- launch wrappers (return cudaError_t of the launch) ----
cudaError_t launch_search(const SearchArgs& a, cudaStream_t s);
cudaError_t launch_levels(const LevelArgs& a, int nsm, cudaStream_t s);
cudaError_t launch_level_order(int64_t N, const int32_t* level, int nlevels, int32_t* lcount,
                               int32_t* loff, int32_t* lfill, int32_t* order, cudaStream_t s);
cudaError_t launch_solve_fp64(const SolveArgs& a, const SweepTables<double>& t, cudaStream_t s);
cudaError_t launch_solve_fp32(const SolveArgs& a, const SweepTables<float>& t, cudaStream_t s);
cudaError_t launch_solve_fp64_into_fp32(const SolveArgs& a, const SweepTables<float>& t, cudaStream_t s);
// batches of domains (doms: device descriptors, noff: ndom + 1 global node
// offsets, order: level-ordered global node ids; the positions to solve are
// list[desc[1] .. desc[1] + desc[0]), desc on the device)
// *out += the number of nonzero entries of v[0, n) (device counter)
cudaError_t launch_count_nonzero(int64_t n, const int8_t* v, unsigned long long* out, int nsm, cudaStream_t s);
cudaError_t launch_search_batch(const SearchArgs* doms, const int64_t* noff, int ndom, int64_t total,
                                unsigned long long* ticket, int nsm, cudaStream_t s);
cudaError_t launch_solve_fp32_batch(int nmax, const SolveArgs* doms, const int64_t* noff, int ndom,
                                    const int32_t* order, const int32_t* list, const int32_t* desc,
                                    const SweepTables<float>& t, int nsm, cudaStream_t s);
cudaError_t launch_solve_fp64_batch(int kl, const SolveArgs* doms, const int64_t* noff, int ndom,
                                    const int32_t* order, const int32_t* list, const int32_t* desc,
                                    const SweepTables<double>& t, int nsm, cudaStream_t s);
cudaError_t launch_solve_fp64_into_fp32_batch(int kl, const SolveArgs* doms, const int64_t* noff, int ndom,
                                              const int32_t* order, const int32_t* list, const int32_t* desc,
                                              const SweepTables<float>& t, int nsm, cudaStream_t s);
// pairs = 2 or 4: one thread per 2 or 4 chunks of 4 realizations (rows of a
// multiple of 8 or 16 realizations, more than 64 of them); otherwise one
// thread per chunk.  split = 1 (rows of a multiple of 8 realizations): one
// block per node, the neighbour list split over its warps (small levels).
cudaError_t launch_sweep_fp32(const SweepTables<float>& t, int k, int64_t p0, int64_t p1, int Rp,
                              const float* z, uint64_t seed, float* V, cudaStream_t s, int pairs = 1,
                              int split = 0);
cudaError_t launch_sweep_fp64(const SweepTables<double>& t, int k, int64_t p0, int64_t p1, int Rp,
                              const double* z, uint64_t seed, double* V, cudaStream_t s);
// all levels in one cooperative launch (loff: device level offsets, nlevels + 1)
cudaError_t launch_sweep_all_fp32(const SweepTables<float>& t, int k, const int32_t* loff, int nlevels, int Rp,
                                  const float* z, uint64_t seed, float* V, cudaStream_t s);
cudaError_t launch_sweep_all_fp64(const SweepTables<double>& t, int k, const int32_t* loff, int nlevels, int Rp,
                                  const double* z, uint64_t seed, double* V, cudaStream_t s);
// all levels in one persistent dataflow launch (no level barriers); W lanes
// per slice of the neighbour list and G chunks of 4 realizations per lane,
// as returned by flow_layout, which also gives the pieces per row
int flow_layout(int Rp, int& W, int& G);
cudaError_t launch_flow_wait_selftest(const float* row, const FlowArgs& f, cudaStream_t s);
cudaError_t launch_sweep_flow_fp32(const SweepTables<float>& t, int k, int Rp, int W, int G, const float* z,
                                   uint64_t seed, float* V, const FlowArgs& f, int nsm, cudaStream_t s);
cudaError_t launch_sweep_flow_fp64(const SweepTables<double>& t, int k, int Rp, int W, int G, const double* z,
                                   uint64_t seed, double* V, const FlowArgs& f, int nsm, cudaStream_t s);
// mean + b0 and sigma^2 of the kriged nodes, NaN elsewhere, by node
template <typename T>
cudaError_t launch_krige_moments(const SweepTables<T>& t, const int8_t* status, double mean, int64_t N, double* m,
                                 double* v, cudaStream_t s);
// the rows of positions [p0, p1) (all N: every row) cleared for a dataflow launch
cudaError_t launch_flow_clear(const int32_t* node, int64_t p0, int64_t p1, int64_t N, size_t row_bytes, void* V,
                              cudaStream_t s);
// host z (R x N, realization-major double) on device -> node-major [N][Rp] of T
cudaError_t launch_z_to_rows_fp32(const double* zin, int64_t N, int R, int Rp, float* z, cudaStream_t s);
cudaError_t launch_z_to_rows_fp64(const double* zin, int64_t N, int R, int Rp, double* z, cudaStream_t s);
// node-major centred values -> realization-major double with the mean added
cudaError_t launch_rows_to_out_fp32(const float* V, int64_t N, int R, int Rp, double mu, double* out, cudaStream_t s);
cudaError_t launch_rows_to_out_fp64(const double* V, int64_t N, int R, int Rp, double mu, double* out, cudaStream_t s);
// FP64 copies of packed (hi, lo) sweep tables: w of `entries` weights, b0 and
// sigma of P positions (node, m, idx and off are shared with the source)
cudaError_t launch_tables_to_fp64(const SweepTables<float>& src, SweepTables<double>& dst, int64_t P,
                                  int64_t entries, cudaStream_t s);
cudaError_t launch_fill_cov_lut(const GridDev& g, const VarioDev& v, CovLut lut, double* c64, int2* cn, cudaStream_t s);
// learned warm start (learned.cu)
cudaError_t launch_nn_features(const GridDev& G, const VarioDev& v, const int32_t* nbr, const int32_t* cnt, int k,
                               const double* data_xyz, float* feat, cudaStream_t s);
cudaError_t launch_nn_predict_plan(const GridDev& G, const VarioDev& v, const int32_t* nbr, const int32_t* cnt, int k,
                                   const double* data_xyz, const float* params, float* out, cudaStream_t s);
// BF16 tensor-core inference (learned_tc.cu); err: device flag set when an
// MMA completion wait gave up
cudaError_t launch_nn_predict_tc(const GridDev& G, const VarioDev& v, const int32_t* nbr, const int32_t* cnt, int k,
                                 const double* data_xyz, const float* params, float* out, int32_t* err, int nsm,
                                 cudaStream_t s);
cudaError_t launch_nn_forward(const float* params, const float* feat, const int32_t* count, int64_t nsys, int k,
                              float* pred, cudaStream_t s);
cudaError_t launch_nn_backward(const float* params, const float* feat, const int32_t* count, const float* target,
                               int64_t nsys, int k, float* grad, float* loss, cudaStream_t s);
cudaError_t launch_nn_adam(float* p, const float* g, float* m, float* v, int step, float lr, float scale,
                           cudaStream_t s);

}  // namespace sgs

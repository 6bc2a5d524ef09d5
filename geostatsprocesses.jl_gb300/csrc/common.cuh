// common.cuh — device helpers shared by the SGS kernels: the canonical FP64
// lag metric, the variogram covariance, Philox draws and warp utilities.
//
// Canonical formulas (identical operation order on host and device; the
// device uses the _rn intrinsics so nothing is contracted into an FMA):
//   grid lag      h_j = (double)(i_c - i_p) * spacing_j
//   data lag      h_j = X_j - (origin_j + ((double)i_j + 0.5) * spacing_j)
//   isotropic     d2 = h0*h0 + h1*h1 (+ h2*h2), inside iff d2 <= r*r
//   ellipsoid     u_j = R(0,j)h0 + R(1,j)h1 (+ R(2,j)h2), q_j = u_j * inv_j
//                 with inv_j = 1 / radius_j rounded once, d2 = sum_j q_j^2,
//                 inside iff d2 <= 1
#pragma once

#include <climits>
#include <cstdint>
#include <cuda_runtime.h>

#include "internal.h"

#define FULL_MASK 0xffffffffu

namespace sgs {

__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }

// canonical squared distance of a lag under a search metric
__device__ __forceinline__ double metric_d2(const MetricDev& m, int dim, double h0, double h1, double h2) {
    if (m.kind != METRIC_ELLIPSOID) {
        double s = dmul(h0, h0);
        s = dadd(s, dmul(h1, h1));
        if (dim == 3) s = dadd(s, dmul(h2, h2));
        return s;
    }
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        if (j < dim) {
            double u = dmul(m.R[0 + 3 * j], h0);
            u = dadd(u, dmul(m.R[1 + 3 * j], h1));
            if (dim == 3) u = dadd(u, dmul(m.R[2 + 3 * j], h2));
            double q = dmul(u, m.inv[j]);
            s = (j == 0) ? dmul(q, q) : dadd(s, dmul(q, q));
        }
    }
    return s;
}

// FP32 evaluation of the same metric, used only to discard candidates that
// are clearly outside `bound` (bound_f, or a tighter bound for a smaller
// distance; each carries a 1e-3 relative margin and a slack above the FP32
// rounding of these few operations), so the FP64 decision is unchanged.
__device__ __forceinline__ bool metric_maybe_within(const MetricDev& m, int dim, float h0, float h1, float h2,
                                                    float bound) {
    float s;
    if (m.kind != METRIC_ELLIPSOID) {
        s = h0 * h0 + h1 * h1 + (dim == 3 ? h2 * h2 : 0.0f);
    } else {
        s = 0.0f;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (j < dim) {
                float u = m.Rf[0 + 3 * j] * h0 + m.Rf[1 + 3 * j] * h1 + (dim == 3 ? m.Rf[2 + 3 * j] * h2 : 0.0f);
                float q = u * m.invf[j];
                s += q * q;
            }
        }
    }
    return s <= bound;
}

__device__ __forceinline__ bool metric_inside(const MetricDev& m, double d2) {
    if (m.kind == METRIC_ISO) return d2 <= m.rr;
    if (m.kind == METRIC_ELLIPSOID) return d2 <= 1.0;
    return true;
}

// grid centroid coordinate along axis j
__device__ __forceinline__ double centroid(const GridDev& g, int j, int i) {
    double t = dadd((double)i, 0.5);
    t = dmul(t, g.spacing[j]);
    return dadd(g.origin[j], t);
}

// node -> cell: divisions by the grid's sides as multiplications by host-made
// reciprocals (GridDev::magic), exact for every node id below 2^31
__device__ __forceinline__ int grid_div(const GridDev& g, int j, int x) {
    return g.n[j] == 1 ? x : (int)(__umulhi((uint32_t)x, g.magic[j]) >> g.shift[j]);
}

__device__ __forceinline__ void cell_of(const GridDev& g, int node, int& i0, int& i1, int& i2) {
    const int r = grid_div(g, 0, node);
    i0 = node - r * g.n[0];
    i2 = grid_div(g, 1, r);
    i1 = r - i2 * g.n[1];
}

// FP64 on this GPU issues one warp instruction in 64 cycles per scheduler, so
// the covariance below counts its FP64 instructions: about 40 for an
// exponential structure in 3D instead of about 150 with the library's exp and
// sqrt, whose many special cases its arguments never need.
//
// 2^(j/64), j = 0 .. 63, rounded to double.
static __device__ const double kExp2J64[64] = {
    0x1.0000000000000p+0, 0x1.02c9a3e778061p+0, 0x1.059b0d3158574p+0, 0x1.0874518759bc8p+0,
    0x1.0b5586cf9890fp+0, 0x1.0e3ec32d3d1a2p+0, 0x1.11301d0125b51p+0, 0x1.1429aaea92de0p+0,
    0x1.172b83c7d517bp+0, 0x1.1a35beb6fcb75p+0, 0x1.1d4873168b9aap+0, 0x1.2063b88628cd6p+0,
    0x1.2387a6e756238p+0, 0x1.26b4565e27cddp+0, 0x1.29e9df51fdee1p+0, 0x1.2d285a6e4030bp+0,
    0x1.306fe0a31b715p+0, 0x1.33c08b26416ffp+0, 0x1.371a7373aa9cbp+0, 0x1.3a7db34e59ff7p+0,
    0x1.3dea64c123422p+0, 0x1.4160a21f72e2ap+0, 0x1.44e086061892dp+0, 0x1.486a2b5c13cd0p+0,
    0x1.4bfdad5362a27p+0, 0x1.4f9b2769d2ca7p+0, 0x1.5342b569d4f82p+0, 0x1.56f4736b527dap+0,
    0x1.5ab07dd485429p+0, 0x1.5e76f15ad2148p+0, 0x1.6247eb03a5585p+0, 0x1.6623882552225p+0,
    0x1.6a09e667f3bcdp+0, 0x1.6dfb23c651a2fp+0, 0x1.71f75e8ec5f74p+0, 0x1.75feb564267c9p+0,
    0x1.7a11473eb0187p+0, 0x1.7e2f336cf4e62p+0, 0x1.82589994cce13p+0, 0x1.868d99b4492edp+0,
    0x1.8ace5422aa0dbp+0, 0x1.8f1ae99157736p+0, 0x1.93737b0cdc5e5p+0, 0x1.97d829fde4e50p+0,
    0x1.9c49182a3f090p+0, 0x1.a0c667b5de565p+0, 0x1.a5503b23e255dp+0, 0x1.a9e6b5579fdbfp+0,
    0x1.ae89f995ad3adp+0, 0x1.b33a2b84f15fbp+0, 0x1.b7f76f2fb5e47p+0, 0x1.bcc1e904bc1d2p+0,
    0x1.c199bdd85529cp+0, 0x1.c67f12e57d14bp+0, 0x1.cb720dcef9069p+0, 0x1.d072d4a07897cp+0,
    0x1.d5818dcfba487p+0, 0x1.da9e603db3285p+0, 0x1.dfc97337b9b5fp+0, 0x1.e502ee78b3ff6p+0,
    0x1.ea4afa2a490dap+0, 0x1.efa1bee615a27p+0, 0x1.f50765b6e4540p+0, 0x1.fa7c1819e90d8p+0,
};

// exp(x) for x <= 0, table-driven (Tang 1989): x = (64 m + j) ln2 / 64 + r with
// |r| <= ln2 / 128, exp(x) = 2^m 2^(j/64) exp(r), exp(r) by its Taylor
// polynomial of degree 5 (truncation below 4e-17); 0 below -700.
__device__ __forceinline__ double exp_nonpos(double x) {
    if ((uint32_t)__double2hiint(x) > 0xC085E000u) return 0.0;  // x < -700
    const double shift = 6755399441055744.0;  // 1.5 x 2^52: the sum's low word is the rounded integer
    const double t = fma(x, 0x1.71547652b82fep+6, shift);
    const int n = __double2loint(t);
    const double nd = t - shift;
    double r = fma(nd, -0x1.62e42fef00000p-7, x);  // ln2 / 64 in two parts, the first exact times nd
    r = fma(nd, -0x1.473de6af278edp-40, r);
    double p = fma(r, 1.0 / 120.0, 1.0 / 24.0);
    p = fma(p, r, 1.0 / 6.0);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    p = p * r;
    const double T = __ldg(&kExp2J64[n & 63]);
    const double e = fma(T, p, T);
    return __hiloint2double(__double2hiint(e) + ((n >> 6) << 20), __double2loint(e));
}

// sqrt(s): FP32 reciprocal root and two Goldschmidt steps in FP64 (within an
// ulp); values far outside FP32's range go to the library
__device__ __forceinline__ double sqrt_fp64(double s) {
    const uint32_t hi = (uint32_t)__double2hiint(s);
    if (hi - 0x39B00000u > 0x46300000u - 0x39B00000u) return sqrt(s);  // outside 2^-100 .. 2^100
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"((float)s));
    const double yd = (double)y;
    double g = s * yd, h = 0.5 * yd;
    double e = fma(-g, h, 0.5);
    g = fma(g, e, g);
    h = fma(h, e, h);
    e = fma(-g, g, s);
    return fma(e, h, g);
}

// normalized variogram (0 at the origin, 1 at the sill) of a squared
// normalized lag s
__device__ __forceinline__ double structure_shape(int type, double s) {
    if (type == 3) return 1.0 - exp_nonpos(-3.0 * s);
    const double hn = sqrt_fp64(s);
    if (type == 1) return hn < 1.0 ? 1.5 * hn - 0.5 * hn * hn * hn : 1.0;
    return 1.0 - exp_nonpos(-3.0 * hn);
}

// gamma(h) of one structure at a nonzero lag (GeoStatsFunctions conventions:
// practical ranges, nugget for nonzero lags only)
__device__ __forceinline__ double structure_gamma(const VarioStructDev& v, int dim, double h0, double h1, double h2) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        if (j < dim) {
            double u = v.R[0 + 3 * j] * h0 + v.R[1 + 3 * j] * h1;
            if (dim == 3) u += v.R[2 + 3 * j] * h2;
            double q = u * v.inv_range[j];
            s += q * q;
        }
    }
    return v.nugget + (v.sill - v.nugget) * structure_shape(v.type, s);
}

__device__ __forceinline__ bool is_zero(double h) { return (__double_as_longlong(h) << 1) == 0; }

// covariance C(h) = sill - gamma(h) in FP64, gamma summed over the model's
// structures
__device__ __forceinline__ double cov_fp64(const VarioDev& v, int dim, double h0, double h1, double h2) {
    if (is_zero(h0) && is_zero(h1) && (dim == 2 || is_zero(h2))) return v.sill;
    double g = 0.0;
#pragma unroll 1
    for (int i = 0; i < v.ns; ++i) g += structure_gamma(v.st[i], dim, h0, h1, h2);
    return v.sill - g;
}

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw 2011) on counter (c0..c3), key (k0,k1)
__device__ __forceinline__ uint4 philox10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        uint4 n;
        n.x = hi1 ^ c.y ^ k0;
        n.y = lo1;
        n.z = hi0 ^ c.w ^ k1;
        n.w = lo0;
        c = n;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c;
}

// four standard normals of node g, realizations 4q..4q+3 (Box-Muller on
// 24-bit uniforms (2m+1)/2^24, exactly representable in float)
__device__ __forceinline__ float4 normals4(uint64_t seed, int64_t g, int q) {
    uint4 c = philox10(make_uint4((uint32_t)g, (uint32_t)((uint64_t)g >> 32), (uint32_t)q, 0u),
                       (uint32_t)seed, (uint32_t)(seed >> 32));
    const float sc = 1.0f / 16777216.0f;
    float u0 = (float)((c.x >> 9) * 2u + 1u) * sc;
    float u1 = (float)((c.y >> 9) * 2u + 1u) * sc;
    float u2 = (float)((c.z >> 9) * 2u + 1u) * sc;
    float u3 = (float)((c.w >> 9) * 2u + 1u) * sc;
    float r0 = sqrtf(-2.0f * logf(u0)), r1 = sqrtf(-2.0f * logf(u2));
    float s0, c0, s1, c1;
    sincospif(2.0f * u1, &s0, &c0);
    sincospif(2.0f * u3, &s1, &c1);
    return make_float4(r0 * c0, r0 * s0, r1 * c1, r1 * s1);
}

// two FP32 values in one 64-bit register pair; fma.rn.f32x2 is one
// instruction for both
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2_pack(float lo, float hi) {
    F2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float f2_lo(F2 v) {
    float lo;
    asm("mov.b64 {%0, _}, %1;" : "=f"(lo) : "l"(v));
    return lo;
}
__device__ __forceinline__ float f2_hi(F2 v) {
    float hi;
    asm("mov.b64 {_, %0}, %1;" : "=f"(hi) : "l"(v));
    return hi;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// ---- double-FP32 ("float-float") arithmetic: a value is an unevaluated sum
// hi + lo of two floats, |lo| <= ulp(hi)/2, about 48 significant bits.  Error-
// free transformations after Knuth (TwoSum), Dekker (Fast2Sum) and the FMA
// form of TwoProduct; every operation is an explicit _rn intrinsic so the
// compiler cannot contract or reorder them.
struct DF {
    float hi, lo;
};

__device__ __forceinline__ DF df_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bp = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
    return {s, e};
}

__device__ __forceinline__ DF df_fast_two_sum(float a, float b) {  // |a| >= |b|
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}

__device__ __forceinline__ DF df_from_double(double v) {
    const float hi = (float)v;
    return {hi, (float)(v - (double)hi)};
}

__device__ __forceinline__ DF df_add(DF a, DF b) {
    const DF s = df_two_sum(a.hi, b.hi);
    return df_fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}

__device__ __forceinline__ DF df_neg(DF a) { return {-a.hi, -a.lo}; }

// Compensated dot-product accumulator (Dot2, Ogita-Rump-Oishi 2005) with
// double-FP32 operands: adds (xh + xl) * (yh + yl) dropping only xl*yl.
struct DFAcc {
    float s, c;
    __device__ __forceinline__ void init(DF v) {
        s = v.hi;
        c = v.lo;
    }
    __device__ __forceinline__ void add_prod(DF x, DF y) {
        const float p = __fmul_rn(x.hi, y.hi);
        const float pe = __fmaf_rn(x.hi, y.hi, -p);
        const DF t = df_two_sum(s, p);
        s = t.hi;
        const float cross = __fmaf_rn(x.hi, y.lo, __fmul_rn(x.lo, y.hi));
        c = __fadd_rn(c, __fadd_rn(t.lo, __fadd_rn(pe, cross)));
    }
    __device__ __forceinline__ DF value() const { return df_two_sum(s, c); }
};

// square root of a non-negative double-FP32 value: FP32 root plus one
// Newton correction evaluated with an exact square (TwoProduct)
__device__ __forceinline__ DF df_sqrt(DF v) {
    if (!(v.hi > 0.0f)) return {0.0f, 0.0f};
    const float r = sqrtf(v.hi);
    const float p = __fmul_rn(r, r);
    const float pe = __fmaf_rn(r, r, -p);
    const float d = __fadd_rn(__fsub_rn(__fsub_rn(v.hi, p), pe), v.lo);
    return df_fast_two_sum(r, __fdiv_rn(d, __fmul_rn(2.0f, r)));
}

__device__ __forceinline__ DF shfl_xor_df(DF v, int o) {
    return {__shfl_xor_sync(FULL_MASK, v.hi, o), __shfl_xor_sync(FULL_MASK, v.lo, o)};
}

__device__ __forceinline__ DF warp_sum_df(DF v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = df_add(v, shfl_xor_df(v, o));
    return v;
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Dependency levels of 32 consecutive tickets, one node per lane: the lane's
// node g (active: it has one) has neighbours row[0, n), of which those below
// N are grid nodes; lev[c] is node c's level, -1 while unknown.  On a linear
// path first is the rank, and so the id, of lane 0's node (else negative): a
// neighbour in [first, first + 32) is another lane's node, whose level is read
// from s_lev (this warp's 32 words) instead of global memory.
//
// Every lane reads all its neighbours' levels once, remembers the unknown
// ones in a mask, and then polls eight of them per turn (the farthest first:
// along a path the last neighbour to be done is usually the nearest) until
// none is left.  Lanes finish in any order.  Waits end because tickets are
// taken in path order by running warps; they are bounded all the same by
// wait_ns of wall-clock time without progress of the warp (and, should the
// timer stall, by a count of polls reached no earlier), and stop soon after
// another warp has raised *err.  A warp that gives up raises *err and returns
// with its remaining levels unwritten.  Returns the lane's level (0 if none).
__device__ __forceinline__ int warp_levels(bool active, int g, const int32_t* __restrict__ row, int n, int64_t N,
                                           volatile int32_t* lev, int64_t first, volatile int32_t* s_lev, int32_t* err,
                                           uint64_t wait_ns, int lane) {
    int lv = 0;
    unsigned long long mask = 0, near = 0;  // unknown levels: elsewhere, in this warp
    s_lev[lane] = -1;
    if (!active) n = 0;
    int nmax = n;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nmax = max(nmax, __shfl_xor_sync(FULL_MASK, nmax, o));
    for (int q = 0; q < nmax; q += 8) {  // eight levels in flight per lane
        int c[8], l[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) c[h] = q + h < n ? row[q + h] : INT_MAX;
#pragma unroll
        for (int h = 0; h < 8; ++h) l[h] = c[h] < N ? lev[c[h]] : -2;
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            if (l[h] != -1) lv = max(lv, l[h] + 1);
            else if (first >= 0 && (uint64_t)(c[h] - first) < 32) near |= 1ull << (q + h);
            else mask |= 1ull << (q + h);
        }
    }
    bool pending = active;
    const volatile int32_t* verr = err;
    const uint64_t max_polls = wait_ns / 32 + 1024;
    uint64_t t0 = 0, idle = 0;
    __syncwarp();
    for (;;) {
        // hand levels over within the warp for as long as that moves a lane
        for (bool any = true; any;) {
            bool moved = false;
            if (pending && near) {
                const int q = 63 - __clzll((long long)near);
                const int l = s_lev[row[q] - first];
                if (l >= 0) {
                    lv = max(lv, l + 1);
                    near &= ~(1ull << q);
                    moved = true;
                }
            }
            if (pending && !(near | mask)) {
                lev[g] = lv;
                s_lev[lane] = lv;
                pending = false;
                moved = true;
            }
            __syncwarp();
            any = __any_sync(FULL_MASK, moved);
        }
        if (!__any_sync(FULL_MASK, pending)) return lv;
        // one turn over global memory
        bool moved = false;
        if (pending && mask) {
            unsigned long long left = mask;
            int c[8], q[8], l[8];
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                q[h] = left ? 63 - __clzll((long long)left) : -1;
                left = left ? left & ~(1ull << q[h]) : 0;
                c[h] = q[h] >= 0 ? row[q[h]] : 0;
            }
#pragma unroll
            for (int h = 0; h < 8; ++h) l[h] = q[h] >= 0 ? lev[c[h]] : -1;
#pragma unroll
            for (int h = 0; h < 8; ++h)
                if (l[h] >= 0) {
                    lv = max(lv, l[h] + 1);
                    mask &= ~(1ull << q[h]);
                    moved = true;
                }
        }
        if (__any_sync(FULL_MASK, moved)) {
            idle = 0;
            t0 = 0;
            continue;
        }
        __nanosleep(64);
        if ((++idle & 31) == 0) {
            bool stop = *verr != 0;
            if (!stop) {
                const uint64_t now = global_ns();
                if (t0 == 0) t0 = now;
                stop = now - t0 > wait_ns || idle > max_polls;
                if (stop) atomicExch(err, 1);
            }
            if (__any_sync(FULL_MASK, stop)) return 0;
        }
    }
}

// 1 / d of a pivot (positive, normal): an FP32 reciprocal r of its mantissa,
// off by e = 1 - d r of some 2^-22, and one step of third order, r (1 + e +
// e^2).  The exponents are handled as integers, off the FP64 pipe.
__device__ __forceinline__ double reciprocal(double d) {
    const unsigned hi = __double2hiint(d), lo = __double2loint(d);
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(__uint_as_float(0x3f800000u | (hi & 0xfffffu) << 3 | lo >> 29)));
    const unsigned u = __float_as_uint(rf);
    const double r = __hiloint2double((int)((u >> 3) + (896u << 20) + (1023u << 20) - (hi & 0x7ff00000u)), (int)(u << 29));
    const double e = fma(-d, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// Rows of a symmetric FP64 system in shared memory: ld of them apart, 8 more
// than a multiple of 16 doubles, so that 2 x 8 entries use all banks.
__host__ __device__ constexpr int ldl_stride(int rows) { return (rows + 7) / 16 * 16 + 8; }

// L D L' of the leading m rows of K (lower triangle) by one warp, carried on
// through rows m .. M - 1: right-hand sides c, which end up as D^-1 L^-1 c,
// with the lower triangle of any symmetric block C beyond column m, which
// becomes the Schur complement C - c' K^-1 c.  False at the first pivot not
// above tau.  Steps take 4 rows x 8 columns at a time, one FP64 instruction
// each: about (M - j)^2 / 64 for step j instead of M - j with a row per lane,
// and a reciprocal instead of a square root and three divisions a column.
// av, fv: M entries of scratch.
__device__ __forceinline__ bool warp_ldl(double* K, int ld, int m, int M, double tau, double* av, double* fv, int lane) {
    const int r = lane >> 3, c = lane & 7;
    for (int j = 0; j < m; ++j) {
        const double d = K[j * ld + j];
        if (!(d > tau)) return false;
        const double inv = reciprocal(d);
        for (int i = j + 1 + lane; i < M; i += 32) {
            const double a = K[i * ld + j], f = a * inv;
            av[i] = a;
            fv[i] = -f;
            K[i * ld + j] = f;
        }
        __syncwarp();
        for (int i0 = j + 1; i0 < M; i0 += 4) {
            const int i = i0 + r, top = min(i, M - 1);
            const double f = fv[top];
            double* row = K + top * ld;
#pragma unroll 4
            for (int l = j + 1 + c; l - c <= min(i0 + 3, M - 1); l += 8)
                if (i < M && l <= i) row[l] = fma(f, av[l], row[l]);
        }
        __syncwarp();
    }
    return true;
}

// Row `rhs` of a system warp_ldl has been through, D^-1 L^-1 c, becomes the
// solution K^-1 c (m <= 64).
__device__ __forceinline__ void warp_ldl_solve(double* K, int ld, int m, int rhs, int lane) {
    double* z = K + rhs * ld;
    double z0 = lane < m ? z[lane] : 0.0, z1 = lane + 32 < m ? z[lane + 32] : 0.0;
    for (int j = m - 1; j > 0; --j) {
        const double zj = __shfl_sync(FULL_MASK, j < 32 ? z0 : z1, j & 31);
        const double* row = K + j * ld;
        if (lane < j) z0 = fma(-row[lane], zj, z0);
        if (j > 32 && lane + 32 < j) z1 = fma(-row[lane + 32], zj, z1);
    }
    if (lane < m) z[lane] = z0;
    if (lane + 32 < m) z[lane + 32] = z1;
    __syncwarp();
}

// ---- batches of domains: global numbering and per-domain descriptors ----
// Domain d owns the global ids [off[d], off[d+1]); returns d for id x
// (0 <= x < off[nd]) by binary search over the nd + 1 offsets.
__device__ __forceinline__ int find_domain(const int64_t* __restrict__ off, int nd, int64_t x) {
    int lo = 0, hi = nd - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= x) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Copy a descriptor (a plain struct, 4-byte multiple) from global into this
// warp's shared-memory slot, all lanes cooperating; the caller __syncwarp()s.
template <typename T>
__device__ __forceinline__ void warp_copy_struct(T* dst, const T* src, int lane) {
    static_assert(sizeof(T) % 4 == 0, "descriptor size");
    int* d = reinterpret_cast<int*>(dst);
    const int* s = reinterpret_cast<const int*>(src);
    for (int i = lane; i < (int)(sizeof(T) / 4); i += 32) d[i] = __ldg(s + i);
}

// First table entry of sweep-table row `pos`: rows of k entries, or CSR
// offsets when the tables are packed (batches of domains with different k).
template <typename T>
__device__ __forceinline__ int64_t table_row(const SweepTables<T>& t, int64_t pos, int k) {
    return t.off ? t.off[pos] : pos * (int64_t)k;
}

}  // namespace sgs

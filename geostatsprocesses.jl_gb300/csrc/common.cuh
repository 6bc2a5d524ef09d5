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
// the covariance below keeps to three of them past the squared lag: square
// roots are put together from FP32 corrections of exact FP64 remainders, and
// the exponential is evaluated in 64-bit integers (some 85 instructions of a
// cycle or two).  Errors below 2^-56 of the sill, which is also what small
// covariances are accurate to (sill - gamma, their other form, loses its bits to
// the same cancellation from 2^-52 of the sill on); the library's exp and sqrt
// took about 100 FP64 instructions, FP64 forms of these two 30.
//
// 2^(-j/64) in units of 2^-63, j = 0 .. 63.
static __device__ const unsigned long long kExp2J64[64] = {
    0x8000000000000000ull, 0x7e9f06067a4360baull, 0x7d41d96db915019dull, 0x7be86fb985689ddcull,
    0x7a92be8a92436616ull, 0x7940bb9e2cffd89dull, 0x77f25ccdee6d7ae6ull, 0x76a7980f6cca15c2ull,
    0x75606373ee921c97ull, 0x741cb5281e25ee34ull, 0x72dc8373be41a454ull, 0x719fc4b95f452d29ull,
    0x70666f76154a7089ull, 0x6f307a412f074892ull, 0x6dfddbcbed791babull, 0x6cce8ae13c57ebdbull,
    0x6ba27e656b4eb57aull, 0x6a79ad55e7f6fd10ull, 0x69540ec8f895722dull, 0x683199ed779592caull,
    0x6712460a8fc24072ull, 0x65f60a7f79393e2eull, 0x64dcdec3371793d1ull, 0x63c6ba6455dcd8aeull,
    0x62b39508aa836d6full, 0x61a3666d124bb204ull, 0x6096266533384a2bull, 0x5f8bccdb3d398841ull,
    0x5e8451cfac061b5full, 0x5d7fad59099f22feull, 0x5c7dd7a3b17dcf75ull, 0x5b7ec8f19468bbc9ull,
    0x5a827999fcef3242ull, 0x5988e20954889245ull, 0x5891fac0e95612c8ull, 0x579dbc56b48521baull,
    0x56ac1f752150a563ull, 0x55bd1cdad49f699cull, 0x54d0ad5a753e077cull, 0x53e6c9da74b29ab5ull,
    0x52ff6b54d8a89c75ull, 0x521a8ad704f3404full, 0x513821818624b40cull, 0x50582887dcb8a7e1ull,
    0x4f7a993048d088d7ull, 0x4e9f6cd3967fdba8ull, 0x4dc69cdceaa72a9cull, 0x4cf022c9905bfd32ull,
    0x4c1bf828c6dc54b8ull, 0x4b4a169b900c2d00ull, 0x4a7a77d47f7b84b1ull, 0x49ad159789f37496ull,
    0x48e1e9b9d588e19bull, 0x4818ee218a3358eeull, 0x47521cc5a2e6a9e0ull, 0x468d6fadbf2dd4f3ull,
    0x45cae0f1f545eb73ull, 0x450a6abaa4b77ecdull, 0x444c0740496d4294ull, 0x438fb0cb4f468808ull,
    0x42d561b3e6243d8aull, 0x421d1461d66f2023ull, 0x4166c34c5615d0ecull, 0x40b268f9de0183baull,
};

// exp(-3 x) in units of 2^-62 of x < 16 in units of 2^-59, table-driven (Tang
// 1989): 3 x / ln 2 = n + j / 64 + g with g < 1 / 64, exp(-3 x) = 2^-n 2^(-j/64)
// exp(-z), z = g ln 2, exp(-z) by its Taylor polynomial of degree 7 as 1 - z
// + z^2 q(z), with as many bits in each term as its size leaves to matter.
__device__ __forceinline__ unsigned long long exp3_fixed(unsigned long long x) {
    const unsigned long long C = 0x8a7fac5f0511f48dull;  // 3 / ln 2, 2^-61
    const unsigned long long hi = __umul64hi(x, C);
    if (hi >> 62) return 0;  // below 2^-64
    const unsigned long long y = hi << 2 | (x * C) >> 62;  // 2^-58
    const int n = (int)(y >> 58), j = (int)(y >> 52) & 63;
    const unsigned long long z = __umul64hi(y << 12, 0xb17217f7d1cf79acull);  // g ln 2, 2^-70
    const unsigned long long w = __umul64hi(z, z);                           // z^2, 2^-76
    const uint32_t z32 = (uint32_t)(z >> 38), w32 = (uint32_t)(w >> 44);     // 2^-32
    // z^2 / 24 (1 - z / 5 + z^2 / 30 - z^3 / 210), 2^-44
    const uint32_t d = __umulhi(z32, 858993459u) - __umulhi(w32, 143165577u) + __umulhi(__umulhi(z32, w32), 20452225u);
    uint32_t r = (uint32_t)(w >> 32);
    r = __umulhi(r - __umulhi(r, d), 178956971u);
    // q = 1/2 - z / 6 + .., 2^-64
    const unsigned long long q = (1ull << 63) - __umul64hi(z >> 6, 0x2aaaaaaaaaaaaaabull) + ((unsigned long long)r << 20);
    const unsigned long long p = (1ull << 63) - (z >> 7) + (__umul64hi(w, q) >> 13);
    return __umul64hi(p, __ldg(&kExp2J64[j])) >> n;
}

// a positive double below 16 in units of 2^-59 (rounded down)
__device__ __forceinline__ unsigned long long fixed59(double v) {
    const unsigned hi = __double2hiint(v);
    const unsigned long long m = (unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | (unsigned)__double2loint(v);
    const int s = (int)(hi >> 20) - 1016;
    return s >= 0 ? m << s : (s > -64 ? m >> -s : 0);
}

// the float nearest below a double's magnitude, its sign kept, and a float as
// a double; by their bits (conversions use the FP64 pipe).  Magnitudes below
// FP32's count as zero.
__device__ __forceinline__ float to_float_bits(double v) {
    const unsigned hi = __double2hiint(v), lo = __double2loint(v);
    const unsigned u = ((hi << 3) | (lo >> 29)) - (896u << 23);
    return (hi & 0x7ff00000u) > (896u << 20) ? __uint_as_float((u & 0x7fffffffu) | (hi & 0x80000000u)) : 0.0f;
}
__device__ __forceinline__ double to_double_bits(float v) {
    const unsigned u = __float_as_uint(v);
    return __hiloint2double((int)((((u & 0x7fffffffu) >> 3) + (896u << 20)) | (u & 0x80000000u)), (int)(u << 29));
}

// sqrt(s) in units of 2^-59 for s below 225: an FP32 root, corrected by e r / 2
// (r the reciprocal root, e = s - h^2 exact) to some 46 bits, and once more
__device__ __forceinline__ unsigned long long sqrt_fixed(double s) {
    if ((unsigned)__double2hiint(s) < (1023u - 120u) << 20) return 0;
    const float sf = to_float_bits(s);
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(sf));
    double h = to_double_bits(__fmul_rn(sf, r));
    const float half = 0.5f * r;
    h += to_double_bits(__fmul_rn(to_float_bits(fma(-h, h, s)), half));
    const float c = __fmul_rn(to_float_bits(fma(-h, h, s)), half);
    return fixed59(h) + (long long)__float2int_rn(__fmul_rn(c, 576460752303423488.0f));
}

// covariance at a squared normalized lag s, as a part of its value short of
// the nugget, in units of 2^-62
__device__ __forceinline__ unsigned long long shape_fixed(int type, double s) {
    if (!(s < 220.0)) return 0;
    if (type == 3) return s < 16.0 ? exp3_fixed(fixed59(s)) : 0;
    if (type == 1) {
        if (!(s < 1.0)) return 0;
        const unsigned long long h = sqrt_fixed(s), h64 = h >> 59 ? ~0ull : h << 5;  // below 1, 2^-64
        const unsigned long long h3 = __umul64hi(__umul64hi(h64, h64), h64);
        const long long v = (long long)((1ull << 62) - (h64 >> 2) - (h64 >> 3) + (h3 >> 3));  // 1 - 3/2 h + h^3 / 2
        return v > 0 ? v : 0;
    }
    return exp3_fixed(sqrt_fixed(s));
}

// covariance of one structure at a nonzero lag (GeoStatsFunctions conventions:
// practical ranges, nugget for nonzero lags only)
__device__ __forceinline__ double structure_cov_nonzero(const VarioStructDev& v, int dim, double h0, double h1, double h2) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        if (j < dim) {
            double u = fma(v.W[j], h0, v.W[3 + j] * h1);
            if (dim == 3) u = fma(v.W[6 + j], h2, u);
            s = fma(u, u, s);
        }
    }
    return v.psill62 * (double)(long long)shape_fixed(v.type, s);
}

__device__ __forceinline__ bool is_zero(double h) { return (__double_as_longlong(h) << 1) == 0; }

// covariance C(h) = sill - gamma(h), summed over the model's structures
__device__ __forceinline__ double cov_fp64(const VarioDev& v, int dim, double h0, double h1, double h2) {
    if (is_zero(h0) && is_zero(h1) && (dim == 2 || is_zero(h2))) return v.sill;
    double c = 0.0;
#pragma unroll 1
    for (int i = 0; i < v.ns; ++i) c += structure_cov_nonzero(v.st[i], dim, h0, h1, h2);
    return c;
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
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// a - b: the product with -1 is exact, so one rounding as in a subtraction
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { return f2_fma(b, 0xbf800000bf800000ull, a); }

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
    constexpr int SLOTS = 8;
    int ask[SLOTS], open = 0;  // neighbours asked for (-1: a free slot)
#pragma unroll
    for (int h = 0; h < SLOTS; ++h) ask[h] = -1;
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
            if (pending && !(near | mask) && !open) {
                lev[g] = lv;
                s_lev[lane] = lv;
                pending = false;
                moved = true;
            }
            __syncwarp();
            any = __any_sync(FULL_MASK, moved);
        }
        if (!__any_sync(FULL_MASK, pending)) return lv;
        // one turn over global memory: up to SLOTS neighbours are asked for at
        // a time, their ids kept in registers until they answer (found again in
        // the mask and row every turn, and 4 or 16 at a time, 5 to 30 % slower)
        bool moved = false;
        if (pending && (mask || open)) {
            if (mask && open < SLOTS) {
#pragma unroll
                for (int h = 0; h < SLOTS; ++h)
                    if (ask[h] < 0 && mask) {
                        const int q = 63 - __clzll((long long)mask);
                        mask &= ~(1ull << q);
                        ask[h] = row[q];
                        ++open;
                    }
            }
            int l[SLOTS];
#pragma unroll
            for (int h = 0; h < SLOTS; ++h) l[h] = ask[h] >= 0 ? lev[ask[h]] : -1;
#pragma unroll
            for (int h = 0; h < SLOTS; ++h)
                if (l[h] >= 0) {
                    lv = max(lv, l[h] + 1);
                    ask[h] = -1;
                    --open;
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
// off by e = 1 - d r of some 2^-22, and one step of the third-order iteration
// for reciprocals, r (1 + e + e^2) (Householder 1970), off by e^3 and a
// rounding.  The exponents are handled as integers, off the FP64 pipe.
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

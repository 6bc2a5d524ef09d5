// flow.cuh — what the dataflow launches share (sweep.cu, indicator.cu): values
// that are their own "stored" flags, bounded waits, and the hand-out of items.
// The scheme is described at the dataflow sweep in sweep.cu.
#pragma once
#include "common.cuh"

namespace sgs {

struct D4 {
    double x, y, z, w;
};
// All ones in a value's words stands for "not yet stored" in a dataflow launch;
// no other NaN does, and a stored value never has it.
__device__ __forceinline__ bool missing(float v) { return __float_as_uint(v) == 0xffffffffu; }
__device__ __forceinline__ bool missing(double v) { return __double2hiint(v) == -1 && __double2loint(v) == -1; }
template <typename T>
__device__ __forceinline__ T unstored();
template <>
__device__ __forceinline__ float unstored<float>() { return __uint_as_float(0xffffffffu); }
template <>
__device__ __forceinline__ double unstored<double>() { return __hiloint2double(-1, -1); }
__device__ __forceinline__ bool missing4(const float4& v) {  // the largest word is all ones
    return max(max(__float_as_uint(v.x), __float_as_uint(v.y)), max(__float_as_uint(v.z), __float_as_uint(v.w))) == ~0u;
}
__device__ __forceinline__ bool missing4(const D4& v) {
    return missing(v.x) || missing(v.y) || missing(v.z) || missing(v.w);
}
__device__ __forceinline__ float settle(float v) { return missing(v) ? __uint_as_float(0x7fffffffu) : v; }
__device__ __forceinline__ double settle(double v) { return missing(v) ? __hiloint2double(0x7fffffff, -1) : v; }

__device__ __forceinline__ float4 ld_value4(const float* p) {
    float4 v;
    asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ D4 ld_value4(const double* p) {
    D4 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.z), "=d"(v.w) : "l"(p + 2) : "memory");
    return v;
}
__device__ __forceinline__ void st_value4(float* p, float4 v) {
    asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(settle(v.x)), "f"(settle(v.y)),
                 "f"(settle(v.z)), "f"(settle(v.w))
                 : "memory");
}
__device__ __forceinline__ void st_value4(double* p, D4 v) {
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(settle(v.x)), "d"(settle(v.y)) : "memory");
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p + 2), "d"(settle(v.z)), "d"(settle(v.w))
                 : "memory");
}
__device__ __forceinline__ double ld_value(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_value(double* p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(settle(v)) : "memory");
}
__device__ __forceinline__ void st_value(float* p, float v) {
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(settle(v)) : "memory");
}
// a category, 0xff where none is stored yet
__device__ __forceinline__ uint32_t ld_category(const uint8_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_category(uint8_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u8 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// A wait's bound: wait_ns of wall-clock time or, should the timer stall, a
// count of polls (each a load from L2, far above 16 ns, so the count is
// reached no earlier).  False once it has run out or another wait has.
struct FlowBound {
    uint64_t t0 = 0, polls = 0;
    __device__ __forceinline__ bool more(int32_t* err, uint64_t wait_ns) {
        if (++polls > 16) __nanosleep(32);
        if (polls & 63) return true;
        const uint64_t now = global_ns();
        if (t0 == 0) t0 = now;
        if (!*(volatile int32_t*)err && now - t0 <= wait_ns && polls <= wait_ns / 16 + 1024) return true;
        atomicExch(err, 1);
        return false;
    }
};

// The items of a warp: tickets of its class (FLOW_CLASSES), taken one ahead,
// f.chunk items each; `it` runs to items and past it at the end, or once an
// error is raised.
struct FlowItems {
    const FlowArgs& f;
    const int lane, cls;
    unsigned long long ticket;
    int64_t it = 0, end = 0;
    __device__ __forceinline__ explicit FlowItems(const FlowArgs& f_)
        : f(f_), lane(threadIdx.x & 31), cls(threadIdx.x >> 5), ticket(take()) {
        step();
    }
    __device__ __forceinline__ unsigned long long take() {
        unsigned long long base = 0;
        if (lane == 0) {  // the two reads overlap
            base = f.item0 + (atomicAdd(f.ticket + cls * FLOW_TICKET_STRIDE, 1ull) * FLOW_CLASSES + cls) * f.chunk;
            if (*(volatile int32_t*)f.err) base = (unsigned long long)f.item1;
        }
        return base;
    }
    __device__ __forceinline__ bool live() const { return it < f.item1; }
    __device__ __forceinline__ void step() {
        if (++it < end) return;
        it = (int64_t)__shfl_sync(FULL_MASK, ticket, 0);
        end = min(it + f.chunk, f.item1);
        if (it < f.item1) ticket = take();
    }
    // it / H by a reciprocal: exact while it * H < 2^64
    __device__ __forceinline__ int64_t position() const {
        return f.H == 1 ? it : (int64_t)__umul64hi((uint64_t)it, f.rec);
    }
};

}  // namespace sgs

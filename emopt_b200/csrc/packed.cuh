// packed.cuh -- 16-byte vectors of x cells with explicitly rounded arithmetic.
//
// Vec<float> holds 4 cells as two register pairs and computes with the packed
// f32x2 instructions (two IEEE single operations per instruction); Vec<double>
// holds 2 cells.  Every operation rounds once, exactly as the scalar
// instruction of the same name, so a kernel written with them gives the same
// bits as the scalar bodies whose multiply-adds contract in the same places.
#pragma once

#include <cuda_runtime.h>

namespace fdtdb {
namespace pk {

template <typename T>
struct Vec;

// A scalar kernel argument in the form the vector operations take: for float
// the pair of equal values, built on the host.
template <typename T>
struct DupOf;
template <>
struct DupOf<float> {
    using type = unsigned long long;
    static type make(float a) {
        union { float f; unsigned u; } x;
        x.f = a;
        return (unsigned long long)x.u << 32 | x.u;
    }
};
template <>
struct DupOf<double> {
    using type = double;
    static type make(double a) { return a; }
};

template <>
struct Vec<float> {
    static constexpr int N = 4;
    unsigned long long v[2];

    static __device__ __forceinline__ unsigned long long pack(float a, float b) {
        unsigned long long r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
        return r;
    }
    static __device__ __forceinline__ void unpack(unsigned long long r, float& a, float& b) {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
    }
    // a pair of equal values (DupOf<float>)
    static __device__ __forceinline__ Vec dup(unsigned long long a) {
        Vec r;
        r.v[0] = r.v[1] = a;
        return r;
    }
    static __device__ __forceinline__ Vec zero() {
        Vec r;
        r.v[0] = r.v[1] = 0ull;
        return r;
    }
    static __device__ __forceinline__ Vec load(const float* p) {
        const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(p);
        Vec r;
        r.v[0] = q.x;
        r.v[1] = q.y;
        return r;
    }
    __device__ __forceinline__ void get(float* f) const {
        unpack(v[0], f[0], f[1]);
        unpack(v[1], f[2], f[3]);
    }
    __device__ __forceinline__ void set(const float* f) {
        v[0] = pack(f[0], f[1]);
        v[1] = pack(f[2], f[3]);
    }
    __device__ __forceinline__ float at0() const {
        float a, b;
        unpack(v[0], a, b);
        return a;
    }
    // f[k + 1] - f[k] (beyond lane 31: 0 - f) and f[k] - f[k - 1] (the value below
    // the first cell of the lane is `below` when `first`)
    __device__ __forceinline__ Vec diff_down() const {
        float f[4];
        get(f);
        float n = __shfl_down_sync(0xffffffffu, f[0], 1);
        if ((threadIdx.x & 31) == 31) n = 0.0f;
        const float d[4] = {__fsub_rn(f[1], f[0]), __fsub_rn(f[2], f[1]), __fsub_rn(f[3], f[2]), __fsub_rn(n, f[3])};
        Vec r;
        r.set(d);
        return r;
    }
    __device__ __forceinline__ Vec diff_up(bool first, float below) const {
        float f[4];
        get(f);
        float n = __shfl_up_sync(0xffffffffu, f[3], 1);
        if (first) n = below;
        const float d[4] = {__fsub_rn(f[0], n), __fsub_rn(f[1], f[0]), __fsub_rn(f[2], f[1]), __fsub_rn(f[3], f[2])};
        Vec r;
        r.set(d);
        return r;
    }
};

template <>
struct Vec<double> {
    static constexpr int N = 2;
    double v[2];

    static __device__ __forceinline__ Vec bcast(double a) {
        Vec r;
        r.v[0] = r.v[1] = a;
        return r;
    }
    static __device__ __forceinline__ Vec dup(double a) { return bcast(a); }
    static __device__ __forceinline__ Vec zero() { return bcast(0.0); }
    static __device__ __forceinline__ Vec load(const double* p) {
        const double2 q = *reinterpret_cast<const double2*>(p);
        Vec r;
        r.v[0] = q.x;
        r.v[1] = q.y;
        return r;
    }
    __device__ __forceinline__ void get(double* f) const { f[0] = v[0]; f[1] = v[1]; }
    __device__ __forceinline__ void set(const double* f) { v[0] = f[0]; v[1] = f[1]; }
    __device__ __forceinline__ double at0() const { return v[0]; }
    __device__ __forceinline__ Vec diff_down() const {
        double n = __shfl_down_sync(0xffffffffu, v[0], 1);
        if ((threadIdx.x & 31) == 31) n = 0.0;
        Vec r;
        r.v[0] = __dsub_rn(v[1], v[0]);
        r.v[1] = __dsub_rn(n, v[1]);
        return r;
    }
    __device__ __forceinline__ Vec diff_up(bool first, double below) const {
        double n = __shfl_up_sync(0xffffffffu, v[1], 1);
        if (first) n = below;
        Vec r;
        r.v[0] = __dsub_rn(v[0], n);
        r.v[1] = __dsub_rn(v[1], v[0]);
        return r;
    }
};

#define PK_OP2(name, ins, scalar)                                                                          \
    __device__ __forceinline__ Vec<float> name(const Vec<float>& a, const Vec<float>& b) {                 \
        Vec<float> r;                                                                                      \
        asm(ins " %0, %1, %2;" : "=l"(r.v[0]) : "l"(a.v[0]), "l"(b.v[0]));                                 \
        asm(ins " %0, %1, %2;" : "=l"(r.v[1]) : "l"(a.v[1]), "l"(b.v[1]));                                 \
        return r;                                                                                          \
    }                                                                                                      \
    __device__ __forceinline__ Vec<double> name(const Vec<double>& a, const Vec<double>& b) {              \
        Vec<double> r;                                                                                     \
        r.v[0] = scalar(a.v[0], b.v[0]);                                                                   \
        r.v[1] = scalar(a.v[1], b.v[1]);                                                                   \
        return r;                                                                                          \
    }
PK_OP2(sub, "sub.rn.f32x2", __dsub_rn)
PK_OP2(mul, "mul.rn.f32x2", __dmul_rn)
#undef PK_OP2

__device__ __forceinline__ Vec<float> fma(const Vec<float>& a, const Vec<float>& b, const Vec<float>& c) {
    Vec<float> r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v[0]) : "l"(a.v[0]), "l"(b.v[0]), "l"(c.v[0]));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v[1]) : "l"(a.v[1]), "l"(b.v[1]), "l"(c.v[1]));
    return r;
}
__device__ __forceinline__ Vec<double> fma(const Vec<double>& a, const Vec<double>& b, const Vec<double>& c) {
    Vec<double> r;
    r.v[0] = __fma_rn(a.v[0], b.v[0], c.v[0]);
    r.v[1] = __fma_rn(a.v[1], b.v[1], c.v[1]);
    return r;
}
// a - b where b is a product: the assembler fuses a packed multiply with the
// packed add of its result (whatever -fmad says), so the difference is written
// as a fused multiply-add by a run-time -1 (an exact product).
__device__ __forceinline__ Vec<float> diff(const Vec<float>& a, const Vec<float>& b, const Vec<float>& mone) {
    return fma(b, mone, a);
}
__device__ __forceinline__ Vec<double> diff(const Vec<double>& a, const Vec<double>& b, const Vec<double>&) {
    return sub(a, b);
}
// c - a b, rounded once
__device__ __forceinline__ Vec<double> fnma(const Vec<double>& a, const Vec<double>& b, const Vec<double>& c) {
    Vec<double> r;
    r.v[0] = __fma_rn(-a.v[0], b.v[0], c.v[0]);
    r.v[1] = __fma_rn(-a.v[1], b.v[1], c.v[1]);
    return r;
}
__device__ __forceinline__ Vec<float> neg(const Vec<float>& a) {
    Vec<float> r;
    r.v[0] = a.v[0] ^ 0x8000000080000000ull;
    r.v[1] = a.v[1] ^ 0x8000000080000000ull;
    return r;
}
__device__ __forceinline__ Vec<double> neg(const Vec<double>& a) {
    Vec<double> r;
    r.v[0] = -a.v[0];
    r.v[1] = -a.v[1];
    return r;
}

__device__ __forceinline__ Vec<float> fnma(const Vec<float>& a, const Vec<float>& b, const Vec<float>& c) {
    return fma(neg(a), b, c);
}
template <typename T>
__device__ __forceinline__ Vec<T> sel(bool p, const Vec<T>& a, const Vec<T>& b) {
    Vec<T> r;
    r.v[0] = p ? a.v[0] : b.v[0];
    r.v[1] = p ? a.v[1] : b.v[1];
    return r;
}

}  // namespace pk
}  // namespace fdtdb

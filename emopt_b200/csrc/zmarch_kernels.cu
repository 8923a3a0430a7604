// zmarch_kernels.cu -- one fused time step (H half step, then E half step)
// per launch, each CTA marching a tile of rows up through the planes.
//
// Arithmetic per cell: src/fdtd.cpp:175-310 (H) and :503-669 (E), with the
// roundings of the vector pair (vec_body.cuh) written out as explicit
// multiplies, adds and fused multiply-adds, so both give the same bits.
//
// Work of one CTA: rows j0 .. j0+R-1 of one x tile for the planes i0 .. i1-1.
// Warp w updates row j0 - 1 + w; a lane holds one 16-byte vector (4 float or
// 2 double cells).  Warp 0 only recomputes H of row j0-1, lane 0 of a tile
// (but the first) only H of the cells before it, lane 31 of a tile (but the
// last) only supplies E, and the plane before the chunk is stepped for its H
// alone: everything recomputed is read from the field set the step does not
// write, so no CTA waits for another.  Each array crosses DRAM once per step.
//
// Data path: the tile's rows of E, H and the E coefficients come by TMA box
// copies one to two planes ahead (rows, cells and planes outside the grid
// arrive as zeros, the boundary value of E) into rings in shared memory; new
// Hx, Hz go to the row above through shared memory.  One CTA barrier per plane
// both publishes them and frees the ring slots the next copies overwrite.
//
// What bounds it: without CPML DRAM (321 x 161 x 101 cells in float32: 71 us a
// step, 313 MB; 4.4 TB/s); with 20-cell slabs the latency of a plane, 3650
// cycles for a CTA in no slab and up to 8300 in all three of them, of which the
// slab state read from DRAM is the largest part.  16 warps per SM is what 112 KB
// of shared memory and 128 registers (120 lossless in float32) leave, and any
// register spilled inside the plane loop costs more than it saves (the L1 is all
// shared memory: 16 bytes spilled took 193 us instead of 126).  us per step,
// before (vector pair, in the large slab the interior/rim pair) and now, 10- to
// 20-cell slabs, a line of current (801x401x201: a plane):
//   float32  80x80x80 24.9 -> 15.3, 161x81x51 22.1 -> 17.3, 321x161x101 121.6 ->
//            100.7, 801x401x201 1043 -> 905
//   float64  101x76x65 26.8 -> 22.5, 161x81x51 27.0 -> 25.2, 321x161x101 205.0 ->
//            181.8
// Steps are launched with programmatic serialization: a step's CTAs start up in
// the slots the last CTAs of the step before leave and wait there for its end
// (16.6 -> 14.4 us on 64x64x64, 21.2 -> 20.0 on 161x81x51 in float32, 920 -> 905
// on the slab).
#include <algorithm>
#include <cmath>
#include <queue>
#include <utility>
#include <vector>

#include "kernels.h"
#include "packed.cuh"
#include "vec_body.cuh"

namespace fdtdb {

namespace {

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

// The statements below touch shared memory and nothing else does; being
// volatile they keep their order among themselves and against the barriers.
__device__ __forceinline__ void mbar_init(unsigned bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes));
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done) : "r"(bar), "r"(parity));
    return done != 0;
}
// Bounded wait for a copy group.  A wait that gives up reports through *err
// (FDTD_solve_cw then fails) and returns true; the warp then runs on to its
// end with single tries.
__device__ __forceinline__ bool mbar_wait_slow(unsigned bar, unsigned parity, int* err, bool gave_up) {
    for (int n = gave_up ? 0 : 1 << 16; n > 0; n--)
        if (mbar_try(bar, parity)) return false;
    atomicExch(err, 1);
    return true;
}
__device__ __forceinline__ void l1_prefetch(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
// One vector in shared memory, at address a + OFF.
template <typename T, unsigned OFF>
__device__ __forceinline__ pk::Vec<T> sh_load(unsigned a) {
    pk::Vec<T> r;
    if constexpr (sizeof(T) == 4)
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2+%3];" : "=l"(r.v[0]), "=l"(r.v[1]) : "r"(a), "n"(OFF));
    else
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2+%3];" : "=d"(r.v[0]), "=d"(r.v[1]) : "r"(a), "n"(OFF));
    return r;
}
template <unsigned OFF>
__device__ __forceinline__ void sh_store(unsigned a, const pk::Vec<float>& r) {
    asm volatile("st.shared.v2.b64 [%0+%3], {%1, %2};" ::"r"(a), "l"(r.v[0]), "l"(r.v[1]), "n"(OFF));
}
template <unsigned OFF>
__device__ __forceinline__ void sh_store(unsigned a, const pk::Vec<double>& r) {
    asm volatile("st.shared.v2.f64 [%0+%3], {%1, %2};" ::"r"(a), "d"(r.v[0]), "d"(r.v[1]), "n"(OFF));
}
// Box copy of the rows y .. of plane z, cells x .. (x a multiple of 16 bytes).
__device__ __forceinline__ void tma_box(unsigned dst, const CUtensorMap* map, int x, int y, int z, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar));
}

// Global vectors, predicated without a branch, read once.
__device__ __forceinline__ pk::Vec<float> gload(const float* p, unsigned ok) {
    pk::Vec<float> r;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n mov.b64 %0, 0;\n mov.b64 %1, 0;\n"
        " @p ld.global.v2.b64 {%0, %1}, [%2];\n}"
        : "=l"(r.v[0]), "=l"(r.v[1]) : "l"(p), "r"(ok));
    return r;
}
__device__ __forceinline__ pk::Vec<double> gload(const double* p, unsigned ok) {
    pk::Vec<double> r;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n mov.f64 %0, 0d0000000000000000;\n mov.f64 %1, 0d0000000000000000;\n"
        " @p ld.global.v2.f64 {%0, %1}, [%2];\n}"
        : "=d"(r.v[0]), "=d"(r.v[1]) : "l"(p), "r"(ok));
    return r;
}
__device__ __forceinline__ void gstore(float* p, const pk::Vec<float>& v, unsigned ok) {
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p st.global.v2.b64 [%0], {%1, %2};\n}"
                 ::"l"(p), "l"(v.v[0]), "l"(v.v[1]), "r"(ok));
}
__device__ __forceinline__ void gstore(double* p, const pk::Vec<double>& v, unsigned ok) {
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p st.global.v2.f64 [%0], {%1, %2};\n}"
                 ::"l"(p), "d"(v.v[0]), "d"(v.v[1]), "r"(ok));
}
// 1/kappa, b, c of one half step of a y or z slab entry (MarchArgs::ytab, ztab).
template <typename T>
struct Coef {
    pk::Vec<T> k, b, c;
};
template <typename T>
__device__ __forceinline__ Coef<T> coef(const typename pk::DupOf<T>::type* t) {
    Coef<T> r;
    r.k = pk::Vec<T>::dup(__ldg(t)); r.b = pk::Vec<T>::dup(__ldg(t + 1)); r.c = pk::Vec<T>::dup(__ldg(t + 2));
    return r;
}

// One array element block at a 32-bit byte offset: the base stays in uniform
// registers, and all fields and coefficients share one offset register.
template <typename T>
__device__ __forceinline__ const T* at(const T* base, unsigned off) {
    return reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + off);
}
template <typename T>
__device__ __forceinline__ T* at(T* base, unsigned off) {
    return reinterpret_cast<T*>(reinterpret_cast<char*>(base) + off);
}

// Builds with FDTD_BOUNDS_CHECK: `want`, if the 16 bytes at offset off lie in an
// array of `bytes`; else the site is recorded and the access left out.  (The box
// copies need no check: what lies outside their arrays arrives as zeros.)
template <typename T>
__device__ __forceinline__ unsigned inside(const GridView<T>& g, unsigned want, unsigned off, long long bytes, int site) {
#ifdef FDTD_BOUNDS_CHECK
    return want && vecb::in_range(g, off, 0, bytes - 15, site) ? 1u : 0u;
#else
    return want;
#endif
}

// ... and the local slab index l, if it is one of n; else -1.
template <typename T>
__device__ __forceinline__ int slab_inside(const GridView<T>& g, int l, int n, int site) {
#ifdef FDTD_BOUNDS_CHECK
    return l >= 0 && vecb::in_range(g, l, 0, n, site) ? l : -1;
#else
    return l;
#endif
}

// Shared memory, in bytes.  Ex and Ez sit in a ring of three planes (the tile's
// rows, the row below and the row above); everything else in two stages that
// alternate by plane: Ey, H (with the row below), the E coefficients, the new
// Hx, Hz of the plane, the x-slab state (two accumulators of the H, two of
// the E update, kXRow bytes a row).  Then the x-axis CPML tables, one vector
// of zeros and the mbarriers.
constexpr unsigned kRow = 512, kXRow = kMarchXBytes;
template <int NW>
struct MarchSmem {
    static constexpr unsigned ring = 2 * (NW + 1) * kRow;            // one plane of Ex, Ez
    static constexpr unsigned ez = (NW + 1) * kRow;                  // Ez within it
    // within a stage
    static constexpr unsigned ey = 0, h = ey + NW * kRow, b = h + 3 * NW * kRow, x = b + 3 * (NW - 1) * kRow,
                              psx = x + 2 * NW * kRow, stage = (psx + 4 * NW * kXRow + 127) / 128 * 128;
    static_assert(NW * kRow % 128 == 0 && NW * kXRow % 128 == 0, "box copies land on 128-byte boundaries");
    static constexpr unsigned stage0 = 3 * ring, xt = stage0 + 2 * stage, zero = xt + 6 * kRow, bars = zero + 128;
    static constexpr size_t bytes = bars + 64;
};

__device__ __forceinline__ float sfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double sfma(double a, double b, double c) { return __fma_rn(a, b, c); }

// The coefficient pair of one source cell, or zeros.
__device__ __forceinline__ void pair_load(const float* p, bool in, float& re, float& im) {
    const float2 v = in ? *reinterpret_cast<const float2*>(p) : make_float2(0, 0);
    re = v.x; im = v.y;
}
__device__ __forceinline__ void pair_load(const double* p, bool in, double& re, double& im) {
    const double2 v = in ? *reinterpret_cast<const double2*>(p) : make_double2(0, 0);
    re = v.x; im = v.y;
}

// Adds (magnetic, sign +) or subtracts (electric) the currents of the sources
// in `mask` that drive this half step (base 3: M, 0: J) to one vector of cells,
// in source order.  Bound by the latency of the coefficients (~350 cycles from
// L2, on every plane of a march): the pairs of a vector are loaded together,
// without branches between them, not one cell after the other (161 x 81 x 51 in
// float32 with a 34 x 64 x 4 box of Jy and Mz: 27.7 -> 21.0 us a step).
template <typename T, int BASE>
__device__ __forceinline__ void vec_sources(const GridView<T>& g, const SourceList<T>& src, unsigned mask, int i, int j, int c0, T S, T C,
                                            pk::Vec<T>& a, pk::Vec<T>& b, pk::Vec<T>& c) {
    constexpr int VW = pk::Vec<T>::N;
    T f[3][VW];
    a.get(f[0]); b.get(f[1]); c.get(f[2]);
    for (; mask; mask &= mask - 1) {
        const DevSource<T>& s = src.s[__ffs(mask) - 1];
        const int lk = c0 - s.k0;
        const long long m = 2 * (((long long)(i - s.i0) * s.J + (j - s.j0)) * s.K + lk);
#ifdef FDTD_BOUNDS_CHECK
        if (!vecb::in_range(g, i, s.i0, s.i0 + s.I, 27) || !vecb::in_range(g, j, s.j0, s.j0 + s.J, 27)) continue;
#endif
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const T* p = s.comp[BASE + q];
            if (!p) continue;
            T re[VW], im[VW];
#pragma unroll
            for (int e = 0; e < VW; e++) pair_load(p + m + 2 * e, (unsigned)(lk + e) < (unsigned)s.K, re[e], im[e]);
#pragma unroll
            for (int e = 0; e < VW; e++) {
                const T t = sfma(S, re[e], C * im[e]);
                if ((unsigned)(lk + e) < (unsigned)s.K) f[q][e] = BASE ? f[q][e] + t : f[q][e] - t;
            }
        }
    }
    a.set(f[0]); b.set(f[1]); c.set(f[2]);
}

// The curl terms oA fA - dB of a half step.  The vector pair's general body
// rounds both products; its float32 body without CPML code (a plain cell)
// fuses the first.  A warp's cells are all general (mode 0), all plain (1) or
// mixed (2).  m: the rounded products dB on entry, the terms on return.
template <typename T>
__device__ __forceinline__ void curls(int mode, bool plain, const pk::Vec<T> (&oA)[3], const pk::Vec<T> (&fA)[3],
                                      pk::Vec<T> (&m)[3], const pk::Vec<T>& mone) {
    if (sizeof(T) == 8 || mode == 0) {
#pragma unroll
        for (int c = 0; c < 3; c++) m[c] = pk::diff(pk::mul(oA[c], fA[c]), m[c], mone);
    } else if (mode == 1) {
#pragma unroll
        for (int c = 0; c < 3; c++) m[c] = pk::fma(oA[c], fA[c], pk::neg(m[c]));
    } else {
#pragma unroll
        for (int c = 0; c < 3; c++)
            m[c] = pk::sel(plain, pk::fma(oA[c], fA[c], pk::neg(m[c])), pk::diff(pk::mul(oA[c], fA[c]), m[c], mone));
    }
}

// The value below a min face from the boundary rule (h_min_ghost of each cell).
template <typename T>
__device__ __forceinline__ pk::Vec<T> ghost(char bc, const pk::Vec<T>& first) {
    if (bc == '0') return pk::Vec<T>::zero();
    return bc == 'E' ? pk::neg(first) : first;
}

// psi <- c d + b psi, and the correction (psi - d) + d / kappa that is added
// to the curl term d.
template <typename T>
__device__ __forceinline__ pk::Vec<T> cpml(pk::Vec<T>& p, const pk::Vec<T>& d, const pk::Vec<T>& kinv,
                                           const pk::Vec<T>& b, const pk::Vec<T>& c, const pk::Vec<T>& mone) {
    p = pk::fma(c, d, pk::mul(b, p));
    return pk::fma(d, kinv, pk::diff(p, d, mone));
}

}  // namespace

template <typename T, int NW, int MINB, bool LOSSY, bool MUARR>
__global__ void __launch_bounds__(32 * NW, MINB)
k_step_march(const __grid_constant__ MarchArgs<T> A, const __grid_constant__ SourceList<T> src,
             const int4* work, const long long* step_base, int off) {
    using V = pk::Vec<T>;
    using L = MarchSmem<NW>;
    constexpr int VW = V::N, R = NW - 1;
    constexpr unsigned SZ = sizeof(T);
    extern __shared__ __align__(128) unsigned char smem[];
    const GridView<T>& g = A.g;
    const PmlAxis<T>& PX = g.pml[0];
    const PmlAxis<T>& PY = g.pml[1];
    const PmlAxis<T>& PZ = g.pml[2];
    const int lane = threadIdx.x & 31, w = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    // The next step may take the slots this one leaves (its copies wait below for
    // the whole of this grid), so its start-up overlaps this step's last CTAs.
    asm volatile("griddepcontrol.launch_dependents;");
    const unsigned bars = smem_u32(smem) + L::bars;
    const bool leader = threadIdx.x == 0;
    if (leader) {
        for (int q = 0; q < 4; q++) mbar_init(bars + 8 * q);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const int4 job = work[blockIdx.x];              // x tile, row tile, planes job.z .. job.w - 1
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("fence.proxy.async.global;" ::: "memory");   // the box copies read what the last step stored
    const int x0 = job.x * (30 * VW), c0 = x0 + lane * VW;
    const int j0 = job.y * R, j = j0 - 1 + w;
    const int i0 = job.z, i1 = job.w, is = i0 > 0 ? i0 - 1 : 0;
#ifdef FDTD_BOUNDS_CHECK
    if (!vecb::in_range(g, x0, 0, g.Nx, 20) || !vecb::in_range(g, job.y * R, 0, g.Ny, 20) ||
        !vecb::in_range(g, i0, 0, i1, 20) || !vecb::in_range(g, i1, 1, g.Nz + 1, 20))
        return;
#endif
    const bool row = j >= 0 && j < g.Ny;
    const bool ok = row && c0 < g.Nx;
    const bool own = ok && w > 0 && (lane > 0 || job.x == 0) && (lane < 31 || job.x == A.x_tiles - 1);
    // byte offsets: a plane, this vector in a plane
    const unsigned pb = (unsigned)g.Ny * g.px * SZ;
    const unsigned rb = ok ? (unsigned)(j * g.px + c0) * SZ : 0u;
    const unsigned sbase = smem_u32(smem);
    const int ly = slab_inside(g, row ? slab_local(PY, j, false) : -1, PY.wsum, 22);
    // x slab: slot of this vector in the whole-vector psi rows, or -1
    int sx = -1;
    if (c0 < PX.w0) sx = c0;
    else if (c0 < g.Nx && c0 + VW > PX.edge_max && PX.w1 > 0) sx = A.x_max_slot + c0;
    const bool inx = __any_sync(0xffffffffu, sx >= 0);
    // the tile's slots, when they fit one box row, come by TMA as well
    const int slo = __reduce_min_sync(0xffffffffu, sx >= 0 ? sx : 1 << 30), shi = __reduce_max_sync(0xffffffffu, sx);
    const bool xtma = inx && (shi + VW - slo) * (int)SZ <= (int)kXRow;
    const unsigned xoff = L::psx + w * kXRow + (unsigned)(sx >= 0 ? sx - slo : 0) * SZ;
    if (!ok) sx = -1;
    // float32: does the vector pair update this cell's 64-cell task by its
    // body without CPML code in the planes of no z slab?
    const int xb0 = c0 & ~63;
    const bool plain = SZ == 4 && ly < 0 && xb0 >= PX.w0 && xb0 + 63 < PX.edge_max;
    const int mode_xy = SZ == 8 ? 0
                        : __all_sync(0xffffffffu, plain || !ok) ? 1
                        : __any_sync(0xffffffffu, plain && ok)  ? 2
                                                                : 0;
    // sources whose box holds cells of this warp's row (bit q: M currents, 16 + q:
    // J currents), and those that touch this cell's 64-cell task of the pair
    unsigned touch = 0, task = 0;
    if (row)
        for (int q = 0; q < src.n; q++) {
            const DevSource<T>& s = src.s[q];
            if (j < s.j0 || j >= s.j0 + s.J) continue;
            const unsigned bits = (s.comp[3] || s.comp[4] || s.comp[5] ? 1u << q : 0u) |
                                  (s.comp[0] || s.comp[1] || s.comp[2] ? 0x10000u << q : 0u);
            if (s.k0 < x0 + 32 * VW && s.k0 + s.K > x0) touch |= bits;
            if (A.src_general && s.k0 < xb0 + 64 && s.k0 + s.K > xb0) task |= bits;
        }
    const unsigned near = __reduce_or_sync(0xffffffffu, touch | task);
    T srcS[2] = {T(0), T(0)}, srcC[2] = {T(0), T(0)};     // step constants of the M and J currents
    if (near) {
        const double4 st = g.step_tab[*step_base + off];
        srcS[0] = T(st.x); srcC[0] = T(st.y); srcS[1] = T(st.z); srcC[1] = T(st.w);
    }

    bool gave_up = false;
    auto wait = [&](unsigned bar, unsigned parity) {
        if (!mbar_try(bar, parity)) gave_up = mbar_wait_slow(bar, parity, A.err, gave_up) || gave_up;
    };
    // Copies of one thread: E of plane p (Ez unless only read from below) into
    // a ring slot; Ey of plane p and H of plane q into their stages; the
    // coefficients of plane q.
    auto stage_at = [&](int i) { return sbase + L::stage0 + (((i - is) & 1) ? L::stage : 0u); };
    auto fetch_e = [&](int p, unsigned slot, bool full, unsigned bar) {
        tma_box(slot, &A.tm_in[0], x0, j0 - 1, p, bar);
        if (full) tma_box(slot + L::ez, &A.tm_in[2], x0, j0 - 1, p, bar);
    };
    auto fetch_x = [&](int q, int e, unsigned bar) {
        if (!xtma) return;
        const unsigned s = stage_at(q) + L::psx + 2 * e * NW * kXRow;
        tma_box(s, &A.tm_x[2 * e], slo, j0 - 1, q, bar);
        tma_box(s + NW * kXRow, &A.tm_x[2 * e + 1], slo, j0 - 1, q, bar);
    };
    auto fetch_eyh = [&](int p, int q, unsigned bar) {
        tma_box(stage_at(p) + L::ey, &A.tm_in[1], x0, j0 - 1, p, bar);
#pragma unroll
        for (int c = 0; c < 3; c++)
            tma_box(stage_at(q) + L::h + c * NW * kRow, &A.tm_in[3 + c], x0, j0 - 1, q, bar);
        fetch_x(q, 0, bar);
    };
    const unsigned xbytes = xtma ? 2 * NW * kXRow : 0;
    auto fetch_b = [&](int q, unsigned bar) {
        mbar_expect(bar, 3 * (NW - 1) * kRow + xbytes);
        fetch_x(q, 1, bar);
#pragma unroll
        for (int c = 0; c < 3; c++)
            tma_box(stage_at(q) + L::b + c * (NW - 1) * kRow, &A.tm_b[c], x0, j0, q, bar);
    };
    const unsigned a_bytes = (2 * (NW + 1) + NW + 3 * NW) * kRow + xbytes;

    // Per-thread addresses: E ring slots of planes i, i + 1, i + 2 (own row),
    // stages of planes i and i + 1, and the barriers (A, then B 16 bytes on)
    unsigned r0 = sbase, r1 = sbase + L::ring, r2 = sbase + 2 * L::ring;
    unsigned sa = sbase + L::stage0, sb = sa + L::stage, ba = bars, bb = bars + 8;
    if (leader) {
        // E(is), E(is+1), H(is) for the first plane; E(is+2), H(is+1) for the next
        mbar_expect(ba, a_bytes + 2 * (NW + 1) * kRow - (is + 1 < i1 ? 0 : (NW + 1) * kRow));
        fetch_e(is, r0, true, ba);
        fetch_e(is + 1, r1, is + 1 < i1, ba);
        fetch_eyh(is + 1, is, ba);
        fetch_b(is, ba + 16);
        if (is + 1 < i1) {
            mbar_expect(bb, a_bytes - (is + 2 < i1 ? 0 : (NW + 1) * kRow));
            fetch_e(is + 2, r2, is + 2 < i1, bb);
            fetch_eyh(is + 2, is + 1, bb);
        }
    }
    static_assert(NW == 8, "the copies are spread over eight warps");
    const unsigned lrow = w * kRow + lane * 16;
    r0 += lrow; r1 += lrow; r2 += lrow; sa += lrow; sb += lrow;
    if (w == NW - 1)
        for (int q = 0; q < 6; q++)
            sh_store<0>(sbase + L::xt + q * kRow + lane * 16, V::load(A.xtab[q] + (c0 < g.px ? c0 : 0)));
    if (threadIdx.x == 32) sh_store<0>(sbase + L::zero, V::zero());
    const unsigned xta = sbase + L::xt + lane * 16;
    V ey = V::zero(), hpy = V::zero();      // Ey of the plane, new Hy of the plane below
    // array sizes of the checked build: fields, x-, y- and z-slab state
    const long long fbytes = (long long)g.Nz * pb, xbytes_all = (long long)g.Nz * g.Ny * A.x_pitch * SZ;
    const long long ybytes = (long long)g.Nz * PY.wsum * g.px * SZ, zbytes = (long long)PZ.wsum * pb;
    if (inside(g, ok, (unsigned)is * pb + rb, fbytes, 21)) ey = V::load(at(A.in.c[1], (unsigned)is * pb + rb));
    __syncthreads();

    const bool iny = ly >= 0, xmin = job.x == 0;
    unsigned o = (unsigned)is * pb + rb;                              // this vector in the fields,
    unsigned oX = ((unsigned)(is * g.Ny + j) * A.x_pitch + sx) * SZ;  // in the x- and y-slab state
    unsigned oY = ((unsigned)(is * PY.wsum + ly) * g.px + (ok ? c0 : 0)) * SZ;
    const unsigned strideY = (unsigned)PY.wsum * g.px * SZ, strideX = (unsigned)g.Ny * A.x_pitch * SZ;
    const unsigned sxu = sx >= 0, ownu = own, ownxu = own && sx >= 0;
    // x-slab state in a stage relative to sa (lanes without a slot read zeros)
    const unsigned xz = sbase + L::zero;
    const V ox = V::dup(A.o[0]), oy = V::dup(A.o[1]), oz = V::dup(A.o[2]), mone = V::dup(A.mone);
    unsigned phase = 0;

#pragma unroll 1
    for (int i = is; i < i1; i++) {
        const int lz = slab_inside(g, slab_local(PZ, i + PZ.off, true), PZ.wsum, 23);
        const bool inz = lz >= 0, emit = i >= i0;      // the plane before the chunk: H only
        const unsigned oZ = (unsigned)lz * pb + rb;
        const unsigned eo = inside(g, emit ? ownu : 0u, o, fbytes, 21), eox = inside(g, emit ? ownxu : 0u, oX, xbytes_all, 24);

        // ---- CPML state of the H update
        V py0, py1, pz0, pz1;
        if (iny) {
            const unsigned in = inside(g, 1u, oY, ybytes, 25);
            py0 = gload(at(A.ph_in[1][0], oY), in); py1 = gload(at(A.ph_in[1][1], oY), in);
        }
        if (inz) {
            const unsigned in = inside(g, 1u, oZ, zbytes, 26);
            pz0 = gload(at(A.ph_in[2][0], oZ), in); pz1 = gload(at(A.ph_in[2][1], oZ), in);
        }

        // ---- which cells round their curls as the vector pair's plain body;
        // the sources of this row in this plane
        int modeH = inz ? 0 : mode_xy, modeE = modeH;
        bool plH = plain, plE = plain;
        unsigned now = 0;
        if (near) {
            for (int q = 0; q < src.n; q++)
                if (i >= src.s[q].i0 && i < src.s[q].i0 + src.s[q].I) now |= 0x10001u << q;
            now &= near;
            if (modeH && A.src_general && now) {
                // a task that a source touches takes the general body
                plH = plain && !(task & now & 0xffffu);
                plE = plain && !(task & now & 0xffff0000u);
                modeH = modeE = 2;
            }
            now &= touch;
        }

        // ---- E of the plane, the row above and the plane above; H
        wait(ba, phase);
        if (i + 1 < i1) {
            if (MUARR && ok)
                for (int c = 0; c < 3; c++) l1_prefetch(at(g.bHarr[c], o + pb));
            if (iny) { l1_prefetch(at(A.ph_in[1][0], oY + strideY)); l1_prefetch(at(A.ph_in[1][1], oY + strideY)); }
            if (inz) { l1_prefetch(at(A.ph_in[2][0], oZ + pb)); l1_prefetch(at(A.ph_in[2][1], oZ + pb)); }
        }
        V ex = sh_load<T, 0>(r0), ez = sh_load<T, L::ez>(r0);
        const V exj = sh_load<T, kRow>(r0), ezj = sh_load<T, L::ez + kRow>(r0);
        const V exi = sh_load<T, 0>(r1), eyi = sh_load<T, L::ey>(sb);
        V hx = sh_load<T, L::h>(sa), hy = sh_load<T, L::h + NW * kRow>(sa), hz = sh_load<T, L::h + 2 * NW * kRow>(sa);

        // ---- H update
        {
            const V fzdy = pk::sub(ezj, ez), fydz = pk::sub(eyi, ey), fxdz = pk::sub(exi, ex);
            const V fzdx = ez.diff_down(), fydx = ey.diff_down(), fxdy = pk::sub(exj, ex);
            V m0, m1, m2;
            if (MUARR) {
                const unsigned in = inside(g, ok ? 1u : 0u, o, fbytes, 21);
                m0 = gload(at(g.bHarr[0], o), in); m1 = gload(at(g.bHarr[1], o), in); m2 = gload(at(g.bHarr[2], o), in);
            } else {
                m0 = V::dup(A.m[0]); m1 = V::dup(A.m[1]); m2 = V::dup(A.m[2]);
            }
            const V oA[3] = {oz, ox, oy}, fA[3] = {fydz, fzdx, fxdy};
            V t[3] = {pk::mul(oy, fzdy), pk::mul(oz, fxdz), pk::mul(ox, fydx)};
            curls<T>(modeH, plH, oA, fA, t, mone);
            hx = pk::fma(m0, t[0], hx);
            hy = pk::fma(m1, t[1], hy);
            hz = pk::fma(m2, t[2], hz);
            if (inx) {
                const V kv = sh_load<T, 0>(xta), bv = sh_load<T, kRow>(xta), cv = sh_load<T, 2 * kRow>(xta);
                V p0, p1;
                if (xtma) {
                    const unsigned q = sxu ? sa - lrow + xoff : xz;
                    p0 = sh_load<T, 0>(q);
                    p1 = sh_load<T, 0>(sxu ? q + NW * kXRow : q);
                } else {
                    const unsigned in = inside(g, sxu, oX, xbytes_all, 24);
                    p0 = gload(at(A.ph_in[0][0], oX), in); p1 = gload(at(A.ph_in[0][1], oX), in);
                }
                hz = pk::fnma(m2, cpml(p0, pk::mul(ox, fydx), kv, bv, cv, mone), hz);
                hy = pk::fma(m1, cpml(p1, pk::mul(ox, fzdx), kv, bv, cv, mone), hy);
                gstore(at(A.ph_out[0][0], oX), p0, eox); gstore(at(A.ph_out[0][1], oX), p1, eox);
            }
            if (iny) {
                const Coef<T> c = coef<T>(A.ytab + 6 * ly);
                hz = pk::fma(m2, cpml(py0, pk::mul(oy, fxdy), c.k, c.b, c.c, mone), hz);
                hx = pk::fnma(m0, cpml(py1, pk::mul(oy, fzdy), c.k, c.b, c.c, mone), hx);
                const unsigned in = inside(g, eo, oY, ybytes, 25);
                gstore(at(A.ph_out[1][0], oY), py0, in); gstore(at(A.ph_out[1][1], oY), py1, in);
            }
            if (inz) {
                const Coef<T> c = coef<T>(A.ztab + 6 * lz);
                hx = pk::fma(m0, cpml(pz1, pk::mul(oz, fydz), c.k, c.b, c.c, mone), hx);
                hy = pk::fnma(m1, cpml(pz0, pk::mul(oz, fxdz), c.k, c.b, c.c, mone), hy);
                const unsigned in = inside(g, eo, oZ, zbytes, 26);
                gstore(at(A.ph_out[2][0], oZ), pz0, in); gstore(at(A.ph_out[2][1], oZ), pz1, in);
            }
        }
        if (now & 0xffffu) vec_sources<T, 3>(g, src, now & 0xffffu, i, j, c0, srcS[0], srcC[0], hx, hy, hz);
        sh_store<L::x>(sa, hx);
        sh_store<L::x + NW * kRow>(sa, hz);
        gstore(at(A.out.c[3], o), hx, eo);
        gstore(at(A.out.c[4], o), hy, eo);
        gstore(at(A.out.c[5], o), hz, eo);

        // ---- CPML state of the E update
        if (iny) {
            const unsigned in = inside(g, eo, oY, ybytes, 25);
            py0 = gload(at(A.pe[1][0], oY), in); py1 = gload(at(A.pe[1][1], oY), in);
        }
        if (inz) {
            const unsigned in = inside(g, eo, oZ, zbytes, 26);
            pz0 = gload(at(A.pe[2][0], oZ), in); pz1 = gload(at(A.pe[2][1], oZ), in);
        }
        V a0, a1, a2;                                  // E-update factors of lossy media
        if (LOSSY) { a0 = gload(at(g.aE[0], o), eo); a1 = gload(at(g.aE[1], o), eo); a2 = gload(at(g.aE[2], o), eo); }
        __syncthreads();
        // E(i), Ey(i+1), H(i) and the coefficients of plane i - 1 have been read:
        // the next copies, spread over the warps (one issue takes ~200 cycles)
        if (lane == 0) {
            int v = w;
            asm volatile("" : "+r"(v));              // keeps what follows out of registers between planes
            if (v == 0) {
                if (i + 2 < i1) {
                    const bool full = i + 3 < i1;
                    mbar_expect(ba, a_bytes - (full ? 0 : (NW + 1) * kRow));
                    fetch_e(i + 3, r0, full, ba);
                    fetch_x(i + 2, 0, ba);
                }
                if (i + 1 < i1) {
                    mbar_expect(bb + 16, 3 * (NW - 1) * kRow + xbytes);
                    fetch_x(i + 1, 1, bb + 16);
                }
            } else if (v < 5) {
                // Ey of plane i + 3 (warp 1), H of plane i + 2 (2..4)
                if (i + 2 < i1)
                    tma_box((v == 1 ? sb + L::ey : sa + L::h + (v - 2) * NW * kRow) - v * kRow, &A.tm_in[v == 1 ? 1 : v + 1],
                            x0, j0 - 1, v == 1 ? i + 3 : i + 2, ba);
            } else if (i + 1 < i1) {
                // the coefficients of plane i + 1
                tma_box(sb + L::b + (v - 5) * (NW - 1) * kRow - v * kRow, &A.tm_b[v - 5], x0, j0, i + 1, bb + 16);
            }
        }
        if (w > 0) {
            wait(ba + 16, phase);
            if (emit) {
                const V bx = sh_load<T, L::b - kRow>(sa), by = sh_load<T, L::b + (NW - 2) * kRow>(sa),
                        bz = sh_load<T, L::b + (2 * NW - 3) * kRow>(sa);
                V hxj = sh_load<T, L::x - kRow>(sa), hzj = sh_load<T, L::x + (NW - 1) * kRow>(sa);   // the row below's
                V hpx = sh_load<T, L::x>(sb);                                                       // the plane below's
                if (j == 0) {
                    hxj = ghost<T>(g.bc[1], hx);
                    hzj = ghost<T>(g.bc[1], hz);
                }
                if (i == 0) { hpx = ghost<T>(g.bc[2], hx); hpy = ghost<T>(g.bc[2], hy); }
                const V fzdy = pk::sub(hz, hzj), fydz = pk::sub(hy, hpy), fxdz = pk::sub(hx, hpx), fxdy = pk::sub(hx, hxj);
                // differences to the cells k - 1
                const bool first = xmin && c0 == 0;
                const V fzdx = hz.diff_up(first, first ? h_min_ghost<T>(g.bc[0], hz.at0(), T(0)) : T(0));
                const V fydx = hy.diff_up(first, first ? h_min_ghost<T>(g.bc[0], hy.at0(), T(0)) : T(0));
                const V oA[3] = {oy, oz, ox}, fA[3] = {fzdy, fxdz, fydx};
                V t[3] = {pk::mul(oz, fydz), pk::mul(ox, fzdx), pk::mul(oy, fxdy)};
                curls<T>(modeE, plE, oA, fA, t, mone);
                if (LOSSY) {
                    ex = pk::fma(a0, ex, pk::mul(t[0], bx));
                    ey = pk::fma(a1, ey, pk::mul(t[1], by));
                    ez = pk::fma(a2, ez, pk::mul(t[2], bz));
                } else {
                    ex = pk::fma(t[0], bx, ex); ey = pk::fma(t[1], by, ey); ez = pk::fma(t[2], bz, ez);
                }
                if (inx) {
                    const V kv = sh_load<T, 3 * kRow>(xta), bv = sh_load<T, 4 * kRow>(xta), cv = sh_load<T, 5 * kRow>(xta);
                    V p0, p1;
                    if (xtma) {
                        const unsigned q = sxu ? sa - lrow + xoff + 2 * NW * kXRow : xz;
                        p0 = sh_load<T, 0>(q);
                        p1 = sh_load<T, 0>(sxu ? q + NW * kXRow : q);
                    } else {
                        const unsigned in = inside(g, ownxu, oX, xbytes_all, 24);
                        p0 = gload(at(A.pe[0][0], oX), in); p1 = gload(at(A.pe[0][1], oX), in);
                    }
                    ez = pk::fma(cpml(p0, pk::mul(ox, fydx), kv, bv, cv, mone), bz, ez);
                    ey = pk::fnma(cpml(p1, pk::mul(ox, fzdx), kv, bv, cv, mone), by, ey);
                    const unsigned in = inside(g, ownxu, oX, xbytes_all, 24);
                    gstore(at(A.pe[0][0], oX), p0, in); gstore(at(A.pe[0][1], oX), p1, in);
                }
                if (iny) {
                    const Coef<T> c = coef<T>(A.ytab + 6 * ly + 3);
                    ez = pk::fnma(cpml(py0, pk::mul(oy, fxdy), c.k, c.b, c.c, mone), bz, ez);
                    ex = pk::fma(cpml(py1, pk::mul(oy, fzdy), c.k, c.b, c.c, mone), bx, ex);
                    const unsigned in = inside(g, ownu, oY, ybytes, 25);
                    gstore(at(A.pe[1][0], oY), py0, in); gstore(at(A.pe[1][1], oY), py1, in);
                }
                if (inz) {
                    const Coef<T> c = coef<T>(A.ztab + 6 * lz + 3);
                    ex = pk::fnma(cpml(pz1, pk::mul(oz, fydz), c.k, c.b, c.c, mone), bx, ex);
                    ey = pk::fma(cpml(pz0, pk::mul(oz, fxdz), c.k, c.b, c.c, mone), by, ey);
                    const unsigned in = inside(g, ownu, oZ, zbytes, 26);
                    gstore(at(A.pe[2][0], oZ), pz0, in); gstore(at(A.pe[2][1], oZ), pz1, in);
                }
                if (now >> 16) vec_sources<T, 0>(g, src, now >> 16, i, j, c0, srcS[1], srcC[1], ex, ey, ez);
                const unsigned in = inside(g, ownu, o, fbytes, 21);
                gstore(at(A.out.c[0], o), ex, in);
                gstore(at(A.out.c[1], o), ey, in);
                gstore(at(A.out.c[2], o), ez, in);
            }
        }
        ey = eyi;
        hpy = hy;
        unsigned q = r0;
        r0 = r1; r1 = r2; r2 = q;
        q = sa; sa = sb; sb = q;
        phase ^= (unsigned)(i - is) & 1u;
        q = ba; ba = bb; bb = q;
        o += pb; oX += strideX; oY += strideY;
    }
    // after a wait that gave up, time for copies still in flight to land
    if (gave_up)
        for (int n = 0; n < 4096; n++) __nanosleep(1000);
}

namespace {

// Rows per CTA plus one: 8 warps, 2 CTAs (16 warps) per SM.
constexpr int kNW = 8, kMinB = 2;

template <typename T, bool LOSSY, bool MUARR>
cudaError_t launch_one(const MarchArgs<T>& a, const SourceList<T>& src, const int4* work, int nwork,
                       const long long* step_base, int off, cudaStream_t st) {
    constexpr size_t bytes = MarchSmem<kNW>::bytes;
    auto k = k_step_march<T, kNW, kMinB, LOSSY, MUARR>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nwork);
    cfg.blockDim = dim3(32 * kNW);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a, src, work, step_base, off);
}

template <typename T>
int x_tiles(int Nx) {
    constexpr int V = pk::Vec<T>::N;
    return std::max(1, (Nx - 2 * V + 30 * V - 1) / (30 * V));
}

}  // namespace

template <typename T>
cudaError_t march_maps(MarchArgs<T>& a) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult st;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &st);
    if (e != cudaSuccess) return e;
    if (st != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    const GridView<T>& g = a.g;
    a.x_tiles = x_tiles<T>(g.Nx);
    const CUtensorMapDataType type = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
    auto map = [&](CUtensorMap* m, const T* p, int rows) {
        const cuuint64_t dims[3] = {(cuuint64_t)g.Nx, (cuuint64_t)g.Ny, (cuuint64_t)g.Nz};
        const cuuint64_t strides[2] = {(cuuint64_t)g.px * sizeof(T), (cuuint64_t)g.plane * sizeof(T)};
        const cuuint32_t box[3] = {(cuuint32_t)(512 / sizeof(T)), (cuuint32_t)rows, 1}, one[3] = {1, 1, 1};
        return ((Encode)fn)(m, type, 3, const_cast<T*>(p), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = CUDA_SUCCESS;
    for (int c = 0; c < 6 && r == CUDA_SUCCESS; c++)
        r = map(&a.tm_in[c], a.in.c[c], c == 0 || c == 2 ? kNW + 1 : kNW);   // Ex, Ez: the row above too
    for (int c = 0; c < 3 && r == CUDA_SUCCESS; c++) r = map(&a.tm_b[c], g.bE[c], kNW - 1);
    for (int c = 0; c < 4 && a.x_pitch > 0 && r == CUDA_SUCCESS; c++) {
        const cuuint64_t dims[3] = {(cuuint64_t)a.x_pitch, (cuuint64_t)g.Ny, (cuuint64_t)g.Nz};
        const cuuint64_t strides[2] = {(cuuint64_t)a.x_pitch * sizeof(T), (cuuint64_t)a.x_pitch * g.Ny * sizeof(T)};
        const cuuint32_t box[3] = {(cuuint32_t)(kMarchXBytes / sizeof(T)), kNW, 1}, one[3] = {1, 1, 1};
        r = ((Encode)fn)(&a.tm_x[c], type, 3, c < 2 ? const_cast<T*>(a.ph_in[0][c]) : a.pe[0][c - 2], dims, strides,
                         box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_step_march(const MarchArgs<T>& a, const SourceList<T>& src, const int4* work, int nwork,
                              const long long* step_base, int off, cudaStream_t st) {
    const bool lossy = a.g.aE[0] != nullptr, mu = a.g.bHarr[0] != nullptr;
    if (lossy) return mu ? launch_one<T, true, true>(a, src, work, nwork, step_base, off, st)
                         : launch_one<T, true, false>(a, src, work, nwork, step_base, off, st);
    return mu ? launch_one<T, false, true>(a, src, work, nwork, step_base, off, st)
              : launch_one<T, false, false>(a, src, work, nwork, step_base, off, st);
}

namespace {

// Estimated cycles (thousands) of a plane of each tile column.  A CTA takes as
// long as its slowest warp, and CPML state makes planes slow (cycles per plane on
// the 321 x 161 x 101 grid in float32 with 20-cell slabs: 3650 in none, 4600 in an
// x slab, 5900 z, 6700 y, 8300 in all three).
template <typename T>
struct MarchCost {
    static constexpr int V = pk::Vec<T>::N, R = kNW - 1;
    const GridView<T>& g;
    const int ntx, nty, ncol;
    std::vector<char> inz;           // planes in a z slab, and their number
    int nz = 0;

    explicit MarchCost(const GridView<T>& g)
        : g(g), ntx(x_tiles<T>(g.Nx)), nty((g.Ny + R - 1) / R), ncol(ntx * nty), inz(g.Nz) {
        for (int i = 0; i < g.Nz; i++) nz += inz[i] = slab_local(g.pml[2], i + g.pml[2].off, true) >= 0;
    }
    double plane(int col, bool z) const {
        const int x = col % ntx, y = col / ntx;
        const PmlAxis<T>*P = g.pml;
        const int c0 = x * 30 * V, c1 = std::min(c0 + 32 * V, g.Nx), j0 = std::max(0, y * R - 1), j1 = std::min(y * R + R, g.Ny);
        const bool sx = c0 < P[0].w0 || (P[0].w1 > 0 && c1 > P[0].edge_max);
        const bool sy = j0 < P[1].w0 || (P[1].w1 > 0 && j1 > P[1].edge_max);
        return 3.65 + (sx ? 0.9 : 0.0) + (sy && z ? 3.8 : sy ? 3.0 : z ? 2.2 : 0.0);
    }
    double column(int col) const { return nz * plane(col, true) + (g.Nz - nz) * plane(col, false); }
    // Does the tile hold more x-slab state than a box copy brings (cells of both
    // slabs, mostly)?
    bool wide_x(int x) const {
        const PmlAxis<T>& P = g.pml[0];
        auto up = [](int k) { return (k + V - 1) / V * V; };
        const int c0 = x * 30 * V, c1 = std::min(c0 + 32 * V, up(g.Nx));
        const int first = P.edge_max & ~(V - 1);            // the vector the max slab starts in
        const int lo = std::min(c1, up(P.w0)) - c0, hi = P.w1 > 0 ? c1 - std::max(c0, first) : 0;
        return (std::max(lo, 0) + std::max(hi, 0)) * (int)sizeof(T) > (int)kXRow;
    }
};

}  // namespace

// Is the fused step faster than the pair that would run in its place (split: the
// split pair)?  Its time goes with the cycles per CTA slot (t, thousands), the
// pair's with its warp tasks of 64 cells (q: their number per thousand cycles of
// the fused step).  A CTA works for seven rows whether they are there or not, and
// in slab code where one of them lies in a slab, so grids of few rows, or mostly
// slab, leave the fused step behind once they are too large to be bound by
// launches and latency.  us per step, pair and fused:
//   float32  512x1x300 (t 21, q 0.11) 10.6 13.9 (split pair 20.8), 150x2x1008 (31,
//            0.19) 15.6 19.6, 580x1x947 (65, 0.15) 18.6 33.8 (split 28.0);
//            256x16x100 (23, 0.27) 16.7 15.1, 59x105x114 (37, 0.33) 24.0 21.9
//   float64  88x1x486 (15, 0.06) 10.6 12.4, 179x2x791 (29, 0.16) 14.7 17.8,
//            324x1x1082 (80, 0.08) 16.8 39.4, 126x33x171 (62, 0.18) 30.5 36.2,
//            374x36x39 (40, 0.21) 22.9 25.8, 119x31x163 (40, 0.25) 27.1 30.0;
//            128x1x100 (5, 0.04) 10.6 8.1, 128x16x100 (23, 0.14) 16.7 14.7,
//            305x34x34 (25, 0.23) 19.7 16.8, 101x76x65 (33, 0.30) 26.6 22.2
// Where a tile's x-slab state does not come by box copies its planes take about
// a quarter longer in float64: 72x90x90 with 15-cell slabs (51, 0.32) 35.1 40.0,
// 62x79x136 with 12 (34, 0.32) 27.0 30.7, 93x141x73 with 20 (67, 0.31) 51.5 54.3,
// but 62x90x90 (26, 0.32) 24.9 21.4.  Over 710 grids of up to 3 M cells the pair's
// time over the chosen one's is 1.256 in float64 and 1.432 in float32 (geometric
// mean; the better of both: 1.261, 1.433); near the lines either side wins by up
// to 8%.
template <typename T>
bool march_pays(const GridView<T>& g, int sms, bool split) {
    const MarchCost<T> c(g);
    double t = 0.0;
    for (int q = 0; q < c.ncol; q++) t += c.column(q);
    t /= kMinB * (sms > 0 ? sms : 148);
    const double q = 1e-3 * ((g.Nx + 63) / 64) * g.Ny * g.Nz / t;
    if (sizeof(T) == 4) return t <= (split ? 33.0 : 20.5) || q >= 0.25;
    bool wide = false;
    for (int x = 0; x < c.ntx; x++) wide = wide || c.wide_x(x);
    if (wide && t > 31.0 && q < 0.36) return false;
    return t <= 13.0 || q >= (t <= 25.0 ? 0.12 : t <= 33.0 ? 0.17 : 0.29);
}

// The chunks of the tile columns: every column is cut into chunks of equal
// estimated time (MarchCost), the column with the longest ones first.  Chunks of 8
// planes on average, in as many waves as that takes, keep neighbouring tiles close
// in z (their halo rows hit L2) and the last wave short: 105.6 us a step on the
// 321 x 161 x 101 grid against 107.5 with 9-13 planes, 118 in one wave and 125.6 in
// equal chunks of 26; in float64 185 against 227 in one wave.  Grids that fill
// less than a wave take one wave.
template <typename T>
void march_work(const GridView<T>& g, int sms, int zc, std::vector<int4>& work) {
    const MarchCost<T> cost(g);
    const int ntx = cost.ntx, nty = cost.nty, ncol = cost.ncol, Nz = g.Nz;
    work.clear();
    if (zc > 0) {
        for (int i = 0; i < Nz; i += zc)
            for (int y = 0; y < nty; y++)
                for (int x = 0; x < ntx; x++) work.push_back(make_int4(x, y, i, std::min(i + zc, Nz)));
        return;
    }
    const int slots = std::max(1, kMinB * (sms > 0 ? sms : 148));
    const double fill = 8.0;                       // first copies and the plane before the chunk
    std::vector<double> total(ncol);
    for (int c = 0; c < ncol; c++) total[c] = cost.column(c);
    // kChunk planes a chunk on average, one wave of CTAs at least; the column with
    // the longest chunks is cut first
    constexpr double kChunk = 8.0;
    const int waves = std::max(1, (int)std::lround((double)ncol * Nz / (kChunk * slots)));
    std::vector<int> best(ncol, 1);
    std::priority_queue<std::pair<double, int>> longest;
    for (int c = 0; c < ncol; c++) longest.push({total[c] + fill, c});
    for (long long k = ncol; k < (long long)waves * slots; k++) {
        const int c = longest.top().second;
        if (best[c] >= Nz) break;
        longest.pop();
        best[c]++;
        longest.push({total[c] / best[c] + fill, c});
    }
    // cut the columns; chunk k of every column before chunk k + 1 of any
    std::vector<std::vector<int4>> rank;
    for (int c = 0; c < ncol; c++) {
        const double in = cost.plane(c, true), out = cost.plane(c, false);
        double acc = 0.0;
        int from = 0, k = 1;
        for (int i = 0; i < Nz; i++) {
            acc += cost.inz[i] ? in : out;
            if (i + 1 < Nz && !(k < best[c] && acc >= total[c] * k / best[c])) continue;
            if ((int)rank.size() < k) rank.resize(k);
            rank[k - 1].push_back(make_int4(c % ntx, c / ntx, from, i + 1));
            from = i + 1;
            k++;
        }
    }
    for (const auto& r : rank) work.insert(work.end(), r.begin(), r.end());
}

template cudaError_t launch_step_march<float>(const MarchArgs<float>&, const SourceList<float>&, const int4*, int,
                                              const long long*, int, cudaStream_t);
template cudaError_t launch_step_march<double>(const MarchArgs<double>&, const SourceList<double>&, const int4*, int,
                                               const long long*, int, cudaStream_t);
template cudaError_t march_maps<float>(MarchArgs<float>&);
template cudaError_t march_maps<double>(MarchArgs<double>&);
template bool march_pays<float>(const GridView<float>&, int, bool);
template bool march_pays<double>(const GridView<double>&, int, bool);
template void march_work<float>(const GridView<float>&, int, int, std::vector<int4>&);
template void march_work<double>(const GridView<double>&, int, int, std::vector<int4>&);

}  // namespace fdtdb

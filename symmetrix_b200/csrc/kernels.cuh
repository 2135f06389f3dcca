// CUDA kernels of the MACE energy+force path for sm_100a.
//
// Data layout in HBM (all row-major, channel index fastest, one arithmetic type T per evaluator):
//   node features  A0/A1 [N][16][K], M0/H1 [rows][nLM][K], Phi1 [N][Q][K], M1/H2 [N][K]
//   spline tables  [pair][bin][function block][2][V][2] with V lanes (see Lane): one double channel or two float channels
//                  (16-byte vector loads that a warp issues over contiguous 512-byte spans)
//   contraction    coefficients [element][monomial][K]
// One thread owns one lane -- one channel in double, two neighbouring channels in float -- of one receiver
// node, so every global access is a contiguous run of values across the CTA. Per-edge quantities that do not depend on the channel
// (harmonics, their gradients, coupling blocks, spline bin) are computed once per edge into
// shared memory and broadcast. No per-edge channel array (R0, R1, Y, Phi1r of the reference,
// libsymmetrix/source/mace.hpp:44-113) is ever written to HBM.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include <utility>

#include "common.cuh"
#include "tp_tables.hpp"
#include "generated/poly_canon.hpp"
#include "generated/tp_scale.hpp"

namespace smx {

#ifndef SMX_EDGE_BATCH
#define SMX_EDGE_BATCH 32
#endif
constexpr int kEdgeBatch = SMX_EDGE_BATCH;   // edges staged in shared memory per pass (one staging latency and two barriers per batch)
// thread t of a CTA stages edge t of a batch and a CTA may be a single warp, so a batch holds at most 32 edges (the 40-edge
// measurement was a build for 128-channel models only, with this check lifted)
#ifndef SMX_EDGE_BATCH_UNCHECKED
static_assert(kEdgeBatch >= 1 && kEdgeBatch <= 32, "SMX_EDGE_BATCH must be between 1 and 32");
#endif
constexpr int kChannelBlock = 128;  // threads per CTA of the edge kernels; more channels are done in chunks
constexpr int kMaxWarps = kChannelBlock / 32;

// Compile-time loop: f(std::integral_constant<int, 0>{}), ..., f(std::integral_constant<int, N-1>{}).
// The tensor-product kernels index their register accumulators with path-dependent offsets, which
// must be constants for the accumulators to stay in registers.
template <typename F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
    static_for_impl(f, std::make_integer_sequence<int, N>{});
}
template <int LF>
struct TPConst {
    static constexpr TPTable t = make_tp_table(LF);
};

// ---------------------------------------------------------------------------------------------
// What a thread of the edge kernels computes on: 64 bits, a double or a pair of floats of two neighbouring channels. The pair
// goes through the packed instructions (fma.rn.f32x2 and its kin: two multiply-adds per issue slot, each rounded like the
// scalar one): every broadcast of edge data, address computation and reduction step is then paid per two channels. Measured
// instructions per (edge, 128 channels) at 1,372 atoms: forward 571 in pairs against 1,131 of a double each.
// ---------------------------------------------------------------------------------------------
struct alignas(8) F2 {
    unsigned long long v;
    __device__ __forceinline__ F2() {}
    __device__ __forceinline__ F2(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
    __device__ __forceinline__ explicit F2(float a) : F2(a, a) {}
    __device__ __forceinline__ explicit F2(double a) : F2(static_cast<float>(a)) {}
    __device__ __forceinline__ explicit F2(unsigned lo, unsigned hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi)); }
    __device__ __forceinline__ float lo() const { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return a; }
    __device__ __forceinline__ float hi() const { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return b; }
};
using ::fma;
__device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v)); return r; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 operator-(F2 a) { return F2(-1.0f) * a; }

template <typename T> struct Lane;               // lane type that most kernels use for a memory type
template <> struct Lane<double> { using type = double; };
template <> struct Lane<float> { using type = F2; };
template <typename V> struct LaneScalar { using type = V; };
template <> struct LaneScalar<F2> { using type = float; };
template <typename V> __host__ __device__ __forceinline__ constexpr int lane_channels() { return static_cast<int>(sizeof(V) / sizeof(typename LaneScalar<V>::type)); }
// Lanes of a row of K channels; the second half of the last pair of an odd row is idle.
template <typename V> __host__ __device__ __forceinline__ constexpr int lanes_of(int K) { return (K + lane_channels<V>() - 1) / lane_channels<V>(); }
// Channels of a row of the spline tables: padded to whole lanes.
template <typename T> __host__ __device__ __forceinline__ constexpr int table_channels(int K) { return lanes_of<typename Lane<T>::type>(K) * lane_channels<typename Lane<T>::type>(); }

__device__ __forceinline__ double lane_sum(double x) { return x; }
__device__ __forceinline__ float lane_sum(float x) { return x; }
__device__ __forceinline__ float lane_sum(F2 x) { return x.lo() + x.hi(); }
__device__ __forceinline__ unsigned lane_lo(double x) { return static_cast<unsigned>(__double2loint(x)); }
__device__ __forceinline__ unsigned lane_hi(double x) { return static_cast<unsigned>(__double2hiint(x)); }
__device__ __forceinline__ unsigned lane_lo(F2 x) { return __float_as_uint(x.lo()); }
__device__ __forceinline__ unsigned lane_hi(F2 x) { return __float_as_uint(x.hi()); }
template <typename V> __device__ __forceinline__ V lane_from_bits(unsigned lo, unsigned hi) {
    if constexpr (lane_channels<V>() == 1) return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
    else return F2(lo, hi);
}

// Lane `l` of a row of K channels at `p`. Rows of an even number of floats start on 8-byte boundaries; odd ones take scalars. WHOLE
// (a template parameter of the edge kernels: K is even) says so at compile time: a branch on K at every load ends the block of
// instructions that the compiler may reorder, so the loads of an edge went out a few at a time (reverse tensor product on pairs,
// float32, 4,000 atoms, K = 128: 1,130 us with the branches, 790 without). Layer 0 forward and the forward tensor product at
// L_max = 0 do little per load and lose with it (see Evaluator::with_rows): they keep the branch for every K.
enum class Cache { kDefault, kReadOnly, kStream };
template <Cache C, typename U> __device__ __forceinline__ U cached_load(const U* p) {
    if constexpr (C == Cache::kReadOnly) return __ldg(p);
    else if constexpr (C == Cache::kStream) return __ldcs(p);
    else return *p;
}
template <typename V, bool WHOLE, Cache C = Cache::kDefault>
__device__ __forceinline__ V lane_load(const typename LaneScalar<V>::type* p, int l, int K) {
    if constexpr (lane_channels<V>() == 1) {
        return cached_load<C>(p + l);
    } else {
        if (WHOLE || (K & 1) == 0) {
            V r;
            r.v = cached_load<C>(reinterpret_cast<const unsigned long long*>(p) + l);
            return r;
        }
        return V(cached_load<C>(p + 2 * l), 2 * l + 1 < K ? cached_load<C>(p + 2 * l + 1) : 0.0f);
    }
}
template <bool STREAM, bool WHOLE, typename V>
__device__ __forceinline__ void lane_store(typename LaneScalar<V>::type* p, int l, int K, V x) {
    auto put = [](auto* q, auto v) { if constexpr (STREAM) __stcs(q, v); else *q = v; };
    if constexpr (lane_channels<V>() == 1) {
        put(p + l, x);
    } else if (WHOLE || (K & 1) == 0) {
        put(reinterpret_cast<unsigned long long*>(p) + l, x.v);
    } else {
        put(p + 2 * l, x.lo());
        if (2 * l + 1 < K) put(p + 2 * l + 1, x.hi());
    }
}
// Adds a float lane to memory with vector reductions where the row allows.
template <bool WHOLE> __device__ __forceinline__ void lane_atomic_add(float* p, int l, int, float x) { atomicAdd(p + l, x); }
template <bool WHOLE> __device__ __forceinline__ void lane_atomic_add(float* p, int l, int K, F2 x) {
    if (WHOLE || (K & 1) == 0) {
        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p + 2 * l), "f"(x.lo()), "f"(x.hi()) : "memory");
    } else {
        atomicAdd(p + 2 * l, x.lo());
        if (2 * l + 1 < K) atomicAdd(p + 2 * l + 1, x.hi());
    }
}

// The four cubic coefficients of lane l from one (pair, bin, function-block) row of 4 * Kt values, Kt = table_channels(K), stored
// [2][L][2] lanes (c0, c1 of every lane, then c2, c3 of every lane): each of the two 16-byte loads of a warp covers 512 contiguous
// bytes, i.e. 4 L1 wavefronts instead of the 8 that an interleaved [L][4] row (32-byte stride between threads) costs.
template <typename V> struct Coef { V x, y, z, w; };
// Single floats have tables of their own, [K][4]: one 16-byte load per channel.
// `block`: the function block in row 0 of the table (the same for all threads); `at`: 16-byte units from there to the lane's
// first load (row of the edge + lane), so that a load's address is one multiply-add of a 32-bit register.
template <typename V, typename I>
__device__ __forceinline__ Coef<V> load_coef(const typename LaneScalar<V>::type* block, I at, int L) {
    if constexpr (sizeof(V) == 4) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(block) + at);
        return {v.x, v.y, v.z, v.w};
    } else {
        const ulonglong2* q = reinterpret_cast<const ulonglong2*>(block);
        const ulonglong2 a = __ldg(q + at), b = __ldg(q + L + at);
        Coef<V> c;
        if constexpr (lane_channels<V>() == 1) {
            c.x = __longlong_as_double(a.x); c.y = __longlong_as_double(a.y); c.z = __longlong_as_double(b.x); c.w = __longlong_as_double(b.y);
        } else {
            c.x.v = a.x; c.y.v = a.y; c.z.v = b.x; c.w.v = b.y;
        }
        return c;
    }
}
// Position of coefficient q (0..3) of channel k in such a row.
template <typename T> __host__ __device__ __forceinline__ constexpr int coef_offset(int k, int q, int Kt) {
    constexpr int C = lane_channels<typename Lane<T>::type>();
    return (q >> 1) * 2 * Kt + (2 * (k / C) + (q & 1)) * C + k % C;
}
// Value and derivative of the cubic at x (x15 = 1.5 x, x2 = 2 x).
template <typename V>
__device__ __forceinline__ V cubic_value(const Coef<V>& c, V x) { return fma(x, fma(x, fma(x, c.w, c.z), c.y), c.x); }
template <typename V>
__device__ __forceinline__ V cubic_slope(const Coef<V>& c, V x2, V x15) { return fma(x2, fma(x15, c.w, c.z), c.y); }

// ---------------------------------------------------------------------------------------------
// Bulk asynchronous copies (TMA, cp.async.bulk) of spline rows into shared memory, completed on an
// mbarrier. Every wait is bounded: a wait that runs out returns false and the caller records it.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1;\n\t}" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
constexpr unsigned kMbarSpinLimit = 1u << 22;
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, unsigned limit = kMbarSpinLimit) {
    const uint32_t addr = smem_u32(bar);
    for (unsigned spin = 0; spin < limit; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
// global -> shared, both addresses 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// Channel `kl` of a staged row chunk of `Kc` channels: the layout of load_coef with K = Kc (float64 only).
__device__ __forceinline__ Coef<double> lds_coef(const double* slot, int p, int kl, int Kc) {
    const double2 a = reinterpret_cast<const double2*>(slot)[(2 * p) * Kc + kl];
    const double2 b = reinterpret_cast<const double2*>(slot)[(2 * p + 1) * Kc + kl];
    return {a.x, a.y, b.x, b.y};
}

// One thread: start the copy of the chunk [kc, kc + Kc) of all P function blocks of a spline row into a slot.
__device__ __forceinline__ void issue_row_copy(double* slot, const double* row, int P, int K, int kc, int Kc, unsigned long long* bar) {
    const unsigned bytes = 4u * P * Kc * sizeof(double);
    mbar_expect_tx(bar, bytes);
    if (Kc == K) {
        bulk_copy_g2s(slot, row, bytes, bar);
    } else {
        for (int q = 0; q < 2 * P; ++q) bulk_copy_g2s(slot + 2 * q * Kc, row + 2 * (q * K + kc), 16u * Kc, bar);
    }
}

// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum each of 16 per-lane values over the warp with 16 shuffles instead of 80: every step halves the
// number of values a lane carries by exchanging the other half with its partner. On return the lane
// holds the warp-wide sum of value `index` (lanes that differ only in bit 0 hold the same value).
template <typename T>
__device__ __forceinline__ T warp_reduce_scatter16(const T (&v)[16], int lane, int& index) {
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4, b1 = lane & 2;
    T w8[8], w4[4], w2[2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const T send = b4 ? v[i] : v[i + 8], keep = b4 ? v[i + 8] : v[i];
        w8[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const T send = b3 ? w8[i] : w8[i + 4], keep = b3 ? w8[i + 4] : w8[i];
        w4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const T send = b2 ? w4[i] : w4[i + 2], keep = b2 ? w4[i + 2] : w4[i];
        w2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
    const T send = b1 ? w2[0] : w2[1], keep = b1 ? w2[1] : w2[0];
    T w1 = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    w1 += __shfl_xor_sync(0xffffffffu, w1, 1);
    index = (b4 ? 8 : 0) + (b3 ? 4 : 0) + (b2 ? 2 : 0) + (b1 ? 1 : 0);
    return w1;
}

// Sums over the lanes of a warp of the 16 adjoints of one edge: W[0] of the edge length, W[lm] of the harmonic lm > 0 (the adjoint of
// the harmonic of degree zero is not needed: its gradient is zero; as a seventeenth value it cost 6 % of the float64 reverse
// tensor product, 1,515 against 1,427 us at 4,000 atoms). Through shuffles, or with a scratch area through shared memory (every lane
// stores its 16 values, then each pair of lanes adds up one of them with 16-byte loads): 40 instead of 72 instructions. For the
// reverse tensor product in float32, 750 against 791 us at 4,000 atoms; its float64 form, where each value is two words,
// took 1,554 against 1,427 us, and layer 0 in float32, whose CTAs are limited by shared memory, 297 against 283. The CTAs of one and two
// warps that narrow rows of single floats take are limited by it too (see Evaluator::launch_tp).
constexpr int kSumStride = 40;      // floats per value: rows of 16-byte loads that a quarter warp reads start in different banks
template <typename T> struct SumScratch {};      // none: shuffles
template <> struct alignas(16) SumScratch<float> { float v[kNumLm * kSumStride]; };      // per warp
template <typename V, typename S>
__device__ __forceinline__ void warp_edge_sums(const V (&W)[kNumLm], int lane, SumScratch<S>* scratch, typename LaneScalar<V>::type (&red)[17]) {
    using T = typename LaneScalar<V>::type;
    if constexpr (!std::is_same_v<S, float>) {
        T w[kNumLm];
#pragma unroll
        for (int q = 0; q < kNumLm; ++q) w[q] = lane_sum(W[q]);
        int idx;
        const T s = warp_reduce_scatter16(w, lane, idx);
        if ((lane & 1) == 0) red[idx] = s;
    } else {
        __syncwarp();               // the sums of the previous edge have been read
#pragma unroll
        for (int q = 0; q < kNumLm; ++q) scratch->v[q * kSumStride + lane] = lane_sum(W[q]);
        __syncwarp();
        const float4* q = reinterpret_cast<const float4*>(scratch->v + (lane >> 1) * kSumStride) + (lane & 1);
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float4 v = q[2 * i]; s0 += v.x + v.y; s1 += v.z + v.w; }
        float s = s0 + s1;
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if ((lane & 1) == 0) red[lane >> 1] = s;
    }
}

// Per-edge partial force from the warp-reduced adjoints, written by one thread per edge:
//   nf -= xhat * dE/dr + sum_lm dE/dY_lm * grad Y_lm
// red[w][e][0], w in [warp0, warp0 + nwarps): dE/dr summed over the channels of warp w, red[w][e][lm]: dE/dY_lm.
template <typename T, int EB>
__device__ __forceinline__ void finish_edge_force(const T (*red)[EB][17], int warp0, int nwarps, int e, const T* dY0, const T* dY1, const T* dY2,
                                                  T ux, T uy, T uz, double* nf) {
    double tr = 0, fx = 0, fy = 0, fz = 0;
    for (int w = warp0; w < warp0 + nwarps; ++w) tr += red[w][e][0];
#pragma unroll
    for (int lm = 1; lm < kNumLm; ++lm) {
        double wv = 0;
        for (int w = warp0; w < warp0 + nwarps; ++w) wv += red[w][e][lm];
        fx += wv * double(dY0[lm]); fy += wv * double(dY1[lm]); fz += wv * double(dY2[lm]);
    }
    nf[0] -= double(ux) * tr + fx;
    nf[1] -= double(uy) * tr + fy;
    nf[2] -= double(uz) * tr + fz;
}

// ---------------------------------------------------------------------------------------------
// Real spherical harmonics up to l = 3 of the direction (a, b, c) = xyz / r, in the convention the
// reference feeds its tensor products with (mace.cpp:118-148: orthonormal real harmonics of the
// axis-shuffled vector (z, x, y), times 2 sqrt(pi), lm = l*l + l + m), written as polynomials in
// the un-shuffled components. g[c][lm] receives the Cartesian gradient d Y_lm / d xyz_c.
// ---------------------------------------------------------------------------------------------
template <typename T, bool GRAD>
__host__ __device__ inline void real_sh3(T a, T b, T c, T inv_r, T* __restrict__ Y, T (*__restrict__ g)[kNumLm]) {
    const T s3 = T(1.7320508075688772935), s15 = T(3.8729833462074168852), s5h = T(1.1180339887498948482);
    const T s105 = T(10.246950765959598383), s7h = T(1.3228756555322952953);
    const T k9 = T(2.0916500663351888699);   // sqrt(35/8)
    const T k11 = T(1.6201851746019651311);  // sqrt(21/8)
    const T aa = a * a, bb = b * b, cc = c * c;
    Y[0] = T(1);
    Y[1] = s3 * a; Y[2] = s3 * b; Y[3] = s3 * c;
    Y[4] = s15 * c * a;
    Y[5] = s15 * a * b;
    Y[6] = s5h * (T(3) * bb - T(1));
    Y[7] = s15 * c * b;
    Y[8] = T(0.5) * s15 * (cc - aa);
    Y[9] = k9 * a * (T(3) * cc - aa);
    Y[10] = s105 * a * b * c;
    Y[11] = k11 * a * (T(5) * bb - T(1));
    Y[12] = s7h * b * (T(5) * bb - T(3));
    Y[13] = k11 * c * (T(5) * bb - T(1));
    Y[14] = T(0.5) * s105 * b * (cc - aa);
    Y[15] = k9 * c * (cc - T(3) * aa);
    if constexpr (GRAD) {
        T d[3][kNumLm];
        d[0][0] = 0; d[1][0] = 0; d[2][0] = 0;
        d[0][1] = s3; d[1][1] = 0; d[2][1] = 0;
        d[0][2] = 0; d[1][2] = s3; d[2][2] = 0;
        d[0][3] = 0; d[1][3] = 0; d[2][3] = s3;
        d[0][4] = s15 * c; d[1][4] = 0; d[2][4] = s15 * a;
        d[0][5] = s15 * b; d[1][5] = s15 * a; d[2][5] = 0;
        d[0][6] = 0; d[1][6] = T(6) * s5h * b; d[2][6] = 0;
        d[0][7] = 0; d[1][7] = s15 * c; d[2][7] = s15 * b;
        d[0][8] = -s15 * a; d[1][8] = 0; d[2][8] = s15 * c;
        d[0][9] = k9 * T(3) * (cc - aa); d[1][9] = 0; d[2][9] = k9 * T(6) * a * c;
        d[0][10] = s105 * b * c; d[1][10] = s105 * a * c; d[2][10] = s105 * a * b;
        d[0][11] = k11 * (T(5) * bb - T(1)); d[1][11] = k11 * T(10) * a * b; d[2][11] = 0;
        d[0][12] = 0; d[1][12] = s7h * (T(15) * bb - T(3)); d[2][12] = 0;
        d[0][13] = 0; d[1][13] = k11 * T(10) * b * c; d[2][13] = k11 * (T(5) * bb - T(1));
        d[0][14] = -s105 * a * b; d[1][14] = T(0.5) * s105 * (cc - aa); d[2][14] = s105 * b * c;
        d[0][15] = -k9 * T(6) * a * c; d[1][15] = 0; d[2][15] = k9 * T(3) * (cc - aa);
        // chain rule through u = xyz / r: grad = (d - u (u . d)) / r
#pragma unroll
        for (int lm = 0; lm < kNumLm; ++lm) {
            const T rad = d[0][lm] * a + d[1][lm] * b + d[2][lm] * c;
            g[0][lm] = (d[0][lm] - rad * a) * inv_r;
            g[1][lm] = (d[1][lm] - rad * b) * inv_r;
            g[2][lm] = (d[2][lm] - rad * c) * inv_r;
        }
    }
}

// Per-edge, channel-independent quantities staged in shared memory.
// Where the edge's row of a spline table starts.
template <int ALIGN> struct EdgeRow;
template <> struct EdgeRow<8> {
    long long coef_base;      // (pair * num_bins + bin) * F * 4 values
    int spare[2];             // keeps the stride of the array at two (float) and four (double) bank conflicts per store
};
template <> struct EdgeRow<16> {
    unsigned coef_row;        // the same in units of 16 bytes
    unsigned coef_row_dir;    // the same with the ordered pair (type_i * num_elements + type_j): folded layer-0 table
};
// ALIGN = 16 lets load_harmonics use 16-byte loads. It suits the kernels whose shared-memory reads count (layer 0: one harmonics
// read per multiply-add; float32 forward at 4,000 atoms 178 -> 147 us; the float64 tensor-memory kernel, 1 to 4 %); in the others
// the staging threads' stores, one edge per thread, then meet more bank conflicts than the loads save (forward +3 %).
template <typename V, int ALIGN = 8>
struct alignas(ALIGN) EdgeStage {
    using T = typename LaneScalar<V>::type;
    V Y[kNumLm];              // harmonics, one copy per channel of a lane (first: 16-byte loads start here)
    T dY[3][kNumLm];          // gradients (reverse kernels only)
    T x;                      // r - h * bin
    T ux, uy, uz;             // unit vector
    EdgeRow<ALIGN> row;
    int j;                    // sender row
    int tj;                   // sender type
};

// What the 16-byte harmonics loads rely on, for every element of an array of stages in shared memory.
template <typename V>
constexpr bool edge_stage_loads_aligned() {
    using Stage = EdgeStage<V, 16>;
    return offsetof(Stage, Y) == 0 && alignof(Stage) == 16 && sizeof(Stage) % 16 == 0 && sizeof(V) * kNumLm % 16 == 0;
}
static_assert(edge_stage_loads_aligned<double>() && edge_stage_loads_aligned<F2>(), "load_harmonics reads 16 bytes at a time from the start of a stage");

// All harmonics of an edge.
template <typename V>
__device__ __forceinline__ void load_harmonics(const EdgeStage<V, 8>& s, V (&Y)[kNumLm]) {
#pragma unroll
    for (int lm = 0; lm < kNumLm; ++lm) Y[lm] = s.Y[lm];
}
template <typename V>
__device__ __forceinline__ void load_harmonics(const EdgeStage<V, 16>& s, V (&Y)[kNumLm]) {
    constexpr int n = 16 / static_cast<int>(sizeof(V));
    struct alignas(16) Pack { V v[n]; };
#pragma unroll
    for (int q = 0; q < kNumLm / n; ++q) {
        const Pack p = reinterpret_cast<const Pack*>(s.Y)[q];
#pragma unroll
        for (int m = 0; m < n; ++m) Y[q * n + m] = p.v[m];
    }
}

struct SplineMeta {
    double h;
    int num_bins;
    int num_elements;
};

// ---------------------------------------------------------------------------------------------
// Work distribution of the edge kernels. The grids are persistent (resident CTAs per SM x SMs) and the work items are
// handed out through a device counter, in order, so that a CTA that shares its SM with fewer others, or drew shorter
// items, simply takes more of them: with a static split the kernel lasts as long as the CTA with the most items
// (4000 receivers over 444 CTAs: ten rounds for an average of nine). sched[0] = next item, sched[1] = CTAs that have left;
// the last CTA to leave re-arms both, so no launch needs a memset.
// The reverse kernels write per-edge outputs only, so their item is (receiver, batch of <= kEdgeBatch of its edges, equal
// sizes), listed once per edge set by work_items_fill_kernel; measured on the 4000-atom float64 case: tensor-product reverse
// 2.01 -> 1.87 ms. The forward kernels accumulate over a receiver's edges (item = receiver) and keep the static split: with
// the counter they measured 2-3 % slower.
// ---------------------------------------------------------------------------------------------
// The item after the current one is requested when the current one starts, so the counter's latency hides behind the work;
// two slots alternate, and the barrier that ends an item orders the slot's write before its read.
__device__ __forceinline__ int work_first(int* __restrict__ sched, int (&s_next)[2]) {
    if (threadIdx.x == 0) s_next[0] = atomicAdd(sched, 1);
    __syncthreads();
    return s_next[0];
}
__device__ __forceinline__ void work_prefetch(int* __restrict__ sched, int (&s_next)[2], int& par) {
    par ^= 1;
    if (threadIdx.x == 0) s_next[par] = atomicAdd(sched, 1);
}
__device__ __forceinline__ int work_next(const int (&s_next)[2], int par) {
    __syncthreads();                 // everyone is done with the current item (shared memory); s_next[par] is written
    return s_next[par];
}
__device__ __forceinline__ void work_leave(int* __restrict__ sched) {
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(sched + 1, 1) == static_cast<int>(gridDim.x) - 1) { sched[0] = 0; sched[1] = 0; __threadfence(); }
    }
}
// Edges per work item: kEdgeBatch, or fewer when that would leave CTAs of a full GPU without an item.
__host__ __device__ __forceinline__ int work_batch(long long edges, int want_items) {
    const long long b = (edges + want_items - 1) / want_items;
    return b < 1 ? 1 : (b > kEdgeBatch ? kEdgeBatch : static_cast<int>(b));
}
static __global__ void work_items_count_kernel(int N, int want_items, const int* __restrict__ order, const long long* __restrict__ first_neigh, int* __restrict__ counts) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= N) return;
    const int i = order ? order[slot] : slot;
    const int batch = work_batch(first_neigh[N], want_items);
    counts[slot] = static_cast<int>((first_neigh[i + 1] - first_neigh[i] + batch - 1) / batch);
}
// items[q] = (receiver, first edge relative to the receiver's row, number of edges, 0)
static __global__ void work_items_fill_kernel(int N, int want_items, const int* __restrict__ order, const long long* __restrict__ first_neigh,
                                              const int* __restrict__ item_ptr, int4* __restrict__ items, int* __restrict__ n_items) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= N) return;
    const int i = order ? order[slot] : slot;
    const int deg = static_cast<int>(first_neigh[i + 1] - first_neigh[i]);
    const int batch = work_batch(first_neigh[N], want_items);
    const int nb = (deg + batch - 1) / batch;
    const int size = nb ? (deg + nb - 1) / nb : 0;
    for (int b = 0; b < nb; ++b) {
        const int begin = b * size;
        items[item_ptr[slot] + b] = make_int4(i, begin, deg - begin < size ? deg - begin : size, 0);
    }
    if (slot == N - 1) *n_items = item_ptr[slot] + nb;
}

// Fill stage[e] for the edges [e0, e0 + nb) of node i; executed by threads 0..nb-1.
template <typename V, bool GRAD, int ALIGN>
__device__ __forceinline__ void stage_edge(EdgeStage<V, ALIGN>& s, long long edge, int type_i, const int* __restrict__ neigh_indices,
                                           const int* __restrict__ neigh_types, const double* __restrict__ xyz,
                                           const double* __restrict__ r, const SplineMeta sm, int F) {
    const double rr = r[edge];
    const double inv = 1.0 / rr;
    const double ax = xyz[3 * edge] * inv, ay = xyz[3 * edge + 1] * inv, az = xyz[3 * edge + 2] * inv;
    using T = typename LaneScalar<V>::type;
    s.ux = T(ax); s.uy = T(ay); s.uz = T(az);
    if constexpr (lane_channels<V>() == 1) {
        real_sh3<T, GRAD>(T(ax), T(ay), T(az), T(inv), s.Y, s.dY);
    } else {
        T y[kNumLm];
        real_sh3<T, GRAD>(T(ax), T(ay), T(az), T(inv), y, s.dY);
#pragma unroll
        for (int lm = 0; lm < kNumLm; ++lm) s.Y[lm] = V(y[lm]);
    }
    // bin and offset exactly as CubicSplineSet::evaluate_derivs (cubic_spline_set.cpp:55-56),
    // clamped to the last interval so that r within rounding of r_cut stays inside the table
    int bin = static_cast<int>(rr / sm.h);
    bin = bin < 0 ? 0 : (bin > sm.num_bins - 1 ? sm.num_bins - 1 : bin);
    s.x = T(rr - sm.h * bin);
    const int tj = neigh_types[edge];
    s.tj = tj;
    s.j = neigh_indices[edge];
    const int lo = type_i <= tj ? type_i : tj, hi = type_i <= tj ? tj : type_i;
    const int pair = lo * (2 * sm.num_elements - lo - 1) / 2 + hi;   // mace.cpp:81-83
    if constexpr (ALIGN == 16) {
        const unsigned row16 = static_cast<unsigned>(F) * (sizeof(T) / 4);
        s.row.coef_row = (static_cast<unsigned>(pair) * sm.num_bins + bin) * row16;
        s.row.coef_row_dir = (static_cast<unsigned>(type_i * sm.num_elements + tj) * sm.num_bins + bin) * row16;
    } else {
        s.row.coef_base = (static_cast<long long>(pair) * sm.num_bins + bin) * F * 4;
    }
}

// ---------------------------------------------------------------------------------------------
// Folded layer-0 table. A0[i, lm, k'] = sum_k Phi0[i, lm, k] W[a][l][k, k'] with Phi0 a sum over edges of
// R0_ab(r)[l, k] Y[lm] H0[b, k] (a, b = receiver, sender type). The spline is linear in its coefficients, so
//   c'[(a, b), bin, l, k', q] = sum_k c[pair(a, b), bin, l, k, q] H0[b, k] W[a][l][k, k']        (q = 0..3)
// is again a table of cubics, per ordered pair, whose edge sum is A0 itself (the reference's device code folds the same
// two factors into its table, mace_kokkos.cpp). Built once per model in float64 from the file's numbers and stored in the
// evaluator's precision and row layout. One CTA per (a, b, bin, l), thread = output channel k'.
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void fold_layer0_kernel(int E, int bins, int K, const double* __restrict__ coef /* [pairs][bins][4][K][4] */,
                                   const double* __restrict__ H0 /* [E][K] */, const double* __restrict__ W /* [E][4][K][K] */,
                                   T* __restrict__ out) {
    extern __shared__ double fold_v[];     // [K][4]: coefficients of input channel k times H0[b, k]
    const int l = blockIdx.x & 3;
    const long long rest = blockIdx.x >> 2;
    const int bin = static_cast<int>(rest % bins);
    const int ab = static_cast<int>(rest / bins);
    const int a = ab / E, b = ab % E;
    const int lo = a <= b ? a : b, hi = a <= b ? b : a;
    const int pair = lo * (2 * E - lo - 1) / 2 + hi;
    const double* in = coef + ((static_cast<size_t>(pair) * bins + bin) * 4 + l) * 4 * K;
    for (int t = threadIdx.x; t < 4 * K; t += blockDim.x) fold_v[t] = in[t] * H0[static_cast<size_t>(b) * K + (t >> 2)];
    __syncthreads();
    const double* w = W + (static_cast<size_t>(a) * 4 + l) * K * K;
    const int Kt = table_channels<T>(K);
    T* row = out + ((static_cast<size_t>(ab) * bins + bin) * 4 + l) * 4 * Kt;
    if (K < Kt) for (int q = threadIdx.x; q < 4; q += blockDim.x) row[coef_offset<T>(K, q, Kt)] = T(0);
    for (int kp = threadIdx.x; kp < K; kp += blockDim.x) {
        double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
        for (int k = 0; k < K; ++k) {
            const double wk = w[static_cast<size_t>(k) * K + kp];
            s0 += fold_v[4 * k] * wk; s1 += fold_v[4 * k + 1] * wk; s2 += fold_v[4 * k + 2] * wk; s3 += fold_v[4 * k + 3] * wk;
        }
        const double c4[4] = {s0, s1, s2, s3};
#pragma unroll
        for (int q = 0; q < 4; ++q) row[coef_offset<T>(kp, q, Kt)] = T(c4[q]);
    }
}

// =============================================================================================
// Layer 0, forward: Phi0[i, lm, k] = sum_j R0_ab(r_ij)[l, k] * Y_ij[lm] * H0[b, k]
// (first half of MACE::compute_A0, mace.cpp:159-178, with compute_Y / compute_R0 fused in).
// =============================================================================================
template <typename T>
struct Layer0Args {
    int N, K;
    const int* node_types; const long long* first_neigh; const int* neigh_indices; const int* neigh_types;
    const double* xyz; const double* r;
    const T* coef0; SplineMeta sm;
    const T* H0_w;          // [E][K]
    // Folded table (optional): per ORDERED element pair (receiver type a, sender type b) the radial coefficients already
    // multiplied by H0[b] and by the per-type channel mix W[a][l] (fold_layer0_kernel), so that the edge sum gives A0
    // directly: Phi0 / Phi0_adj then point at A0 / A0_adj and the two channel-mixing GEMMs of layer 0 are not run.
    const T* coef0_folded;
    // Optional processing order of the receivers (node ids sorted by element type). All CTAs then work on receivers of
    // one type at a time, whose edges touch only the pair tables of that type: for five elements 5 of 15 tables (73 MB of
    // 220 MB), which stay resident in the 126 MB L2 instead of being re-fetched from HBM.
    const int* order;
    T* Phi0;                // [N][16][K]          (forward output)
    const T* Phi0_adj;      // [N][16][K]          (reverse input)
    double* node_forces;    // [3 * num_edges]     (reverse: accumulated into)
    int* sched;             // work counters (see work_first)
    const int4* items;      // reverse kernel: (receiver, first edge, edges) batches
    const int* n_items;
};

// Forward edge kernels: which receiver, channel chunk and edges a CTA works on. Items are (receiver, chunk of blockDim.x
// lanes), walked with the grid's stride. SPLIT: the CTAs of a cluster share one item, each summing a contiguous part of
// the receiver's edges; the parts are added through distributed shared memory in rank order, so the result does not depend
// on timing. It is launched when there are fewer items than resident CTAs (see Evaluator::forward_split): an edge of a CTA
// that has its SM to itself takes about 0.9 us in float64, all of it latency, and a receiver of a crystal has 75 of them.
template <bool SPLIT>
struct ForwardWork {
    int rank = 0, ranks = 1;
    int first, stride;
    __device__ __forceinline__ ForwardWork() {
        if constexpr (SPLIT) {
            const auto cl = cooperative_groups::this_cluster();
            rank = static_cast<int>(cl.block_rank());
            ranks = static_cast<int>(cl.num_blocks());
        }
        first = static_cast<int>(blockIdx.x) / ranks;
        stride = static_cast<int>(gridDim.x) / ranks;
    }
    __device__ __forceinline__ void edges(long long& e_begin, long long& e_end) const {
        if constexpr (SPLIT) {
            const long long per = (e_end - e_begin + ranks - 1) / ranks;
            e_begin = e_begin + per * rank < e_end ? e_begin + per * rank : e_end;
            e_end = e_begin + per < e_end ? e_begin + per : e_end;
        }
    }
    // out(q, value) for every accumulator q: directly, or for every ranks-th q the sum over the cluster's CTAs
    template <typename V, int Q, typename F>
    __device__ __forceinline__ void finish(const V (&acc)[Q], F&& out) const {
        if constexpr (SPLIT) {
            extern __shared__ __align__(16) unsigned char forward_part_raw[];
            V* part = reinterpret_cast<V*>(forward_part_raw);
            auto cl = cooperative_groups::this_cluster();
#pragma unroll
            for (int q = 0; q < Q; ++q) part[q * blockDim.x + threadIdx.x] = acc[q];
            cl.sync();
            for (int q = rank; q < Q; q += ranks) {
                V s = cl.map_shared_rank(part, 0)[q * blockDim.x + threadIdx.x];
                for (int w = 1; w < ranks; ++w) s = s + cl.map_shared_rank(part, w)[q * blockDim.x + threadIdx.x];
                out(q, s);
            }
            cl.sync();      // nobody overwrites or leaves while its part is being read
        } else {
#pragma unroll
            for (int q = 0; q < Q; ++q) out(q, acc[q]);
        }
    }
};

template <typename T, bool SPLIT>
__global__ void __launch_bounds__(kChannelBlock) layer0_forward_kernel(const Layer0Args<T> a) {
    chain_begin();
    using V = typename Lane<T>::type;
    __shared__ EdgeStage<V, 16> st[kEdgeBatch];
    const int L = lanes_of<V>(a.K), Kt = table_channels<T>(a.K), row = 4 * Kt, F = (kLmaxSH + 1) * Kt;
    const ForwardWork<SPLIT> fw;
    const int chunks = (L + blockDim.x - 1) / blockDim.x;
    for (int w = fw.first; w < a.N * chunks; w += fw.stride) {
        const int slot = w / chunks;
        const int i = a.order ? a.order[slot] : slot;     // nodes in element-type order: see Layer0Args::order
        const int k = (w - slot * chunks) * blockDim.x + threadIdx.x;
        const bool active = k < L;
        long long e_begin = a.first_neigh[i], e_end = a.first_neigh[i + 1];
        fw.edges(e_begin, e_end);
        const int type_i = a.node_types[i];
        V acc[kNumLm];
#pragma unroll
        for (int lm = 0; lm < kNumLm; ++lm) acc[lm] = V(0.0);
        for (long long e0 = e_begin; e0 < e_end; e0 += kEdgeBatch) {
            const int nb = static_cast<int>(e_end - e0 < kEdgeBatch ? e_end - e0 : kEdgeBatch);
            __syncthreads();
            if (threadIdx.x < nb)
                stage_edge<V, false>(st[threadIdx.x], e0 + threadIdx.x, type_i, a.neigh_indices, a.neigh_types, a.xyz, a.r, a.sm, F);
            __syncthreads();
            if (active) {
                for (int e = 0; e < nb; ++e) {
                    const EdgeStage<V, 16>& s = st[e];
                    const V h0 = a.coef0_folded ? V(1.0) : lane_load<V, false>(a.H0_w + s.tj * a.K, k, a.K);
                    const V x = V(s.x);
                    const T* cb = a.coef0_folded ? a.coef0_folded : a.coef0;
                    const unsigned cr = a.coef0_folded ? s.row.coef_row_dir : s.row.coef_row;
                    V Y[kNumLm];
                    load_harmonics(s, Y);
#pragma unroll
                    for (int l = 0; l <= kLmaxSH; ++l) {
                        V R = cubic_value(load_coef<V>(cb + l * row, cr + k, L), x);
                        if (!a.coef0_folded) R = R * h0;
#pragma unroll
                        for (int lm = l * l; lm < (l + 1) * (l + 1); ++lm) acc[lm] = fma(R, Y[lm], acc[lm]);
                    }
                }
            }
        }
        T* out = a.Phi0 + (static_cast<size_t>(i) * kNumLm) * a.K;
        fw.template finish<V, kNumLm>(acc, [&](int lm, V v) { if (active) lane_store<false, false>(out + static_cast<size_t>(lm) * a.K, k, a.K, v); });
    }
}

// =============================================================================================
// Layer 0, reverse: per-edge partial forces
//   nf[ij] -= sum_{lm,k} Phi0_adj[i,lm,k] H0[b,k] (xhat R0'[l,k] Y[lm] + R0[l,k] grad Y[lm])
// (second half of MACE::reverse_A0, mace.cpp:238-269).
// =============================================================================================
// CPT lanes per thread (k, k + blockDim.x, ...): the per-edge sums over channels (15 harmonic adjoints + 1 radial
// adjoint, reduced across the warp with shuffles and across warps through shared memory) are what this kernel spends
// most of its instructions on, and a thread that adds up CPT lanes before the reduction needs 1 / CPT of them.
template <typename T, int CPT, bool WHOLE>
__global__ void __launch_bounds__(kChannelBlock) layer0_reverse_kernel(const Layer0Args<T> a) {
    chain_begin();
    using V = typename Lane<T>::type;
    __shared__ EdgeStage<V, 16> st[kEdgeBatch];
    __shared__ T red[kMaxWarps][kEdgeBatch][17];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int L = lanes_of<V>(a.K), Kt = table_channels<T>(a.K), row = 4 * Kt, F = (kLmaxSH + 1) * Kt;
    __shared__ int s_next[2];
    int par = 0;
    const int n_items = *a.n_items;
    for (int item = work_first(a.sched, s_next); item < n_items; item = work_next(s_next, par))
    for (int kc = 0; kc < L; kc += CPT * blockDim.x) {
        if (kc == 0) work_prefetch(a.sched, s_next, par);     // ask for the next item while this one is computed
        const int4 it = a.items[item];                    // one batch of one receiver's edges, receivers in element-type order
        const int i = it.x;
        int kk[CPT];
        bool active[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) { kk[c] = kc + c * blockDim.x + threadIdx.x; active[c] = kk[c] < L; }
        const long long e_begin = a.first_neigh[i] + it.y, e_end = e_begin + it.z;
        const int type_i = a.node_types[i];
        V d[CPT][kNumLm];
#pragma unroll
        for (int c = 0; c < CPT; ++c)
#pragma unroll
            for (int lm = 0; lm < kNumLm; ++lm)
                d[c][lm] = active[c] ? lane_load<V, WHOLE>(a.Phi0_adj + (static_cast<size_t>(i) * kNumLm + lm) * a.K, kk[c], a.K) : V(0.0);
        for (long long e0 = e_begin; e0 < e_end; e0 += kEdgeBatch) {
            const int nb = static_cast<int>(e_end - e0 < kEdgeBatch ? e_end - e0 : kEdgeBatch);
            __syncthreads();
            if (threadIdx.x < nb)
                stage_edge<V, true>(st[threadIdx.x], e0 + threadIdx.x, type_i, a.neigh_indices, a.neigh_types, a.xyz, a.r, a.sm, F);
            __syncthreads();
            for (int e = 0; e < nb; ++e) {
                const EdgeStage<V, 16>& s = st[e];
                V Wl[kNumLm];      // adjoints of the edge length (Wl[0]) and of the harmonics, summed over this thread's lanes
#pragma unroll
                for (int lm = 0; lm < kNumLm; ++lm) Wl[lm] = V(0.0);
                const V x = V(s.x), x2 = x * V(2.0), x15 = x * V(1.5);
                const T* cb = a.coef0_folded ? a.coef0_folded : a.coef0;
                const unsigned cr = a.coef0_folded ? s.row.coef_row_dir : s.row.coef_row;
                V Y[kNumLm];
                load_harmonics(s, Y);
#pragma unroll
                for (int c = 0; c < CPT; ++c) {
                    if (!active[c]) continue;
                    V h0 = V(1.0);
                    if (!a.coef0_folded) h0 = lane_load<V, WHOLE>(a.H0_w + s.tj * a.K, kk[c], a.K);
#pragma unroll
                    for (int l = 0; l <= kLmaxSH; ++l) {
                        const Coef<V> cf = load_coef<V>(cb + l * row, cr + kk[c], L);
                        V R = cubic_value(cf, x), Rd = cubic_slope(cf, x2, x15);
                        if (!a.coef0_folded) { R = R * h0; Rd = Rd * h0; }
                        V sv = l == 0 ? d[c][0] : d[c][l * l] * Y[l * l];
                        if (l > 0) Wl[l * l] = fma(R, d[c][l * l], Wl[l * l]);
#pragma unroll
                        for (int lm = l * l + 1; lm < (l + 1) * (l + 1); ++lm) {
                            sv = fma(d[c][lm], Y[lm], sv);
                            Wl[lm] = fma(R, d[c][lm], Wl[lm]);
                        }
                        Wl[0] = fma(Rd, sv, Wl[0]);
                    }
                }
                warp_edge_sums(Wl, lane, static_cast<SumScratch<void>*>(nullptr), red[warp][e]);
            }
            __syncthreads();
            if (threadIdx.x < nb) {
                const int e = threadIdx.x;
                finish_edge_force<T, kEdgeBatch>(red, 0, nwarps, e, st[e].dY[0], st[e].dY[1], st[e].dY[2], st[e].ux, st[e].uy, st[e].uz,
                                                 a.node_forces + 3 * (e0 + e));
            }
        }
    }
    work_leave(a.sched);
}

// =============================================================================================
// Layer 1 tensor product. Per (edge, channel):
//     Phi1[i, (l m e_p), k] += R1_p(r_ij)[k] * sum_{m1 m2} C^{l m}_{l1 m1, l2 m2} Y_ij[l1 m1] H1[j, (l2 m2), k]
// which is the reference's two-step form (Phi1r, then the Clebsch-Gordan COO contraction,
// mace.cpp:453-502) with the sums merged; Phi1r is never formed. The non-zeros of the coupling are
// written out as straight-line code (generated/tp_L*_forward.inc), so the accumulators stay in
// registers and the coupling constants are immediates; the only shared-memory traffic per edge is
// the 16 harmonics. Any per-path scale of a model file's coupling table is folded into R1_p at load.
// =============================================================================================
template <typename T>
struct TPArgs {
    int N, K;
    const int* node_types; const long long* first_neigh; const int* neigh_indices; const int* neigh_types;
    const double* xyz; const double* r;
    const T* coef1; SplineMeta sm;
    const T* coef1_single;  // the same table for single-float lanes (float: reverse pass of odd and of narrow rows up to L_max = 1, forward
                            // pass at L_max = 2; see Evaluator::may_use_single_floats)
    const T* H;             // sender features [rows][nLM][K]
    T* Phi1;                // forward output [N][Q][K]
    const T* dPhi1;         // reverse input  [N][Q][K]
    T* Hmsg;                // reverse output [num_edges][nLM][K]: adjoint message of each edge to its sender (float64)
    T* H_adj;               // float32: the messages are added straight into H_adj[sender] with red.global.add
    double* node_forces;    // reverse: accumulated into
    int* status;            // set non-zero by a bounded wait that ran out (staged reverse kernel)
    const int* order;       // optional processing order of the receivers (see Layer0Args::order)
    // Run-time radial mode: the radial functions of every edge (and their derivatives, reverse pass) evaluated from the
    // un-splined network by radial_hidden_kernel + a tensor-core GEMM, [num_edges][P * K]; null: cubic splines (coef1).
    const T* R_edge;
    const T* Rd_edge;
    int* sched;             // work counters (see work_first)
    const int4* items;      // reverse kernels: (receiver, first edge, edges) batches
    const int* n_items;
};

// Resident CTAs (of 128 threads) per SM the compiler is asked to allow for in the forward pass, i.e. the register budget: 3 up to
// L_max = 1 (168 registers, no spills; pairs of floats with 5, i.e. 96 registers, spill 230 bytes), 1 beyond. Single floats, which
// L_max = 2 uses where there is work for all SMs (see launch_tp): 4, i.e. 128 registers (2,664 atoms, 48 edges each, K = 256: 1,017 us;
// with 3 1,335, with 2 1,264). Pairs have 255 registers for 71 accumulators (2,916 atoms, 78 edges each, K = 256: 1,444 us, single
// floats 1,313).
template <typename V> constexpr int tp_min_blocks(int LF) { return sizeof(V) == 4 ? 4 : (LF >= 2 ? 1 : 3); }

template <typename V, int LF, bool SPLIT, bool WHOLE>
__global__ void __launch_bounds__(kChannelBlock, tp_min_blocks<V>(LF)) tp_forward_kernel(const TPArgs<typename LaneScalar<V>::type> a) {
    chain_begin();
    using T = typename LaneScalar<V>::type;
    constexpr TPTable tp = make_tp_table(LF);
    constexpr TPScale<LF> scale{};
    __shared__ EdgeStage<V> st[kEdgeBatch];
    const int L = lanes_of<V>(a.K), Kt = sizeof(V) == 4 ? a.K : table_channels<T>(a.K), row = 4 * Kt, F = tp.P * Kt;
    const ForwardWork<SPLIT> fw;
    const int chunks = (L + blockDim.x - 1) / blockDim.x;
    for (int w = fw.first; w < a.N * chunks; w += fw.stride) {
        const int slot = w / chunks;
        const int i = a.order ? a.order[slot] : slot;     // nodes in element-type order: see Layer0Args::order
        const int k = (w - slot * chunks) * blockDim.x + threadIdx.x;
        const bool active = k < L;
        long long e_begin = a.first_neigh[i], e_end = a.first_neigh[i + 1];
        fw.edges(e_begin, e_end);
        const int type_i = a.node_types[i];
        V acc[tp.Q];
#pragma unroll
        for (int q = 0; q < tp.Q; ++q) acc[q] = V(0.0);
        for (long long e0 = e_begin; e0 < e_end; e0 += kEdgeBatch) {
            const int nb = static_cast<int>(e_end - e0 < kEdgeBatch ? e_end - e0 : kEdgeBatch);
            __syncthreads();
            if (threadIdx.x < nb)
                stage_edge<V, false>(st[threadIdx.x], e0 + threadIdx.x, type_i, a.neigh_indices, a.neigh_types, a.xyz, a.r, a.sm, F);
            __syncthreads();
            if (active) {
                for (int e = 0; e < nb; ++e) {
                    const EdgeStage<V>& s = st[e];
                    const V x = V(s.x);
                    const T* cb = (sizeof(V) == 4 ? a.coef1_single : a.coef1) + s.row.coef_base;
                    const T* hrow = a.H + static_cast<size_t>(s.j) * tp.nLM * a.K;
                    V h[tp.nLM], R[tp.P], Y[kNumLm];
#pragma unroll
                    for (int lm2 = 0; lm2 < tp.nLM; ++lm2) h[lm2] = lane_load<V, WHOLE, Cache::kReadOnly>(hrow + static_cast<size_t>(lm2) * a.K, k, a.K);
                    if (a.R_edge) {
                        const T* re = a.R_edge + static_cast<size_t>(e0 + e) * tp.P * a.K;
#pragma unroll
                        for (int p = 0; p < tp.P; ++p) R[p] = lane_load<V, WHOLE, Cache::kStream>(re + static_cast<size_t>(p) * a.K, k, a.K);
                    } else {
#pragma unroll
                        for (int p = 0; p < tp.P; ++p) R[p] = cubic_value(load_coef<V>(cb + p * row, k, L), x);
                    }
                    load_harmonics(s, Y);
                    {
                        using T = V;      // the generated code's name for what it computes on
                        if constexpr (LF == 0) {
#include "generated/tp_L0_forward.inc"
                        } else if constexpr (LF == 1) {
#include "generated/tp_L1_forward.inc"
                        } else if constexpr (LF == 2) {
#include "generated/tp_L2_forward.inc"
                        } else {
#include "generated/tp_L3_forward.inc"
                        }
                    }
                }
            }
        }
        T* out = a.Phi1 + static_cast<size_t>(i) * tp.Q * a.K;
#pragma unroll
        for (int q = 0; q < tp.Q; ++q) acc[q] = V(scale.q[q]) * acc[q];
        // written once, read by the GEMM: stream past L2 residents
        fw.template finish<V, tp.Q>(acc, [&](int q, V v) { if (active) lane_store<true, WHOLE>(out + static_cast<size_t>(q) * a.K, k, a.K, v); });
    }
}

// Reverse of the tensor product (MACE::reverse_Phi1, mace.cpp:504-605) for one receiver per CTA.
// Per (edge, channel) the generated code (generated/tp_L*_reverse.inc) produces the three adjoints of
// the trilinear form: msg = dE/dH1_j (written to Hmsg, summed per sender afterwards), W[lm > 0] = dE/dY_ij and
// W[0] = dE/dr_ij. W is summed over channels (warp_edge_sums, then across warps in shared
// memory) and one thread per edge turns it into the partial force
//   nf[ij] -= xhat * W[0] + sum_lm W[lm] * grad Y[lm].
//
// STAGED = true: the spline row of every edge (4*P*K values, 40 KB in float64 for K = 128, L_max = 1) is brought
// into shared memory by one bulk asynchronous copy (TMA) that a single thread starts one edge ahead of its use,
// through two slots guarded by a full/empty mbarrier pair each, so the coefficient reads are shared-memory loads
// instead of global loads that only 8 resident warps per SM would have to cover. A bounded wait that runs out
// sets *status, stops further copies and waits, and the kernel finishes (with results the host discards).
// The adjoint message of an edge to its sender. float64: deterministic two-step scatter (per-edge message, then a fixed-order sum
// per sender by sender_gather_kernel); the stores stream, because the buffer is written once and read once and must not push
// the spline tables out of L2. float32: reductions directly into the sender's row (no message buffer).
template <int NLM, bool WHOLE, typename T, typename V>
__device__ __forceinline__ void tp_reverse_message(const TPArgs<T>& a, long long edge, int j, int k, const V (&msg)[NLM]) {
    if constexpr (sizeof(T) == 8) {
        T* mrow = a.Hmsg + static_cast<size_t>(edge) * NLM * a.K;
        static_for<NLM>([&](auto q) { lane_store<true, WHOLE>(mrow + static_cast<size_t>(q) * a.K, k, a.K, msg[q]); });
    } else {
        T* arow = a.H_adj + static_cast<size_t>(j) * NLM * a.K;
        static_for<NLM>([&](auto q) { lane_atomic_add<WHOLE>(arow + static_cast<size_t>(q) * a.K, k, a.K, msg[q]); });
    }
}
template <bool STAGED> constexpr int tp_reverse_batch() { return STAGED ? 24 : kEdgeBatch; }

template <typename V, int LF, bool STAGED, bool WHOLE, bool SHARED>
__global__ void __launch_bounds__(kChannelBlock, sizeof(V) == 4 ? 4 : 1) tp_reverse_kernel(const TPArgs<typename LaneScalar<V>::type> a) {
    chain_begin();
    using T = typename LaneScalar<V>::type;
    static_assert(!STAGED || sizeof(T) == 8, "row staging is a float64 variant");
    constexpr TPTable tp = make_tp_table(LF);
    constexpr TPScale<LF> scale{};
    constexpr int EB = tp_reverse_batch<STAGED>();
    __shared__ EdgeStage<V> st[EB];
    __shared__ T red[kMaxWarps][EB][17];
    __shared__ SumScratch<std::conditional_t<SHARED, T, void>> scratch[kMaxWarps];
    __shared__ __align__(8) unsigned long long full_bar[2], empty_bar[2];
    __shared__ int failed;
    extern __shared__ __align__(128) unsigned char tp_dyn_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int L = lanes_of<V>(a.K), Kt = sizeof(V) == 4 ? a.K : table_channels<T>(a.K), row = 4 * Kt, F = tp.P * Kt;
    unsigned full_par = 0, empty_par = 0;     // bit s: parity of the phase slot s is in
    if constexpr (STAGED) {
        if (threadIdx.x == 0) {
            failed = 0;
            mbar_init(&full_bar[0], 1); mbar_init(&full_bar[1], 1);
            mbar_init(&empty_bar[0], blockDim.x); mbar_init(&empty_bar[1], blockDim.x);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
    }
    // Work items: the row-staging variant walks whole receivers (static split; its copies run ahead inside a receiver's
    // edge list), the plain variant takes (receiver, batch) items from the work counter.
    __shared__ int s_next[2];
    int par = 0;
    const int n_work = STAGED ? a.N : *a.n_items;
    for (int w = STAGED ? static_cast<int>(blockIdx.x) : work_first(a.sched, s_next); w < n_work;
         w = STAGED ? w + static_cast<int>(gridDim.x) : work_next(s_next, par))
    for (int kc = 0; kc < L; kc += blockDim.x) {
        if constexpr (!STAGED) { if (kc == 0) work_prefetch(a.sched, s_next, par); }     // ask for the next item while this one is computed
        int i;
        long long e_begin, e_end;
        if constexpr (STAGED) {
            i = a.order ? a.order[w] : w;                 // nodes in element-type order: see Layer0Args::order
            e_begin = a.first_neigh[i]; e_end = a.first_neigh[i + 1];
        } else {
            const int4 it = a.items[w];
            i = it.x;
            e_begin = a.first_neigh[i] + it.y; e_end = e_begin + it.z;
        }
        const int k = kc + threadIdx.x;
        const bool active = k < L;
        const int Kc = L - kc < static_cast<int>(blockDim.x) ? L - kc : static_cast<int>(blockDim.x);      // STAGED only (lane = channel)
        T* const slot0 = reinterpret_cast<T*>(tp_dyn_smem);
        T* const slot1 = slot0 + 4 * tp.P * Kc;
        const int type_i = a.node_types[i];
        V d[tp.Q];
#pragma unroll
        for (int q = 0; q < tp.Q; ++q)
            d[q] = active ? V(scale.q[q]) * lane_load<V, WHOLE, Cache::kStream>(a.dPhi1 + (static_cast<size_t>(i) * tp.Q + q) * a.K, k, a.K) : V(0.0);
        for (long long e0 = e_begin; e0 < e_end; e0 += EB) {
            const int nb = static_cast<int>(e_end - e0 < EB ? e_end - e0 : EB);
            __syncthreads();
            if (threadIdx.x < nb)
                stage_edge<V, true>(st[threadIdx.x], e0 + threadIdx.x, type_i, a.neigh_indices, a.neigh_types, a.xyz, a.r, a.sm, F);
            __syncthreads();
            if constexpr (STAGED) {
                if (threadIdx.x == 0 && !failed) {
                    issue_row_copy(slot0, a.coef1 + st[0].row.coef_base, tp.P, a.K, kc, Kc, &full_bar[0]);
                    if (nb > 1) issue_row_copy(slot1, a.coef1 + st[1].row.coef_base, tp.P, a.K, kc, Kc, &full_bar[1]);
                }
            }
            for (int e = 0; e < nb; ++e) {
                const EdgeStage<V>& s = st[e];
                V W[kNumLm];      // assigned by the generated code (first contribution of each entry), zero for idle lanes
                const int sl = e & 1;
                V R[tp.P], Rd[tp.P];
                const V x = V(s.x), x2 = x * V(2.0), x15 = x * V(1.5);
                if constexpr (STAGED) {
                    if (!*reinterpret_cast<volatile int*>(&failed)) {
                        if (!mbar_wait(&full_bar[sl], (full_par >> sl) & 1u)) { failed = 1; atomicMax(a.status, 3); }
                    }
                    full_par ^= 1u << sl;
                    const T* slot = sl ? slot1 : slot0;
                    if (active) {
#pragma unroll
                        for (int p = 0; p < tp.P; ++p) {
                            const Coef<V> c = lds_coef(slot, p, threadIdx.x, Kc);
                            R[p] = cubic_value(c, x);
                            Rd[p] = cubic_slope(c, x2, x15);
                        }
                    }
                    mbar_arrive(&empty_bar[sl]);                 // this thread has read its part of the slot
                    if (threadIdx.x == 0) {
                        if (e + 2 < nb && !failed) {
                            if (!mbar_wait(&empty_bar[sl], (empty_par >> sl) & 1u)) { failed = 1; atomicMax(a.status, 4); }
                            else issue_row_copy(sl ? slot1 : slot0, a.coef1 + st[e + 2].row.coef_base, tp.P, a.K, kc, Kc, &full_bar[sl]);
                        }
                    }
                    empty_par ^= 1u << sl;
                }
                if (active) {
                    const T* hrow = a.H + static_cast<size_t>(s.j) * tp.nLM * a.K;
                    V h[tp.nLM], msg[tp.nLM], Y[kNumLm];
#pragma unroll
                    for (int lm2 = 0; lm2 < tp.nLM; ++lm2) h[lm2] = lane_load<V, WHOLE, Cache::kReadOnly>(hrow + static_cast<size_t>(lm2) * a.K, k, a.K);
                    if constexpr (!STAGED) {
                        if (sizeof(T) == 4 && a.R_edge) {
                            const T* re = a.R_edge + static_cast<size_t>(e0 + e) * tp.P * a.K;
                            const T* rde = a.Rd_edge + static_cast<size_t>(e0 + e) * tp.P * a.K;
#pragma unroll
                            for (int p = 0; p < tp.P; ++p) {
                                R[p] = lane_load<V, WHOLE, Cache::kStream>(re + static_cast<size_t>(p) * a.K, k, a.K);
                                Rd[p] = lane_load<V, WHOLE, Cache::kStream>(rde + static_cast<size_t>(p) * a.K, k, a.K);
                            }
                        } else {
                            const T* cb = (sizeof(V) == 4 ? a.coef1_single : a.coef1) + s.row.coef_base;
#pragma unroll
                            for (int p = 0; p < tp.P; ++p) {
                                const Coef<V> c = load_coef<V>(cb + p * row, k, L);
                                R[p] = cubic_value(c, x);
                                Rd[p] = cubic_slope(c, x2, x15);
                            }
                        }
                    }
                    load_harmonics(s, Y);
                    {
                        using T = V;      // the generated code's name for what it computes on
                        if constexpr (LF == 0) {
#include "generated/tp_L0_reverse.inc"
                        } else if constexpr (LF == 1) {
#include "generated/tp_L1_reverse.inc"
                        } else if constexpr (LF == 2) {
#include "generated/tp_L2_reverse.inc"
                        } else {
#include "generated/tp_L3_reverse.inc"
                        }
                    }
                    tp_reverse_message<tp.nLM, WHOLE>(a, e0 + e, s.j, k, msg);
                } else {
#pragma unroll
                    for (int lm = 0; lm < kNumLm; ++lm) W[lm] = V(0.0);
                }
                warp_edge_sums(W, lane, &scratch[warp], red[warp][e]);
            }
            __syncthreads();
            if (threadIdx.x < nb) {
                const int e = threadIdx.x;
                finish_edge_force<T, EB>(red, 0, nwarps, e, st[e].dY[0], st[e].dY[1], st[e].dY[2], st[e].ux, st[e].uy, st[e].uz,
                                         a.node_forces + 3 * (e0 + e));
            }
        }
    }
    if constexpr (!STAGED) work_leave(a.sched);
    if constexpr (STAGED) {
        // after a failed wait: give copies that may still be in flight one more bounded wait before the CTA exits
        __syncthreads();
        if (threadIdx.x == 0 && failed) {
            mbar_wait(&full_bar[0], (full_par & 1u) ^ 1u);
            mbar_wait(&full_bar[1], ((full_par >> 1) & 1u) ^ 1u);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Reverse of the tensor product with the receiver's adjoint in tensor memory.
//
// tp_reverse_kernel keeps d[Q] (the adjoint of the receiver's tensor product, 2 registers per value: 80 registers
// for Q = 40) in registers for the whole walk over the receiver's edges; with the 16 harmonic adjoints, the messages, the
// radial values and the coupling temporaries that is 254 registers, i.e. two resident CTAs (8 warps) per SM, too few to
// cover the latency of the coefficient loads that start every edge. Blackwell's tensor memory (TMEM, 512 columns x 128
// lanes x 32 bits per SM, normally the accumulator of tcgen05.mma) is used here as a per-thread scratchpad instead: thread
// t of the CTA owns TMEM lane t and keeps its d values there (tcgen05.st once per receiver), fetching the 2l+1 values of
// one path at a time (tcgen05.ld) while it works on the previous path. TMEM has its own data path, so this costs neither
// registers nor shared-memory / L1 bandwidth, which the coefficient stream needs. The register budget then allows three
// resident CTAs per SM.
//
// Column layout (per lane): path p starts at tp_tmem_col(p), aligned to its padded width (2, 8, 16 or 16 columns for
// l = 0, 1, 2, 3; a value takes two 32-bit columns). A CTA allocates the next power of two >= the total; the host
// checks that the resident CTAs of one SM fit into the 512 columns.
//
// A CTA always has 128 threads, since a warp reaches only the 32 TMEM lanes of its quadrant: where a row has 64 or 32 lanes
// (K = 128 in float, 64 in double, ...) two or four groups of threads share the receiver and take its edges in turn.
// ---------------------------------------------------------------------------------------------
constexpr int tp_tmem_width(int l) { return l == 0 ? 2 : (l == 1 ? 8 : 16); }
constexpr int tp_tmem_col(const TPTable& tp, int p) {
    int col = 0;
    for (int q = 0; q < p; ++q) {
        const int w = tp_tmem_width(tp.l[q]);
        col = (col + w - 1) / w * w + w;
    }
    const int w = tp_tmem_width(tp.l[p]);
    return (col + w - 1) / w * w;
}
constexpr int tp_tmem_cols(int LF) {
    const TPTable tp = make_tp_table(LF);
    const int used = tp_tmem_col(tp, tp.P - 1) + tp_tmem_width(tp.l[tp.P - 1]);
    int alloc = 32;
    while (alloc < used) alloc *= 2;
    return alloc;
}

// Starts the asynchronous fetch of W 32-bit columns of this thread's TMEM lane into `v` (W = 2, 8 or 16).
template <int W>
__device__ __forceinline__ void tmem_ld_issue(uint32_t taddr, uint32_t (&v)[16]) {
    if constexpr (W == 2) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(taddr) : "memory");
    } else if constexpr (W == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr) : "memory");
    } else {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                       "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(taddr) : "memory");
    }
}
// Waits for the fetches this thread started; the registers are operands so that no use of them moves above the wait.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                   "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]) :: "memory");
}
template <typename V>
__device__ __forceinline__ void tmem_st2(uint32_t taddr, V x) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(lane_lo(x)), "r"(lane_hi(x)) : "memory");
}

template <typename T, int LF, int MINB, bool WHOLE>
__global__ void __launch_bounds__(kChannelBlock, MINB) tp_reverse_tmem_kernel(const TPArgs<T> a) {
    chain_begin();
    using V = typename Lane<T>::type;
    constexpr TPTable tp = make_tp_table(LF);
    constexpr TPScale<LF> scale{};
    constexpr int kAlign = sizeof(T) == 8 ? 16 : 8;      // see EdgeStage
    constexpr int EB = kEdgeBatch;
    constexpr int kCols = tp_tmem_cols(LF);
    __shared__ EdgeStage<V, kAlign> st[EB];
    __shared__ T red[kMaxWarps][EB][17];
    __shared__ SumScratch<T> scratch[kMaxWarps];
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int L = lanes_of<V>(a.K), Kt = table_channels<T>(a.K), row = 4 * Kt, F = tp.P * Kt;
    const int gthreads = L <= 32 ? 32 : (L <= 64 ? 64 : 128);      // threads of a group
    const int groups = kChannelBlock / gthreads, group = threadIdx.x / gthreads, gwarps = gthreads / 32;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // this thread's lane: 32 * (warp % 4) + lane, in bits 16.. of the address (a warp reaches the 32 lanes of its quadrant)
    const uint32_t tbase = tmem_slot + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    // two sets of staging registers, used by the paths of even and odd index: the set a path has just consumed is dead
    // until the path after the next one refills it, so its registers can become the path's double-precision values in place
    uint32_t stage0[16], stage1[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) { stage0[q] = 0u; stage1[q] = 0u; }

    __shared__ int s_next[2];
    int par = 0;
    const int n_items = *a.n_items;
    for (int item = work_first(a.sched, s_next); item < n_items; item = work_next(s_next, par))
    for (int kc = 0; kc < L; kc += gthreads) {
        if (kc == 0) work_prefetch(a.sched, s_next, par);     // ask for the next item while this one is computed
        const int4 it = a.items[item];                    // one batch of one receiver's edges, receivers in element-type order
        const int i = it.x;
        const int kt = kc + static_cast<int>(threadIdx.x) % gthreads;
        const bool active = kt < L;
        const int k = active ? kt : L - 1;                // idle threads shadow the last lane with a zero adjoint: the
                                                          // tensor-memory instructions need the whole warp
        const long long e_begin = a.first_neigh[i] + it.y, e_end = e_begin + it.z;
        const int type_i = a.node_types[i];
        // the receiver's adjoint into this thread's TMEM lane, path by path
        static_for<tp.P>([&](auto pc) {
            constexpr int p = decltype(pc)::value;
            static_for<2 * tp.l[p] + 1>([&](auto mc) {
                constexpr int m = decltype(mc)::value, q = tp.lme(p, m);
                constexpr double factor = scale.q[q];
                const V v = active ? V(factor) * lane_load<V, WHOLE, Cache::kStream>(a.dPhi1 + (static_cast<size_t>(i) * tp.Q + q) * a.K, k, a.K) : V(0.0);
                tmem_st2(tbase + tp_tmem_col(tp, p) + 2 * m, v);
            });
        });
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tmem_ld_issue<tp_tmem_width(tp.l[0])>(tbase + tp_tmem_col(tp, 0), stage0);     // path 0 of the first edge
        for (long long e0 = e_begin; e0 < e_end; e0 += EB) {
            const int nb = static_cast<int>(e_end - e0 < EB ? e_end - e0 : EB);
            __syncthreads();
            if (threadIdx.x < nb)
                stage_edge<V, true>(st[threadIdx.x], e0 + threadIdx.x, type_i, a.neigh_indices, a.neigh_types, a.xyz, a.r, a.sm, F);
            __syncthreads();
            for (int e = group; e < nb; e += groups) {
                const EdgeStage<V, kAlign>& s = st[e];
                V W[kNumLm];      // assigned by the generated code (first contribution of each entry)
                V R[tp.P], Rd[tp.P];
                const V x = V(s.x), x2 = x * V(2.0), x15 = x * V(1.5);
                V h[tp.nLM], msg[tp.nLM], Y[kNumLm];
                const T* hrow = a.H + static_cast<size_t>(s.j) * tp.nLM * a.K;
                static_for<tp.nLM>([&](auto q) { h[q] = lane_load<V, WHOLE, Cache::kReadOnly>(hrow + static_cast<size_t>(q) * a.K, k, a.K); });
                const T* cb = a.coef1;
                unsigned cr = k;
                if constexpr (kAlign == 16) cr += s.row.coef_row; else cb += s.row.coef_base;
                static_for<tp.P>([&](auto p) {
                    const Coef<V> c = load_coef<V>(cb + p * row, cr, L);
                    R[p] = cubic_value(c, x);
                    Rd[p] = cubic_slope(c, x2, x15);
                });
                load_harmonics(s, Y);
                // Path p's adjoint values arrive in `stage` (fetch started while path p - 1 was computed); they are moved
                // into dp and the fetch of the next path (path 0 again after the last: the adjoint belongs to the receiver,
                // not to the edge) starts before path p is computed.
#define TP_PATH_D(p, n, dp)                                                                                   \
                {                                                                                             \
                    uint32_t (&cur_)[16] = ((p) & 1) ? stage1 : stage0;                                       \
                    uint32_t (&nxt_)[16] = ((((p) + 1) % tp.P) & 1) ? stage1 : stage0;                        \
                    tmem_ld_wait(cur_);                                                                       \
                    static_for<(n)>([&](auto m_) { dp[m_] = lane_from_bits<V>(cur_[2 * m_], cur_[2 * m_ + 1]); }); \
                    tmem_ld_issue<tp_tmem_width(tp.l[((p) + 1) % tp.P])>(tbase + tp_tmem_col(tp, ((p) + 1) % tp.P), nxt_); \
                }
                {
                    using T = V;      // the generated code's name for what it computes on
                    if constexpr (LF == 0) {
#include "generated/tp_L0_reverse_bypath.inc"
                    } else if constexpr (LF == 1) {
#include "generated/tp_L1_reverse_bypath.inc"
                    } else if constexpr (LF == 2) {
#include "generated/tp_L2_reverse_bypath.inc"
                    } else {
#include "generated/tp_L3_reverse_bypath.inc"
                    }
                }
#undef TP_PATH_D
                if (active) tp_reverse_message<tp.nLM, WHOLE>(a, e0 + e, s.j, k, msg);
                warp_edge_sums(W, lane, &scratch[warp], red[warp][e]);
            }
            __syncthreads();
            if (threadIdx.x < nb) {
                const int e = threadIdx.x;
                finish_edge_force<T, EB>(red, e % groups * gwarps, gwarps, e, st[e].dY[0], st[e].dY[1], st[e].dY[2], st[e].ux, st[e].uy, st[e].uz,
                                         a.node_forces + 3 * (e0 + e));
            }
        }
        tmem_ld_wait(stage0);     // the fetch started after the last path of the last edge: nothing may be in flight when d is rewritten
    }
    work_leave(a.sched);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot), "r"(kCols) : "memory");
}

// ---------------------------------------------------------------------------------------------
// Run-time radial mode, first part: the hidden activations of the radial network and their derivatives with respect
// to the edge length, per edge. The network is what the reference's exporter tabulates into its cubic splines
// (symmetrix/source/symmetrix/extract_mace_data.py:144-172):
//   f_n(r) = sqrt(2 / r_cut) sin(n pi r / r_cut) / r * cutoff_p(r / r_cut) * pair_scale[pair][n]
//   x <- s silu(x W) per hidden layer (s = silu_scale),  dx/dr by the chain rule alongside.
// The last layer (hidden -> P K values per edge) is a dense GEMM over all edges and runs on the tensor cores
// (gemm_rows_tcgen05_kernel). One group of `hidden` threads per edge, four groups per CTA; the weights sit in shared
// memory, thread j of a group owns neuron j.
// ---------------------------------------------------------------------------------------------
struct RadialNetArgs {
    int N, num_bessel, poly_p, hidden, num_hidden_layers, num_elements;
    float r_cut, silu_scale;
    const int* node_types; const long long* first_neigh; const int* neigh_types; const double* r;
    const float* w_first;      // [num_bessel][hidden]
    const float* w_hidden;     // [num_hidden_layers - 1][hidden][hidden]
    const float* pair_scale;   // [pairs][num_bessel]
    float* x_out;              // [num_edges][hidden]
    float* dx_out;             // [num_edges][hidden]
};
constexpr int kRadialGroups = 4;

static __global__ void __launch_bounds__(kRadialGroups * 64) radial_hidden_kernel(const RadialNetArgs a) {
    extern __shared__ float radial_smem[];
    const int H = a.hidden;
    float* w1 = radial_smem;                                        // [num_bessel][H]
    float* wh = w1 + a.num_bessel * H;                              // [(layers - 1)][H][H]
    float* act = wh + (a.num_hidden_layers - 1) * H * H;            // [groups][2 buffers][2 (x, dx)][64]
    for (int t = threadIdx.x; t < a.num_bessel * H; t += blockDim.x) w1[t] = a.w_first[t];
    for (int t = threadIdx.x; t < (a.num_hidden_layers - 1) * H * H; t += blockDim.x) wh[t] = a.w_hidden[t];
    __syncthreads();
    const int group = threadIdx.x / 64, j = threadIdx.x % 64;
    float* mine = act + group * 4 * 64;
    const double pi = 3.14159265358979323846;
    for (int i = blockIdx.x; i < a.N; i += gridDim.x) {
        const int type_i = a.node_types[i];
        const long long e_begin = a.first_neigh[i], e_end = a.first_neigh[i + 1];
        const long long rounds = (e_end - e_begin + kRadialGroups - 1) / kRadialGroups;
        for (long long rd = 0; rd < rounds; ++rd) {
            const long long e = e_begin + rd * kRadialGroups + group;
            const bool live = e < e_end;
            if (live && j < a.num_bessel) {
                const double rr = a.r[e], rc = a.r_cut;
                const int tj = a.neigh_types[e];
                const int lo = type_i <= tj ? type_i : tj, hi = type_i <= tj ? tj : type_i;
                const int pair = lo * (2 * a.num_elements - lo - 1) / 2 + hi;
                const double kn = (j + 1) * pi / rc, amp = sqrt(2.0 / rc);
                double sn, cs;
                sincos(kn * rr, &sn, &cs);
                const double b = amp * sn / rr, db = amp * (kn * cs / rr - sn / (rr * rr));
                const double x = rr / rc, p = a.poly_p;
                double c = 0.0, dc = 0.0;
                if (x < 1.0) {
                    double xp1 = 1.0;                              // x^(p - 1) by repeated multiplication (p is a small integer)
                    for (int q = 1; q < a.poly_p; ++q) xp1 *= x;
                    const double xp = xp1 * x, xq = xp * x, xr = xq * x;
                    c = 1.0 - (p + 1.0) * (p + 2.0) / 2.0 * xp + p * (p + 2.0) * xq - p * (p + 1.0) / 2.0 * xr;
                    dc = (-(p + 1.0) * (p + 2.0) / 2.0 * p * xp1 + p * (p + 2.0) * (p + 1.0) * xp - p * (p + 1.0) / 2.0 * (p + 2.0) * xq) / rc;
                }
                const double sc = a.pair_scale[pair * a.num_bessel + j];
                mine[j] = static_cast<float>(b * c * sc);
                mine[64 + j] = static_cast<float>((db * c + b * dc) * sc);
            }
            __syncthreads();
            int cur = 0;
            for (int layer = 0; layer < a.num_hidden_layers; ++layer) {
                const float* xin = mine + cur * 128;
                float* xout = mine + (cur ^ 1) * 128;
                const int n_in = layer == 0 ? a.num_bessel : H;
                const float* w = layer == 0 ? w1 : wh + (layer - 1) * H * H;
                if (live && j < H) {
                    float z = 0.f, dz = 0.f;
                    for (int q = 0; q < n_in; ++q) {
                        const float wv = w[q * H + j];
                        z = fmaf(xin[q], wv, z);
                        dz = fmaf(xin[64 + q], wv, dz);
                    }
                    const float sig = 1.f / (1.f + expf(-z));
                    xout[j] = a.silu_scale * z * sig;
                    xout[64 + j] = a.silu_scale * sig * (1.f + z * (1.f - sig)) * dz;
                }
                __syncthreads();
                cur ^= 1;
            }
            if (live && j < H) {
                a.x_out[static_cast<size_t>(e) * H + j] = mine[cur * 128 + j];
                a.dx_out[static_cast<size_t>(e) * H + j] = mine[cur * 128 + 64 + j];
            }
            __syncthreads();
        }
    }
}

// Input check for callers that cannot vouch for their edge arrays: counts, per kind, the entries that would make the
// evaluation read out of bounds or produce non-finite values. Reads only inside the given arrays.
//   0 node type outside [0, num_elements)      1 negative neighbour count      2 counts do not add up to the edge total
//   3 sender index outside [0, feature_rows)   4 sender type outside the model  5 r not finite, <= 0 or beyond r_cut
//   6 r differs from |xyz| by more than 1e-6 relative
constexpr int kNumInputChecks = 7;
static __global__ void validate_inputs_kernel(int N, long long E, int num_elements, int feature_rows, double r_cut,
                                       const int* __restrict__ node_types, const int* __restrict__ num_neigh,
                                       const long long* __restrict__ first_neigh, const int* __restrict__ neigh_indices,
                                       const int* __restrict__ neigh_types, const double* __restrict__ xyz, const double* __restrict__ r,
                                       unsigned long long* __restrict__ counts) {
    const long long t0 = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    unsigned long long bad[kNumInputChecks] = {};
    for (long long i = t0; i < N; i += stride) {
        if (node_types[i] < 0 || node_types[i] >= num_elements) bad[0] += 1;
        if (num_neigh[i] < 0) bad[1] += 1;
    }
    if (t0 == 0 && N > 0 && first_neigh[N - 1] + num_neigh[N - 1] != E) bad[2] += 1;
    for (long long e = t0; e < E; e += stride) {
        if (neigh_indices[e] < 0 || neigh_indices[e] >= feature_rows) bad[3] += 1;
        if (neigh_types[e] < 0 || neigh_types[e] >= num_elements) bad[4] += 1;
        const double rr = r[e];
        if (!(rr > 0.0) || !(rr <= r_cut * (1.0 + 1e-12)) || !isfinite(rr)) bad[5] += 1;
        const double x = xyz[3 * e], y = xyz[3 * e + 1], z = xyz[3 * e + 2];
        const double d = sqrt(x * x + y * y + z * z);
        if (!(fabs(d - rr) <= 1e-6 * fmax(d, rr))) bad[6] += 1;
    }
    for (int c = 0; c < kNumInputChecks; ++c)
        if (bad[c]) atomicAdd(counts + c, bad[c]);
}

// Measurement probe: streams, for every edge of the current edge set, the spline row the edge kernels read
// (same (pair, bin) addressing, same per-thread 16-byte loads) and does nothing else; its duration is the
// floor the L2 -> SM path sets for one pass of an edge kernel over the edge set. No barriers and few
// registers, so the SMs run it at full occupancy.
template <typename T>
__global__ void row_stream_probe_kernel(int N, int K, int P, const int* __restrict__ node_types, const long long* __restrict__ first_neigh,
                                        const int* __restrict__ neigh_types, const double* __restrict__ r, const T* __restrict__ coef,
                                        SplineMeta sm, const int* __restrict__ order, T* __restrict__ sink) {
    using V = typename Lane<T>::type;
    const int L = lanes_of<V>(K), Kt = table_channels<T>(K), stride = 4 * Kt;
    V acc = V(0.0);
    for (int slot = blockIdx.x; slot < N; slot += gridDim.x) {
        const int i = order ? order[slot] : slot;
        const int type_i = node_types[i];
        const long long e_begin = first_neigh[i], e_end = first_neigh[i + 1];
        for (int k = threadIdx.x; k < L; k += blockDim.x)
            for (long long e = e_begin; e < e_end; ++e) {
                int bin = static_cast<int>(r[e] / sm.h);
                bin = bin < 0 ? 0 : (bin > sm.num_bins - 1 ? sm.num_bins - 1 : bin);
                const int tj = neigh_types[e];
                const int lo = type_i <= tj ? type_i : tj, hi = type_i <= tj ? tj : type_i;
                const int pair = lo * (2 * sm.num_elements - lo - 1) / 2 + hi;
                const T* row = coef + (static_cast<long long>(pair) * sm.num_bins + bin) * P * stride;
                for (int p = 0; p < P; ++p) {
                    const Coef<V> c = load_coef<V>(row + p * stride, k, L);
                    acc = acc + ((c.x + c.y) + (c.z + c.w));
                }
            }
    }
    if (lane_sum(acc) == T(1.2345e30)) *sink = lane_sum(acc);     // never true for real tables; keeps the loads alive
}

// Sum of the adjoint messages of all edges that have row j as their sender, in the fixed order
// of the sender-sorted edge list (deterministic; takes the place of the atomic scatter the
// reference's device code uses, mace_kokkos.cpp:1008-1010):
//   H_adj[j, :, :] += sum_{e in in_edges(j)} Hmsg[e, :, :]
// VEC: a thread sums two neighbouring values with 16-byte loads (float64 rows of even width; the rows start 16-byte aligned).
template <typename T, bool VEC>
__global__ void sender_gather_kernel(int rows, int width, const long long* __restrict__ in_ptr,
                                     const int* __restrict__ in_edge, const T* __restrict__ Hmsg, T* __restrict__ H_adj) {
    chain_begin();
    for (int j = blockIdx.x; j < rows; j += gridDim.x) {
        const long long b = in_ptr[j], e = in_ptr[j + 1];
        if constexpr (VEC && sizeof(T) == 8) {
            for (int c = 2 * threadIdx.x; c < width; c += 2 * blockDim.x) {
                // eight rows in flight per thread; the additions stay in list order
                double a0 = 0, a1 = 0;
                long long n = b;
                for (; n + 8 <= e; n += 8) {
                    double2 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        v[u] = __ldcs(reinterpret_cast<const double2*>(Hmsg + static_cast<size_t>(in_edge[n + u]) * width + c));
#pragma unroll
                    for (int u = 0; u < 8; ++u) { a0 += v[u].x; a1 += v[u].y; }
                }
                for (; n < e; ++n) {
                    const double2 v = __ldcs(reinterpret_cast<const double2*>(Hmsg + static_cast<size_t>(in_edge[n]) * width + c));
                    a0 += v.x; a1 += v.y;
                }
                double2* out = reinterpret_cast<double2*>(H_adj + static_cast<size_t>(j) * width + c);
                double2 o = *out;
                o.x += a0; o.y += a1;
                *out = o;
            }
            continue;
        }
        for (int c = threadIdx.x; c < width; c += blockDim.x) {
            // eight rows in flight per thread; the additions stay in list order
            T acc = 0;
            long long n = b;
            for (; n + 8 <= e; n += 8) {
                T v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = __ldcs(Hmsg + static_cast<size_t>(in_edge[n + u]) * width + c);
#pragma unroll
                for (int u = 0; u < 8; ++u) acc += v[u];
            }
            for (; n < e; ++n) acc += __ldcs(Hmsg + static_cast<size_t>(in_edge[n]) * width + c);
            H_adj[static_cast<size_t>(j) * width + c] += acc;
        }
    }
}

// =============================================================================================
// Symmetric contraction (MACE::compute_M0 / compute_M1, mace.cpp:348-370,759-777, and their
// reverses :372-395,779-794). One thread per (node, channel) walks the nested Horner program of
// each output component; the 16 inputs of the thread live in shared memory.
// =============================================================================================
template <typename T>
struct PolyArgs {
    int N, K;
    int num_out;                 // output components (nLM for M0, 1 for M1)
    int num_mono;                // monomial rows per element in `coef`
    const int* node_types;
    const int* perm;             // nodes sorted by element type
    const int* type_seg;         // [E + 1] segment of each type in perm
    int num_types;               // E
    const int* prog;             // concatenated operation streams (see compile_polynomial)
    const int* prog_off;         // [num_out] first word of each stream
    const int* prog_cnt;         // [num_out] operations to execute (a multiple of the prefetch distance)
    const int* mono_off;         // [num_out] first coefficient row of each stream
    const T* coef;               // [E][num_mono][K]
    const T* A;                  // [N][16][K]
    T* M;                        // forward output [N][num_out][K]
    const T* M_adj;              // reverse input  [N][num_out][K]
    T* A_adj;                    // reverse output [N][16][K] (overwritten)
};

constexpr int kPolyAhead = 8;    // must equal kPolyPrefetch of the program builder

__device__ __forceinline__ int poly_kind(int w) { return w & 7; }
__device__ __forceinline__ int poly_var(int w) { return (w >> 3) & 31; }
template <typename T>
__device__ __forceinline__ T poly_coef(const T* c, int w, int K) {
    const int row = (w >> 8) - 1;
    return row >= 0 ? __ldg(c + static_cast<size_t>(row) * K) : T(0);
}

// One thread owns one channel of NB nodes of the same element type (blockIdx.y = type, blockIdx.x =
// group of NB nodes in the type's segment of the sorted node list, blockIdx.z = channel chunk), so
// every coefficient fetched from L2 is used NB times, and the operation words and coefficients of
// the next kPolyAhead operations are already in flight while one executes. Inputs live in shared
// memory as [node slot][variable][thread].
template <typename T, int NB>
__global__ void poly_forward_kernel(const PolyArgs<T> a) {
    chain_begin();
    extern __shared__ unsigned char smem_raw[];
    T* As = reinterpret_cast<T*>(smem_raw);           // [NB][16][blockDim.x]
    const int nt = blockDim.x, t = threadIdx.x;
    const int type = blockIdx.y;
    const int seg_begin = a.type_seg[type], seg_count = a.type_seg[type + 1] - seg_begin;
    const int first = blockIdx.x * NB;
    if (first >= seg_count) return;
    const int k = blockIdx.z * nt + t;
    if (k >= a.K) return;
    int node[NB];
#pragma unroll
    for (int n = 0; n < NB; ++n) {
        const bool valid = first + n < seg_count;
        node[n] = valid ? a.perm[seg_begin + first + n] : -1;
#pragma unroll
        for (int q = 0; q < kNumLm; ++q)
            As[(n * kNumLm + q) * nt + t] = valid ? a.A[(static_cast<size_t>(node[n]) * kNumLm + q) * a.K + k] : T(0);
    }
    const T* cf = a.coef + static_cast<size_t>(type) * a.num_mono * a.K + k;
    for (int o = 0; o < a.num_out; ++o) {
        const int* w = a.prog + a.prog_off[o];
        const int count = a.prog_cnt[o];
        const T* c = cf + static_cast<size_t>(a.mono_off[o]) * a.K;
        int wr[kPolyAhead];
        T cr[kPolyAhead];
#pragma unroll
        for (int u = 0; u < kPolyAhead; ++u) { wr[u] = __ldg(w + u); cr[u] = poly_coef(c, wr[u], a.K); }
        T total_v[NB], s1[NB], s2[NB];
#pragma unroll
        for (int n = 0; n < NB; ++n) total_v[n] = s1[n] = s2[n] = T(0);
        for (int base = 0; base < count; base += kPolyAhead) {
#pragma unroll
            for (int u = 0; u < kPolyAhead; ++u) {
                const int word = wr[u];
                const T cv = cr[u];
                wr[u] = __ldg(w + base + kPolyAhead + u);          // streams are padded, so this stays in bounds
                cr[u] = poly_coef(c, wr[u], a.K);
                const int kind = poly_kind(word), q = poly_var(word);
                if (kind == 0) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) s2[n] += cv * As[(n * kNumLm + q) * nt + t];
                } else if (kind == 1) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) s2[n] = cv;
                } else if (kind == 2) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) s1[n] += s2[n] * As[(n * kNumLm + q) * nt + t];
                } else if (kind == 3) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) s1[n] = cv;
                } else if (kind == 4) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) total_v[n] += s1[n] * As[(n * kNumLm + q) * nt + t];
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NB; ++n)
            if (node[n] >= 0) a.M[(static_cast<size_t>(node[n]) * a.num_out + o) * a.K + k] = total_v[n];
    }
}

template <typename T, int NB>
__global__ void poly_reverse_kernel(const PolyArgs<T> a) {
    chain_begin();
    extern __shared__ unsigned char smem_raw[];
    const int nt = blockDim.x, t = threadIdx.x;
    T* As = reinterpret_cast<T*>(smem_raw);           // [NB][16][nt]
    T* Gs = As + NB * kNumLm * nt;                    // [NB][16][nt] gradient accumulators
    const int type = blockIdx.y;
    const int seg_begin = a.type_seg[type], seg_count = a.type_seg[type + 1] - seg_begin;
    const int first = blockIdx.x * NB;
    if (first >= seg_count) return;
    const int k = blockIdx.z * nt + t;
    if (k >= a.K) return;
    int node[NB];
#pragma unroll
    for (int n = 0; n < NB; ++n) {
        const bool valid = first + n < seg_count;
        node[n] = valid ? a.perm[seg_begin + first + n] : -1;
#pragma unroll
        for (int q = 0; q < kNumLm; ++q) {
            As[(n * kNumLm + q) * nt + t] = valid ? a.A[(static_cast<size_t>(node[n]) * kNumLm + q) * a.K + k] : T(0);
            Gs[(n * kNumLm + q) * nt + t] = T(0);
        }
    }
    const T* cf = a.coef + static_cast<size_t>(type) * a.num_mono * a.K + k;
    for (int o = 0; o < a.num_out; ++o) {
        T seed[NB];
#pragma unroll
        for (int n = 0; n < NB; ++n) seed[n] = node[n] >= 0 ? a.M_adj[(static_cast<size_t>(node[n]) * a.num_out + o) * a.K + k] : T(0);
        const int* w = a.prog + a.prog_off[o];
        const int count = a.prog_cnt[o];
        const T* c = cf + static_cast<size_t>(a.mono_off[o]) * a.K;
        int wr[kPolyAhead];
        T cr[kPolyAhead];
#pragma unroll
        for (int u = 0; u < kPolyAhead; ++u) { wr[u] = __ldg(w + u); cr[u] = poly_coef(c, wr[u], a.K); }
        // s1/s2: values of the open head / pair brackets; a2: A[q2]; adj1/adj2: adjoints of the brackets
        T s1[NB], s2[NB], a2[NB], adj1[NB], adj2[NB];
#pragma unroll
        for (int n = 0; n < NB; ++n) s1[n] = s2[n] = a2[n] = adj1[n] = adj2[n] = T(0);
        for (int base = 0; base < count; base += kPolyAhead) {
#pragma unroll
            for (int u = 0; u < kPolyAhead; ++u) {
                const int word = wr[u];
                const T cv = cr[u];
                wr[u] = __ldg(w + base + kPolyAhead + u);
                cr[u] = poly_coef(c, wr[u], a.K);
                const int kind = poly_kind(word), q = poly_var(word);
                if (kind == 0) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) {
                        s2[n] += cv * As[(n * kNumLm + q) * nt + t];
                        Gs[(n * kNumLm + q) * nt + t] += adj2[n] * cv;
                    }
                } else if (kind == 1) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) { a2[n] = As[(n * kNumLm + q) * nt + t]; s2[n] = cv; adj2[n] = adj1[n] * a2[n]; }
                } else if (kind == 2) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) { Gs[(n * kNumLm + q) * nt + t] += adj1[n] * s2[n]; s1[n] += s2[n] * a2[n]; }
                } else if (kind == 3) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) { s1[n] = cv; adj1[n] = seed[n] * As[(n * kNumLm + q) * nt + t]; }
                } else if (kind == 4) {
#pragma unroll
                    for (int n = 0; n < NB; ++n) Gs[(n * kNumLm + q) * nt + t] += seed[n] * s1[n];
                }
            }
        }
    }
#pragma unroll
    for (int n = 0; n < NB; ++n)
        if (node[n] >= 0)
#pragma unroll
            for (int q = 0; q < kNumLm; ++q) a.A_adj[(static_cast<size_t>(node[n]) * kNumLm + q) * a.K + k] = Gs[(n * kNumLm + q) * nt + t];
}

// Straight-line variant for models whose monomial lists are the symmetry-complete ones of
// generated/poly_canon.hpp (l_max = 3, correlation 3): one thread per (node, channel), the 16 inputs and the
// 16 gradient accumulators in registers, every coefficient one load at a compile-time offset. `coef` is then
// ordered canonically, [element][canonical monomial][K]. NOUT = number of output components (1, 4 or 9).
// NB nodes of one element type share a thread: every coefficient load then feeds NB multiply-adds (the coefficient stream
// from L2, one load per multiply-add for NB = 1, is what these kernels wait for). The generated code is written for a
// type T with fma and *; here T is a short vector over the NB nodes. Grid: one thread per (node group, channel).
template <typename S, int NB>
struct PolyVec {
    S v[NB];
    __device__ __forceinline__ PolyVec() {}
    __device__ __forceinline__ PolyVec(S x) {
#pragma unroll
        for (int n = 0; n < NB; ++n) v[n] = x;
    }
    __device__ __forceinline__ PolyVec(int x) : PolyVec(S(static_cast<float>(x))) {}      // the generated code's zero
};
template <typename S, int NB>
__device__ __forceinline__ PolyVec<S, NB> fma(const PolyVec<S, NB>& x, const PolyVec<S, NB>& y, const PolyVec<S, NB>& z) {
    PolyVec<S, NB> r;
#pragma unroll
    for (int n = 0; n < NB; ++n) r.v[n] = fma(x.v[n], y.v[n], z.v[n]);
    return r;
}
template <typename S, int NB>
__device__ __forceinline__ PolyVec<S, NB> operator*(const PolyVec<S, NB>& x, const PolyVec<S, NB>& y) {
    PolyVec<S, NB> r;
#pragma unroll
    for (int n = 0; n < NB; ++n) r.v[n] = x.v[n] * y.v[n];
    return r;
}

// SPLIT: the NOUT warps of a CTA share 32 (node group, channel) pairs, one output component each (reverse: their gradients are
// added in shared memory in the order of the components). For structures that do not fill the GPU: a thread's chain of some
// hundred dependent multiply-adds per component is what they wait for (nine atoms, four components: 16 us for M0).
template <int NOUT, bool SPLIT> constexpr int poly_fixed_threads() { return SPLIT ? 32 * NOUT : 128; }

template <typename S, int NOUT, int NB, bool SPLIT>
__global__ void __launch_bounds__(poly_fixed_threads<NOUT, SPLIT>()) poly_fixed_forward_kernel(const PolyArgs<typename LaneScalar<S>::type> a) {
    chain_begin();
    using T = PolyVec<S, NB>;
    const int L = lanes_of<S>(a.K);
    // flat index -> (element type, group of NB nodes of that type, lane); groups of all types are numbered consecutively
    const int comp = SPLIT ? static_cast<int>(threadIdx.x >> 5) : 0;      // SPLIT: this warp's output component
    const long long idx = static_cast<long long>(blockIdx.x) * (SPLIT ? 32 : blockDim.x) + (SPLIT ? threadIdx.x & 31 : threadIdx.x);
    int g = static_cast<int>(idx / L);
    const int at = static_cast<int>(idx - static_cast<long long>(g) * L);
    int type = 0, seg_begin = 0, count = 0;
    for (; type < a.num_types; ++type) {
        seg_begin = a.type_seg[type];
        count = a.type_seg[type + 1] - seg_begin;
        const int groups = (count + NB - 1) / NB;
        if (g < groups) break;
        g -= groups;
    }
    if (type == a.num_types) return;
    int node[NB];
    bool live[NB];
#pragma unroll
    for (int n = 0; n < NB; ++n) {
        const int jn = g * NB + n;
        live[n] = jn < count;
        node[n] = a.perm[seg_begin + (live[n] ? jn : count - 1)];   // an empty slot repeats the last node; its results are dropped
    }
    const int k = at * lane_channels<S>();      // first channel of the lane
    const auto* cf = a.coef + static_cast<size_t>(type) * a.num_mono * a.K + k;
    T A[kNumLm];
#pragma unroll
    for (int q = 0; q < kNumLm; ++q)
#pragma unroll
        for (int n = 0; n < NB; ++n) A[q].v[n] = lane_load<S, true>(a.A + (static_cast<size_t>(node[n]) * kNumLm + q) * a.K + k, 0, a.K);
    {
        if (!SPLIT || comp == 0) {
            constexpr int kOff = kCanonPolyOffset[0];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
#include "generated/poly_lm0_forward.inc"
#pragma unroll
            for (int n = 0; n < NB; ++n)
                if (live[n]) lane_store<false, true>(a.M + (static_cast<size_t>(node[n]) * NOUT + 0) * a.K + k, 0, a.K, total.v[n]);
        }
    }
    if constexpr (NOUT > 1) {
        if (!SPLIT || comp == 1) {
            constexpr int kOff = kCanonPolyOffset[1];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
#include "generated/poly_lm1_forward.inc"
#pragma unroll
            for (int n = 0; n < NB; ++n)
                if (live[n]) lane_store<false, true>(a.M + (static_cast<size_t>(node[n]) * NOUT + 1) * a.K + k, 0, a.K, total.v[n]);
        }
        if (!SPLIT || comp == 2) {
            constexpr int kOff = kCanonPolyOffset[2];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
#include "generated/poly_lm2_forward.inc"
#pragma unroll
            for (int n = 0; n < NB; ++n)
                if (live[n]) lane_store<false, true>(a.M + (static_cast<size_t>(node[n]) * NOUT + 2) * a.K + k, 0, a.K, total.v[n]);
        }
        if (!SPLIT || comp == 3) {
            constexpr int kOff = kCanonPolyOffset[3];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
#include "generated/poly_lm3_forward.inc"
#pragma unroll
            for (int n = 0; n < NB; ++n)
                if (live[n]) lane_store<false, true>(a.M + (static_cast<size_t>(node[n]) * NOUT + 3) * a.K + k, 0, a.K, total.v[n]);
        }
    }
    if constexpr (NOUT > 4) {
        if (!SPLIT || comp == 4) {
            constexpr int kOff = kCanonPolyOffset[4];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
#include "generated/poly_lm4_forward.inc"
#pragma unroll
            for (int n = 0; n < NB; ++n)
                if (live[n]) lane_store<false, true>(a.M + (static_cast<size_t>(node[n]) * NOUT + 4) * a.K + k, 0, a.K, total.v[n]);
        }
        if (!SPLIT || comp == 5) {
            constexpr int kOff = kCanonPolyOffset[5];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
#include "generated/poly_lm5_forward.inc"
#pragma unroll
            for (int n = 0; n < NB; ++n)
                if (live[n]) lane_store<false, true>(a.M + (static_cast<size_t>(node[n]) * NOUT + 5) * a.K + k, 0, a.K, total.v[n]);
        }
        if (!SPLIT || comp == 6) {
            constexpr int kOff = kCanonPolyOffset[6];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
#include "generated/poly_lm6_forward.inc"
#pragma unroll
            for (int n = 0; n < NB; ++n)
                if (live[n]) lane_store<false, true>(a.M + (static_cast<size_t>(node[n]) * NOUT + 6) * a.K + k, 0, a.K, total.v[n]);
        }
        if (!SPLIT || comp == 7) {
            constexpr int kOff = kCanonPolyOffset[7];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
#include "generated/poly_lm7_forward.inc"
#pragma unroll
            for (int n = 0; n < NB; ++n)
                if (live[n]) lane_store<false, true>(a.M + (static_cast<size_t>(node[n]) * NOUT + 7) * a.K + k, 0, a.K, total.v[n]);
        }
        if (!SPLIT || comp == 8) {
            constexpr int kOff = kCanonPolyOffset[8];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
#include "generated/poly_lm8_forward.inc"
#pragma unroll
            for (int n = 0; n < NB; ++n)
                if (live[n]) lane_store<false, true>(a.M + (static_cast<size_t>(node[n]) * NOUT + 8) * a.K + k, 0, a.K, total.v[n]);
        }
    }
}

// LATE (one component): the adjoint multiplies the gradient at the end, the products of node_head_kernel, which knows the gradient before
// the adjoint. Small structures only, where stage calls must give that kernel's bits: float64 at 4,000 atoms takes 47 instead of 45 us.
template <typename S, int NOUT, int NB, bool SPLIT, bool LATE = false>
__global__ void __launch_bounds__(poly_fixed_threads<NOUT, SPLIT>()) poly_fixed_reverse_kernel(const PolyArgs<typename LaneScalar<S>::type> a) {
    chain_begin();
    using T = PolyVec<S, NB>;
    const int L = lanes_of<S>(a.K);
    // flat index -> (element type, group of NB nodes of that type, lane); groups of all types are numbered consecutively
    const int comp = SPLIT ? static_cast<int>(threadIdx.x >> 5) : 0;      // SPLIT: this warp's output component
    const long long idx = static_cast<long long>(blockIdx.x) * (SPLIT ? 32 : blockDim.x) + (SPLIT ? threadIdx.x & 31 : threadIdx.x);
    int g = static_cast<int>(idx / L);
    const int at = static_cast<int>(idx - static_cast<long long>(g) * L);
    int type = 0, seg_begin = 0, count = 0;
    for (; type < a.num_types; ++type) {
        seg_begin = a.type_seg[type];
        count = a.type_seg[type + 1] - seg_begin;
        const int groups = (count + NB - 1) / NB;
        if (g < groups) break;
        g -= groups;
    }
    bool in_range = true;
    if (type == a.num_types) {
        if constexpr (!SPLIT) return;
        in_range = false;      // idle lane: repeats some node, its results are dropped
        type = 0; seg_begin = 0; count = a.type_seg[a.num_types]; g = 0;
    }
    int node[NB];
    bool live[NB];
#pragma unroll
    for (int n = 0; n < NB; ++n) {
        const int jn = g * NB + n;
        live[n] = in_range && jn < count;
        node[n] = a.perm[seg_begin + (jn < count ? jn : count - 1)];   // an empty slot repeats the last node; its results are dropped
    }
    const int k = at * lane_channels<S>();      // first channel of the lane
    const auto* cf = a.coef + static_cast<size_t>(type) * a.num_mono * a.K + k;
    T A[kNumLm], G[kNumLm];
#pragma unroll
    for (int q = 0; q < kNumLm; ++q) {
#pragma unroll
        for (int n = 0; n < NB; ++n) A[q].v[n] = lane_load<S, true>(a.A + (static_cast<size_t>(node[n]) * kNumLm + q) * a.K + k, 0, a.K);
        G[q] = T(0);
    }
    {
        if (!SPLIT || comp == 0) {
            constexpr int kOff = kCanonPolyOffset[0];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
            T seed;
#pragma unroll
            for (int n = 0; n < NB; ++n) seed.v[n] = lane_load<S, true>(a.M_adj + (static_cast<size_t>(node[n]) * NOUT + 0) * a.K + k, 0, a.K);
            if constexpr (LATE) {
                static_assert(NOUT == 1, "one component");
                const T adjoint = seed;
                {
                    const T seed(1);
#include "generated/poly_lm0_reverse.inc"
                }
#pragma unroll
                for (int q = 0; q < kNumLm; ++q) G[q] = adjoint * G[q];
            } else {
#include "generated/poly_lm0_reverse.inc"
            }
        }
    }
    if constexpr (NOUT > 1) {
        if (!SPLIT || comp == 1) {
            constexpr int kOff = kCanonPolyOffset[1];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
            T seed;
#pragma unroll
            for (int n = 0; n < NB; ++n) seed.v[n] = lane_load<S, true>(a.M_adj + (static_cast<size_t>(node[n]) * NOUT + 1) * a.K + k, 0, a.K);
#include "generated/poly_lm1_reverse.inc"
        }
        if (!SPLIT || comp == 2) {
            constexpr int kOff = kCanonPolyOffset[2];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
            T seed;
#pragma unroll
            for (int n = 0; n < NB; ++n) seed.v[n] = lane_load<S, true>(a.M_adj + (static_cast<size_t>(node[n]) * NOUT + 2) * a.K + k, 0, a.K);
#include "generated/poly_lm2_reverse.inc"
        }
        if (!SPLIT || comp == 3) {
            constexpr int kOff = kCanonPolyOffset[3];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
            T seed;
#pragma unroll
            for (int n = 0; n < NB; ++n) seed.v[n] = lane_load<S, true>(a.M_adj + (static_cast<size_t>(node[n]) * NOUT + 3) * a.K + k, 0, a.K);
#include "generated/poly_lm3_reverse.inc"
        }
    }
    if constexpr (NOUT > 4) {
        if (!SPLIT || comp == 4) {
            constexpr int kOff = kCanonPolyOffset[4];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
            T seed;
#pragma unroll
            for (int n = 0; n < NB; ++n) seed.v[n] = lane_load<S, true>(a.M_adj + (static_cast<size_t>(node[n]) * NOUT + 4) * a.K + k, 0, a.K);
#include "generated/poly_lm4_reverse.inc"
        }
        if (!SPLIT || comp == 5) {
            constexpr int kOff = kCanonPolyOffset[5];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
            T seed;
#pragma unroll
            for (int n = 0; n < NB; ++n) seed.v[n] = lane_load<S, true>(a.M_adj + (static_cast<size_t>(node[n]) * NOUT + 5) * a.K + k, 0, a.K);
#include "generated/poly_lm5_reverse.inc"
        }
        if (!SPLIT || comp == 6) {
            constexpr int kOff = kCanonPolyOffset[6];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
            T seed;
#pragma unroll
            for (int n = 0; n < NB; ++n) seed.v[n] = lane_load<S, true>(a.M_adj + (static_cast<size_t>(node[n]) * NOUT + 6) * a.K + k, 0, a.K);
#include "generated/poly_lm6_reverse.inc"
        }
        if (!SPLIT || comp == 7) {
            constexpr int kOff = kCanonPolyOffset[7];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
            T seed;
#pragma unroll
            for (int n = 0; n < NB; ++n) seed.v[n] = lane_load<S, true>(a.M_adj + (static_cast<size_t>(node[n]) * NOUT + 7) * a.K + k, 0, a.K);
#include "generated/poly_lm7_reverse.inc"
        }
        if (!SPLIT || comp == 8) {
            constexpr int kOff = kCanonPolyOffset[8];
            auto C = [&](int slot) { return T(lane_load<S, true, Cache::kReadOnly>(cf + static_cast<size_t>(kOff + slot) * a.K, 0, a.K)); };
            T seed;
#pragma unroll
            for (int n = 0; n < NB; ++n) seed.v[n] = lane_load<S, true>(a.M_adj + (static_cast<size_t>(node[n]) * NOUT + 8) * a.K + k, 0, a.K);
#include "generated/poly_lm8_reverse.inc"
        }
    }
    if constexpr (SPLIT) {
        static_assert(NB == 1, "one node per thread");
        __shared__ S part[NOUT][kNumLm][32];
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int q = 0; q < kNumLm; ++q) part[comp][q][lane] = G[q].v[0];
        __syncthreads();
        for (int q = comp; q < kNumLm; q += NOUT) {
            S sum = part[0][q][lane];
#pragma unroll
            for (int o = 1; o < NOUT; ++o) sum += part[o][q][lane];
            if (live[0]) a.A_adj[(static_cast<size_t>(node[0]) * kNumLm + q) * a.K + k] = sum;
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < kNumLm; ++q)
#pragma unroll
        for (int n = 0; n < NB; ++n)
            if (live[n]) lane_store<false, true>(a.A_adj + (static_cast<size_t>(node[n]) * kNumLm + q) * a.K + k, 0, a.K, G[q].v[n]);
}

// =============================================================================================
// Channel-mixing linears as row-gathered GEMMs: C[row, :] (+)= A[row, :] . B  (or . B^T).
// A row of a problem is addressed as (node, sub): node = perm ? perm[seg_begin + r / sub_count]
// : r / sub_count, sub = r % sub_count, at A + node*a_node_stride + a_off + sub*a_sub_stride.
// One problem list entry per (element type, degree l) block; blockIdx.z selects the problem.
// Covers the dgemm/dgemv calls of compute_A0/H1/A1/H2 and their reverses (mace.cpp:184-198,
// 406-420, 623-637, 804-830 and :215-229, 434-448, 659-674, 846-872).
// =============================================================================================
template <typename T>
struct GemmProblem {
    const T* A; T* C; const T* B;
    const int* perm;         // optional node permutation (nodes sorted by element type)
    const int* seg;          // optional device array of segment offsets into perm
    int seg_index;           // this problem covers perm[seg[seg_index] .. seg[seg_index + 1])
    int num_nodes;           // used when seg == nullptr
    int sub_count;           // rows per node
    long long a_node_stride, a_off, a_sub_stride;
    long long c_node_stride, c_off, c_sub_stride;
    int Kd, Nc;              // inner dimension, output columns
    int ldb;                 // leading dimension of B
    int transB;              // 0: B is [Kd][Nc]; 1: B is [Nc][Kd] and used transposed
    int accumulate;          // 0: C = A.B ; 1: C += A.B
    const T* B_image;        // float32 tcgen05 path: B as pre-split, pre-swizzled operand tiles (gemm_tcgen05.cuh)
    // Optional second product into the same rows of C (gemm_rows_small_kernel only; null otherwise): C (+)= A.B + A2.B2,
    // with B2 laid out like B. Row r of A2 belongs to the node of row r of C.
    const T* A2; const T* B2;
    long long a2_node_stride, a2_off, a2_sub_stride;
};

// The problems of one launch. Up to kNear of them travel in the kernel's parameters (28 fill the classic 4 KB): a copy to
// the device in front of every GEMM launch cost about 4 us of stream time each, nine times per evaluation. Longer lists
// (many element types) go through the device ring.
template <typename T>
struct GemmList {
    static constexpr int kNear = 24;
    const GemmProblem<T>* far;
    GemmProblem<T> near[kNear];
    __device__ __forceinline__ const GemmProblem<T>& operator[](int q) const { return far ? far[q] : near[q]; }
};

constexpr int kGemmBM = 64, kGemmBN = 64, kGemmBK = 16, kGemmThreads = 128;

// Tensor-core fragments. float64 uses the DMMA instruction mma.sync.m8n8k4 (sm_100a has no 5th-generation
// tensor-core kind for float64); float32 uses TF32 mma.sync.m16n8k8 with the operands split into a TF32 head
// and a TF32 remainder and three products per tile (head*head + head*rem + rem*head), which keeps float32-level
// accuracy for the 1e-4 energy gate while running on the tensor pipe.
__device__ __forceinline__ void dmma_m8n8k4(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};" : "+d"(c0), "+d"(c1) : "d"(a), "d"(b));
}
__device__ __forceinline__ unsigned to_tf32(float x) {
    unsigned r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void mma_tf32_m16n8k8(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <typename T> struct GemmSmem;
template <> struct GemmSmem<double> { static constexpr int SA = kGemmBK + 4, SB = kGemmBN + 4; };   // conflict-free fragment reads
template <> struct GemmSmem<float> { static constexpr int SA = kGemmBK + 4, SB = kGemmBN + 8; };

// Warp tile 32 x 32 of the 64 x 64 CTA tile; accumulators and the k-loop body per precision.
template <typename T> struct WarpTile;
template <>
struct WarpTile<double> {
    double c[4][4][2];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) c[i][j][0] = c[i][j][1] = 0.0;
    }
    __device__ __forceinline__ void step(const double* As, const double* Bs, int wm, int wn, int lane) {
        constexpr int SA = GemmSmem<double>::SA, SB = GemmSmem<double>::SB;
#pragma unroll
        for (int kk = 0; kk < kGemmBK; kk += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[(wm * 32 + i * 8 + (lane >> 2)) * SA + kk + (lane & 3)];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[(kk + (lane & 3)) * SB + wn * 32 + j * 8 + (lane >> 2)];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma_m8n8k4(c[i][j][0], c[i][j][1], a[i], b[j]);
        }
    }
    template <typename F>
    __device__ __forceinline__ void for_each(int wm, int wn, int lane, F&& f) const {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) f(wm * 32 + i * 8 + (lane >> 2), wn * 32 + j * 8 + 2 * (lane & 3) + e, c[i][j][e]);
    }
};
template <>
struct WarpTile<float> {
    float c[2][4][4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[i][j][e] = 0.f;
    }
    __device__ __forceinline__ void step(const float* As, const float* Bs, int wm, int wn, int lane) {
        constexpr int SA = GemmSmem<float>::SA, SB = GemmSmem<float>::SB;
#pragma unroll
        for (int kk = 0; kk < kGemmBK; kk += 8) {
            unsigned ah[2][4], al[2][4], bh[4][2], bl[4][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = wm * 32 + i * 16 + (lane >> 2), cidx = kk + (lane & 3);
                const float v[4] = {As[r * SA + cidx], As[(r + 8) * SA + cidx], As[r * SA + cidx + 4], As[(r + 8) * SA + cidx + 4]};
#pragma unroll
                for (int e = 0; e < 4; ++e) { ah[i][e] = to_tf32(v[e]); al[i][e] = to_tf32(v[e] - __uint_as_float(ah[i][e])); }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int n = wn * 32 + j * 8 + (lane >> 2);
                const float v[2] = {Bs[(kk + (lane & 3)) * SB + n], Bs[(kk + 4 + (lane & 3)) * SB + n]};
#pragma unroll
                for (int e = 0; e < 2; ++e) { bh[j][e] = to_tf32(v[e]); bl[j][e] = to_tf32(v[e] - __uint_as_float(bh[j][e])); }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    mma_tf32_m16n8k8(c[i][j], al[i], bh[j]);
                    mma_tf32_m16n8k8(c[i][j], ah[i], bl[j]);
                    mma_tf32_m16n8k8(c[i][j], ah[i], bh[j]);
                }
        }
    }
    template <typename F>
    __device__ __forceinline__ void for_each(int wm, int wn, int lane, F&& f) const {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    f(wm * 32 + i * 16 + (lane >> 2) + (e >> 1) * 8, wn * 32 + j * 8 + 2 * (lane & 3) + (e & 1), c[i][j][e]);
    }
};

template <typename T>
__global__ void __launch_bounds__(kGemmThreads) gemm_rows_kernel(const __grid_constant__ GemmList<T> problems) {
    chain_begin();
    const GemmProblem<T> pb = problems[blockIdx.z];
    int node_begin = 0, node_count = pb.num_nodes;
    if (pb.seg) { node_begin = pb.seg[pb.seg_index]; node_count = pb.seg[pb.seg_index + 1] - node_begin; }
    const long long M = static_cast<long long>(node_count) * pb.sub_count;
    const long long row0 = static_cast<long long>(blockIdx.x) * kGemmBM;
    const int col0 = blockIdx.y * kGemmBN;
    if (row0 >= M || col0 >= pb.Nc) return;

    constexpr int SA = GemmSmem<T>::SA, SB = GemmSmem<T>::SB;
    __shared__ T As[kGemmBM * SA];
    __shared__ T Bs[kGemmBK * SB];
    __shared__ long long a_base[kGemmBM];
    __shared__ long long c_base[kGemmBM];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp >> 1, wn = warp & 1;
    if (tid < kGemmBM) {
        const long long r = row0 + tid;
        if (r < M) {
            const long long n = r / pb.sub_count;
            const int sub = static_cast<int>(r - n * pb.sub_count);
            const long long node = pb.perm ? pb.perm[node_begin + n] : (node_begin + n);
            a_base[tid] = node * pb.a_node_stride + pb.a_off + sub * pb.a_sub_stride;
            c_base[tid] = node * pb.c_node_stride + pb.c_off + sub * pb.c_sub_stride;
        } else {
            a_base[tid] = -1;
            c_base[tid] = -1;
        }
    }
    __syncthreads();

    constexpr int kPer = kGemmBM * kGemmBK / kGemmThreads;   // 8 elements of each tile per thread
    T ra[kPer], rb[kPer];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int it = 0; it < kPer; ++it) {
            const int lin = tid + it * kGemmThreads;
            const int rr = lin >> 4, kk = lin & 15;
            ra[it] = (a_base[rr] >= 0 && k0 + kk < pb.Kd) ? pb.A[a_base[rr] + k0 + kk] : T(0);
            if (!pb.transB) {
                const int kb = lin >> 6, cc = lin & 63;
                rb[it] = (k0 + kb < pb.Kd && col0 + cc < pb.Nc) ? pb.B[static_cast<size_t>(k0 + kb) * pb.ldb + col0 + cc] : T(0);
            } else {
                const int cc = lin >> 4, kb = lin & 15;
                rb[it] = (k0 + kb < pb.Kd && col0 + cc < pb.Nc) ? pb.B[static_cast<size_t>(col0 + cc) * pb.ldb + k0 + kb] : T(0);
            }
        }
    };
    auto stash = [&]() {
#pragma unroll
        for (int it = 0; it < kPer; ++it) {
            const int lin = tid + it * kGemmThreads;
            As[(lin >> 4) * SA + (lin & 15)] = ra[it];
            if (!pb.transB) Bs[(lin >> 6) * SB + (lin & 63)] = rb[it];
            else Bs[(lin & 15) * SB + (lin >> 4)] = rb[it];
        }
    };

    WarpTile<T> acc;
    acc.zero();
    fetch(0);
    for (int k0 = 0; k0 < pb.Kd; k0 += kGemmBK) {
        stash();
        __syncthreads();
        if (k0 + kGemmBK < pb.Kd) fetch(k0 + kGemmBK);     // next tile's global loads overlap the tensor-core work
        acc.step(As, Bs, wm, wn, lane);
        __syncthreads();
    }
    acc.for_each(wm, wn, lane, [&](int r, int cidx, T v) {
        const long long cb = c_base[r];
        const int col = col0 + cidx;
        if (cb >= 0 && col < pb.Nc) {
            T* dst = pb.C + cb + col;
            *dst = pb.accumulate ? (*dst + v) : v;
        }
    });
}

// float64 variant with asynchronous tile loads: the 64 x 16 tile of gathered A rows and the 16 x 64 tile of B go from
// global to shared memory with 16-byte cp.async copies (no staging registers), two stages deep, so the copies of tile
// t + 1 run while the DMMA instructions work on tile t and there is one barrier pair per tile instead of a
// load - store - barrier sequence. Needs 16-byte aligned rows (even strides and offsets, even leading dimension); the
// launch code falls back to gemm_rows_kernel otherwise. Out-of-range rows, columns and k values are zero-filled by the
// copy's source-size operand.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem)), "l"(gmem), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

static __global__ void __launch_bounds__(kGemmThreads) gemm_rows_f64_async_kernel(const __grid_constant__ GemmList<double> problems) {
    chain_begin();
    const GemmProblem<double> pb = problems[blockIdx.z];
    int node_begin = 0, node_count = pb.num_nodes;
    if (pb.seg) { node_begin = pb.seg[pb.seg_index]; node_count = pb.seg[pb.seg_index + 1] - node_begin; }
    const long long M = static_cast<long long>(node_count) * pb.sub_count;
    const long long row0 = static_cast<long long>(blockIdx.x) * kGemmBM;
    const int col0 = blockIdx.y * kGemmBN;
    if (row0 >= M || col0 >= pb.Nc) return;

    constexpr int SA = GemmSmem<double>::SA, SB = GemmSmem<double>::SB;      // 20 and 68 doubles: rows start on 16-byte boundaries
    constexpr int kBTile = kGemmBK * SB > kGemmBN * SA ? kGemmBK * SB : kGemmBN * SA;
    __shared__ __align__(16) double As[2][kGemmBM * SA];
    __shared__ __align__(16) double Bs[2][kBTile];          // [k][n] rows of SB, or for transposed B [n][k] rows of SA
    __shared__ long long a_base[kGemmBM];
    __shared__ long long c_base[kGemmBM];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp >> 1, wn = warp & 1;
    if (tid < kGemmBM) {
        const long long r = row0 + tid;
        if (r < M) {
            const long long n = r / pb.sub_count;
            const int sub = static_cast<int>(r - n * pb.sub_count);
            const long long node = pb.perm ? pb.perm[node_begin + n] : (node_begin + n);
            a_base[tid] = node * pb.a_node_stride + pb.a_off + sub * pb.a_sub_stride;
            c_base[tid] = node * pb.c_node_stride + pb.c_off + sub * pb.c_sub_stride;
        } else {
            a_base[tid] = -1;
            c_base[tid] = -1;
        }
    }
    __syncthreads();

    auto issue = [&](int stage, int k0) {
        // A: 64 rows x 8 chunks of two doubles; B: 16 x 32 chunks (or 64 x 8 for transposed B): 4 + 4 chunks per thread
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int lin = tid + it * kGemmThreads;
            const int rr = lin >> 3, kk = (lin & 7) * 2;
            const long long ab = a_base[rr];
            const int left = pb.Kd - (k0 + kk);
            const int bytes = ab >= 0 ? (left >= 2 ? 16 : (left == 1 ? 8 : 0)) : 0;
            cp_async16(&As[stage][rr * SA + kk], pb.A + (bytes ? ab + k0 + kk : 0), bytes);
        }
        if (!pb.transB) {
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int lin = tid + it * kGemmThreads;
                const int kb = lin >> 5, cc = (lin & 31) * 2;
                const int left = pb.Nc - (col0 + cc);
                const int bytes = (k0 + kb < pb.Kd) ? (left >= 2 ? 16 : (left == 1 ? 8 : 0)) : 0;
                cp_async16(&Bs[stage][kb * SB + cc], pb.B + (bytes ? static_cast<size_t>(k0 + kb) * pb.ldb + col0 + cc : 0), bytes);
            }
        } else {
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int lin = tid + it * kGemmThreads;
                const int cc = lin >> 3, kb = (lin & 7) * 2;
                const int left = pb.Kd - (k0 + kb);
                const int bytes = (col0 + cc < pb.Nc) ? (left >= 2 ? 16 : (left == 1 ? 8 : 0)) : 0;
                cp_async16(&Bs[stage][cc * SA + kb], pb.B + (bytes ? static_cast<size_t>(col0 + cc) * pb.ldb + k0 + kb : 0), bytes);
            }
        }
        cp_async_commit();
    };

    double c[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j][0] = c[i][j][1] = 0.0;
    const int num_tiles = (pb.Kd + kGemmBK - 1) / kGemmBK;
    issue(0, 0);
    for (int t = 0; t < num_tiles; ++t) {
        const int stage = t & 1;
        if (t + 1 < num_tiles) { issue(stage ^ 1, (t + 1) * kGemmBK); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncthreads();
        const double* Asm = As[stage];
        const double* Bsm = Bs[stage];
#pragma unroll
        for (int kk = 0; kk < kGemmBK; kk += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = Asm[(wm * 32 + i * 8 + (lane >> 2)) * SA + kk + (lane & 3)];
            if (!pb.transB) {
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = Bsm[(kk + (lane & 3)) * SB + wn * 32 + j * 8 + (lane >> 2)];
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = Bsm[(wn * 32 + j * 8 + (lane >> 2)) * SA + kk + (lane & 3)];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma_m8n8k4(c[i][j][0], c[i][j][1], a[i], b[j]);
        }
        __syncthreads();      // this stage is refilled by the copies issued in the next iteration
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = wm * 32 + i * 8 + (lane >> 2), cidx = wn * 32 + j * 8 + 2 * (lane & 3) + e;
                const long long cb = c_base[r];
                const int col = col0 + cidx;
                if (cb >= 0 && col < pb.Nc) {
                    double* dst = pb.C + cb + col;
                    *dst = pb.accumulate ? (*dst + c[i][j][e]) : c[i][j][e];
                }
            }
}

// =============================================================================================
// Few rows (a molecule, a unit cell): the 64 x 64 and 128 x 128 tiles above leave a handful of CTAs that walk the inner
// dimension alone, one exposed L2 latency per 16 or 32 values (Kd = 384: 24 of them, 28 us for nine rows). Here a CTA owns
// 16 x 32 outputs, so there are eight (float32: thirty-two) times as many, and four stages of 32 inner values are in flight
// at once: for Kd = 128 every load of the CTA is issued before the first wait. float64: DMMA, two accumulator sets
// (alternate k-steps) so that four multiply chains run side by side; float32: plain FFMA, so no operand splitting.
// A problem with a second product (A2, B2) is walked as one longer inner dimension.
// Needs rows and leading dimensions that start on 16-byte boundaries.
// =============================================================================================
constexpr int kSmallBM = 16, kSmallBN = 32, kSmallBK = 32, kSmallStages = 4, kSmallThreads = 128;
constexpr int kSmallStride = kSmallBK + 4;       // rows of both tiles (BN = BK): 16-byte aligned, conflict-free fragment reads
template <typename T> constexpr int gemm_small_stage() { return (kSmallBM + kSmallBK) * kSmallStride; }
template <typename T> constexpr int gemm_small_smem() { return kSmallStages * gemm_small_stage<T>() * static_cast<int>(sizeof(T)); }

template <typename T>
__global__ void __launch_bounds__(kSmallThreads) gemm_rows_small_kernel(const __grid_constant__ GemmList<T> problems) {
    chain_begin();
    static_assert(kSmallBN == kSmallBK, "the B tile uses one stride for both orientations");
    constexpr int S = kSmallStride, V = 16 / static_cast<int>(sizeof(T));      // values per 16-byte copy
    const GemmProblem<T> pb = problems[blockIdx.z];
    int node_begin = 0, node_count = pb.num_nodes;
    if (pb.seg) { node_begin = pb.seg[pb.seg_index]; node_count = pb.seg[pb.seg_index + 1] - node_begin; }
    const long long M = static_cast<long long>(node_count) * pb.sub_count;
    const long long row0 = static_cast<long long>(blockIdx.x) * kSmallBM;
    const int col0 = blockIdx.y * kSmallBN;
    if (row0 >= M || col0 >= pb.Nc) return;
    extern __shared__ __align__(16) unsigned char gemm_small_raw[];
    T* const smem = reinterpret_cast<T*>(gemm_small_raw);
    __shared__ long long a_base[2][kSmallBM], c_base[kSmallBM];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < kSmallBM) {
        const long long r = row0 + tid;
        a_base[0][tid] = a_base[1][tid] = c_base[tid] = -1;
        if (r < M) {
            const long long n = r / pb.sub_count;
            const int sub = static_cast<int>(r - n * pb.sub_count);
            const long long node = pb.perm ? pb.perm[node_begin + n] : (node_begin + n);
            a_base[0][tid] = node * pb.a_node_stride + pb.a_off + sub * pb.a_sub_stride;
            a_base[1][tid] = node * pb.a2_node_stride + pb.a2_off + sub * pb.a2_sub_stride;
            c_base[tid] = node * pb.c_node_stride + pb.c_off + sub * pb.c_sub_stride;
        }
    }
    __syncthreads();
    const bool transB = pb.transB != 0;
    const int Kd = pb.Kd, tiles_1 = (Kd + kSmallBK - 1) / kSmallBK, num_tiles = pb.A2 ? 2 * tiles_1 : tiles_1;
    auto issue = [&](int t) {
        if (t < num_tiles) {
            const int src = t >= tiles_1 ? 1 : 0, k0 = (t - src * tiles_1) * kSmallBK;
            const T* A = src ? pb.A2 : pb.A;
            const T* B = src ? pb.B2 : pb.B;
            T* As = smem + (t % kSmallStages) * gemm_small_stage<T>();
            T* Bs = As + kSmallBM * S;
            auto bytes_of = [](int left) { return left >= V ? 16 : (left > 0 ? left * static_cast<int>(sizeof(T)) : 0); };
#pragma unroll
            for (int lin = tid; lin < kSmallBM * kSmallBK / V; lin += kSmallThreads) {
                const int rr = lin / (kSmallBK / V), kk = lin % (kSmallBK / V) * V;
                const long long ab = a_base[src][rr];
                const int bytes = ab >= 0 ? bytes_of(Kd - (k0 + kk)) : 0;
                cp_async16(&As[rr * S + kk], A + (bytes ? ab + k0 + kk : 0), bytes);
            }
#pragma unroll
            for (int lin = tid; lin < kSmallBN * kSmallBK / V; lin += kSmallThreads) {
                const int row = lin / (kSmallBK / V), v = lin % (kSmallBK / V) * V;
                // [k][n] for plain B, [n][k] for transposed B
                const int k = k0 + (transB ? v : row), n = col0 + (transB ? row : v);
                const int bytes = transB ? (n < pb.Nc ? bytes_of(Kd - k) : 0) : (k < Kd ? bytes_of(pb.Nc - n) : 0);
                cp_async16(&Bs[row * S + v], B + (bytes ? (transB ? static_cast<size_t>(n) * pb.ldb + k : static_cast<size_t>(k) * pb.ldb + n) : 0), bytes);
            }
        }
        cp_async_commit();      // possibly empty: keeps the group count in step
    };
#pragma unroll
    for (int t = 0; t < kSmallStages - 1; ++t) issue(t);
    auto store = [&](int r, int cidx, T v) {
        const long long cb = c_base[r];
        const int col = col0 + cidx;
        if (cb >= 0 && col < pb.Nc) {
            T* dst = pb.C + cb + col;
            *dst = pb.accumulate ? (*dst + v) : v;
        }
    };
    if constexpr (sizeof(T) == 8) {
        double c[2][2][2] = {};      // [k parity][row half][2]
        for (int t = 0; t < num_tiles; ++t) {
            cp_async_wait<kSmallStages - 2>();
            __syncthreads();
            issue(t + kSmallStages - 1);      // refills the stage that every thread left before the barrier
            const double* As = smem + (t % kSmallStages) * gemm_small_stage<T>();
            const double* Bs = As + kSmallBM * S;
            const int n = warp * 8 + (lane >> 2);
#pragma unroll
            for (int kk = 0; kk < kSmallBK; kk += 4) {
                const int k = kk + (lane & 3), par = (kk >> 2) & 1;
                const double b = transB ? Bs[n * S + k] : Bs[k * S + n];
#pragma unroll
                for (int i = 0; i < 2; ++i) dmma_m8n8k4(c[par][i][0], c[par][i][1], As[(i * 8 + (lane >> 2)) * S + k], b);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) store(i * 8 + (lane >> 2), warp * 8 + 2 * (lane & 3) + e, c[0][i][e] + c[1][i][e]);
    } else {
        // two rows and two columns per thread; columns side by side for plain B, 16 apart for transposed B (bank conflicts)
        const int ty = tid >> 4, tx = tid & 15;
        const int n0 = transB ? tx : 2 * tx, n1 = transB ? tx + 16 : 2 * tx + 1;
        float c[2][2] = {};
        for (int t = 0; t < num_tiles; ++t) {
            cp_async_wait<kSmallStages - 2>();
            __syncthreads();
            issue(t + kSmallStages - 1);
            const float* As = reinterpret_cast<const float*>(smem) + (t % kSmallStages) * gemm_small_stage<T>();
            const float* Bs = As + kSmallBM * S;
#pragma unroll
            for (int kk = 0; kk < kSmallBK; kk += 4) {
                const float4 a0 = *reinterpret_cast<const float4*>(&As[ty * S + kk]), a1 = *reinterpret_cast<const float4*>(&As[(ty + 8) * S + kk]);
                const float av[2][4] = {{a0.x, a0.y, a0.z, a0.w}, {a1.x, a1.y, a1.z, a1.w}};
                float bv[2][4];
                if (transB) {
                    const float4 b0 = *reinterpret_cast<const float4*>(&Bs[n0 * S + kk]), b1 = *reinterpret_cast<const float4*>(&Bs[n1 * S + kk]);
                    bv[0][0] = b0.x; bv[0][1] = b0.y; bv[0][2] = b0.z; bv[0][3] = b0.w;
                    bv[1][0] = b1.x; bv[1][1] = b1.y; bv[1][2] = b1.z; bv[1][3] = b1.w;
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float2 b = *reinterpret_cast<const float2*>(&Bs[(kk + q) * S + n0]);
                        bv[0][q] = b.x; bv[1][q] = b.y;
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int j = 0; j < 2; ++j) c[i][j] = fmaf(av[i][q], bv[j][q], c[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) { store(ty + 8 * i, n0, c[i][0]); store(ty + 8 * i, n1, c[i][1]); }
    }
}

// =============================================================================================
// Readouts (MACE::compute_readouts, mace.cpp:876-903 with MultilayerPerceptron::evaluate_gradient,
// multilayer_perceptron.cpp:76-150, hidden width 16): one warp per node.
//   E_i += E0[a] + w1 . H1[i,0,:] + w2 . (s * silu(W1 H2[i]))
//   H1_adj[i,0,:] = w1 ;  H2_adj[i,:] = W1^T (w2 * s * silu'(W1 H2[i]))
// Writes the nodes' whole rows of H1_adj (Hm_adj), zero beyond the scalar part; rows of ghosts are the caller's to clear.
// =============================================================================================
template <typename T>
struct ReadoutArgs {
    int N, K, nLM;
    const int* node_types;
    const double* E0;
    const T* ro1; const T* W1; const T* w2; T scale;
    const T* H1; const T* H2;
    double* node_energies;
    T* H1_adj; T* H2_adj;
    // three-block models: linear readout of the middle block's scalar features (null otherwise)
    const T* ro_m; const T* Hm; T* Hm_adj;
};

// A lane in which warp_reduce_scatter16 leaves value q.
__device__ __forceinline__ constexpr int readout_lane(int q) { return ((q & 8) ? 16 : 0) + ((q & 4) ? 8 : 0) + ((q & 2) ? 4 : 0) + ((q & 1) ? 2 : 0); }

template <typename T>
__global__ void readout_kernel(const ReadoutArgs<T> a) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int warps_total = (gridDim.x * blockDim.x) >> 5;
    for (int i = warp_global; i < a.N; i += warps_total) {
        const T* h1 = a.H1 + static_cast<size_t>(i) * a.nLM * a.K;
        const T* h2 = a.H2 + static_cast<size_t>(i) * a.K;
        T lin = 0;
        T z[16];
#pragma unroll
        for (int h = 0; h < 16; ++h) z[h] = 0;
        for (int k = lane; k < a.K; k += 32) {
            lin += a.ro1[k] * h1[k];
            a.H1_adj[static_cast<size_t>(i) * a.nLM * a.K + k] = a.ro1[k];
            for (int lm = 1; lm < a.nLM; ++lm) a.H1_adj[(static_cast<size_t>(i) * a.nLM + lm) * a.K + k] = T(0);
            if (a.ro_m) {
                lin += a.ro_m[k] * a.Hm[static_cast<size_t>(i) * a.nLM * a.K + k];
                a.Hm_adj[static_cast<size_t>(i) * a.nLM * a.K + k] = a.ro_m[k];
                for (int lm = 1; lm < a.nLM; ++lm) a.Hm_adj[(static_cast<size_t>(i) * a.nLM + lm) * a.K + k] = T(0);
            }
            const T v = h2[k];
#pragma unroll
            for (int h = 0; h < 16; ++h) z[h] += a.W1[h * a.K + k] * v;
        }
        lin = warp_sum(lin);
        // hidden unit h belongs to the lanes that the reduction leaves its sum in (two each): one sigmoid per lane, not sixteen
        int h;
        const T zz = warp_reduce_scatter16(z, lane, h);
        const T sig = T(1) / (T(1) + exp(-zz));
        const T e2 = warp_sum((lane & 1) ? T(0) : a.w2[h] * (a.scale * zz * sig));
        const T gh = a.w2[h] * (a.scale * sig + a.scale * zz * sig * (T(1) - sig));
        T g[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) g[q] = __shfl_sync(0xffffffffu, gh, readout_lane(q));
        if (lane == 0) a.node_energies[i] += a.E0[a.node_types[i]] + double(lin) + double(e2);
        for (int k = lane; k < a.K; k += 32) {
            T s = 0;
#pragma unroll
            for (int h = 0; h < 16; ++h) s += g[h] * a.W1[h * a.K + k];
            a.H2_adj[static_cast<size_t>(i) * a.K + k] = s;
        }
    }
}

// =============================================================================================
// Small structures: everything between the last block's A1 and its adjoint in one launch -- M1, H2, readouts, and the reverse
// of H2 and M1 (compute_M1 .. reverse_M1), all of which act on one node at a time. Each is 6 to 10 us of latency as a launch of its own
// while there are fewer nodes than SMs: start, first loads from L2, a chain of multiply-adds, drain.
//
// A cluster of CTAs per node. Every CTA computes all of M1 (94 coefficients a channel: cheaper again than a cluster barrier),
// its slice of the channels of H2 and that slice's part of the 16 hidden units, which the cluster exchanges through distributed
// shared memory (the one cluster barrier); from the units' gradients every CTA has the whole H2_adj and takes its slice of the
// rows of the transposed products and of A1_adj. dM1/dA1, which does not depend on the adjoint, is computed by the CTA's second half
// while the first computes M1. Bound by L2 latency: a handful of dependent loads and barriers; the weights are split
// over the cluster so that a thread has all of its loads in flight at once. Nine atoms, K = 128, float64: the call takes 157 us
// instead of 172 (see Evaluator::node_cluster for where the line lies).
//
// The steps that sum over channels are functions of their own, because stage calls (and evaluations whose stages are timed) run
// them one launch each (node_features_kernel, node_readout_kernel, node_rows_kernel below): the same sums in the same order, so
// that a sequence of stages gives a whole evaluation bit for bit. M1 and its reverse need no such launch: the contraction kernels
// run the same generated code, the reverse in its LATE form.
// =============================================================================================
template <typename T>
struct NodeHeadArgs {
    PolyArgs<T> poly;             // of the last block (M1)
    ReadoutArgs<T> ro;
    const T* W_M1;                // [K][K]
    const T* W_H1;                // [E][K][K]: residual of the first block's scalar features, by element type
    T* H2; T* M1_adj;
    int slice;                    // channels per CTA of a node
    int ranks;                    // CTAs per node
};
constexpr int kHeadMaxK = 256, kHeadMaxCluster = 8, kHeadMaxSlice = 160;      // (slice: see Evaluator::node_cluster)
// A channel of H2 is a sum of sixteen partial sums over the rows, however many threads share them: the same bits from a cluster's slices
// as from node_features_kernel, whose CTAs take kHeadFine channels each.
constexpr int kHeadParts = 16, kHeadFine = 16;
__host__ __device__ constexpr int node_head_threads(int K) { return K <= 128 ? 256 : 512; }      // two per channel (see below)

// The node of this CTA and its slice of the channels: [k0, k0 + cols). A node's CTAs are consecutive (and a cluster, where they
// exchange anything), and every one of them has channels: see Evaluator::node_cluster.
struct HeadSlice { int i, rank, k0, cols; };
template <typename T>
__device__ __forceinline__ HeadSlice head_slice(const NodeHeadArgs<T>& a) {
    const int i = static_cast<int>(blockIdx.x) / a.ranks, rank = static_cast<int>(blockIdx.x) - i * a.ranks, k0 = rank * a.slice;
    return {i, rank, k0, a.ro.K - k0 < a.slice ? a.ro.K - k0 : a.slice};
}

// This slice of H2 = m1 . W_M1 + prev . W_H1[type], returned by thread (channel - k0). Thread (column, share of the partial sums);
// part: kHeadParts rows of the slice.
template <typename T>
__device__ __forceinline__ T head_features(const NodeHeadArgs<T>& a, const HeadSlice& s, int type, const T* m1, const T* prev, T* part) {
    const int K = a.ro.K, tid = threadIdx.x, nthreads = static_cast<int>(blockDim.x);
    const int c = tid % a.slice, g = tid / a.slice, groups = nthreads / a.slice;
    if (g < groups && c < s.cols) {
        const T* w = a.W_M1 + s.k0 + c;
        const T* r = a.W_H1 + static_cast<size_t>(type) * K * K + s.k0 + c;
        for (int p = g; p < kHeadParts; p += groups) {
            T acc = T(0);
#pragma unroll 8
            for (int j = p; j < K; j += kHeadParts) acc = fma(m1[j], __ldg(w + static_cast<size_t>(j) * K), fma(prev[j], __ldg(r + static_cast<size_t>(j) * K), acc));
            part[p * a.slice + c] = acc;
        }
    }
    __syncthreads();
    T h2 = T(0);
    if (tid < s.cols) {
#pragma unroll
        for (int p = 0; p < kHeadParts; ++p) h2 += part[p * a.slice + tid];
        a.H2[static_cast<size_t>(s.i) * K + s.k0 + tid] = h2;
    }
    return h2;
}

// Readouts of one node by its cluster: `h2` of thread (channel - k0), `prev` the previous block's scalar features. Adds the node's
// energy, leaves the gradients of the hidden units in shared memory for head_features_adjoint. The caller waits at the cluster
// barrier that this function arrives at (other CTAs read this one's shared memory until then).
template <typename T>
struct HeadReadoutShared {
    T units[16][16];                        // [warp][hidden unit]
    T slice_units[16];                      // this slice's part of the hidden units, read by the cluster
    T unit_grad[16];
    T linear;
};
template <typename T>
__device__ __forceinline__ void head_readout(const NodeHeadArgs<T>& a, const HeadSlice& s, int type, T h2, const T* prev, HeadReadoutShared<T>& sh) {
    namespace cg = cooperative_groups;
    auto cl = cg::this_cluster();
    const int K = a.ro.K, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = static_cast<int>(blockDim.x) >> 5;
    T z[16];
#pragma unroll
    for (int h = 0; h < 16; ++h) z[h] = tid < s.cols ? a.ro.W1[h * K + s.k0 + tid] * h2 : T(0);
    if (warp * 32 < a.slice) {
        int h;
        const T sum = warp_reduce_scatter16(z, lane, h);
        if ((lane & 1) == 0) sh.units[warp][h] = sum;
    }
    if (s.rank == 0 && warp == nwarps - 1) {         // the linear readout
        T lin = T(0);
        for (int k = lane; k < K; k += 32) lin = fma(a.ro.ro1[k], prev[k], lin);
        lin = warp_sum(lin);
        if (lane == 0) sh.linear = lin;
    }
    __syncthreads();
    if (tid < 16) {
        T sum = T(0);
        for (int w = 0; w * 32 < a.slice; ++w) sum += sh.units[w][tid];
        sh.slice_units[tid] = sum;
    }
    cl.sync();
    if (warp == 0) {
        const int h = lane & 15;
        T zz = T(0);
        for (int q = 0; q < a.ranks; ++q) zz += *cl.map_shared_rank(&sh.slice_units[h], q);
        const T sig = T(1) / (T(1) + exp(-zz));
        const T e2 = warp_sum(lane < 16 ? a.ro.w2[h] * (a.ro.scale * zz * sig) : T(0));
        if (lane < 16) sh.unit_grad[h] = a.ro.w2[h] * (a.ro.scale * sig + a.ro.scale * zz * sig * (T(1) - sig));
        if (s.rank == 0 && lane == 0) a.ro.node_energies[s.i] += a.ro.E0[type] + double(sh.linear) + double(e2);
    }
    cl.barrier_arrive();        // no more reads of other CTAs' memory
    __syncthreads();
}
// H2_adj[k] from the hidden units' gradients; stored, and the rows of H1_adj beyond the scalars cleared, by the CTA whose channel it is.
template <typename T>
__device__ __forceinline__ T head_features_adjoint(const NodeHeadArgs<T>& a, const HeadSlice& s, const T* unit_grad, int k) {
    const int K = a.ro.K;
    T sum = T(0);
#pragma unroll
    for (int h = 0; h < 16; ++h) sum = fma(unit_grad[h], a.ro.W1[h * K + k], sum);
    if (k >= s.k0 && k < s.k0 + s.cols) {
        a.ro.H2_adj[static_cast<size_t>(s.i) * K + k] = sum;
        for (int lm = 1; lm < a.ro.nLM; ++lm) a.ro.H1_adj[(static_cast<size_t>(s.i) * a.ro.nLM + lm) * K + k] = T(0);
    }
    return sum;
}
// Rows [k0, k0 + cols) of W . H2_adj for both matrices: four rows of a matrix per warp at a time, lanes along the row. Lane 0 to 3
// calls put(residual?, channel, value).
template <typename T, typename Put>
__device__ __forceinline__ void head_rows(const NodeHeadArgs<T>& a, const HeadSlice& s, int type, const T* h2_adj, Put&& put) {
    const int K = a.ro.K, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = static_cast<int>(blockDim.x) >> 5;
    const int quads = (s.cols + 3) / 4;
    for (int q = warp; q < 2 * quads; q += nwarps) {
        const bool residual = q >= quads;
        const int r0 = 4 * (residual ? q - quads : q);
        const T* w = (residual ? a.W_H1 + static_cast<size_t>(type) * K * K : a.W_M1) + static_cast<size_t>(s.k0) * K;
        T sum[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 4
        for (int k = lane; k < K; k += 32) {
            const T g = h2_adj[k];
#pragma unroll
            for (int t = 0; t < 4; ++t) sum[t] = fma(g, __ldg(w + static_cast<size_t>(r0 + t < s.cols ? r0 + t : s.cols - 1) * K + k), sum[t]);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) sum[t] = warp_sum(sum[t]);
        if (lane < 4 && r0 + lane < s.cols) put(residual, s.k0 + r0 + lane, lane == 0 ? sum[0] : lane == 1 ? sum[1] : lane == 2 ? sum[2] : sum[3]);
    }
}

template <typename T>
__global__ void __launch_bounds__(512) node_head_kernel(const NodeHeadArgs<T> a) {
    chain_begin();
    const HeadSlice s = head_slice(a);
    const int i = s.i, k0 = s.k0, cols = s.cols, K = a.ro.K, nLM = a.ro.nLM, tid = threadIdx.x;
    const int nthreads = static_cast<int>(blockDim.x), half = nthreads >> 1;
    const int type = a.ro.node_types[i];
    __shared__ T m1[kHeadMaxK], prev[kHeadMaxK], h2_adj[kHeadMaxK], m1_adj[kHeadMaxSlice], part[kHeadParts * kHeadMaxSlice];
    __shared__ HeadReadoutShared<T> readout;

    // M1 by the first half of the threads; dM1/dA1 of this CTA's slice, kept in registers until the end, by the second half
    PolyVec<T, 1> G[kNumLm];
    const int kg = k0 + tid - half;
    const bool grad_thread = tid >= half && tid - half < cols;
    {
        const int k = tid < half ? tid : kg;
        const bool forward = tid < K && tid < half;
        if (forward || grad_thread) {
            const T* cf = a.poly.coef + static_cast<size_t>(type) * a.poly.num_mono * K + k;
            constexpr int kOff = kCanonPolyOffset[0];
            auto C = [&](int slot) { return PolyVec<T, 1>(__ldg(cf + static_cast<size_t>(kOff + slot) * K)); };
            PolyVec<T, 1> A[kNumLm];
#pragma unroll
            for (int q = 0; q < kNumLm; ++q) A[q].v[0] = a.poly.A[(static_cast<size_t>(i) * kNumLm + q) * K + k];
            if (forward) {
                prev[k] = a.ro.H1[static_cast<size_t>(i) * nLM * K + k];
                using T = PolyVec<std::remove_const_t<std::remove_reference_t<decltype(m1[0])>>, 1>;
#include "generated/poly_lm0_forward.inc"
                m1[k] = total.v[0];
                if (k >= k0 && k < k0 + cols) a.poly.M[static_cast<size_t>(i) * K + k] = total.v[0];
            } else {
#pragma unroll
                for (int q = 0; q < kNumLm; ++q) G[q] = PolyVec<T, 1>(T(0));
                using T = PolyVec<std::remove_const_t<std::remove_reference_t<decltype(m1[0])>>, 1>;
                const T seed(1);
#include "generated/poly_lm0_reverse.inc"
            }
        }
    }
    __syncthreads();
    const T h2 = head_features(a, s, type, m1, prev, part);
    head_readout(a, s, type, h2, prev, readout);
    for (int k = tid; k < K; k += nthreads) h2_adj[k] = head_features_adjoint(a, s, readout.unit_grad, k);
    __syncthreads();
    head_rows(a, s, type, h2_adj, [&](bool residual, int k, T v) {
        if (residual) {
            a.ro.H1_adj[static_cast<size_t>(i) * nLM * K + k] = a.ro.ro1[k] + v;      // linear readout, residual
        } else {
            m1_adj[k - k0] = v;
            a.M1_adj[static_cast<size_t>(i) * K + k] = v;
        }
    });
    __syncthreads();
    if (grad_thread) {
        const T seed = m1_adj[tid - half];
#pragma unroll
        for (int q = 0; q < kNumLm; ++q) a.poly.A_adj[(static_cast<size_t>(i) * kNumLm + q) * K + kg] = seed * G[q].v[0];
    }
    cooperative_groups::this_cluster().barrier_wait();
}

// The steps as launches of their own. Sums over a row's channels (node_rows_kernel) and over the rows (node_features_kernel) do not depend
// on the slices, so these two take small ones, a warp's worth of work per warp: with the cluster's slices they took 13.2 and 9.1 us at
// 144 atoms, K = 128, float64, where the matrix products of larger structures take 8.7 and 7.6. The readout's sums are the cluster's.
template <typename T>
__global__ void __launch_bounds__(16 * kHeadFine) node_features_kernel(const NodeHeadArgs<T> a) {      // compute_H2
    chain_begin();
    const HeadSlice s = head_slice(a);
    const int K = a.ro.K;
    __shared__ T m1[kHeadMaxK], prev[kHeadMaxK], part[kHeadParts * kHeadFine];
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        m1[k] = a.poly.M[static_cast<size_t>(s.i) * K + k];
        prev[k] = a.ro.H1[static_cast<size_t>(s.i) * a.ro.nLM * K + k];
    }
    __syncthreads();
    head_features(a, s, a.ro.node_types[s.i], m1, prev, part);
}
template <typename T>
__global__ void __launch_bounds__(512) node_readout_kernel(const NodeHeadArgs<T> a) {       // compute_readouts
    chain_begin();
    const HeadSlice s = head_slice(a);
    const int K = a.ro.K;
    __shared__ HeadReadoutShared<T> readout;
    const T h2 = static_cast<int>(threadIdx.x) < s.cols ? a.ro.H2[static_cast<size_t>(s.i) * K + s.k0 + threadIdx.x] : T(0);
    head_readout(a, s, a.ro.node_types[s.i], h2, a.ro.H1 + static_cast<size_t>(s.i) * a.ro.nLM * K, readout);
    for (int c = threadIdx.x; c < s.cols; c += blockDim.x) {
        const int k = s.k0 + c;
        head_features_adjoint(a, s, readout.unit_grad, k);
        a.ro.H1_adj[static_cast<size_t>(s.i) * a.ro.nLM * K + k] = a.ro.ro1[k];
    }
    cooperative_groups::this_cluster().barrier_wait();
}
template <typename T>
__global__ void __launch_bounds__(16 * kHeadFine) node_rows_kernel(const NodeHeadArgs<T> a) {          // reverse_H2
    chain_begin();
    const HeadSlice s = head_slice(a);
    const int K = a.ro.K, nLM = a.ro.nLM;
    __shared__ T h2_adj[kHeadMaxK];
    for (int k = threadIdx.x; k < K; k += blockDim.x) h2_adj[k] = a.ro.H2_adj[static_cast<size_t>(s.i) * K + k];
    __syncthreads();
    head_rows(a, s, a.ro.node_types[s.i], h2_adj, [&](bool residual, int k, T v) {
        if (residual) a.ro.H1_adj[static_cast<size_t>(s.i) * nLM * K + k] += v;
        else a.M1_adj[static_cast<size_t>(s.i) * K + k] = v;
    });
}

// =============================================================================================
// ZBL pair repulsion (ZBL::compute_ZBL, zbl.cpp:96-125 with compute / compute_gradient / envelope :22-94):
// screened Coulomb term times a polynomial envelope that vanishes at the sum of the covalent radii. Half of each
// pair energy goes to the receiver's node energy, the radial derivative to the edge's partial force. One thread
// per node walks its row, so the energy sum needs no atomics. Always float64.
// =============================================================================================
struct ZblParams {
    double a_exp, a_prefactor, c[4];
    int p;
    const double* covalent_radii;   // indexed by atomic number
    const int* atomic_numbers;      // per model type
};

// A warp per receiver: 32 lanes test 32 edges at a time, and the few within the sum of the covalent radii (one to four of a
// liquid's fifty) are collected into a list so that the lanes evaluate them side by side, in rounds of 32. Every pow and exp of an
// edge is a long serial chain in float64: bound by that chain, not by bytes. With a thread per receiver, which walked its edges one
// after the other through those chains, 1,029 atoms took 200 us, now 18.
constexpr int kZblThreads = 128;
static __global__ void __launch_bounds__(kZblThreads) zbl_kernel(int N, const int* __restrict__ node_types, const long long* __restrict__ first_neigh,
                           const int* __restrict__ neigh_types, const double* __restrict__ xyz, const double* __restrict__ r,
                           ZblParams z, double* __restrict__ node_energies, double* __restrict__ node_forces) {
    chain_begin();
    const double ce[4] = {-3.2, -0.9423, -0.4028, -0.2016};     // screening exponents, zbl.hpp:49-52
    const double v_prefactor = 14.3996;                          // zbl.hpp:53
    __shared__ int hits[kZblThreads / 32][64];                   // edges of the receiver's row still to be evaluated
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* const list = hits[warp];
    for (int i = (blockIdx.x * kZblThreads + threadIdx.x) >> 5; i < N; i += gridDim.x * (kZblThreads / 32)) {
        const int Zi = z.atomic_numbers[node_types[i]];
        const double radius_i = z.covalent_radii[Zi];
        const long long begin = first_neigh[i], count = first_neigh[i + 1] - begin;
        double e_sum = 0.0;
        int pending = 0;
        for (long long at = 0; at < count || pending > 0; at += 32) {
            bool hit = false;
            if (at + lane < count) {
                const long long e = begin + at + lane;
                hit = !(r[e] >= radius_i + z.covalent_radii[z.atomic_numbers[neigh_types[e]]]);      // envelope and its gradient vanish beyond (zbl.cpp:76,86)
            }
            const unsigned found = __ballot_sync(0xffffffffu, hit);
            if (hit) list[pending + __popc(found & ((1u << lane) - 1u))] = static_cast<int>(at) + lane;
            pending += __popc(found);
            __syncwarp();
            if (pending < 32 && at + 32 < count) continue;        // fewer than a round and more edges to test
            const int now = pending < 32 ? pending : 32;
            if (lane < now) {
                const long long e = begin + list[lane];
                const int Zj = z.atomic_numbers[neigh_types[e]];
                const double rr = r[e];
                const double r_max = radius_i + z.covalent_radii[Zj];
                const double Zu = Zi, Zv = Zj;
                const double a = z.a_prefactor * 0.529 / (pow(Zu, z.a_exp) + pow(Zv, z.a_exp));
                const double roa = rr / a;
                double phi = 0.0, dphi = 0.0;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const double t = z.c[q] * exp(ce[q] * roa);
                    phi += t;
                    dphi += ce[q] * t;
                }
                dphi /= a;
                const double v = v_prefactor * Zu * Zv / rr * phi;
                const double dv = v_prefactor * Zu * Zv * (rr * dphi - phi) / (rr * rr);
                const double x = rr / r_max, p = z.p;
                const double env = 1.0 - ((p + 1.0) * (p + 2.0) / 2.0) * pow(x, p) + p * (p + 2.0) * pow(x, p + 1.0) - (p * (p + 1.0) / 2.0) * pow(x, p + 2.0);
                const double denv = (-((p + 1.0) * (p + 2.0) / 2.0) * p * pow(x, p - 1.0) + p * (p + 2.0) * (p + 1.0) * pow(x, p)
                                     - (p * (p + 1.0) / 2.0) * (p + 2.0) * pow(x, p + 1.0)) / r_max;
                e_sum += 0.5 * v * env;
                const double g = 0.5 * (v * denv + dv * env);
                node_forces[3 * e] -= xyz[3 * e] / rr * g;
                node_forces[3 * e + 1] -= xyz[3 * e + 1] / rr * g;
                node_forces[3 * e + 2] -= xyz[3 * e + 2] / rr * g;
            }
            __syncwarp();
            const int rest = pending - now;                       // at most 31: the list never holds more than 63
            const int moved = lane < rest ? list[32 + lane] : 0;
            __syncwarp();
            if (lane < rest) list[lane] = moved;
            pending = rest;
            __syncwarp();
        }
        e_sum = warp_sum(e_sum);
        if (lane == 0) node_energies[i] += e_sum;
    }
}

// =============================================================================================
// Density normalisation of a layer's A features (MACE::compute_A0_scaled / reverse_A0_scaled and the A1 twins,
// mace.cpp:273-346, 681-757): A[i] /= 1 + sum_j f_ab(r_ij) with one scalar cubic spline per element pair.
// One CTA per node. The reverse pass recomputes the factor, adds dE/dr of the factor to the edge forces and
// scales the adjoint.
// =============================================================================================
struct ScalarSplines {
    const double* coef;   // [pair][bin][4]
    double h;
    int bins, num_elements;
};

__device__ __forceinline__ void scalar_spline(const ScalarSplines& sp, int type_i, int type_j, double rr, double& f, double& d) {
    const int lo = type_i <= type_j ? type_i : type_j, hi = type_i <= type_j ? type_j : type_i;
    const int pair = lo * (2 * sp.num_elements - lo - 1) / 2 + hi;
    int bin = static_cast<int>(rr / sp.h);
    bin = bin < 0 ? 0 : (bin > sp.bins - 1 ? sp.bins - 1 : bin);
    const double x = rr - sp.h * bin;
    const double* c = sp.coef + (static_cast<size_t>(pair) * sp.bins + bin) * 4;
    f = c[0] + c[1] * x + c[2] * x * x + c[3] * x * x * x;
    d = c[1] + 2 * c[2] * x + 3 * c[3] * x * x;
}

__device__ __forceinline__ double block_sum(double v, double* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double t = 0;
    for (int w = 0; w < nw; ++w) t += sh[w];
    return t;
}

template <typename T>
__global__ void density_scale_forward_kernel(int N, int K, const int* __restrict__ node_types, const long long* __restrict__ first_neigh,
                                             const int* __restrict__ neigh_types, const double* __restrict__ r, ScalarSplines sp,
                                             T* __restrict__ A) {
    chain_begin();
    __shared__ double sh[32];
    for (int i = blockIdx.x; i < N; i += gridDim.x) {
        const int ti = node_types[i];
        double part = 0;
        for (long long e = first_neigh[i] + threadIdx.x; e < first_neigh[i + 1]; e += blockDim.x) {
            double f, d;
            scalar_spline(sp, ti, neigh_types[e], r[e], f, d);
            part += f;
        }
        const double factor = 1.0 + block_sum(part, sh);
        T* row = A + static_cast<size_t>(i) * kNumLm * K;
        for (int c = threadIdx.x; c < kNumLm * K; c += blockDim.x) row[c] = static_cast<T>(double(row[c]) / factor);
    }
}

template <typename T>
__global__ void density_scale_reverse_kernel(int N, int K, const int* __restrict__ node_types, const long long* __restrict__ first_neigh,
                                             const int* __restrict__ neigh_types, const double* __restrict__ xyz, const double* __restrict__ r,
                                             ScalarSplines sp, const T* __restrict__ A, T* __restrict__ A_adj, double* __restrict__ node_forces) {
    chain_begin();
    __shared__ double sh[32];
    for (int i = blockIdx.x; i < N; i += gridDim.x) {
        const int ti = node_types[i];
        double part = 0;
        for (long long e = first_neigh[i] + threadIdx.x; e < first_neigh[i + 1]; e += blockDim.x) {
            double f, d;
            scalar_spline(sp, ti, neigh_types[e], r[e], f, d);
            part += f;
        }
        const double factor = 1.0 + block_sum(part, sh);
        const T* arow = A + static_cast<size_t>(i) * kNumLm * K;
        T* grow = A_adj + static_cast<size_t>(i) * kNumLm * K;
        double dot = 0;
        for (int c = threadIdx.x; c < kNumLm * K; c += blockDim.x) dot += double(grow[c]) * double(arow[c]);
        dot = block_sum(dot, sh);
        for (long long e = first_neigh[i] + threadIdx.x; e < first_neigh[i + 1]; e += blockDim.x) {
            double f, d;
            scalar_spline(sp, ti, neigh_types[e], r[e], f, d);
            const double g = dot / factor * d / r[e];
            node_forces[3 * e] += g * xyz[3 * e];
            node_forces[3 * e + 1] += g * xyz[3 * e + 1];
            node_forces[3 * e + 2] += g * xyz[3 * e + 2];
        }
        __syncthreads();
        for (int c = threadIdx.x; c < kNumLm * K; c += blockDim.x) grow[c] = static_cast<T>(double(grow[c]) / factor);
    }
}

// =============================================================================================
// Small helpers
// =============================================================================================
static __global__ void iota_kernel(int n, int* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = i;
}

// offsets[v] = first position in the sorted key array with key >= v, for v = 0..num_values
static __global__ void segment_offsets_kernel(long long n, const int* __restrict__ sorted_keys, int num_values, long long* __restrict__ offsets) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v <= num_values; v += gridDim.x * blockDim.x) {
        long long lo = 0, hi = n;
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if (sorted_keys[mid] < v) lo = mid + 1; else hi = mid;
        }
        offsets[v] = lo;
    }
}
static __global__ void segment_offsets_int_kernel(int n, const int* __restrict__ sorted_keys, int num_values, int* __restrict__ offsets) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v <= num_values; v += gridDim.x * blockDim.x) {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (sorted_keys[mid] < v) lo = mid + 1; else hi = mid;
        }
        offsets[v] = lo;
    }
}

template <typename S, typename D>
__global__ void convert_kernel(long long n, const S* __restrict__ src, D* __restrict__ dst) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n; i += static_cast<long long>(gridDim.x) * blockDim.x)
        dst[i] = static_cast<D>(src[i]);
}

// Per-atom forces from per-edge partial forces, without atomics:
//   f[i] = - sum_{e in row i} nf[e] + sum_{e in in_edges(i)} nf[e]
// (pair_symmetrix/pair_symmetrix_mace.cpp:334-347; symmetrix_calc.py:93-97)
// One warp per atom: lane l takes the edges l, l + 32, ... of the atom's own row and of its incoming list in order, and the
// lanes are combined by a fixed shuffle tree (same bits on every run).
static __global__ void atom_forces_kernel(int rows, int N, const long long* __restrict__ first_neigh, const long long* __restrict__ in_ptr,
                                   const int* __restrict__ in_edge, const double* __restrict__ nf, double* __restrict__ f) {
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int i = blockIdx.x * warps + (threadIdx.x >> 5); i < rows; i += gridDim.x * warps) {
        double fx = 0, fy = 0, fz = 0;
        if (i < N)
            for (long long e = first_neigh[i] + lane; e < first_neigh[i + 1]; e += 32) { fx -= nf[3 * e]; fy -= nf[3 * e + 1]; fz -= nf[3 * e + 2]; }
        for (long long n = in_ptr[i] + lane; n < in_ptr[i + 1]; n += 32) {
            const long long e = in_edge[n];
            fx += nf[3 * e]; fy += nf[3 * e + 1]; fz += nf[3 * e + 2];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            fx += __shfl_down_sync(0xffffffffu, fx, off);
            fy += __shfl_down_sync(0xffffffffu, fy, off);
            fz += __shfl_down_sync(0xffffffffu, fz, off);
        }
        if (lane == 0) { f[3 * i] = fx; f[3 * i + 1] = fy; f[3 * i + 2] = fz; }
    }
}

// ---------------------------------------------------------------------------------------------
// Halo rows of a decomposed run (what the reference's pair style does in pack_forward_comm / unpack_forward_comm /
// pack_reverse_comm / unpack_reverse_comm, pair_symmetrix/pair_symmetrix_mace.cpp:194-238, and as device kernels in
// pair_symmetrix_mace_kokkos.cpp:240-290, 351-367). Rows of `width` values, one thread per value.
//   gather:       buf[m, :]        = array[rows[m], :]
//   scatter:      array[rows[m], :] = buf[m, :]
//   scatter_add:  array[row, :]   += sum of buf[m, :] over the positions m with rows[m] == row, in ascending m
// The reference adds with atomics (order of the additions undefined); here the positions are grouped by row with a
// stable sort (`sorted_rows`, `sorted_pos`) and one thread adds a row's contributions in list order, so two runs give
// the same bits even when a row occurs several times in the list (an atom that is a ghost of the same peer twice).
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void rows_gather_kernel(const T* __restrict__ array, int width, const int* __restrict__ rows, long long total, T* __restrict__ buf) {
    for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total; t += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long m = t / width;
        const int c = static_cast<int>(t - m * width);
        buf[t] = array[static_cast<size_t>(rows[m]) * width + c];
    }
}
template <typename T>
__global__ void rows_scatter_kernel(T* __restrict__ array, int width, const int* __restrict__ rows, long long total, const T* __restrict__ buf) {
    for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total; t += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long m = t / width;
        const int c = static_cast<int>(t - m * width);
        array[static_cast<size_t>(rows[m]) * width + c] = buf[t];
    }
}
template <typename T>
__global__ void rows_scatter_add_kernel(T* __restrict__ array, int width, const int* __restrict__ sorted_rows, const int* __restrict__ sorted_pos,
                                        int n, const T* __restrict__ buf) {
    const long long total = static_cast<long long>(n) * width;
    for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total; t += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int s = static_cast<int>(t / width);
        const int c = static_cast<int>(t - static_cast<long long>(s) * width);
        const int row = sorted_rows[s];
        if (s > 0 && sorted_rows[s - 1] == row) continue;        // not the first list position of this row
        T acc = array[static_cast<size_t>(row) * width + c];
        for (int q = s; q < n && sorted_rows[q] == row; ++q) acc += buf[static_cast<size_t>(sorted_pos[q]) * width + c];
        array[static_cast<size_t>(row) * width + c] = acc;
    }
}

// Block-wise partial sums of {energy, virial xx yy zz xy xz yz}; partials[block][7].
// Virial convention of pair_symmetrix_mace.cpp:349-368.
static __global__ void energy_virial_partial_kernel(int N, long long E, const double* __restrict__ node_energies, const double* __restrict__ xyz,
                                             const double* __restrict__ nf, double* __restrict__ partials) {
    __shared__ double sh[7][256];
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < N; i += stride) v[0] += node_energies[i];
    for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < E; e += stride) {
        const double x = xyz[3 * e], y = xyz[3 * e + 1], z = xyz[3 * e + 2];
        const double fx = nf[3 * e], fy = nf[3 * e + 1], fz = nf[3 * e + 2];
        v[1] += x * fx; v[2] += y * fy; v[3] += z * fz;
        v[4] += 0.5 * (x * fy + y * fx); v[5] += 0.5 * (x * fz + z * fx); v[6] += 0.5 * (y * fz + z * fy);
    }
    for (int c = 0; c < 7; ++c) sh[c][threadIdx.x] = v[c];
    __syncthreads();
    for (int s = blockDim.x >> 1; s > 0; s >>= 1) {
        if (threadIdx.x < s)
            for (int c = 0; c < 7; ++c) sh[c][threadIdx.x] += sh[c][threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x < 7) partials[blockIdx.x * 7 + threadIdx.x] = sh[threadIdx.x][0];
}
// One warp per component (launch with 7 warps): lane l adds the rows l, l + 32, ... in order, then the lanes are combined
// by a fixed shuffle tree, so the sum has the same bits on every run.
static __global__ void energy_virial_final_kernel(int num_blocks, const double* __restrict__ partials, double* __restrict__ out7) {
    const int comp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (comp >= 7) return;
    double s = 0;
    for (int b = lane; b < num_blocks; b += 32) s += partials[b * 7 + comp];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) out7[comp] = s;
}

}  // namespace smx

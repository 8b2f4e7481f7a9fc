// Activation quantisers: the step that feeds the W8A8 GEMMs.  The reference ships none (its benchmark only rounds
// and clamps, benchmark.py:17-18); these follow the package's torch quantisers bit for bit:
//     s = amax / 127  (s = 1 where the block is all zero),  q = clamp(rint(v / s), -127, 127)
// with IEEE division and round-half-even.  Every element is read once with 16-byte loads and written once (5 bytes per fp32
// element, 3 per bf16 element; the row quantiser reads what does not fit its registers twice).
#pragma once

#include <cuda_bf16.h>

#include "ptx.cuh"

namespace gi8 {

constexpr int kQuantThreads = 256;

// First statement of every quantiser: it may have been started while the kernel before it was still running, so nothing
// is read or written before that kernel has ended.  Only then may a dependent kernel start: the GEMM behind a quantiser
// reads its weights without waiting for the quantiser, and must find what the kernel before the quantiser wrote.
// release_late: it may start only as the CTAs end (see the host's release_late).
GI8_DEVICE void quant_dependency(bool release_late = false)
{
    pdl_wait();
    if (!release_late) pdl_launch_dependents();
}

GI8_DEVICE float warp_max(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// q = clamp(rint(v / s)) with the IEEE quotient, at the price of a multiplication for all but one element in
// several thousand: v * r, r an approximate 1/s (one unit in the last place), is within 2^-15 of the correctly rounded
// quotient (|v / s| <= 127: 127 * (2^-23 of r, 2^-24 of the quotient) = 2.3e-5, and 2^-24 of the product where that is rounded
// first, 3.1e-5), so rounding it gives the same integer unless it lies within 7e-5 of a half-integer -- only then is the
// division carried out.
// r is NaN for blocks whose scale is so small or large that 1/s overflows or loses accuracy: every comparison with it
// then fails and all their elements take the division.
struct QuantScale {
    float s, r;
};

GI8_DEVICE QuantScale make_quant_scale(float amax)
{
    QuantScale qs;
    qs.s = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 1.0f;
    asm("rcp.approx.f32 %0, %1;" : "=f"(qs.r) : "f"(qs.s));
    if (!(qs.s > 1e-30f && qs.s < 1e30f)) qs.r = __int_as_float(0x7fffffff);
    return qs;
}

// Arithmetic on packed fp32 pairs: one instruction for two elements; each half rounds like the scalar instruction.
GI8_DEVICE uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
GI8_DEVICE uint64_t sub2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
GI8_DEVICE uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
GI8_DEVICE uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// Largest magnitude of N pairs (NaN ignored, as fmaxf does).
template <int N>
GI8_DEVICE float amax_pairs(const uint64_t* v)
{
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float lo, hi;
        f32x2_split(v[i], lo, hi);
        m = max3_abs(lo, hi, m);
    }
    return m;
}

// Largest magnitude of 16 loaded bytes (NaN ignored).  bf16: on the packed pairs as they came, one instruction for two elements.
template <typename T>
GI8_DEVICE float amax16(const uint4& u);

template <>
GI8_DEVICE float amax16<float>(const uint4& u)
{
    return max3_abs(__uint_as_float(u.x), __uint_as_float(u.y), max3_abs(__uint_as_float(u.z), __uint_as_float(u.w), 0.0f));
}

template <>
GI8_DEVICE float amax16<__nv_bfloat16>(const uint4& u)
{
    // (the magnitudes' maximum with the product of the signs, which the last step drops; it starts at zero, so that two NaN do not meet)
    uint32_t m = 0u;
    asm("max.xorsign.abs.bf16x2 %0, %0, %1;\n\tmax.xorsign.abs.bf16x2 %0, %0, %2;\n\tmax.xorsign.abs.bf16x2 %0, %0, %3;\n\t"
        "max.xorsign.abs.bf16x2 %0, %0, %4;"
        : "+r"(m)
        : "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w));
    return max3_abs(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u), 0.0f);
}

// The exact rule for one element.
GI8_DEVICE int quant_exact(float v, float s)
{
    float t = rintf(__fdiv_rn(v, s));
    t = fminf(fmaxf(t, -127.0f), 127.0f);
    return static_cast<int>(t);
}

GI8_DEVICE uint32_t pack_i8x4(int a, int b, int c, int d)
{
    return (static_cast<uint32_t>(a) & 0xff) | ((static_cast<uint32_t>(b) & 0xff) << 8) |
           ((static_cast<uint32_t>(c) & 0xff) << 16) | ((static_cast<uint32_t>(d) & 0xff) << 24);
}

// Four elements (two pairs) -> four packed int8.  Fast path, full-rate instructions only: v * r + 1.5 * 2^23 in one rounding
// leaves the nearest integer n of v * r in the low mantissa bits, whose low byte is the int8 result; the constant minus that
// is -n as a float, and v * r - n, again in one rounding, the distance for the half-integer test.  |n| <= 127 because
// |v| <= amax, so no clamp.
// The largest of the four distances decides (a NaN among them fails the test): packed arithmetic and three-operand
// maxima make that about 3.5 instructions an element, where scalar ones with a comparison each took seven.
// FUSED = false: the product is rounded first, one packed instruction more for two elements (what the row quantiser takes: see there).
template <bool FUSED = true>
GI8_DEVICE uint32_t quant_pack4(uint64_t v0, uint64_t v1, const QuantScale& qs)
{
    const uint64_t magic = f32x2(12582912.0f, 12582912.0f);
    const uint64_t r2 = f32x2(qs.r, qs.r);
    uint64_t u0, u1, d0, d1;
    if constexpr (FUSED) {
        u0 = fma2(v0, r2, magic), u1 = fma2(v1, r2, magic);
        d0 = fma2(v0, r2, sub2(magic, u0)), d1 = fma2(v1, r2, sub2(magic, u1));
    } else {
        const uint64_t t0 = mul2(v0, r2), t1 = mul2(v1, r2);
        u0 = add2(t0, magic), u1 = add2(t1, magic);
        d0 = sub2(t0, sub2(u0, magic)), d1 = sub2(t1, sub2(u1, magic));
    }
    float a, b, c, d;
    f32x2_split(d0, a, b), f32x2_split(d1, c, d);
    if (max3_abs_nan(max3_abs_nan(a, b, c), d, 0.0f) <= 0.49993f) {
        float x, y, z, w;
        f32x2_split(u0, x, y), f32x2_split(u1, z, w);
        const uint32_t lo = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x0040);
        const uint32_t hi = __byte_perm(__float_as_uint(z), __float_as_uint(w), 0x0040);
        return __byte_perm(lo, hi, 0x5410);
    }
    float x, y, z, w;
    f32x2_split(v0, x, y), f32x2_split(v1, z, w);
    return pack_i8x4(quant_exact(x, qs.s), quant_exact(y, qs.s), quant_exact(z, qs.s), quant_exact(w, qs.s));
}

// 16 loaded bytes as fp32 pairs: four floats, or eight bf16.
template <typename T>
GI8_DEVICE void unpack16(const uint4& u, uint64_t (&v)[8 / sizeof(T)]);

template <>
GI8_DEVICE void unpack16<float>(const uint4& u, uint64_t (&v)[2])
{
    v[0] = f32x2(__uint_as_float(u.x), __uint_as_float(u.y)), v[1] = f32x2(__uint_as_float(u.z), __uint_as_float(u.w));
}

template <>
GI8_DEVICE void unpack16<__nv_bfloat16>(const uint4& u, uint64_t (&v)[4])
{
    v[0] = f32x2(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u));
    v[1] = f32x2(__uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
    v[2] = f32x2(__uint_as_float(u.z << 16), __uint_as_float(u.z & 0xffff0000u));
    v[3] = f32x2(__uint_as_float(u.w << 16), __uint_as_float(u.w & 0xffff0000u));
}

// Maxima over groups of 16 (or 32) consecutive lanes of U = 4 or 8 values per lane, and what the quantiser derives from
// them, at the price of one division per lane instead of U: the butterfly halves the values a lane is in charge of
// while it doubles the lanes each has been reduced over, so that in the end every lane holds the maximum of ONE value
// index, makes its scale, and fetches the others' scales by shuffles.  After the call r[u], s[u] are the scale of value
// u of this lane's group.  Value u is held by the group's lanes with lane % U == bit_reverse(u).
template <int U, int LANES>
GI8_DEVICE void group_scales(float (&m)[U], float (&s)[U], float (&r)[U])
{
    const int lane = threadIdx.x & 31;
    int n = U;
#pragma unroll
    for (int o = 1; o < U; o <<= 1) {
        n >>= 1;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < U / 2; ++i) {
            if (i < n) {
                const float keep = up ? m[i + n] : m[i], give = up ? m[i] : m[i + n];
                m[i] = fmaxf(keep, __shfl_xor_sync(0xffffffffu, give, o));
            }
        }
    }
#pragma unroll
    for (int o = U; o < LANES; o <<= 1) m[0] = fmaxf(m[0], __shfl_xor_sync(0xffffffffu, m[0], o));
    const QuantScale mine = make_quant_scale(m[0]);
    const int first = lane & ~(LANES - 1);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        // the lane whose bits 0, 1, .. are the bits of u from the highest down
        const int src = first + (U == 8 ? ((u >> 2) & 1) | (u & 2) | ((u & 1) << 2) : ((u >> 1) & 1) | ((u & 1) << 1));
        s[u] = __shfl_sync(0xffffffffu, mine.s, src);
        r[u] = __shfl_sync(0xffffffffu, mine.r, src);
    }
}

// 16-byte loads: lane l of a group of LPB = 128 / EPL lanes owns EPL = 16 / sizeof(T) consecutive elements of one
// 128-wide K block, a warp covers 32 / LPB blocks per load, and kQuantUnroll loads are issued before the first is
// used so that enough bytes are in flight to cover the DRAM latency (one block per warp at a time reached a
// quarter of the copy bandwidth).  The loaded 16 bytes stay in registers as they came (four registers per load whatever
// the type) and are unpacked at each use: a byte in flight costs a register byte.  fp32 input takes eight loads per lane,
// bf16 input, which is closer to the bound of instruction issue, four.
// Bound: HBM for fp32 (16384 x 8192: 128 -> 113 us, 6.0 TB/s, 0.91 of the copy bandwidth); for bf16 (103 -> 88 us, 4.6 TB/s, 0.71) no
// single unit; fewer instructions help: maxima on packed bf16 and quant_pack4 with two packed multiply-adds 90.4 -> 85.4 us (another
// machine), 4096 x 14336 40.7 -> 38.6.  Both with the packed arithmetic and one division per lane instead of one or two per block and lane (group_scales).
// a [M,K] (K % EPL == 0, rows 16-byte aligned) -> q int8 [M,K], s fp32 [M, ceil(K/128)].
constexpr int kQuantBlocksPerItem = 8;  // 128-wide blocks per warp and iteration, whatever the type (1 x 8 or 2 x 4)

// Residency: four CTAs per SM (64 registers); five spill the loads of bf16 input, and cost fp32 input a tenth.
template <typename T>
__global__ void __launch_bounds__(kQuantThreads, 4)
quantize_token_block_kernel(const T* __restrict__ a, int8_t* __restrict__ q, float* __restrict__ s, int64_t M, int K,
                            int KB, bool release_late)
{
    quant_dependency(release_late);
    constexpr int EPL = 16 / sizeof(T);   // elements per lane and load
    constexpr int LPB = 128 / EPL;        // lanes per 128-wide block
    constexpr int BPL = 32 / LPB;         // blocks per warp and load
    constexpr int kQuantUnroll = sizeof(T) == 4 ? 8 : 4;  // 16-byte loads per lane in flight
    constexpr int BPI = BPL * kQuantUnroll;  // blocks per warp and iteration
    static_assert(BPI == kQuantBlocksPerItem, "the host sizes the grid by this");
    const int lane = threadIdx.x & 31;
    const int sub = lane / LPB, ll = lane % LPB;
    // Work item = BPI consecutive blocks of one row (one 32-bit division per item instead of one 64-bit division
    // per block: the index arithmetic, not the memory system, bounded the first version of this kernel).
    const uint32_t groups = static_cast<uint32_t>((KB + BPI - 1) / BPI);
    const uint32_t warps_total = gridDim.x * (kQuantThreads / 32);
    const uint32_t items_total = static_cast<uint32_t>(M) * groups;  // the host checks that this fits
    for (uint32_t item = blockIdx.x * (kQuantThreads / 32) + (threadIdx.x >> 5); item < items_total; item += warps_total) {
        const uint32_t row = item / groups;
        const int kb0 = static_cast<int>(item - row * groups) * BPI + sub;   // this lane's block of load 0
        const int col0 = kb0 * 128 + ll * EPL;                               // load u: BPL blocks further per u
        const int64_t off0 = static_cast<int64_t>(row) * K + col0;
        uint4 raw[kQuantUnroll];
#pragma unroll
        for (int u = 0; u < kQuantUnroll; ++u) {
            const bool ok = col0 + u * (BPL * 128) < K;   // also false for blocks past the end of the row
            raw[u] = ok ? __ldg(reinterpret_cast<const uint4*>(a + (off0 + u * (BPL * 128)))) : make_uint4(0u, 0u, 0u, 0u);
        }
        float m[kQuantUnroll], sc[kQuantUnroll], rc[kQuantUnroll];
#pragma unroll
        for (int u = 0; u < kQuantUnroll; ++u) {
            m[u] = amax16<T>(raw[u]);
        }
        group_scales<kQuantUnroll, LPB>(m, sc, rc);
#pragma unroll
        for (int u = 0; u < kQuantUnroll; ++u) {
            const int kb = kb0 + u * BPL;
            if (ll == 0 && kb < KB) s[static_cast<int64_t>(row) * KB + kb] = sc[u];
            if (col0 + u * (BPL * 128) < K) {
                uint64_t v[EPL / 2];
                unpack16<T>(raw[u], v);
                uint32_t w[EPL / 4];
#pragma unroll
                for (int j = 0; j < EPL / 4; ++j) w[j] = quant_pack4(v[2 * j], v[2 * j + 1], QuantScale{sc[u], rc[u]});
                int8_t* dst = q + (off0 + u * (BPL * 128));
                if constexpr (EPL == 8) *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
                else *reinterpret_cast<uint32_t*>(dst) = w[0];
            }
        }
    }
}

// One CTA per row at a time: per-token scale over the whole row.  LOADS 16-byte loads per thread stay in registers between
// the maximum and the quantisation, so that the row is read once; what lies beyond them is read again (it hits L1 or L2).
// The host takes the smallest of 2, 4 and 8 that holds the row (eight: 16384 bf16 or 8192 fp32 elements): registers that
// a short row leaves unused would cost resident CTAs.
// 16384 x 8192, row read twice -> held in registers: fp32 149 -> 102 us (6.6 TB/s), bf16 126 -> 88.5, since then 85.
// Beyond the registers the second read stays: 8192 x 28672 fp32 322 -> 240 us.
// bf16 with eight loads: four CTAs per SM, which the maximum on packed bf16 makes room for (64 registers; without the bound 72 and three
// fit): 4096 x 14336 43.6 -> 39.1 us, 8192 x 28672 208 -> 146.  fp32 with two loads: six (40 registers for 42), 2048 x 2048 6.9 -> 6.4.  The
// other forms are left to the compiler, and fp32 keeps the plain maximum and all of them the rounded product (quant_pack4<false>): with
// bounds everywhere, the nested maximum and the fused product fp32 8192 x 28672 took 250 us for 240, 4096 x 14336 58.0 for 55.8, 4096 x
// 4096 16.7 for 16.1, bf16 4096 x 4096 16.3 for 15.6, 8192 x 28672 151 for 146 (a bound of one CTA per SM: fp32 380).
template <typename T, int LOADS>
__global__ void __launch_bounds__(kQuantThreads, sizeof(T) == 2 ? (LOADS == 8 ? 4 : 0) : (LOADS == 2 ? 6 : 0))
quantize_token_row_kernel(const T* __restrict__ a, int8_t* __restrict__ q, float* __restrict__ s, int64_t M, int K,
                          bool release_late)
{
    quant_dependency(release_late);
    constexpr int EPL = 16 / sizeof(T);
    constexpr int kStep = kQuantThreads * EPL;
    __shared__ float warp_amax[2][kQuantThreads / 32];
    int parity = 0;
    for (int64_t row = blockIdx.x; row < M; row += gridDim.x, parity ^= 1) {
        const T* src = a + row * K;
        const int col0 = threadIdx.x * EPL;
        uint4 raw[LOADS];
#pragma unroll
        for (int u = 0; u < LOADS; ++u)
            raw[u] = col0 + u * kStep < K ? __ldg(reinterpret_cast<const uint4*>(src + col0 + u * kStep)) : make_uint4(0u, 0u, 0u, 0u);
        auto amax_of = [](const uint4& u) {
            if constexpr (sizeof(T) == 2) {
                return amax16<T>(u);
            } else {
                uint64_t v[EPL / 2];
                unpack16<T>(u, v);
                return amax_pairs<EPL / 2>(v);
            }
        };
        float amax = 0.0f;
#pragma unroll
        for (int u = 0; u < LOADS; ++u) amax = fmaxf(amax, amax_of(raw[u]));
        for (int col = col0 + LOADS * kStep; col < K; col += kStep) amax = fmaxf(amax, amax_of(__ldg(reinterpret_cast<const uint4*>(src + col))));
        amax = warp_max(amax);
        // (two sets of slots in turn: one barrier per row is enough)
        if ((threadIdx.x & 31) == 0) warp_amax[parity][threadIdx.x >> 5] = amax;
        __syncthreads();
        float m = warp_amax[parity][threadIdx.x % (kQuantThreads / 32)];
#pragma unroll
        for (int o = kQuantThreads / 64; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const QuantScale sc = make_quant_scale(m);
        if (threadIdx.x == 0) s[row] = sc.s;
        auto put = [&](const uint4& u, int col) {
            uint64_t v[EPL / 2];
            unpack16<T>(u, v);
            int8_t* dst = q + row * K + col;
            if constexpr (EPL == 8) *reinterpret_cast<uint2*>(dst) = make_uint2(quant_pack4<false>(v[0], v[1], sc), quant_pack4<false>(v[2], v[3], sc));
            else *reinterpret_cast<uint32_t*>(dst) = quant_pack4<false>(v[0], v[1], sc);
        };
#pragma unroll
        for (int u = 0; u < LOADS; ++u)
            if (col0 + u * kStep < K) put(raw[u], col0 + u * kStep);
        for (int col = col0 + LOADS * kStep; col < K; col += kStep) put(__ldg(reinterpret_cast<const uint4*>(src + col)), col);
    }
}

// Walsh-Hadamard rotation along K in blocks of H = 2^LOGH (128 <= H <= 8192, H | K) fused with the per-token
// per-128-block quantiser: out = quantise( FWHT_H(row block) * H^-1/2 ).
// The transform is the textbook in-place butterfly, strides h = 1, 2, 4, ... ascending, (a, b) -> (a + b, a - b):
// every output of a stage is ONE fp32 add or subtract of two outputs of the stage before, so the result does not
// depend on which thread computes it and equals a sequential CPU loop bit for bit.
// Rows and blocks are consecutive in memory, so the matrix is one sequence of H-blocks; a unit of 2^LOGU = max(H, 2048)
// elements is held by 2^LOGU / 64 threads (one, two or four warps), 64 elements each, in two arrangements of the index
// bits between which it passes twice through shared memory:
//   L: a thread holds bits 0-2 and the top three (eight runs of eight consecutive elements: loads and stores of a warp
//      are contiguous, a 128-wide block is one run of 16 lanes),
//   M: a thread holds the bits in the middle, 3 .. LOGU - 4 (of the 8192 unit all but bit 3, which is one shuffle in L;
//      of the 2048 unit also bit 10, which has no stage there).
// Stages on bits 0-2 run in L, the middle ones in M, the top ones back in L: four shared-memory accesses an element,
// where a chain of five shuffle stages and up to three shared-memory stages took up to eleven, each with its selects.
// Words are padded and bit 2 of the word index is flipped by bit 5, which makes both arrangements free of bank conflicts.
// Measured, before and after: 2048 x 28672 bf16, H = 4096, 115 -> 56 us (3.1 TB/s); 499 x 8192 fp32, H = 8192, 18.4 -> 8.9 us;
// 4096 x 8192 bf16, H = 128, 137 -> 32 us.  What bounds it now is no single unit either: at 8192 x 8192 bf16 and H = 8192 23
// instructions an element issue on 62 % of the cycles, the load-store pipe (shared memory above all, 3 % of its accesses in conflict) is
// at 46 %, and 96 registers allow five CTAs of four warps.
template <int LOGH>
struct HadamardShape {
    static constexpr int LOGU = LOGH < 11 ? 11 : LOGH;
    static constexpr int THREADS = 1 << (LOGU - 6);           // of one unit
    static constexpr int UNITS = LOGU == 11 ? 4 : 1;          // units of a CTA
    static constexpr int PAD = LOGU == 13 ? 16 : 8;           // words behind each eighth of the unit
    static constexpr int RUN = 8 * THREADS;                   // elements of an eighth
    static constexpr int WORDS = 8 * (RUN + PAD);
};

GI8_DEVICE void butterfly(uint64_t& a, uint64_t& b)
{
    const uint64_t x = a, y = b;
    a = add2(x, y), b = sub2(x, y);
}
GI8_DEVICE void butterfly_inside(uint64_t& a)
{
    float x, y;
    f32x2_split(a, x, y);
    a = f32x2(x + y, x - y);
}

template <typename T, int LOGH>
__global__ void __launch_bounds__(HadamardShape<LOGH>::THREADS * HadamardShape<LOGH>::UNITS)
hadamard_quantize_token_block_kernel(const T* __restrict__ a, int8_t* __restrict__ q, float* __restrict__ s, int64_t total,
                                     float norm)
{
    quant_dependency();
    using S = HadamardShape<LOGH>;
    __shared__ __align__(16) float stage[S::UNITS][S::WORDS];
    const int t = threadIdx.x % S::THREADS;
    const int64_t unit = static_cast<int64_t>(blockIdx.x) * S::UNITS + threadIdx.x / S::THREADS;
    const int64_t first = (unit << S::LOGU) + 8 * t;   // this thread's run j: 8 elements from first + j * RUN on
    auto sync = [] {
        if constexpr (S::THREADS == 32) __syncwarp();
        else __syncthreads();
    };

    uint64_t v[32];  // L: pair p of run j in v[4 j + p]
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int64_t at = first + j * S::RUN;
        uint4 raw[sizeof(T) / 2];
#pragma unroll
        for (int h = 0; h < static_cast<int>(sizeof(T)) / 2; ++h)
            raw[h] = at < total ? __ldg(reinterpret_cast<const uint4*>(a + at) + h) : make_uint4(0u, 0u, 0u, 0u);
        if constexpr (sizeof(T) == 2) {
            unpack16<T>(raw[0], reinterpret_cast<uint64_t(&)[4]>(v[4 * j]));
        } else {
            unpack16<T>(raw[0], reinterpret_cast<uint64_t(&)[2]>(v[4 * j]));
            unpack16<T>(raw[1], reinterpret_cast<uint64_t(&)[2]>(v[4 * j + 2]));
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        uint64_t* w = v + 4 * j;
#pragma unroll
        for (int p = 0; p < 4; ++p) butterfly_inside(w[p]);
        butterfly(w[0], w[1]), butterfly(w[2], w[3]);
        butterfly(w[0], w[2]), butterfly(w[1], w[3]);
    }
    if constexpr (S::LOGU == 13) {  // bit 3: the neighbouring lane's run
        const float sign = (t & 1) ? -1.0f : 1.0f;   // upper: other - mine = fma(-1, mine, other)
        const uint64_t sign2 = f32x2(sign, sign);
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = fma2(sign2, v[i], __shfl_xor_sync(0xffffffffu, v[i], 1));
    }

    float* const base = stage[threadIdx.x / S::THREADS];
    // L: run j, half h (four elements) of this thread
    float* const l0 = base + 8 * t + 4 * ((t >> 2) & 1);
    float* const l1 = base + 8 * t + 4 * (((t >> 2) & 1) ^ 1);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        *reinterpret_cast<ulonglong2*>(l0 + j * (S::RUN + S::PAD)) = make_ulonglong2(v[4 * j], v[4 * j + 1]);
        *reinterpret_cast<ulonglong2*>(l1 + j * (S::RUN + S::PAD)) = make_ulonglong2(v[4 * j + 2], v[4 * j + 3]);
    }
    sync();
    {
        // M: element b of this thread.  Bits 0-2 of the unit's index are t % 8, the rest of t is bit 3 (8192 unit) and
        // the top bits; the flip of bit 2 by bit 5 makes two base addresses.
        constexpr int kBits = S::LOGU == 11 ? 5 : 6;                    // middle bits held
        constexpr int kStride = S::LOGU == 13 ? 16 : 8;                 // words between neighbours
        constexpr int kFlip = S::LOGU == 13 ? 2 : 4;                    // bit of b that is bit 5 of the index
        const int rest = S::LOGU == 13 ? ((t >> 3) & 1) * 8 + (t >> 4) * (S::RUN + S::PAD) : (t >> 3) * (S::RUN + S::PAD);
        float* const m0 = base + (t & 7) + rest;
        float* const m1 = base + ((t & 7) ^ 4) + rest;
        auto word = [&](int e) -> float* {  // e in [0, 64): b and, of the 2048 unit, bit 10
            const int b = e & ((1 << kBits) - 1);
            return ((b & kFlip) ? m1 : m0) + b * kStride + (e >> kBits) * 4 * (S::RUN + S::PAD);
        };
        uint64_t w[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) w[i] = f32x2(*word(2 * i), *word(2 * i + 1));
        constexpr int kFirstBit = S::LOGU == 13 ? 4 : 3;
        constexpr int kStages = LOGH - kFirstBit < kBits ? LOGH - kFirstBit : kBits;
#pragma unroll
        for (int i = 0; i < 32; ++i) butterfly_inside(w[i]);
#pragma unroll
        for (int st = 1; st < kStages; ++st) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if ((i & (1 << (st - 1))) == 0) butterfly(w[i], w[i | (1 << (st - 1))]);
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) f32x2_split(w[i], *word(2 * i), *word(2 * i + 1));
    }
    sync();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(l0 + j * (S::RUN + S::PAD));
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(l1 + j * (S::RUN + S::PAD));
        v[4 * j] = x.x, v[4 * j + 1] = x.y, v[4 * j + 2] = y.x, v[4 * j + 3] = y.y;
    }
    constexpr int kTopStages = LOGH - (S::LOGU - 3) > 0 ? LOGH - (S::LOGU - 3) : 0;
#pragma unroll
    for (int st = 0; st < kTopStages; ++st) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if ((j & (1 << st)) == 0) {
#pragma unroll
                for (int p = 0; p < 4; ++p) butterfly(v[4 * j + p], v[4 * (j | (1 << st)) + p]);
            }
        }
    }
    // normalise, then the quantiser's rule on each 128-wide block (16 consecutive lanes)
    const uint64_t norm2 = f32x2(norm, norm);
    float m[8], sc[8], rc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int p = 0; p < 4; ++p) v[4 * j + p] = mul2(v[4 * j + p], norm2);
        m[j] = amax_pairs<4>(v + 4 * j);
    }
    group_scales<8, 16>(m, sc, rc);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int64_t at = first + j * S::RUN;
        if (at < total) {
            const QuantScale qs{sc[j], rc[j]};
            if ((t & 15) == 0) s[at >> 7] = qs.s;
            *reinterpret_cast<uint2*>(q + at) = make_uint2(quant_pack4(v[4 * j], v[4 * j + 1], qs), quant_pack4(v[4 * j + 2], v[4 * j + 3], qs));
        }
    }
}

}  // namespace gi8

// w4a8_quantize.cuh -- activation rows -> int8 codes in the Xq layout, for rows that allow 16-byte loads.
//
// Byte work: every element is read once and a code is written for it.  A CTA owns a token and keeps what it has read in registers
// between the maximum and the codes; only what exceeds its threads' UN loads is read a second time.  A warp loads 512 neighbouring
// bytes and stores the codes of the same elements, side by side where a token's codes are a row (T = 1).  What bounds a launch of
// few tokens is latency: a trip to HBM, two barriers, and code that runs for the first time and is fetched from L2, so there is
// little of it.  (With codes in groups of eight tokens two tokens a CTA were needed to store whole sectors, and eight CTAs wrote
// into every line: 700 x 4096 binary16 -> 4096 22.7 -> 18.1 us with the GEMM behind it, 100 x 4096 13.4 -> 10.2.)
#pragma once
#include "w4a8_device.h"
#include "w4a8_math.cuh"
#include "w4a8_ptx.cuh"
#include <type_traits>

namespace rkb200 {

// Elements of a lane's 16 bytes.
template <bool HALF> constexpr int PIECE = HALF ? 8 : 4;

// Codes of eight binary16 values.
template <class Word>
__device__ __forceinline__ uint2 codes_of_halves(Word word, const uint4& r, float inv)
{
    float v[8];
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        v[2 * e] = __half2float(__ushort_as_half((uint16_t)(w[e] & 0xffffu)));
        v[2 * e + 1] = __half2float(__ushort_as_half((uint16_t)(w[e] >> 16)));
    }
    return make_uint2(word(v[0], v[1], v[2], v[3], inv), word(v[4], v[5], v[6], v[7], inv));
}

// The block's row pulled towards L2 while the launch in front still runs: only a hint, and L2 is the point of coherence, so whatever the
// producer still writes is what the loads see.  (2000 x 4096 fp32 -> 4096 38.0 us, 36.2; 2048 binary16 34.0, 33.0; the projections of a layer
// of 5120 / 13824 with 16 tokens 74.0, 72.8; rows loaded element by element gain nothing.)
__device__ __forceinline__ void prefetch_row(const void* A, size_t row_bytes)
{
    const char* const row = static_cast<const char*>(A) + blockIdx.x * row_bytes;
    for (size_t at = 32 * threadIdx.x; at < row_bytes; at += 32 * blockDim.x) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + at));
}

// UN: 16-byte loads a thread keeps.  Op: max_of(best, 16 bytes as loaded) -> best; join(best, best) -> best, join_warp over a warp;
// begin(token, best) -> inverse scale, called by one thread of the row's, which writes the scale; word(x0..x3, inverse) -> four
// codes.  SCAN false: the maxima are collected(token).
template <bool HALF, bool SCAN, int UN, class Op>
__device__ __forceinline__ void quantize_rows(const void* A, uint8_t* Xq, int K, int Kp, int T, Op op)
{
    constexpr int EPW = PIECE<HALF>, LPU = 16 / EPW;     // lanes per 16-element unit
    __shared__ uint32_t s_part[16];
    __shared__ float s_inverse;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x, m = blockIdx.x;
    const uint4* const row = reinterpret_cast<const uint4*>(static_cast<const char*>(A) + (size_t)m * K * (16 / EPW));
    const int pieces = K / EPW, padded = Kp / EPW;       // 16-byte pieces of a row: K is a multiple of EPW
    auto load = [&](int piece) { return piece < pieces ? __ldcg(row + piece) : make_uint4(0u, 0u, 0u, 0u); };
    uint4 kept[UN];
    auto fill = [&](int from) {
#pragma unroll
        for (int i = 0; i < UN; ++i) kept[i] = load(from + i * threads);
    };
    fill(tid);
    if (SCAN) {
        uint32_t best = 0;
#pragma unroll
        for (int i = 0; i < UN; ++i) best = op.max_of(best, kept[i]);
        for (int piece = tid + UN * threads; piece < pieces; piece += threads) best = op.max_of(best, load(piece));
        if constexpr (Op::CHECKS)
            if (best >= Op::LEAST_BAD) {
                best = 0;
                for (int piece = tid; piece < pieces; piece += threads) best = op.max_checked(best, load(piece));
            }
        best = op.join_warp(best);
        if (lane == 0) s_part[warp] = best;
        __syncthreads();
        if (tid == 0) {
            uint32_t all = 0;
            for (int w = 0; w < threads >> 5; ++w) all = op.join(all, s_part[w]);
            s_inverse = op.begin(m, all);
        }
    } else if (tid == 0) s_inverse = op.begin(m, op.collected(m));
    __syncthreads();
    const float inv = s_inverse;
    const int mt = m / T, t = m - mt * T;
    uint8_t* const dst = Xq + ((size_t)mt * (Kp / 16) * T + t) * 16;
    for (int from = tid;;) {
#pragma unroll
        for (int i = 0; i < UN; ++i) {
            const int piece = from + i * threads;
            if (piece < padded) {
                const uint4 r = kept[i];
                uint8_t* const to = dst + (uint32_t)(piece / LPU) * (T * 16u) + piece % LPU * EPW;
                if constexpr (HALF) *reinterpret_cast<uint2*>(to) = codes_of_halves([&](float a, float b, float c, float d, float by) { return op.word(a, b, c, d, by); }, r, inv);
                else *reinterpret_cast<uint32_t*>(to) = op.word(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z), __uint_as_float(r.w), inv);
            }
        }
        from += UN * threads;
        if (from >= padded) break;
        fill(from);
    }
}

// ---- what a row's maximum and its elements become: the W4A8 rule and the W8A8 one (the operators' definitions: w4a8_kernels.cu,
// w8a8_kernels.cu)
template <bool HALF>
struct RowQuant {
    float* scales;
    const uint32_t* rowmax;      // collected maxima, or NULL: scanned
    volatile int* bad_word;      // set where a row is rejected
    static __device__ __forceinline__ uint32_t join(uint32_t a, uint32_t b) { return max(a, b); }
    static __device__ __forceinline__ uint32_t join_warp(uint32_t a) { return __reduce_max_sync(0xffffffffu, a); }
    static __device__ __forceinline__ uint32_t max_of(uint32_t best, const uint4& r)
    {
        if constexpr (HALF) {
            // pairs of magnitudes in one word: both halves order like unsigned 16-bit numbers
            uint32_t m = __vmaxu2(__vmaxu2(r.x & 0x7fff7fffu, r.y & 0x7fff7fffu), __vmaxu2(r.z & 0x7fff7fffu, r.w & 0x7fff7fffu));
            return max(best, max(m & 0xffffu, m >> 16));
        }
        return max(max(best, max(r.x & 0x7fffffffu, r.y & 0x7fffffffu)), max(r.z & 0x7fffffffu, r.w & 0x7fffffffu));
    }
    static constexpr bool CHECKS = false;
    static constexpr uint32_t LEAST_BAD = 0xffffffffu;
    // a row's maximum where it was collected and not scanned; the inverse of its scale
    __device__ __forceinline__ uint32_t collected(int m) const { return __ldcg(rowmax + m); }
    __device__ __forceinline__ float begin(int m, uint32_t bits) const
    {
        float maximum;
        int bad;
        if (HALF && !rowmax) {
            bad = bits >= 0x7c00u ? 1 : 0;
            maximum = __half2float(__ushort_as_half((uint16_t)bits));
        } else {
            bad = bits >= 0x7f800000u ? (rowmax ? 2 : 1) : 0;
            maximum = __uint_as_float(bits);
        }
        float s, inv;
        scale_from_max(maximum, bad != 0, s, inv);
        scales[m] = s;
        if (bad) *bad_word = bad;         // (the same value from every bad row of a launch)
        return inv;
    }
    __device__ __forceinline__ uint32_t word(float a, float b, float c, float d, float inv) const
    {
        return quantize4_scaled(a, b, c, d, inv);
    }
};
// round_half_away + clamp of one product; NaN gives +127 like the reference's min/max chain
__device__ __forceinline__ int w8_code(float x, float inv)
{
    const float y = __fmul_rn(x, inv);
    return (y != y) ? 127 : round_clamp(y);
}

// Scale (dynamic scan or the caller's), then codes in the Xq layout, for rows that allow 16-byte loads.
template <bool HALF>
struct W8RowQuant {
    const float* static_scale;   // the caller's, or NULL: scanned
    float* scales;
    // Magnitude bits order like magnitudes; a NaN pattern (above infinity) never raises the maximum.  The top bit says that there is a
    // NaN or an infinity among them.
    static constexpr uint32_t CAREFUL = 0x80000000u, INF = HALF ? 0x7c00u : 0x7f800000u;
    static __device__ __forceinline__ uint32_t join(uint32_t a, uint32_t b) { return max(a & ~CAREFUL, b & ~CAREFUL) | ((a | b) & CAREFUL); }
    static __device__ __forceinline__ uint32_t join_warp(uint32_t a) { return __reduce_max_sync(0xffffffffu, a & ~CAREFUL) | (__any_sync(0xffffffffu, (a & CAREFUL) != 0) ? CAREFUL : 0u); }
    static constexpr bool CHECKS = true;
    static constexpr uint32_t LEAST_BAD = INF;
    static __device__ __forceinline__ uint32_t max_of(uint32_t best, const uint4& r) { return RowQuant<HALF>::max_of(best, r); }
    // for a thread whose maximum is LEAST_BAD or more: its pieces once more
    static __device__ __forceinline__ uint32_t max_checked(uint32_t best, const uint4& r)
    {
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t a = w[i] & (HALF ? 0x7fffu : 0x7fffffffu), b = HALF ? (w[i] >> 16) & 0x7fffu : 0u;
            if (a <= INF) best = join(best, a);
            if (HALF && b <= INF) best = join(best, b);
        }
        return best | CAREFUL;
    }
    __device__ __forceinline__ uint32_t collected(int) const { return 0u; }
    // The sign of the inverse says how its row is rounded: positive, no product is a NaN or rounds beyond 127 (the scale is that of
    // the row, and normal), as in the W4A8 rule; negative, with the checks; a NaN: the scale is not positive (an underflowed maximum),
    // the codes are zeros.
    __device__ __forceinline__ float begin(int m, uint32_t bits) const
    {
        float s;
        const uint32_t magnitude = bits & ~CAREFUL;
        if (static_scale) s = static_scale[m];
        else {
            const float maximum = HALF ? __half2float(__ushort_as_half((uint16_t)magnitude)) : __uint_as_float(magnitude);
            s = maximum > 0.f ? __fdiv_rn(maximum, 127.0f) : 1.0f;
        }
        scales[m] = s;
        if (!(s > 0.f)) return __int_as_float(0x7fffffff);
        const float inv = __frcp_rn(s);
        return static_scale || (bits & CAREFUL) || s < FLT_MIN ? -inv : inv;
    }
    __device__ __forceinline__ uint32_t word(float a, float b, float c, float d, float inv) const
    {
        if (inv > 0.f) return quantize4_scaled(a, b, c, d, inv);
        if (inv != inv) return 0u;
        return __byte_perm(__byte_perm((uint32_t)w8_code(a, -inv), (uint32_t)w8_code(b, -inv), 0x0040),
                           __byte_perm((uint32_t)w8_code(c, -inv), (uint32_t)w8_code(d, -inv), 0x0040), 0x5410);
    }
};

// Rows that do not allow 16-byte loads: a warp takes 512 elements at a time, a lane element 32 i + lane, so that every load
// covers neighbouring elements, and hands them to the lane whose 16-element unit they belong to through shared memory, a word
// per element, units seventeen words apart (no bank conflicts in either direction).  (A thread loading its unit element by
// element touched 32 lines with every load: 193 rows of 3070 fp32 9 us where 3072 values take 5.5.)
constexpr int PIECE_WORDS = 32 * 17;
template <bool HALF>
__device__ __forceinline__ void load_piece(const typename ActType<HALF>::type* row, int k0, int K, int lane, uint32_t (&raw)[16])
{
    using Bits = std::conditional_t<HALF, unsigned short, unsigned int>;
    const Bits* const at = reinterpret_cast<const Bits*>(row) + k0 + lane;
    const int left = K - k0 - lane;
#pragma unroll
    for (int i = 0; i < 16; ++i) raw[i] = 32 * i < left ? (uint32_t)__ldcg(at + 32 * i) : 0u;
}
// The sixteen values of unit `lane` of a piece (between two barriers of the warp).
template <bool HALF>
__device__ __forceinline__ void exchange_piece(uint32_t* words, int lane, const uint32_t (&raw)[16], float (&v)[16])
{
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) words[(2 * i + (lane >> 4)) * 17 + (lane & 15)] = raw[i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const uint32_t w = words[lane * 17 + i];
        v[i] = HALF ? __half2float(__ushort_as_half((uint16_t)w)) : __uint_as_float(w);
    }
}

// 16-byte loads are possible for every row.
template <bool HALF>
inline bool quantize_rows_ok(const void* A, int K) { return (reinterpret_cast<uintptr_t>(A) & 15u) == 0 && K % PIECE<HALF> == 0; }
// Calls f with the shape of the launch: <threads, loads a thread keeps>, a CTA for each token.  The threads' loads just hold the row,
// as far as they go.  Up to 591 tokens (four a SM) all CTAs of up to 256 threads are resident and half the loads on twice the threads
// are faster (with the GEMM behind it, 512 x 8 loads against 128 x 4: 200 x 1024 binary16 11.6 -> 9.7 us, 400 x 2048 fp32 11.0 -> 9.7), but of
// 512 threads only two an SM are, up to 296 tokens; from there on rows that 256 x 8 loads hold take these (512 x 4 against 256 x 8: 350 x
// 5120 fp32 16.4 -> 15.8, 400 x 8192 22.3 -> 21.4, 591 x 8192 24.8 -> 24.6, 400 x 11008 binary16 25.9 -> 25.1).  Longer ones stay, read a second
// time in part (300 x 14336 fp32 27.3 and 27.7, 400 x 14336 33.6 and 32.3), and rows with known maxima, where it hardly matters (FFN of 300 x
// 6144 35.1 and 35.5, of 500 41.7 and 41.2).  Beyond, CTAs in line behind each other: fewer threads a row, more of the row
// each (2000 x 4096 fp32 256 x 4 23.1, 128 x 8 22.6; 3000 x 8192 fp32 512 x 4 50.9, 256 x 8 47.6, 128 x 8 54.1; 3000 x 11008
// binary16 50.1, 47.9 and 50.5).  Short rows: 128 x 4 (2048 x 4096 binary16 18.1 us, 128 x 8 18.6; 700 x 2048 fp32 10.1 and 11.1),
// but many with known maxima, which have less to wait for, 128 x 8 (FFN of 1000 x 2048 28.5 -> 27.6).
template <bool HALF, bool SCAN, class F>
inline auto with_quantize_rows_shape(int M, int K, F f)
{
    using std::integral_constant;
    using I4 = integral_constant<int, 4>;
    using I8 = integral_constant<int, 8>;
    using B128 = integral_constant<int, 128>;
    using B256 = integral_constant<int, 256>;
    using B512 = integral_constant<int, 512>;
    const int bytes = K * (16 / PIECE<HALF>);
    if (bytes <= 8192 && (SCAN || M < 592)) return f(B128{}, I4{});
    if (M < 592) {
        if (bytes <= 16384) return f(B256{}, I4{});
        return SCAN && M > 296 && bytes <= 32768 ? f(B256{}, I8{}) : f(B512{}, I4{});
    }
    return bytes <= 16384 ? f(B128{}, I8{}) : f(B256{}, I8{});
}

} // namespace rkb200

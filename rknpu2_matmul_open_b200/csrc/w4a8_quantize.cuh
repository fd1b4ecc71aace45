// w4a8_quantize.cuh -- activation rows -> int8 codes in the Xq layout, for rows that allow 16-byte loads.
//
// Byte work: every element is read once and a code is written for it.  A CTA owns TG tokens (one or two, neighbours in their
// token tile) and keeps what it has read in registers between the maximum and the codes; only what exceeds a thread's UN loads is
// read a second time.  Lanes are dealt so that both sides move whole sectors: a warp's load covers 512 / TG contiguous bytes
// of each token's row, and the store that follows puts the TG tokens' 16-byte units, which are neighbours in the layout,
// side by side.  (One CTA per token with a thread per 16-element unit loaded every row twice, each load at a stride of 32 or
// 64 bytes, and stored half sectors: 4096 x 14336 fp32 with known maxima 88-98 -> 60 us, 4096 x 4096 fp32 27 -> 21,
// 128 x 11008 half 7.7 -> 5.8, 50 x 8192 fp32 6.8 -> 5.2, each with cold caches and a launch's own 2.5 us.)
#pragma once
#include "w4a8_device.h"
#include "w4a8_math.cuh"
#include "w4a8_ptx.cuh"
#include <type_traits>

namespace rkb200 {

template <bool HALF, int TG>
struct QuantRows {
    static constexpr int EPW = HALF ? 8 : 4;             // elements of a lane's 16 bytes
    static constexpr int LPU = 16 / EPW;                 // lanes per 16-element unit
    static constexpr int UPW = 32 / (LPU * TG);          // units of each token per warp and step
};

// UN: 16-byte loads a thread keeps.  Op: max_of(best, 16 bytes as loaded) -> best; begin(token, best) -> inverse scale, called by one thread per token, which
// also writes the scales; word(y0..y3) -> four codes of products x * inverse.
// SCAN false: the maxima are not needed (begin ignores its argument).
template <bool HALF, int TG, bool SCAN, int UN, class Op>
__device__ __forceinline__ void quantize_rows(const void* A, uint8_t* Xq, int M, int K, int Kp, int T, Op& op)
{
    using Q = QuantRows<HALF, TG>;
    __shared__ uint32_t s_part[16][TG];
    __shared__ float s_inverse[TG];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    const int j = lane % Q::LPU, tg = lane / Q::LPU % TG, u = lane / (Q::LPU * TG);
    const int m0 = blockIdx.x * TG, m = m0 + tg;
    const bool mine = TG == 1 || m < M;
    const uint4* const row = reinterpret_cast<const uint4*>(static_cast<const char*>(A) + (size_t)(mine ? m : m0) * K * (16 / Q::EPW));
    const int pieces = K / Q::EPW;                       // 16-byte pieces of a row: K is a multiple of EPW
    const int units = Kp / 16, step = warps * Q::UPW, first = warp * Q::UPW + u;
    auto load = [&](int unit) {
        const int piece = unit * Q::LPU + j;
        return mine && piece < pieces ? __ldcg(row + piece) : make_uint4(0u, 0u, 0u, 0u);
    };
    uint4 kept[UN];
    auto fill = [&](int from) {
#pragma unroll
        for (int i = 0; i < UN; ++i) kept[i] = load(from + i * step);
    };
    fill(first);
    if (SCAN) {
        uint32_t best = 0;
#pragma unroll
        for (int i = 0; i < UN; ++i) best = op.max_of(best, kept[i]);
        for (int unit = first + UN * step; unit * Q::LPU < pieces; unit += step) best = op.max_of(best, load(unit));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            if (TG == 1 || (o != Q::LPU)) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
        if (lane % Q::LPU == 0 && lane < Q::LPU * TG) s_part[warp][tg] = best;
        __syncthreads();
        if (tid < TG && m0 + tid < M) {
            uint32_t all = 0;
            for (int w = 0; w < warps; ++w) all = max(all, s_part[w][tid]);
            s_inverse[tid] = op.begin(m0 + tid, all);
        }
    } else if (tid < TG && m0 + tid < M) s_inverse[tid] = op.begin(m0 + tid, 0u);
    __syncthreads();
    if (!mine) return;
    const float inv = s_inverse[tg];
    const int mt = m / T, t = m - mt * T;
    uint8_t* const dst = Xq + ((size_t)mt * units * T + t) * 16 + j * Q::EPW;
    for (int from = first;;) {
#pragma unroll
        for (int i = 0; i < UN; ++i) {
            const int unit = from + i * step;
            if (unit < units) {
                const uint4 r = kept[i];
                if constexpr (HALF) {
                    float v[8];
                    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        v[2 * e] = __half2float(__ushort_as_half((uint16_t)(w[e] & 0xffffu)));
                        v[2 * e + 1] = __half2float(__ushort_as_half((uint16_t)(w[e] >> 16)));
                    }
                    *reinterpret_cast<uint2*>(dst + (size_t)unit * T * 16) = make_uint2(op.word(v[0], v[1], v[2], v[3], inv), op.word(v[4], v[5], v[6], v[7], inv));
                } else {
                    *reinterpret_cast<uint32_t*>(dst + (size_t)unit * T * 16) =
                        op.word(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z), __uint_as_float(r.w), inv);
                }
            }
        }
        from += UN * step;
        if (from >= units) break;
        fill(from);
    }
}

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
inline bool quantize_rows_ok(const void* A, int K) { return (reinterpret_cast<uintptr_t>(A) & 15u) == 0 && K % QuantRows<HALF, 1>::EPW == 0; }
// Calls f with the shape of the launch: <tokens per CTA, threads, loads a thread keeps>.
// Rows that are scanned.  Up to 296 tokens (two CTAs of 512 threads an SM, all resident) a token per CTA, and all the
// threads that help with a row work on it.  Up to 591 these CTAs would come in two waves: 256 threads (in front of 4096
// channels 448 x 1024 binary16 13.8 -> 12.1 us, 448 x 4096 fp32 18.4 -> 16.9), but not for long fp32 rows, whose CTAs take
// twice as long then (300 x 11008 -> 4096 28.0 us, 29.5 with 256; FFN of 400 x 8192 54.7 and 56.7). From 592 tokens on
// binary16 rows of up to 4096 elements take 128 threads with two loads and 32 registers, sixteen CTAs an SM (in front of
// 4096 channels 3000 x 1024 32.2 -> 28.8 us, 1024 x 4096 27.3 -> 25.8); the others two tokens per CTA, which make whole
// sectors of codes (6144 and 8192 binary16 -6 to -10 % against a token per CTA).  (The two fp32 forms of eight loads and two
// tokens spill six words.)
// Rows whose maxima are known: two tokens per CTA, up to 591 tokens of 512 threads (FFN of 64 x 1024 -> 2 x 2048 24.2 ->
// 21.6 us, of 591 x 4096 -> 2 x 14336 116 -> 103), beyond of 256 with 32 registers (4096 x 14336 fp32 60 us, 70 with twice
// the registers).  Few long rows want a CTA each (20 x 11008 40.3 us against 42.3,
// 20 x 4096 26.8 against 27.6).
template <bool HALF, bool SCAN, class F>
inline auto with_quantize_rows_shape(int M, int K, F f)
{
    constexpr int EPW = QuantRows<HALF, 1>::EPW;
    using std::integral_constant;
    using I1 = integral_constant<int, 1>;
    using I2 = integral_constant<int, 2>;
    using I4 = integral_constant<int, 4>;
    using I8 = integral_constant<int, 8>;
    using B128 = integral_constant<int, 128>;
    using B256 = integral_constant<int, 256>;
    using B512 = integral_constant<int, 512>;
    if constexpr (!SCAN) {
        if (M >= 592) return f(I2{}, B256{}, I4{});
        return (M <= 296 && K > 8192) || (M < 24 && K >= 4096) ? f(I1{}, B512{}, I8{}) : f(I2{}, B512{}, I8{});
    } else {
        if (M <= 296) return f(I1{}, B512{}, I8{});
        if (M < 592) return HALF || K < 8192 ? f(I1{}, B256{}, I8{}) : f(I1{}, B512{}, I8{});
        if constexpr (HALF) {
            if (K <= 4096) return f(I1{}, B128{}, I2{});
        } else if (K <= 2048) return f(I2{}, B256{}, I4{});
        return K <= 256 * 8 * EPW / 2 ? f(I2{}, B256{}, I8{}) : f(I2{}, B512{}, I8{});
    }
}

} // namespace rkb200

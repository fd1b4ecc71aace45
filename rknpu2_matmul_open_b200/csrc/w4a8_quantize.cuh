// w4a8_quantize.cuh -- activation rows -> int8 codes in the Xq layout, for rows that allow 16-byte loads.
//
// Byte work: every element is read once and a code is written for it.  A CTA owns TG tokens (neighbours in their token
// tile) and keeps what it has read in registers between the maximum and the codes; only what exceeds a thread's UN loads is
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

// 16-byte loads are possible for every row.
template <bool HALF>
inline bool quantize_rows_ok(const void* A, int K, int T) { return (reinterpret_cast<uintptr_t>(A) & 15u) == 0 && K % QuantRows<HALF, 1>::EPW == 0 && T % 2 == 0; }
// Calls f with the shape of the launch: <tokens per CTA, threads, loads a thread keeps>.
// Two tokens per CTA once that leaves two CTAs per SM; below, a token per CTA spreads the rows over more SMs, and all the
// threads that help with a row work on it.  There, four loads a thread and 32 registers where these hold the rows (or nothing
// has to be held): twice the CTAs on an SM, in different phases (4096 x 14336 fp32 with known maxima 70 -> 60 us).
template <bool HALF, bool SCAN, class F>
inline auto with_quantize_rows_shape(int M, int K, F f)
{
    constexpr int EPW = QuantRows<HALF, 1>::EPW;
    using std::integral_constant;
    using I1 = integral_constant<int, 1>;
    using I2 = integral_constant<int, 2>;
    using I4 = integral_constant<int, 4>;
    using I8 = integral_constant<int, 8>;
    using B256 = integral_constant<int, 256>;
    using B512 = integral_constant<int, 512>;
    if (M < 4 * 148) return f(I1{}, B512{}, I8{});
    if (!SCAN || K <= 256 * 4 * EPW / 2) return f(I2{}, B256{}, I4{});
    return K <= 256 * 8 * EPW / 2 ? f(I2{}, B256{}, I8{}) : f(I2{}, B512{}, I8{});
}

} // namespace rkb200

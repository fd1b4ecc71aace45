// w4a8_kernels.cu -- weight repacking, per-token activation quantisation and the
// mma.sync W4A8 GEMM (decode / small-batch path and general fallback) for sm_100a.
//
// Reference behaviour reproduced (paths inside the reference project):
//   quantise_kernel : src/rk_npu_w4a8_quant.cpp:52-85 (scales), :119-121 (codes),
//                     :145-161 (scales from collected row maxima)
//   gemm epilogues  : src/rk_npu_w4a8_output.cpp:70-76 (dequantise),
//                     src/rk_npu_w4a8_swiglu.cpp:12-91 + src/rk_npu_swiglu_fp32_neon.h:13-51
//   pack_weights    : src/rk_npu_w4a8.cpp:236-242 (code range check); layout is new.
#include "w4a8_device.h"
#include "w4a8_host.h"
#include "w4a8_ptx.cuh"
#include "w4a8_math.cuh"
#include "w4a8_quantize.cuh"
#include <cuda_fp16.h>
#include <float.h>

namespace rkb200 {

// =============================================================== weight repacking
// One thread builds one 32-bit word of the packed layout: eight codes of one output
// channel.  Consecutive threads take consecutive channels so the reads of B[k, :] are
// coalesced; the 4-byte writes of a warp land 16 bytes apart and are merged in L2.
__global__ void __launch_bounds__(256) pack_weights_kernel(const PackParams p)
{
    const long long total = (long long)p.NG * p.KC * 4 * GROUP;
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int r = (int)(idx % GROUP);
    long long rest = idx / GROUP;
    const int j = (int)(rest % 4);
    rest /= 4;
    const int c = (int)(rest % p.KC);
    const int g = (int)(rest / p.KC);
    const int n = g * GROUP + r;
    uint32_t word = 0;
    int bad = 0;
    if (n < p.N) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int k_lo = c * 32 + 4 * j + b, k_hi = k_lo + 16;
            int lo = 0, hi = 0;
            if (k_lo < p.K) lo = p.B[(size_t)k_lo * p.N + n];
            if (k_hi < p.K) hi = p.B[(size_t)k_hi * p.N + n];
            bad |= (lo < -8) | (lo > 7) | (hi < -8) | (hi > 7);
            word |= (uint32_t)((lo & 15) | ((hi & 15) << 4)) << (8 * b);
        }
    }
    if (bad) atomicOr(p.error, 1);
    reinterpret_cast<uint32_t*>(p.Wp)[(((size_t)g * p.KC + c) * GROUP + r) * 4 + j] = word;
}

cudaError_t launch_pack_weights(const PackParams& p, cudaStream_t stream)
{
    const long long total = (long long)p.NG * p.KC * 4 * GROUP;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    pack_weights_kernel<<<blocks, 256, 0, stream>>>(p);
    return cudaGetLastError();
}

// =============================================================== activation quantisation
// Pass 1: max |x| over the full row on the raw bit patterns (for binary16 and fp32 alike the
// magnitude bits order like the magnitudes, and anything at or above the infinity pattern is
// NaN/Inf).  Pass 2: q = clamp(round_half_away(x * inverse), -127, 127), written as 16-byte units of
// the Xq layout.  Rows that allow 16-byte loads: quantize_rows (w4a8_quantize.cuh).
template <bool HALF, bool SCAN, int BS, int UN>
__global__ void __launch_bounds__(BS, (UN <= 4 ? 1280 : 896) / BS) quantize_rows_kernel(const QuantParams p)
{
    pdl_launch_dependents();   // the GEMM behind this kernel may start prefetching weights
    if (SCAN) prefetch_row(p.A, (size_t)p.K * (HALF ? 2 : 4));
    pdl_wait();                // A may be the output of the kernel in front of this one
    quantize_rows<HALF, SCAN, UN>(p.A, p.Xq, p.K, p.Kp, p.T, RowQuant<HALF>{p.scales, p.rowmax, &p.status->bad_accum});
}

// Any row: one CTA per token.
template <bool HALF>
__global__ void __launch_bounds__(256, 6) quantize_kernel(const QuantParams p)
{
    constexpr int BS = 256;
    using T = typename ActType<HALF>::type;
    pdl_launch_dependents();   // the GEMM behind this kernel may start prefetching weights
    pdl_wait();                // A may be the output of the kernel in front of this one
    const int m = blockIdx.x, tid = threadIdx.x;
    const T* row = reinterpret_cast<const T*>(p.A) + (size_t)m * p.K;
    const int lane = tid & 31, first = tid & ~31;   // units of this warp: 32 from `first` on, and every BS further
    const int chunks = p.Kp / 16;
    __shared__ uint32_t s_words[BS / 32][PIECE_WORDS];
    __shared__ uint32_t s_part[BS / 32];
    __shared__ float s_inverse;

    uint32_t maxbits = 0;
    int bad = 0;
    if (p.rowmax == nullptr) {
        for (int u = first; u * 16 < p.K; u += BS) {
            uint32_t raw[16];
            load_piece<HALF>(row, u * 16, p.K, lane, raw);
#pragma unroll
            for (int i = 0; i < 16; ++i) maxbits = max(maxbits, raw[i] & (HALF ? 0x7fffu : 0x7fffffffu));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) maxbits = max(maxbits, __shfl_xor_sync(0xffffffffu, maxbits, o));
        if ((tid & 31) == 0) s_part[tid >> 5] = maxbits;
        __syncthreads();
        if (tid == 0) {
            uint32_t mx = 0;
#pragma unroll
            for (int i = 0; i < BS / 32; ++i) mx = max(mx, s_part[i]);
            float maximum;
            if constexpr (HALF) {
                bad = mx >= 0x7c00u ? 1 : 0;
                maximum = __half2float(__ushort_as_half((uint16_t)mx));
            } else {
                bad = mx >= 0x7f800000u ? 1 : 0;
                maximum = __uint_as_float(mx);
            }
            const float s = (maximum == 0.f || bad) ? 1.0f : fmaxf(__fdiv_rn(maximum, 127.0f), FLT_MIN);
            const float inv = __fdiv_rn(1.0f, s);
            p.scales[m] = s;
            s_inverse = inv;
        }
    } else if (tid == 0) {
        const uint32_t bits = p.rowmax[m];
        bad = bits >= 0x7f800000u ? 2 : 0;
        const float maximum = __uint_as_float(bits);
        const float s = (maximum == 0.f || bad) ? 1.0f : fmaxf(__fdiv_rn(maximum, 127.0f), FLT_MIN);
        const float inv = __fdiv_rn(1.0f, s);
        p.scales[m] = s;
        s_inverse = inv;
    }
    __syncthreads();
    const float inv = s_inverse;
    const int mt = m / p.T, t = m - mt * p.T;
    uint4* dst = reinterpret_cast<uint4*>(p.Xq) + ((size_t)mt * chunks) * p.T + t;
    for (int u = first; u < chunks; u += BS) {
        uint32_t raw[16];
        float v[16];
        load_piece<HALF>(row, u * 16, p.K, lane, raw);
        exchange_piece<HALF>(s_words[tid >> 5], lane, raw, v);
        const int kc = u + lane;
        if (kc < chunks) dst[(size_t)kc * p.T] = kc * 16 < p.K ? quantize16(v, inv, kc * 16, p.K) : make_uint4(0u, 0u, 0u, 0u);
    }
    if (tid == 0) {
        if (bad) p.status->bad_accum = bad;     // (the same value from every bad row of a launch)
    }
}

template <bool HALF, bool SCAN>
static cudaError_t launch_quantize_rows(const QuantParams& p, cudaLaunchConfig_t& cfg)
{
    return with_quantize_rows_shape<HALF, SCAN>(p.M, p.K, [&](auto bs, auto un) {
        constexpr int BS = decltype(bs)::value, UN = decltype(un)::value;
        cfg.gridDim = dim3((unsigned)p.M);
        cfg.blockDim = dim3((unsigned)BS);
        return cudaLaunchKernelEx(&cfg, quantize_rows_kernel<HALF, SCAN, BS, UN>, p);
    });
}

cudaError_t launch_quantize(const QuantParams& p, cudaStream_t stream, bool pdl)
{
    cudaLaunchConfig_t cfg = {};
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cfg.dynamicSmemBytes = 0;
    const bool scan = p.rowmax == nullptr;      // (collected maxima come with an fp32 middle)
    if (!(p.half ? scan && quantize_rows_ok<true>(p.A, p.K) : quantize_rows_ok<false>(p.A, p.K))) {
        cfg.gridDim = dim3((unsigned)p.M);
        cfg.blockDim = dim3(256);
        return p.half ? cudaLaunchKernelEx(&cfg, quantize_kernel<true>, p) : cudaLaunchKernelEx(&cfg, quantize_kernel<false>, p);
    }
    if (p.half) return launch_quantize_rows<true, true>(p, cfg);
    return scan ? launch_quantize_rows<false, true>(p, cfg) : launch_quantize_rows<false, false>(p, cfg);
}

// =============================================================== mma.sync GEMM
// Output-stationary, swap-AB: the 128 output channels of a CTA are the M side of
// mma.m16n8k32 (weights = A fragments built from the packed nibbles with three ALU
// instructions per eight codes), the tokens are the N side (8 per instruction).
// One producer thread streams weight and activation k-blocks with bulk async copies
// into a ring of stages; four consumer warps (one weight group each) do the math.
// Split-K runs as a thread-block cluster along y: partial sums are exchanged through
// distributed shared memory, each rank finishing a slice of the channels.
// Behind the contraction every access is a trip: the channels' scales are asked for before the wait for the kernel in front, the
// tokens' before the contraction, and a thread asks all ranks for their sums at once.  (One after the other, and the scales at the
// end: 16 x 4096 -> 4096 binary16 7.4 us against 7.2, 24 x 1024 -> 3000 6.7 against 6.2, the projections of a layer of 2048 / 5632
// with 16 tokens 44.7 against 42.8.)  The turns of this part are not unrolled: code that runs once is fetched from L2, which made
// 64 x 2048 -> 1000 7.5 us instead of 7.1; sums stored to the rank that finishes them, word by word with st.async, 8.5 at 16 x 4096.
constexpr int MMA_STAGES = 8;
constexpr int RED_STRIDE = 132;   // int32 words per token row of the reduction buffer

__host__ __device__ constexpr int mma_stage_bytes(int tc) { return 4 * 2048 + 128 * tc; }
__host__ __device__ constexpr size_t mma_smem_bytes(int tc)
{
    return (size_t)MMA_STAGES * mma_stage_bytes(tc) + (size_t)tc * RED_STRIDE * 4 + 2 * MMA_STAGES * 8 + 16;
}
size_t gemm_mma_smem_bytes(int tokens_per_cta) { return mma_smem_bytes(tokens_per_cta); }

template <int NT, bool BIGK>
__global__ void __launch_bounds__(160, 1) gemm_mma_kernel(const GemmParams p)
{
    constexpr int TC = 8 * NT;
    constexpr int XB = 128 * TC;
    constexpr int STAGE = mma_stage_bytes(TC);
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* const stages = smem;
    int32_t* const red = reinterpret_cast<int32_t*>(smem + MMA_STAGES * STAGE);
    uint64_t* const full = reinterpret_cast<uint64_t*>(smem + MMA_STAGES * STAGE + TC * RED_STRIDE * 4);
    uint64_t* const empty = full + MMA_STAGES;
    __shared__ int s_verdict;
    __shared__ float s_sx[TC];

    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x, rank = blockIdx.y, S = p.split;
    const int tok0 = blockIdx.z * TC;
    const bool swiglu = p.epi == EPI_SWIGLU;
    const int KC = p.KB * 4;
    const int kb0 = (int)(((long long)p.KB * rank) / S), kb1 = (int)(((long long)p.KB * (rank + 1)) / S);
    const int nkb = kb1 - kb0;
    const unsigned long long deadline = global_ns() + p.timeout_ns;

    if (tid == 0) {
        for (int s = 0; s < MMA_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 4); }
        mbar_fence_init();
    }
    __syncthreads();
    // What a thread finishes: four channels of this rank's share (SwiGLU: of the gate, and the same of up), 128 / IPT tokens apart.
    const int CH = (swiglu ? 64 : TILE_N) / S;
    const int IPT = CH / 4, first_token = tid / IPT, c4 = (tid - first_token * IPT) * 4;
    const int columns = swiglu ? p.F : p.N;
    const int n0 = swiglu ? tile * 64 + rank * CH + c4 : tile * TILE_N + rank * CH + c4;
    float sw[4], sw_up[4];
    if (warp < 4) {      // scales of channels never change
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            sw[e] = n0 + e < columns ? p.sw[n0 + e] : 0.f;
            sw_up[e] = swiglu && n0 + e < p.F ? p.sw[p.F + n0 + e] : 0.f;
        }
    }

    int acc[2][NT][4];
    int hi[BIGK ? 2 : 1][BIGK ? NT : 1][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[a][j][e] = 0;
    if constexpr (BIGK) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) hi[a][j][e] = 0;
    }

    if (warp == 4) {
        if (lane == 0) {
            // ---------------- producer
            int group[4];
#pragma unroll
            for (int w = 0; w < 4; ++w)
                group[w] = swiglu ? (w < 2 ? tile * 2 + w : p.F / GROUP + tile * 2 + (w - 2)) : tile * 4 + w;
            const int mt = tok0 / p.T, r0 = tok0 - mt * p.T;
            const size_t kc16_total = (size_t)p.KB * 8;
            auto copy_w = [&](int it, int s) {
#pragma unroll
                for (int w = 0; w < 4; ++w)
                    bulk_g2s(stages + (size_t)s * STAGE + w * 2048,
                             p.Wp + ((size_t)group[w] * KC + (size_t)(kb0 + it) * 4) * 512, 2048, &full[s]);
            };
            auto copy_x = [&](int it, int s) {
                uint8_t* dst = stages + (size_t)s * STAGE + 8192;
                const size_t kc16 = (size_t)(kb0 + it) * 8;
                if (p.T == TC) {
                    bulk_g2s(dst, p.Xq + ((size_t)mt * kc16_total + kc16) * p.T * 16, XB, &full[s]);
                } else {
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        bulk_g2s(dst + c * TC * 16, p.Xq + (((size_t)mt * kc16_total + kc16 + c) * p.T + r0) * 16,
                                 TC * 16, &full[s]);
                }
            };
            const int pre = nkb < MMA_STAGES ? nkb : MMA_STAGES;
            // Weights never change, so their first stages are requested before waiting
            // for the kernel in front (which produces the activation codes).
            for (int it = 0; it < pre; ++it) { mbar_expect_tx(&full[it], 8192); copy_w(it, it); }
            pdl_wait();
            for (int it = 0; it < pre; ++it) { mbar_arrive_expect_tx(&full[it], XB); copy_x(it, it); }
            for (int it = pre; it < nkb; ++it) {
                const int s = it % MMA_STAGES;
                if (!mbar_wait(&empty[s], ((it / MMA_STAGES) - 1) & 1, deadline)) {
                    report_device_error(p.report);
                    break;
                }
                mbar_arrive_expect_tx(&full[s], STAGE);
                copy_w(it, s);
                copy_x(it, s);
            }
        }
        __syncwarp();
    } else {
        // ---------------- consumers: warp w owns weight group w (32 channels = two m16 tiles)
        pdl_wait();
        // (the contraction does not wait for the verdict: only the results depend on it)
        if (tid == 0) s_verdict = take_verdict(p.status, p.report);
        const float sx_own = tid < TC && tok0 + tid < p.M ? __ldcg(p.sx + tok0 + tid) : 0.f;     // (on its way while the contraction runs)
        if ((blockIdx.x | blockIdx.y | blockIdx.z) == 0) clear_maxima(p.rowmax_in, p.M, tid, 128);
        const int g8 = lane >> 2, t4 = lane & 3;
        for (int it = 0; it < nkb; ++it) {
            const int s = it % MMA_STAGES;
            if (!mbar_wait(&full[s], (it / MMA_STAGES) & 1, deadline)) {
                if (lane == 0) report_device_error(p.report);
                break;
            }
            {
                const uint32_t wbase = smem_u32(stages + (size_t)s * STAGE + warp * 2048) + g8 * 16 + t4 * 4;
                const uint32_t xbase = smem_u32(stages + (size_t)s * STAGE + 8192) + g8 * 16 + t4 * 4;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t a[2][4];
#pragma unroll
                    for (int mtile = 0; mtile < 2; ++mtile) {
                        const uint32_t w0 = lds32(wbase + (c * 32 + mtile * 16) * 16);
                        const uint32_t w1 = lds32(wbase + (c * 32 + mtile * 16 + 8) * 16);
                        a[mtile][0] = (w0 << 4) & 0xF0F0F0F0u;
                        a[mtile][1] = (w1 << 4) & 0xF0F0F0F0u;
                        a[mtile][2] = w0 & 0xF0F0F0F0u;
                        a[mtile][3] = w1 & 0xF0F0F0F0u;
                    }
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        const uint32_t b0 = lds32(xbase + ((2 * c) * TC + 8 * j) * 16);
                        const uint32_t b1 = lds32(xbase + ((2 * c + 1) * TC + 8 * j) * 16);
                        mma_s8(acc[0][j], a[0][0], a[0][1], a[0][2], a[0][3], b0, b1);
                        mma_s8(acc[1][j], a[1][0], a[1][1], a[1][2], a[1][3], b0, b1);
                    }
                }
                if constexpr (BIGK) {
                    // 16*|sum| stays below 2^31 for 512 k-blocks; fold the exact quotient away.
                    if ((it & 511) == 511) {
#pragma unroll
                        for (int a = 0; a < 2; ++a)
#pragma unroll
                            for (int j = 0; j < NT; ++j)
#pragma unroll
                                for (int e = 0; e < 4; ++e) { hi[a][j][e] += acc[a][j][e] >> 4; acc[a][j][e] = 0; }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
        }
        if (tid < TC) s_sx[tid] = sx_own;
        // partial sums -> reduction buffer [token][channel]
#pragma unroll
        for (int mtile = 0; mtile < 2; ++mtile)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    int v = acc[mtile][j][e] >> 4;
                    if constexpr (BIGK) v += hi[mtile][j][e];
                    const int ch = warp * 32 + mtile * 16 + g8 + (e >> 1) * 8;
                    const int tok = 8 * j + 2 * t4 + (e & 1);
                    red[tok * RED_STRIDE + ch] = v;
                }
    }
    __syncthreads();
    if (S > 1) { cluster_arrive(); cluster_wait(); }
    const uint32_t sums = smem_u32(red);

    if (warp < 4 && !s_verdict) {
#pragma unroll 1
        for (int tok = first_token; tok - first_token < TC; tok += 128 / IPT) {      // (the same turns for all threads)
            const int m = tok0 + tok;
            const bool finish = tok < TC && m < p.M && n0 < columns;      // only what is stored is asked for, see the end
            int v[4] = {}, u[4] = {};
            if (finish) {
                const uint32_t at = sums + (uint32_t)(tok * RED_STRIDE + rank * CH + c4) * 4u;
                auto add = [&](uint32_t at, int (&to)[4]) {
                    int4 a[8];           // all ranks' sums on their way at once
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q < S) a[q] = lds128_cluster(S > 1 ? map_to_cta(at, (uint32_t)q) : at);
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q < S) { to[0] += a[q].x; to[1] += a[q].y; to[2] += a[q].z; to[3] += a[q].w; }
                };
                add(at, v);
                if (swiglu) add(at + 256u, u);
            }
            const float sx = finish ? s_sx[tok] : 0.f;
            if (!swiglu) {
                if (finish) {
                    if (p.epi == EPI_I32) {
                        int* out = reinterpret_cast<int*>(p.out) + (size_t)m * p.N + n0;
                        if (n0 + 3 < p.N && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) *reinterpret_cast<int4*>(out) = make_int4(v[0], v[1], v[2], v[3]);
                        else for (int e = 0; e < 4; ++e) if (n0 + e < p.N) out[e] = v[e];
                    } else {
                        float y[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) y[e] = dequant(v[e], sx, sw[e]);
                        if (p.epi == EPI_F32) {
                            float* out = reinterpret_cast<float*>(p.out) + (size_t)m * p.N + n0;
                            if (n0 + 3 < p.N && (reinterpret_cast<uintptr_t>(out) & 15u) == 0)
                                *reinterpret_cast<float4*>(out) = make_float4(y[0], y[1], y[2], y[3]);
                            else for (int e = 0; e < 4; ++e) if (n0 + e < p.N) out[e] = y[e];
                        } else {
                            __half* out = reinterpret_cast<__half*>(p.out) + (size_t)m * p.N + n0;
                            if (n0 + 3 < p.N && (reinterpret_cast<uintptr_t>(out) & 7u) == 0) {
                                const __half2 h0 = __halves2half2(__float2half_rn(y[0]), __float2half_rn(y[1]));
                                const __half2 h1 = __halves2half2(__float2half_rn(y[2]), __float2half_rn(y[3]));
                                uint2 pk;
                                pk.x = *reinterpret_cast<const uint32_t*>(&h0);
                                pk.y = *reinterpret_cast<const uint32_t*>(&h1);
                                *reinterpret_cast<uint2*>(out) = pk;
                            } else for (int e = 0; e < 4; ++e) if (n0 + e < p.N) out[e] = __float2half_rn(y[e]);
                        }
                    }
                }
            } else {
                uint32_t mx = 0;
                if (finish) {
                    float y[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float g = dequant(v[e], sx, sw[e]);
                        const float up = dequant(u[e], sx, sw_up[e]);
                        y[e] = __fmul_rn(silu_poly(g), up);
                        mx = max(mx, __float_as_uint(y[e]) & 0x7fffffffu);
                    }
                    float* out = reinterpret_cast<float*>(p.out) + (size_t)m * p.F + n0;
                    if ((reinterpret_cast<uintptr_t>(out) & 15u) == 0) *reinterpret_cast<float4*>(out) = make_float4(y[0], y[1], y[2], y[3]);
                    else for (int e = 0; e < 4; ++e) out[e] = y[e];
                }
                if (p.rowmax) {
                    // lanes of an aligned group of IPT share the token: one atomic per group
                    for (int o = 1; o < IPT && o < 32; o <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    if ((lane & (IPT - 1) & 31) == 0 && mx) atomicMax(&p.rowmax[m], mx);
                }
            }
        }
    }
    // Nobody leaves while a peer may still read its sums.  A relaxed arrival does not wait for loads, so no load may be on its way here:
    // each one's sums went into a store above, which needed them.
    if (S > 1) {
        __syncwarp();
        cluster_arrive_relaxed();
        cluster_wait();
    }
}

template <int NT, bool BIGK>
static cudaError_t launch_mma_inst(const GemmParams& p, cudaStream_t stream, bool pdl)
{
    constexpr int TC = 8 * NT;
    const size_t smem = mma_smem_bytes(TC);
    static PerDeviceOnce configured;
    int configured_device = -1;
    auto kernel = gemm_mma_kernel<NT, BIGK>;
    if (configured.needed(configured_device)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured.mark(configured_device);
    }
    const int tiles = p.epi == EPI_SWIGLU ? (p.F + 63) / 64 : (p.N + TILE_N - 1) / TILE_N;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tiles, (unsigned)p.split, (unsigned)((p.M + TC - 1) / TC));
    cfg.blockDim = dim3(160);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = 1;
    attr[n].val.clusterDim.y = (unsigned)p.split;
    attr[n].val.clusterDim.z = 1;
    ++n;
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

cudaError_t launch_gemm_mma(const GemmParams& p, int tokens_per_cta, cudaStream_t stream, bool pdl)
{
    if (p.split != 1 && p.split != 2 && p.split != 4 && p.split != 8) return cudaErrorInvalidValue;
    if (p.T % tokens_per_cta) return cudaErrorInvalidValue;
    const bool big = (long long)p.KB * KBLOCK > 131072;
    switch (tokens_per_cta) {
    case 8: return big ? launch_mma_inst<1, true>(p, stream, pdl) : launch_mma_inst<1, false>(p, stream, pdl);
    case 16: return big ? launch_mma_inst<2, true>(p, stream, pdl) : launch_mma_inst<2, false>(p, stream, pdl);
    case 32: return big ? launch_mma_inst<4, true>(p, stream, pdl) : launch_mma_inst<4, false>(p, stream, pdl);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace rkb200

// =============================================================== linear without any allocation
// Some callers may not allocate at the moment they need a linear: an inference engine that
// sized its one device pool at start-up and forbids cudaMalloc afterwards, a plugin running
// inside somebody else's real-time loop, code on a path where an allocation (and the implicit
// device synchronisation cudaMalloc and cudaFree bring) is not acceptable.  A workspace is
// what normally owns the scratch of a call -- the quantised activation codes, the per-token
// scales and the status word -- and creating one allocates.  The entry point below runs the
// same two kernels as a small-batch workspace (quantise, then the mma.sync split-K GEMM) with
// that scratch in a fixed array that is part of the library image, so the call itself
// allocates nothing.  Every GPU that loads the library carries the array until exit.
namespace {
constexpr int STATIC_MAX_TOKENS = 32;
constexpr size_t STATIC_CODE_BYTES = size_t(2) << 20;               // activation codes: tokens_per_cta x padded K bytes
constexpr size_t STATIC_SCRATCH_BYTES = STATIC_CODE_BYTES + 4096;   // + scales, status block
}
static __device__ __align__(256) unsigned char g_static_scratch[STATIC_SCRATCH_BYTES];

namespace {
std::mutex g_static_lock;
unsigned char* g_static_ptr[64] = {};   // device address of the array, per CUDA ordinal

// The array's name is only a host-side handle; kernels need its address on the current device.
int static_scratch(int device, unsigned char** out)
{
    if (device < 0 || device >= 64) return RK_NPU_ERR_PARAM;
    std::lock_guard<std::mutex> guard(g_static_lock);
    if (!g_static_ptr[device]) {
        void* ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_static_scratch) != cudaSuccess || !ptr) { cudaGetLastError(); return RK_NPU_ERR_IOCTL; }
        g_static_ptr[device] = static_cast<unsigned char*>(ptr);
    }
    *out = g_static_ptr[device];
    return RK_NPU_OK;
}
} // namespace

namespace {
// Makes `device` current for the duration of a call and restores what the caller had.
struct DeviceScope {
    int previous = -1;
    bool ok = false;
    explicit DeviceScope(int device)
    {
        if (cudaGetDevice(&previous) != cudaSuccess) { cudaGetLastError(); previous = -1; }
        ok = previous == device || cudaSetDevice(device) == cudaSuccess;
        if (!ok) cudaGetLastError();
        if (previous == device) previous = -1;
    }
    ~DeviceScope() { if (previous >= 0) cudaSetDevice(previous); }
};
} // namespace

// What the last allocation-free linear on `weights`' GPU left in the array's status block.  Copies 16 bytes
// into the caller's variables; allocates nothing.  The caller has synchronised the stream of that call.
extern "C" int rk_npu_b200_w4a8_static_status(const rk_npu_w4a8_weights* weights, int* bad_input, int* device_error)
{
    using namespace rkb200;
    if (!weights || !bad_input || !device_error) return RK_NPU_ERR_PARAM;
    const rk_npu_ctx* ctx = weights->domain->ctx;
    DeviceScope scope(ctx->device);
    if (!scope.ok) return RK_NPU_ERR_SUBMIT;
    unsigned char* base = nullptr;
    const int rc = static_scratch(ctx->device, &base);
    if (rc) return rc;
    Status host{};
    if (cudaMemcpy(&host, base + STATIC_CODE_BYTES + 1024, sizeof(Status), cudaMemcpyDeviceToHost) != cudaSuccess) {
        cudaGetLastError();
        return RK_NPU_ERR_SUBMIT;
    }
    *bad_input = host.bad_input;
    *device_error = host.device_error;
    return host.device_error ? RK_NPU_ERR_SUBMIT : host.bad_input ? RK_NPU_ERR_PARAM : RK_NPU_OK;
}

extern "C" int rk_npu_b200_w4a8_enqueue_f16_static(const rk_npu_w4a8_weights* weights, const uint16_t* dA, uint16_t* dC,
                                                   int M, void* cuda_stream)
{
    using namespace rkb200;
    if (!weights || !dA || !dC || dA == dC || M < 1) return RK_NPU_ERR_PARAM;
    const int K = weights->info.config.K, N = weights->info.config.N;
    const int tokens = M <= 8 ? 8 : M <= 16 ? 16 : 32;
    const size_t code_bytes = size_t(tokens) * weights->KB * KBLOCK;
    // sizes beyond the fixed array are refused, never truncated
    if (M > STATIC_MAX_TOKENS || code_bytes > STATIC_CODE_BYTES) return RK_NPU_ERR_NOMEM;
    const rk_npu_ctx* ctx = weights->domain->ctx;
    if (ctx->world > 1) return RK_NPU_ERR_PARAM;   // sharded weights: the exchange behind a group linear needs a workspace
    DeviceScope scope(ctx->device);   // the caller's current device is put back on return
    if (!scope.ok) return RK_NPU_ERR_SUBMIT;
    unsigned char* base = nullptr;
    const int rc = static_scratch(ctx->device, &base);
    if (rc) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    uint8_t* codes = base;
    float* scales = reinterpret_cast<float*>(base + STATIC_CODE_BYTES);
    Status* status = reinterpret_cast<Status*>(base + STATIC_CODE_BYTES + 1024);
    // The array keeps whatever the previous call left: padding rows of the code tile and the
    // status block must start at zero.
    if (cudaMemsetAsync(codes, 0, code_bytes, stream) != cudaSuccess ||
        cudaMemsetAsync(status, 0, sizeof(Status), stream) != cudaSuccess) { cudaGetLastError(); return RK_NPU_ERR_SUBMIT; }
    QuantParams q{};
    q.A = dA;
    q.Xq = codes;
    q.scales = scales;
    q.status = status;
    q.M = M;
    q.K = K;
    q.Kp = weights->KB * KBLOCK;
    q.T = tokens;
    q.half = 1;
    if (launch_quantize(q, stream, false) != cudaSuccess) { cudaGetLastError(); return RK_NPU_ERR_SUBMIT; }
    GemmParams g{};
    g.Wp = weights->packed;
    g.Xq = codes;
    g.sx = scales;
    g.sw = weights->scales;
    g.out = dC;
    g.status = g.report = status;
    g.M = M;
    g.N = N;
    g.K = K;
    g.KB = weights->KB;
    g.NG = weights->NG;
    g.T = tokens;
    g.epi = EPI_F16;
    g.timeout_ns = 500ull * 1000000ull;
    const int tiles = (N + TILE_N - 1) / TILE_N;
    int split = 1;
    while (split < 8 && (long long)tiles * split * 2 <= (long long)(5 * ctx->sm_count) / 2 && weights->KB / (split * 2) >= 2) split *= 2;
    g.split = split;
    if (launch_gemm_mma(g, tokens, stream, false) != cudaSuccess) { cudaGetLastError(); return RK_NPU_ERR_SUBMIT; }
    return RK_NPU_OK;
}

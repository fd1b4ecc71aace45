// w4a8_gemm_tc_persist.cu -- persistent two-CTA tcgen05 W4A8 GEMM from 17 tokens on (sm_100a).
//
// Packed int4 weights -> tensor memory as the A operand, int8 activation codes as shared-memory B operand, kind::i8
// MMA over a CTA pair with cta_group::2, int32 accumulators in tensor memory, organised so that nothing but the
// tensor pipe sits on the critical path:
//   * one cluster of two CTAs per SM pair stays resident and walks a run of 256-channel x (64, 128, 192, 224 or
//     256)-token tiles; barriers, tensor memory and descriptors are set up once.  Where the tiles are few, K is cut into parts;
//   * weights and activations travel through SEPARATE rings of bulk copies.  A weight slot is
//     free again as soon as the unpack warps have read it (the unpacked copy lives in tensor
//     memory), an activation slot when the MMAs that read it retire.  Together the rings take all of shared memory,
//     because the copies (L2 hits) take several MMA-stage times to arrive and the pipe starves on a
//     shallower ring;
//   * eight dedicated epilogue warps read the accumulator out of tensor memory, hand it back
//     after the last read and store straight from registers: the 32 lanes of a warp hold 32
//     neighbouring channels of one token, i.e. 64..128 contiguous bytes per store;
//   * for SwiGLU the unpack warps place gate channels in lanes 0-15 and the matching up
//     channels in lanes 16-31 of every tensor-memory lane quarter, so the epilogue pairs them
//     with one warp shuffle.
// Outputs: binary16 / fp32 / int32 [M,N], or the fused SwiGLU middle [M,F] fp32 (row maxima
// collected).
#include "w4a8_device.h"
#include "w4a8_math.cuh"
#include "w4a8_rules.h"
#include "w4a8_ptx.cuh"
#include "w4a8_tc.cuh"
#include <algorithm>

namespace rkb200 {

constexpr int PS_ROLE_WARPS = 4;             // warp 0: activation producer, 1: MMA issuer, 2: weight producer, 3: activation voucher
constexpr int PS_UNPACK_WARPS = 8;
// (With twelve or sixteen, at 80 and 72 registers a thread, the finishing gets the issue slots that the unpacking and the MMA
// issuer need: SwiGLU at 192 tokens 426 -> 458 and 558 us.)
constexpr int PS_EPI_WARPS = 8;
constexpr int PS_EPI_SETS = PS_EPI_WARPS / 4;  // per tensor-memory lane quarter, taking 32-token chunks in turn
constexpr int PS_UNPACK_WARP0 = PS_ROLE_WARPS;
constexpr int PS_EPI_WARP0 = PS_UNPACK_WARP0 + PS_UNPACK_WARPS;
constexpr int PS_THREADS = 32 * (PS_EPI_WARP0 + PS_EPI_WARPS);   // 640
constexpr int PS_TMEM_COLS = 512;
constexpr unsigned long long PS_DRAIN_NS = 50000;


// One instantiation's resources.  TOK = tokens of the MMA tile (accumulator columns), half of them in each CTA.
// Stages are 2 k-blocks.  Tensor memory holds the accumulator (two of them where they fit, so that the epilogue of a
// segment overlaps the MMAs of the next) and the unpacked weights, 64 columns per stage.
template <bool W8, int TOK>
struct PsShape {
    static constexpr int T = TOK / 2;                                            // tokens of one CTA's activation tile
    static constexpr int XA = TOK == 256 ? (W8 ? 3 : 5) : TOK == 224 ? (W8 ? 3 : 4) : TOK == 192 ? (W8 ? 4 : 5) : TOK == 128 && W8 ? 4 : 6;   // activation ring
    static constexpr int XW = TOK == 256 || W8 ? 4 : TOK >= 128 ? 6 : 8;        // weight ring
    static constexpr int ACC = TOK > 192 ? 1 : 2;                                // accumulators
    static constexpr int ABUF = TOK == 64 ? 6 : TOK == 192 ? 2 : 4;              // unpacked weight stages
    static constexpr int A_COL0 = ACC * TOK;
    static constexpr size_t XA_BYTES = 2 * (size_t)T * 128;
    static constexpr uint32_t GB = W8 ? 4096 : 2048;                             // one k-block of one 32-channel group
    static constexpr size_t XW_BYTES = 2 * 4 * (size_t)GB;
    static constexpr int BARRIERS = 3 * XA + 2 * XW + 2 * ABUF + 2 * ACC;
    static constexpr size_t SMEM = XA * XA_BYTES + XW * XW_BYTES + 2 * TOK * 4 + BARRIERS * 8 + 32;
    static constexpr size_t SLOT_INTS = 128 * (size_t)TOK;                       // one CTA's partial sums of a segment
    static_assert(SMEM <= 232448, "exceeds the shared memory of one CTA");
    static_assert(A_COL0 + 64 * ABUF <= PS_TMEM_COLS, "exceeds tensor memory");
    // The two unpack sets take alternate stages, so with an even ring every slot belongs to one set, which sees all of its
    // phases.  (With an odd one a set could ask for a slot's second phase while the first, the other set's, is still open;
    // a parity wait takes that for completed.)
    static_assert(XW % 2 == 0 && ABUF % 2 == 0, "a ring slot would change between the unpack sets");
};

// A position in a ring of N barriers: slot and phase parity.
template <int N>
struct RingPos {
    int slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next() { if (++slot == N) { slot = 0; phase ^= 1u; } }
};

// Barrier of the eight epilogue warps that also tells every one of them whether `ok` holds in all.
__device__ __forceinline__ bool epilogue_all(bool ok)
{
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.and.pred p, 1, %2, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(all)
        : "r"(ok ? 1u : 0u), "n"(32 * PS_EPI_WARPS)
        : "memory");
    return all != 0;
}

// The same barrier; true: `here` holds in one of them.
__device__ __forceinline__ bool epilogue_any(bool here)
{
    uint32_t any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.or.pred p, 1, %2, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(any)
        : "r"(here ? 1u : 0u), "n"(32 * PS_EPI_WARPS)
        : "memory");
    return any != 0;
}

// (Linear and SwiGLU launches have kernels of their own: less to fetch, and neither finishing pays for the other's registers.)
// W8: the weights are int8 codes in the W8 layout (w8a8_kernels.cu): "unpacking" is a copy into tensor memory and the sums
// are not scaled by 16.
template <bool W8, bool SWIGLU, int TOK>
__global__ void __launch_bounds__(PS_THREADS, 1) gemm_tc_persist_kernel(const GemmParams p, int num_clusters)
{
    using S = PsShape<W8, TOK>;
    constexpr uint32_t GB = S::GB;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* const acts = smem;
    uint8_t* const wts = acts + S::XA * S::XA_BYTES;
    float* const s_sx = reinterpret_cast<float*>(wts + S::XW * S::XW_BYTES);     // token scales of the tile being finished
    uint32_t* const s_tilemax = reinterpret_cast<uint32_t*>(s_sx + TOK);         // SwiGLU: the CTA's row maxima of that tile
    uint64_t* const xfull = reinterpret_cast<uint64_t*>(s_tilemax + TOK);
    uint64_t* const xempty = xfull + S::XA;
    uint64_t* const x_ready = xempty + S::XA;    // leader: both CTAs' activations of the stage have landed
    uint64_t* const wfull = x_ready + S::XA;
    uint64_t* const wempty = wfull + S::XW;
    uint64_t* const a_ready = wempty + S::XW;    // leader: both CTAs' weights of the stage are in tensor memory
    uint64_t* const a_free = a_ready + S::ABUF;
    uint64_t* const acc_full = a_free + S::ABUF;
    uint64_t* const acc_empty = acc_full + S::ACC;
    uint32_t* const s_tmem = reinterpret_cast<uint32_t*>(acc_empty + S::ACC);
    int* const s_error = reinterpret_cast<int*>(s_tmem + 1);
    int* const s_finish = s_error + 1;           // this CTA completed the tile whose partial sums it just stored

    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const int cluster_id = blockIdx.x >> 1;
    constexpr bool swiglu = SWIGLU;
    const int KB = p.KB;
    const int nst = (KB + 1) / 2;                                      // stage iterations per tile
    const int tiles_n = swiglu ? (p.F + 63) / 64 : (p.N + TILE_N - 1) / TILE_N;
    const int pairs_n = (tiles_n + 1) / 2;
    const int pairs_m = (p.M + TOK - 1) / TOK;
    // Every cluster takes a run of whole tiles, or (split > 1) one of the `split` parts of one tile's stages.
    const int tiles = pairs_n * pairs_m, split = p.split;
    const int part = cluster_id % split;
    const int tile0 = split > 1 ? cluster_id / split : (int)((long long)tiles * cluster_id / num_clusters);
    const int it0 = nst * part / split;
    const int n_items = split > 1 ? nst * (part + 1) / split - it0 : ((int)((long long)tiles * (cluster_id + 1) / num_clusters) - tile0) * nst;
    const unsigned long long deadline = global_ns() + p.timeout_ns;
    // optional cycle stamps of cluster 0's leader: [segment j < 16][8] = MMA wait-begin, MMA first issue,
    // MMA last commit, epilogue acc_full seen, tensor memory handed back, stored, [6] cycles the MMA
    // issuer waited for operands; [128] / [129] cycles unpack warp 0 waited for weights / for a free
    // tensor-memory buffer, [160] cycles for activations; [200] = clusters in the grid
    unsigned long long* const trace = (p.trace && blockIdx.x == 0) ? p.trace : nullptr;
    const long long c0 = clock64();
#define PS_STAMP(j, slot) do { if (trace && (j) < 16) trace[(j) * 8 + (slot)] = (unsigned long long)(clock64() - c0); } while (0)
    if (trace && tid == 0) trace[200] = (unsigned long long)num_clusters;

    if (tid == 0) {
        for (int s = 0; s < S::XA; ++s) { mbar_init(&xfull[s], 1); mbar_init(&xempty[s], 1); mbar_init(&x_ready[s], 2); }
        for (int s = 0; s < S::XW; ++s) { mbar_init(&wfull[s], 1); mbar_init(&wempty[s], 4); }
        for (int b = 0; b < S::ABUF; ++b) { mbar_init(&a_ready[b], 8); mbar_init(&a_free[b], 1); }
        for (int b = 0; b < S::ACC; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * PS_EPI_WARPS); }   // every epilogue warp of both CTAs
        mbar_fence_init();
        *s_error = 0;
        *s_finish = 0;
    }
    if (tid < TOK) s_tilemax[tid] = 0u;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(PS_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_arrive();
    cluster_wait();   // the peer's barriers and tensor memory exist from here on
    tc_fence_after();
    const uint32_t tmem_base = *s_tmem;

    // What does not depend on the kernel in front -- requesting weights, unpacking the first of them into tensor
    // memory -- starts before the dependency wait; every other warp waits here.
    auto dependency_met = [&]() -> bool {   // false: the quantiser rejected the input, nothing is to be written
        pdl_wait();
        return *reinterpret_cast<volatile const int*>(&p.status->bad_input) == 0;
    };

    if (warp == 2) {
        // ---------------------------------------------------------------- weight producer
        // (the whole warp walks the loop and one elected lane issues, as in the MMA issuer below: copy requests take their
        // operands from uniform registers, and four lanes issuing one request each took 1000 cycles per stage)
        RingPos<S::XW> r;
        int it = it0;
        bool ok = true, live = true;
        const uint8_t* src = nullptr;                              // group 0 of this CTA's channel tile, stage `it`
        const size_t group_bytes = (size_t)KB * GB;
        const size_t upper = swiglu ? (size_t)(p.F / GROUP) * group_bytes : 2 * group_bytes;   // groups 2, 3 behind groups 0, 1
        for (int gi = 0, tile = tile0; gi < n_items; ++gi, r.next()) {
            if (gi == S::XW) {
                live = dependency_met();
                if (!live) break;
            }
            if (src == nullptr) {
                const int ct = 2 * (tile % pairs_n) + (int)rank;
                src = p.Wp + (size_t)(swiglu ? ct * 2 : ct * 4) * group_bytes + (size_t)it * 2 * GB;
            }
            const uint32_t bytes = (uint32_t)min(2, KB - 2 * it) * GB;
            if (gi >= S::XW) ok = __all_sync(0xffffffffu, mbar_wait(&wempty[r.slot], r.phase ^ 1u, deadline));
            if (!ok) { *s_error = 1; break; }
            uint8_t* const dst = wts + (size_t)r.slot * S::XW_BYTES;
            if (elect_one()) {
                mbar_arrive_expect_tx(&wfull[r.slot], 4u * bytes);
                bulk_g2s(dst, src, bytes, &wfull[r.slot]);
                bulk_g2s(dst + 2 * GB, src + group_bytes, bytes, &wfull[r.slot]);
                bulk_g2s(dst + 4 * GB, src + upper, bytes, &wfull[r.slot]);
                bulk_g2s(dst + 6 * GB, src + upper + group_bytes, bytes, &wfull[r.slot]);
            }
            __syncwarp();
            src += 2 * GB;
            if (++it == nst) { it = 0; ++tile; src = nullptr; }
        }
        if (n_items <= S::XW) live = dependency_met();
        if (!live && lane == 0)   // nobody will consume: let the copies already requested land before leaving
            for (int s = 0; s < min(n_items, S::XW); ++s)
                if (!mbar_wait(&wfull[s], 0, deadline)) { *s_error = 1; break; }
    } else if (warp == 0) {
        // ---------------------------------------------------------------- activation producer
        if (dependency_met()) {
            RingPos<S::XA> r;
            int it = it0;
            const uint8_t* src = nullptr;
            for (int gi = 0, tile = tile0; gi < n_items; ++gi, r.next()) {
                if (src == nullptr) src = p.Xq + ((size_t)(2 * (tile / pairs_n) + (int)rank) * KB + (size_t)it * 2) * (S::T * 128);
                const uint32_t bytes = (uint32_t)min(2, KB - 2 * it) * S::T * 128u;
                bool ok = true;
                if (gi >= S::XA) ok = __all_sync(0xffffffffu, mbar_wait_cluster(&xempty[r.slot], r.phase ^ 1u, deadline));
                if (!ok) { *s_error = 1; break; }
                if (elect_one()) {
                    mbar_arrive_expect_tx(&xfull[r.slot], bytes);
                    bulk_g2s(acts + (size_t)r.slot * S::XA_BYTES, src, bytes, &xfull[r.slot]);
                }
                __syncwarp();
                src += S::XA_BYTES;
                if (++it == nst) { it = 0; ++tile; src = nullptr; }
            }
            // The MMAs' commits arrive on this CTA's barriers asynchronously, the peer's among them: the CTA may not leave
            // (and its shared memory change hands) before the last of them is here.
            for (int gi = n_items; gi < n_items + S::XA && !*reinterpret_cast<volatile int*>(s_error); ++gi, r.next())
                if (gi >= S::XA && !mbar_wait_cluster(&xempty[r.slot], r.phase ^ 1u, deadline)) *s_error = 1;
        }
    } else if (warp == 3) {
        // ---------------------------------------------------------------- activation voucher
        // The leader's MMAs read both CTAs' activations: this warp passes on that this CTA's copy has landed.  It runs
        // ahead of the MMAs by the depth of the ring.  (When the unpack warps vouched for it, with an arrival that released
        // everything at cluster scope, that release bounded the whole loop: 730 cycles per k-block at K = 11008 against 525.)
        if (dependency_met() && lane == 0) {
            RingPos<S::XA> r;
            long long waited = 0;
            for (int gi = 0; gi < n_items; ++gi, r.next()) {
                const long long w0 = trace ? clock64() : 0;
                if (!mbar_wait(&xfull[r.slot], r.phase, deadline)) { *s_error = 1; break; }
                if (trace) waited += clock64() - w0;
                if (rank != 0) mbar_arrive_remote(&x_ready[r.slot], 0); else mbar_arrive(&x_ready[r.slot]);
            }
            if (trace) trace[160] = (unsigned long long)waited;
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer (leader CTA)
        // The whole warp walks the loop, so that descriptors and addresses are warp-uniform values, and one elected lane
        // issues.  (A loop that only lane 0 enters moves every operand of every MMA into uniform registers first: 85
        // cycles per MMA, which bounded a stage at 1190 cycles whatever the token tile; 1050 now at 256 tokens, of 1024.)
        if (dependency_met() && rank == 0) {
            const uint32_t idesc = tc_idesc_s8(256, TOK);
            bool ok = true;
            RingPos<S::XA> rx;
            RingPos<S::ABUF> ra;
            RingPos<S::ACC> rc;
            int it = it0;
            for (int gi = 0, j = 0; gi < n_items && ok; ++j, rc.next()) {
                const int n = min(nst - it, n_items - gi);
                if (lane == 0) PS_STAMP(j, 0);
                if (j >= S::ACC) {   // the epilogue warps of both CTAs have read this accumulator's previous segment
                    ok = __all_sync(0xffffffffu, mbar_wait_cluster(&acc_empty[rc.slot], rc.phase ^ 1u, deadline));
                    if (!ok) { *s_error = 1; break; }
                    tc_fence_after();
                }
                const uint32_t d_tmem = tmem_base + rc.slot * TOK;
                long long waited = 0;
                for (int i = 0; i < n; ++i, ++it, rx.next(), ra.next()) {
                    const int kbs = min(2, KB - 2 * it);
                    const long long w0 = trace ? clock64() : 0;
                    ok = mbar_wait_cluster(&x_ready[rx.slot], rx.phase, deadline) && mbar_wait_cluster(&a_ready[ra.slot], ra.phase, deadline);
                    ok = __all_sync(0xffffffffu, ok);
                    if (trace) waited += clock64() - w0;
                    if (!ok) { *s_error = 1; break; }
                    if (i == 0 && lane == 0) PS_STAMP(j, 1);
                    tc_fence_after();
                    const uint32_t xaddr = smem_u32(acts + (size_t)rx.slot * S::XA_BYTES);
                    const uint32_t a_tmem = tmem_base + S::A_COL0 + ra.slot * 64;
                    // k-step q: k-block q / 4 of the stage, 32 k = two 16-byte chunks per token: the descriptor's
                    // address field advances by 2 * T (16-byte units) per step
                    const uint64_t desc0 = tc_smem_desc(xaddr, S::T * 16u, 128u);
                    if (elect_one()) {
                        tc_mma_i8_ts_pair(d_tmem, a_tmem, desc0, idesc, i > 0 ? 1u : 0u);
#pragma unroll
                        for (int q = 1; q < 4; ++q) tc_mma_i8_ts_pair_acc(d_tmem, a_tmem + q * 8, desc0 + (uint64_t)(q * 2 * S::T), idesc);
                        if (kbs == 2) {
#pragma unroll
                            for (int q = 4; q < 8; ++q) tc_mma_i8_ts_pair_acc(d_tmem, a_tmem + q * 8, desc0 + (uint64_t)(q * 2 * S::T), idesc);
                        }
                        tc_commit_pair(&xempty[rx.slot]);   // the activation stage may be refilled once these MMAs retire
                        tc_commit_pair(&a_free[ra.slot]);   // and the weight buffer rewritten, in both CTAs
                        if (i == n - 1) tc_commit_pair(&acc_full[rc.slot]);
                    }
                    __syncwarp();
                }
                if (!ok) break;
                if (lane == 0) {
                    PS_STAMP(j, 2);
                    if (trace && j < 16) trace[j * 8 + 6] = (unsigned long long)waited;
                }
                gi += n;
                if (it == nst) it = 0;
            }
        }
    } else if (warp < PS_EPI_WARP0) {
        // ---------------------------------------------------------------- weight unpack -> TMEM
        const int q = warp & 3;
        const int set = (warp - PS_UNPACK_WARP0) >> 2;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        // which rows of the staged weight groups feed this thread's tensor-memory lane:
        // plain: group q, row lane.  SwiGLU: lanes 0-15 gate rows, lanes 16-31 the matching
        // up rows (staged groups 0,1 = gate, 2,3 = up of the same 64 features).
        const int src_group = swiglu ? (q >> 1) + (lane >= 16 ? 2 : 0) : q;
        const int src_row = swiglu ? (q & 1) * 16 + (lane & 15) : lane;
        const bool tr = trace && warp == PS_UNPACK_WARP0 && lane == 0;
        long long wait_full = 0, wait_free = 0;
        RingPos<S::XW> rw;
        RingPos<S::ABUF> ra;
        // The two sets take alternate stages.  A stage's packed words are read from shared memory while the previous
        // stage's stores to tensor memory are still on their way, so that the two latencies overlap.
        constexpr int NV = W8 ? 16 : 8;                        // 16-byte pieces a lane takes from a stage
        uint4 w[NV];
        bool ok = true;
        auto fetch = [&](int it) {
            const int kbs = min(2, KB - 2 * it);
            const long long w0 = tr ? clock64() : 0;
            ok = __all_sync(0xffffffffu, mbar_wait(&wfull[rw.slot], rw.phase, deadline));
            if (tr) wait_full += clock64() - w0;
            const uint4* src = reinterpret_cast<const uint4*>(wts + (size_t)rw.slot * S::XW_BYTES + src_group * 2 * GB) + src_row;
#pragma unroll
            for (int c = 0; c < NV; ++c) w[c] = (c < NV / 2 * kbs) ? src[c * 32] : make_uint4(0u, 0u, 0u, 0u);
        };
        int it = it0;
        auto advance = [&]() { rw.next(); ra.next(); if (++it == nst) it = 0; };
        if (set == 1) advance();
        if (set < n_items) fetch(it);
        for (int g = set; g < n_items && ok; g += 2) {
            const int kbs = min(2, KB - 2 * it), b = ra.slot;
            // (before the first buffer comes back from the MMAs, which need the activations)
            if ((g == S::ABUF || g == S::ABUF + 1) && !dependency_met()) break;
            const long long w0 = tr ? clock64() : 0;
            if (g >= S::ABUF) ok = __all_sync(0xffffffffu, mbar_wait_cluster(&a_free[b], ra.phase ^ 1u, deadline));
            if (tr) wait_free += clock64() - w0;
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (h < kbs) {
                    uint32_t r[32];
                    if constexpr (W8) {
                        // int8 codes: a lane's sixteen 16-byte pieces of the stage are the words of its tensor-memory row in order
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            const uint4 v = w[8 * h + c];
                            r[4 * c] = v.x; r[4 * c + 1] = v.y; r[4 * c + 2] = v.z; r[4 * c + 3] = v.w;
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const uint4 v = w[4 * h + c];
                            const uint32_t ww[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int jj = 0; jj < 4; ++jj) {
                                r[c * 8 + jj] = (ww[jj] << 4) & 0xF0F0F0F0u;
                                r[c * 8 + 4 + jj] = ww[jj] & 0xF0F0F0F0u;
                            }
                        }
                    }
                    tc_st32(lane_addr + S::A_COL0 + b * 64 + h * 32, r);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&wempty[rw.slot]);      // the packed copy has been read
            advance();
            advance();
            if (g + 2 < n_items) fetch(it);
            tc_wait_st();
            tc_fence_before();
            // Tensor-memory writes are ordered by the wait and the fences; the arrival itself carries nothing, so it is
            // relaxed (see mbar_arrive_remote for what a release at cluster scope costs).
            __syncwarp();
            if (lane == 0) { if (rank != 0) mbar_arrive_remote_relaxed(&a_ready[b], 0); else mbar_arrive_relaxed(&a_ready[b]); }
        }
        if (!ok) *s_error = 1;
        // (the commits on the buffers have to be here before the CTA leaves, as for the activation ring; none come where
        // the input was rejected)
        if (ok && dependency_met())
            for (int g = n_items + ((n_items ^ set) & 1); g < n_items + S::ABUF; g += 2, ra.next(), ra.next())
                if (g >= S::ABUF && !mbar_wait_cluster(&a_free[ra.slot], ra.phase ^ 1u, deadline)) { *s_error = 1; break; }
        if (tr) { trace[128] = (unsigned long long)wait_full; trace[129] = (unsigned long long)wait_free; }
    } else {
        // ---------------------------------------------------------------- epilogue warps
        // A warp finishes sixteen tokens (of its 32 accumulator rows) per turn of a rolled loop.  What bounds it is the
        // number of instructions: eight warps share the issue slots with the unpack warps, so the arithmetic works on pairs
        // of tokens (one instruction per two operations), the int4 records' 1/16 is in the token scales, one look at the
        // magnitudes of four gate values settles that none needs the slow division, and maxima are taken of floats, whose
        // signs the instruction drops (4096 tokens, 4096 -> 2 x 14336: 424 -> 405 us; 300 tokens 54.4 -> 49.6).
        const int q = warp & 3;                        // TMEM lane quarter this warp may read
        const int eset = (warp - PS_EPI_WARP0) >> 2;   // takes 32-token chunks eset, eset + PS_EPI_SETS, ...
        const int sid = (warp - PS_EPI_WARP0) * 32 + lane;   // 0..255 among the epilogue threads
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        const int out_cols = swiglu ? p.F : p.N;
        // output column (inside the CTA's tile) this thread's accumulator row belongs to
        const int col = swiglu ? (q >> 1) * 32 + (q & 1) * 16 + (lane & 15) : q * 32 + lane;
        const bool up_lane = swiglu && lane >= 16;
        const int odd = lane & 1;
        const bool quad_ok = (out_cols % 4 == 0) && (reinterpret_cast<uintptr_t>(p.out) & 7u) == 0;
        constexpr int STEP = 32 * PS_EPI_SETS;
        constexpr int SHIFT = W8 ? 0 : 4;             // int4 records enter the MMA times 16
        bool ok = dependency_met();
        RingPos<S::ACC> rc;
        int tile = tile0, it = it0;
        for (int gi = 0, j = 0; gi < n_items && ok; ++j, rc.next()) {
            const int n_seg = min(nst - it, n_items - gi);
            const int ct = 2 * (tile % pairs_n) + (int)rank;
            const int tok_base = (tile / pairs_n) * TOK;
            const int col0 = swiglu ? ct * 64 : ct * TILE_N;
            const int n = col0 + col;
            const bool n_ok = n < out_cols;
            const float sw = n_ok ? p.sw[(up_lane ? p.F : 0) + n] : 0.f;
            // 32-token chunks of this warp that hold live tokens: those at 32 eset + STEP c, c < chunks
            const int chunks = max(0, (min(TOK, p.M - tok_base) - 32 * eset + STEP - 1) / STEP);
            // Token scales, staged with the int4 records' 1/16 in them: (float)(16 s) * (sx / 16) is (float)s * sx, exactly,
            // unless sx / 16 is subnormal.  (The barrier at the end of a tile keeps stragglers out.)
            float sx_here = 0.f;
            bool tiny = false;
            if (sid < TOK) {
                const int m = tok_base + sid;
                if (m < p.M) {
                    sx_here = p.sx[m];
                    tiny = !W8 && sx_here < 7.8886e-31f;
                }
                s_sx[sid] = W8 ? sx_here : sx_here * 0.0625f;
            }
            tiny = epilogue_any(tiny);
            if (tiny) {
                if (sid < TOK) s_sx[sid] = sx_here;
                asm volatile("bar.sync 1, %0;" ::"n"(32 * PS_EPI_WARPS) : "memory");
            }
            ok = epilogue_all(mbar_wait_cluster(&acc_full[rc.slot], rc.phase, deadline));   // one verdict for all eight warps
            if (!ok) { *s_error = 1; break; }
            if (sid == 0) PS_STAMP(j, 3);
            tc_fence_after();
            const uint32_t acc_addr = lane_addr + rc.slot * TOK + 32 * eset;
            const int row = q * 32 + lane;
            auto hand_back = [&]() {   // this warp is done with the accumulator: another segment's MMAs may overwrite it
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { if (rank != 0) mbar_arrive_remote_relaxed(&acc_empty[rc.slot], 0); else mbar_arrive_relaxed(&acc_empty[rc.slot]); }
                if (sid == 0) PS_STAMP(j, 4);
            };
            // ---- a part of a tile's K: the raw sums go to this CTA's slot, the tile's part counter is advanced, and the CTA
            // that completes it adds the other parts' slots to its own sums, which are still in tensor memory (integer
            // addition: exact in any order), and finishes the tile.  Nobody waits for anybody, and no slot needs clearing.
            const size_t part_stride = 2 * (S::SLOT_INTS / 4);            // from one part's slot to the next one's
            const int4* const slots = reinterpret_cast<const int4*>(p.partials) + (size_t)(2 * split * tile + (int)rank) * (S::SLOT_INTS / 4) + (size_t)(8 * eset) * 128 + row;   // [token / 4][row][4 tokens]
            bool finish = true;
            if (split > 1) {
                int4* const slot = const_cast<int4*>(slots) + part * part_stride;
#pragma unroll 1
                for (int c = 0; c < chunks; ++c) {
                    uint32_t r[32];
                    tc_ld32(acc_addr + STEP * c, r);
                    tc_wait_ld();
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        __stcg(slot + (size_t)(STEP / 4 * c + i) * 128, make_int4((int)r[4 * i], (int)r[4 * i + 1], (int)r[4 * i + 2], (int)r[4 * i + 3]));
                }
                __threadfence();
                asm volatile("bar.sync 1, %0;" ::"n"(32 * PS_EPI_WARPS) : "memory");
                if (sid == 0) {
                    // (a tile with a part whose wait ran out is never completed; the launch reports the error and the host
                    // clears the counters)
                    unsigned* const count = p.counts + 2 * tile + (int)rank;
                    const bool done = atomicAdd(count, 1u) == (unsigned)split - 1u;
                    if (done) *count = 0u;
                    *s_finish = done ? 1 : 0;
                    __threadfence();
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * PS_EPI_WARPS) : "memory");
                finish = *reinterpret_cast<volatile int*>(s_finish) != 0;
            }
            const int turns = finish ? 2 * chunks : 0;
            const int other = part == 0 ? 1 : 0;                          // the first of the other parts
            int4 ahead[4];                                                // its sums of the next turn, on their way
            auto fetch_part = [&](int4 (&v)[4], int which, int k) {
                const int4* const src = slots + which * part_stride + (size_t)(STEP / 4 * (k >> 1) + 4 * (k & 1)) * 128;
#pragma unroll
                for (int h = 0; h < 4; ++h) v[h] = __ldcg(src + (size_t)h * 128);
            };
            if (split > 1 && turns) fetch_part(ahead, other, 0);
            if (split == 1 && chunks == 0) hand_back();
#pragma unroll 1
            for (int k = 0; k < turns; ++k) {
                const int t0 = 32 * eset + STEP * (k >> 1) + 16 * (k & 1), m0 = tok_base + t0;
                uint32_t r[16];
                tc_ld16(lane_addr + rc.slot * TOK + t0, r);
                tc_wait_ld();
                if (split == 1) {
                    if (k + 1 == turns) hand_back();
                } else {
                    auto add = [&](const int4 (&v)[4]) {
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            r[4 * h] += (uint32_t)v[h].x; r[4 * h + 1] += (uint32_t)v[h].y; r[4 * h + 2] += (uint32_t)v[h].z; r[4 * h + 3] += (uint32_t)v[h].w;
                        }
                    };
                    add(ahead);
#pragma unroll 1
                    for (int which = other + 1; which < split; ++which)
                        if (which != part) {
                            int4 v[4];
                            fetch_part(v, which, k);
                            add(v);
                        }
                    if (k + 1 < turns) fetch_part(ahead, other, k + 1);
                }
                if (m0 >= p.M) continue;
                if (!SWIGLU && p.epi == EPI_I32) {
                    int* const row0 = reinterpret_cast<int*>(p.out) + (size_t)m0 * out_cols + n;
                    if (n_ok) {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (m0 + i < p.M) row0[(size_t)i * out_cols] = (int)r[i] >> SHIFT;
                    }
                    continue;
                }
                // y[i]: tokens m0 + 2i and m0 + 2i + 1.  (float)(16 s) / 16 is (float)s, exactly.
                F2 y[8];
                {
                    const ulonglong2* const sx2 = reinterpret_cast<const ulonglong2*>(s_sx + t0);
                    const F2 sw2 = f2_all(sw);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const ulonglong2 sx = sx2[i];
                        y[2 * i] = f2_pack(__int2float_rn((int)r[4 * i]), __int2float_rn((int)r[4 * i + 1]));
                        y[2 * i + 1] = f2_pack(__int2float_rn((int)r[4 * i + 2]), __int2float_rn((int)r[4 * i + 3]));
                        if (tiny) { y[2 * i] = f2_mul(y[2 * i], f2_all(0.0625f)); y[2 * i + 1] = f2_mul(y[2 * i + 1], f2_all(0.0625f)); }
                        y[2 * i] = f2_mul(f2_mul(y[2 * i], sx.x), sw2);
                        y[2 * i + 1] = f2_mul(f2_mul(y[2 * i + 1], sx.y), sw2);
                    }
                }
                if (!SWIGLU && p.epi == EPI_F16) {
                    // a lane holds one channel of sixteen tokens; two exchange rounds turn that into four neighbouring
                    // channels of four tokens: lanes 4g..4g+3 end up with tokens 4i + (lane & 3)
                    uint32_t word[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        float lo, hi;
                        f2_unpack(y[i], lo, hi);
                        const __half2 h = __floats2half2_rn(lo, hi);
                        word[i] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                    const uint32_t selector = odd ? 0x3276u : 0x5410u;     // even lanes: low halves (own, peer's); odd lanes: high halves (peer's, own)
#pragma unroll
                    for (int i = 0; i < 8; ++i) word[i] = __byte_perm(word[i], __shfl_xor_sync(0xffffffffu, word[i], 1), selector);
                    const bool upper = (lane & 2) != 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t recv = __shfl_xor_sync(0xffffffffu, upper ? word[2 * i] : word[2 * i + 1], 2);
                        if (upper) word[2 * i] = recv; else word[2 * i + 1] = recv;
                        // now (word[2i], word[2i+1]) = channels n4 .. n4+3 of token m0 + 4i + (lane & 3)
                    }
                    const int n4 = n - (lane & 3);
                    const int mrow = m0 + (lane & 3);
                    __half* dst = reinterpret_cast<__half*>(p.out) + (size_t)mrow * out_cols + n4;
                    const size_t step = 4 * (size_t)out_cols;
#pragma unroll
                    for (int i = 0; i < 4; ++i, dst += step)
                        if (mrow + 4 * i < p.M) {
                            if (quad_ok && n4 + 3 < out_cols) *reinterpret_cast<uint2*>(dst) = make_uint2(word[2 * i], word[2 * i + 1]);
                            else {
                                const uint32_t ww[2] = {word[2 * i], word[2 * i + 1]};
#pragma unroll
                                for (int e = 0; e < 4; ++e)
                                    if (n4 + e < out_cols) dst[e] = __ushort_as_half((unsigned short)((ww[e >> 1] >> (16 * (e & 1))) & 0xffffu));
                            }
                        }
                } else if (!SWIGLU) {
                    float* dst = reinterpret_cast<float*>(p.out) + (size_t)m0 * out_cols + n;
                    if (n_ok) {
#pragma unroll
                        for (int i = 0; i < 8; ++i, dst += 2 * (size_t)out_cols) {
                            float lo, hi;
                            f2_unpack(y[i], lo, hi);
                            if (m0 + 2 * i < p.M) dst[0] = lo;
                            if (m0 + 2 * i + 1 < p.M) dst[out_cols] = hi;
                        }
                    }
                } else {
                    // Lanes 0-15 hold the gate rows g, lanes 16-31 the matching up rows u of 16 features.  The gate lanes
                    // finish the even token of every pair and the up lanes the odd one: each sends the half of the pair
                    // that the other finishes and evaluates eight SiLUs.
                    float v[8];
                    const int mine_row = m0 + (up_lane ? 1 : 0);
                    const int left = n_ok ? p.M - mine_row : 0;         // rows from here on that are stored
                    float* dst = reinterpret_cast<float*>(p.out) + (size_t)mine_row * out_cols + n;
#pragma unroll
                    for (int h = 0; h < 8; h += 4) {           // (four at a time: one look at the magnitudes, few values waiting)
                        float g[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float even_token, odd_token;
                            f2_unpack(y[h + i], even_token, odd_token);
                            const float recv = __shfl_xor_sync(0xffffffffu, up_lane ? even_token : odd_token, 16);
                            g[i] = up_lane ? recv : even_token;
                            v[h + i] = up_lane ? odd_token : recv;
                        }
                        if (left < 16) {                        // what does not exist has zeros: keep it off the slow path below
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (2 * (h + i) >= left) g[i] = 1.f;
                        }
                        if (silu_plain(min_abs(min_abs(g[0], g[1]), min_abs(g[2], g[3])), max_abs(max_abs(g[0], g[1]), max_abs(g[2], g[3])))) {
#pragma unroll
                            for (int i = 0; i < 4; i += 2) {
                                float a, b;
                                minus_silu_poly2(g[i], g[i + 1], a, b);
                                v[h + i] = __fmul_rn(-a, v[h + i]);
                                v[h + i + 1] = __fmul_rn(-b, v[h + i + 1]);
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) v[h + i] = __fmul_rn(silu_poly(g[i]), v[h + i]);
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i, dst += 2 * (size_t)out_cols)
                            if (2 * (h + i) < left) *dst = v[h + i];
                    }
                    if (p.rowmax) {
                        // Maxima over the 16 lanes of each half, one token per value: three folding steps that halve the
                        // values a lane holds and a plain one; lanes 2i of a half end up with the maximum of their token.
                        // (Tokens and channels that do not exist have zero scales, and zeros here.)
#pragma unroll
                        for (int width = 8; width > 1; width >>= 1) {
                            const bool upper = (lane & width) != 0;
#pragma unroll
                            for (int i = 0; i < width / 2; ++i) {
                                const float keep = upper ? v[i + width / 2] : v[i];
                                const float give = upper ? v[i] : v[i + width / 2];
                                v[i] = max_abs(keep, __shfl_xor_sync(0xffffffffu, give, width));
                            }
                        }
                        const uint32_t most = __float_as_uint(max_abs(v[0], __shfl_xor_sync(0xffffffffu, v[0], 1)));
                        // collected per CTA and tile in shared memory first: one global atomic per token and tile
                        // instead of one per token, tile and 16 features
                        if (!odd && most) atomicMax(&s_tilemax[t0 + (up_lane ? 1 : 0) + 2 * ((lane >> 1) & 7)], most);
                    }
                }
            }
            if (sid == 0) PS_STAMP(j, 5);
            asm volatile("bar.sync 1, %0;" ::"n"(32 * PS_EPI_WARPS) : "memory");   // every epilogue warp is done with this tile's scales and maxima
            if (swiglu && p.rowmax && sid < TOK) {
                const uint32_t m = s_tilemax[sid];
                if (m) {
                    atomicMax(&p.rowmax[tok_base + sid], m);
                    s_tilemax[sid] = 0u;
                }
            }
            gi += n_seg;
            it += n_seg;
            if (it == nst) { it = 0; ++tile; }
        }
    }

    // ------------------------------------------------------------------------ teardown
    tc_fence_before();
    __syncthreads();
    // A wait that ran out ends its role at once, and copies requested just before may still be on their way into this CTA's
    // shared memory: they land within microseconds, so the CTA stays that long before it leaves.
    if (*reinterpret_cast<volatile int*>(s_error))
        for (const unsigned long long until = global_ns() + PS_DRAIN_NS; global_ns() < until;) __nanosleep(1000);
    cluster_arrive();
    cluster_wait();   // neither CTA frees tensor memory or leaves while the other may still use it
    if (tid == 0 && *s_error) report_device_error(p.status, p.report);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(PS_TMEM_COLS) : "memory");
    }
}

namespace {
constexpr long long PS_MAX_K = 131072;

template <bool W8, bool SWIGLU, int TOK>
cudaError_t launch_persist_inst(const GemmParams& p, cudaStream_t stream, bool pdl)
{
    using S = PsShape<W8, TOK>;
    auto kernel = gemm_tc_persist_kernel<W8, SWIGLU, TOK>;
    static PerDeviceOnce configured;
    static int clusters_of_device[64] = {};   // resident CTA pairs, per CUDA ordinal
    int device = -1;
    int max_clusters = 0;
    const bool setup = configured.needed(device);
    if (!setup) max_clusters = clusters_of_device[device];
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(PS_THREADS);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    if (setup || !max_clusters) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
        if (e != cudaSuccess) return e;
        // how many CTA pairs can be resident at once
        cfg.gridDim = dim3(2, 1, 1);
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
        if (e != cudaSuccess || n < 1) { cudaGetLastError(); int dev = 0, sms = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); n = sms / 2; }
        max_clusters = n;
        if (device >= 0 && device < 64) { clusters_of_device[device] = n; configured.mark(device); }
    }
    const int tiles = gemm_tc_persist_tiles(p.epi == EPI_SWIGLU ? 2 * p.F : p.N, p.M, TOK);
    const int clusters = persist_clusters(tiles, p.split, max_clusters);
    cfg.gridDim = dim3((unsigned)(2 * clusters), 1, 1);
    int n = 1;
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, p, clusters);
}
template <int TOK>
cudaError_t launch_persist_tok(const GemmParams& p, cudaStream_t stream, bool pdl)
{
    if (p.w8) return p.epi == EPI_SWIGLU ? cudaErrorInvalidValue : launch_persist_inst<true, false, TOK>(p, stream, pdl);
    return p.epi == EPI_SWIGLU ? launch_persist_inst<false, true, TOK>(p, stream, pdl) : launch_persist_inst<false, false, TOK>(p, stream, pdl);
}
} // namespace

int gemm_tc_persist_tiles(int columns, int M, int tok) { return (columns + 255) / 256 * ((M + tok - 1) / tok); }

// The token tile and the number of parts a tile's K is cut into: the cheapest by a model of the kernel's time in cycles,
// fitted to 80 shapes (M 33..4096, K 2048..14336, N 1024..28672, both epilogues).  On 27 others, K 1024..11008, it is within
// 2 % of the best choice but just above 64 tokens (a second tile of 64 would be nearly empty: 20 % at worst, 65 x 8192 -> 2048
// 19.0 us where 64-token tiles take 15.8) and for 400 to 448 tokens of K = 1024 (23.9 against 22.0):
//   * a k-block takes 270 to 390 cycles at 64 tokens and 310 to 370 at 128, more with more SMs busy (the operands come
//     out of L2 at about 45 bytes per SM and cycle when all SMs ask), and 530 at 256, where the MMAs bound it; int8
//     weights are delivery-bound (52 bytes per cycle).  At 192 tokens two accumulators leave two buffers of unpacked
//     weights: 560, and 780 with int8 weights;
//   * finishing a tile takes 33 cycles per token, 1500 at least; 80 and 4800 with SwiGLU, which bounds the kernel at
//     K = 4096 (192 tokens instead of 128 amortise it better: 4096 x 4096 -> 14336 450 -> 422 us); two accumulators hide
//     it behind the next tile's MMAs up to 192 tokens, beyond there is room for one and nothing is hidden;
//   * 224 tokens are for what 256 would cut worse (777 tokens, 14336 -> 4096 50 -> 46 us);
//   * K in parts costs an exchange through L2: so much per part and pair, more for wide token tiles;
//   * a launch on more than half of the SMs leaves the one behind it no room to set itself up meanwhile.
PersistPlan gemm_tc_persist_plan(int columns, int M, int KB, bool w8, bool swiglu, int sm_count)
{
    PersistPlan best{256, 1};
    double best_time = 0;
    const int pairs = std::max(1, sm_count / 2);
    for (const int tok : {64, 128, 192, 224, 256}) {
        if (tok > 64 && M <= 64) break;                        // half of the tile would be padding
        const long long tiles = (long long)((columns + 255) / 256) * ((M + tok - 1) / tok);
        for (const int split : {1, 2, 3, 4, 6, 8}) {
            if (split > 1 && (tok > 128 || tiles * split > pairs || KB < 4 * split)) break;
            const long long clusters = std::min<long long>(tiles * split, pairs), rounds = (tiles + pairs - 1) / pairs;
            const double busy = double(clusters) / pairs;
            double block = tok == 64 ? 270 + 120 * busy : tok == 128 ? 310 + 60 * busy : tok == 192 ? 480 + 80 * busy : tok == 224 ? 470 : 530;
            if (swiglu) block += 20;
            if (w8) block = tok == 192 ? 780 : std::max(block, (16384 + 64 * tok) / 52.0);
            const double mma = KB * block / split, live = std::min(tok, M), finish = swiglu ? 4800 + 80 * live : 1500 + 33 * live;
            double time = tok > 192 ? rounds * (mma + finish) : mma + (rounds - 1) * std::max(mma, finish) + finish;
            if (split > 1) time += (1500 + 1000 * (split - 1) + 30 * clusters) * (1 + 1.5 * std::max(0.0, live - 64) / 64);
            if (2 * clusters > pairs) time += 3000;
            if (best_time == 0 || time < best_time) { best_time = time; best = {tok, split}; }
        }
    }
    return best;
}
size_t gemm_tc_persist_slot_bytes(int columns, int M, const PersistPlan& plan)
{
    return plan.split > 1 ? 2 * size_t(gemm_tc_persist_tiles(columns, M, plan.tok)) * size_t(plan.split) * 128 * size_t(plan.tok) * sizeof(int) : 0;
}
size_t gemm_tc_persist_count_bytes(int columns, int M, const PersistPlan& plan)
{
    return plan.split > 1 ? 2 * size_t(gemm_tc_persist_tiles(columns, M, plan.tok)) * sizeof(unsigned) : 0;
}

cudaError_t launch_gemm_tc_persist(const GemmParams& p, cudaStream_t stream, bool pdl)
{
    if ((long long)p.KB * KBLOCK > PS_MAX_K || p.split < 1 || (p.split > 1 && !(p.partials && p.counts))) return cudaErrorInvalidValue;
    switch (2 * p.T) {
    case 64: return launch_persist_tok<64>(p, stream, pdl);
    case 128: return launch_persist_tok<128>(p, stream, pdl);
    case 192: return launch_persist_tok<192>(p, stream, pdl);
    case 224: return launch_persist_tok<224>(p, stream, pdl);
    case 256: return launch_persist_tok<256>(p, stream, pdl);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace rkb200

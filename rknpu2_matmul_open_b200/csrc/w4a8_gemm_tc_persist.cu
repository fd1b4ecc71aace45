// w4a8_gemm_tc_persist.cu -- persistent two-CTA tcgen05 W4A8 GEMM, from 9 or 17 tokens on by the width of the output (sm_100a).
//
// Packed int4 weights -> tensor memory as the A operand (int8 weights stay in shared memory), int8 activation codes as
// shared-memory B operand, kind::i8 MMA over a CTA pair with cta_group::2, int32 accumulators in tensor memory, organised so
// that nothing but the tensor pipe sits on the critical path:
//   * one cluster of two CTAs per SM pair stays resident and walks a run of items: 256 channels x any multiple of 32 tokens up to
//     the kernel's width (64, 160 or 256; int8 weights 64 or 256), so that equal runs leave no nearly empty last round
//     (4096 -> 14336, 2048 tokens: 13 rounds of 128-token tiles for 12.1 of work before).  Barriers, tensor memory and
//     descriptors are set up once.  Where the tiles are few, K is cut into parts (persist_plan.h);
//   * weights (bulk copies) and activations (tensor copies with the 128-byte swizzle) travel through SEPARATE rings.  A weight slot is free again as soon as the unpack
//     warps have read it (the unpacked copy lives in tensor memory), an activation slot when the MMAs that read it retire;
//   * the MMA issuer is one warp whose every instruction counts: the tensor pipe queues about two MMAs, and what the issuer
//     does between the last MMA of a stage and the first of the next has to fit under them.  So there is ONE barrier to wait
//     for (activations and unpacked weights of a stage arrive on the same one) and ONE commit per stage.  (With a barrier and
//     a commit per operand a stage of two k-blocks cost the issuer 610 cycles where the MMAs of 128 tokens take 512; leaving
//     the copies, the unpacking or the finishing out changed that by less than 12 %, the waits for operands not at all);
//   * 160 tokens: two accumulators and three unpacked stages fill tensor memory exactly, and per token the weights are
//     unpacked, and shared memory is written and read, a quarter less often than with 128 (4096 -> 14336, MMA issue to MMA
//     issue: 345 cycles per k-block at 128 tokens before, 300 at 128 and 336 of 320 at 160 now, without the finishing);
//   * eight dedicated epilogue warps read the accumulator out of tensor memory, hand it back after the last read and store
//     straight from registers.  They read it as fragments of sixteen lanes x 256 bits, and the unpack warps choose which
//     channel goes to which lane: a thread then holds four neighbouring channels of a token (SwiGLU: two features' gate and up
//     values), so that nothing has to be exchanged between lanes but row maxima (and the sums of rows whose length does not
//     allow four channels in one store).
// Outputs: binary16 / fp32 / int32 [M,N], or the fused SwiGLU middle [M,F] fp32 (row maxima collected).
#include "w4a8_device.h"
#include "w4a8_math.cuh"
#include "w4a8_ptx.cuh"
#include "w4a8_tc.cuh"
#include <cstdio>
#include <cstdlib>

namespace rkb200 {

constexpr int PS_ROLE_WARPS = 4;             // warp 0: activation producer, 1: MMA issuer, 2: weight producer, 3: voucher
constexpr int PS_UNPACK_SETS = 2;            // of four warps, taking stages in turn (three: the same time, unpacking no longer bounds it)
constexpr int PS_UNPACK_WARPS = 4 * PS_UNPACK_SETS;
// (With twelve or sixteen, at 80 and 72 registers a thread, the finishing gets the issue slots that the unpacking and the MMA
// issuer need: 160 tokens 4096 -> 14336 80 -> 82 and 83 us, SwiGLU 181 -> 181 and 185.)
constexpr int PS_EPI_WARPS = 8;
constexpr int PS_EPI_SETS = PS_EPI_WARPS / 4;  // per tensor-memory lane quarter, taking pieces of sixteen tokens in turn
constexpr int PS_UNPACK_WARP0 = PS_ROLE_WARPS;
constexpr int PS_TMEM_COLS = 512;
constexpr int PS_SK = 2;                     // k-blocks of a stage
constexpr unsigned long long PS_DRAIN_NS = 50000;
constexpr float PS_LOW = 9.5367431640625e-7f;   // 2^-20: the product of two scales of at least that is at least 2^-40

// One instantiation's resources.  TOK = the widest item (accumulator columns), half of its tokens in each CTA.
// Tensor memory holds two accumulators, so that the epilogue of an item overlaps the MMAs of the next, and the unpacked int4
// weights, 64 columns per stage.  (256 tokens leave room for one: for few, long items, whose finishing is not worth hiding.)
// int8 weights are an operand as they lie in shared memory, in the slot of the activations they are multiplied with.
template <bool W8, int TOK>
struct PsShape {
    static constexpr int T = TOK / 2;                                            // tokens of one CTA's half
    static constexpr int ACC = !W8 && TOK == 256 ? 1 : 2;                        // accumulators
    static constexpr int XA = W8 ? (TOK == 64 ? 5 : 3) : TOK == 64 ? 8 : 4;      // activation ring, stages
    static constexpr int XW = W8 ? XA : TOK == 64 ? 10 : TOK == 256 ? 6 : 8;     // weight ring
    static constexpr int ABUF = W8 ? 0 : TOK == 64 ? 6 : TOK == 256 ? 4 : 3;     // unpacked weight stages
    static constexpr int NR = XA > ABUF ? XA : ABUF;                             // barriers of stages ready for / done by the MMAs
    static constexpr int EPI_WARP0 = PS_UNPACK_WARP0 + (W8 ? 0 : PS_UNPACK_WARPS);
    static constexpr int THREADS = 32 * (EPI_WARP0 + PS_EPI_WARPS);              // 640; 384 where nothing is unpacked (1 to 2 % of a call of 24 us)
    static constexpr int WB = W8 ? 0 : XW;                                       // weight slots with barriers of their own
    static constexpr int A_COL0 = ACC * TOK;
    static constexpr size_t XA_BYTES = PS_SK * (size_t)T * 128;
    static constexpr uint32_t GB = W8 ? 4096 : 2048;                             // one k-block of one 32-channel group
    static constexpr size_t XW_BYTES = PS_SK * 4 * (size_t)GB;
    static constexpr int BARRIERS = XA + 2 * WB + 2 * NR + 2 * ACC;
    // barriers in the order in which they lie: xfull, wfull, wempty, ready, done, acc_full, acc_empty
    static __device__ __forceinline__ uint32_t arrivals(int i)
    {
        if (i < XA) return W8 ? 2 : 1;
        if ((i -= XA) < 2 * WB) return i < WB ? 1 : 4;
        if ((i -= 2 * WB) < 2 * NR) return i < NR ? (W8 ? 0 : 8) + 2 : 1;
        return i - 2 * NR < ACC ? 1 : 2 * PS_EPI_WARPS;           // acc_empty: every epilogue warp of both CTAs
    }
    static constexpr size_t SMEM = XA * XA_BYTES + XW * XW_BYTES + 2 * TOK * 4 + BARRIERS * 8 + 32;
    static_assert(TOK % 32 == 0 && TOK <= 256, "not the width of an MMA");
    static_assert(SMEM <= 232448, "exceeds the shared memory of one CTA");
    static_assert(A_COL0 + 64 * ABUF <= PS_TMEM_COLS, "exceeds tensor memory");
    // The two unpack sets take alternate stages, so with an even ring every weight slot belongs to one set, which sees all of
    // its phases.  (With an odd one a set could ask for a slot's second phase while the first, the other set's, is still
    // open; a parity wait takes that for completed.  The barriers of retired MMAs complete in order, whoever waits.)
    static_assert(W8 || XW % PS_UNPACK_SETS == 0, "a ring slot would change between the unpack sets");
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

// Four neighbouring channels of one token, held in the order (turn, turn + 1, ...) mod 4, in one store.
__device__ __forceinline__ void store_four(uint32_t* dst, const uint32_t (&held)[4], int turn)
{
    uint32_t half[4], v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) half[i] = turn & 1 ? held[(i + 3) & 3] : held[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = turn & 2 ? half[(i + 2) & 3] : half[i];
    *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store_four_halves(__half* dst, uint32_t held01, uint32_t held23, int turn)
{
    // channel i is held at (i - turn) mod 4
    const uint32_t a = (0u - turn) & 3u, b = (1u - turn) & 3u, c = (2u - turn) & 3u, d = (3u - turn) & 3u;
    *reinterpret_cast<uint2*>(dst) = make_uint2(__byte_perm(held01, held23, 0x1010u + 0x22u * a + 0x2200u * b), __byte_perm(held01, held23, 0x1010u + 0x22u * c + 0x2200u * d));
}

// (Linear and SwiGLU launches have kernels of their own: less to fetch, and neither finishing pays for the other's registers.)
// W8: the weights are int8 codes in the W8 layout (w8a8_kernels.cu), and the sums are not scaled by 16.
template <bool W8, bool SWIGLU, int TOK>
__global__ void __launch_bounds__(PsShape<W8, TOK>::THREADS, 1) gemm_tc_persist_kernel(const GemmParams p, const __grid_constant__ PersistMaps maps, int num_clusters)
{
    using S = PsShape<W8, TOK>;
    constexpr uint32_t GB = S::GB;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* const acts = smem;
    uint8_t* const wts = acts + S::XA * S::XA_BYTES;
    float* const s_sx = reinterpret_cast<float*>(wts + S::XW * S::XW_BYTES);     // token scales of the item being finished
    uint32_t* const s_tilemax = reinterpret_cast<uint32_t*>(s_sx + TOK);         // SwiGLU: the CTA's row maxima of that item
    uint64_t* const xfull = reinterpret_cast<uint64_t*>(s_tilemax + TOK);        // W8: the weights of the stage as well
    uint64_t* const wfull = xfull + S::XA;
    uint64_t* const wempty = wfull + S::WB;
    uint64_t* const ready = wempty + S::WB;      // leader: both CTAs' operands of the stage are where the MMAs read them
    uint64_t* const done = ready + S::NR;        // the stage's MMAs have retired: its operands may be overwritten
    uint64_t* const acc_full = done + S::NR;
    uint64_t* const acc_empty = acc_full + S::ACC;
    uint32_t* const s_tmem = reinterpret_cast<uint32_t*>(acc_empty + S::ACC);
    int* const s_error = reinterpret_cast<int*>(s_tmem + 1);
    int* const s_finish = s_error + 1;           // this CTA completed the tile whose partial sums it just stored
    int* const s_verdict = s_finish + 1;         // the quantiser rejected the input: nothing is to be written

    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const int cluster_id = blockIdx.x >> 1;
    constexpr bool swiglu = SWIGLU;
    const int KB = p.KB;
    const int nst = (KB + PS_SK - 1) / PS_SK;                          // stages of a tile
    // Every cluster takes a run of items over all of K, or (split > 1) one of the `split` parts of one tile's stages.
    const int per_tile = (p.M + p.unit - 1) / p.unit, split = p.split;
    const int part = cluster_id % split;
    const int it0 = nst * part / split, it1 = nst * (part + 1) / split;
    const unsigned unit0 = split > 1 ? (unsigned)(cluster_id / split) : persist_bound(p.share, per_tile, p.snap, cluster_id);
    const unsigned unit1 = split > 1 ? unit0 + 1 : persist_bound(p.share, per_tile, p.snap, cluster_id + 1);
    // an item: pair of channel tiles, first token, tokens the MMAs take (a multiple of 32)
    struct Item { int tile, tok0, width; };
    PersistItems items(unit0, unit1, per_tile, p.most);
    auto next_item = [&](Item& item) -> bool {
        int first, n;
        if (!items.next(item.tile, first, n)) return false;
        item.tok0 = first * p.unit;
        item.width = min(n * p.unit, (p.M - item.tok0 + 31) & ~31);
        return true;
    };
    Item item;
    const unsigned long long deadline = global_ns() + p.timeout_ns;
    // optional cycle stamps of cluster 0's leader: [item j < 16][8] = MMA issuer begins, [2] its last
    // commit, [3] epilogue sees the accumulator, [4] tensor memory handed back, [5] stored; [128] / [129] cycles unpack warp 0 waited
    // for weights / for a free tensor-memory buffer, [160] cycles for activations; [200] = clusters in the grid
    unsigned long long* const trace = (p.trace && blockIdx.x == 0) ? p.trace : nullptr;
    const long long c0 = clock64();
#define PS_STAMP(j, slot) do { if (trace && (j) < 16) trace[(j) * 8 + (slot)] = (unsigned long long)(clock64() - c0); } while (0)
    if (trace && tid == 0) trace[200] = (unsigned long long)num_clusters;

    // Set-up: a CTA that could only start when one of the launch in front left is late with its weights and everything behind them,
    // so nobody waits for more than it needs.  The weight producer makes the barriers (a lane each) and requests weights at once; it
    // and the epilogue warps report here and settle later.
    if (warp == 2) {
        for (int i = lane; i < S::BARRIERS; i += 32) mbar_init(&xfull[i], S::arrivals(i));
        mbar_fence_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (lane == 0) { *s_error = 0; *s_finish = 0; }
        __syncwarp();
    } else if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(PS_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    if (warp == 2 || warp >= S::EPI_WARP0) {
        asm volatile("bar.arrive 2, %0;" ::"n"(S::THREADS) : "memory");
        cluster_arrive();
    } else {
        asm volatile("bar.sync 2, %0;" ::"n"(S::THREADS) : "memory");
        asm volatile("bar.arrive 3, %0;" ::"n"(S::THREADS) : "memory");
        cluster_arrive();
        cluster_wait();   // the peer's barriers and tensor memory exist from here on
        tc_fence_after();
    }
    auto settle = [&]() {
        asm volatile("bar.sync 3, %0;" ::"n"(S::THREADS) : "memory");
        cluster_wait();
        tc_fence_after();
    };

    // What does not depend on the kernel in front -- requesting weights, unpacking the first of them into tensor
    // memory -- starts before the dependency wait.  Where the quantiser rejected the input the contraction runs all the same
    // and the epilogue drops its sums: whoever loads activations need not wait for the verdict (a trip to L2).

    if (warp == 2) {
        // ---------------------------------------------------------------- weight producer
        // (the whole warp walks the loop and one elected lane issues, as in the MMA issuer below: copy requests take their
        // operands from uniform registers, and four lanes issuing one request each took 1000 cycles per stage)
        RingPos<S::XW> r;
        bool ok = true, settled = false;
        int g = 0;
        const size_t group_bytes = (size_t)KB * GB;
        const size_t upper = swiglu ? (size_t)(p.F / GROUP) * group_bytes : 2 * group_bytes;   // groups 2, 3 behind groups 0, 1
        while (ok && next_item(item)) {
            const int ct = 2 * item.tile + (int)rank;
            const uint8_t* src = p.Wp + (size_t)(swiglu ? ct * 2 : ct * 4) * group_bytes + (size_t)it0 * (W8 ? 4 : 1) * PS_SK * GB;
            for (int it = it0; it < it1; ++it, ++g, r.next()) {
                if (g == S::XW) {                              // (slots come back once the MMAs have activations)
                    settle();
                    pdl_wait();
                    settled = true;
                }
                const uint32_t bytes = (uint32_t)min(PS_SK, KB - PS_SK * it) * GB;
                if (ok && g >= S::XW) ok = __all_sync(0xffffffffu, W8 ? mbar_wait_cluster(&done[r.slot], r.phase ^ 1u, deadline) : mbar_wait(&wempty[r.slot], r.phase ^ 1u, deadline));
                if (!ok) { *s_error = 1; break; }
                uint8_t* const dst = wts + (size_t)r.slot * S::XW_BYTES;
                if (elect_one()) {
                    if constexpr (W8) {                        // a k-block of a channel tile is contiguous
                        mbar_arrive_expect_tx(&xfull[r.slot], 4u * bytes);
                        bulk_g2s(dst, src, 4u * bytes, &xfull[r.slot]);
                    } else {
                        mbar_arrive_expect_tx(&wfull[r.slot], 4u * bytes);
                        bulk_g2s(dst, src, bytes, &wfull[r.slot]);
                        bulk_g2s(dst + PS_SK * GB, src + group_bytes, bytes, &wfull[r.slot]);
                        bulk_g2s(dst + 2 * PS_SK * GB, src + upper, bytes, &wfull[r.slot]);
                        bulk_g2s(dst + 3 * PS_SK * GB, src + upper + group_bytes, bytes, &wfull[r.slot]);
                    }
                }
                __syncwarp();
                src += (W8 ? 4 : 1) * PS_SK * GB;
            }
        }
        if (!settled) settle();
    } else if (warp == 0) {
        // ---------------------------------------------------------------- activation producer
        {
            PersistItems first = items;
            int tile, at, n;
            if (lane == 0 && first.next(tile, at, n)) tensor_prefetch_map(&maps.box[min(n * p.unit, (p.M - at * p.unit + 31) & ~31) / 32 - 1]);
        }
        pdl_wait();
        RingPos<S::XA> r;
        bool ok = true;
        int g = 0;
        while (ok && next_item(item)) {
            const int rows = item.width / 2;               // of this CTA's half
            const int row0 = item.tok0 + (int)rank * rows;
            const CUtensorMap* const box = &maps.box[rows / 16 - 1];
            for (int it = it0; it < it1; ++it, ++g, r.next()) {
                if (g >= S::XA) ok = __all_sync(0xffffffffu, mbar_wait_cluster(&done[(g - S::XA) % S::NR], (g - S::XA) / S::NR & 1, deadline));
                if (!ok) { *s_error = 1; break; }
                if (elect_one()) {
                    // (a stage's second k-block that does not exist is filled with zeros)
                    mbar_arrive_expect_tx(&xfull[r.slot], (uint32_t)rows * (PS_SK * 128u));
                    tensor_g2s(acts + (size_t)r.slot * S::XA_BYTES, box, row0, it * PS_SK, &xfull[r.slot]);
                }
                __syncwarp();
            }
        }
        // The MMAs' commits arrive on this CTA's barriers asynchronously, the peer's among them: the CTA may not leave
        // (and its shared memory change hands) before the last of them is here.
        for (int k = max(0, g - S::XA); k < g && !*reinterpret_cast<volatile int*>(s_error); ++k)
            if (!mbar_wait_cluster(&done[k % S::NR], k / S::NR & 1, deadline)) *s_error = 1;
    } else if (warp == 3) {
        // ---------------------------------------------------------------- voucher
        // The leader's MMAs read both CTAs' shared memory: this warp passes on that this CTA's copies have landed.  It runs
        // ahead of the MMAs by the depth of the ring.  (When the unpack warps vouched for it, with an arrival that released
        // everything at cluster scope, that release bounded the whole loop: 730 cycles per k-block at K = 11008 against 525.)
        pdl_wait();
        if (lane == 0) {
            RingPos<S::XA> r;
            RingPos<S::NR> to;
            long long waited = 0;
            bool ok = true;
            while (ok && next_item(item))
                for (int it = it0; it < it1; ++it, r.next(), to.next()) {
                    const long long w0 = trace ? clock64() : 0;
                    ok = mbar_wait(&xfull[r.slot], r.phase, deadline);
                    if (!ok) { *s_error = 1; break; }
                    if (trace) waited += clock64() - w0;
                    if (rank != 0) mbar_arrive_remote(&ready[to.slot], 0); else mbar_arrive(&ready[to.slot]);
                }
            if (trace) trace[160] = (unsigned long long)waited;
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer (leader CTA)
        // The whole warp walks the loop, so that descriptors and addresses are warp-uniform values, and one elected lane
        // issues.  (A loop that only lane 0 enters moves every operand of every MMA into uniform registers first: 85
        // cycles per MMA.)  Everything a stage needs is known before the one in front is issued; what stands between two
        // stages' MMAs is one wait, one commit and a few additions.
        pdl_wait();
        if (rank == 0) {
            bool dead = false;                                     // (the elected lane's, always the same one)
            int issued = 0;                                        // items
            RingPos<S::ACC> rc;
            const uint32_t ready0 = smem_u32(ready), done0 = smem_u32(done);
            const uint64_t b_first = tc_smem_desc_rows128(smem_u32(acts));
            const uint64_t a_first = tc_smem_desc(smem_u32(wts), 2048u, 128u);        // W8
            const uint32_t b_hi = (uint32_t)(b_first >> 32), a_hi = (uint32_t)(a_first >> 32);
            const uint32_t b_lo0 = (uint32_t)b_first, a_lo0 = (uint32_t)a_first;
            const uint32_t b_lo_end = b_lo0 + (uint32_t)(S::XA * S::XA_BYTES / 16);
            const uint32_t tmem_base = *s_tmem, a_tmem0 = tmem_base + S::A_COL0;
            uint32_t b_lo = b_lo0, a_lo = a_lo0, a_tmem = a_tmem0, bar = 0, phase = 0;
            for (int j = 0; next_item(item); ++j, rc.next()) {
                const uint32_t idesc = tc_idesc_s8(256, item.width);
                const uint32_t block = 4u * (uint32_t)item.width;  // of descriptor address between a stage's k-blocks
                if (lane == 0) PS_STAMP(j, 0);
                if (j >= S::ACC) {   // the epilogue warps of both CTAs have read this accumulator's previous item
                    if (!__all_sync(0xffffffffu, mbar_wait_cluster(&acc_empty[rc.slot], rc.phase ^ 1u, deadline))) { *s_error = 1; break; }
                    tc_fence_after();
                }
                const uint32_t d_tmem = tmem_base + rc.slot * TOK;
                const bool odd_end = (KB & 1) && it1 == nst;       // the last stage has one k-block
                for (int it = it0; it < it1; ++it) {
                    // k-step q: 32 k: 32 bytes of the activations' rows, two 128-channel columns of int8 weights
                    const uint64_t b_desc = (uint64_t)b_hi << 32 | b_lo, a_desc = (uint64_t)a_hi << 32 | a_lo;
                    const uint32_t a_now = a_tmem;
                    const bool whole = !(odd_end && it == nst - 1);
                    if (elect_one()) {
                        if (!dead && !mbar_wait_cluster_at(ready0 + bar, phase, deadline)) { *s_error = 1; dead = true; }
                        if (!dead) {
                            tc_fence_after();
                            if constexpr (W8) {
                                tc_mma_i8_ss_pair(d_tmem, a_desc, b_desc, idesc, it != it0 ? 1u : 0u);
#pragma unroll
                                for (int q = 1; q < 4; ++q) tc_mma_i8_ss_pair(d_tmem, a_desc + 256u * q, b_desc + 2u * q, idesc, 1u);
                                if (whole) {
#pragma unroll
                                    for (int q = 4; q < 8; ++q) tc_mma_i8_ss_pair(d_tmem, a_desc + 256u * q, b_desc + block + 2u * (q - 4), idesc, 1u);
                                }
                            } else {
                                tc_mma_i8_ts_pair(d_tmem, a_now, b_desc, idesc, it != it0 ? 1u : 0u);
#pragma unroll
                                for (int q = 1; q < 4; ++q) tc_mma_i8_ts_pair_acc(d_tmem, a_now + 8 * q, b_desc + 2u * q, idesc);
                                if (whole) {
#pragma unroll
                                    for (int q = 4; q < 8; ++q) tc_mma_i8_ts_pair_acc(d_tmem, a_now + 8 * q, b_desc + block + 2u * (q - 4), idesc);
                                }
                            }
                            tc_commit_pair_at(done0 + bar);   // in both CTAs: the stage's operands may be overwritten once these MMAs retire
                            if (it == it1 - 1) tc_commit_pair(&acc_full[rc.slot]);
                        }
                    }
                    bar = bar == (S::NR - 1) * 8 ? 0 : bar + 8;
                    phase ^= bar == 0 ? 1u : 0u;
                    b_lo += (uint32_t)(S::XA_BYTES / 16);
                    if (W8) a_lo += (uint32_t)(S::XW_BYTES / 16);
                    if (b_lo == b_lo_end) { b_lo = b_lo0; a_lo = a_lo0; }
                    if constexpr (!W8) a_tmem = a_tmem == a_tmem0 + (S::ABUF - 1) * 64 ? a_tmem0 : a_tmem + 64;
                }
                __syncwarp();
                if (lane == 0) PS_STAMP(j, 2);
                ++issued;
            }
            // (the peer's last arrivals are waited for, so that none is on its way when this CTA leaves)
            if (split == 1)
                for (int j = max(0, issued - S::ACC); j < issued && !*reinterpret_cast<volatile int*>(s_error); ++j)
                    if (!mbar_wait_cluster(&acc_empty[j % S::ACC], j / S::ACC & 1, deadline)) *s_error = 1;
        }
    } else if (warp < S::EPI_WARP0) {
        // ---------------------------------------------------------------- weight unpack -> TMEM
        if constexpr (!W8) {
        const int q = warp & 3;
        const int set = (warp - PS_UNPACK_WARP0) >> 2;
        const uint32_t lane_addr = *s_tmem + ((uint32_t)(q * 32) << 16);
        // Which row of the staged weight groups feeds this thread's tensor-memory lane.  The epilogue's thread t reads lanes
        // t / 4 + 8 c; they hold channels 4 (t / 4) .. + 3 of the warp's group, or (SwiGLU) features 2 (t / 4), + 1 of sixteen,
        // gate values in lanes 0-15 and up values in lanes 16-31 (staged groups 0, 1 = gate, 2, 3 = up of the same 64
        // features).  The order inside those four (two) turns with t, so that eight neighbouring lanes read rows that are
        // different modulo eight: no bank conflicts.
        const int i8 = lane & 7;
        const int src_group = swiglu ? (q >> 1) + (lane >= 16 ? 2 : 0) : q;
        const int src_row = swiglu ? (q & 1) * 16 + 2 * i8 + (((lane >> 3) + (i8 >> 2)) & 1) : 4 * i8 + (((lane >> 3) + (i8 >> 1)) & 3);
        const bool tr = trace && warp == PS_UNPACK_WARP0 && lane == 0;
        long long wait_full = 0, wait_free = 0;
        RingPos<S::XW> rw;
        // The two sets take alternate stages.  A stage's packed words are read from shared memory while the previous
        // stage's stores to tensor memory are still on their way, so that the two latencies overlap.
        uint4 w[4 * PS_SK];                                    // 16-byte pieces of this lane's row
        bool ok = true;
        int n_stages = (int)(unit1 - unit0);                   // one item a unit, or fewer
        if (p.most != 1)
            for (n_stages = 0; next_item(item);) ++n_stages;
        n_stages *= it1 - it0;
        int it = it0;
        auto advance = [&]() { rw.next(); if (++it == it1) it = it0; };
        auto fetch = [&]() {
            const int kbs = min(PS_SK, KB - PS_SK * it);
            const long long w0 = tr ? clock64() : 0;
            ok = __all_sync(0xffffffffu, mbar_wait(&wfull[rw.slot], rw.phase, deadline));
            if (tr) wait_full += clock64() - w0;
            const uint4* src = reinterpret_cast<const uint4*>(wts + (size_t)rw.slot * S::XW_BYTES + src_group * PS_SK * GB) + src_row;
#pragma unroll
            for (int c = 0; c < 4 * PS_SK; ++c) w[c] = (c < 4 * kbs) ? src[c * 32] : make_uint4(0u, 0u, 0u, 0u);
        };
        for (int k = 0; k < set; ++k) advance();
        if (set < n_stages) fetch();
        for (int g = set; g < n_stages && ok; g += PS_UNPACK_SETS) {
            const int kbs = min(PS_SK, KB - PS_SK * it), b = g % S::ABUF;
            const bool reuse = g >= S::ABUF;
            // (before the first buffer comes back from the MMAs, which need the activations)
            if (reuse && g - PS_UNPACK_SETS < S::ABUF) pdl_wait();
            const long long w0 = tr ? clock64() : 0;
            if (reuse) ok = __all_sync(0xffffffffu, mbar_wait_cluster(&done[(g - S::ABUF) % S::NR], (g - S::ABUF) / S::NR & 1, deadline));
            if (tr) wait_free += clock64() - w0;
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < PS_SK; ++h)
                if (h < kbs) {
#pragma unroll
                    for (int e = 0; e < 2; ++e) {              // (sixteen columns at a time: fewer registers)
                        uint32_t r[16];
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const uint4 v = w[4 * h + 2 * e + c];
                            const uint32_t ww[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int jj = 0; jj < 4; ++jj) {
                                r[c * 8 + jj] = (ww[jj] << 4) & 0xF0F0F0F0u;
                                r[c * 8 + 4 + jj] = ww[jj] & 0xF0F0F0F0u;
                            }
                        }
                        tc_st16(lane_addr + S::A_COL0 + b * 64 + h * 32 + e * 16, r);
                    }
                }
            __syncwarp();
            if (lane == 0) mbar_arrive(&wempty[rw.slot]);      // the packed copy has been read
#pragma unroll
            for (int k = 0; k < PS_UNPACK_SETS; ++k) advance();
            if (g + PS_UNPACK_SETS < n_stages) fetch();
            tc_wait_st();
            tc_fence_before();
            // Tensor-memory writes are ordered by the wait and the fences; the arrival itself carries nothing, so it is
            // relaxed (see mbar_arrive_remote for what a release at cluster scope costs).
            __syncwarp();
            if (lane == 0) { if (rank != 0) mbar_arrive_remote_relaxed(&ready[g % S::NR], 0); else mbar_arrive_relaxed(&ready[g % S::NR]); }
        }
        if (!ok) *s_error = 1;
        if (tr) { trace[128] = (unsigned long long)wait_full; trace[129] = (unsigned long long)wait_free; }
        }
    } else {
        // ---------------------------------------------------------------- epilogue warps
        // A warp finishes sixteen tokens of its 32 accumulator rows per turn of a rolled loop.  What bounds it is the
        // number of instructions: eight warps share the issue slots with the unpack warps and the MMA issuer, so nothing is
        // exchanged between lanes but row maxima, the arithmetic works on pairs of tokens (one instruction per two
        // operations), the int4 records' 1/16 is in the token scales, one look at the largest magnitude of eight gate values
        // settles that none needs the slow division, and maxima are taken of floats, whose signs the instruction drops.
        // (Small ones are settled by the scales: a sum is zero, where the fast form is exact, or at least one.  Looking for
        // the smallest magnitude as well sent every fourth turn to the slow form, one sum in eight hundred being zero.)
        const int q = warp & 3;                        // TMEM lane quarter this warp may read
        const int eset = (warp - S::EPI_WARP0) >> 2;   // takes pieces eset, eset + PS_EPI_SETS, ...
        const int sid = (warp - S::EPI_WARP0) * 32 + lane;   // 0..255 among the epilogue threads
        const int out_cols = swiglu ? p.F : p.N;
        // This thread's fragment: channels 4 i8 .. + 3 of its group (features 2 i8, + 1 of sixteen), the one in its c-th
        // tensor-memory lane is number (c + turn) of them; tokens 2 tq, 2 tq + 1 and eight further of a piece.
        const int i8 = lane >> 2, tq = lane & 3;
        const int turn = W8 ? 0 : swiglu ? i8 >> 2 : i8 >> 1;
        const int col = swiglu ? q * 16 + 2 * i8 : q * 32 + 4 * i8;      // its first channel inside the CTA's tile
        const int holder = 8 * (((lane & 3) - (W8 ? 0 : lane >> 3)) & 3) + (lane >> 2);       // the tensor-memory lane of the group's channel `lane`
        constexpr int CH = swiglu ? 2 : 4;
        const size_t elem = swiglu || p.epi != EPI_F16 ? 4 : 2;
        // All of them in one store; where the rows do not allow it a thread takes sixteen tokens of one channel instead, and a
        // warp's store covers 32 neighbouring channels of a token, in order (224 tokens of fp32 3070 -> 4911 20 us; 28 with
        // four scattered stores a token, and with the channels in the order of the tensor-memory lanes).
        const bool wide_ok = out_cols % CH == 0 && reinterpret_cast<uintptr_t>(p.out) % (CH * elem) == 0;
        const bool fragments = swiglu || wide_ok;
        constexpr int STEP = 16 * PS_EPI_SETS;
        constexpr int SHIFT = W8 ? 0 : 4;              // int4 records enter the MMA times 16
        if (sid < TOK) s_tilemax[sid] = 0u;            // (read behind barriers of the epilogue warps)
        pdl_wait();
        settle();
        const uint32_t lane_addr = *s_tmem + ((uint32_t)(q * 32) << 16);
        bool ok = true, good = true;
        if constexpr (!W8) {
            if (sid == 0) *s_verdict = take_verdict(p.status, p.report);
            if (blockIdx.x == 0) clear_maxima(p.rowmax_in, p.M, sid, 32 * PS_EPI_WARPS);
        }
        RingPos<S::ACC> rc;
        for (int j = 0; ok && next_item(item); ++j, rc.next()) {
            const int ct = 2 * item.tile + (int)rank;
            const int tok_base = item.tok0;
            const int n0 = (swiglu ? ct * 64 : ct * TILE_N) + col;
            float sw[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int n = n0 + ((c + turn) & (CH - 1));
                sw[c] = n < out_cols ? p.sw[(swiglu && c >= 2 ? p.F : 0) + n] : 0.f;
                if (swiglu && c >= 2) sw[c] = -sw[c];  // (the SiLU comes negated)
            }
            // pieces of sixteen tokens of this warp that hold live tokens: those at 16 eset + STEP k, k < pieces
            const int live = min(item.width, p.M - tok_base);
            int pieces = max(0, (live - 16 * eset + STEP - 1) / STEP);
            // Token scales, staged with the int4 records' 1/16 in them: (float)(16 s) * (sx / 16) is (float)s * sx, exactly,
            // unless sx / 16 is subnormal.  (The barrier at the end of an item keeps stragglers out.)
            float sx_here = 0.f;
            const bool mine = sid < live && sid < TOK;
            if (mine) sx_here = p.sx[tok_base + sid];
            if (sid < TOK) s_sx[sid] = W8 ? sx_here : sx_here * 0.0625f;
            const bool low = epilogue_any(mine && sx_here < PS_LOW);      // any scale that small: the careful ways below
            bool tiny = false;
            if (!W8 && low) {
                tiny = epilogue_any(mine && sx_here < 7.8886e-31f);
                if (tiny) {
                    if (sid < TOK) s_sx[sid] = sx_here;
                    asm volatile("bar.sync 1, %0;" ::"n"(32 * PS_EPI_WARPS) : "memory");
                }
            }
            // SwiGLU: no gate value of this thread is too small for the fast SiLU, whatever the sums are (zero is not)
            const bool gates_ok = swiglu && !low && (n0 >= out_cols || (sw[0] >= PS_LOW && sw[1] >= PS_LOW));
            ok = epilogue_all(mbar_wait_cluster(&acc_full[rc.slot], rc.phase, deadline));   // all eight warps or none
            if (!ok) { *s_error = 1; break; }
            if constexpr (!W8) good = *reinterpret_cast<volatile const int*>(s_verdict) == 0;
            if (sid == 0) PS_STAMP(j, 3);
            tc_fence_after();
            const uint32_t acc_addr = lane_addr + rc.slot * TOK + 16 * eset;
            auto hand_back = [&]() {   // this warp is done with the accumulator: another item's MMAs may overwrite it
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { if (rank != 0) mbar_arrive_remote_relaxed(&acc_empty[rc.slot], 0); else mbar_arrive_relaxed(&acc_empty[rc.slot]); }
                if (sid == 0) PS_STAMP(j, 4);
            };
            auto read_sums = [&](int k, uint32_t (&r)[16]) {
                if (fragments) {
                    tc_ld_16x256b_x2(acc_addr + STEP * k, r);
                    tc_ld_16x256b_x2(acc_addr + (16u << 16) + STEP * k, r + 8);
                } else tc_ld16(acc_addr + STEP * k, r);
                tc_wait_ld();
            };
            // ---- a part of a tile's K: the raw sums go to this CTA's slot, the tile's part counter is advanced, and the CTA
            // that completes it adds the other parts' slots to its own sums, which are still in tensor memory (integer
            // addition: exact in any order), and finishes the tile.  Nobody waits for anybody, and no slot needs clearing.
            // A slot holds what a thread reads in one turn, four sums at a time: [piece][4][thread of the lane quarters].
            const size_t tile_index = (size_t)unit0;
            const size_t slot_quads = 32 * (size_t)p.unit, part_stride = 2 * slot_quads;
            const int4* const slots = reinterpret_cast<const int4*>(p.partials) + (2 * split * tile_index + rank) * slot_quads + (size_t)(4 * eset) * 128 + q * 32 + lane;
            bool finish = true;
            if (!W8 && !good) pieces = 0;                  // a rejected input: the sums are dropped
            else if (split > 1) {
                int4* const slot = const_cast<int4*>(slots) + part * part_stride;
#pragma unroll 1
                for (int k = 0; k < pieces; ++k) {
                    uint32_t r[16];
                    read_sums(k, r);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        __stcg(slot + (size_t)(STEP / 4 * k + i) * 128, make_int4((int)r[4 * i], (int)r[4 * i + 1], (int)r[4 * i + 2], (int)r[4 * i + 3]));
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * PS_EPI_WARPS) : "memory");
                if (sid == 0) {
                    // (a tile with a part whose wait ran out is never completed; the launch reports the error and the host
                    // clears the counters)
                    // One addition that releases all of the warps' stores, behind the barrier, and acquires the other parts':
                    // a sequentially consistent fence on either side of it took longer (24 x 4096 -> 4096 8.95 us, now 8.45;
                    // 64 x 8192 -> 8192 14.1 and 13.6; 128 x 11008 -> 4096 17.9 and 17.5).
                    unsigned* const count = p.counts + 2 * tile_index + rank;
                    const bool last = atomic_add_acq_rel(count, 1u) == (unsigned)split - 1u;
                    if (last) *count = 0u;
                    *s_finish = last ? 1 : 0;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * PS_EPI_WARPS) : "memory");
                finish = *reinterpret_cast<volatile int*>(s_finish) != 0;
            }
            const int turns = finish ? pieces : 0;
            const int other = part == 0 ? 1 : 0;                          // the first of the other parts
            int4 ahead[4];                                                // its sums of the next turn, on their way
            auto fetch_part = [&](int4 (&v)[4], int which, int k) {
                const int4* const src = slots + which * part_stride + (size_t)(STEP / 4 * k) * 128;
#pragma unroll
                for (int h = 0; h < 4; ++h) v[h] = __ldcg(src + (size_t)h * 128);
            };
            if (split > 1 && turns) fetch_part(ahead, other, 0);
            if (pieces == 0 && split == 1) hand_back();
#pragma unroll 1
            for (int k = 0; k < turns; ++k) {
                const int t0 = 16 * eset + STEP * k + 2 * tq;             // this thread's first token of the turn
                const int left = live - t0;                              // its tokens t0 + {0, 1, 8, 9} below t0 + left exist
                uint32_t r[16];
                read_sums(k, r);
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
                if (!SWIGLU && !fragments) {
                    const int first = 16 * eset + STEP * k, rows = live - first;
                    const int n = ct * TILE_N + q * 32 + lane;
#pragma unroll
                    for (int i = 0; i < 16; ++i) r[i] = __shfl_sync(0xffffffffu, r[i], holder);
                    if (n < out_cols) {
                        const size_t at = (size_t)(tok_base + first) * out_cols + n;
                        auto store_rows = [&](auto* dst, auto value) {
                            if (rows >= 16) {
#pragma unroll
                                for (int i = 0; i < 16; ++i, dst += out_cols) *dst = value(i);
                            } else {
#pragma unroll
                                for (int i = 0; i < 16; ++i, dst += out_cols)
                                    if (i < rows) *dst = value(i);
                            }
                        };
                        if (p.epi == EPI_I32) store_rows(reinterpret_cast<int*>(p.out) + at, [&](int i) { return (int)r[i] >> SHIFT; });
                        else {
                            const F2 sw_own = f2_all(p.sw[n]);
#pragma unroll
                            for (int i = 0; i < 16; i += 2) {
                                F2 v = f2_pack(__int2float_rn((int)r[i]), __int2float_rn((int)r[i + 1]));
                                if (tiny) v = f2_mul(v, f2_all(0.0625f));
                                float lo, hi;
                                f2_unpack(f2_mul(f2_mul(v, *reinterpret_cast<const F2*>(s_sx + first + i)), sw_own), lo, hi);
                                r[i] = __float_as_uint(lo);
                                r[i + 1] = __float_as_uint(hi);
                            }
                            if (p.epi == EPI_F16) store_rows(reinterpret_cast<__half*>(p.out) + at, [&](int i) { return __float2half_rn(__uint_as_float(r[i])); });
                            else store_rows(reinterpret_cast<float*>(p.out) + at, [&](int i) { return __uint_as_float(r[i]); });
                        }
                    }
                    continue;
                }
                // r[8 (c / 2) + 4 h + 2 (c % 2) + e]: tensor-memory lane c, token t0 + 8 h + e
                if (!SWIGLU && p.epi == EPI_I32) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (8 * h + e < left && n0 < out_cols) {
                                uint32_t v[4];
#pragma unroll
                                for (int c = 0; c < 4; ++c) v[c] = (uint32_t)((int)r[8 * (c >> 1) + 4 * h + 2 * (c & 1) + e] >> SHIFT);
                                store_four(reinterpret_cast<uint32_t*>(p.out) + (size_t)(tok_base + t0 + 8 * h + e) * out_cols + n0, v, turn);
                            }
                    continue;
                }
                F2 y[4][2];                                               // [lane c][h]: tokens t0 + 8 h, + 1
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const F2 sx = *reinterpret_cast<const F2*>(s_sx + t0 + 8 * h);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t* const pair = r + 8 * (c >> 1) + 4 * h + 2 * (c & 1);
                        y[c][h] = f2_pack(__int2float_rn((int)pair[0]), __int2float_rn((int)pair[1]));
                        if (tiny) y[c][h] = f2_mul(y[c][h], f2_all(0.0625f));   // (float)(16 s) / 16 is (float)s, exactly
                        y[c][h] = f2_mul(f2_mul(y[c][h], sx), f2_all(sw[c]));
                    }
                }
                if (!SWIGLU) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float v[4][2];
#pragma unroll
                        for (int c = 0; c < 4; ++c) f2_unpack(y[c][h], v[c][0], v[c][1]);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const size_t at = (size_t)(tok_base + t0 + 8 * h + e) * out_cols + n0;
                            if (8 * h + e >= left || n0 >= out_cols) continue;
                            if (p.epi == EPI_F16) {
                                const __half2 lo = __floats2half2_rn(v[0][e], v[1][e]), hi = __floats2half2_rn(v[2][e], v[3][e]);
                                store_four_halves(reinterpret_cast<__half*>(p.out) + at, *reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi), turn);
                            } else {
                                const uint32_t four[4] = {__float_as_uint(v[0][e]), __float_as_uint(v[1][e]), __float_as_uint(v[2][e]), __float_as_uint(v[3][e])};
                                store_four(reinterpret_cast<uint32_t*>(p.out) + at, four, turn);
                            }
                        }
                    }
                } else {
                    // lanes 0, 1: gate values of two features, lanes 2, 3: their up values, negated
                    const bool n_ok = n0 < out_cols;                      // (features come in whole groups of 32)
                    F2 v[2][2];
                    float most = 0.f;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            float a, b;
                            f2_unpack(y[c][h], a, b);
                            most = max_abs(most, max_abs(a, b));
                        }
                    if (gates_ok && silu_fast(most)) {
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                float a, b, ya, yb;
                                f2_unpack(y[c][h], a, b);
                                minus_silu_poly2(a, b, ya, yb);
                                v[c][h] = f2_mul(f2_pack(ya, yb), y[c + 2][h]);
                            }
                    } else {
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                float a, b, ua, ub;
                                f2_unpack(y[c][h], a, b);
                                f2_unpack(y[c + 2][h], ua, ub);
                                v[c][h] = f2_pack(__fmul_rn(silu_poly(a), -ua), __fmul_rn(silu_poly(b), -ub));
                            }
                    }
                    float top[4];                                         // [2 h + e]: the larger of the two features
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float a[2], b[2];
                        f2_unpack(v[0][h], a[0], a[1]);
                        f2_unpack(v[1][h], b[0], b[1]);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            top[2 * h + e] = max_abs(a[e], b[e]);
                            if (n_ok && 8 * h + e < left) {
                                float* const dst = reinterpret_cast<float*>(p.out) + (size_t)(tok_base + t0 + 8 * h + e) * out_cols + n0;
                                const float first = turn ? b[e] : a[e], second = turn ? a[e] : b[e];
                                if (wide_ok) *reinterpret_cast<float2*>(dst) = make_float2(first, second);
                                else { dst[0] = first; dst[1] = second; }
                            }
                        }
                    }
                    if (p.rowmax) {
                        // Maxima over the sixteen features, one token per value: two folding steps that halve the values a
                        // lane holds and a plain one.  (Tokens and features that do not exist have zero scales, and zeros here.)
                        const bool far = (lane & 16) != 0, near = (lane & 8) != 0;
#pragma unroll
                        for (int e = 0; e < 2; ++e) top[e] = max_abs(far ? top[2 + e] : top[e], __shfl_xor_sync(0xffffffffu, far ? top[e] : top[2 + e], 16));
                        top[0] = max_abs(near ? top[1] : top[0], __shfl_xor_sync(0xffffffffu, near ? top[0] : top[1], 8));
                        const uint32_t bits = __float_as_uint(max_abs(top[0], __shfl_xor_sync(0xffffffffu, top[0], 4)));
                        // collected per CTA and item in shared memory first: one global atomic per token and item
                        // instead of one per token, item and sixteen features
                        if (!(lane & 4) && bits) atomicMax(&s_tilemax[t0 + (far ? 8 : 0) + (near ? 1 : 0)], bits);
                    }
                }
            }
            if (sid == 0) PS_STAMP(j, 5);
            asm volatile("bar.sync 1, %0;" ::"n"(32 * PS_EPI_WARPS) : "memory");   // every epilogue warp is done with this item's scales and maxima
            if (swiglu && good && p.rowmax && sid < TOK) {
                const uint32_t m = s_tilemax[sid];
                if (m) {
                    atomicMax(&p.rowmax[tok_base + sid], m);
                    s_tilemax[sid] = 0u;
                }
            }
        }
    }

    // ------------------------------------------------------------------------ teardown
    tc_fence_before();
    __syncthreads();
    // A wait that ran out ends its role at once, and copies requested just before may still be on their way into this CTA's
    // shared memory: they land within microseconds, so the CTA stays that long before it leaves.
    if (*reinterpret_cast<volatile int*>(s_error))
        for (const unsigned long long until = global_ns() + PS_DRAIN_NS; global_ns() < until;) __nanosleep(1000);
    // Neither CTA frees tensor memory or leaves while the other may still use it.  (Every arrival from the other CTA has been
    // waited for, so the barrier need not order memory: an arrival with a release waits for this CTA's results to be stored.)
    cluster_arrive_relaxed();
    cluster_wait();
    if (tid == 0 && *s_error) report_device_error(p.report);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(*s_tmem), "r"(PS_TMEM_COLS) : "memory");
    }
}

namespace {
constexpr long long PS_MAX_K = 131072;

int units_of(int columns, int M, int unit) { return ((columns - 1) / 256 + 1) * ((M - 1) / unit + 1); }

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
    cfg.blockDim = dim3(S::THREADS);
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
    const int units = units_of(p.epi == EPI_SWIGLU ? 2 * p.F : p.N, p.M, p.unit), clusters = persist_clusters(units, p.split, max_clusters);
    GemmParams q = p;
    q.share = persist_share((unsigned)units, (unsigned)clusters);
    cfg.gridDim = dim3((unsigned)(2 * clusters), 1, 1);
    int n = 1;
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, q, *p.maps, clusters);
}
} // namespace


PersistPlan gemm_tc_persist_plan(int columns, int M, int KB, bool w8, bool swiglu, int sm_count)
{
    PersistPlan cut{};
    const char* const text = std::getenv("RK_NPU_B200_PERSIST_CUT");   // experiments and tests: "unit,most,snap,split"
    if (text && std::sscanf(text, "%d,%d,%d,%d", &cut.unit, &cut.most, &cut.snap, &cut.split) == 4 && persist_cut_ok(cut, KB)) return cut;
    return persist_plan(columns, M, KB, w8, swiglu, sm_count);
}
size_t gemm_tc_persist_slot_bytes(int columns, int M, const PersistPlan& plan)
{
    return plan.split > 1 ? 2 * size_t(units_of(columns, M, plan.unit)) * size_t(plan.split) * 128 * size_t(plan.unit) * sizeof(int) : 0;
}
size_t gemm_tc_persist_count_bytes(int columns, int M, const PersistPlan& plan)
{
    return plan.split > 1 ? 2 * size_t(units_of(columns, M, plan.unit)) * sizeof(unsigned) : 0;
}

bool make_persist_maps(PersistMaps& maps, const uint8_t* codes, int M, int KB)
{
    static const auto encode = []() {
        void* entry = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &entry, 12000, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            entry = nullptr;
        }
        return reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(entry);
    }();
    if (!encode) return false;
    const cuuint64_t dims[3] = {128, (cuuint64_t(M) + PERSIST_TOKENS - 1) / PERSIST_TOKENS * PERSIST_TOKENS, cuuint64_t(KB)};
    const cuuint64_t strides[2] = {cuuint64_t(KB) * 128, 128};
    const cuuint32_t steps[3] = {1, 1, 1};
    for (int i = 0; i < 8; ++i) {
        const cuuint32_t box[3] = {128, 16u * (i + 1), PS_SK};
        if (encode(&maps.box[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(codes), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    return true;
}

cudaError_t launch_gemm_tc_persist(const GemmParams& p, cudaStream_t stream, bool pdl)
{
    if (!p.maps) return cudaErrorInvalidValue;
    const int width = p.unit * p.most;   // picks the kernel
    if ((long long)p.KB * KBLOCK > PS_MAX_K || p.T != PERSIST_T || p.unit < 32 || p.unit % 32 || p.most < 1 || width > PS_WIDEST || p.split < 1 ||
        (p.split > 1 && !(p.most == 1 && p.partials && p.counts)))
        return cudaErrorInvalidValue;
    if (p.w8) {
        if (p.epi == EPI_SWIGLU) return cudaErrorInvalidValue;
        return width <= PS_NARROW ? launch_persist_inst<true, false, PS_NARROW>(p, stream, pdl) : launch_persist_inst<true, false, PS_WIDEST>(p, stream, pdl);
    }
    if (p.epi == EPI_SWIGLU)
        return width <= PS_NARROW ? launch_persist_inst<false, true, PS_NARROW>(p, stream, pdl)
             : width <= PS_WIDE   ? launch_persist_inst<false, true, PS_WIDE>(p, stream, pdl)
                                  : launch_persist_inst<false, true, PS_WIDEST>(p, stream, pdl);
    return width <= PS_NARROW ? launch_persist_inst<false, false, PS_NARROW>(p, stream, pdl)
         : width <= PS_WIDE   ? launch_persist_inst<false, false, PS_WIDE>(p, stream, pdl)
                              : launch_persist_inst<false, false, PS_WIDEST>(p, stream, pdl);
}

} // namespace rkb200

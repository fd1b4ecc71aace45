// moe_kernels.cu -- routed SwiGLU experts with int8 weights (the original's rk_npu_moe_w8 operator) for sm_100a.
//
// The original gathers each expert's rows on the NPU, runs int8 GEMMs there and does the middle stage
// (dequantise, SwiGLU, row maximum, nearest-even re-quantisation; src/rk_npu_moe_cpu.cpp:47-115) and the
// weighted combine (src/rk_npu_moe_w8.cpp:786-816) on the CPU.  Here the whole operator is byte work streamed
// from HBM/L2: an expert's weights are read once per job of up to 16 assignments, in records laid out in the
// register order of mma.sync.m16n8k32 so that every warp load is 512 contiguous bytes; the gathered activation
// rows sit in shared memory; sums are exact int32.
//
//   moe_intake_kernel     a small run's piece from page-locked host memory to the device; fp32 rows -> int8 codes + scales,
//                         nearest-even, scale = max/127 (1 for a zero row)
//   moe_project_kernel    gate/up: (float(sum) * s_in) * s_w, y = silu(gate) * up (degree-7 polynomial shared with the dense
//                         path), fp32 middle rows + atomicMax of |y| bit patterns per assignment;
//                         down: re-quantised middle rows, int8 GEMM over I, (float(sum) * s_mid) * s_w
//   moe_combine_kernel    out[token] = sum over the token's slots, in slot order, one fused multiply-add each
#include "moe_device.h"
#include "w4a8_math.cuh"
#include "w4a8_ptx.cuh"
#include "w4a8_tc.cuh"
#include <algorithm>

namespace rkb200 {

namespace {
constexpr int MOE_WARPS = 8;                 // contraction warps of a group
constexpr int MOE_GROUP = 32 * MOE_WARPS;    // and its threads; one more warp of the CTA streams the weights
constexpr int MOE_STAGE_RECORDS = 16;        // 16-channel x 128-k records in a stage
constexpr int MOE_STAGE_BYTES = MOE_STAGE_RECORDS * 2048;            // 32 KB (half of it for int4 records)
constexpr int MOE_RING_MOST = 5;
constexpr int MOE_TURNS = 16;                // announced items: more than the ring can hold, with the closing ones
constexpr int MOE_PARTIAL = MOE_WARPS * 8 * 32;                      // int32 sums of an item
constexpr int MOE_ROW_PAD = 16;              // bytes between activation rows in shared memory beyond K: conflict-free fragment loads
constexpr size_t MOE_SMEM_MOST = 218 * 1024;     // (scales, barriers and announced items are static shared memory)

__host__ __device__ constexpr int moe_row_bytes(int K) { return (K + MOE_KQ - 1) / MOE_KQ * MOE_KQ + MOE_ROW_PAD; }
__host__ __device__ constexpr size_t moe_group_bytes(int K) { return size_t(MOE_JOB_ROWS) * moe_row_bytes(K) + 2 * MOE_PARTIAL * 4; }
// Two groups of warps wherever two stages fit beside their rows; one for the longest rows.
__host__ __device__ constexpr int moe_groups(int K) { return 2 * moe_group_bytes(K) + 2 * MOE_STAGE_BYTES <= MOE_SMEM_MOST ? 2 : 1; }
__host__ __device__ constexpr int moe_ring(int K)
{
    const int fit = int((MOE_SMEM_MOST - moe_groups(K) * moe_group_bytes(K)) / MOE_STAGE_BYTES);
    return fit < MOE_RING_MOST ? fit : MOE_RING_MOST;
}
static_assert(moe_ring(8192) >= 2, "two stages fit beside the longest rows");

__device__ __forceinline__ int8_t nearest_even_code(float v)
{
    return (int8_t)__float2int_rn(fminf(fmaxf(v, -127.f), 127.f));
}

// `kqs` 128-k records of one 16-channel block in shared memory against up to 16 activation rows: c[half] += W(16 x k) * X^T.
// Fragment mapping of m16n8k32 (g = lane / 4, t = lane % 4): A regs = channels g / g + 8 at k = 4t.. and 16 + 4t..; B regs
// = token g at the same k; C regs = channels g, g + 8 x tokens 2t, 2t + 1.  NIB: int4 records (two 16-byte pieces per 128 k
// instead of four); the sums come out times 16.
template <bool TWO, bool NIB>
__device__ __forceinline__ void block_mma(const uint4* w, const uint8_t* x0, int row_bytes, int kqs, int lane, int (&c)[2][4])
{
    const uint8_t* x1 = x0 + (size_t)8 * row_bytes;
#pragma unroll 2
    for (int kq = 0; kq < kqs; ++kq, w += NIB ? 64 : 128, x0 += MOE_KQ, x1 += MOE_KQ) {
        uint4 a[NIB ? 2 : 4];
#pragma unroll
        for (int s = 0; s < (NIB ? 2 : 4); ++s) a[s] = w[s * 32 + lane];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t b0 = *reinterpret_cast<const uint32_t*>(x0 + s * 32), b1 = *reinterpret_cast<const uint32_t*>(x0 + s * 32 + 16);
            uint32_t d0 = 0, d1 = 0;
            if (TWO) { d0 = *reinterpret_cast<const uint32_t*>(x1 + s * 32); d1 = *reinterpret_cast<const uint32_t*>(x1 + s * 32 + 16); }
            uint32_t a0, a1, a2, a3;
            if (NIB) {
                const uint4 v = a[s >> 1];
                const uint32_t wx = (s & 1) ? v.z : v.x, wy = (s & 1) ? v.w : v.y;
                a0 = (wx << 4) & 0xF0F0F0F0u; a2 = wx & 0xF0F0F0F0u;
                a1 = (wy << 4) & 0xF0F0F0F0u; a3 = wy & 0xF0F0F0F0u;
            } else {
                const uint4 v = a[NIB ? 0 : s];
                a0 = v.x; a1 = v.y; a2 = v.z; a3 = v.w;
            }
            mma_s8(c[TWO ? 0 : s & 1], a0, a1, a2, a3, b0, b1);      // (one half of tokens: two chains of sums instead)
            if (TWO) mma_s8(c[1], a0, a1, a2, a3, d0, d1);
        }
    }
}
} // namespace

// ------------------------------------------------------------------ weights -> records
__global__ void __launch_bounds__(256) moe_pack_kernel(const MoePackParams p)
{
    const int kq_count = (p.K + MOE_KQ - 1) / MOE_KQ;
    const int pieces = p.nibbles ? 2 : 4;
    const size_t total = (size_t)(p.N / 16) * kq_count * pieces * 32;
    auto code = [&](int k, int n) -> uint32_t { return k < p.K ? (uint32_t)(uint8_t)p.W[(size_t)k * p.N + n] : 0u; };
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int lane = (int)(i & 31), piece = (int)((i >> 5) % pieces);
        const size_t rec = (i >> 5) / pieces;
        const int kq = (int)(rec % kq_count), cb = (int)(rec / kq_count);
        const int g = lane >> 2, t = lane & 3;
        uint32_t word[4];
        if (p.nibbles) {
            // piece = k-steps 2 piece, 2 piece + 1; words: (step, channel g), (step, g + 8), (step + 1, g), (step + 1, g + 8)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int k0 = kq * MOE_KQ + (2 * piece + (r >> 1)) * 32 + 4 * t, n = cb * 16 + g + (r & 1) * 8;
                uint32_t v = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) v |= ((code(k0 + j, n) & 15u) | ((code(k0 + 16 + j, n) & 15u) << 4)) << (8 * j);
                word[r] = v;
            }
        } else {
            const int k0 = kq * MOE_KQ + piece * 32 + 4 * t, n0 = cb * 16 + g;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int k = k0 + (r >> 1) * 16, n = n0 + (r & 1) * 8;
                uint32_t v = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) v |= code(k + j, n) << (8 * j);
                word[r] = v;
            }
        }
        reinterpret_cast<uint4*>(p.packed)[i] = make_uint4(word[0], word[1], word[2], word[3]);
    }
}

// ------------------------------------------------------------------ intake (fp32 rows -> codes: src/rk_npu_moe_w8.cpp:317-343)
// Blocks below row_blocks take a row each; the others carry the rest of a piece that is still in host memory (header and
// schedule) to the device.  Nothing is asked of the header where that can be avoided: an fp32 row is requested before the
// header is known to name it (moe_row_plan keeps every row of the grid inside the piece) and stays in registers between its
// maximum and its codes: one trip over the bus, not three.
constexpr int MOE_INTAKE_THREADS = 256, MOE_INTAKE_MOVERS = 8;
constexpr int MOE_INTAKE_BLIND = MOE_INTAKE_MOVERS * MOE_INTAKE_THREADS * 16;    // moved without asking how much of it is in use
__global__ void __launch_bounds__(MOE_INTAKE_THREADS) moe_intake_kernel(const MoeIntakeParams p)
{
    __shared__ uint32_t s_max[MOE_INTAKE_THREADS / 32];
    pdl_launch_dependents();
    const uint8_t* const piece = p.from ? p.from : p.upload;
    const MoeRun* const run = moe_piece<MoeRun>(piece, 0);
    const int row_blocks = gridDim.x - (p.from ? MOE_INTAKE_MOVERS : 0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if ((int)blockIdx.x >= row_blocks) {
        const int step = MOE_INTAKE_MOVERS * MOE_INTAKE_THREADS;
        const uint4* const src = reinterpret_cast<const uint4*>(piece);
        uint4* const dst = reinterpret_cast<uint4*>(p.upload);
        const int end = (int)((p.input_at <= MOE_INTAKE_BLIND ? p.input_at : run->used) / 16);
#pragma unroll 4
        for (int i = ((int)blockIdx.x - row_blocks) * MOE_INTAKE_THREADS + tid; i < end; i += step) dst[i] = src[i];
        return;
    }
    const int row = blockIdx.x;
    if (!p.f32) {
        const uint4* const src = reinterpret_cast<const uint4*>(piece + p.input_at + (size_t)row * p.H);       // H is a multiple of 32
        uint4* const dst = reinterpret_cast<uint4*>(p.upload + p.input_at + (size_t)row * p.H);
        if (row < run->rows)
            for (int i = tid; i < p.H / 16; i += MOE_INTAKE_THREADS) dst[i] = src[i];
        return;
    }
    constexpr int MOST = 8192 / 4 / MOE_INTAKE_THREADS;
    const float4* const x = reinterpret_cast<const float4*>(piece + p.input_at) + (size_t)row * (p.H / 4);
    const int quads = p.H / 4;
    float4 v[MOST];
#pragma unroll
    for (int k = 0; k < MOST; ++k) {
        const int i = k * MOE_INTAKE_THREADS + tid;
        v[k] = i < quads ? x[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (row >= run->rows) return;
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < MOST; ++k)
        m = max(m, max(max(__float_as_uint(v[k].x) & 0x7fffffffu, __float_as_uint(v[k].y) & 0x7fffffffu),
                       max(__float_as_uint(v[k].z) & 0x7fffffffu, __float_as_uint(v[k].w) & 0x7fffffffu)));
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) s_max[warp] = m;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MOE_INTAKE_THREADS / 32; ++i) m = max(m, s_max[i]);
    const float scale = m ? __fdiv_rn(__uint_as_float(m), 127.f) : 1.f;
    const float inverse = __frcp_rn(scale);
    if (m >= 0x7f800000u || !(scale > 0.f) || (__float_as_uint(inverse) & 0x7fffffffu) >= 0x7f800000u) {     // an infinite or NaN element is the largest pattern
        if (tid == 0) p.status->bad_input = 1;
        return;
    }
    if (tid == 0) p.scales[row] = scale;
    uint32_t* const q = reinterpret_cast<uint32_t*>(p.codes + (size_t)row * p.H);
#pragma unroll
    for (int k = 0; k < MOST; ++k) {
        const int i = k * MOE_INTAKE_THREADS + tid;
        if (i < quads)
            q[i] = (uint32_t)(uint8_t)nearest_even_code(__fmul_rn(v[k].x, inverse)) | (uint32_t)(uint8_t)nearest_even_code(__fmul_rn(v[k].y, inverse)) << 8 |
                   (uint32_t)(uint8_t)nearest_even_code(__fmul_rn(v[k].z, inverse)) << 16 | (uint32_t)(uint8_t)nearest_even_code(__fmul_rn(v[k].w, inverse)) << 24;
    }
}

// ------------------------------------------------------------------ the two projections
// Byte work: every expert's weights cross HBM once per job of up to 16 assignments.  The work is a flat list of items for one
// persistent CTA per SM: a job and two 16-channel gate blocks with their two up blocks, or a job and eight 16-column blocks of
// the down projection.  One warp streams the items' records and scales through a ring of 32 KB stages with bulk copies, ahead
// of the contraction, so that 64 to 160 KB per SM are on their way whatever the other warps do.  Two groups of eight warps
// take the items in turn, each with activation rows of its own, so that one finishes or gathers while the other contracts
// (one group alone cannot keep up with the memory).  Down: a warp has a block and all of K (at most 512), and its sums never
// leave its registers.  Gate/up: a warp has a block and half of each stage's K; the sums of an item meet in shared memory.
// A job's activation rows are brought into shared memory when a group's job changes: the int8 codes, or, for the down
// projection, the middle rows re-quantised with their row scale max/127 (nearest-even; src/rk_npu_moe_cpu.cpp:78-80).
// SMs do not get equal shares of the memory: with the list cut evenly the first CTA was done after 26 us and the last after
// 38.  So a CTA owns a contiguous share of three quarters of a long list and takes the rest from a common counter, item by
// item; a list of fewer than eight items per CTA is cut evenly (a turn at the counter costs a microsecond).
// 64 rows over 128 + 1 int8 experts of 1536 x 512, 305 MB of weights, with an event on either side of each launch: gate/up
// 53 -> 43 us, down 39 -> 33 us (before: a CTA per item with register double buffering, a quarter as much in flight, and a
// CTA's start and its gather paid per item).  The whole call 190 -> 150 us, one token over int4 experts 36 -> 29 us, of which
// the launch takes 11 us, and the trips over the bus at either end 16 + 20 us at 64 rows.
template <bool DOWN>
__global__ void __launch_bounds__(2 * MOE_GROUP + 32, 1) moe_project_kernel(const MoeProjectParams p)
{
    extern __shared__ __align__(128) uint8_t smem[];
    // A stage's full barrier belongs to the group that reads it: a group waits on a parity only after it has seen the phase
    // before (copies land out of order, and a slot's last stage may be the other group's and still on its way).
    __shared__ __align__(8) uint64_t full[2][MOE_RING_MOST], empty[MOE_RING_MOST], told[MOE_TURNS];
    __shared__ int4 s_turn[MOE_TURNS];                                     // item (-1: no more), first assignment, rows, int4 records
    __shared__ __align__(16) float s_w[MOE_TURNS][(DOWN ? 8 : 4) * 16];        // and the scales of its channels
    __shared__ float s_scales[2][MOE_JOB_ROWS];
    const int K = DOWN ? p.I : p.H;
    const int kq_count = (K + MOE_KQ - 1) / MOE_KQ, row_bytes = moe_row_bytes(K);
    const int R = moe_ring(K), groups = moe_groups(K);
    constexpr int BLOCKS = DOWN ? 8 : 4, STAGE_KQ = MOE_STAGE_RECORDS / BLOCKS;    // of a stage: its blocks, and 128-k records of each
    constexpr int PER_ITEM = DOWN ? BLOCKS : BLOCKS / 2, BLOCK_STAGE = STAGE_KQ * 2048;
    const int stages = (kq_count + STAGE_KQ - 1) / STAGE_KQ;               // of an item
    uint8_t* const ring = smem;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < R; ++i) { mbar_init(&full[0][i], 1); mbar_init(&full[1][i], 1); mbar_init(&empty[i], MOE_WARPS); }
        for (int i = 0; i < MOE_TURNS; ++i) mbar_init(&told[i], 1);
        mbar_fence_init();
    }
    __syncthreads();
    // The schedule is the intake's work: gate/up waits for it before it lets the down projection's CTAs in, which can then
    // read the schedule and request weights (these never change) while gate/up still runs.
    if (!DOWN) pdl_wait();
    pdl_launch_dependents();
    const MoeRun* const run = moe_piece<MoeRun>(p.upload, 0);
    const int* const job_expert = moe_piece<int>(p.upload, run->job_expert), *const job_first = moe_piece<int>(p.upload, run->job_first);
    const int* const job_rows = moe_piece<int>(p.upload, run->job_rows);
    const MoeBank bank = DOWN ? run->down.bank : run->gate_up.bank;
    const float* const all_scales = DOWN ? run->down.scales : run->gate_up.scales;
    const int blocks = DOWN ? p.H / 16 : p.I / 16;                       // 16-channel blocks to cover per job (gate blocks)
    const int per_job = (blocks + PER_ITEM - 1) / PER_ITEM;
    const int total = run->jobs * per_job;

    if (tid >= groups * MOE_GROUP) {
        // ---------------------------------------------------------------- the copy warp
        const int owned = total >= 8 * (int)gridDim.x ? total - total / 4 : total;
        int item = (int)((long long)owned * blockIdx.x / gridDim.x), last = (int)((long long)owned * (blockIdx.x + 1) / gridDim.x);
        int slot = 0, issued = 0, turn = 0;
        uint32_t phase = 0;
        unsigned long long deadline = 0;
        int job = -1, first = 0, rows = 0;
        bool nib = false, failed = false;
        const uint8_t* base = nullptr;
        const float* ws = nullptr;
        uint32_t armed[2] = {}, used[2] = {};                            // per group: the phase each slot is armed in, and whether it ever was
        size_t block_bytes = 0;
        for (;;) {
            if (item == last) {
                if (owned == total) break;
                if (lane == 0) item = owned + (int)atomicAdd(p.tickets + DOWN, 1u);
                item = __shfl_sync(0xffffffffu, item, 0);
                if (item >= total) break;
                last = item + 1;
            }
            if (item / per_job != job) {
                job = item / per_job;
                const int expert = job_expert[job];
                first = job_first[job];
                rows = job_rows[job];
                base = bank.expert(expert);
                nib = bank.nibbles(expert);
                ws = bank.scales(expert, all_scales, DOWN ? p.H : 2 * p.I);
                block_bytes = (size_t)kq_count * (nib ? 1024 : 2048);
            }
            const int b0 = (item - job * per_job) * PER_ITEM, live = min(PER_ITEM, blocks - b0);
            for (int kq = 0; kq < kq_count; kq += STAGE_KQ, ++issued) {
                const uint32_t bytes = (uint32_t)min(STAGE_KQ, kq_count - kq) * (nib ? 1024u : 2048u);
                if (issued >= R) {
                    if (deadline == 0) { if (DOWN) pdl_wait(); deadline = global_ns() + p.timeout_ns; }   // slots come back once the activations exist
                    if (!__all_sync(0xffffffffu, mbar_wait(&empty[slot], phase ^ 1u, deadline))) {
                        if (lane == 0) *reinterpret_cast<volatile int*>(&p.status->device_error) = 1;
                        failed = true;
                        break;
                    }
                }
                uint8_t* const dst = ring + (size_t)slot * MOE_STAGE_BYTES;
                const uint8_t* const src = base + (size_t)b0 * block_bytes + (size_t)kq * (nib ? 1024 : 2048);
                const int reader = turn % groups, entry = turn % MOE_TURNS;
                uint64_t* const bar = &full[reader][slot];
                if (used[reader] >> slot & 1u) armed[reader] ^= 1u << slot;
                used[reader] |= 1u << slot;
                if (elect_one()) {
                    const uint32_t scale_bytes = kq == 0 ? (uint32_t)live * 64u : 0u;
                    mbar_arrive_expect_tx(bar, (bytes * (uint32_t)live + scale_bytes) * (DOWN ? 1u : 2u));
                    if (kq == 0) {       // (an entry is used again 16 turns later: its readers have freed a later stage since)
                        s_turn[entry] = make_int4(item, first, rows, nib);
                        mbar_arrive(&told[entry]);
                        bulk_g2s(s_w[entry], ws + b0 * 16, scale_bytes, bar);
                        if (!DOWN) bulk_g2s(s_w[entry] + PER_ITEM * 16, ws + p.I + b0 * 16, scale_bytes, bar);
                    }
                    for (int b = 0; b < live; ++b) bulk_g2s(dst + b * BLOCK_STAGE, src + (size_t)b * block_bytes, bytes, bar);
                    if (!DOWN)
                        for (int b = 0; b < live; ++b)
                            bulk_g2s(dst + (PER_ITEM + b) * BLOCK_STAGE, src + (size_t)(blocks + b) * block_bytes, bytes, bar);
                }
                __syncwarp();
                if (++slot == R) { slot = 0; phase ^= 1u; }
            }
            if (failed) break;
            ++item;
            ++turn;
        }
        if (!failed && elect_one())
            for (int i = 0; i < groups; ++i, ++turn) {                   // no more
                s_turn[turn % MOE_TURNS] = make_int4(-1, 0, 0, 0);
                mbar_arrive(&told[turn % MOE_TURNS]);
            }
        __syncwarp();
        // the CTA stays until its copies have landed, whoever still waits for them
        if (deadline == 0 || failed) deadline = global_ns() + p.timeout_ns;
        for (int g = 0; g < groups; ++g)
            for (int i = 0; i < R; ++i)
                if (used[g] >> i & 1u) mbar_wait(&full[g][i], armed[g] >> i & 1u, deadline);
        return;
    }

    // ------------------------------------------------------------------ contraction warps
    const int group = tid / MOE_GROUP, gtid = tid - group * MOE_GROUP, warp = gtid >> 5;
    uint8_t* const xs = ring + (size_t)R * MOE_STAGE_BYTES + (size_t)group * moe_group_bytes(K);
    int* const partials = reinterpret_cast<int*>(xs + (size_t)MOE_JOB_ROWS * row_bytes);      // two buffers
    float* const s_scale = s_scales[group];
    const int8_t* const codes = run->f32 ? p.codes : moe_piece<int8_t>(p.upload, p.input_at);
    const float* const in_scales = run->f32 ? p.in_scales : moe_piece<float>(p.upload, run->scales);
    const int* const assign_token = moe_piece<int>(p.upload, run->assign_token);
    const int g = lane >> 2, t = lane & 3;
    const int block = DOWN ? warp : warp & 3, k_half = DOWN ? 0 : warp >> 2;
    const uint8_t* const x0 = xs + (size_t)g * row_bytes + 4 * t;
    unsigned long long deadline = 0;
    bool waited = !DOWN;
    auto wait = [&](uint64_t* bar, uint32_t parity) {        // false: it ran out
        if (mbar_test(bar, parity)) return true;
        if (deadline == 0) deadline = global_ns() + p.timeout_ns;
        if (mbar_wait(bar, parity, deadline)) return true;
        *reinterpret_cast<volatile int*>(&p.status->device_error) = 1;
        return false;
    };
    // The group's eight warps meet; true: one of them could not wait any longer, and all of them leave (a warp that gives up
    // takes part in one more meeting, whichever the others come to next, so that none is left waiting for it).
    auto meet = [&](bool failed) {
        uint32_t any;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %3, 0;\n\tbarrier.cta.red.or.pred p, %1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(any) : "r"(1 + group), "n"(MOE_GROUP), "r"((uint32_t)failed) : "memory");
        return any != 0;
    };
    int job = -1;
    uint32_t phases = 0;                                     // of the group's full barriers, one bit per slot
    for (int turn = group;; turn += groups) {
        const bool knows = __all_sync(0xffffffffu, wait(&told[turn % MOE_TURNS], (uint32_t)(turn / MOE_TURNS) & 1u));
        const int4 told_item = s_turn[turn % MOE_TURNS];
        const int item = told_item.x, first = told_item.y, rows = told_item.z;
        const bool nib = told_item.w;
        if (!knows || item < 0) {
            meet(!knows);
            break;
        }
        if (item / per_job != job) {
            job = item / per_job;
            if (!waited) { pdl_wait(); waited = true; }      // middle rows and their maxima come from the gate/up launch
            if (meet(false)) break;                          // the rows of the job before are no longer read
            // rows beyond the job are not read (their columns of the sums are not used); k beyond K meets zero weights
            const int live_rows = rows > 8 ? 16 : 8;
            auto row_scale = [&](int r) {
                const uint32_t m = __ldcg(p.row_max + first + r);
                return m ? __fdiv_rn(__uint_as_float(m), 127.f) : 1.f;
            };
            if (gtid < MOE_JOB_ROWS) s_scale[gtid] = gtid >= rows ? 0.f : DOWN ? row_scale(gtid) : in_scales[assign_token[first + gtid]];
            if (DOWN) {
                const int quads = p.I / 4;                   // I is a multiple of 32
#pragma unroll 4
                for (int i = gtid; i < live_rows * quads; i += MOE_GROUP) {
                    const int r = i / quads, w = i - r * quads;
                    uint32_t packed = 0;
                    if (r < rows) {
                        const float4 v = __ldcg(reinterpret_cast<const float4*>(p.middle + (size_t)(first + r) * p.I + 4 * w));
                        const float inv = __frcp_rn(row_scale(r));
                        packed = (uint32_t)(uint8_t)nearest_even_code(__fmul_rn(v.x, inv)) | (uint32_t)(uint8_t)nearest_even_code(__fmul_rn(v.y, inv)) << 8 |
                                 (uint32_t)(uint8_t)nearest_even_code(__fmul_rn(v.z, inv)) << 16 | (uint32_t)(uint8_t)nearest_even_code(__fmul_rn(v.w, inv)) << 24;
                    }
                    *reinterpret_cast<uint32_t*>(xs + (size_t)r * row_bytes + 4 * w) = packed;
                }
            } else {
                const int vecs = p.H / 16;                   // H is a multiple of 32
#pragma unroll 4
                for (int i = gtid; i < live_rows * vecs; i += MOE_GROUP) {
                    const int r = i / vecs, v = i - r * vecs;
                    uint4 val = make_uint4(0u, 0u, 0u, 0u);
                    if (r < rows) val = *(reinterpret_cast<const uint4*>(codes + (size_t)assign_token[first + r] * p.H) + v);
                    *reinterpret_cast<uint4*>(xs + (size_t)r * row_bytes + 16 * v) = val;
                }
            }
            if (meet(false)) break;
        }
        const int b0 = (item - job * per_job) * PER_ITEM, live = min(PER_ITEM, blocks - b0);
        const bool mine = DOWN ? block < live : (block & 1) < live;      // this warp's block exists
        int c[2][4] = {};
        int slot = turn * stages % R;
        bool failed = false;
        for (int kq = 0; kq < kq_count; kq += STAGE_KQ) {
            const int n = min(STAGE_KQ, kq_count - kq), lead = DOWN ? n : (n + 1) / 2;
            if (!__all_sync(0xffffffffu, wait(&full[group][slot], phases >> slot & 1u))) failed = true;
            const int from = k_half ? lead : 0, count = k_half ? n - lead : lead;
            if (mine && count > 0) {
                const uint4* const w = reinterpret_cast<const uint4*>(ring + (size_t)slot * MOE_STAGE_BYTES + block * BLOCK_STAGE) + from * (nib ? 64 : 128);
                const uint8_t* const x = x0 + (kq + from) * MOE_KQ;
                if (nib) {
                    if (rows > 8) block_mma<true, true>(w, x, row_bytes, count, lane, c);
                    else block_mma<false, true>(w, x, row_bytes, count, lane, c);
                } else {
                    if (rows > 8) block_mma<true, false>(w, x, row_bytes, count, lane, c);
                    else block_mma<false, false>(w, x, row_bytes, count, lane, c);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[slot]);
            phases ^= 1u << slot;
            if (++slot == R) slot = 0;
        }
        if (rows <= 8) {
#pragma unroll
            for (int i = 0; i < 4; ++i) c[0][i] += c[1][i];
        }
        const int shift = nib ? 4 : 0;                       // int4 records: every code entered times 16
        const float* const scales = s_w[turn % MOE_TURNS];
        if (DOWN) {
            if (failed) { meet(true); break; }
            if (!mine) continue;
            const int column = (b0 + block) * 16 + g;
            const float w0 = scales[block * 16 + g], w1 = scales[block * 16 + g + 8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = (i >> 2) * 8 + 2 * t + (i & 1);
                if (r < rows) p.expert_out[(size_t)(first + r) * p.H + column + (i & 2 ? 8 : 0)] = dequant(c[i >> 2][i & 3] >> shift, s_scale[r], i & 2 ? w1 : w0);
            }
        } else {
            // the halves of K meet in shared memory; a warp finishes feature block fbi, features g + 8 h, tokens 8 half ..
            int* const partial = partials + (turn / groups & 1) * MOE_PARTIAL;
#pragma unroll
            for (int i = 0; i < 8; ++i) partial[(warp * 8 + i) * 32 + lane] = c[i >> 2][i & 3];
            if (meet(failed)) break;
            const int half = (warp >> 1) & 1, fbi = warp & 1, h = warp >> 2;
            if (fbi >= live || (half == 1 && rows <= 8)) continue;
            const int feature = (b0 + fbi) * 16 + g + 8 * h;
            const float w0 = scales[fbi * 16 + g + 8 * h], w1 = scales[(PER_ITEM + fbi) * 16 + g + 8 * h];
            auto sum = [&](int b, int i) { return (partial[(b * 8 + i) * 32 + lane] + partial[((b + 4) * 8 + i) * 32 + lane]) >> shift; };
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = half * 8 + 2 * t + e;
                uint32_t m = 0;
                if (r < rows) {
                    const int i = half * 4 + 2 * h + e;
                    const float sc = s_scale[r];
                    const float y = __fmul_rn(silu_poly(dequant(sum(fbi, i), sc, w0)), dequant(sum(2 + fbi, i), sc, w1));
                    p.middle[(size_t)(first + r) * p.I + feature] = y;
                    m = __float_as_uint(y) & 0x7fffffffu;
                }
                m = max(m, __shfl_xor_sync(0xffffffffu, m, 4));
                m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
                m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
                if (g == 0 && r < rows && m) atomicMax(&p.row_max[first + r], m);
            }
        }
    }
    if (!waited) pdl_wait();        // (the next kernel relies on this one to have waited)
}

// ------------------------------------------------------------------ weighted sum over a token's slots (src/rk_npu_moe_w8.cpp:786-816)
// Four columns per thread.  Where the result goes to host memory, the last block of every 16 rows to have stored its part
// raises these rows' flag, and the host carries them on while later rows still cross the bus.
constexpr int MOE_COMBINE_THREADS = 128;
__global__ void __launch_bounds__(MOE_COMBINE_THREADS) moe_combine_kernel(const MoeCombineParams p)
{
    const MoeRun* const run = moe_piece<MoeRun>(p.upload, 0);
    const int token = blockIdx.y, rows = run->rows;
    const int n = (blockIdx.x * MOE_COMBINE_THREADS + threadIdx.x) * 4;
    if (token >= rows) return;
    const int* const assign = moe_piece<int>(p.upload, run->slot_assign) + token * p.slots;
    const float* const coefficients = moe_piece<float>(p.upload, run->coefficients) + token * p.slots;
    constexpr int MOST = 9;                           // top-8 and the shared expert
    int at[MOST];
    float c[MOST];
#pragma unroll
    for (int slot = 0; slot < MOST; ++slot) {
        at[slot] = slot < p.slots ? assign[slot] : -1;
        c[slot] = slot < p.slots ? coefficients[slot] : 0.f;
    }
    float* const out = run->out;
    const uint32_t serial = run->serial;
    pdl_wait();
    // the row maxima have been consumed by the down projection: leave them zero for the next run
    if (blockIdx.x == 0 && threadIdx.x < p.slots) {
        const int a = assign[threadIdx.x];
        if (a >= 0) p.row_max[a] = 0u;
    }
    if (blockIdx.x == 0 && token == 0 && threadIdx.x < 2) p.tickets[threadIdx.x] = 0u;
    if (n < p.H) {
        float4 v[MOST];
#pragma unroll
        for (int slot = 0; slot < MOST; ++slot)
            v[slot] = at[slot] >= 0 ? *reinterpret_cast<const float4*>(p.expert_out + (size_t)at[slot] * p.H + n) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int slot = 0; slot < MOST; ++slot)
            if (at[slot] >= 0) {                          // slot order, one fused multiply-add each
                sum.x = __fmaf_rn(v[slot].x, c[slot], sum.x);
                sum.y = __fmaf_rn(v[slot].y, c[slot], sum.y);
                sum.z = __fmaf_rn(v[slot].z, c[slot], sum.z);
                sum.w = __fmaf_rn(v[slot].w, c[slot], sum.w);
            }
        *reinterpret_cast<float4*>(out + (size_t)token * p.H + n) = sum;
    }
    if (!serial) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        const int chunk = token / MOE_CHUNK_ROWS;
        const unsigned all = gridDim.x * (unsigned)min(MOE_CHUNK_ROWS, rows - chunk * MOE_CHUNK_ROWS);
        __threadfence_system();                       // the block's rows are in host memory: the one trip over the bus that is waited for
        if (atomicAdd(&p.arrived[chunk], 1u) + 1 == all) {
            p.arrived[chunk] = 0u;
            __threadfence();
            *reinterpret_cast<volatile uint32_t*>(&p.flags[chunk]) = serial;
        }
    }
}

// ------------------------------------------------------------------ launchers
cudaError_t launch_moe_pack(const MoePackParams& p, cudaStream_t stream)
{
    const size_t total = (p.nibbles ? moe_packed_nibble_bytes(p.K, p.N) : moe_packed_bytes(p.K, p.N)) / 16;
    const unsigned blocks = (unsigned)std::min<size_t>((total + 255) / 256, 148 * 8);
    moe_pack_kernel<<<blocks, 256, 0, stream>>>(p);
    return cudaGetLastError();
}

// one launch that may start while the kernel in front of it on the stream still runs (each kernel above waits
// with griddepcontrol.wait before it touches what that kernel writes)
template <class Params>
static cudaError_t launch_dependent(void (*kernel)(const Params), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, const Params& p)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

cudaError_t launch_moe_intake(const MoeIntakeParams& p, int max_rows, cudaStream_t stream)
{
    moe_intake_kernel<<<unsigned(max_rows + (p.from ? MOE_INTAKE_MOVERS : 0)), MOE_INTAKE_THREADS, 0, stream>>>(p);
    return cudaGetLastError();
}

template <bool DOWN>
static cudaError_t launch_project(const MoeProjectParams& p, int sm_count, cudaStream_t stream)
{
    static PerDeviceOnce once;
    int device = -1;
    if (once.needed(device)) {
        const cudaError_t e = cudaFuncSetAttribute(moe_project_kernel<DOWN>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(MOE_SMEM_MOST));
        if (e != cudaSuccess) return e;
        once.mark(device);
    }
    const int K = DOWN ? p.I : p.H, groups = moe_groups(K);
    return launch_dependent(moe_project_kernel<DOWN>, dim3(unsigned(sm_count)), unsigned(groups * MOE_GROUP + 32),
                            groups * moe_group_bytes(K) + size_t(moe_ring(K)) * MOE_STAGE_BYTES, stream, p);
}
cudaError_t launch_moe_gate_up(const MoeProjectParams& p, int sm_count, cudaStream_t stream) { return launch_project<false>(p, sm_count, stream); }
cudaError_t launch_moe_down(const MoeProjectParams& p, int sm_count, cudaStream_t stream) { return launch_project<true>(p, sm_count, stream); }

cudaError_t launch_moe_combine(const MoeCombineParams& p, int max_rows, cudaStream_t stream)
{
    return launch_dependent(moe_combine_kernel, dim3(unsigned((p.H / 4 + MOE_COMBINE_THREADS - 1) / MOE_COMBINE_THREADS), unsigned(max_rows)), MOE_COMBINE_THREADS, 0, stream, p);
}

} // namespace rkb200

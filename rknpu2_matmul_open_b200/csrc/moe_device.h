// moe_device.h -- device side of the routed-experts operator (rk_npu_moe_w8.h): parameter blocks and launchers.
//
// A run is a list of JOBS: up to 16 (token, slot) assignments that use the same expert.  After the intake of the rows
// three launches work on the list: gate/up projection + SwiGLU (fp32 middle rows and their maxima), down projection (re-quantises
// the middle rows on the way into shared memory), and the weighted sum over each token's slots.
#pragma once
#include "w4a8_device.h"
#include <cuda_runtime.h>
#include <stdint.h>

namespace rkb200 {

constexpr int MOE_JOB_ROWS = 16;     // assignments per job: two 8-token halves of mma.m16n8k32
constexpr int MOE_KQ = 128;          // k extent of one packed weight record (four k-steps of 32)

// Packed int8 expert matrix W[K][N] (N a multiple of 16): records of 16 channels x 128 k in the register order
// of the m16n8k32 A operand, [channel block][k quarter-kilo][k-step 0..3][lane][16 B = a0 a1 a2 a3], zero beyond K.
inline size_t moe_packed_bytes(int K, int N) { return size_t((K + MOE_KQ - 1) / MOE_KQ) * MOE_KQ * size_t(N); }
// Int4 experts keep two codes per byte: [channel block][k quarter-kilo][half 0..1][lane][16 B], the 16 bytes being the
// words of k-steps 2 half and 2 half + 1 for channels g and g + 8; a word w holds the codes at k = 4t.. in its low
// nibbles and those at k = 16 + 4t.. in its high nibbles, so that (w << 4) & 0xF0F0F0F0 and w & 0xF0F0F0F0 are the two
// A registers of the channel with every code times 16 (the sums are shifted back, exactly).  Half the bytes.
inline size_t moe_packed_nibble_bytes(int K, int N) { return moe_packed_bytes(K, N) / 2; }
// A bank of experts: the first `nibble_experts` hold int4 records, the rest int8 records.  An immutable bank is one
// allocation (`base`, experts at fixed strides) with its scales in one array; a slot bank keeps every expert in an
// allocation of its own, which can change hands between banks, and gives the kernels two tables of pointers instead
// (`table`: each expert's records; `scale_table`: each expert's scales).
struct MoeBank {
    const uint8_t* base;
    size_t nibble_bytes, byte_bytes;   // one expert's records in either form
    int nibble_experts;
    const uint8_t* const* table;       // slot banks only, else null
    const float* const* scale_table;   // slot banks only, else null
    __host__ __device__ const uint8_t* expert(int e) const
    {
        if (table) return table[e];
        return e < nibble_experts ? base + size_t(e) * nibble_bytes
                                  : base + size_t(nibble_experts) * nibble_bytes + size_t(e - nibble_experts) * byte_bytes;
    }
    // the scales of expert e: `all` holds `stride` per expert where there is no table
    __host__ __device__ const float* scales(int e, const float* all, int stride) const
    {
        return scale_table ? scale_table[e] : all + size_t(e) * stride;
    }
    __host__ __device__ bool nibbles(int e) const { return e < nibble_experts; }
};

struct MoePackParams {
    const int8_t* W;      // [K][N] row-major, on the device
    uint8_t* packed;
    int K, N;
    int nibbles;          // 1: int4 codes, two per byte
};

// One projection's weights: the experts' records and their scales.
struct MoeMatrix {
    MoeBank bank;
    const float* scales;       // [E][channels] (immutable banks)
};
// What one run hands to the device, in one piece, begins with this: what there is and where it lies (bytes from the start
// of the piece).  The kernels of a run read everything that changes from call to call from here, so that their parameters,
// and with them a kept graph of the launches, depend on the workspace alone.
struct MoeRun {
    int rows, jobs, assignments;
    int f32;                   // the rows are fp32 and the intake kernel quantises them; else int8 codes
    uint32_t job_expert;       // [jobs]
    uint32_t job_first;        // [jobs] first assignment of the job (a job's assignments are consecutive)
    uint32_t job_rows;         // [jobs] 1..16
    uint32_t assign_token;     // [assignments] source row of each assignment
    uint32_t slot_assign;      // [rows][slots] assignment index, -1: the slot takes no part
    uint32_t coefficients;     // [rows][slots]
    uint32_t scales;           // [rows] (int8 rows)
    uint32_t used;             // bytes of header, schedule and tables: a multiple of 16
    MoeMatrix gate_up, down;
    float* out;                // [rows][H], on the device or the device alias of page-locked host memory
    uint32_t serial;           // not 0: the combine kernel stores this number into a chunk's flag when its rows are complete
    uint32_t pad;
};
constexpr int MOE_CHUNK_ROWS = 16;                                   // output rows per flag
template <class T> __host__ __device__ inline const T* moe_piece(const uint8_t* upload, uint32_t offset) { return reinterpret_cast<const T*>(upload + offset); }

struct MoeIntakeParams {
    const uint8_t* from;  // device alias of the piece in page-locked host memory, or NULL: it has been copied to `upload` already
    uint8_t* upload;
    int8_t* codes;        // [rows][H]
    float* scales;        // [rows]
    Status* status;       // bad_input: a non-finite element, or a scale whose reciprocal is not finite
    uint32_t input_at;    // where the input rows [rows][H] begin: behind all that header, schedule and tables can take
    int H, f32;
};

// One projection of every job: gate/up with SwiGLU, or down.
struct MoeProjectParams {
    const uint8_t* upload;
    const int8_t* codes;         // gate/up: [rows][H] and
    const float* in_scales;      // [rows], where the run's rows are fp32
    float* middle;               // [assignments][I]
    uint32_t* row_max;           // [assignments] bit patterns of max |middle|, zero before the first launch
    float* expert_out;           // down: [assignments][H]
    unsigned* tickets;           // [2] items handed out by gate/up and by down; zero before the first launch
    Status* status;              // device_error: a bounded wait ran out
    uint32_t input_at;
    int H, I;
    unsigned long long timeout_ns;
};

struct MoeCombineParams {
    const uint8_t* upload;
    const float* expert_out;     // [assignments][H]
    uint32_t* row_max;           // [assignments] cleared here for the next run
    unsigned* tickets;           // [2] cleared here as well
    unsigned* arrived;           // [chunks] blocks that have stored their part; zero between runs
    uint32_t* flags;             // [chunks] in page-locked host memory
    int slots, H;
};

cudaError_t launch_moe_pack(const MoePackParams& p, cudaStream_t stream);
// max_rows: the rows a grid has to be able to cover (the run's own count is read on the device)
cudaError_t launch_moe_intake(const MoeIntakeParams& p, int max_rows, cudaStream_t stream);
cudaError_t launch_moe_gate_up(const MoeProjectParams& p, int sm_count, cudaStream_t stream);
cudaError_t launch_moe_down(const MoeProjectParams& p, int sm_count, cudaStream_t stream);
cudaError_t launch_moe_combine(const MoeCombineParams& p, int max_rows, cudaStream_t stream);

} // namespace rkb200

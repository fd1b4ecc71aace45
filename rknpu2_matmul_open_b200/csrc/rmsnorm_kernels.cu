// rmsnorm_kernels.cu -- residual add + RMSNorm on fp16 tensors (rk_npu_add_rmsnorm_f16.h), one launch.
//
//   sum  = fp16(float(x) + float(residual))                                   -> residual_out
//   norm = fp16(float(double(sum) * inv * double(gamma))),  inv = 1 / sqrt(sum of double(sum)^2 / D + eps)   -> norm_out
//
// the double-precision statement of the original's board test (tests/test_add_rmsnorm_f16.cpp:96-113), which is what
// the original device's result is checked against.  Double-precision conversions run at a quarter of the fp32 rate and
// would be the busiest pipe of this kernel, so the second pass proves per value that single precision
// gives the same fp16 bits and falls back to the defining expression where it cannot (scale_pair).
//
// HBM-bound: 4 tensors of 2 M D bytes cross DRAM once each.  Two forms.  Rows that fit a CTA's registers take
// add_rmsnorm_row_kernel; longer block-8 rows, and block-8 tensors across the bus, take add_rmsnorm_kernel, where a tile of TM
// tokens is shared by a CLUSTER of CS CTAs, each taking a slice of D: the sums stay in that CTA's shared memory between the two
// passes (both outputs are stored in the second one, so that no global store is in flight at the cluster barrier), the
// per-token sums of squares are exchanged through distributed shared memory and added in rank order by every CTA, so that the
// result does not depend on the schedule.  Both tensor layouts move 16-byte chunks
// (8 elements): in the block-8 layout (D/8, M, 8) consecutive TOKENS of one chunk column are contiguous, in row-major
// [M, D] consecutive CHUNKS of one token are; the thread index is split accordingly so that a warp touches 512
// contiguous bytes either way.
#include "rmsnorm_device.h"
#include "w4a8_math.cuh"
#include "w4a8_ptx.cuh"
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <atomic>
#include <cstdio>
#include <cstdlib>

namespace cg = cooperative_groups;

namespace rkb200 {
namespace {

constexpr int RN_THREADS = 512;
constexpr int RN_BATCH = 4;     // chunks of each input a thread requests before it uses the first
constexpr int RN_CTAS = 2;      // CTAs per SM the register allocation is bounded for
constexpr int RN_MAX_DEVICES = 64;
constexpr int RN_SMEM_SUMS = 64 * 1024;   // most bytes of sums one CTA keeps: TM * ceil(D/8/CS) * 16

// (x and the residual of a kernel that starts behind the one in front, and is not launched before that has finished)
__device__ __forceinline__ uint4 ld_stream(const uint4* p)
{
    uint4 v;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// The same for a kernel that may start before the one in front has finished writing what it reads: a coherent load that the
// compiler leaves behind the dependency wait.
__device__ __forceinline__ uint4 ld_dependent(const uint4* p)
{
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_stream(uint4* p, const uint4& v)
{
    asm volatile("st.global.cs.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// fp16(float(a) + float(b)) for a packed pair.  With 24 >= 2 * 11 + 2 mantissa bits the float sum rounded to fp16 equals
// the correctly rounded fp16 sum (double rounding is innocuous), which is what the packed fp16 add returns.  The squares
// of the two sums are added to acc in element order.
__device__ __forceinline__ uint32_t add_pair(uint32_t a, uint32_t b, double& acc)
{
    const __half2 s = __hadd2_rn(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    const float2 fs = __half22float2(s);
    const double lo = double(fs.x), hi = double(fs.y);
    acc += lo * lo;       // a product of two fp16 values is exact in double
    acc += hi * hi;
    return *reinterpret_cast<const uint32_t*>(&s);
}
// One output: fp16(float(double(v) * inv * double(g))), the defining expression, evaluated in double only when needed.
// y = fl32(fl32(v * inv_f) * g) with inv_f = fl32(inv) differs from the exact product x by at most 3 * 2^-24 |x|, and
// the float the defining expression rounds to fp16 by at most (2^-24 + 2^-52) |x|: that float lies between
// y (1 - 2^-21) and y (1 + 2^-21) (for the magnitudes |v| < 2^16, 2^-16 < inv, |g| < 2^16 nothing leaves the normal float
// range).  Rounding is monotone, so when both ends -- taken at 2^-20, which covers their own rounding -- round to the same
// fp16, that IS the defined result.  About 0.4 % of the values, and rows whose inv is not a normal float, are evaluated
// in double.

// The defining expression, for a pair.  A real call, so that this rare path is branched around instead of being
// evaluated for every value.
__device__ __noinline__ uint32_t scale_defined(float2 v, float2 g, double inv)
{
    const __half2 o = __floats2half2_rn(__double2float_rn(double(v.x) * inv * double(g.x)), __double2float_rn(double(v.y) * inv * double(g.y)));
    return *reinterpret_cast<const uint32_t*>(&o);
}
__device__ __forceinline__ uint32_t scale_pair(uint32_t v, uint32_t g, double inv, float inv_f, bool fast)
{
    const float2 fv = __half22float2(*reinterpret_cast<const __half2*>(&v));
    const float2 fg = __half22float2(*reinterpret_cast<const __half2*>(&g));
    const F2 y = f2_mul(f2_mul(f2_pack(fv.x, fv.y), f2_all(inv_f)), f2_pack(fg.x, fg.y));
    float a0, a1, b0, b1;
    f2_unpack(f2_mul(y, f2_all(1.f - 9.5367431640625e-07f)), a0, a1);
    f2_unpack(f2_mul(y, f2_all(1.f + 9.5367431640625e-07f)), b0, b1);
    const __half2 lower = __floats2half2_rn(a0, a1), upper = __floats2half2_rn(b0, b1);
    uint32_t o = *reinterpret_cast<const uint32_t*>(&lower);
    if (!fast || o != *reinterpret_cast<const uint32_t*>(&upper)) o = scale_defined(fv, fg, inv);
    return o;
}

// Block-8 (D/8, M, 8).  grid = tiles * CS CTAs in clusters of CS.
__global__ void __launch_bounds__(RN_THREADS, RN_CTAS) add_rmsnorm_kernel(AddRmsNormParams p)
{
    extern __shared__ __align__(16) uint8_t smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int CS = int(cluster.num_blocks()), rank = int(cluster.block_rank());
    const int TM = p.tile_tokens, JL = RN_THREADS / TM;       // tokens of the tile x chunk lanes
    const int tid = threadIdx.x;
    const int dm = tid % TM, jl = tid / TM;
    const int m = int(blockIdx.x / CS) * TM + dm;
    const int chunks = p.D / 8, per = (chunks + CS - 1) / CS;
    const int j0 = min(chunks, rank * per), j1 = min(chunks, j0 + per);
    const bool live = m < p.M;

    uint4* s_sum = reinterpret_cast<uint4*>(smem);                               // this CTA's slice of the tile's sums
    double* s_part = reinterpret_cast<double*>(smem + size_t(TM) * per * 16);    // [RN_THREADS]
    double* s_token = s_part + RN_THREADS;                                       // [TM] this CTA's sum of squares per token
    auto lane_of = [&](int token, int lane) { return lane * TM + token; };
    auto global_at = [&](int j) { return size_t(j) * p.M + m; };
    auto shared_at = [&](int j) { return (j - j0) * TM + dm; };

    double acc = 0.0;
    if (live) {
        for (int j = j0 + jl; j < j1; j += RN_BATCH * JL) {      // RN_BATCH chunks of both inputs in flight per thread
            uint4 a[RN_BATCH], b[RN_BATCH];
#pragma unroll
            for (int u = 0; u < RN_BATCH; ++u)
                if (j + u * JL < j1) {
                    const size_t at = global_at(j + u * JL);
                    a[u] = ld_stream(p.x + at);
                    b[u] = ld_stream(p.residual + at);
                }
#pragma unroll
            for (int u = 0; u < RN_BATCH; ++u)
                if (j + u * JL < j1) {
                    uint4 s;
                    s.x = add_pair(a[u].x, b[u].x, acc);
                    s.y = add_pair(a[u].y, b[u].y, acc);
                    s.z = add_pair(a[u].z, b[u].z, acc);
                    s.w = add_pair(a[u].w, b[u].w, acc);
                    s_sum[shared_at(j + u * JL)] = s;
                }
        }
    }
    s_part[tid] = acc;
    __syncthreads();
    if (JL <= 16) {                                            // few lanes per token: one thread adds them in lane order
        if (jl == 0) {
            double sum = acc;
            for (int lane = 1; lane < JL; ++lane) sum += s_part[lane_of(dm, lane)];
            s_token[dm] = sum;
        }
    } else {
        for (int step = JL / 2; step > 0; step >>= 1) {        // fixed tree over the chunk lanes of each token
            if (jl < step) s_part[tid] += s_part[lane_of(dm, jl + step)];
            __syncthreads();
        }
        if (jl == 0) s_token[dm] = s_part[tid];
    }
    if (CS > 1) cluster.sync(); else __syncthreads();
    double total = 0.0;
    for (int r = 0; r < CS; ++r) total += CS > 1 ? cluster.map_shared_rank(s_token, r)[dm] : s_token[dm];
    const double inv = 1.0 / sqrt(total / double(p.D) + double(p.eps));
    const float inv_f = __double2float_rn(inv);
    const bool fast = inv_f >= 1.17549435e-38f && inv_f <= 3.402823466e38f;       // a normal float (false for NaN)

    if (live) {
#pragma unroll 4
        for (int j = j0 + jl; j < j1; j += JL) {
            const uint4 s = s_sum[shared_at(j)];
            const uint4 g = __ldg(p.gamma + j);
            st_stream(p.residual_out + global_at(j), s);
            uint4 o;
            o.x = scale_pair(s.x, g.x, inv, inv_f, fast);
            o.y = scale_pair(s.y, g.y, inv, inv_f, fast);
            o.z = scale_pair(s.z, g.z, inv, inv_f, fast);
            o.w = scale_pair(s.w, g.w, inv, inv_f, fast);
            st_stream(p.norm_out + global_at(j), o);
        }
    }
    // A CTA's s_token must stay readable until every peer has read it.  Nothing this CTA wrote has to become visible
    // for that, so the arrival is relaxed: a releasing one would wait for the output stores still in flight.
    if (CS > 1) {
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    }
}


// The form for rows that fit a CTA's registers.  A row's JL threads keep its sums in registers (CPL chunks each) between
// the passes: no shared-memory round trip of the sums, no cluster, one barrier.  What bounds the operator is how many
// loads an SM has in flight and how long a CTA lives behind them, so the CTAs are small (their phases interleave) and
// every thread requests all of its chunks before it uses the first.  4096 x 4096 row-major: 36.9 -> 25.6 us
// (134 MB; the copy rate of this GPU gives 20.5), 8192 x 8192 118 -> 89 us (82), 16 x 4096 3.9 -> 2.6 us.
template <bool ROWS, int CPL>
__global__ void __launch_bounds__(RN_THREADS) add_rmsnorm_row_kernel(AddRmsNormParams p)
{
    pdl_launch_dependents();
    pdl_wait();                                               // x or the residual may come from the kernel in front
    __shared__ double s_part[RN_THREADS / 32 * 8];
    const int TM = p.tile_tokens, JL = int(blockDim.x) / TM;  // tokens of the CTA x threads per token
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dm = ROWS ? tid / JL : tid % TM, jl = ROWS ? tid % JL : tid / TM;
    const int m = int(blockIdx.x) * TM + dm;
    const int chunks = p.D / 8;
    const bool live = m < p.M;
    auto global_at = [&](int j) { return ROWS ? size_t(m) * chunks + j : size_t(j) * p.M + m; };
    uint4 sum[CPL];
    double acc = 0.0;
    {
        uint4 b[CPL];
#pragma unroll
        for (int u = 0; u < CPL; ++u) {
            sum[u] = b[u] = make_uint4(0u, 0u, 0u, 0u);
            const int j = jl + u * JL;
            if (live && j < chunks) {
                const size_t at = global_at(j);
                sum[u] = ld_dependent(p.x + at);
                b[u] = ld_dependent(p.residual + at);
            }
        }
#pragma unroll
        for (int u = 0; u < CPL; ++u) {
            sum[u].x = add_pair(sum[u].x, b[u].x, acc);
            sum[u].y = add_pair(sum[u].y, b[u].y, acc);
            sum[u].z = add_pair(sum[u].z, b[u].z, acc);
            sum[u].w = add_pair(sum[u].w, b[u].w, acc);
        }
    }
    // a fixed tree over the lanes of a token inside each warp, then the warps in order
    for (int step = ROWS ? 1 : TM; step < 32; step <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, step);
    if (ROWS ? lane == 0 : lane < TM) s_part[ROWS ? warp : warp * TM + lane] = acc;
    __syncthreads();
    double total = 0.0;
    if (ROWS) {
        const int per = JL / 32;
        for (int w = 0; w < per; ++w) total += s_part[dm * per + w];
    } else {
        for (int w = 0; w < int(blockDim.x) / 32; ++w) total += s_part[w * TM + dm];
    }
    const double inv = 1.0 / sqrt(total / double(p.D) + double(p.eps));
    const float inv_f = __double2float_rn(inv);
    const bool fast = inv_f >= 1.17549435e-38f && inv_f <= 3.402823466e38f;       // a normal float (false for NaN)
    if (!live) return;
#pragma unroll
    for (int u = 0; u < CPL; ++u) {
        const int j = jl + u * JL;
        if (j < chunks) {
            const uint4 s = sum[u], g = __ldg(p.gamma + j);
            st_stream(p.residual_out + global_at(j), s);
            uint4 o;
            o.x = scale_pair(s.x, g.x, inv, inv_f, fast);
            o.y = scale_pair(s.y, g.y, inv, inv_f, fast);
            o.z = scale_pair(s.z, g.z, inv, inv_f, fast);
            o.w = scale_pair(s.w, g.w, inv, inv_f, fast);
            st_stream(p.norm_out + global_at(j), o);
        }
    }
}

} // namespace

// Tile and cluster.  Candidates: tokens per tile a power of two up to 32 and up to the batch (at least 8 where the
// batch has them, so that a tile's chunks of one column are 128 contiguous bytes); clusters of
// 1, 2, 4 or 8 CTAs over D; the CTA's slice of the sums within RN_SMEM_SUMS; every thread of a cluster member with at
// least one chunk.  Taken: the candidate with the most CTAs up to 128 (small batches are spread over the GPU), then
// the smallest cluster, then the most tokens per tile.  Measured on 4096 rows: time falls with the work per CTA (a
// CTA's fixed cost -- start, load latency, two barriers, store drain -- is about 4 us) and rises with the cluster size.
static void add_rmsnorm_geometry(int M, int D, int& tile_tokens, int& cluster)
{
    int top = 1;
    while (top < 32 && top < M) top <<= 1;
    const int floor_tokens = top < 8 ? top : 8;
    const int chunks = D / 8;
    if (const char* text = std::getenv("RK_NPU_B200_RMSNORM_TILE")) {      // experiments: "tokens,cluster"
        int tm = 0, cs = 0;
        if (std::sscanf(text, "%d,%d", &tm, &cs) == 2 && tm >= 1 && tm <= 32 && (tm & (tm - 1)) == 0 && (cs == 1 || cs == 2 || cs == 4 || cs == 8) &&
            size_t(tm) * ((chunks + cs - 1) / cs) * 16 <= size_t(RN_SMEM_SUMS)) {
            tile_tokens = tm;
            cluster = cs;
            return;
        }
    }
    int best_score = -1;
    tile_tokens = 1;
    cluster = 8;        // D <= 32768: 512 chunks per CTA, one per thread
    for (int pass = 0; pass < 2 && best_score < 0; ++pass)      // second pass: without the floor, if nothing fitted
        for (int cs = 1; cs <= 8; cs <<= 1)
            for (int tm = top; tm >= (pass ? 1 : floor_tokens); tm >>= 1) {
                const int per = (chunks + cs - 1) / cs;
                if (size_t(tm) * per * 16 > size_t(RN_SMEM_SUMS)) continue;
                if (cs > 1 && tm * per < RN_THREADS) continue;
                const int ctas = (M + tm - 1) / tm * cs;
                const int score = ctas < 128 ? ctas : 128;
                if (score > best_score) {
                    best_score = score;
                    tile_tokens = tm;
                    cluster = cs;
                }
            }
}

// Threads of a CTA, its tokens and the chunks per thread of the register form; false where the cluster form is taken:
// block-8 rows too long for the registers of a CTA that covers four tokens (whose chunks of one column are the two
// sectors a warp should touch at least), and tensors across the bus, which wants 128 contiguous bytes and more (128 x
// 4096: 93 us against 180).  Measured on shapes from 1 x 1024 to 8192 x 8192: large tensors want many loads
// per thread in small CTAs (4096 x 4096 row-major, 128 threads: four chunks 25.6 us, two 27.9, eight 30; block-8, four
// tokens and eight chunks 33.3, two tokens 34.1), small ones want the whole GPU and short chains (16 x 4096: one chunk 2.6,
// two 2.8 us; block-8 128 x 4096: two tokens 4.0, four 4.9 us, 16 x 4096: one token 3.2 us, two 3.7).
static bool row_geometry(const AddRmsNormParams& p, int& threads, int& tokens, int& cpl)
{
    const int M = p.M, D = p.D, row_major = p.row_major;
    if (p.over_bus && M > 1) return false;
    const int chunks = D / 8;
    const long long work = (long long)M * chunks;
    auto power = [](int least, int x) { while (least < x) least <<= 1; return least; };
    if (row_major) {
        cpl = work >= (1 << 20) ? 4 : work >= (1 << 15) ? 2 : 1;
        while (power(32, (chunks + cpl - 1) / cpl) > RN_THREADS) cpl <<= 1;          // (D <= 32768: eight at most)
        const int lanes = power(32, (chunks + cpl - 1) / cpl);
        threads = lanes < 128 ? 128 : lanes;
        tokens = threads / lanes;
        return true;
    }
    tokens = work >= (1 << 18) ? 4 : work >= (1 << 15) ? 2 : 1;
    while (tokens > 1 && tokens / 2 >= M) tokens >>= 1;
    cpl = tokens == 4 ? 8 : 1;
    while (cpl < 8 && RN_THREADS / tokens * cpl < chunks) cpl <<= 1;
    if (RN_THREADS / tokens * cpl < chunks && work >= (1 << 15)) return false;
    while (RN_THREADS / tokens * cpl < chunks) tokens >>= 1;                          // (a few long rows: D <= 32768 fits one token)
    threads = power(64, tokens * ((chunks + cpl - 1) / cpl));
    return true;
}

template <bool ROWS>
static cudaError_t launch_rows(const AddRmsNormParams& p, int threads, int cpl, cudaStream_t stream)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned((p.M + p.tile_tokens - 1) / p.tile_tokens));
    cfg.blockDim = dim3(unsigned(threads));
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    switch (cpl) {
    case 1: return cudaLaunchKernelEx(&cfg, add_rmsnorm_row_kernel<ROWS, 1>, p);
    case 2: return cudaLaunchKernelEx(&cfg, add_rmsnorm_row_kernel<ROWS, 2>, p);
    case 4: return cudaLaunchKernelEx(&cfg, add_rmsnorm_row_kernel<ROWS, 4>, p);
    default: return cudaLaunchKernelEx(&cfg, add_rmsnorm_row_kernel<ROWS, 8>, p);
    }
}

cudaError_t launch_add_rmsnorm(const AddRmsNormParams& q, cudaStream_t stream)
{
    AddRmsNormParams p = q;
    int threads = 0, cpl = 0;
    if (row_geometry(p, threads, p.tile_tokens, cpl))
        return p.row_major ? launch_rows<true>(p, threads, cpl, stream) : launch_rows<false>(p, threads, cpl, stream);
    int cs = 1;
    add_rmsnorm_geometry(p.M, p.D, p.tile_tokens, cs);
    const int per = (p.D / 8 + cs - 1) / cs;
    const size_t shared = size_t(p.tile_tokens) * per * 16 + size_t(RN_THREADS + p.tile_tokens) * sizeof(double);
    // function attributes are per device: remember what this device's copy of the kernel already allows
    static std::atomic<int> allowed[RN_MAX_DEVICES];
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) return err;
    std::atomic<int>* known = device >= 0 && device < RN_MAX_DEVICES ? &allowed[device] : nullptr;
    if (!known || known->load(std::memory_order_relaxed) < int(shared)) {
        err = cudaFuncSetAttribute(add_rmsnorm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(RN_SMEM_SUMS + (RN_THREADS + 32) * sizeof(double)));
        if (err != cudaSuccess) return err;
        err = cudaFuncSetAttribute(add_rmsnorm_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, int(cudaSharedmemCarveoutMaxShared));
        if (err != cudaSuccess) return err;
        if (known) known->store(int(RN_SMEM_SUMS + (RN_THREADS + 32) * sizeof(double)), std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg{};
    const int tiles = (p.M + p.tile_tokens - 1) / p.tile_tokens;
    cfg.gridDim = dim3(unsigned(tiles) * unsigned(cs));
    cfg.blockDim = dim3(RN_THREADS);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(cs);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, add_rmsnorm_kernel, p);
}

} // namespace rkb200

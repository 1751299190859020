// Internal definitions shared by the translation units of libferrograd_b200.
#pragma once
#include <nvtx3/nvToolsExt.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <utility>

#include "../../include/ferrograd_b200.h"
#include "conv_plan.cuh"

// Device error word bits, set by kernels whose bounded waits ran out.
#define FG_DEVERR_TMA_WAIT 1
#define FG_DEVERR_MMA_WAIT 2
#define FG_DEVERR_EPI_WAIT 4

struct fg_buf {
    void* ptr;
    uint64_t bytes;
    uint64_t version;   // bumped by every entry point that writes the buffer through its handle (fg_upload, fg_copy, ...)
    bool view;          // a window into a larger allocation owned by someone else: fg_free releases the handle only
};

struct fg_plan {
    cudaGraph_t graph;
    cudaGraphExec_t exec;
    uint64_t launches;  // kernels recorded in the graph
    uint64_t ws_generation;   // the scratch arena whose addresses the recorded kernels carry
    fg_ctx* ctx;
    bool has_comm;            // the recording contains an exchange: it holds the communicator until it is destroyed
};

// One timed launch: events on the launching stream around a single kernel.
struct fg_time_rec {
    cudaEvent_t a, b;
    int kind;
    double work;   // flop for GEMMs, bytes for bandwidth-bound kernels
};
#define FG_TIME_MAX_RECS 65536

struct fg_ctx {
    int device;
    cudaStream_t stream;
    bool own_stream;
    cudaStream_t comm_stream;
    cudaEvent_t ev_fork, ev_join;
    bool comm_pending;
    cudaEvent_t ev_ckpt[8];             // exchange checkpoints (fg_comm_checkpoint / fg_comm_wait)
    int comm_reserved_sms;              // SMs the persistent GEMMs leave free while an exchange is in flight
    cudaStream_t copy_stream;           // host->device prefetches that overlap compute
    cudaEvent_t ev_copy_done, ev_main_mark;
    bool mark_valid;
    char err[512];
    uint64_t launches;          // kernels launched so far (eager + replayed plans)
    bool capturing;
    uint64_t capture_launches;  // kernels recorded since fg_plan_begin
    // Scratch arena: operand planes of the tensor-core GEMM, reduction partials.
    char* ws;
    uint64_t ws_bytes;
    uint64_t ws_used;           // bump pointer, reset at the start of every entry point
    int* dev_status;            // device error word (see FG_DEVERR_*)
    void* tmap_encode;          // cuTensorMapEncodeTiled, resolved at context creation
    int sm_count;
    // Optional per-kernel timing (eager mode only)
    bool timing_on;
    fg_time_rec* time_recs;
    int time_count;       // records in use
    int time_created;     // records whose events exist
    // NCCL (loaded at run time)
    void* nccl_lib;
    void* comm;
    int nranks, rank;
    // Options (fg_ctx_set_option); the FG_* environment variables give their initial values once, at creation.
    int opt_tile_group;         // pair kernel: tile rows per group of the tile order (0: the default, eight)
    int opt_tile_pair;          // -1: chosen per shape; 1: CTA pairs whenever the shape allows; 0: opt_tile_bn x opt_tile_bk
    int opt_tile_bn, opt_tile_bk;
    int opt_conv_bn, opt_conv_split;      // conversion kernel: its tile width and K-shares wherever it can run (0: by estimate)
    bool opt_split_k;           // split-K tail of the pair kernel
    bool opt_pairs;             // multiply f32 tensors as they lie (bf16 pairs) where the shape allows
    int opt_exec_plans;         // the graph engine records each dispatch as a CUDA graph: 1 always, 0 never, -1 when launch-bound
    int opt_comm_max_ctas;      // CTAs the communicator may use (fg_comm_init)
    uint64_t opt_min_exchange;  // elements: the graph engine starts an exchange once this much is complete
    uint64_t ws_generation;     // bumped whenever the scratch arena is reallocated
    bool capture_has_comm;      // an exchange was recorded since fg_plan_begin
    int comm_plans;             // live plans that contain an exchange
};

inline int32_t fg_fail(fg_ctx* ctx, int32_t code, const char* msg) {
    if (ctx) {
        strncpy(ctx->err, msg, sizeof(ctx->err) - 1);
        ctx->err[sizeof(ctx->err) - 1] = 0;
    }
    return code;
}

inline int32_t fg_fail_cuda(fg_ctx* ctx, int32_t code, const char* what, cudaError_t e) {
    if (ctx) snprintf(ctx->err, sizeof(ctx->err), "%s: %s", what, cudaGetErrorString(e));
    return code;
}

#define FG_REQUIRE(ctx, cond, msg) \
    do { if (!(cond)) return fg_fail((ctx), FG_ERR_INVALID_ARGUMENT, msg); } while (0)

#define FG_CUDA(ctx, code, call) \
    do { cudaError_t _e = (call); if (_e != cudaSuccess) return fg_fail_cuda((ctx), (code), #call, _e); } while (0)

// Every compute entry point starts with this: valid context, right device, fresh scratch.
#define FG_ENTER(ctx) \
    do { if (!(ctx)) return FG_ERR_NOT_INITIALIZED; \
         FG_CUDA(ctx, FG_ERR_INVALID_DEVICE, cudaSetDevice((ctx)->device)); \
         (ctx)->ws_used = 0; } while (0)

// A named range on the calling host thread for timeline tools (NVTX, header-only: without a tool attached a
// range costs one pointer test).  The four dispatches of a training step, plan replays and gradient exchanges
// carry one each.
struct FgRange {
    explicit FgRange(const char* name) { nvtxRangePushA(name); }
    ~FgRange() { nvtxRangePop(); }
    FgRange(const FgRange&) = delete;
    FgRange& operator=(const FgRange&) = delete;
};

// After a kernel launch: count it and surface launch-configuration errors.
#define FG_LAUNCHED(ctx) \
    do { cudaError_t _e = cudaGetLastError(); \
         if (_e != cudaSuccess) return fg_fail_cuda((ctx), FG_ERR_LAUNCH_FAILURE, "kernel launch", _e); \
         if ((ctx)->capturing) (ctx)->capture_launches++; else (ctx)->launches++; } while (0)

// Back-to-back launches of short kernels.  A kernel launched with fg_launch (or, in clusters, fg_launch_cluster) is set up while the
// kernel before it on the stream drains (programmatic stream serialization); fg_grid_enter(), which comes in every thread before
// anything that reads or writes memory of the device, waits until
// everything before it has finished and is visible.  Nothing is triggered early: blocks of the next kernel that wait on the
// SMs from the start of this one's work on slow it several times over, once the host is ahead (18 x (88 x 24 x 256) backward,
// two launches: 14.4 us in plain order, 10.8 like this, 30 to 37 with a trigger on entry).  Seven launches of a ragged layer's
// backward pass 71.6 -> 53.6 us, the 16 of a 2-16-2 training step 36.2 -> 30.1 us.
template <typename... P, typename... A>
inline void fg_launch_cluster(fg_ctx* ctx, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, unsigned cluster, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (!ctx->comm) {      // with a communicator the stream also forks and joins: plain order there
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = cluster;
        attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
        ++cfg.numAttrs;
    }
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);      // FG_LAUNCHED reports its error
}
template <typename... P, typename... A>
inline void fg_launch(fg_ctx* ctx, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
    fg_launch_cluster(ctx, kernel, grid, block, smem, 1, std::forward<A>(args)...);
}
__device__ __forceinline__ void fg_grid_enter() { cudaGridDependencySynchronize(); }

// Sums over the blocks of a launch: every block leaves its part in memory, and the parts are added in an order that does not depend
// on who adds them, by the block that counts itself last or by a launch of its own.  The counters (behind the device error word)
// start at zero and wrap back to it; the kernels of a context run one after the other, so one set serves all of them.
constexpr uint32_t kFgArrivals = 1024;
inline unsigned* fg_arrivals(const fg_ctx* ctx) { return reinterpret_cast<unsigned*>(ctx->dev_status) + 64; }
constexpr size_t kFgStatusBytes = 256 + kFgArrivals * sizeof(unsigned);
// Does the last block add?  Recorded in a plan, a second launch costs the device 0.9 us, and the fence, the counter and the way to the
// other parts 1.7 us or more, for every wave of blocks; called one by one, every launch costs the host 2 us, which is more than
// either while the blocks are few.  MSE of 4096 and of 1 Mi elements, column sums of 384 x 256 and of 16384 x 1000, us:
// in a plan 2.2 / 4.3 / 2.8 / 8.3 with a second launch and 3.2 / 6.7 / 3.4 / 13.3 in one; called one by one 6.2 / 6.2 / 6.1 /
// 8.9 and 4.1 / 7.0 / 4.5 / 13.4.
inline bool fg_fold_in_launch(const fg_ctx* ctx, uint64_t blocks) { return !ctx->capturing && blocks <= 2 * (uint64_t)ctx->sm_count; }
// Called by all threads of a block after they have written their part; true in the block that is the last of `blocks`.
__device__ __forceinline__ bool fg_last_block(unsigned* arrivals, unsigned blocks) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) last = atomicInc(arrivals, blocks - 1) == blocks - 1;
    __syncthreads();
    if (last) __threadfence();
    return last != 0;
}
// The sum of n partial sums, in thread 0 of 256: in strides of 256, then across the threads.
__device__ __forceinline__ float fg_sum_partials(const float* partials, uint32_t n, float* red) {
    float s = 0.0f;
    for (uint32_t i = threadIdx.x; i < n; i += 256) s += __ldcg(partials + i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    s = 0.0f;
    if (threadIdx.x == 0)
        for (int w = 0; w < 8; ++w) s += red[w];
    return s;
}
// A block's sum (in thread 0 of 256) goes to the partials; with `out`, the last block adds them.
__device__ __forceinline__ void fg_leave_sum(float s, float* partials, unsigned* arrivals, float* out, float* red) {
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
    if (!out || !fg_last_block(arrivals, gridDim.x)) return;
    s = fg_sum_partials(partials, gridDim.x, red);
    if (threadIdx.x == 0) *out = s;
}

// Brackets one kernel launch with events when timing is enabled (never while capturing).
inline fg_time_rec* fg_time_begin(fg_ctx* ctx, int kind, double work) {
    if (!ctx->timing_on || ctx->capturing || !ctx->time_recs || ctx->time_count >= FG_TIME_MAX_RECS) return nullptr;
    fg_time_rec* r = &ctx->time_recs[ctx->time_count];
    if (ctx->time_count >= ctx->time_created) {
        if (cudaEventCreate(&r->a) != cudaSuccess || cudaEventCreate(&r->b) != cudaSuccess) return nullptr;
        ctx->time_created = ctx->time_count + 1;
    }
    r->kind = kind;
    r->work = work;
    cudaEventRecord(r->a, ctx->stream);
    ctx->time_count++;
    return r;
}
inline void fg_time_end(fg_ctx* ctx, fg_time_rec* r) {
    if (r) cudaEventRecord(r->b, ctx->stream);
}

inline bool fg_aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Returns a 256-byte aligned slice of the scratch arena, growing it when allowed.
int32_t fg_ws_alloc(fg_ctx* ctx, uint64_t bytes, void** out);
// Room for `bytes` more in the arena (grows it when nothing has been carved yet for this operation).
int32_t fg_ws_ensure(fg_ctx* ctx, uint64_t bytes);
bool fg_ws_try(fg_ctx* ctx, uint64_t bytes);      // the same, but a failure changes nothing and is no error

// SMs for a kernel whose CTAs take one each and stay to its end.
inline uint64_t fg_free_sms(const fg_ctx* ctx) { return fg_sms_beside(ctx->sm_count, ctx->comm_pending, ctx->comm_reserved_sms); }

// Grid for a bandwidth-bound grid-stride kernel: a multiple of the SM count.
inline int fg_stream_grid(const fg_ctx* ctx, uint64_t work_items, int threads, int per_sm) {
    uint64_t need = (work_items + threads - 1) / threads;
    uint64_t cap = (uint64_t)ctx->sm_count * per_sm;
    if (need < 1) need = 1;
    return (int)(need < cap ? need : cap);
}

// ---- activation maths shared by the GEMM epilogue and the elementwise kernels ----
// Constants of the reference's tanh-approximated GELU (op/unary.rs:493-494).
#define FG_GELU_A 0.044715f
#define FG_GELU_B 0.7978846f

__device__ __forceinline__ float fg_ex2_fast(float a) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a)); return r; }
__device__ __forceinline__ float fg_rcp_fast(float a) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a)); return r; }

// With u the argument of GELU's tanh, e = exp(-2|u|) <= 1, r = 1 / (1 + e) and q = e * r, 0.5 * (1 + tanh(u)) is 1 - q for
// x > 0 and q for x < 0, so gelu(x) = max(x, 0) - |x| * q and gelu'(x) = [x > 0 ? 1 - q : q] + 2x * q * r * du/dx: a
// third of the instructions of the tanhf form and nothing cancels (1 + tanh(u) does for negative x).  The reciprocal takes
// one Newton step (its residual is exact by fma).  Error against 64 bits over N(0,1): 3.7e-8 of the result (2-norm),
// 3.8e-8 with tanhf.
__device__ __forceinline__ void fg_gelu_terms(float x, float& q, float& r) {
    constexpr double kB = 0.7978846, kA = 0.044715, kC1 = -1.4426950408889634 * 2.0 * kB;
    const float e = fg_ex2_fast(fabsf(x) * __fmaf_rn(x * x, (float)(kC1 * kA), (float)kC1));
    const float d = 1.0f + e;
    r = fg_rcp_fast(d);
    r = __fmaf_rn(r, __fmaf_rn(-d, r, 1.0f), r);
    q = e * r;
}
__device__ __forceinline__ float fg_gelu_fwd(float x) {
    float q, r;
    fg_gelu_terms(x, q, r);
    const float p = x > 1e30f ? 0.0f : fabsf(x) * q;      // +inf stays +inf (q is zero there)
    return fmaxf(x, 0.0f) - p;
}
__device__ __forceinline__ float fg_gelu_grad(float x) {
    float q, r;
    fg_gelu_terms(x, q, r);
    const float du = __fmaf_rn(x * x, FG_GELU_B * FG_GELU_A * 3.0f, FG_GELU_B);
    return __fmaf_rn((x + x) * (r * q), du, x > 0.0f ? 1.0f - q : q);
}

__device__ __forceinline__ float fg_act_fwd(int act, float z) {
    switch (act) {
        case FG_ACT_RELU: return z > 0.0f ? z : 0.0f;
        case FG_ACT_TANH: return tanhf(z);
        case FG_ACT_GELU: return fg_gelu_fwd(z);
        default: return z;
    }
}

// d act / d z given the saved value (output y for relu/tanh, pre-activation z for gelu).
__device__ __forceinline__ float fg_act_grad(int act, float saved) {
    switch (act) {
        case FG_ACT_RELU: return saved > 0.0f ? 1.0f : 0.0f;
        case FG_ACT_TANH: return 1.0f - saved * saved;
        case FG_ACT_GELU: return fg_gelu_grad(saved);
        default: return 1.0f;
    }
}

// ---- the same activations for GEMM epilogues ----
// An epilogue runs while the tensor core is already on the next tile and must be done before the two
// accumulators it can run ahead by are full; eight warps do it, so it is bound by instruction issue and its
// arithmetic is kept short: tanh through one exponential and one reciprocal (both the hardware approximations,
// 1-2 ulp), 0.5*(1 + tanh(u)) = 1 / (1 + exp(-2u)), polynomials as explicit fused multiply-adds.  For GELU this
// form has no cancellation; results agree with the libm forms above to a few 1e-7 of the output's scale.
// 1 / (1 + exp(-a)) with a given pre-multiplied by -log2(e): sigmoid(a) = 1 / (1 + 2^(a * -log2 e)).
__device__ __forceinline__ float fg_sigmoid_l2(float a_neg_l2) { return fg_rcp_fast(1.0f + fg_ex2_fast(a_neg_l2)); }
#define FG_NEG_LOG2E (-1.4426950408889634f)
// -log2(e) * 2 * FG_GELU_B * (x + FG_GELU_A x^3) = x * (c1 + c3 x^2)
#define FG_GELU_C1 (FG_NEG_LOG2E * 2.0f * FG_GELU_B)
#define FG_GELU_C3 (FG_NEG_LOG2E * 2.0f * FG_GELU_B * FG_GELU_A)

__device__ __forceinline__ float fg_act_fwd_fast(int act, float z) {
    switch (act) {
        case FG_ACT_RELU: return z > 0.0f ? z : 0.0f;
        case FG_ACT_TANH: return __fmaf_rn(2.0f, fg_sigmoid_l2(z * (2.0f * FG_NEG_LOG2E)), -1.0f);
        case FG_ACT_GELU: return z * fg_sigmoid_l2(z * __fmaf_rn(z * z, FG_GELU_C3, FG_GELU_C1));
        default: return z;
    }
}

__device__ __forceinline__ float fg_act_grad_fast(int act, float saved) {
    switch (act) {
        case FG_ACT_RELU: return saved > 0.0f ? 1.0f : 0.0f;
        case FG_ACT_TANH: return __fmaf_rn(-saved, saved, 1.0f);
        case FG_ACT_GELU: {
            // s = 0.5*(1 + tanh(u)); 1 - tanh(u)^2 = 4*s*(1 - s); gelu' = s + 0.5*x*(1 - tanh^2)*du/dx
            const float xx = saved * saved;
            const float s = fg_sigmoid_l2(saved * __fmaf_rn(xx, FG_GELU_C3, FG_GELU_C1));
            const float du = __fmaf_rn(xx, FG_GELU_B * FG_GELU_A * 3.0f, FG_GELU_B);
            return __fmaf_rn((saved + saved) * (s * (1.0f - s)), du, s);
        }
        default: return 1.0f;
    }
}

// Compact forms of the two functions above for code that is unrolled or must stay small: one uniform branch
// separates the activations that need an exponential from those that do not, and selects do the rest (instead
// of a switch whose every case is expanded at every call site).
__device__ __forceinline__ float fg_act_fwd_sel(int act, float z) {
    if (act >= FG_ACT_TANH) {
        const float arg = act == FG_ACT_TANH ? z * (2.0f * FG_NEG_LOG2E) : z * __fmaf_rn(z * z, FG_GELU_C3, FG_GELU_C1);
        const float s = fg_sigmoid_l2(arg);
        return act == FG_ACT_TANH ? __fmaf_rn(2.0f, s, -1.0f) : z * s;
    }
    return act == FG_ACT_RELU ? fmaxf(z, 0.0f) : z;
}
__device__ __forceinline__ float fg_act_grad_sel(int act, float saved) {
    const float xx = saved * saved;
    if (act == FG_ACT_GELU) {
        const float s = fg_sigmoid_l2(saved * __fmaf_rn(xx, FG_GELU_C3, FG_GELU_C1));
        const float du = __fmaf_rn(xx, FG_GELU_B * FG_GELU_A * 3.0f, FG_GELU_B);
        return __fmaf_rn((saved + saved) * (s * (1.0f - s)), du, s);
    }
    const float relu = saved > 0.0f ? 1.0f : 0.0f;
    return act == FG_ACT_TANH ? 1.0f - xx : act == FG_ACT_RELU ? relu : 1.0f;
}

// ---- bf16 pairs of an f32 tensor (operands of the default GEMM mode) ----
// A kind::tf32 MMA that reads an f32 word from shared memory uses sign, exponent and the top 10 mantissa
// bits: it sees trunc(x).  The pairs carry what the split product needs beside that: plane 0 = bf16(x),
// plane 1 = bf16(x - trunc(x)).  Whoever writes a tensor writes its pairs in the same pass.
__device__ __forceinline__ float fg_trunc_tf32(float x) { return __uint_as_float(__float_as_uint(x) & 0xffffe000u); }
__device__ __forceinline__ void fg_store_pairs4(__nv_bfloat16* pairs, uint64_t plane_stride, size_t idx, float4 v) {
    const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
    const __nv_bfloat162 l0 = __floats2bfloat162_rn(v.x - fg_trunc_tf32(v.x), v.y - fg_trunc_tf32(v.y));
    const __nv_bfloat162 l1 = __floats2bfloat162_rn(v.z - fg_trunc_tf32(v.z), v.w - fg_trunc_tf32(v.w));
    uint2 h, l;
    h.x = *reinterpret_cast<const uint32_t*>(&h0); h.y = *reinterpret_cast<const uint32_t*>(&h1);
    l.x = *reinterpret_cast<const uint32_t*>(&l0); l.y = *reinterpret_cast<const uint32_t*>(&l1);
    *reinterpret_cast<uint2*>(pairs + idx) = h;
    *reinterpret_cast<uint2*>(pairs + plane_stride + idx) = l;
}
__device__ __forceinline__ void fg_store_pairs1(__nv_bfloat16* pairs, uint64_t plane_stride, size_t idx, float v) {
    pairs[idx] = __float2bfloat16_rn(v);
    pairs[plane_stride + idx] = __float2bfloat16_rn(v - fg_trunc_tf32(v));
}

// ---- internal launchers used across translation units ----
int32_t fg_gemm_simt_launch(fg_ctx* ctx, int transA, int transB, uint32_t M, uint32_t N, uint32_t K,
                            const float* A, const float* B, float* C, const float* bias, int act,
                            float* preact_out);
// The same for `batch` matrices in one launch (grid z = matrix; strides in elements).
int32_t fg_gemm_simt_batched_launch(fg_ctx* ctx, int transA, int transB, uint32_t batch, uint32_t M, uint32_t N, uint32_t K,
                                    const float* A, uint64_t sA, const float* B, uint64_t sB, float* C, uint64_t sC,
                                    const float* bias, int act, float* preact_out);
// Is the exact path the faster one for a small forward product whose order of sums is free?
bool fg_gemm_simt_suits(uint32_t M, uint32_t N, uint32_t K);
// Does the exact path take its 64 x 64 tiles for these products?
bool fg_gemm_simt_large(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t batch);
// dB = Aᵀ·dZ and dA = dZ·Bᵀ of a batch in one launch, where fg_gemm_simt_large says no for both.
int32_t fg_gemm_simt_batched_bwd_launch(fg_ctx* ctx, uint32_t batch, uint32_t M, uint32_t N, uint32_t K, const float* A, uint64_t sA, const float* B,
                                        uint64_t sB, const float* dZ, uint64_t sC, float* dA, float* dB);
// Do two ranges of bytes overlap (NULL: no)?
bool fg_ranges_meet(const void* p, uint64_t np, const void* q, uint64_t nq);
// One product of the FMA kernel: C[M,N] = op(A)[M,K] · op(B)[K,N], operands dense as they are stored (ta: A is [K,M], tb: B is
// [N,K]), batch strides in elements.  All pointers but A, B and C may be NULL.
struct FgFmaOp {
    int ta, tb;
    uint32_t M, N, K;
    const float *A, *B;
    float* C;
    const float* factor;              // ta xor tb: the operand that is not transposed is x * act'(factor)
    int factor_act;
    const float* bias;                // C = act(sum + bias), or (sum + bias) * act'(mul_saved)
    int act;
    float* preact;
    const float* mul_saved;
    int mul_act;
    __nv_bfloat16* pairs;             // of C
    uint64_t pairs_stride;
    float *colsum_b, *colsum_c;       // [N]: sums over k of the B operand (ta only), over the rows of C
    uint64_t sA, sB, sC;
};
// One product, or two in one launch (the first with ta, the second with tb).  in_order: every sum is one chain of FMAs in the order of
// k, the exact path's results (forward, or both gradients).  Room in the arena for one row of C's column sums per 32 rows.
int32_t fg_gemm_fma_launch(fg_ctx* ctx, const FgFmaOp* ops, int n, uint32_t batch, bool in_order);
// Is it the kernel for the forward product of [M,K] x [K,N], or for one or both of its gradients?  kFgFactor: dZ is formed on the way;
// kFgBelow: dA becomes the dZ of the layer below; kFgBias: with the bias gradient.
enum { kFgForward = 0, kFgGradB = 1, kFgGradA = 2, kFgFactor = 4, kFgBelow = 8, kFgBias = 16 };
bool fg_gemm_fma_suits(uint32_t M, uint32_t N, uint32_t K, int products);
// The same for products too small for the tensor cores: the narrow layer's own kernels take the gradients of up to 16 columns and many rows.
bool fg_gemm_fma_suits_small(uint32_t M, uint32_t N, uint32_t K, int products);
// A layer's backward pass with it: dZ = dZ * act'(factor); dB, dbias; the exchange; dA (* act'(mul_saved), pairs, column sums).
struct FgFmaBwd {
    uint32_t M, N, K;
    const float *A, *B, *dZ, *factor;
    int factor_act;
    float *dA, *dB, *dbias;
    const float* mul_saved;
    int mul_act;
    __nv_bfloat16* pairs;
    uint64_t pairs_stride;
    float* below_dbias;
    float* exch_buf;
    uint64_t exch_count;
};
int32_t fg_gemm_fma_bwd(fg_ctx* ctx, const FgFmaBwd& b);
uint64_t fg_gemm_fma_bwd_scratch(const FgFmaBwd& b);      // what it carves from the arena, beside column sums of dA
// Does the backward pass of this layer sum dZ's columns on its way (fg_gemm_bwd_paired_f32's dbias costs nothing)?
bool fg_gemm_bwd_sums_bias(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, bool dA);
uint64_t fg_gemm_skinny_scratch_bytes(uint32_t M, uint32_t N, uint32_t K);   // enough for any one skinny launch
int32_t fg_gemm_skinny_n_launch(fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, const float* A, const float* B, float* C,
                                const float* bias, int act, float* preact_out);
// Optional extras of the dA kernel: dA = (dZ·Bᵀ) * act'(mul_saved), its bf16 pairs, and partial column sums
// (the partials of the bias gradient of the layer below): room for [fg_gemm_skinny_colsum_rows(M)][K]; the launch
// reports how many rows it wrote.
uint32_t fg_gemm_skinny_colsum_rows(uint32_t M);
struct fg_skinny_extras {
    const float* mul_saved;
    int mul_act;
    __nv_bfloat16* pairs;
    uint64_t pairs_stride;
    float* colsum_part;
};
int32_t fg_gemm_skinny_nt_launch(fg_ctx* ctx, uint32_t M, uint32_t K, uint32_t N, const float* dZ, const float* B,
                                 float* dA, const fg_skinny_extras* extras = nullptr, uint32_t* colsum_rows = nullptr);
int32_t fg_gemm_skinny_tn_launch(fg_ctx* ctx, uint32_t M, uint32_t Kd, uint32_t N, const float* A, const float* dZ,
                                 float* dB);
int32_t fg_convert_launch(fg_ctx* ctx, const void* src, int src_dtype, void* dst, int dst_dtype, uint64_t n);
int32_t fg_act_bwd_launch(fg_ctx* ctx, uint64_t n, int act, const float* dy, const float* saved, float* dz);
// Which tensors' bf16 pairs the forward and backward products of [M,K] x [K,N] read when they exist: 1 A, 2 B, 4 dZ.
uint32_t fg_gemm_reads_pairs(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K);
// fg_ce_loss_grad with the sum of the losses; its arguments have been checked.
int32_t fg_ce_loss_grad_sum(fg_ctx* ctx, const float* probs, const uint32_t* labels, uint32_t rows, uint32_t cols, float* loss_out,
                            float* grad_out, float* loss_sum_out);
// fg_adamw_step_multi (gradients zeroed) of step *counter + 1; `count`: the counter is that step afterwards.
int32_t fg_adamw_next_step(fg_ctx* ctx, const fg_update_tensor* tensors, uint32_t n, const fg_adamw_hyper* h, uint32_t* counter, bool count);
// Where `grid` blocks leave their partial sums (scratch, or *sum itself for one block), where the last of them leaves the sum, if it
// adds them; fg_block_sums_end(), after the launch, has them added otherwise.  No sum wanted: both NULL.
struct FgBlockSums { float *partials, *out, *sum; int grid; };
int32_t fg_block_sums(fg_ctx* ctx, int grid, float* sum, FgBlockSums* b);
int32_t fg_block_sums_end(fg_ctx* ctx, const FgBlockSums& b);
int32_t fg_colsum_launch(fg_ctx* ctx, uint32_t rows, uint32_t cols, const float* x, float* out);
int32_t fg_colsum_fold_launch(fg_ctx* ctx, uint32_t cols, uint32_t nchunks, const float* part, void* out, int out_dtype = FG_DTYPE_F32);

// Dense f32 and 16-bit GEMM on the tcgen05 tensor cores, and the GEMM entry points (forward with fused bias +
// activation epilogue, backward dA / dB / dbias).
//
// What it replaces: the reference's tiled scalar-FMA matmul and its backward edges
// (crates/ferrograd-nn/src/op/matmul/mod.rs:17-188, generic.rs:13-325; dA = dC·Bᵀ via
// transpose_b, dB = Aᵀ·dC via transpose_a, mod.rs:75-101) together with the epilogue
// fusion of trailing elementwise ops (crates/fused_gpu/src/dispatch/backend/kernel/forward.rs:373-457)
// and the activation-derivative factor of the backward chains (op/unary.rs:281-309,
// :453-472, :588-714).
//
// Method.  An f32 product is a split product: x = hi + lo with hi = tf32(x); A·B ~= hi·hi on kind::tf32 plus the two
// cross terms, on kind::f16 from bf16 planes (bf16(x), bf16(lo)) or, in the strict 3xTF32 mode, on kind::tf32 from
// tf32(lo).  Accumulators are f32 in tensor memory, drained in chunks of k; the dropped lo·lo term is ~2^-23 relative.
// Four ways to get hi and lo to the tensor core, chosen by estimates of their times (pick_route and its callers):
//   * pairs: the f32 tensor as it lies (the MMA truncates it) beside bf16 planes kept with it or made in one pass;
//     256 x 256 tiles on SM pairs.  Large products.
//   * conversion kernel: the f32 tensors alone; warps round and split each k-block, one operand into tensor memory and the
//     other in shared memory.  Small and middling products, batches.
//   * operand planes: a pre-pass writes hi and lo planes of each operand into the scratch arena, contraction index
//     contiguous, transposing on the way; dY * act'(saved) is applied there.  Any shape; the strict mode.
//   * 16-bit tensors go to kind::f16 as they lie, with a padded copy where rows are not 16-byte aligned.
// Every kernel is a warp-specialised pipeline: one warp issues bulk-tensor loads (no multicast) into swizzled shared
// memory, one warp issues tcgen05.mma (a lane of each, elected where the warp runs the role as a whole), other warps read the
// accumulators back with tcgen05.ld and apply bias and activation while storing.
#include <atomic>
#include <cuda_bf16.h>
#include <stdlib.h>

#include <type_traits>

#include "fg_internal.cuh"
#include "ptx_sm100.cuh"

using namespace fgptx;

namespace {

constexpr int BM = 128;         // rows of the output tile = UMMA M
static_assert(BM == (int)kConvTileM, "the plan's tiles");
// BK (template parameter): f32 per k-block = one swizzled shared-memory row: 32 (128-byte swizzle) or 16 (64-byte).
constexpr int UK = 8;           // K of one tcgen05.mma kind::tf32
constexpr long long kWaitCycles = 2000000000LL;   // bound on every device-side wait (about 1 s)

struct Epilogue {
    float* C;
    const float* bias;   // in the storage type, see epi_bias
    float* preact;
    uint32_t M, N, K;
    int act;
    int* dev_status;
    // Split-K tail of the pair kernel: tiles [0, t_full) are whole; each later tile is computed as `split`
    // partial sums over equal shares of the K chunks, written raw to `partial` and folded by a second kernel.
    float* partial;
    uint32_t t_full, split;
    int out_dtype;       // storage type of C, preact and bias (fg_dtype); partial is always f32
    // ---- pair kernel on f32 tensors with bf16 pairs (FMT 1) ----
    uint32_t a_mn, b_mn;              // the operand's storage has the non-contraction index contiguous
    __nv_bfloat16* c_pairs;           // optional: bf16 pairs of the stored C (see pairs_kernel)
    uint64_t c_pairs_stride;          // elements between the two planes of c_pairs
    const float* mul_saved;           // optional [M,N]: C = (acc + bias) * act'(mul_saved), act = mul_act
    int mul_act;
    float* colsum_part;               // optional [ceil(M/32)][N]: column sums of the stored C per 32-row block
    uint32_t group;                   // tile rows per group of the tile order (see pair_tile_origin)
    uint64_t c_batch;                 // conversion kernel: elements between two matrices of a batch in C and preact
#ifdef FG_GEMM_PROFILE
    uint32_t dbg;                     // diagnostic build: bit 0 = leave out the global stores of the epilogue
#endif
};

// Element stores in the output's storage type (idx in elements).
__device__ __forceinline__ void store_out4(void* base, size_t idx, float4 v, int dt) {
    if (dt == FG_DTYPE_F32) {
        *reinterpret_cast<float4*>(static_cast<float*>(base) + idx) = v;
    } else if (dt == FG_DTYPE_F16) {
        const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
        uint2 u;
        u.x = *reinterpret_cast<const uint32_t*>(&lo);
        u.y = *reinterpret_cast<const uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(static_cast<__half*>(base) + idx) = u;
    } else {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
        uint2 u;
        u.x = *reinterpret_cast<const uint32_t*>(&lo);
        u.y = *reinterpret_cast<const uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(base) + idx) = u;
    }
}
// The bias of column c, which lies in the output's storage type.
__device__ __forceinline__ float epi_bias(const float* bias, uint32_t c, int dt) {
    if (dt == FG_DTYPE_F32) return bias[c];
    return dt == FG_DTYPE_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[c]) : __half2float(reinterpret_cast<const __half*>(bias)[c]);
}
__device__ __forceinline__ void store_out1(void* base, size_t idx, float v, int dt) {
    if (dt == FG_DTYPE_F32) static_cast<float*>(base)[idx] = v;
    else if (dt == FG_DTYPE_F16) static_cast<__half*>(base)[idx] = __float2half_rn(v);
    else static_cast<__nv_bfloat16*>(base)[idx] = __float2bfloat16_rn(v);
}

// Origin of pair tile `tile`: tiles are numbered so that eight consecutive pair-rows sweep all columns
// before the next eight start.  The pairs working at the same time then cover a squarish block of C and
// re-use both its A rows and its B rows from L2 (with rows-fastest order every wave streamed all of A
// again: 7.7x the operand bytes from DRAM at 8192^3).
__host__ __device__ __forceinline__ void pair_tile_origin(uint32_t tile, uint32_t pairs_m, uint32_t pairs_n,
                                                          uint32_t tile_m, uint32_t tile_n, uint32_t kGroup, uint32_t& m0,
                                                          uint32_t& n0) {
    const uint32_t grp = tile / (kGroup * pairs_n);
    const uint32_t left = pairs_m - grp * kGroup;
    const uint32_t grp_rows = left < kGroup ? left : kGroup;
    const uint32_t rem = tile - grp * kGroup * pairs_n;
    m0 = (grp * kGroup + rem % grp_rows) * tile_m;
    n0 = (rem / grp_rows) * tile_n;
}

// One shared copy of the activation code.  fg_act_fwd inlines tanhf and the GELU polynomial at every call
// site; an epilogue that is unrolled over a thread's 128 accumulators would carry 128 copies and run out
// of instruction cache (measured on the pair kernel: 45,000 cycles for ~1,000 useful instructions).
__device__ __noinline__ float4 act_fwd4(int act, float4 z) {
    return make_float4(fg_act_fwd_fast(act, z.x), fg_act_fwd_fast(act, z.y), fg_act_fwd_fast(act, z.z), fg_act_fwd_fast(act, z.w));
}
// z * act'(saved): the backward factor of the layer below, applied while a dA tile is stored.
__device__ __noinline__ float4 act_mul4(int act, float4 z, float4 sv) {
    return make_float4(z.x * fg_act_grad_fast(act, sv.x), z.y * fg_act_grad_fast(act, sv.y), z.z * fg_act_grad_fast(act, sv.z),
                       z.w * fg_act_grad_fast(act, sv.w));
}

// Four columns of one row, element by element: the ragged right edge of a matrix whose width is not a multiple
// of four, or unaligned pointers.  A cold path, kept out of line so that it does not sit in the unrolled epilogue.
__device__ __noinline__ float4 epi_store_edge(float4 zin, size_t off, uint32_t col, uint32_t col_lim, char* out, char* pre,
                                               __nv_bfloat16* pairs, uint64_t pairs_stride, const float* mul, int mul_act, int act,
                                               int odt) {
    const float z[4] = {zin.x, zin.y, zin.z, zin.w};
    float o4[4] = {0.f, 0.f, 0.f, 0.f};
    for (int t = 0; t < 4; ++t)
        if (col + t < col_lim) {
            const float o = mul ? z[t] * fg_act_grad_fast(mul_act, mul[off + t]) : fg_act_fwd_fast(act, z[t]);
            if (pre) store_out1(pre, off + t, z[t], odt);
            store_out1(out, off + t, o, odt);
            if (pairs) fg_store_pairs1(pairs, pairs_stride, off + t, o);
            o4[t] = o;
        }
    return make_float4(o4[0], o4[1], o4[2], o4[3]);
}

template <int BN, int BK>
struct TileCfg {
    static constexpr int kABytes = 2 * BM * BK * 4;   // hi + lo tiles of A
    static constexpr int kBBytes = 2 * BN * BK * 4;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kStages = (200 * 1024) / kStageBytes > 8 ? 8 : (200 * 1024) / kStageBytes;
    static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
    static constexpr int kTmemCols = 2 * BN < 32 ? 32 : 2 * BN;   // two accumulators (ping-pong)
    static constexpr int kColsPerThread = BN / 2;                 // each lane quarter is shared by two warps
};

#ifdef FG_GEMM_PROFILE
// Diagnostic build only (-DFG_GEMM_PROFILE): cycle counters of the pair kernel's roles, summed over CTAs.
// 0 MMA wait for a drained accumulator, 1 MMA wait for loads, 2 MMA loop total, 3 epilogue (warp 2) wait for a
// finished chunk, 4 epilogue store phase, 5 units, 6 producer wait for a free stage, 7 reporting CTAs.
__device__ unsigned long long g_prof[8];
#define PROF_T0() const long long _pt0 = clock64()
#define PROF_ADD(var) var += clock64() - _pt0
#else
#define PROF_T0()
#define PROF_ADD(var)
#endif

constexpr int kThreads = 320;      // warp 0: loads, warp 1: MMA issue, warps 2..9: accumulate + epilogue
// The pair kernel runs three warpgroups: warps 0..3 (loads, MMA issue, two idle warps) keep kPairRegsLow registers
// per thread, the eight accumulate + epilogue warps 4..11 take kPairRegsHigh.  A thread of those owns 128 running
// sums; with the 168 registers a 384-thread CTA gets by default, the store phase spilled, and with 227 KB of the
// SM's memory configured as shared memory there is next to no L1 behind local memory: every spill access cost an
// L2 round trip (measured: ~50 cycles per instruction in the store phase, 20,000 cycles per tile).
constexpr int kPairThreads = 384;
constexpr int kPairRegsLow = 72, kPairRegsHigh = 216;     // 128 * 72 + 256 * 216 = 64,512 <= 65,536
constexpr int kPairEpiWarp0 = 4;
constexpr int kChunkK = 256;       // values of k per accumulation chunk

// The tensor core adds into its f32 accumulator with truncation, so a long chain of
// tcgen05.mma drifts linearly with K (measured: 1.9e-4 relative at K = 8192).  The K loop is
// therefore cut into chunks of kChunkK values of k.  Each chunk accumulates in one of two
// tensor-memory accumulators, starting from zero; when it completes, the eight epilogue
// warps read it back and add it, rounding to nearest, to running sums held in registers
// while the tensor core is already working on the next chunk in the other accumulator.
//
// FMT selects the operand planes and the MMA sequence per k-block:
//   0  [hi | lo] f32 planes; three kind::tf32 MMAs per 8-wide k-step (lo*hi, hi*lo, hi*hi): "3xTF32".
//   1  hi as f32 (tf32-rounded) plus a bf16 pair [bf16(x) | bf16(x - hi)]; the dominant term hi*hi
//      runs as kind::tf32, the two cross terms as kind::f16 (bf16) MMAs, which take half the time of a
//      tf32 MMA per k: two tf32-units of tensor work per product instead of three.  The cross terms
//      are 2^-12 of the product, so bf16's 2^-9 relative rounding costs ~2^-20 relative per product.
template <int BN, int BK, int FMT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmA16, const __grid_constant__ CUtensorMap tmB16, Epilogue ep) {
    static_assert(FMT == 0 || BK == 32, "the bf16 planes use 64-byte rows: 32 values of k per block");
    using Cfg = TileCfg<BN, BK>;
    constexpr int S = Cfg::kStages;
    constexpr int CPT = Cfg::kColsPerThread;
    extern __shared__ unsigned char smem_raw[];
    // 1024-byte alignment: required by the 128-byte swizzle (descriptor base offset 0).
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* base_ptr = smem_raw + (base - raw);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(base_ptr + S * Cfg::kStageBytes);
    const uint32_t bar0 = base + S * Cfg::kStageBytes;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (S + s); };
    auto acc_full_bar = [&](int b) { return bar0 + 8u * (2 * S + b); };
    auto acc_empty_bar = [&](int b) { return bar0 + 8u * (2 * S + 2 + b); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * S + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const uint32_t nkb = (ep.K + BK - 1) / BK;
    constexpr uint32_t kChunkKB = kChunkK / BK;   // k-blocks per accumulation chunk
    const uint32_t nchunks = (nkb + kChunkKB - 1) / kChunkKB;

    // A wait that expired earlier (this launch or a previous one) makes every CTA leave at once.
    // One thread reads the word so that the whole CTA takes the same branch.
    __shared__ int s_abort;
    if (threadIdx.x == 0) s_abort = *reinterpret_cast<volatile int*>(ep.dev_status);
    __syncthreads();
    if (s_abort != 0) return;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full_bar(b), 1); mbar_init(acc_empty_bar(b), 8); }
        fence_mbar_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        if (FMT == 1) { prefetch_tmap(&tmA16); prefetch_tmap(&tmB16); }
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), Cfg::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ---- producer: bulk-tensor loads ----
            for (uint32_t kb = 0; kb < nkb; ++kb) {
                const int s = kb % S;
                const uint32_t ph = (kb / S) & 1u;
                if (!mbar_wait_bounded(empty_bar(s), ph ^ 1u, kWaitCycles)) {
                    atomicOr(ep.dev_status, FG_DEVERR_TMA_WAIT);
                    break;
                }
                mbar_expect_tx(full_bar(s), Cfg::kStageBytes);
                const uint32_t sa = base + s * Cfg::kStageBytes;
                tma_load_3d(sa, &tmA, full_bar(s), (int)(kb * BK), (int)m0, 0);
                tma_load_3d(sa + Cfg::kABytes, &tmB, full_bar(s), (int)(kb * BK), (int)n0, 0);
                if (FMT == 1) {   // the bf16 pairs follow their operand's f32 tile
                    tma_load_3d(sa + BM * BK * 4, &tmA16, full_bar(s), (int)(kb * BK), (int)m0, 0);
                    tma_load_3d(sa + Cfg::kABytes + BN * BK * 4, &tmB16, full_bar(s), (int)(kb * BK), (int)n0, 0);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issuer ----
            constexpr uint32_t idesc = make_idesc(2u /*tf32*/, BM, BN < 16 ? 16 : BN);
            bool ok = true;
            for (uint32_t c = 0; c < nchunks && ok; ++c) {
                const uint32_t buf = c & 1u;
                // the accumulator must have been drained by the epilogue warps (two chunks ago)
                if (!mbar_wait_bounded(acc_empty_bar(buf), ((c >> 1) & 1u) ^ 1u, kWaitCycles)) {
                    atomicOr(ep.dev_status, FG_DEVERR_MMA_WAIT);
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                const uint32_t kb_end = min(nkb, (c + 1) * kChunkKB);
                for (uint32_t kb = c * kChunkKB; kb < kb_end; ++kb) {
                    const int s = kb % S;
                    const uint32_t ph = (kb / S) & 1u;
                    if (!mbar_wait_bounded(full_bar(s), ph, kWaitCycles)) {
                        atomicOr(ep.dev_status, FG_DEVERR_MMA_WAIT);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = base + s * Cfg::kStageBytes;
                    const uint64_t a_hi = make_desc_kmajor<BK * 4>(sa);
                    const uint64_t a_lo = make_desc_kmajor<BK * 4>(sa + BM * BK * 4);
                    const uint64_t b_hi = make_desc_kmajor<BK * 4>(sa + Cfg::kABytes);
                    const uint64_t b_lo = make_desc_kmajor<BK * 4>(sa + Cfg::kABytes + BN * BK * 4);
                    const uint32_t first = (kb == c * kChunkKB) ? 0u : 1u;   // a chunk starts from zero
                    if (FMT == 0) {
#pragma unroll
                        for (int kk = 0; kk < BK / UK; ++kk) {
                            // advance along K inside the swizzled row: +32 bytes, i.e. +2 in the address field
                            const uint64_t adv = (uint64_t)(kk * UK * 4 >> 4);
                            mma_tf32(d_tmem, a_lo + adv, b_hi + adv, idesc, first | (uint32_t)kk);
                            mma_tf32(d_tmem, a_hi + adv, b_lo + adv, idesc, 1u);
                            mma_tf32(d_tmem, a_hi + adv, b_hi + adv, idesc, 1u);
                        }
                    } else {
                        // bf16 tiles: rows of 64 bytes (32 values of k), two 16-wide k-steps of 32 bytes each
                        constexpr uint32_t idesc16 = make_idesc(1u /*bf16*/, BM, BN < 16 ? 16 : BN);
                        const uint32_t a16 = sa + BM * BK * 4, b16 = sa + Cfg::kABytes + BN * BK * 4;
                        const uint64_t a_h16 = make_desc_kmajor<64>(a16), a_l16 = make_desc_kmajor<64>(a16 + BM * BK * 2);
                        const uint64_t b_h16 = make_desc_kmajor<64>(b16), b_l16 = make_desc_kmajor<64>(b16 + BN * BK * 2);
#pragma unroll
                        for (int kk = 0; kk < BK / 16; ++kk) {
                            const uint64_t adv = (uint64_t)(kk * 16 * 2 >> 4);
                            mma_f16(d_tmem, a_l16 + adv, b_h16 + adv, idesc16, first | (uint32_t)kk);
                            mma_f16(d_tmem, a_h16 + adv, b_l16 + adv, idesc16, 1u);
                        }
#pragma unroll
                        for (int kk = 0; kk < BK / UK; ++kk) {
                            const uint64_t adv = (uint64_t)(kk * UK * 4 >> 4);
                            mma_tf32(d_tmem, a_hi + adv, b_hi + adv, idesc, 1u);
                        }
                    }
                    mma_commit(empty_bar(s));   // frees the stage once these MMAs have read it
                }
                if (ok) mma_commit(acc_full_bar(buf));   // this chunk's accumulator is complete
            }
        }
    } else {
        // ---- accumulate + epilogue: warps 2..9.  Warp w may touch TMEM lanes 32*(w%4) .. +31;
        //      warps 2..5 take the first half of the tile's columns, warps 6..9 the second. ----
        const int q = warp & 3;
        const int half = (warp - 2) >> 2;
        float sum[CPT];
#pragma unroll
        for (int j = 0; j < CPT; ++j) sum[j] = 0.0f;
        bool ok = true;
        for (uint32_t c = 0; c < nchunks; ++c) {
            const uint32_t buf = c & 1u;
            bool got = mbar_wait_bounded(acc_full_bar(buf), (c >> 1) & 1u, kWaitCycles + kWaitCycles / 2);
            got = __all_sync(0xffffffffu, got);
            if (!got) {
                if (lane == 0) atomicOr(ep.dev_status, FG_DEVERR_EPI_WAIT);
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN + half * CPT;
            if constexpr (CPT >= 32) {
#pragma unroll
                for (int g = 0; g < CPT / 32; ++g) {
                    uint32_t r[32];
                    tmem_ld_32x32(t0 + g * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[g * 32 + j] += __uint_as_float(r[j]);
                }
            } else {
                uint32_t r[16];
                tmem_ld_32x16(t0, r);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) sum[j] += __uint_as_float(r[j]);
            }
            tc_fence_before();
            if (lane == 0) mbar_arrive(acc_empty_bar(buf));
        }
        if (ok && *reinterpret_cast<volatile int*>(ep.dev_status) == 0) {
            const uint32_t row = m0 + q * 32 + lane;
            const uint32_t cbase = n0 + half * CPT;
            const bool vec_ok = (ep.N % 4 == 0) && ((reinterpret_cast<uintptr_t>(ep.C) & 15u) == 0) &&
                                (!ep.preact || (reinterpret_cast<uintptr_t>(ep.preact) & 15u) == 0);
            if (row < ep.M) {
                float* crow = ep.C + (size_t)row * ep.N;
                float* prow = ep.preact ? ep.preact + (size_t)row * ep.N : nullptr;
#pragma unroll
                for (int j = 0; j < CPT; j += 4) {
                    const uint32_t col = cbase + j;
                    if (col >= ep.N) break;
                    float z[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        z[t] = sum[j + t];
                        if (ep.bias && col + t < ep.N) z[t] += ep.bias[col + t];
                    }
                    const float4 o = ep.act == FG_ACT_NONE ? make_float4(z[0], z[1], z[2], z[3])
                                                           : act_fwd4(ep.act, make_float4(z[0], z[1], z[2], z[3]));
                    if (vec_ok && col + 3 < ep.N) {
                        if (prow) *reinterpret_cast<float4*>(prow + col) = make_float4(z[0], z[1], z[2], z[3]);
                        *reinterpret_cast<float4*>(crow + col) = o;
                    } else {
                        const float ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                        for (int t = 0; t < 4; ++t)
                            if (col + t < ep.N) {
                                if (prow) prow[col + t] = z[t];
                                crow[col + t] = ov[t];
                            }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

// ------------------------------------------------------------------------------------
// CTA-pair kernel (cta_group::2): two CTAs on neighbouring SMs compute one 256 x 256 tile.
// Each CTA loads its own 128 rows of A and HALF of the B tile (128 of its 256 rows); the
// pair's MMA reads both halves, so the bytes each SM pulls from L2 per k-block drop from
// 96 KiB to 64 KiB.  (The single-CTA kernel is limited by exactly that stream: it takes the
// same time with two thirds of the tensor work.)  CTA 0 of the pair issues all MMAs; both
// CTAs keep their 128 rows of the accumulators in their own tensor memory and run their own
// epilogue.  Loads carry no multicast; the only cross-CTA traffic is signalling
// (load-completion bytes counted on the leader's mbarrier, commit arrivals on both CTAs'
// mbarriers, accumulator-drained arrivals on the leader's mbarrier).
// ------------------------------------------------------------------------------------
constexpr long long kPairWaitCycles = 400000000LL;   // about 0.2 s

template <int BK, int FMT>
struct PairCfg {
    static constexpr int kBN = 256;
    static constexpr int kPlanes = FMT >= 2 ? 1 : 2;         // 16-bit operands are loaded as they are: one 128-byte row
    static constexpr int kABytes = kPlanes * BM * BK * 4;          // this CTA's 128 rows of A: hi + lo (or f32 + bf16 pair)
    static constexpr int kBBytes = kPlanes * (kBN / 2) * BK * 4;   // this CTA's half of the B tile
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kStages = (200 * 1024) / kStageBytes > 8 ? 8 : (200 * 1024) / kStageBytes;
    static constexpr int kStoreBytes = 8 * 32 * 32 * 4;       // the epilogue warps' staging blocks (32 x 32 f32 each)
    static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256 + kStoreBytes;
    static_assert(kSmemBytes <= 232448, "exceeds the 227 KB a CTA may use");
    static constexpr int kTmemCols = 512;                     // two 256-column accumulators
};

// Persistent: the grid is one CTA pair per SM pair (or fewer); pair p computes tiles p, p + P, p + 2P, ...
// The load ring, the MMA issue and the accumulator ping-pong run straight across tile boundaries, so
// while the epilogue warps apply bias/activation and store tile t from their registers, the loads and
// MMAs of tile t+1 are already under way (per-tile set-up, fill and store cost 20-55 us per wave when
// every tile was its own CTA pair: 17 % of a 4096^3 GEMM, more than half of a K = 784 one).
// Two products in a launch (both gradients of a 16-bit layer): a pair takes tiles pair, pair + P, ... of the first, then a run of the
// second's, as long as evens the pairs out (the host's counts, see pair_runs): 384 tiles of which 128 have twice the k are seven
// times of the short ones on 74 pairs instead of the eight of two launches.
template <bool TWO>
struct PairArgs {
    Epilogue ep[TWO ? 2 : 1];
    uint32_t extra;          // pairs with one tile of the first product more than the others: pairs 0 ... extra - 1
    uint32_t run[2];         // tiles of the second product for one of those, and for one of the others
};
template <int BK, int FMT, bool TWO>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmA16, const __grid_constant__ CUtensorMap tmB16,
                    const __grid_constant__ PairArgs<TWO> pa) {
    static_assert(!TWO || FMT >= 2, "the second product's maps take the place of the f32 ones");
    static_assert(FMT == 0 || BK == 32, "the bf16 planes use 64-byte rows: 32 values of k per block");
    // FMT 2 (bf16) and 3 (f16): the operands ARE 16-bit tensors, loaded as they lie (64 values of k per k-block)
    // and multiplied by one kind::f16 MMA per 16 values of k.
    constexpr bool kDirect16 = FMT >= 2;
    constexpr uint32_t KBE = kDirect16 ? 2 * BK : BK;            // values of k per k-block
    constexpr uint32_t kChunk = kDirect16 ? 1024 : kChunkK;      // 16-bit results tolerate the longer chain
    using Cfg = PairCfg<BK, FMT>;
    constexpr int BN = Cfg::kBN, HB = BN / 2;
    constexpr int S = Cfg::kStages;
    constexpr int CPT = BN / 2;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* base_ptr = smem_raw + (base - raw);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(base_ptr + S * Cfg::kStageBytes);
    const uint32_t bar0 = base + S * Cfg::kStageBytes;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (S + s); };
    auto acc_full_bar = [&](int b) { return bar0 + 8u * (2 * S + b); };
    auto acc_empty_bar = [&](int b) { return bar0 + 8u * (2 * S + 2 + b); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * S + 4);

    // (known to be the same in all lanes, as the roles' branches and loops then are: the addresses and descriptors of the loading and
    // the MMA warp live in uniform registers.  From one lane of a divergent branch, issuing the eight MMAs of a k-block took 770 cycles.)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = __shfl_sync(0xffffffffu, cluster_ctarank(), 0);
    const bool leader = rank == 0;
    const uint32_t npairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
    constexpr uint32_t kChunkKB = kChunk / KBE;
    int* const dev_status = pa.ep[0].dev_status;
    // One product's tiles and units.  Work units: whole tiles first, then the tail tiles in `split` K-shares each (the host sizes the
    // tail so that it fills one last wave instead of leaving most pairs idle for a whole tile time).
    struct Units {
        uint32_t pairs_m, pairs_n, nkb, nchunks, n;
    };
    auto units_of = [&](const Epilogue& ep) -> Units {
        Units w;
        w.pairs_m = (ep.M + 2 * BM - 1) / (2 * BM);
        w.pairs_n = (ep.N + BN - 1) / BN;
        w.nkb = (ep.K + KBE - 1) / KBE;
        w.nchunks = (w.nkb + kChunkKB - 1) / kChunkKB;
        w.n = ep.t_full + (w.pairs_m * w.pairs_n - ep.t_full) * ep.split;
        return w;
    };
    auto tile_origin = [&](const Epilogue& ep, const Units& w, uint32_t tile, uint32_t& m0, uint32_t& n0) {
        pair_tile_origin(tile, w.pairs_m, w.pairs_n, 2 * BM, BN, ep.group, m0, n0);
        m0 += rank * BM;                                               // this CTA's rows of A and C
    };
    auto unit_at = [&](const Epilogue& ep, const Units& w, uint32_t u, uint32_t& tile, uint32_t& c0, uint32_t& c1, uint32_t& slot) -> bool {
        if (u < ep.t_full) { tile = u; c0 = 0; c1 = w.nchunks; slot = 0; return false; }
        const uint32_t v = u - ep.t_full, p = v % ep.split;
        tile = ep.t_full + v / ep.split;
        c0 = p * w.nchunks / ep.split;
        c1 = (p + 1) * w.nchunks / ep.split;
        slot = v;
        return true;
    };
    // This pair's run of the second product.
    uint32_t run0 = 0, run1 = 0;
    if constexpr (TWO) {
        const bool more = pair < pa.extra;
        run0 = more ? pair * pa.run[0] : pa.extra * pa.run[0] + (pair - pa.extra) * pa.run[1];
        run1 = min(run0 + pa.run[more ? 0 : 1], units_of(pa.ep[1]).n);
    }

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full_bar(b), 1); mbar_init(acc_empty_bar(b), 16); }
        fence_mbar_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        if (FMT >= 1) { prefetch_tmap(&tmA16); prefetch_tmap(&tmB16); }
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), Cfg::kTmemCols);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();      // the peer's barriers exist before anything is signalled across CTAs
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    if (warp < kPairEpiWarp0) {
    reg_release<kPairRegsLow>();
    if (warp == 0) {
        {
            // ---- producer (both CTAs): own rows of A, own half of B; completion counted on the leader ----
            uint32_t g = 0;      // k-blocks issued so far, across tiles: ring position and phase
            bool ok = true;
            long long prof_a = 0;
            (void)prof_a;
            auto produce = [&](const Epilogue& ep, const CUtensorMap& map_a, const CUtensorMap& map_b, uint32_t first, uint32_t end, uint32_t step) {
            const Units w = units_of(ep);
            for (uint32_t u = first; u < end && ok; u += step) {
                uint32_t tile, c0, c1, slot, m0, n0;
                unit_at(ep, w, u, tile, c0, c1, slot);
                tile_origin(ep, w, tile, m0, n0);
                const uint32_t nb0 = n0 + rank * HB;                    // the rows of B this CTA loads
                const uint32_t kb_last = min(w.nkb, c1 * kChunkKB);
                for (uint32_t kb = c0 * kChunkKB; kb < kb_last; ++kb, ++g) {
                    const int s = g % S;
                    const uint32_t ph = (g / S) & 1u;
                    {
                        PROF_T0();
                        const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(empty_bar(s), ph ^ 1u, kPairWaitCycles));
                        PROF_ADD(prof_a);
                        if (!got) {
                            if (lane == 0) atomicOr(dev_status, FG_DEVERR_TMA_WAIT);
                            ok = false;
                            break;
                        }
                    }
                    if (!elect_one()) continue;
                    const uint32_t lf = map_to_cta(full_bar(s), 0);
                    const uint32_t sa = base + s * Cfg::kStageBytes;
                    if (kDirect16) {
                        if (leader) mbar_expect_tx(full_bar(s), 2 * Cfg::kStageBytes);   // both CTAs' bytes
                        // One operand tile = 128 rows x 64 values of k.  K-major storage: one box; MN-major storage
                        // ([k][rows]): two boxes of 64 rows x 64 k, each [k][64 rows], 8 KiB.
                        auto load16 = [&](uint32_t dst, const CUtensorMap* t16, bool mn, uint32_t r0) {
                            if (!mn) {
                                tma_load_3d_pair(dst, t16, lf, (int)(kb * KBE), (int)r0, 0);
                            } else {
                                tma_load_3d_pair(dst, t16, lf, (int)r0, (int)(kb * KBE), 0);
                                tma_load_3d_pair(dst + 8192, t16, lf, (int)(r0 + 64), (int)(kb * KBE), 0);
                            }
                        };
                        load16(sa, &map_a, ep.a_mn != 0, m0);
                        load16(sa + Cfg::kABytes, &map_b, ep.b_mn != 0, nb0);
                        continue;
                    }
                    if (leader) mbar_expect_tx(full_bar(s), 2 * Cfg::kStageBytes);   // both CTAs' bytes
                    if (FMT == 1) {
                        // One operand tile = 128 rows x 32 values of k as f32 (16 KiB) followed by its two
                        // bf16 planes (2 x 8 KiB).  K-major storage: one box each.  MN-major storage
                        // ([k][rows]): the f32 tile arrives as four boxes of 32 rows x 32 k (each [k][32 rows],
                        // 4 KiB), the bf16 planes as two boxes of 64 rows x 32 k x 2 planes ([plane][k][64 rows]).
                        auto load_tile = [&](uint32_t dst, const CUtensorMap* t32, const CUtensorMap* t16, bool mn, uint32_t r0) {
                            if (!mn) {
                                tma_load_3d_pair(dst, t32, lf, (int)(kb * BK), (int)r0, 0);
                                tma_load_3d_pair(dst + BM * BK * 4, t16, lf, (int)(kb * BK), (int)r0, 0);
                            } else {
#pragma unroll
                                for (int i = 0; i < 4; ++i)
                                    tma_load_3d_pair(dst + i * 4096, t32, lf, (int)(r0 + 32 * i), (int)(kb * BK), 0);
#pragma unroll
                                for (int i = 0; i < 2; ++i)
                                    tma_load_3d_pair(dst + BM * BK * 4 + i * 8192, t16, lf, (int)(r0 + 64 * i), (int)(kb * BK), 0);
                            }
                        };
                        load_tile(sa, &tmA, &map_a, ep.a_mn != 0, m0);
                        load_tile(sa + Cfg::kABytes, &tmB, &map_b, ep.b_mn != 0, nb0);
                    } else {
                        tma_load_3d_pair(sa, &tmA, lf, (int)(kb * BK), (int)m0, 0);
                        tma_load_3d_pair(sa + Cfg::kABytes, &tmB, lf, (int)(kb * BK), (int)nb0, 0);
                    }
                }
            }
            };
            produce(pa.ep[0], tmA16, tmB16, pair, units_of(pa.ep[0]).n, npairs);
            if constexpr (TWO) produce(pa.ep[1], tmA, tmB, run0, run1, 1);
#ifdef FG_GEMM_PROFILE
            if (lane == 0) atomicAdd(&g_prof[6], (unsigned long long)prof_a);
#endif
        }
    } else if (warp == 1) {
        if (leader) {
            // ---- MMA issuer (leader CTA only): M = 256 across the pair, N = 256 ----
            constexpr uint32_t idesc = make_idesc(2u /*tf32*/, 2 * BM, BN);
            bool ok = true;
            uint32_t g = 0, gc = 0;     // k-blocks and chunks consumed so far, across tiles
            long long prof_e = 0, prof_f = 0;
            (void)prof_e; (void)prof_f;
#ifdef FG_GEMM_PROFILE
            const long long prof_start = clock64();
#endif
            auto issue = [&](const Epilogue& ep, uint32_t first_unit, uint32_t end, uint32_t step) {
            const Units w = units_of(ep);
            for (uint32_t u = first_unit; u < end && ok; u += step) {
                uint32_t tile, c0, c1, slot;
                unit_at(ep, w, u, tile, c0, c1, slot);
                for (uint32_t c = c0; c < c1 && ok; ++c, ++gc) {
                    const uint32_t buf = gc & 1u;
                    // the accumulator must have been drained by both CTAs' epilogue warps (two chunks ago)
                    {
                        PROF_T0();
                        const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(acc_empty_bar(buf), ((gc >> 1) & 1u) ^ 1u, kPairWaitCycles));
                        PROF_ADD(prof_e);
                        if (!got) {
                            if (lane == 0) atomicOr(dev_status, FG_DEVERR_MMA_WAIT);
                            ok = false;
                            break;
                        }
                    }
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_base + buf * BN;
                    const uint32_t kb_end = min(w.nkb, (c + 1) * kChunkKB);
                    for (uint32_t kb = c * kChunkKB; kb < kb_end; ++kb, ++g) {
                        const int s = g % S;
                        const uint32_t ph = (g / S) & 1u;
                        {
                            PROF_T0();
                            const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(full_bar(s), ph, kPairWaitCycles));
                            PROF_ADD(prof_f);
                            if (!got) {
                                if (lane == 0) atomicOr(dev_status, FG_DEVERR_MMA_WAIT);
                                ok = false;
                                break;
                            }
                        }
                        tc_fence_after();
                        const uint32_t sa = base + s * Cfg::kStageBytes;
                        const uint64_t a_hi = make_desc_kmajor<BK * 4>(sa);
                        const uint64_t b_hi = make_desc_kmajor<BK * 4>(sa + Cfg::kABytes);
                        const uint32_t first = (kb == c * kChunkKB) ? 0u : 1u;   // a chunk starts from zero
                        if (kDirect16) {
                            // K-major: 16 values of k are 32 bytes inside the swizzled row.  MN-major: 16 k-rows are two
                            // 1024-byte atoms, and the tile's two 64-row column blocks are 8 KiB apart.
                            const uint32_t idesc16 = make_idesc(FMT == 2 ? 1u /*bf16*/ : 0u /*f16*/, 2 * BM, BN) |
                                                     (ep.a_mn ? kIdescAMnMajor : 0u) | (ep.b_mn ? kIdescBMnMajor : 0u);
                            const uint64_t a_d = ep.a_mn ? make_desc_mnmajor(sa, 8192, 1024, 2) : a_hi;
                            const uint64_t b_d = ep.b_mn ? make_desc_mnmajor(sa + Cfg::kABytes, 8192, 1024, 2) : b_hi;
                            const uint32_t a_adv = ep.a_mn ? 128u : 2u, b_adv = ep.b_mn ? 128u : 2u;
                            if (elect_one()) {
#pragma unroll
                                for (int kk = 0; kk < (int)KBE / 16; ++kk)
                                    mma_f16_pair(d_tmem, a_d + (uint64_t)(kk * a_adv), b_d + (uint64_t)(kk * b_adv), idesc16,
                                                 first | (uint32_t)kk);
                            }
                        } else if (FMT == 0) {
                            const uint64_t a_lo = make_desc_kmajor<BK * 4>(sa + BM * BK * 4);
                            const uint64_t b_lo = make_desc_kmajor<BK * 4>(sa + Cfg::kABytes + HB * BK * 4);
                            if (elect_one()) {
#pragma unroll
                                for (int kk = 0; kk < BK / UK; ++kk) {
                                    const uint64_t adv = (uint64_t)(kk * UK * 4 >> 4);
                                    mma_tf32_pair(d_tmem, a_lo + adv, b_hi + adv, idesc, first | (uint32_t)kk);
                                    mma_tf32_pair(d_tmem, a_hi + adv, b_lo + adv, idesc, 1u);
                                    mma_tf32_pair(d_tmem, a_hi + adv, b_hi + adv, idesc, 1u);
                                }
                            }
                        } else {
                            // Per operand: descriptors of the f32 tile and of its two bf16 planes, and how far
                            // one MMA's worth of k advances them (address field, 16-byte units).  K-major: 32 bytes
                            // inside the swizzled row.  MN-major: eight k-rows = 1024 bytes per tf32 MMA (two 512-byte
                            // atoms of the 32-byte-atomicity swizzle), sixteen k-rows = two 1024-byte atoms per bf16
                            // MMA; column blocks are 4 KiB (f32) / 8 KiB (bf16) apart.
                            const uint32_t idesc_t = idesc | (ep.a_mn ? kIdescAMnMajor : 0u) | (ep.b_mn ? kIdescBMnMajor : 0u);
                            const uint32_t idesc16 = make_idesc(1u /*bf16*/, 2 * BM, BN) | (ep.a_mn ? kIdescAMnMajor : 0u) |
                                                     (ep.b_mn ? kIdescBMnMajor : 0u);
                            const uint32_t a32 = sa, a16 = sa + BM * BK * 4;
                            const uint32_t b32 = sa + Cfg::kABytes, b16 = b32 + HB * BK * 4;
                            uint64_t a_f, a_h16, a_l16, b_f, b_h16, b_l16;
                            uint32_t a_adv32, a_adv16, b_adv32, b_adv16;
                            if (!ep.a_mn) {
                                a_f = make_desc_kmajor<128>(a32);
                                a_h16 = make_desc_kmajor<64>(a16); a_l16 = make_desc_kmajor<64>(a16 + BM * BK * 2);
                                a_adv32 = 2; a_adv16 = 2;
                            } else {
                                a_f = make_desc_mnmajor(a32, 4096, 512, 1);
                                a_h16 = make_desc_mnmajor(a16, 8192, 1024, 2); a_l16 = make_desc_mnmajor(a16 + 4096, 8192, 1024, 2);
                                a_adv32 = 64; a_adv16 = 128;
                            }
                            if (!ep.b_mn) {
                                b_f = make_desc_kmajor<128>(b32);
                                b_h16 = make_desc_kmajor<64>(b16); b_l16 = make_desc_kmajor<64>(b16 + HB * BK * 2);
                                b_adv32 = 2; b_adv16 = 2;
                            } else {
                                b_f = make_desc_mnmajor(b32, 4096, 512, 1);
                                b_h16 = make_desc_mnmajor(b16, 8192, 1024, 2); b_l16 = make_desc_mnmajor(b16 + 4096, 8192, 1024, 2);
                                b_adv32 = 64; b_adv16 = 128;
                            }
                            if (elect_one()) {
#pragma unroll
                                for (int kk = 0; kk < BK / 16; ++kk) {
                                    mma_f16_pair(d_tmem, a_l16 + (uint64_t)(kk * a_adv16), b_h16 + (uint64_t)(kk * b_adv16), idesc16,
                                                 first | (uint32_t)kk);
                                    mma_f16_pair(d_tmem, a_h16 + (uint64_t)(kk * a_adv16), b_l16 + (uint64_t)(kk * b_adv16), idesc16, 1u);
                                }
#pragma unroll
                                for (int kk = 0; kk < BK / UK; ++kk)
                                    mma_tf32_pair(d_tmem, a_f + (uint64_t)(kk * a_adv32), b_f + (uint64_t)(kk * b_adv32), idesc_t, 1u);
                            }
                        }
                        __syncwarp();
                        if (elect_one()) mma_commit_pair(empty_bar(s), 3);        // frees this stage in both CTAs
                        __syncwarp();
                    }
                    if (ok && elect_one()) mma_commit_pair(acc_full_bar(buf), 3);   // both CTAs may drain their half
                    __syncwarp();
                }
            }
            };
            issue(pa.ep[0], pair, units_of(pa.ep[0]).n, npairs);
            if constexpr (TWO) issue(pa.ep[1], run0, run1, 1);
#ifdef FG_GEMM_PROFILE
            if (lane == 0) {
            atomicAdd(&g_prof[0], (unsigned long long)prof_e);
            atomicAdd(&g_prof[1], (unsigned long long)prof_f);
            atomicAdd(&g_prof[2], (unsigned long long)(clock64() - prof_start));
            atomicAdd(&g_prof[7], 1ull);
            }
#endif
        }
    }
    } else {
        reg_acquire<kPairRegsHigh>();
        // ---- accumulate + epilogue (both CTAs, own 128 rows); see gemm_tc_kernel ----
        const int q = warp & 3;
        const int half = (warp - kPairEpiWarp0) >> 2;
        const uint32_t leader_acc_empty0 = map_to_cta(acc_empty_bar(0), 0);
        float4* tbuf = reinterpret_cast<float4*>(base_ptr + S * Cfg::kStageBytes + 256);   // 8 warps x 32 rows x 8 chunks
        float sum[CPT];
        bool ok = true;
        uint32_t gc = 0;
        long long prof_w = 0, prof_s = 0, prof_n = 0;
        (void)prof_w; (void)prof_s; (void)prof_n;
        auto drain = [&](const Epilogue& ep, uint32_t first, uint32_t end, uint32_t step) {
        const Units w = units_of(ep);
        const bool vec_ok = (ep.N % 4 == 0) && ((reinterpret_cast<uintptr_t>(ep.C) & 15u) == 0) &&
                            (!ep.preact || (reinterpret_cast<uintptr_t>(ep.preact) & 15u) == 0);
        for (uint32_t u = first; u < end && ok; u += step) {
            uint32_t tile, c0, c1, slot, m0, n0;
            const bool part = unit_at(ep, w, u, tile, c0, c1, slot);
            tile_origin(ep, w, tile, m0, n0);
#pragma unroll
            for (int j = 0; j < CPT; ++j) sum[j] = 0.0f;
            // Where this warp's part of the tile goes (a K-share of a tail tile goes out raw into its 256 x 256 slot).
            const uint32_t rsub = lane >> 3, cc = lane & 7;
            const uint32_t out_ld = part ? BN : ep.N, row_lim = part ? 2 * BM : ep.M, col_lim = part ? BN : ep.N;
            const uint32_t row0 = (part ? rank * BM : m0) + q * 32;            // first row of this warp's blocks
            const uint32_t col_base = (part ? 0u : n0) + half * CPT + cc * 4;  // this lane's 4 columns in block 0
            const bool vec = part || vec_ok;
            const float* const mul = part ? nullptr : ep.mul_saved;
            // The saved tensor of the layer below (dA epilogue), rows i*4 + rsub of block `blk`, read a whole block
            // ahead of its use through a rotating set of eight registers per lane: block 0 while the tile's last
            // accumulation chunk is still being computed, block b + 1 while block b is stored.  Read when needed,
            // or only a few rows ahead, each block waited for DRAM two to three times.
            const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
            auto saved_at = [&](int blk, int i) -> float4 {
                const uint32_t row = row0 + i * 4 + rsub, colb = col_base + blk * 32;
                return (mul && vec && blk < CPT / 32 && row < row_lim && colb + 3 < col_lim)
                           ? __ldg(reinterpret_cast<const float4*>(mul + (size_t)row * out_ld + colb)) : zero4;
            };
            float4 s0 = zero4, s1 = zero4, s2 = zero4, s3 = zero4, s4 = zero4, s5 = zero4, s6 = zero4, s7 = zero4;
            for (uint32_t c = c0; c < c1; ++c, ++gc) {
                const uint32_t buf = gc & 1u;
                if (c + 1 == c1 && mul) {
                    s0 = saved_at(0, 0); s1 = saved_at(0, 1); s2 = saved_at(0, 2); s3 = saved_at(0, 3);
                    s4 = saved_at(0, 4); s5 = saved_at(0, 5); s6 = saved_at(0, 6); s7 = saved_at(0, 7);
                }
                PROF_T0();
                bool got = mbar_wait_bounded(acc_full_bar(buf), (gc >> 1) & 1u, kPairWaitCycles + kPairWaitCycles / 2);
                PROF_ADD(prof_w);
                got = __all_sync(0xffffffffu, got);
                if (!got) {
                    if (lane == 0) atomicOr(dev_status, FG_DEVERR_EPI_WAIT);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN + half * CPT;
#pragma unroll
                for (int g4 = 0; g4 < CPT / 32; ++g4) {
                    uint32_t r[32];
                    tmem_ld_32x32(t0 + g4 * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[g4 * 32 + j] += __uint_as_float(r[j]);
                }
                tc_fence_before();
                if (lane == 0) mbar_arrive_cluster(leader_acc_empty0 + 8u * buf);   // 16 warps report to the leader
            }
            if (!ok) break;
#ifdef FG_GEMM_PROFILE
            const long long prof_st = clock64();
#endif
            // Store this tile from registers; the tensor core is already working on the next one.  A thread
            // owns one row, so storing directly would touch 32 different lines per instruction; instead each
            // warp passes 32x32 blocks through a padded shared-memory buffer and writes 4 rows x 128 bytes
            // per instruction (bias and activation are applied on the way out).
            // A K-share of a tail tile goes out raw (no bias, no activation) into its 256x256 slot.
            // The 32 x 32 staging block of this warp: rows of eight 16-byte chunks, chunk c of row r at position
            // c ^ (r & 7), so that both the row-wise writes (a lane owns a row) and the reads (eight lanes sweep a
            // row) are 128-bit accesses without bank conflicts.  A K-share of a tail tile goes out raw (no bias, no
            // activation, no extras: the fold kernel does those) into its 256 x 256 slot.
            // Nothing below may touch local memory: no calls, no dynamically indexed arrays, no spills.
            float4* tb4 = tbuf + (warp - kPairEpiWarp0) * (32 * 8);
            char* const out = part ? (char*)(ep.partial + (size_t)slot * (2 * BM * BN)) : (char*)ep.C;
            char* const pre = part ? nullptr : (char*)ep.preact;
            const int odt = (part || !kDirect16) ? (int)FG_DTYPE_F32 : ep.out_dtype;   // the f32 kernels store f32 only
            const int act = part ? FG_ACT_NONE : ep.act;
            __nv_bfloat16* const pairs = part ? nullptr : ep.c_pairs;
            float* const csp = part ? nullptr : ep.colsum_part;
#ifdef FG_GEMM_PROFILE
            const bool no_store = (ep.dbg & 1u) != 0;
#else
            constexpr bool no_store = false;
#endif
#pragma unroll
            for (int g4 = 0; g4 < CPT / 32; ++g4) {
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    tb4[lane * 8 + (c ^ (lane & 7))] = make_float4(sum[g4 * 32 + 4 * c], sum[g4 * 32 + 4 * c + 1],
                                                                   sum[g4 * 32 + 4 * c + 2], sum[g4 * 32 + 4 * c + 3]);
                __syncwarp();
                const uint32_t col = col_base + g4 * 32;
                const bool fast = vec && col + 3 < col_lim;                    // the whole float4 is inside the matrix
                float4 bz = make_float4(0.f, 0.f, 0.f, 0.f);
                if (ep.bias && !part) {
                    if (kDirect16) {
                        if (col < col_lim) bz.x = epi_bias(ep.bias, col, ep.out_dtype);
                        if (col + 1 < col_lim) bz.y = epi_bias(ep.bias, col + 1, ep.out_dtype);
                        if (col + 2 < col_lim) bz.z = epi_bias(ep.bias, col + 2, ep.out_dtype);
                        if (col + 3 < col_lim) bz.w = epi_bias(ep.bias, col + 3, ep.out_dtype);
                    } else if (col + 3 < col_lim && (reinterpret_cast<uintptr_t>(ep.bias) & 15u) == 0) {
                        bz = __ldg(reinterpret_cast<const float4*>(ep.bias + col));
                    } else {      // the last columns, or a bias that starts off 16 bytes
                        if (col < col_lim) bz.x = ep.bias[col];
                        if (col + 1 < col_lim) bz.y = ep.bias[col + 1];
                        if (col + 2 < col_lim) bz.z = ep.bias[col + 2];
                        if (col + 3 < col_lim) bz.w = ep.bias[col + 3];
                    }
                }
                float4 cs = make_float4(0.f, 0.f, 0.f, 0.f);     // column sums of what this lane stores (rows i*4 + rsub)
                // Rows i*4 + rsub, i = 0..7, one per iteration of a rolled loop (one copy of the activation code per
                // block).  Each iteration takes its row of the saved tensor from the front of the rotating set and
                // refills the back with the same row of the NEXT block.  The staged values come through a rotating
                // set too: the tensor core reads its operands from shared memory at most of the memory's bandwidth,
                // and a shared-memory load issued when its value is needed waits behind that traffic.
                auto staged_row = [&](int i) -> float4 {
                    const uint32_t lr = (uint32_t)(i & 7) * 4 + rsub;
                    return tb4[lr * 8 + (cc ^ (lr & 7))];
                };
                float4 z0 = staged_row(0), z1 = staged_row(1), z2 = staged_row(2), z3 = staged_row(3);
#pragma unroll 1
                for (int i = 0; i < 8; ++i) {
                    const float4 sv = s0;
                    s0 = s1; s1 = s2; s2 = s3; s3 = s4; s4 = s5; s5 = s6; s6 = s7;
                    s7 = saved_at(g4 + 1, i);
                    float4 zin = z0;
                    z0 = z1; z1 = z2; z2 = z3; z3 = staged_row(i + 4);
                    const uint32_t lr = i * 4 + rsub;
                    const uint32_t row = row0 + lr;
                    zin.x += bz.x; zin.y += bz.y; zin.z += bz.z; zin.w += bz.w;
                    if (row < row_lim && col < col_lim) {
                        const size_t off = (size_t)row * out_ld + col;
                        if (fast) {
                            float4 o;
                            if (mul) {
                                o = make_float4(zin.x * fg_act_grad_sel(ep.mul_act, sv.x), zin.y * fg_act_grad_sel(ep.mul_act, sv.y),
                                                zin.z * fg_act_grad_sel(ep.mul_act, sv.z), zin.w * fg_act_grad_sel(ep.mul_act, sv.w));
                            } else if (act != FG_ACT_NONE) {
                                o = make_float4(fg_act_fwd_sel(act, zin.x), fg_act_fwd_sel(act, zin.y), fg_act_fwd_sel(act, zin.z),
                                                fg_act_fwd_sel(act, zin.w));
                            } else o = zin;
                            if (!no_store) {
                                if (pre) store_out4(pre, off, zin, odt);
                                store_out4(out, off, o, odt);
                                if (pairs) fg_store_pairs4(pairs, ep.c_pairs_stride, off, o);
                            }
                            cs.x += o.x; cs.y += o.y; cs.z += o.z; cs.w += o.w;
                        } else {
                            const float4 o = epi_store_edge(zin, off, col, col_lim, out, pre, pairs, ep.c_pairs_stride, mul, ep.mul_act, act, odt);
                            cs.x += o.x; cs.y += o.y; cs.z += o.z; cs.w += o.w;
                        }
                    }
                }
                if (csp) {
                    // the four lanes that share these columns hold rows 0,4,.. / 1,5,.. / 2,6,.. / 3,7,..: add them in a fixed order
                    cs.x += __shfl_xor_sync(0xffffffffu, cs.x, 8); cs.x += __shfl_xor_sync(0xffffffffu, cs.x, 16);
                    cs.y += __shfl_xor_sync(0xffffffffu, cs.y, 8); cs.y += __shfl_xor_sync(0xffffffffu, cs.y, 16);
                    cs.z += __shfl_xor_sync(0xffffffffu, cs.z, 8); cs.z += __shfl_xor_sync(0xffffffffu, cs.z, 16);
                    cs.w += __shfl_xor_sync(0xffffffffu, cs.w, 8); cs.w += __shfl_xor_sync(0xffffffffu, cs.w, 16);
                    if (lane < 8 && row0 < row_lim) {
                        float* d = csp + (size_t)(row0 >> 5) * ep.N + col;
                        if (col < col_lim) d[0] = cs.x;
                        if (col + 1 < col_lim) d[1] = cs.y;
                        if (col + 2 < col_lim) d[2] = cs.z;
                        if (col + 3 < col_lim) d[3] = cs.w;
                    }
                }
                __syncwarp();
            }
#ifdef FG_GEMM_PROFILE
            prof_s += clock64() - prof_st;
            prof_n += 1;
#endif
        }
        };
        drain(pa.ep[0], pair, units_of(pa.ep[0]).n, npairs);
        if constexpr (TWO) drain(pa.ep[1], run0, run1, 1);
#ifdef FG_GEMM_PROFILE
        if (warp == kPairEpiWarp0 && lane == 0 && leader) {
            atomicAdd(&g_prof[3], (unsigned long long)prof_w);
            atomicAdd(&g_prof[4], (unsigned long long)prof_s);
            atomicAdd(&g_prof[5], (unsigned long long)prof_n);
        }
#endif
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();      // neither CTA retires while the peer may still read its shared memory
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
    }
}

// Folds the pair kernel's K-shares of a 256 x 256 tile in a fixed order, then does what its own epilogue does for a whole
// tile: bias, activation (or the act' factor), store, bf16 pairs, column sums.
// A block of 256 threads per 32 x 32 sub-block (so that a block owns whole 32-row column sums); thread t handles four
// consecutive columns of row t / 8.
__global__ void __launch_bounds__(256) gemm_tc_fold_kernel(Epilogue ep) {
    fg_grid_enter();
    __shared__ float cs_sm[8][32];
    constexpr uint32_t TM = 2 * BM, TN = 256;
    constexpr uint32_t kSubN = TN / 32, kSubs = (TM / 32) * kSubN;
    const uint32_t pairs_m = (ep.M + TM - 1) / TM, pairs_n = (ep.N + TN - 1) / TN;
    const uint32_t tail = blockIdx.x / kSubs, sub = blockIdx.x % kSubs;
    uint32_t m0, n0;
    pair_tile_origin(ep.t_full + tail, pairs_m, pairs_n, TM, TN, ep.group, m0, n0);
    const uint32_t lrow = (sub / kSubN) * 32 + (threadIdx.x >> 3), lcol = (sub % kSubN) * 32 + (threadIdx.x & 7u) * 4;
    const uint32_t row = m0 + lrow, col = n0 + lcol;
    const bool live = row < ep.M && col < ep.N;
    float ov[4] = {0.f, 0.f, 0.f, 0.f};
    if (live) {
        const float* p = ep.partial + (size_t)tail * ep.split * (TM * TN) + (size_t)lrow * TN + lcol;
        float4 z = *reinterpret_cast<const float4*>(p);
        for (uint32_t k = 1; k < ep.split; ++k) {
            const float4 t = *reinterpret_cast<const float4*>(p + (size_t)k * (TM * TN));
            z.x += t.x; z.y += t.y; z.z += t.z; z.w += t.w;
        }
        float zz[4] = {z.x, z.y, z.z, z.w};
        if (ep.bias) {
#pragma unroll
            for (int t = 0; t < 4; ++t) if (col + t < ep.N) zz[t] += epi_bias(ep.bias, col + t, ep.out_dtype);
        }
        const size_t off = (size_t)row * ep.N + col;
        const bool vec_ok = (ep.N % 4 == 0) && ((reinterpret_cast<uintptr_t>(ep.C) & 15u) == 0) &&
                            (!ep.preact || (reinterpret_cast<uintptr_t>(ep.preact) & 15u) == 0) &&
                            (!ep.mul_saved || (reinterpret_cast<uintptr_t>(ep.mul_saved) & 15u) == 0);
        if (vec_ok && col + 3 < ep.N) {
            const float4 zin = make_float4(zz[0], zz[1], zz[2], zz[3]);
            float4 o;
            if (ep.mul_saved) o = act_mul4(ep.mul_act, zin, __ldg(reinterpret_cast<const float4*>(ep.mul_saved + off)));
            else o = ep.act == FG_ACT_NONE ? zin : act_fwd4(ep.act, zin);
            if (ep.preact) store_out4(ep.preact, off, zin, ep.out_dtype);
            store_out4(ep.C, off, o, ep.out_dtype);
            if (ep.c_pairs) fg_store_pairs4(ep.c_pairs, ep.c_pairs_stride, off, o);
            ov[0] = o.x; ov[1] = o.y; ov[2] = o.z; ov[3] = o.w;
        } else {
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (col + t < ep.N) {
                    const float o = ep.mul_saved ? zz[t] * fg_act_grad_fast(ep.mul_act, ep.mul_saved[off + t]) : fg_act_fwd_fast(ep.act, zz[t]);
                    if (ep.preact) store_out1(ep.preact, off + t, zz[t], ep.out_dtype);
                    store_out1(ep.C, off + t, o, ep.out_dtype);
                    if (ep.c_pairs) fg_store_pairs1(ep.c_pairs, ep.c_pairs_stride, off + t, o);
                    ov[t] = o;
                }
        }
    }
    if (!ep.colsum_part) return;
    // column sums over this block's 32 rows: four rows inside each warp, then the eight warps in order
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        ov[t] += __shfl_xor_sync(0xffffffffu, ov[t], 8);
        ov[t] += __shfl_xor_sync(0xffffffffu, ov[t], 16);
    }
    if (lane < 8) {
#pragma unroll
        for (int t = 0; t < 4; ++t) cs_sm[warp][lane * 4 + t] = ov[t];
    }
    __syncthreads();
    const uint32_t row0 = m0 + (sub / kSubN) * 32, c = n0 + (sub % kSubN) * 32 + threadIdx.x;
    if (threadIdx.x < 32 && row0 < ep.M && c < ep.N) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += cs_sm[w][threadIdx.x];
        ep.colsum_part[(size_t)(row0 >> 5) * ep.N + c] = t;
    }
}

// ------------------------------------------------------------------------------------
// Pre-pass: operand planes of X [R, C] (row-major), optionally of dY * act'(saved).
// Orientation n keeps X's layout (contraction index = column): rows R, pitch ld*.
// Orientation t is transposed (contraction index = row): rows C.
// Plane formats (FMT):
//   0  p32 = [2][rows][ld32] f32: hi = tf32(x), lo = tf32(x - hi)
//   1  p32 = [rows][ld32] f32: hi;  p16 = [2][rows][ld16] bf16: bf16(x), bf16(x - hi)
// ------------------------------------------------------------------------------------
struct PlaneSet {
    float* p32;
    __nv_bfloat16* p16;
    uint32_t ld32, ld16;
    uint64_t plane16;      // elements between the two bf16 planes (0: rows * ld16, planes back to back)
    bool mn;               // storage is [contraction][rows] (rows contiguous): the f32 tensor itself with its pairs
    uint64_t batch32;      // elements between two matrices of a batch (0: rows * ld32 of the storage)
};

struct SplitArgs {
    const float* x;
    const float* saved;    // non-NULL: value = x * act'(saved)
    int act;
    uint32_t R, C;
    PlaneSet n, t;         // p32 == NULL: orientation not wanted
    float* value_out;      // optional copy of the (fused) value, [R, C]
    float* colsum_part;    // optional [gridDim.y][C]: column sums of the value over each tile's rows (bias gradient)
};

template <int FMT>
__device__ __forceinline__ void store_planes(const PlaneSet& ps, size_t rows, size_t r, size_t c, float hi, float lo,
                                             float v) {
    ps.p32[r * ps.ld32 + c] = hi;
    if (FMT == 0) {
        ps.p32[rows * ps.ld32 + r * ps.ld32 + c] = lo;
    } else {
        ps.p16[r * ps.ld16 + c] = __float2bfloat16_rn(v);
        ps.p16[rows * ps.ld16 + r * ps.ld16 + c] = __float2bfloat16_rn(lo);
    }
}

// Any shape and alignment: 32x32 tiles, 32x8 threads, scalar accesses.
template <int FMT>
__global__ void __launch_bounds__(256) split_kernel(SplitArgs a) {
    __shared__ float tv[32][33];
    __shared__ float cs[8][33];
    const uint32_t c = blockIdx.x * 32 + threadIdx.x;
    const uint32_t r0 = blockIdx.y * 32;
    float csum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t r = r0 + threadIdx.y + i * 8;
        float v = 0.0f;
        if (r < a.R && c < a.C) {
            const size_t idx = (size_t)r * a.C + c;
            v = a.x[idx];
            if (a.saved) v = v * fg_act_grad(a.act, a.saved[idx]);
            if (a.value_out) a.value_out[idx] = v;
            if (a.n.p32) {
                const float hi = __uint_as_float(cvt_tf32(v));
                const float lo = v - hi;
                store_planes<FMT>(a.n, a.R, r, c, hi, FMT == 0 ? __uint_as_float(cvt_tf32(lo)) : lo, v);
            }
        }
        tv[threadIdx.y + i * 8][threadIdx.x] = v;
        csum += v;
    }
    if (a.colsum_part) cs[threadIdx.y][threadIdx.x] = csum;
    if (!a.t.p32 && !a.colsum_part) return;
    __syncthreads();
    if (a.colsum_part && threadIdx.y == 0 && c < a.C) {
        float t = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += cs[k][threadIdx.x];
        a.colsum_part[(size_t)blockIdx.y * a.C + c] = t;
    }
    if (!a.t.p32) return;
    const uint32_t tr = r0 + threadIdx.x;          // source row -> destination column
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t tc = blockIdx.x * 32 + threadIdx.y + i * 8;   // source column -> destination row
        if (tc < a.C && tr < a.R) {
            const float v = tv[threadIdx.x][threadIdx.y + i * 8];
            const float hi = __uint_as_float(cvt_tf32(v));
            const float lo = v - hi;
            store_planes<FMT>(a.t, a.C, tc, tr, hi, FMT == 0 ? __uint_as_float(cvt_tf32(lo)) : lo, v);
        }
    }
}

struct Split4 {
    float4 hi, lo;
};
template <int FMT>
__device__ __forceinline__ Split4 split4(float4 v) {
    Split4 o;
    o.hi = make_float4(__uint_as_float(cvt_tf32(v.x)), __uint_as_float(cvt_tf32(v.y)),
                       __uint_as_float(cvt_tf32(v.z)), __uint_as_float(cvt_tf32(v.w)));
    o.lo = make_float4(v.x - o.hi.x, v.y - o.hi.y, v.z - o.hi.z, v.w - o.hi.w);
    if (FMT == 0)
        o.lo = make_float4(__uint_as_float(cvt_tf32(o.lo.x)), __uint_as_float(cvt_tf32(o.lo.y)),
                           __uint_as_float(cvt_tf32(o.lo.z)), __uint_as_float(cvt_tf32(o.lo.w)));
    return o;
}
__device__ __forceinline__ uint2 pack_bf16x4(float4 v) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    uint2 u;
    u.x = *reinterpret_cast<uint32_t*>(&a);
    u.y = *reinterpret_cast<uint32_t*>(&b);
    return u;
}
// Four consecutive elements of one plane row (c a multiple of 4, pitches multiples of 4 / 8).
template <int FMT>
__device__ __forceinline__ void store_planes4(const PlaneSet& ps, size_t rows, size_t r, size_t c, float4 v) {
    const Split4 s = split4<FMT>(v);
    *reinterpret_cast<float4*>(ps.p32 + r * ps.ld32 + c) = s.hi;
    if (FMT == 0) {
        *reinterpret_cast<float4*>(ps.p32 + rows * ps.ld32 + r * ps.ld32 + c) = s.lo;
    } else {
        *reinterpret_cast<uint2*>(ps.p16 + r * ps.ld16 + c) = pack_bf16x4(v);
        *reinterpret_cast<uint2*>(ps.p16 + rows * ps.ld16 + r * ps.ld16 + c) = pack_bf16x4(s.lo);
    }
}

// 128-bit accesses, for R % 4 == 0 and C % 4 == 0 (every group of four is wholly inside or outside)
// and 16-byte aligned pointers.  64x64 tiles, 256 threads: thread t handles column group t%16
// (4 columns) of rows t/16 + 16*i, then writes 4 consecutive source rows of source column t/16 + 16*i.
template <int FMT>
__global__ void __launch_bounds__(256) split_vec_kernel(SplitArgs a) {
    __shared__ float tv[64][65];
    __shared__ float cs[16][64];
    const uint32_t cg = threadIdx.x & 15, rl = threadIdx.x >> 4;
    const uint32_t c = blockIdx.x * 64 + cg * 4;
    const uint32_t r0 = blockIdx.y * 64;
    const bool want_t = a.t.p32 != nullptr;
    float4 csum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t lr = rl + 16 * i, r = r0 + lr;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < a.R && c < a.C) {
            const size_t idx = (size_t)r * a.C + c;
            v = __ldcs(reinterpret_cast<const float4*>(a.x + idx));
            if (a.saved) {
                const float4 s = __ldcs(reinterpret_cast<const float4*>(a.saved + idx));
                v.x *= fg_act_grad(a.act, s.x); v.y *= fg_act_grad(a.act, s.y);
                v.z *= fg_act_grad(a.act, s.z); v.w *= fg_act_grad(a.act, s.w);
            }
            if (a.value_out) *reinterpret_cast<float4*>(a.value_out + idx) = v;
            if (a.n.p32) store_planes4<FMT>(a.n, a.R, r, c, v);
        }
        if (want_t) {
            tv[lr][cg * 4 + 0] = v.x; tv[lr][cg * 4 + 1] = v.y; tv[lr][cg * 4 + 2] = v.z; tv[lr][cg * 4 + 3] = v.w;
        }
        csum.x += v.x; csum.y += v.y; csum.z += v.z; csum.w += v.w;
    }
    if (a.colsum_part) {
        cs[rl][cg * 4 + 0] = csum.x; cs[rl][cg * 4 + 1] = csum.y; cs[rl][cg * 4 + 2] = csum.z; cs[rl][cg * 4 + 3] = csum.w;
    }
    if (!want_t && !a.colsum_part) return;
    __syncthreads();
    if (a.colsum_part && threadIdx.x < 64 && blockIdx.x * 64 + threadIdx.x < a.C) {
        float t = 0.0f;
#pragma unroll
        for (int k = 0; k < 16; ++k) t += cs[k][threadIdx.x];
        a.colsum_part[(size_t)blockIdx.y * a.C + blockIdx.x * 64 + threadIdx.x] = t;
    }
    if (!want_t) return;
    const uint32_t tr = r0 + cg * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t lc = rl + 16 * i, tc = blockIdx.x * 64 + lc;
        if (tc < a.C && tr < a.R)
            store_planes4<FMT>(a.t, a.C, tc, tr,
                               make_float4(tv[cg * 4 + 0][lc], tv[cg * 4 + 1][lc], tv[cg * 4 + 2][lc], tv[cg * 4 + 3][lc]));
    }
}

// ------------------------------------------------------------------------------------
// One pass over a dense [R, C] tensor of any storage type, for what cannot be read in place: a copy with a padded pitch
// (a bulk-tensor load wants 16-byte row pitches), dZ = dY * act'(saved), and the column sums of the value over each 32 rows
// (the bias gradient's partials).  grid.z is the matrix of a batch.
// ------------------------------------------------------------------------------------
struct PrepArgs {
    const void* x;
    const void* saved;    // non-NULL: value = x * act'(saved), rounded to the storage type
    int act;
    uint32_t R, C;
    uint64_t x_batch;     // elements between two matrices of x and saved
    void* out;            // [R][ld] per matrix, matrices R * ld apart, or NULL
    uint32_t ld;
    void* copy;           // optional second copy, dense, matrices R * C apart
    float* colsum_part;   // [ceil(R/32)][C] f32 or NULL (one matrix)
};

template <typename T> __device__ __forceinline__ float lp_to_float(T v);
template <> __device__ __forceinline__ float lp_to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float lp_to_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float lp_to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T lp_from_float(float v);
template <> __device__ __forceinline__ float lp_from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __half lp_from_float<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 lp_from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// 32 rows x 32 * W columns per block, W columns per thread: 16 bytes of them, or, for any shape and alignment, one in 32.  All loads
// first, and column sums that lie 36 words apart: with eight apart and two blocks an SM, dZ of 2048 x 4096 bf16 through GELU took 20 -
// 30 us for 50 MB.  Blocks an SM by registers: three of bf16, four of f16, five of f32 (asked for three, the compiler took 40 registers
// for f32 and spilled: dB and bias gradient of 9216 x 4096 x 8 93 us, 85 with five; f16 4096 x 4096 x 64 23.8 with three, 21.0 with four).
constexpr int kPrepPitch = 36;
template <typename T, int W, bool VEC>
__device__ __forceinline__ void prep_block(const PrepArgs& a, uint32_t bx, uint32_t by, uint32_t bz, float* cs) {
    const uint32_t x0 = bx * 32 * W, c = VEC ? x0 + threadIdx.x * W : x0 + threadIdx.x, r0 = by * 32 + threadIdx.y;
    struct __align__(VEC ? W * sizeof(T) : sizeof(T)) Vec { T e[W]; };
    const T* const x = static_cast<const T*>(a.x) + bz * a.x_batch;
    const T* const saved = a.saved ? static_cast<const T*>(a.saved) + bz * a.x_batch : nullptr;
    T* const out = a.out ? static_cast<T*>(a.out) + (size_t)bz * a.R * a.ld : nullptr;
    T* const copy = a.copy ? static_cast<T*>(a.copy) + (size_t)bz * a.R * a.C : nullptr;
    auto load = [&](const T* p, uint32_t r, Vec& v) {
        p += (size_t)r * a.C + c;
        if constexpr (VEC) v = *reinterpret_cast<const Vec*>(p);
        else
#pragma unroll
            for (int w = 0; w < W; ++w)
                if (c + 32 * w < a.C) v.e[w] = p[32 * w];
    };
    auto store = [&](T* p, uint32_t r, uint32_t ld, const Vec& v) {
        p += (size_t)r * ld + c;
        if constexpr (VEC) *reinterpret_cast<Vec*>(p) = v;
        else
#pragma unroll
            for (int w = 0; w < W; ++w)
                if (c + 32 * w < a.C) p[32 * w] = v.e[w];
    };
    float sum[W];
#pragma unroll
    for (int w = 0; w < W; ++w) sum[w] = 0.0f;
    if (c < a.C) {
        Vec v[4], sv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (r0 + 8 * k < a.R) {
                load(x, r0 + 8 * k, v[k]);
                if (saved) load(saved, r0 + 8 * k, sv[k]);
            }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t r = r0 + 8 * k;
            if (r >= a.R) continue;
            if (saved) {
                // (the activation is chosen for a row: between choices the W elements' chains run side by side)
                auto factor = [&](auto act) {
#pragma unroll
                    for (int w = 0; w < W; ++w) v[k].e[w] = lp_from_float<T>(lp_to_float(v[k].e[w]) * fg_act_grad(decltype(act)::value, lp_to_float(sv[k].e[w])));
                };
                if (a.act == FG_ACT_GELU) factor(std::integral_constant<int, FG_ACT_GELU>{});
                else if (a.act == FG_ACT_TANH) factor(std::integral_constant<int, FG_ACT_TANH>{});
                else if (a.act == FG_ACT_RELU) factor(std::integral_constant<int, FG_ACT_RELU>{});
            }
            if (out) store(out, r, a.ld, v[k]);
            if (copy) store(copy, r, a.C, v[k]);
#pragma unroll
            for (int w = 0; w < W; ++w) sum[w] += lp_to_float(v[k].e[w]);
        }
    }
    if (!a.colsum_part) return;
#pragma unroll
    for (int w = 0; w < W; ++w) cs[(threadIdx.y * W + w) * kPrepPitch + threadIdx.x] = sum[w];
    __syncthreads();
    const uint32_t t = threadIdx.y * 32 + threadIdx.x, col = x0 + t;
    if (t < 32 * W && col < a.C) {
        float z = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) z += cs[(k * W + (VEC ? t % W : t / 32)) * kPrepPitch + (VEC ? t / W : t % 32)];
        a.colsum_part[(size_t)by * a.C + col] = z;
    }
}

// Up to three passes in a launch, one after the other in the grid: what a product or a backward pass needs beforehand are short,
// independent passes (a ragged layer's dZ and copies of its input and weights, 3.5 - 5 us each: backward of 1000 x 777 x 1001
// 40.9 -> 38 - 39 us).
struct PrepJobs {
    PrepArgs job[3];
    uint32_t width[3], gx[3], gy[3], first[4];      // columns per thread (0: 16 bytes of them); blocks across and down a matrix; the first block of each
};
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 5 : std::is_same_v<T, __half> ? 4 : 3) prep_kernel(const __grid_constant__ PrepJobs p) {
    fg_grid_enter();
    constexpr int W = 16 / sizeof(T);
    __shared__ float room[8 * W * kPrepPitch];
    const uint32_t j = blockIdx.x >= p.first[2] ? 2u : blockIdx.x >= p.first[1] ? 1u : 0u, b = blockIdx.x - p.first[j];
    const uint32_t bx = b % p.gx[j], r = b / p.gx[j], by = r % p.gy[j], bz = r / p.gy[j];
    if (p.width[j] == 0) prep_block<T, W, true>(p.job[j], bx, by, bz, room);
    else if (p.width[j] == 4) prep_block<T, 4, false>(p.job[j], bx, by, bz, room);
    else prep_block<T, 2, false>(p.job[j], bx, by, bz, room);
}

// Passes that have been asked for and not been launched.
struct PrepBatch {
    PrepJobs jobs{};
    int n = 0, dtype = FG_DTYPE_F32;
    double bytes = 0.0;

    // a.out, when given, is scratch: 16-byte aligned with a 16-byte pitch.
    int32_t add(fg_ctx* ctx, int type, const PrepArgs& a, uint32_t batch = 1) {
        if (n == 3 || (n && type != dtype)) {
            const int32_t s = launch(ctx);
            if (s != FG_OK) return s;
        }
        dtype = type;
        const uint32_t per16 = dtype == FG_DTYPE_F32 ? 4 : 8;
        const bool vec = a.C % per16 == 0 && (batch == 1 || a.x_batch % per16 == 0) && fg_aligned16(a.x) && (!a.saved || fg_aligned16(a.saved)) &&
                         (!a.copy || fg_aligned16(a.copy));
        // four columns a thread where that still makes two blocks an SM (backward of 1000 x 777 x 1001 37.8 us, 39.5 with two)
        const uint32_t wide = (uint64_t)((a.C + 127) / 128) * ((a.R + 31) / 32) * batch >= 2ull * (uint64_t)ctx->sm_count ? 4 : 2;
        const uint32_t w = 32 * (vec ? per16 : wide), gx = (a.C + w - 1) / w, gy = (a.R + 31) / 32;
        const uint64_t end = jobs.first[n] + (uint64_t)gx * gy * batch;
        if (gy > 65535 || batch > 65535 || end > 0x7fffffffull) return fg_fail(ctx, FG_ERR_INVALID_ARGUMENT, "GEMM operand has too many rows");
        jobs.job[n] = a;
        jobs.width[n] = vec ? 0 : wide; jobs.gx[n] = gx; jobs.gy[n] = gy;
        for (int k = ++n; k < 4; ++k) jobs.first[k] = (uint32_t)end;
        bytes += (dtype == FG_DTYPE_F32 ? 4.0 : 2.0) * batch * a.R * a.C * (1.0 + (a.saved ? 1.0 : 0.0) + (a.out ? 1.0 : 0.0) + (a.copy ? 1.0 : 0.0));
        return FG_OK;
    }
    int32_t launch(fg_ctx* ctx) {
        if (!n) return FG_OK;
        const dim3 block(32, 8);
        fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SPLIT, bytes);
        if (dtype == FG_DTYPE_F32) fg_launch(ctx, prep_kernel<float>, jobs.first[n], block, 0, jobs);
        else if (dtype == FG_DTYPE_F16) fg_launch(ctx, prep_kernel<__half>, jobs.first[n], block, 0, jobs);
        else fg_launch(ctx, prep_kernel<__nv_bfloat16>, jobs.first[n], block, 0, jobs);
        fg_time_end(ctx, tr);
        n = 0;
        bytes = 0.0;
        jobs.first[0] = 0;
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
};

// ------------------------------------------------------------------------------------
// Conversion kernel: small and middling products of f32 tensors, straight from the tensors.
// The pair kernel needs bf16 pairs in HBM and works in 256 x 256 tiles on two SMs; a product of a
// few such tiles leaves most SMs idle, and making the pairs of a tensor that is read once costs
// as much as reading it twice more.  Here a CTA owns a 128 x BN tile, loads the raw f32 words of
// both operands (half the bytes of tensor plus pairs) and converter warps split each k-block: A into
// tensor memory, from where the MMAs read it, B's bf16 planes beside its words in shared memory, in the
// layout a bulk-tensor load would have given them.  A matrix index rides in the unit number and a K-share in
// the cluster, so that one launch covers a batch, or both gradients of a layer, and fills the SMs.
//   warp 0 loads, warp 1 issues MMAs, warps 4..11 drain accumulators and store, warps 12..27 convert.
// Measured (start: operand planes or pairs, then a 256 x 256 or 128-row tile each; then with A in shared memory, eight converter
// warps, K-shares folded by a second launch and one launch per product; now): 100 x 4096 x 4096 129 -> 35 -> 30 us,
// 16 x (384 x 512 x 320) forward and backward 1530 -> 86 -> 48 us, the 200-256-256-10 step 195 -> 91 -> 70 us.
// Bound by shared-memory bandwidth: per k-block of 32 a 128 x 128 tile moves 32 KB in by TMA, 32 KB into the converters, 32 KB
// out of them (B) and 32 KB into the MMAs (B): 1024 cycles at 128 B per cycle, 1040 measured (128 x 64: 640, 590 - 630 measured).
// ------------------------------------------------------------------------------------
template <int BN>
struct ConvCfg {
    static constexpr int kA32 = BM * 32 * 4, kB32 = BN * 32 * 4;    // f32 tiles; B's two bf16 planes take as much again
    static constexpr int kStageBytes = kA32 + 2 * kB32;
    static constexpr int kStages = BN == 128 ? 4 : 6;
    static constexpr int kACols = 64;                               // tensor memory per stage: A as f32 and as two bf16 planes
    // Converters: groups of warps that take the k-blocks in turn, see the kernel.
    static constexpr int kGroups = 2, kGroup = 256;
    static constexpr int kEpi0 = 4, kConv0 = 12;                    // first epilogue and first converter warp
    static constexpr int kThreads = kConv0 * 32 + kGroups * kGroup;
    // registers after the split between the warpgroups (72 each at launch): loads and MMAs, epilogue, converters
    static constexpr int kRegsLow = 40, kRegsEpi = 104, kRegsConv = 64;
    static_assert(kThreads == 896 && 128 * kRegsLow + 256 * kRegsEpi + 512 * kRegsConv <= 896 * 72, "the launch's registers");
    static constexpr int kStoreBytes = 8 * 32 * 32 * 4;             // the epilogue warps' staging blocks
    static constexpr int kSmemBytes = kStages * kStageBytes + kStoreBytes + 1024 + 256;
    static_assert(kSmemBytes <= 232448, "exceeds the 227 KB a CTA may use");
    static_assert(kStages * kStageBytes >= BM * BN * 4, "a K-share's sums lie in the stages");
    static constexpr int kTmemCols = 512;
    static_assert(2 * BN + kStages * kACols <= kTmemCols, "two accumulators and the stages of A");
};

// The split of a tile of ROWS rows x 32 k, eight elements per thread and step: the words are rounded to tf32
// in place (hi; an MMA would truncate them, which doubles what the cross terms have to carry: 1.9e-6 against 1.5e-6 of the
// result's 2-norm), the planes are bf16(x) and bf16(x - hi).
// K-major f32: rows of 128 bytes, 16-byte chunk c of row r at c ^ (r & 7); bf16: planes of [ROWS][64 bytes], chunk c of row
// r at c ^ (r / 2 & 3).  MN-major f32: blocks of 32 rows, [k][128 bytes] each, 32-byte chunk j of k-row k at j ^ (k & 3);
// bf16: blocks of 64 rows, [plane][k][128 bytes] each, 16-byte chunk c of k-row k at c ^ (k & 7).
// Lanes are dealt so that the 128-bit accesses of eight lanes fall into different banks.
// Nearest tf32 value, ties away from zero (cvt.rna), in two integer operations: the conversion unit is a fraction as wide.
// A NaN may lose its payload here; the planes keep the product NaN.  Values from 0x7f7ff000 on round to infinity; products of
// values from 0x7f7f8000 on are not finite in any format with bf16 planes, because bf16(x) is not.
__device__ __forceinline__ float4 round_tf32(float4 v) {
    auto r = [](float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); };
    return make_float4(r(v.x), r(v.y), r(v.z), r(v.w));
}
template <int ROWS, int GROUP>
__device__ __forceinline__ void convert_tile(unsigned char* t32, bool mn, uint32_t ct) {
    unsigned char* const t16 = t32 + ROWS * 128;
#pragma unroll 2
    for (uint32_t o = ct; o < ROWS * 4; o += GROUP) {
        unsigned char *s0, *s1, *h, *l;
        bool swap = false;
        if (!mn) {
            const uint32_t r = o >> 2, q = o & 3u, x = r & 7u, off = r * 64 + ((q ^ (r >> 1 & 3u)) << 4);
            s0 = t32 + r * 128 + ((2 * q ^ x) << 4);
            s1 = t32 + r * 128 + (((2 * q + 1) ^ x) << 4);
            h = t16 + off;
            l = h + ROWS * 64;
        } else {
            const uint32_t j = o & 3u, lo = o >> 2 & 1u, k = o >> 3 & 31u, blk = o >> 8;    // 64-row block blk, its half lo
            unsigned char* const s = t32 + (blk * 2 + lo) * 4096 + k * 128 + ((j ^ (k & 3u)) << 5);
            swap = lo != 0;
            s0 = s + (swap ? 16 : 0);
            s1 = s + (swap ? 0 : 16);
            h = t16 + blk * 8192 + k * 128 + (((lo * 4 + j) ^ (k & 7u)) << 4);
            l = h + 4096;
        }
        const float4 p = *reinterpret_cast<const float4*>(s0), q4 = *reinterpret_cast<const float4*>(s1);
        const float4 ph = round_tf32(p), qh = round_tf32(q4);
        *reinterpret_cast<float4*>(s0) = ph;
        *reinterpret_cast<float4*>(s1) = qh;
        const uint2 hp = pack_bf16x4(p), hq = pack_bf16x4(q4);
        const uint2 lp = pack_bf16x4(make_float4(p.x - ph.x, p.y - ph.y, p.z - ph.z, p.w - ph.w));
        const uint2 lq = pack_bf16x4(make_float4(q4.x - qh.x, q4.y - qh.y, q4.z - qh.z, q4.w - qh.w));
        const uint2 h0 = swap ? hq : hp, h1 = swap ? hp : hq, l0 = swap ? lq : lp, l1 = swap ? lp : lq;
        *reinterpret_cast<uint4*>(h) = make_uint4(h0.x, h0.y, h1.x, h1.y);
        *reinterpret_cast<uint4*>(l) = make_uint4(l0.x, l0.y, l1.x, l1.y);
    }
}

// The same split of sixteen k of one row of A (128 rows x 32 k, the k from 16 * half on), into tensor memory: the words as the
// kind::tf32 MMA reads them (one column per k), and the planes (two k per column).  A warp fills the 32 lanes it may touch.
__device__ __forceinline__ void convert_a_row(const unsigned char* t32, bool mn, uint32_t q, uint32_t lane, uint32_t half, uint32_t taddr) {
    float x[16];
    if (!mn) {
        const unsigned char* const r = t32 + (q * 32 + lane) * 128;
#pragma unroll
        for (uint32_t c = 0; c < 4; ++c) {
            const float4 v = *reinterpret_cast<const float4*>(r + (((half * 4 + c) ^ (lane & 7u)) << 4));
            x[4 * c] = v.x; x[4 * c + 1] = v.y; x[4 * c + 2] = v.z; x[4 * c + 3] = v.w;
        }
    } else {
        const unsigned char* const b = t32 + q * 4096 + half * 2048 + (lane & 7u) * 4;
#pragma unroll
        for (uint32_t k = 0; k < 16; ++k) x[k] = *reinterpret_cast<const float*>(b + k * 128 + (((lane >> 3) ^ (k & 3u)) << 5));
    }
    uint32_t f[16], h[8], l[8];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float4 v = make_float4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]), r = round_tf32(v);
        f[4 * c] = __float_as_uint(r.x); f[4 * c + 1] = __float_as_uint(r.y); f[4 * c + 2] = __float_as_uint(r.z); f[4 * c + 3] = __float_as_uint(r.w);
        const uint2 hv = pack_bf16x4(v), lv = pack_bf16x4(make_float4(v.x - r.x, v.y - r.y, v.z - r.z, v.w - r.w));
        h[2 * c] = hv.x; h[2 * c + 1] = hv.y;
        l[2 * c] = lv.x; l[2 * c + 1] = lv.y;
    }
    tmem_st_32x16(taddr + half * 16, f);
    tmem_st_32x8(taddr + 32 + half * 8, h);
    tmem_st_32x8(taddr + 48 + half * 8, l);
}

// Descriptors of one converted operand tile: the f32 words, the two planes, and how far one MMA's k advances them.
struct ConvOperand {
    uint64_t f, h, l;
    uint32_t adv32, adv16;
};
template <int ROWS>
__device__ __forceinline__ ConvOperand conv_operand(uint32_t t32, bool mn) {
    const uint32_t t16 = t32 + ROWS * 128;
    ConvOperand o;
    if (!mn) {
        o.f = make_desc_kmajor<128>(t32);
        o.h = make_desc_kmajor<64>(t16);
        o.l = make_desc_kmajor<64>(t16 + ROWS * 64);
        o.adv32 = 2; o.adv16 = 2;
    } else {
        o.f = make_desc_mnmajor(t32, 4096, 512, 1);
        o.h = make_desc_mnmajor(t16, 8192, 1024, 2);
        o.l = make_desc_mnmajor(t16 + 4096, 8192, 1024, 2);
        o.adv32 = 64; o.adv16 = 128;
    }
    return o;
}

// One or two products in a launch (the two gradients of a layer): problem 0's units come first, then problem 1's.
struct ConvArgs {
    Epilogue ep[2];
    uint32_t units0, units;       // units (tile x matrix) of problem 0, and of both
    uint32_t split;               // K-shares of a unit = CTAs of a cluster
    int* dev_status;
};

// Stores groups of four columns from `col` on: bias, activation or act' factor, the optional outputs.  A CTA stores one tile, or
// a few, with one or two warps per scheduler: their instructions come one after the other, so whatever does not change from row
// to row is settled before (asked again for every row, storing a 128 x 128 tile took 8000 - 11000 cycles).
struct ConvStore {
    uint32_t col;
    bool live, vec, plain;
    int kind, act;       // 0: as it is, 1: act, 2: * act'(mul_saved)
    __device__ __forceinline__ ConvStore(const Epilogue& ep, uint32_t c) : col(c), live(c < ep.N) {
        // (with vec, N is a multiple of four: a live group is whole)
        vec = (ep.N % 4 == 0) && (ep.c_batch % 4 == 0) &&
              (((reinterpret_cast<uintptr_t>(ep.C) | reinterpret_cast<uintptr_t>(ep.preact) | reinterpret_cast<uintptr_t>(ep.mul_saved)) & 15u) == 0);
        kind = ep.mul_saved ? 2 : ep.act != FG_ACT_NONE ? 1 : 0;
        act = kind == 2 ? ep.mul_act : ep.act;
        plain = vec && kind == 0 && !ep.preact && !ep.c_pairs;
    }
    // The group at element offset `off`, its bias added.  Returns what was stored in C.
    __device__ __forceinline__ float4 put_plain(const Epilogue& ep, size_t off, float4 z) const {
        *reinterpret_cast<float4*>(ep.C + off) = z;
        return z;
    }
    __device__ __forceinline__ float4 put_vec(const Epilogue& ep, size_t off, float4 z) const {
        float4 o = z;
        if (kind == 1) {
            o = make_float4(fg_act_fwd_sel(act, z.x), fg_act_fwd_sel(act, z.y), fg_act_fwd_sel(act, z.z), fg_act_fwd_sel(act, z.w));
        } else if (kind == 2) {
            const float4 sv = __ldg(reinterpret_cast<const float4*>(ep.mul_saved + off));
            o = make_float4(z.x * fg_act_grad_sel(act, sv.x), z.y * fg_act_grad_sel(act, sv.y), z.z * fg_act_grad_sel(act, sv.z),
                            z.w * fg_act_grad_sel(act, sv.w));
        }
        if (ep.preact) *reinterpret_cast<float4*>(ep.preact + off) = z;
        *reinterpret_cast<float4*>(ep.C + off) = o;
        if (ep.c_pairs) fg_store_pairs4(ep.c_pairs, ep.c_pairs_stride, off, o);
        return o;
    }
};
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
// Sums over the lanes that hold the same four columns (lanes c, c + 8, c + 16, c + 24).
__device__ __forceinline__ float4 sum_column_lanes(float4 v) {
#pragma unroll
    for (int d = 8; d < 32; d *= 2) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, d); v.y += __shfl_xor_sync(0xffffffffu, v.y, d);
        v.z += __shfl_xor_sync(0xffffffffu, v.z, d); v.w += __shfl_xor_sync(0xffffffffu, v.w, d);
    }
    return v;
}
__device__ __forceinline__ void store_colsum(const Epilogue& ep, uint32_t row0, uint32_t col, float4 cs) {
    float* d = ep.colsum_part + (size_t)(row0 >> 5) * ep.N + col;
    if (col < ep.N) d[0] = cs.x;
    if (col + 1 < ep.N) d[1] = cs.y;
    if (col + 2 < ep.N) d[2] = cs.z;
    if (col + 3 < ep.N) d[3] = cs.w;
}

// Units are walked persistently (unit, unit + CTAs, ...): the ring of loads, the conversion and the MMAs run across units, so
// that a tile is stored while the next one is computed; a CTA's last wide tile is stored by the converters, who have nothing else left
// to do and are twice as many (1024 x 256 x 2048 with bias 10.4 -> 10.0 us, with GELU 13.0 -> 11.0, 1000 x 256 x 2001 with GELU 23.8 ->
// 16.8; gradients of 1000 x 777 x 1001 39.8 -> 34.7).  With K-shares a cluster of `split` CTAs takes one unit, a share each, and the shares'
// sums meet through distributed shared memory: every CTA stores every split-th 32 x 32 block of the tile.
template <int BN, bool TWO, bool SHARES>
__global__ void __launch_bounds__(ConvCfg<BN>::kThreads, 1)
gemm_tc_conv_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmB0,
                    const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB1,
                    const __grid_constant__ ConvArgs ca) {
    using Cfg = ConvCfg<BN>;
    constexpr int S = Cfg::kStages, BK = 32, CPT = BN / 2;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* const base_ptr = smem_raw + (base - raw);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(base_ptr + S * Cfg::kStageBytes + Cfg::kStoreBytes);
    const uint32_t bar0 = base + S * Cfg::kStageBytes + Cfg::kStoreBytes;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };            // the f32 words have landed
    auto conv_bar = [&](int s) { return bar0 + 8u * (S + s); };      // both operands are converted
    auto empty_bar = [&](int s) { return bar0 + 8u * (2 * S + s); };
    auto acc_full_bar = [&](int b) { return bar0 + 8u * (3 * S + b); };
    auto acc_empty_bar = [&](int b) { return bar0 + 8u * (3 * S + 2 + b); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 3 * S + 4);

    // (the warp index is known to be the same in all lanes, as in the pair kernel)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t split = SHARES ? ca.split : 1u, share = SHARES ? cluster_ctarank() : 0u;
    const uint32_t first = SHARES ? blockIdx.x / split : blockIdx.x, step = SHARES ? ca.units : gridDim.x;
    struct Unit { uint32_t p, m0, n0, bz, kb0, nkb; };
    // (each problem's fields are read at addresses known to the compiler: through a pointer they are loads from memory)
    auto ep_of = [&](uint32_t p, auto field) { return !TWO || p == 0 ? field(ca.ep[0]) : field(ca.ep[1]); };
    auto unit_at = [&](uint32_t u) -> Unit {
        Unit t;
        t.p = TWO && u >= ca.units0 ? 1u : 0u;
        const uint32_t v = u - (t.p ? ca.units0 : 0u), K = ep_of(t.p, [](const Epilogue& e) { return e.K; });
        const uint32_t tiles_m = ep_of(t.p, [](const Epilogue& e) { return (e.M + BM - 1) / BM; });
        const uint32_t tiles = ep_of(t.p, [](const Epilogue& e) { return ((e.M + BM - 1) / BM) * ((e.N + BN - 1) / BN); }), tile = v % tiles;
        t.bz = v / tiles;
        t.m0 = tile % tiles_m * BM;      // down the columns of tiles: the CTAs at work share a few tile columns of B
        t.n0 = tile / tiles_m * BN;
        const uint32_t all = (K + BK - 1) / BK;      // the host keeps split <= all
        t.kb0 = (uint32_t)((uint64_t)share * all / split);
        t.nkb = (uint32_t)((uint64_t)(share + 1) * all / split) - t.kb0;
        return t;
    };
    auto is_mn = [&](uint32_t p, bool& a, bool& b) {
        a = ep_of(p, [](const Epilogue& e) { return e.a_mn != 0; });
        b = ep_of(p, [](const Epilogue& e) { return e.b_mn != 0; });
    };
    // Do the converters store a CTA's last tile?  (Of narrow tiles, half as long to store, it slowed the others down: gradients of
    // 16 x 384 x 512 x 320 29.7 -> 31.0 us.)
    constexpr bool kHandOn = !SHARES && BN == 128;
    // Chunks of 128 k, half of the other kernels': fewer additions in the tensor core's truncating accumulator, as K-shares of that
    // length had, and the epilogue warps have the time (a tile's drain takes a tenth of its four k-blocks).
    constexpr uint32_t kChunkKB = 128 / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(full_bar(s), 1); mbar_init(conv_bar(s), Cfg::kGroup / 32); mbar_init(empty_bar(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full_bar(b), 1); mbar_init(acc_empty_bar(b), 8); }
        fence_mbar_init();
        prefetch_tmap(&tmA0);
        prefetch_tmap(&tmB0);
        if (TWO) { prefetch_tmap(&tmA1); prefetch_tmap(&tmB1); }
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), Cfg::kTmemCols);
        tmem_relinquish();
    }
    // Everything up to here needs nothing of the kernels before this one: it passes while the last of them drains.
    fg_grid_enter();
    __shared__ int s_abort;      // see gemm_tc_kernel; the CTAs of a cluster stay together to the end, whatever they have read
    __shared__ int s_tail;       // the last tile's sums are in the stages
    if (threadIdx.x == 0) {
        s_abort = *reinterpret_cast<volatile int*>(ca.dev_status);
        s_tail = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const bool go = __all_sync(0xffffffffu, s_abort == 0);

    // A warp stores 32 columns of up to 32 rows of whole sums, which lie in shared memory in float4s: at(row, float4 of the row).
    auto store_rows = [&](const Epilogue& ep, size_t cb, uint32_t row0, uint32_t col0, float bias, uint32_t rows, auto at) {
        const uint32_t rsub = lane >> 3, cc = lane & 7;
        const ConvStore st(ep, col0 + cc * 4);
        if (!st.vec) {
            // Rows that do not start on 16 bytes: a lane per column, a row of 128 bytes per step (four single words per lane
            // and step, 16 bytes apart between lanes, took 11000 cycles for a 128 x 128 tile: backward of 1000 x 777 x 1001 51.0 -> 40.9 us).
            const uint32_t c = col0 + lane;
            if (c >= ep.N) rows = 0;
            size_t off = cb + (size_t)row0 * ep.N + c;
            float cs[4] = {0.f, 0.f, 0.f, 0.f};      // row r in chain r % 4, as the lanes below have it
#pragma unroll 4
            for (uint32_t r = 0; r < 32; ++r, off += ep.N) {
                if (r >= rows) continue;
                const float z = reinterpret_cast<const float*>(at(r, (uint32_t)lane >> 2))[lane & 3] + bias;
                const float o = st.kind == 2 ? z * fg_act_grad_fast(st.act, ep.mul_saved[off]) : st.kind == 1 ? fg_act_fwd_sel(st.act, z) : z;
                if (ep.preact) ep.preact[off] = z;
                ep.C[off] = o;
                if (ep.c_pairs) fg_store_pairs1(ep.c_pairs, ep.c_pairs_stride, off, o);
                cs[r & 3] += o;
            }
            if (ep.colsum_part && rows) ep.colsum_part[(size_t)(row0 >> 5) * ep.N + c] = (cs[0] + cs[1]) + (cs[2] + cs[3]);
            __syncwarp();
            return;
        }
        const float4 bz = make_float4(__shfl_sync(0xffffffffu, bias, cc * 4), __shfl_sync(0xffffffffu, bias, cc * 4 + 1),
                                      __shfl_sync(0xffffffffu, bias, cc * 4 + 2), __shfl_sync(0xffffffffu, bias, cc * 4 + 3));
        float4 cs = make_float4(0.f, 0.f, 0.f, 0.f);
        size_t off = cb + (size_t)(row0 + rsub) * ep.N + st.col;
        const uint32_t mine = st.live && rsub < rows ? (rows - rsub + 3) / 4 : 0u;      // this lane's, of eight
        auto sum_at = [&](uint32_t i) { return add4(*reinterpret_cast<const float4*>(at(i * 4 + rsub, cc)), bz); };
        if (st.plain) {
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i, off += (size_t)4 * ep.N)
                if (i < mine) cs = add4(cs, st.put_plain(ep, off, sum_at(i)));
        } else {
#pragma unroll 2
            for (uint32_t i = 0; i < 8; ++i, off += (size_t)4 * ep.N)
                if (i < mine) cs = add4(cs, st.put_vec(ep, off, sum_at(i)));
        }
        __syncwarp();
        if (ep.colsum_part) {
            cs = sum_column_lanes(cs);
            if (lane < 8 && rows) store_colsum(ep, row0, st.col, cs);
        }
        __syncwarp();
    };

    if (warp < Cfg::kEpi0) {
        reg_release<Cfg::kRegsLow>();
        if (go && warp == 0) {
            // ---- producer ----
            uint32_t g = 0;      // k-blocks so far, across units: ring position and phase
            bool ok = true;
            for (uint32_t u = first; u < ca.units && ok; u += step) {
                const Unit t = unit_at(u);
                const CUtensorMap* const ta = TWO && t.p ? &tmA1 : &tmA0;
                const CUtensorMap* const tb = TWO && t.p ? &tmB1 : &tmB0;
                bool a_mn, b_mn;
                is_mn(t.p, a_mn, b_mn);
                for (uint32_t i = 0; i < t.nkb; ++i, ++g) {
                    const int s = g % S;
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(empty_bar(s), ((g / S) & 1u) ^ 1u, kWaitCycles))) {
                        if (lane == 0) atomicOr(ca.dev_status, FG_DEVERR_TMA_WAIT);
                        ok = false;
                        break;
                    }
                    const uint32_t sa = base + s * Cfg::kStageBytes, sb = sa + Cfg::kA32;
                    const int k = (int)((t.kb0 + i) * BK);
                    if (!elect_one()) continue;
                    mbar_expect_tx(full_bar(s), Cfg::kA32 + Cfg::kB32);
                    if (!a_mn) tma_load_3d(sa, ta, full_bar(s), k, (int)t.m0, (int)t.bz);
                    else
#pragma unroll
                        for (int j = 0; j < BM / 32; ++j) tma_load_3d(sa + j * 4096, ta, full_bar(s), (int)(t.m0 + 32 * j), k, (int)t.bz);
                    if (!b_mn) tma_load_3d(sb, tb, full_bar(s), k, (int)t.n0, (int)t.bz);
                    else
#pragma unroll
                        for (int j = 0; j < BN / 32; ++j) tma_load_3d(sb + j * 4096, tb, full_bar(s), (int)(t.n0 + 32 * j), k, (int)t.bz);
                }
            }
        } else if (go && warp == 1) {
            // ---- MMA issuer ----
            bool ok = true;
            uint32_t g = 0, gc = 0;      // k-blocks and chunks so far, across units
            for (uint32_t u = first; u < ca.units && ok; u += step) {
                const Unit t = unit_at(u);
                bool a_mn, b_mn;
                is_mn(t.p, a_mn, b_mn);
                const uint32_t mnbits = b_mn ? kIdescBMnMajor : 0u;
                const uint32_t idesc32 = make_idesc(2u /*tf32*/, BM, BN) | mnbits, idesc16 = make_idesc(1u /*bf16*/, BM, BN) | mnbits;
                const uint32_t nchunks = (t.nkb + kChunkKB - 1) / kChunkKB;
                for (uint32_t c = 0; c < nchunks && ok; ++c, ++gc) {
                    const uint32_t buf = gc & 1u;
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(acc_empty_bar(buf), ((gc >> 1) & 1u) ^ 1u, kWaitCycles))) {
                        if (lane == 0) atomicOr(ca.dev_status, FG_DEVERR_MMA_WAIT);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_base + buf * BN;
                    const uint32_t end = min(t.nkb, (c + 1) * kChunkKB);
                    for (uint32_t i = c * kChunkKB; i < end; ++i, ++g) {
                        const int s = g % S;
                        if (!__all_sync(0xffffffffu, mbar_wait_bounded(conv_bar(s), (g / S) & 1u, kWaitCycles))) {
                            if (lane == 0) atomicOr(ca.dev_status, FG_DEVERR_MMA_WAIT);
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t sa = base + s * Cfg::kStageBytes;
                        const ConvOperand b = conv_operand<BN>(sa + Cfg::kA32, b_mn);
                        const uint32_t a = tmem_base + 2 * BN + s * Cfg::kACols;
                        const uint32_t acc = (i == c * kChunkKB) ? 0u : 1u;      // a chunk starts from zero
                        if (elect_one()) {
#pragma unroll
                            for (int kk = 0; kk < BK / 16; ++kk) {
                                mma_f16_ta(d_tmem, a + 48 + kk * 8, b.h + (uint64_t)(kk * b.adv16), idesc16, acc | (uint32_t)kk);
                                mma_f16_ta(d_tmem, a + 32 + kk * 8, b.l + (uint64_t)(kk * b.adv16), idesc16, 1u);
                            }
#pragma unroll
                            for (int kk = 0; kk < BK / UK; ++kk)
                                mma_tf32_ta(d_tmem, a + kk * 8, b.f + (uint64_t)(kk * b.adv32), idesc32, 1u);
                            mma_commit(empty_bar(s));
                        }
                        __syncwarp();
                    }
                    if (ok && elect_one()) mma_commit(acc_full_bar(buf));
                    __syncwarp();
                }
            }
        }
        if constexpr (SHARES) { __syncwarp(); cluster_sync_all(); cluster_sync_all(); }      // as the converters
    } else if (warp >= Cfg::kConv0) {
        reg_release<Cfg::kRegsConv>();
        // ---- converters: two groups of eight warps take the k-blocks in turn, so that one's waits (for the loads, shared memory
        // and the proxy fence) pass under the other's work.  Every stage belongs to one group: it is refilled only after its
        // group has converted it, so that no wait, which names a phase by its parity alone, can meet the phase before or after
        // the one it means. ----
        static_assert(S % Cfg::kGroups == 0 && Cfg::kGroup % 128 == 0, "see above");
        const uint32_t ct = (threadIdx.x - Cfg::kConv0 * 32) % Cfg::kGroup, mine = (threadIdx.x - Cfg::kConv0 * 32) / Cfg::kGroup;
        uint32_t g = 0;
        bool ok = go;
        for (uint32_t u = first; u < ca.units && ok; u += step) {
            const Unit t = unit_at(u);
            bool a_mn, b_mn;
            is_mn(t.p, a_mn, b_mn);
            for (uint32_t i = 0; i < t.nkb; ++i, ++g) {
                if (g % Cfg::kGroups != mine) continue;
                const int s = g % S;
                unsigned char* const sa = base_ptr + s * Cfg::kStageBytes;
                const bool got = mbar_wait_bounded(full_bar(s), (g / S) & 1u, kWaitCycles);
                if (!__all_sync(0xffffffffu, got)) {
                    if (lane == 0) atomicOr(ca.dev_status, FG_DEVERR_TMA_WAIT);
                    ok = false;
                    break;
                }
                tc_fence_after();           // the stage's tensor memory has been read: its load was waited for after those MMAs
                const uint32_t ta = tmem_base + ((uint32_t)(warp & 3) << 21) + 2 * BN + s * Cfg::kACols;
                convert_a_row(sa, a_mn, warp & 3, lane, ct >> 7, ta);
                convert_tile<BN, Cfg::kGroup>(sa + Cfg::kA32, b_mn, ct);
                tmem_st_wait();
                tc_fence_before();
                fence_proxy_async();        // the planes are read by the tensor core
                __syncwarp();
                if (lane == 0) mbar_arrive(conv_bar(s));
            }
        }
        if constexpr (kHandOn) {
            // The CTA's last tile, from the stages' room: a warp takes a block of 32 x 32.
            const Unit t = unit_at(first + (ca.units - 1 - first) / step * step);
            const uint32_t lr0 = (uint32_t)(warp - Cfg::kConv0) / (BN / 32) * 32, cb = (uint32_t)(warp - Cfg::kConv0) % (BN / 32);
            auto store = [&](const Epilogue& ep) {
                const uint32_t row0 = t.m0 + lr0, col0 = t.n0 + cb * 32;
                const float bias = ep.bias && col0 + lane < ep.N ? ep.bias[col0 + lane] : 0.0f;
                __syncwarp();
                asm volatile("bar.sync 2, 768;" ::: "memory");      // the sums are there
                if (s_tail && row0 < ep.M)
                    store_rows(ep, (size_t)t.bz * ep.c_batch, row0, col0, bias, min(32u, ep.M - row0),
                               [&](uint32_t r, uint32_t c) { return base_ptr + (((lr0 + r) * (BN / 4) + ((cb * 8 + c) ^ (r & 7))) << 4); });
            };
            if (!TWO || t.p == 0) store(ca.ep[0]);
            else store(ca.ep[1]);
        }
        if constexpr (SHARES) {
            __syncwarp();
            cluster_sync_all();      // every share's sums are in its CTA's shared memory
            if (go) {
                // This CTA's 32 x 32 blocks are every split-th of the tile, from its share's number on; a warp takes four rows of
                // one, a lane four columns of a row.
                const Unit t = unit_at(first);
                const uint32_t rsub = lane >> 3, cc = lane & 7;
                auto fold = [&](const Epilogue& ep, auto ragged) {
                    float4* const csum = reinterpret_cast<float4*>(base_ptr + S * Cfg::kStageBytes);      // [block][eight times four rows][8 lanes]
                    for (uint32_t v = warp - Cfg::kConv0, b; (b = share + split * (v >> 3)) < 4 * (BN / 32); v += 16) {
                        const uint32_t lr = (b & 3u) * 32 + (v & 7u) * 4 + rsub, c0 = (b >> 2) * 32, row = t.m0 + lr;
                        const ConvStore st(ep, t.n0 + c0 + cc * 4);
                        const uint32_t at = base + ((lr * (BN / 4) + (((c0 >> 2) + cc) ^ (lr & 7))) << 4);
                        float4 z[8];
#pragma unroll
                        for (uint32_t r = 0; r < 8; ++r)
                            if (r < split) z[r] = ld_cluster_f4(map_to_cta(at, r));
                        float bz[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) bz[j] = ep.bias && st.col + j < ep.N ? ep.bias[st.col + j] : 0.0f;
#pragma unroll
                        for (uint32_t r = 1; r < 8; ++r)        // in the order of the shares, whoever adds them
                            if (r < split) z[0] = add4(z[0], z[r]);
                        if constexpr (decltype(ragged)::value) {
                            const float4 w = add4(z[0], make_float4(bz[0], bz[1], bz[2], bz[3]));
                            // Rows that do not start on 16 bytes: a lane per column, one of the four rows per step, as in store_rows.
                            const uint32_t c = t.n0 + c0 + lane, r0 = t.m0 + (b & 3u) * 32 + (v & 7u) * 4;
                            size_t off = (size_t)t.bz * ep.c_batch + (size_t)r0 * ep.N + c;
                            float o[4];
#pragma unroll
                            for (uint32_t i = 0; i < 4; ++i, off += ep.N) {
                                const int from = (int)(i * 8 + (lane >> 2));
                                const float x0 = __shfl_sync(0xffffffffu, w.x, from), x1 = __shfl_sync(0xffffffffu, w.y, from);
                                const float x2 = __shfl_sync(0xffffffffu, w.z, from), x3 = __shfl_sync(0xffffffffu, w.w, from);
                                const float x = lane & 2 ? (lane & 1 ? x3 : x2) : (lane & 1 ? x1 : x0);
                                o[i] = 0.0f;
                                if (c >= ep.N || r0 + i >= ep.M) continue;
                                o[i] = st.kind == 2 ? x * fg_act_grad_fast(st.act, ep.mul_saved[off]) : st.kind == 1 ? fg_act_fwd_sel(st.act, x) : x;
                                if (ep.preact) ep.preact[off] = x;
                                ep.C[off] = o[i];
                                if (ep.c_pairs) fg_store_pairs1(ep.c_pairs, ep.c_pairs_stride, off, o[i]);
                            }
                            if (ep.colsum_part) reinterpret_cast<float*>(csum)[v * 32 + lane] = (o[0] + o[1]) + (o[2] + o[3]);
                            __syncwarp();
                            continue;
                        }
                        float4 cs = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (st.live && row < ep.M) {
                            const size_t off = (size_t)t.bz * ep.c_batch + (size_t)row * ep.N + st.col;
                            const float4 w = add4(z[0], make_float4(bz[0], bz[1], bz[2], bz[3]));
                            cs = st.plain ? st.put_plain(ep, off, w) : st.put_vec(ep, off, w);
                        }
                        __syncwarp();
                        if (ep.colsum_part) {
                            cs = sum_column_lanes(cs);
                            if (lane < 8) csum[v * 8 + lane] = cs;
                        }
                    }
                    if (ep.colsum_part) {
                        asm volatile("bar.sync 1, 512;" ::: "memory");      // the converters
                        const uint32_t k = threadIdx.x - Cfg::kConv0 * 32, blk = k >> 3, b = share + split * blk;      // eight lanes per block
                        if (b < 4 * (BN / 32) && t.m0 + (b & 3u) * 32 < ep.M) {
                            float4 w = csum[blk * 64 + cc];
#pragma unroll
                            for (uint32_t j = 1; j < 8; ++j) w = add4(w, csum[blk * 64 + j * 8 + cc]);
                            store_colsum(ep, t.m0 + (b & 3u) * 32, t.n0 + (b >> 2) * 32 + cc * 4, w);
                        }
                    }
                };
                auto fold_of = [&](const Epilogue& ep) {
                    if (ConvStore(ep, 0).vec) fold(ep, std::false_type{});
                    else fold(ep, std::true_type{});
                };
                if (!TWO || t.p == 0) fold_of(ca.ep[0]);
                else fold_of(ca.ep[1]);
            }
            __syncwarp();
            cluster_sync_all();      // no CTA leaves while another reads its sums
        }
    } else {
        reg_acquire<Cfg::kRegsEpi>();
        // ---- accumulate + epilogue: warps 4..11; warp w may touch TMEM lanes 32*(w%4) .. +31 ----
        const int q = warp & 3, half = (warp - Cfg::kEpi0) >> 2;
        bool ok = go;
        uint32_t gc = 0;
        float4* const tb4 = reinterpret_cast<float4*>(base_ptr + S * Cfg::kStageBytes) + (warp - Cfg::kEpi0) * (32 * 8);
        for (uint32_t u = first; u < ca.units && ok; u += step) {
            const Unit t = unit_at(u);
            const uint32_t nchunks = (t.nkb + kChunkKB - 1) / kChunkKB;
            // a lane holds the bias of one column per block: it is here long before the sums are
            float bias[CPT / 32];
            const bool last = SHARES || (kHandOn && u + step >= ca.units);
            if (!last) {
                const float* const bp = ep_of(t.p, [](const Epilogue& e) { return e.bias; });
                const uint32_t N = ep_of(t.p, [](const Epilogue& e) { return e.N; });
#pragma unroll
                for (int gr = 0; gr < CPT / 32; ++gr) {
                    const uint32_t c = t.n0 + half * CPT + gr * 32 + lane;
                    bias[gr] = bp && c < N ? bp[c] : 0.0f;
                }
            }
            float sum[CPT];
#pragma unroll
            for (int j = 0; j < CPT; ++j) sum[j] = 0.0f;
            for (uint32_t c = 0; c < nchunks; ++c, ++gc) {
                const uint32_t buf = gc & 1u;
                bool got = mbar_wait_bounded(acc_full_bar(buf), (gc >> 1) & 1u, kWaitCycles + kWaitCycles / 2);
                got = __all_sync(0xffffffffu, got);
                if (!got) {
                    if (lane == 0) atomicOr(ca.dev_status, FG_DEVERR_EPI_WAIT);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN + half * CPT;
#pragma unroll
                for (int gr = 0; gr < CPT / 32; ++gr) {
                    uint32_t r[32];
                    tmem_ld_32x32(t0 + gr * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[gr * 32 + j] += __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty_bar(buf));
            }
            if (!ok) break;
            if (last) {
                // Every load and MMA of this CTA has finished (its last chunk is complete), so the stages are free: the tile's or
                // the share's sums as [row][BN], float4 c of a row at c ^ (row & 7).
                float4* const part = reinterpret_cast<float4*>(base_ptr) + (q * 32 + lane) * (BN / 4);
#pragma unroll
                for (int c = 0; c < CPT / 4; ++c)
                    part[(half * (CPT / 4) + c) ^ (lane & 7)] = make_float4(sum[4 * c], sum[4 * c + 1], sum[4 * c + 2], sum[4 * c + 3]);
                if (kHandOn && threadIdx.x == Cfg::kEpi0 * 32) s_tail = 1;
            } else {
#pragma unroll 1
                for (int gr = 0; gr < CPT / 32; ++gr) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        float4 v = make_float4(sum[4 * c], sum[4 * c + 1], sum[4 * c + 2], sum[4 * c + 3]);
                        if (CPT > 32 && gr) v = make_float4(sum[CPT - 32 + 4 * c], sum[CPT - 32 + 4 * c + 1], sum[CPT - 32 + 4 * c + 2], sum[CPT - 32 + 4 * c + 3]);
                        tb4[lane * 8 + (c ^ (lane & 7))] = v;
                    }
                    __syncwarp();
                    const uint32_t row0 = t.m0 + q * 32, col0 = t.n0 + half * CPT + gr * 32;
                    const float bv = CPT > 32 && gr ? bias[CPT / 32 - 1] : bias[0];
                    auto store = [&](const Epilogue& ep) {
                        store_rows(ep, (size_t)t.bz * ep.c_batch, row0, col0, bv, row0 < ep.M ? min(32u, ep.M - row0) : 0u,
                                   [&](uint32_t r, uint32_t c) { return reinterpret_cast<const unsigned char*>(tb4 + r * 8 + (c ^ (r & 7))); });
                    };
                    if (!TWO || t.p == 0) store(ca.ep[0]);
                    else store(ca.ep[1]);
                }
            }
        }
        if constexpr (SHARES) { __syncwarp(); cluster_sync_all(); cluster_sync_all(); }      // as the converters
        if constexpr (kHandOn) { __syncwarp(); asm volatile("bar.sync 2, 768;" ::: "memory"); }      // the converters store the last tile
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

// ------------------------------------------------------------------------------------
// Sixteen-bit tensors, small and middling products: the conversion kernel's scheme without its converters.  The pair kernel's 256 x 256
// tiles leave most SMs idle on a product of a few tiles and cost 15 - 20 us whatever the product's size (layers of 100 - 500 samples:
// three of them, 65 us forward and backward).  Here a CTA owns a 128 x BN tile (BN 128 or 64), k-blocks of 64 go from the tensors as
// they lie through shared memory into kind::f16 MMAs, K-shares are the CTAs of a cluster, whose sums meet in distributed shared
// memory, and both gradients of a layer are one launch.
//   warp 0 loads, warp 1 issues MMAs, warps 4..11 drain accumulators, add up the shares and store.
// Bound by shared memory on long k (128 x 128: 32 KB in and 32 KB out of it per k-block, 512 cycles; the tensor core needs 256), by the
// ends of the launch on short ones.
// ------------------------------------------------------------------------------------
template <int BN>
struct HalfCfg {
    static constexpr int kA = BM * 128, kB = BN * 128, kStageBytes = kA + kB;      // 64 values of k: rows of 128 bytes
    static constexpr int kStages = BN == 128 ? 6 : 8;
    static constexpr int kThreads = 384, kEpi0 = 4;
    static constexpr int kStoreBytes = 8 * 32 * 32 * 4;
    static constexpr int kSmemBytes = kStages * kStageBytes + kStoreBytes + 1024 + 256;
    static_assert(kSmemBytes <= 232448, "exceeds the 227 KB a CTA may use");
    static_assert(kStages * kStageBytes >= BM * BN * 4, "a K-share's sums lie in the stages");
    static constexpr int kTmemCols = 2 * BN;
};
struct HalfArgs {
    Epilogue ep[2];
    uint32_t units0, units, split;
    int* dev_status;
};

template <int BN, bool TWO, bool SHARES>
__global__ void __launch_bounds__(HalfCfg<BN>::kThreads, 1)
gemm_tc_half_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmB0,
                    const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB1,
                    const __grid_constant__ HalfArgs ha) {
    using Cfg = HalfCfg<BN>;
    constexpr int S = Cfg::kStages, BK = 64, CPT = BN / 2;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* const base_ptr = smem_raw + (base - raw);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(base_ptr + S * Cfg::kStageBytes + Cfg::kStoreBytes);
    const uint32_t bar0 = base + S * Cfg::kStageBytes + Cfg::kStoreBytes;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (S + s); };
    auto acc_full_bar = [&](int b) { return bar0 + 8u * (2 * S + b); };
    auto acc_empty_bar = [&](int b) { return bar0 + 8u * (2 * S + 2 + b); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * S + 4);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t split = SHARES ? ha.split : 1u, share = SHARES ? cluster_ctarank() : 0u;
    const uint32_t first = SHARES ? blockIdx.x / split : blockIdx.x, step = SHARES ? ha.units : gridDim.x;
    struct Unit { uint32_t p, m0, n0, kb0, nkb; };
    auto ep_of = [&](uint32_t p, auto field) { return !TWO || p == 0 ? field(ha.ep[0]) : field(ha.ep[1]); };
    auto unit_at = [&](uint32_t u) -> Unit {
        Unit t;
        t.p = TWO && u >= ha.units0 ? 1u : 0u;
        const uint32_t tile = u - (t.p ? ha.units0 : 0u), K = ep_of(t.p, [](const Epilogue& e) { return e.K; });
        const uint32_t tiles_m = ep_of(t.p, [](const Epilogue& e) { return (e.M + BM - 1) / BM; });
        t.m0 = tile % tiles_m * BM;
        t.n0 = tile / tiles_m * BN;
        const uint32_t all = (K + BK - 1) / BK;      // the host keeps split <= all
        t.kb0 = (uint32_t)((uint64_t)share * all / split);
        t.nkb = (uint32_t)((uint64_t)(share + 1) * all / split) - t.kb0;
        return t;
    };
    auto is_mn = [&](uint32_t p, bool& a, bool& b) {
        a = ep_of(p, [](const Epilogue& e) { return e.a_mn != 0; });
        b = ep_of(p, [](const Epilogue& e) { return e.b_mn != 0; });
    };
    constexpr uint32_t kChunkKB = 1024 / BK;      // k per accumulation chunk, as in the pair kernel

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full_bar(b), 1); mbar_init(acc_empty_bar(b), 8); }
        fence_mbar_init();
        prefetch_tmap(&tmA0);
        prefetch_tmap(&tmB0);
        if (TWO) { prefetch_tmap(&tmA1); prefetch_tmap(&tmB1); }
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), Cfg::kTmemCols);
        tmem_relinquish();
    }
    // Everything up to here needs nothing of the kernels before this one: it passes while the last of them drains.
    fg_grid_enter();
    __shared__ int s_abort;      // see gemm_tc_kernel; the CTAs of a cluster stay together to the end, whatever they have read
    if (threadIdx.x == 0) s_abort = *reinterpret_cast<volatile int*>(ha.dev_status);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const bool go = __all_sync(0xffffffffu, s_abort == 0);

    if (go && warp == 0) {
        // ---- producer ----
        uint32_t g = 0;      // k-blocks so far, across units: ring position and phase
        bool ok = true;
        for (uint32_t u = first; u < ha.units && ok; u += step) {
            const Unit t = unit_at(u);
            const CUtensorMap* const ta = TWO && t.p ? &tmA1 : &tmA0;
            const CUtensorMap* const tb = TWO && t.p ? &tmB1 : &tmB0;
            bool a_mn, b_mn;
            is_mn(t.p, a_mn, b_mn);
            for (uint32_t i = 0; i < t.nkb; ++i, ++g) {
                const int s = g % S;
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(empty_bar(s), ((g / S) & 1u) ^ 1u, kWaitCycles))) {
                    if (lane == 0) atomicOr(ha.dev_status, FG_DEVERR_TMA_WAIT);
                    ok = false;
                    break;
                }
                const uint32_t sa = base + s * Cfg::kStageBytes, sb = sa + Cfg::kA;
                const int k = (int)((t.kb0 + i) * BK);
                if (!elect_one()) continue;
                mbar_expect_tx(full_bar(s), Cfg::kStageBytes);
                // K-major storage: one box; MN-major ([k][rows]): boxes of 64 rows x 64 k, each [k][64 rows]
                if (!a_mn) tma_load_3d(sa, ta, full_bar(s), k, (int)t.m0, 0);
                else
#pragma unroll
                    for (int j = 0; j < BM / 64; ++j) tma_load_3d(sa + j * 8192, ta, full_bar(s), (int)(t.m0 + 64 * j), k, 0);
                if (!b_mn) tma_load_3d(sb, tb, full_bar(s), k, (int)t.n0, 0);
                else
#pragma unroll
                    for (int j = 0; j < BN / 64; ++j) tma_load_3d(sb + j * 8192, tb, full_bar(s), (int)(t.n0 + 64 * j), k, 0);
            }
        }
    } else if (go && warp == 1) {
        // ---- MMA issuer ----
        bool ok = true;
        uint32_t g = 0, gc = 0;      // k-blocks and chunks so far, across units
        for (uint32_t u = first; u < ha.units && ok; u += step) {
            const Unit t = unit_at(u);
            bool a_mn, b_mn;
            is_mn(t.p, a_mn, b_mn);
            const uint32_t idesc = make_idesc(ha.ep[0].out_dtype == FG_DTYPE_BF16 ? 1u : 0u, BM, BN) | (a_mn ? kIdescAMnMajor : 0u) | (b_mn ? kIdescBMnMajor : 0u);
            const uint32_t a_adv = a_mn ? 128u : 2u, b_adv = b_mn ? 128u : 2u;
            const uint32_t nchunks = (t.nkb + kChunkKB - 1) / kChunkKB;
            for (uint32_t c = 0; c < nchunks && ok; ++c, ++gc) {
                const uint32_t buf = gc & 1u;
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(acc_empty_bar(buf), ((gc >> 1) & 1u) ^ 1u, kWaitCycles))) {
                    if (lane == 0) atomicOr(ha.dev_status, FG_DEVERR_MMA_WAIT);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                const uint32_t end = min(t.nkb, (c + 1) * kChunkKB);
                for (uint32_t i = c * kChunkKB; i < end; ++i, ++g) {
                    const int s = g % S;
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(full_bar(s), (g / S) & 1u, kWaitCycles))) {
                        if (lane == 0) atomicOr(ha.dev_status, FG_DEVERR_MMA_WAIT);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = base + s * Cfg::kStageBytes, sb = sa + Cfg::kA;
                    const uint64_t a_d = a_mn ? make_desc_mnmajor(sa, 8192, 1024, 2) : make_desc_kmajor<128>(sa);
                    const uint64_t b_d = b_mn ? make_desc_mnmajor(sb, 8192, 1024, 2) : make_desc_kmajor<128>(sb);
                    const uint32_t acc = (i == c * kChunkKB) ? 0u : 1u;      // a chunk starts from zero
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < BK / 16; ++kk)
                            mma_f16(d_tmem, a_d + (uint64_t)(kk * a_adv), b_d + (uint64_t)(kk * b_adv), idesc, acc | (uint32_t)kk);
                        mma_commit(empty_bar(s));
                    }
                    __syncwarp();
                }
                if (ok && elect_one()) mma_commit(acc_full_bar(buf));
                __syncwarp();
            }
        }
    } else if (warp >= Cfg::kEpi0) {
        // ---- accumulate + epilogue: warps 4..11; warp w may touch TMEM lanes 32*(w%4) .. +31 ----
        const int q = warp & 3, half = (warp - Cfg::kEpi0) >> 2;
        bool ok = go;
        uint32_t gc = 0;
        float4* const tb4 = reinterpret_cast<float4*>(base_ptr + S * Cfg::kStageBytes) + (warp - Cfg::kEpi0) * (32 * 8);
        const uint32_t rsub = lane >> 3, cc = lane & 7;
        // (a launch of two products, the gradients, has none)
        auto bias_at = [&](uint32_t c) { return !TWO && ha.ep[0].bias && c < ha.ep[0].N ? epi_bias(ha.ep[0].bias, c, ha.ep[0].out_dtype) : 0.0f; };
        // Four columns of a row from their sums with the bias.
        auto put4 = [&](const Epilogue& ep, size_t off, uint32_t col, bool vec, float4 z) {
            if (vec) {      // (N is a multiple of four: a live group is whole)
                const float4 o = ep.act == FG_ACT_NONE ? z : make_float4(fg_act_fwd_sel(ep.act, z.x), fg_act_fwd_sel(ep.act, z.y),
                                                                         fg_act_fwd_sel(ep.act, z.z), fg_act_fwd_sel(ep.act, z.w));
                if (ep.preact) store_out4(ep.preact, off, z, ep.out_dtype);
                store_out4(ep.C, off, o, ep.out_dtype);
            } else {
                epi_store_edge(z, off, col, ep.N, (char*)ep.C, (char*)ep.preact, nullptr, 0, nullptr, 0, ep.act, ep.out_dtype);
            }
        };
        auto vec_ok = [&](const Epilogue& ep) {      // (C and preact start on 16 bytes)
            return ep.N % 4 == 0;
        };
        // A 32 x 32 block of whole sums, swizzled in tb4 (float4 c of row r at c ^ (r & 7)): four rows of 64 bytes per step, or, where
        // rows do not start on eight bytes, a lane per column and a row per step.
        auto store_block = [&](const Epilogue& ep, uint32_t row0, uint32_t col0, float bias) {
            if (!vec_ok(ep)) {
                const uint32_t c = col0 + lane, rows = c < ep.N && row0 < ep.M ? min(32u, ep.M - row0) : 0u;
                const float* const tb = reinterpret_cast<const float*>(tb4);
                size_t off = (size_t)row0 * ep.N + c;
#pragma unroll 4
                for (uint32_t r = 0; r < 32; ++r, off += ep.N) {
                    if (r >= rows) continue;
                    const float z = tb[r * 32 + (((lane >> 2) ^ (r & 7)) << 2) + (lane & 3)] + bias;
                    if (ep.preact) store_out1(ep.preact, off, z, ep.out_dtype);
                    store_out1(ep.C, off, fg_act_fwd_sel(ep.act, z), ep.out_dtype);
                }
                __syncwarp();
                return;
            }
            const float4 bz = make_float4(__shfl_sync(0xffffffffu, bias, cc * 4), __shfl_sync(0xffffffffu, bias, cc * 4 + 1),
                                          __shfl_sync(0xffffffffu, bias, cc * 4 + 2), __shfl_sync(0xffffffffu, bias, cc * 4 + 3));
            const uint32_t col = col0 + cc * 4;
            size_t off = (size_t)(row0 + rsub) * ep.N + col;
            const uint32_t rows = col < ep.N && row0 + rsub < ep.M ? (ep.M - row0 - rsub + 3) / 4 : 0u;      // this lane's, of eight
#pragma unroll 4
            for (uint32_t i = 0; i < 8; ++i, off += (size_t)4 * ep.N) {
                const uint32_t lr = i * 4 + rsub;
                if (i < rows) put4(ep, off, col, true, add4(tb4[lr * 8 + (cc ^ (lr & 7))], bz));
            }
            __syncwarp();
        };
        for (uint32_t u = first; u < ha.units && ok; u += step) {
            const Unit t = unit_at(u);
            const uint32_t nchunks = (t.nkb + kChunkKB - 1) / kChunkKB;
            // a lane holds the bias of one column per block: it is here long before the sums are
            float bias[CPT / 32];
            if constexpr (!SHARES) {
#pragma unroll
                for (int gr = 0; gr < CPT / 32; ++gr) bias[gr] = bias_at(t.n0 + half * CPT + gr * 32 + lane);
            }
            float sum[CPT];
#pragma unroll
            for (int j = 0; j < CPT; ++j) sum[j] = 0.0f;
            for (uint32_t c = 0; c < nchunks; ++c, ++gc) {
                const uint32_t buf = gc & 1u;
                bool got = mbar_wait_bounded(acc_full_bar(buf), (gc >> 1) & 1u, kWaitCycles + kWaitCycles / 2);
                got = __all_sync(0xffffffffu, got);
                if (!got) {
                    if (lane == 0) atomicOr(ha.dev_status, FG_DEVERR_EPI_WAIT);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN + half * CPT;
#pragma unroll
                for (int gr = 0; gr < CPT / 32; ++gr) {
                    uint32_t r[32];
                    tmem_ld_32x32(t0 + gr * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[gr * 32 + j] += __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty_bar(buf));
            }
            if (!ok) break;
            if constexpr (SHARES) {
                // Every load and MMA of this CTA has finished (its last chunk is complete), so the stages are free: the share's
                // sums as [row][BN], float4 c of a row at c ^ (row & 7).
                float4* const part = reinterpret_cast<float4*>(base_ptr) + (q * 32 + lane) * (BN / 4);
#pragma unroll
                for (int c = 0; c < CPT / 4; ++c)
                    part[(half * (CPT / 4) + c) ^ (lane & 7)] = make_float4(sum[4 * c], sum[4 * c + 1], sum[4 * c + 2], sum[4 * c + 3]);
            } else {
#pragma unroll
                for (int gr = 0; gr < CPT / 32; ++gr) {
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        tb4[lane * 8 + (c ^ (lane & 7))] = make_float4(sum[gr * 32 + 4 * c], sum[gr * 32 + 4 * c + 1], sum[gr * 32 + 4 * c + 2], sum[gr * 32 + 4 * c + 3]);
                    __syncwarp();
                    const uint32_t row0 = t.m0 + q * 32, col0 = t.n0 + half * CPT + gr * 32;
                    if (!TWO || t.p == 0) store_block(ha.ep[0], row0, col0, bias[gr]);
                    else store_block(ha.ep[1], row0, col0, bias[gr]);
                }
            }
        }
        if constexpr (SHARES) {
            __syncwarp();
            cluster_sync_all();      // every share's sums are in its CTA's shared memory
            if (go) {
                // This CTA's 32 x 32 blocks are every split-th of the tile, from its share's number on; a warp takes four rows of
                // one, a lane four columns of a row.
                const Unit t = unit_at(first);
                auto fold = [&](const Epilogue& ep) {
                    for (uint32_t v = warp - Cfg::kEpi0, b; (b = share + split * (v >> 3)) < 4 * (BN / 32); v += 8) {
                        const uint32_t lr = (b & 3u) * 32 + (v & 7u) * 4 + rsub, c0 = (b >> 2) * 32, row = t.m0 + lr, col = t.n0 + c0 + cc * 4;
                        const uint32_t at = base + ((lr * (BN / 4) + (((c0 >> 2) + cc) ^ (lr & 7))) << 4);
                        float4 z[8];
#pragma unroll
                        for (uint32_t r = 0; r < 8; ++r)
                            if (r < split) z[r] = ld_cluster_f4(map_to_cta(at, r));
                        float bz[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) bz[j] = bias_at(col + j);
#pragma unroll
                        for (uint32_t r = 1; r < 8; ++r)        // in the order of the shares, whoever adds them
                            if (r < split) z[0] = add4(z[0], z[r]);
                        if (col < ep.N && row < ep.M)
                            put4(ep, (size_t)row * ep.N + col, col, vec_ok(ep), add4(z[0], make_float4(bz[0], bz[1], bz[2], bz[3])));
                        __syncwarp();
                    }
                };
                if (!TWO || t.p == 0) fold(ha.ep[0]);
                else fold(ha.ep[1]);
            }
            __syncwarp();
            cluster_sync_all();      // no CTA leaves while another reads its sums
        }
    }
    if constexpr (SHARES) {
        if (warp < Cfg::kEpi0) { __syncwarp(); cluster_sync_all(); cluster_sync_all(); }      // as the epilogue warps
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

inline uint32_t round4(uint32_t v) { return (v + 3u) & ~3u; }
inline uint32_t round8(uint32_t v) { return (v + 7u) & ~7u; }
inline uint64_t align256(uint64_t v) { return (v + 255u) & ~uint64_t(255); }
// Scratch bytes of one operand's planes (rows x contraction k), including internal alignment.
inline uint64_t planes_bytes(int fmt, uint32_t rows, uint32_t k) {
    if (fmt == 0) return 2ull * rows * round4(k) * 4ull + 256;
    return align256((uint64_t)rows * round4(k) * 4ull) + 2ull * rows * round8(k) * 2ull + 512;
}
int32_t alloc_planes(fg_ctx* ctx, int fmt, uint32_t rows, uint32_t k, PlaneSet* out) {
    void* p;
    int32_t s = fg_ws_alloc(ctx, planes_bytes(fmt, rows, k), &p);
    if (s != FG_OK) return s;
    out->p32 = (float*)p;
    out->ld32 = round4(k);
    out->ld16 = round8(k);
    out->p16 = fmt == 0 ? nullptr
                        : (__nv_bfloat16*)((char*)p + align256((uint64_t)rows * round4(k) * 4ull));
    out->plane16 = 0;
    out->mn = false;
    return FG_OK;
}

// `chunks_out` (may be NULL) receives the number of row tiles = rows of a.colsum_part that get written.
int32_t launch_split(fg_ctx* ctx, int fmt, const SplitArgs& a, uint32_t* chunks_out = nullptr) {
    auto ok16 = [](const PlaneSet& ps) { return !ps.p32 || (fg_aligned16(ps.p32) && (!ps.p16 || fg_aligned16(ps.p16))); };
    const bool vec = (a.R % 4 == 0) && (a.C % 4 == 0) && fg_aligned16(a.x) && (!a.saved || fg_aligned16(a.saved)) &&
                     (!a.value_out || fg_aligned16(a.value_out)) && ok16(a.n) && ok16(a.t);
    const uint32_t tile = vec ? 64 : 32;
    dim3 grid((a.C + tile - 1) / tile, (a.R + tile - 1) / tile);
    if (grid.y > 65535) return fg_fail(ctx, FG_ERR_INVALID_ARGUMENT, "GEMM operand has too many rows");
    if (chunks_out) *chunks_out = grid.y;
    double bytes = 4.0 * a.R * a.C * (1.0 + (a.saved ? 1.0 : 0.0) + (a.value_out ? 1.0 : 0.0) +
                                      (a.n.p32 ? 2.0 : 0.0) + (a.t.p32 ? 2.0 : 0.0));
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SPLIT, bytes);
    if (fmt == 0) {
        if (vec) split_vec_kernel<0><<<grid, 256, 0, ctx->stream>>>(a);
        else split_kernel<0><<<grid, dim3(32, 8), 0, ctx->stream>>>(a);
    } else {
        if (vec) split_vec_kernel<1><<<grid, 256, 0, ctx->stream>>>(a);
        else split_kernel<1><<<grid, dim3(32, 8), 0, ctx->stream>>>(a);
    }
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

typedef CUresult (*pfn_encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Tensor map over planes [nplanes][rows][ld] with contraction extent `kdim`; box {bk, box_rows, nplanes}.
// The swizzle span equals the box's inner extent in bytes: 128 or 64.
// elem: 0 f32, 1 bf16, 2 f16.
int32_t make_tmap(fg_ctx* ctx, CUtensorMap* out, const void* planes, int elem, uint32_t nplanes, uint32_t rows,
                  uint32_t kdim, uint32_t ld, uint32_t box_rows, uint32_t bk) {
    if (!ctx->tmap_encode) return fg_fail(ctx, FG_ERR_UNSUPPORTED_FEATURE, "cuTensorMapEncodeTiled unavailable");
    const uint32_t esz = elem ? 2 : 4;
    cuuint64_t dims[3] = {kdim, rows, nplanes};
    cuuint64_t strides[2] = {(cuuint64_t)ld * esz, (cuuint64_t)rows * ld * esz};
    cuuint32_t box[3] = {bk, box_rows, nplanes};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapSwizzle swz = bk * esz == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    CUresult r = ((pfn_encode)ctx->tmap_encode)(out, elem == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                     : elem == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                                                3, (void*)planes, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                                swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(ctx->err, sizeof(ctx->err), "cuTensorMapEncodeTiled failed with code %d", (int)r);
        return FG_ERR_INTERNAL;
    }
    return FG_OK;
}

// General 3-D tiled map with the 128- or 64-byte swizzle (by the box's inner extent in bytes).
int32_t make_tmap3(fg_ctx* ctx, CUtensorMap* out, const void* base, int elem, uint64_t d0, uint64_t d1, uint64_t d2,
                   uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t b0, uint32_t b1, uint32_t b2, bool atom32 = false) {
    if (!ctx->tmap_encode) return fg_fail(ctx, FG_ERR_UNSUPPORTED_FEATURE, "cuTensorMapEncodeTiled unavailable");
    const uint32_t esz = elem ? 2 : 4;
    cuuint64_t dims[3] = {d0, d1, d2};
    cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
    cuuint32_t box[3] = {b0, b1, b2};
    cuuint32_t estr[3] = {1, 1, 1};
    // atom32: 32-byte chunks permuted within the 128-byte span (what an MN-major tf32 operand needs)
    const CUtensorMapSwizzle swz = atom32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B
                                   : b0 * esz == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    CUresult r = ((pfn_encode)ctx->tmap_encode)(out, elem == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                     : elem == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                                                3, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                                swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(ctx->err, sizeof(ctx->err), "cuTensorMapEncodeTiled failed with code %d", (int)r);
        return FG_ERR_INTERNAL;
    }
    return FG_OK;
}

// The two maps of one operand of the pair kernel in format 1: `rows` x `kdim` values as an f32 tensor
// (hi plane or the tensor itself) plus two bf16 planes, tile_rows rows per tile.
int32_t make_operand_maps(fg_ctx* ctx, const PlaneSet& o, uint32_t rows, uint32_t kdim, uint32_t tile_rows, CUtensorMap* t32,
                          CUtensorMap* t16) {
    const uint64_t plane16 = o.plane16 ? o.plane16 : (uint64_t)rows * o.ld16;
    int32_t s;
    if (!o.mn) {
        if ((s = make_tmap3(ctx, t32, o.p32, 0, kdim, rows, 1, (uint64_t)o.ld32 * 4, (uint64_t)rows * o.ld32 * 4, 32, tile_rows, 1)) != FG_OK) return s;
        return make_tmap3(ctx, t16, o.p16, 1, kdim, rows, 2, (uint64_t)o.ld16 * 2, plane16 * 2, 32, tile_rows, 2);
    }
    // [kdim][rows]: boxes of 128 bytes along rows x 32 values of k
    if ((s = make_tmap3(ctx, t32, o.p32, 0, rows, kdim, 1, (uint64_t)o.ld32 * 4, (uint64_t)kdim * o.ld32 * 4, 32, 32, 1, true)) != FG_OK) return s;
    return make_tmap3(ctx, t16, o.p16, 1, rows, kdim, 2, (uint64_t)o.ld16 * 2, plane16 * 2, 64, 32, 2);
}

template <int BN, int BK, int FMT>
int32_t launch_tc(fg_ctx* ctx, const PlaneSet& a, const PlaneSet& b, const Epilogue& ep) {
    using Cfg = TileCfg<BN, BK>;
    CUtensorMap tmA, tmB, tmA16, tmB16;
    int32_t s;
    if ((s = make_tmap(ctx, &tmA, a.p32, 0, FMT == 0 ? 2 : 1, ep.M, ep.K, a.ld32, BM, BK)) != FG_OK) return s;
    if ((s = make_tmap(ctx, &tmB, b.p32, 0, FMT == 0 ? 2 : 1, ep.N, ep.K, b.ld32, BN, BK)) != FG_OK) return s;
    if (FMT == 1) {
        if ((s = make_tmap(ctx, &tmA16, a.p16, 1, 2, ep.M, ep.K, a.ld16, BM, BK)) != FG_OK) return s;
        if ((s = make_tmap(ctx, &tmB16, b.p16, 1, 2, ep.N, ep.K, b.ld16, BN, BK)) != FG_OK) return s;
    } else {
        tmA16 = tmA;
        tmB16 = tmB;
    }
    // one bit per device; several host threads (one context each) may arrive here together, and setting the
    // attribute twice is harmless
    static std::atomic<uint64_t> attr_done{0};
    if (!(attr_done.load(std::memory_order_acquire) >> (ctx->device & 63) & 1ull)) {
        FG_CUDA(ctx, FG_ERR_INTERNAL,
                cudaFuncSetAttribute(gemm_tc_kernel<BN, BK, FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
        attr_done.fetch_or(1ull << (ctx->device & 63), std::memory_order_release);
    }
    dim3 grid((ep.N + BN - 1) / BN, (ep.M + BM - 1) / BM);
    if (grid.y > 65535) return fg_fail(ctx, FG_ERR_INVALID_ARGUMENT, "GEMM: M too large");
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_GEMM_TC, 2.0 * ep.M * ep.N * ep.K);
    gemm_tc_kernel<BN, BK, FMT><<<grid, kThreads, Cfg::kSmemBytes, ctx->stream>>>(tmA, tmB, tmA16, tmB16, ep);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

// Scratch the pair kernel's split-K tail may need: at most one 256x256 f32 slot per resident pair.
constexpr uint64_t kPairPartialBytes = 80ull * (2 * BM) * 256 * 4 + 256;

// How many clusters of `size` CTAs run at once; false if the runtime does not say (its error is taken off the context's thread).
template <typename Kernel>
bool cluster_query(int* n, Kernel kernel, unsigned grid, unsigned threads, size_t smem, unsigned size) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = size; attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(n, kernel, &cfg) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

// The kernel may use its shared memory, on this device (one bit per device; several host threads, one context each, may arrive here
// together, and setting the attribute twice is harmless).
template <int BK, int FMT, bool TWO>
cudaError_t pair_attr(const fg_ctx* ctx) {
    static std::atomic<uint64_t> done{0};
    if (done.load(std::memory_order_acquire) >> (ctx->device & 63) & 1ull) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(gemm_tc_pair_kernel<BK, FMT, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<BK, FMT>::kSmemBytes);
    if (e == cudaSuccess) done.fetch_or(1ull << (ctx->device & 63), std::memory_order_release);
    return e;
}
// CTA pairs that are resident at once (asked of the runtime: not every SM need be pairable), with room for the gradient exchange that
// runs beside.
template <int BK, int FMT>
uint64_t pair_slots(const fg_ctx* ctx) {
    static std::atomic<int> max_clusters[64];       // zero-initialised
    const uint64_t slots = (uint64_t)fg_asked_once(max_clusters[ctx->device & 63], ctx->sm_count / 2, [&](int* n) {
        return pair_attr<BK, FMT, false>(ctx) == cudaSuccess &&
               cluster_query(n, gemm_tc_pair_kernel<BK, FMT, false>, (unsigned)ctx->sm_count & ~1u, kPairThreads, PairCfg<BK, FMT>::kSmemBytes, 2) && *n >= 1;
    });
    return fg_free_sms(ctx) / 2 < slots ? fg_free_sms(ctx) / 2 : slots;
}
// The map of a 16-bit operand of the pair kernel, 64 values of k per k-block: boxes of `tile_rows` rows x 64 k, or 64 k x 64 rows when
// the rows are contiguous.
template <int FMT>
int32_t pair16_map(fg_ctx* ctx, CUtensorMap* t, const PlaneSet& o, uint32_t rows, uint32_t K, uint32_t tile_rows) {
    const int elem = FMT == 2 ? 1 : 2;
    if (!o.mn) return make_tmap(ctx, t, o.p16, elem, 1, rows, K, o.ld16, tile_rows, 64);
    return make_tmap3(ctx, t, o.p16, elem, rows, K, 1, (uint64_t)o.ld16 * 2, (uint64_t)K * o.ld16 * 2, 64, 64, 1);
}
// Tile rows per group of the tile order: the pairs at work at one time cover `group` tile rows, whose slabs of A
// (256 x K elements each) should stay in the L2 while the B slabs stream past.  Eight rows for long K; sixteen
// when the slabs are small (K <= 2048: the dW products of the eight-layer workload ran 5 % faster, its step
// 23.83 against 23.91 ms; on 784-4096-4096-10, all K = 4096, eight is best: 0.300 ms per launch against
// 0.302 / 0.305 / 0.307 for 12 / 16 / 4).
inline uint32_t pair_group(const fg_ctx* ctx, uint32_t K) { return ctx->opt_tile_group > 0 ? (uint32_t)ctx->opt_tile_group : (K <= 2048 ? 16u : 8u); }

template <int BK, int FMT>
int32_t launch_tc_pair(fg_ctx* ctx, const PlaneSet& a, const PlaneSet& b, const Epilogue& ep_in) {
    Epilogue ep = ep_in;
    using Cfg = PairCfg<BK, FMT>;
    CUtensorMap tmA, tmB, tmA16, tmB16;
    int32_t s;
    constexpr bool kDirect16 = FMT >= 2;
    if (kDirect16) {
        if ((s = pair16_map<FMT>(ctx, &tmA16, a, ep.M, ep.K, BM)) != FG_OK) return s;
        if ((s = pair16_map<FMT>(ctx, &tmB16, b, ep.N, ep.K, Cfg::kBN / 2)) != FG_OK) return s;
        ep.a_mn = a.mn ? 1u : 0u;
        ep.b_mn = b.mn ? 1u : 0u;
        tmA = tmA16;
        tmB = tmB16;
    } else {
        if (FMT == 1) {
            if ((s = make_operand_maps(ctx, a, ep.M, ep.K, BM, &tmA, &tmA16)) != FG_OK) return s;
            if ((s = make_operand_maps(ctx, b, ep.N, ep.K, Cfg::kBN / 2, &tmB, &tmB16)) != FG_OK) return s;
            ep.a_mn = a.mn ? 1u : 0u;
            ep.b_mn = b.mn ? 1u : 0u;
        } else {
            if ((s = make_tmap(ctx, &tmA, a.p32, 0, 2, ep.M, ep.K, a.ld32, BM, BK)) != FG_OK) return s;
            if ((s = make_tmap(ctx, &tmB, b.p32, 0, 2, ep.N, ep.K, b.ld32, Cfg::kBN / 2, BK)) != FG_OK) return s;
            tmA16 = tmA;
            tmB16 = tmB;
        }
    }
    FG_CUDA(ctx, FG_ERR_INTERNAL, (pair_attr<BK, FMT, false>(ctx)));
    const uint64_t ntiles = (uint64_t)((ep.M + 2 * BM - 1) / (2 * BM)) * ((ep.N + Cfg::kBN - 1) / Cfg::kBN);
    if (ntiles > (1ull << 30)) return fg_fail(ctx, FG_ERR_INVALID_ARGUMENT, "GEMM: too many tiles");
    ep.group = pair_group(ctx, ep.K);
    // persistent: one CTA pair per SM pair, each walking tiles pair, pair + P, ...
    const uint64_t slots = pair_slots<BK, FMT>(ctx);
    // The last wave: `rem` tiles for `slots` pairs.  When at least two pairs are free per tile, each tail
    // tile is cut into K-shares (whole accumulation chunks, at least two per share) so that the wave
    // lasts a fraction of a tile time; the shares are folded by a second, bandwidth-bound kernel.
    const uint32_t chunk_k = kDirect16 ? 1024 : kChunkK;          // as in the kernel
    const uint32_t nchunks = (ep.K + chunk_k - 1) / chunk_k;
    const uint64_t rem = ntiles % slots;
    uint64_t split = rem ? slots / rem : 1;
    if (split > nchunks / 2) split = nchunks / 2;
    if (split > 4) split = 4;
    if (!ctx->opt_split_k) split = 1;
    ep.partial = nullptr;
    ep.t_full = (uint32_t)ntiles;
    ep.split = 1;
    if (split >= 2 && rem * split * (2 * BM) * 256 * 4 + 256 <= kPairPartialBytes) {
        void* part;
        if ((s = fg_ws_alloc(ctx, rem * split * (2 * BM) * 256 * 4, &part)) != FG_OK) return s;
        ep.partial = (float*)part;
        ep.t_full = (uint32_t)(ntiles - rem);
        ep.split = (uint32_t)split;
    }
    const uint64_t nunits = ep.t_full + (ntiles - ep.t_full) * ep.split;
    dim3 grid((unsigned)(2 * (nunits < slots ? nunits : slots)));
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_GEMM_TC, 2.0 * ep.M * ep.N * ep.K);
    PairArgs<false> pa{};
    pa.ep[0] = ep;
    gemm_tc_pair_kernel<BK, FMT, false><<<grid, kPairThreads, Cfg::kSmemBytes, ctx->stream>>>(tmA, tmB, tmA16, tmB16, pa);
    FG_LAUNCHED(ctx);
    if (ep.split > 1) {
        fg_launch(ctx, gemm_tc_fold_kernel, (unsigned)((ntiles - ep.t_full) * 64), 256, 0, ep);
        FG_LAUNCHED(ctx);
    }
    fg_time_end(ctx, tr);
    return FG_OK;
}

// ---- conversion kernel, host side ----
template <int BN> int conv_clusters(const fg_ctx* ctx, uint32_t split);
ConvPlan plan_conv(const fg_ctx* ctx, const ConvShape* sh, int n, uint64_t sms) {
    auto clusters = [&](uint32_t bn, uint32_t split) {
        return conv_clusters_beside(bn == 128 ? conv_clusters<128>(ctx, split) : conv_clusters<64>(ctx, split), sms, (uint64_t)ctx->sm_count);
    };
    if (ctx->opt_conv_bn) return conv_plan_fixed(sh, n, (uint32_t)ctx->opt_conv_bn, (uint32_t)ctx->opt_conv_split, clusters);
    return conv_plan(sh, n, sms, clusters);
}
// One product with the whole GPU: what the choice of a kernel goes by, which does not depend on a running exchange.
ConvPlan plan_conv(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, uint32_t batch) {
    const ConvShape sh{M, N, K, batch};
    return plan_conv(ctx, &sh, 1, (uint64_t)ctx->sm_count);
}
// The pair kernel for one matrix: 256 x 256 tiles on SM pairs, plus the passes that make the pairs of `prep` elements.
double pair_cycles(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, double prep_elems, int prep_launches) {
    const uint64_t pairs = (uint64_t)ctx->sm_count / 2, tiles = (uint64_t)((M + 255) / 256) * ((N + 255) / 256);
    // A tile's k-blocks, or, of a few of them, the store that they hide only partly (8192 x 2048 with k of 32 / 128 / 512: 45 / 51 / 70 us); where
    // rows of the result start off 16 bytes, four words to a lane, both (9128 x 1497 with k of 3 / 256 / 1000 113 / 119 / 195 us, 3000 x 3001 x 1000
    // 135; by the conversion kernel 61 / 79 / 164 and 110).
    const double nkb = (double)((K + 31) / 32), store = 12500.0 + nkb * 750.0;
    const double tile = N % 4 ? 45000.0 + nkb * 1300.0 : nkb * 1250.0 > store ? nkb * 1250.0 : store;
    const double whole = (double)(tiles / pairs) * tile;
    const uint64_t rem = tiles % pairs;
    double tail = rem ? tile : 0.0;
    const uint64_t nchunks = (K + kChunkK - 1) / kChunkK;
    uint64_t split = rem ? pairs / rem : 1;
    if (split > nchunks / 2) split = nchunks / 2;
    if (split > 4) split = 4;
    if (split >= 2 && ctx->opt_split_k) tail = tail / (double)split + 8000.0;
    // (512 x 512 x 512: 22 us of which the products are 9; set-up and the last tile's epilogue are the rest)
    return whole + tail + 23000.0 + prep_elems * 8.0 / 2500.0 + 3700.0 * prep_launches;
}
inline bool conv_allowed(const fg_ctx* ctx) { return ctx->opt_pairs && ctx->opt_tile_pair < 0 && ctx->tmap_encode; }

// The kernel may use its shared memory, on this device (one bit per device).
template <int BN, bool TWO, bool SHARES>
cudaError_t conv_attr(const fg_ctx* ctx) {
    static std::atomic<uint64_t> done{0};
    if (done.load(std::memory_order_acquire) >> (ctx->device & 63) & 1ull) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(gemm_tc_conv_kernel<BN, TWO, SHARES>, cudaFuncAttributeMaxDynamicSharedMemorySize, ConvCfg<BN>::kSmemBytes);
    if (e == cudaSuccess) done.fetch_or(1ull << (ctx->device & 63), std::memory_order_release);
    return e;
}
// Clusters of `split` CTAs that are resident at once (asked of the runtime, once per device: how the SMs are grouped is not
// documented); 0 if they cannot be launched.
template <int BN>
int conv_clusters(const fg_ctx* ctx, uint32_t split) {
    static std::atomic<int> known[64][9];       // zero-initialised
    return fg_asked_once(known[ctx->device & 63][split], 0, [&](int* n) {
        if (conv_attr<BN, false, true>(ctx) != cudaSuccess) { cudaGetLastError(); return false; }
        return cluster_query(n, gemm_tc_conv_kernel<BN, false, true>, split * 64, ConvCfg<BN>::kThreads, ConvCfg<BN>::kSmemBytes, split);
    });
}

// One product of a launch: its operands, their roles and the epilogue.
struct ConvProduct {
    PlaneSet a, b;
    Epilogue ep;
    uint32_t batch;
};
template <int BN>
int32_t launch_conv_bn(fg_ctx* ctx, const ConvProduct* pr, int n, uint32_t split) {
    using Cfg = ConvCfg<BN>;
    CUtensorMap tm[4];
    ConvArgs ca{};
    uint64_t units = 0;
    double flop = 0.0;
    for (int j = 0; j < n; ++j) {
        const ConvProduct& c = pr[j];
        const PlaneSet* ops[2] = {&c.a, &c.b};
        const uint32_t rows[2] = {c.ep.M, c.ep.N}, tile[2] = {(uint32_t)BM, (uint32_t)BN};
        for (int i = 0; i < 2; ++i) {
            const PlaneSet& o = *ops[i];
            const uint64_t apart = (o.batch32 ? o.batch32 : (uint64_t)(o.mn ? c.ep.K : rows[i]) * o.ld32) * 4;
            int32_t s;
            if (!o.mn) s = make_tmap3(ctx, &tm[2 * j + i], o.p32, 0, c.ep.K, rows[i], c.batch, (uint64_t)o.ld32 * 4, apart, 32, tile[i], 1);
            else s = make_tmap3(ctx, &tm[2 * j + i], o.p32, 0, rows[i], c.ep.K, c.batch, (uint64_t)o.ld32 * 4, apart, 32, 32, 1, true);
            if (s != FG_OK) return s;
        }
        ca.ep[j] = c.ep;
        ca.ep[j].a_mn = c.a.mn ? 1u : 0u;
        ca.ep[j].b_mn = c.b.mn ? 1u : 0u;
        const uint64_t tiles = (uint64_t)((c.ep.M + BM - 1) / BM) * ((c.ep.N + BN - 1) / BN);
        if (tiles > (1ull << 30) || c.batch > 65535 || units + tiles * c.batch > (1ull << 31))
            return fg_fail(ctx, FG_ERR_INVALID_ARGUMENT, "GEMM: too many tiles");
        units += tiles * c.batch;
        if (j == 0) ca.units0 = (uint32_t)units;
        flop += 2.0 * c.batch * c.ep.M * c.ep.N * c.ep.K;
    }
    if (n == 1) { tm[2] = tm[0]; tm[3] = tm[1]; }
    ca.units = (uint32_t)units;
    ca.split = split;
    ca.dev_status = ctx->dev_status;
    const uint32_t grid = (uint32_t)conv_grid(units, split, fg_free_sms(ctx));
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_GEMM_TC, flop);
    auto launch = [&](auto two, auto shares) -> int32_t {
        constexpr bool T = decltype(two)::value, S = decltype(shares)::value;
        FG_CUDA(ctx, FG_ERR_INTERNAL, (conv_attr<BN, T, S>(ctx)));
        fg_launch_cluster(ctx, gemm_tc_conv_kernel<BN, T, S>, grid, Cfg::kThreads, Cfg::kSmemBytes, split, tm[0], tm[1], tm[2], tm[3], ca);
        FG_LAUNCHED(ctx);
        return FG_OK;
    };
    const std::true_type yes{};
    const std::false_type no{};
    const int32_t s = n == 2 ? (split > 1 ? launch(yes, yes) : launch(yes, no)) : split > 1 ? launch(no, yes) : launch(no, no);
    fg_time_end(ctx, tr);
    return s;
}
inline ConvShape conv_shape(const ConvProduct& c) { return ConvShape{c.ep.M, c.ep.N, c.ep.K, c.batch}; }
int32_t launch_conv(fg_ctx* ctx, const ConvProduct* pr, int n, ConvPlan p) {
    // beside an exchange the units are split for the SMs that it leaves (n = 2 comes from launch_conv_both, which has done so)
    if (n == 1 && fg_free_sms(ctx) != (uint64_t)ctx->sm_count) {
        const ConvShape sh = conv_shape(pr[0]);
        p = plan_conv(ctx, &sh, 1, fg_free_sms(ctx));
    }
    return p.bn == 128 ? launch_conv_bn<128>(ctx, pr, n, p.split) : launch_conv_bn<64>(ctx, pr, n, p.split);
}
int32_t launch_conv(fg_ctx* ctx, const PlaneSet& a, const PlaneSet& b, const Epilogue& ep, const ConvPlan& p, uint32_t batch) {
    const ConvProduct pr{a, b, ep, batch};
    return launch_conv(ctx, &pr, 1, p);
}
// Does what `w` stores (C, and its pairs) lie over an operand of `r`?
bool stores_over(const ConvProduct& w, const ConvProduct& r) {
    auto meets = [](const void* p, uint64_t np, const void* q, uint64_t nq) {      // bytes from the first to behind the last element
        const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(q);
        return p && q && a < b + nq && b < a + np;
    };
    const uint64_t mn = (uint64_t)w.ep.M * w.ep.N, c_bytes = ((uint64_t)(w.batch - 1) * w.ep.c_batch + mn) * 4;
    const PlaneSet* const ops[2] = {&r.a, &r.b};
    const uint32_t rows[2] = {r.ep.M, r.ep.N};
    for (int i = 0; i < 2; ++i) {
        const PlaneSet& o = *ops[i];
        const uint64_t one = (uint64_t)(o.mn ? r.ep.K : rows[i]) * o.ld32, bytes = ((uint64_t)(r.batch - 1) * (o.batch32 ? o.batch32 : one) + one) * 4;
        if (meets(w.ep.C, c_bytes, o.p32, bytes) || meets(w.ep.c_pairs, (w.ep.c_pairs_stride + mn) * 2, o.p32, bytes)) return true;
    }
    return false;
}
// The two gradients of a layer in one launch: more units to share out, and one wave's end instead of two.  The longer k goes
// first, so that the short units fill the last round.  Two launches where each wants K-shares of its own (128 x 4096 x 1024: k of
// 4096 on eight tiles and of 128 on 256 of them, 60 us together, 39 apart), and where dA lies over what dB reads (the gradient of
// an activation may overwrite the activation): dB is then complete before dA is written, as on every other route.
int32_t launch_conv_both(fg_ctx* ctx, const ConvProduct& dB, const ConvProduct& dA) {
    const ConvProduct pr[2] = {dB.ep.K >= dA.ep.K ? dB : dA, dB.ep.K >= dA.ep.K ? dA : dB};
    const ConvShape sh[2] = {conv_shape(pr[0]), conv_shape(pr[1])};
    const uint64_t sms = fg_free_sms(ctx);
    const ConvPlan together = plan_conv(ctx, sh, 2, sms), one = plan_conv(ctx, sh, 1, sms), two = plan_conv(ctx, sh + 1, 1, sms);
    if (together.cycles <= one.cycles + two.cycles && !stores_over(dA, dB)) return launch_conv(ctx, pr, 2, together);
    const bool b_first = dB.ep.K >= dA.ep.K;
    const int32_t s = launch_conv(ctx, &dB, 1, b_first ? one : two);
    return s != FG_OK ? s : launch_conv(ctx, &dA, 1, b_first ? two : one);
}

// ---- the same for sixteen-bit tensors ----
// Costs fitted to 87 products under the pair kernel and every plan (2 % slower than the best of each in the geometric mean).
constexpr ConvCosts kHalfCosts = {64, {520.0, 305.0}, {600.0, 300.0}, {950.0, 1250.0}, {600.0, 300.0}, {950.0, 1250.0}, {800.0, 650.0}, 2400.0, 1600.0};
template <int BN, bool TWO, bool SHARES>
cudaError_t half_attr(const fg_ctx* ctx) {
    static std::atomic<uint64_t> done{0};
    if (done.load(std::memory_order_acquire) >> (ctx->device & 63) & 1ull) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(gemm_tc_half_kernel<BN, TWO, SHARES>, cudaFuncAttributeMaxDynamicSharedMemorySize, HalfCfg<BN>::kSmemBytes);
    if (e == cudaSuccess) done.fetch_or(1ull << (ctx->device & 63), std::memory_order_release);
    return e;
}
template <int BN>
int half_clusters(const fg_ctx* ctx, uint32_t split) {
    static std::atomic<int> known[64][9];       // zero-initialised
    return fg_asked_once(known[ctx->device & 63][split], 0, [&](int* n) {
        if (half_attr<BN, false, true>(ctx) != cudaSuccess) { cudaGetLastError(); return false; }
        return cluster_query(n, gemm_tc_half_kernel<BN, false, true>, split * 64, HalfCfg<BN>::kThreads, HalfCfg<BN>::kSmemBytes, split);
    });
}
ConvPlan plan_half(const fg_ctx* ctx, const ConvShape* sh, int n) {
    const uint64_t sms = fg_free_sms(ctx);
    auto clusters = [&](uint32_t bn, uint32_t split) {
        return conv_clusters_beside(bn == 128 ? half_clusters<128>(ctx, split) : half_clusters<64>(ctx, split), sms, (uint64_t)ctx->sm_count);
    };
    if (ctx->opt_conv_bn) return conv_plan_fixed(sh, n, (uint32_t)ctx->opt_conv_bn, (uint32_t)ctx->opt_conv_split, clusters, kHalfCosts.kblock);
    return conv_plan(sh, n, sms, clusters, kHalfCosts);
}
template <int BN>
int32_t launch_half_bn(fg_ctx* ctx, const ConvProduct* pr, int n, uint32_t split) {
    using Cfg = HalfCfg<BN>;
    CUtensorMap tm[4];
    HalfArgs ha{};
    uint64_t units = 0;
    double flop = 0.0;
    for (int j = 0; j < n; ++j) {
        const ConvProduct& c = pr[j];
        const PlaneSet* ops[2] = {&c.a, &c.b};
        const uint32_t rows[2] = {c.ep.M, c.ep.N}, tile[2] = {(uint32_t)BM, (uint32_t)BN};
        const int elem = c.ep.out_dtype == FG_DTYPE_BF16 ? 1 : 2;
        for (int i = 0; i < 2; ++i) {
            const PlaneSet& o = *ops[i];
            const int32_t s = !o.mn ? make_tmap(ctx, &tm[2 * j + i], o.p16, elem, 1, rows[i], c.ep.K, o.ld16, tile[i], 64)
                                    : make_tmap3(ctx, &tm[2 * j + i], o.p16, elem, rows[i], c.ep.K, 1, (uint64_t)o.ld16 * 2, (uint64_t)c.ep.K * o.ld16 * 2, 64, 64, 1);
            if (s != FG_OK) return s;
        }
        ha.ep[j] = c.ep;
        ha.ep[j].a_mn = c.a.mn ? 1u : 0u;
        ha.ep[j].b_mn = c.b.mn ? 1u : 0u;
        units += (uint64_t)((c.ep.M + BM - 1) / BM) * ((c.ep.N + BN - 1) / BN);
        if (units > (1ull << 28)) return fg_fail(ctx, FG_ERR_INVALID_ARGUMENT, "GEMM: too many tiles");
        if (j == 0) ha.units0 = (uint32_t)units;
        flop += 2.0 * c.ep.M * c.ep.N * c.ep.K;
    }
    if (n == 1) { tm[2] = tm[0]; tm[3] = tm[1]; }
    ha.units = (uint32_t)units;
    ha.split = split;
    ha.dev_status = ctx->dev_status;
    const uint32_t grid = (uint32_t)conv_grid(units, split, fg_free_sms(ctx));
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_GEMM_TC, flop);
    auto launch = [&](auto two, auto shares) -> int32_t {
        constexpr bool T = decltype(two)::value, S = decltype(shares)::value;
        FG_CUDA(ctx, FG_ERR_INTERNAL, (half_attr<BN, T, S>(ctx)));
        fg_launch_cluster(ctx, gemm_tc_half_kernel<BN, T, S>, grid, Cfg::kThreads, Cfg::kSmemBytes, split, tm[0], tm[1], tm[2], tm[3], ha);
        FG_LAUNCHED(ctx);
        return FG_OK;
    };
    const std::true_type yes{};
    const std::false_type no{};
    const int32_t s = n == 2 ? (split > 1 ? launch(yes, yes) : launch(yes, no)) : split > 1 ? launch(no, yes) : launch(no, no);
    fg_time_end(ctx, tr);
    return s;
}
int32_t launch_half(fg_ctx* ctx, const ConvProduct* pr, int n, const ConvPlan& p) {
    return p.bn == 128 ? launch_half_bn<128>(ctx, pr, n, p.split) : launch_half_bn<64>(ctx, pr, n, p.split);
}
// The pair kernel on 16-bit tensors by the same fit: tiles of 256 x 256, K-shares of 2048 or more in the last wave.
constexpr double kPair16Around = 26600.0;
uint64_t pair_tiles(const ConvShape& sh) { return (uint64_t)((sh.M + 255) / 256) * ((sh.N + 255) / 256); }
double pair16_tile(const ConvShape& sh) {
    const double kb = (double)((sh.K + 63) / 64) * 395.0;
    return kb > 2500.0 ? kb : 2500.0;
}
double pair16_cycles(const fg_ctx* ctx, const ConvShape& sh) {
    const uint64_t pairs = fg_free_sms(ctx) / 2, tiles = pair_tiles(sh);
    const double tile = pair16_tile(sh), whole = (double)(tiles / pairs) * tile;
    const uint64_t rem = tiles % pairs, nchunks = (sh.K + 1023) / 1024;
    double tail = rem ? tile : 0.0;
    uint64_t split = rem ? pairs / rem : 1;
    if (split > nchunks / 2) split = nchunks / 2;
    if (split > 4) split = 4;
    if (split >= 2 && ctx->opt_split_k) tail = tail / (double)split + 3300.0;
    return whole + tail + kPair16Around;
}

// A dense [R, C] f32 tensor (`batch` of them, x_batch apart) can be loaded as it lies when rows and matrices start on
// 16-byte boundaries; otherwise from a padded copy (loadable32 leaves it to `prep`).
inline bool in_place32(const float* x, uint32_t C, uint32_t batch, uint64_t x_batch) {
    return fg_aligned16(x) && C % 4 == 0 && (batch == 1 || x_batch % 4 == 0);
}
inline uint64_t copy32_bytes(const float* x, uint32_t R, uint32_t C, uint32_t batch, uint64_t x_batch) {
    return in_place32(x, C, batch, x_batch) ? 0 : (uint64_t)batch * R * round4(C) * 4 + 256;
}
int32_t loadable32(fg_ctx* ctx, const float* x, uint32_t R, uint32_t C, uint32_t batch, uint64_t x_batch, PlaneSet* o, PrepBatch* prep) {
    *o = PlaneSet{};
    o->p32 = const_cast<float*>(x);
    o->ld32 = C;
    o->batch32 = batch > 1 ? x_batch : 0;      // one matrix: its stride need not suit a tensor map
    if (in_place32(x, C, batch, x_batch)) return FG_OK;
    void* p;
    int32_t s = fg_ws_alloc(ctx, (uint64_t)batch * R * round4(C) * 4, &p);
    if (s != FG_OK) return s;
    PrepArgs a{};
    a.x = x; a.R = R; a.C = C; a.x_batch = x_batch; a.out = p; a.ld = round4(C);
    o->p32 = (float*)p;
    o->ld32 = a.ld;
    o->batch32 = (uint64_t)R * a.ld;
    return prep->add(ctx, FG_DTYPE_F32, a, batch);
}
inline PlaneSet as_operand(PlaneSet o, bool mn) { o.mn = mn; return o; }

// C[M,N] = act(Aop·Bopᵀ + bias) where the A operand's planes have M rows and the B operand's N rows.
int32_t tc_gemm(fg_ctx* ctx, int fmt, const PlaneSet& a, const PlaneSet& b, uint32_t M, uint32_t N, uint32_t K, float* C,
                const float* bias, int act, float* preact) {
    Epilogue ep{C, bias, preact, M, N, K, act, ctx->dev_status};
    // Tile choice: one output tile per CTA (or per CTA pair), so the last wave is often part empty.
    // Each candidate is scored by machine fill times its measured relative throughput at 8192^3
    // (hybrid planes: pair 316, 128x256 248, 128x128 ~215 TFLOP/s; hi/lo planes: 262, 260, 217).
    const uint64_t sms = (uint64_t)ctx->sm_count, mt = (M + BM - 1) / BM;
    auto fill = [](uint64_t tiles, uint64_t slots) { return (double)tiles / (double)(((tiles + slots - 1) / slots) * slots); };
    const uint64_t t256 = mt * ((N + 255) / 256), t128 = mt * ((N + 127) / 128);
    const uint64_t tpair = (uint64_t)((M + 2 * BM - 1) / (2 * BM)) * ((N + 255) / 256);
    const double s_pair = (N > 128 && M > BM) ? fill(tpair, sms / 2) * 1.0 : 0.0;
    const double s_256 = N > 128 ? fill(t256, sms) * (fmt == 1 ? 0.78 : 0.98) : 0.0;
    const double s_128 = N > 64 ? fill(t128, sms) * (fmt == 1 ? 0.68 : 0.83) : 0.0;
    int bn = N > 128 ? (s_256 >= s_128 ? 256 : 128) : N > 64 ? 128 : N > 32 ? 64 : 32;
    int bk = (fmt == 0 && bn == 256) ? 16 : 32;
    bool pair = s_pair > 0.0 && s_pair >= s_256 && s_pair >= s_128;
    // Option gemm_tile: "pair" or "<BN>x<BK>" instead of the choice above.
    if (ctx->opt_tile_pair == 1) pair = N > 128;
    else if (ctx->opt_tile_pair == 0 && (ctx->opt_tile_bk == 32 || fmt == 0)) {
        bn = ctx->opt_tile_bn; bk = ctx->opt_tile_bk; pair = false;
    }
    if (pair) return fmt == 1 ? launch_tc_pair<32, 1>(ctx, a, b, ep) : launch_tc_pair<32, 0>(ctx, a, b, ep);
    if (fmt == 1) {
        if (bn == 256) return launch_tc<256, 32, 1>(ctx, a, b, ep);
        if (bn == 128) return launch_tc<128, 32, 1>(ctx, a, b, ep);
        if (bn == 64) return launch_tc<64, 32, 1>(ctx, a, b, ep);
        return launch_tc<32, 32, 1>(ctx, a, b, ep);
    }
    if (bn == 256 && bk == 16) return launch_tc<256, 16, 0>(ctx, a, b, ep);
    if (bn == 128 && bk == 16) return launch_tc<128, 16, 0>(ctx, a, b, ep);
    if (bn == 256) return launch_tc<256, 32, 0>(ctx, a, b, ep);
    if (bn == 128) return launch_tc<128, 32, 0>(ctx, a, b, ep);
    if (bn == 64) return launch_tc<64, 32, 0>(ctx, a, b, ep);
    return launch_tc<32, 32, 0>(ctx, a, b, ep);
}

// ------------------------------------------------------------------------------------
// f32 tensors with bf16 pairs: the pair kernel multiplies the tensors as they lie in HBM.
// The kind::tf32 MMA reads the f32 words themselves (it uses sign, exponent and the top 10
// mantissa bits: hi = trunc(x)); the two cross terms of the split product come from two
// bf16 planes of the same shape and layout, pairs[0] = bf16(x), pairs[1] = bf16(x - trunc(x)).
// An operand whose contraction index is not the contiguous one is read through MN-major
// descriptors, so nothing is ever transposed, and whoever produces a tensor (a GEMM
// epilogue, the optimizer, the kernels below) writes its pairs in the same pass.
// ------------------------------------------------------------------------------------
// (VEC: x starts on 16 bytes)
template <bool VEC>
__global__ void __launch_bounds__(256) pairs_kernel(const float* __restrict__ x, uint64_t n, __nv_bfloat16* __restrict__ pairs,
                                                    uint64_t plane_stride) {
    fg_grid_enter();
    const uint64_t nv = VEC ? n >> 2 : 0, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += stride)
        fg_store_pairs4(pairs, plane_stride, i * 4, __ldcs(reinterpret_cast<const float4*>(x) + i));
    for (uint64_t i = (nv << 2) + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        fg_store_pairs1(pairs, plane_stride, i, x[i]);
}

// dz = dy * act'(saved) over [R, C] with its pairs and the column sums of each 32-row block (the bias
// gradient's partials), in one pass.  A block covers 32 rows x 512 columns; a thread owns four columns.
// dz may alias dy.  Needs C % 4 == 0 and 16-byte aligned pointers.
__global__ void __launch_bounds__(128) dz_pairs_kernel(uint32_t R, uint32_t C, const float* dy, const float* __restrict__ saved,
                                                       int act, float* dz, __nv_bfloat16* __restrict__ pairs,
                                                       uint64_t plane_stride, float* __restrict__ colsum_part) {
    fg_grid_enter();
    const uint32_t c = (blockIdx.x * 128 + threadIdx.x) * 4;
    if (c >= C) return;
    const uint32_t r0 = blockIdx.y * 32, r1 = min(R, r0 + 32);
    float4 cs = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (uint32_t r = r0; r < r1; ++r) {
        const size_t off = (size_t)r * C + c;
        float4 v = __ldcs(reinterpret_cast<const float4*>(dy + off));
        if (saved) v = act_mul4(act, v, __ldcs(reinterpret_cast<const float4*>(saved + off)));
        if (dz) *reinterpret_cast<float4*>(dz + off) = v;
        if (pairs) fg_store_pairs4(pairs, plane_stride, off, v);
        cs.x += v.x; cs.y += v.y; cs.z += v.z; cs.w += v.w;
    }
    if (colsum_part) *reinterpret_cast<float4*>(colsum_part + (size_t)blockIdx.y * C + c) = cs;
}

int32_t launch_pairs(fg_ctx* ctx, const float* x, uint64_t n, __nv_bfloat16* pairs, uint64_t plane_stride) {
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SPLIT, 8.0 * (double)n);
    if (fg_aligned16(x)) fg_launch(ctx, pairs_kernel<true>, fg_stream_grid(ctx, (n + 3) / 4, 256, 8), 256, 0, x, n, pairs, plane_stride);
    else fg_launch(ctx, pairs_kernel<false>, fg_stream_grid(ctx, n, 256, 8), 256, 0, x, n, pairs, plane_stride);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

int32_t launch_dz_pairs(fg_ctx* ctx, uint32_t R, uint32_t C, const float* dy, const float* saved, int act, float* dz,
                        __nv_bfloat16* pairs, uint64_t plane_stride, float* colsum_part) {
    dim3 grid((C + 511) / 512, (R + 31) / 32);
    if (grid.y > 65535) return fg_fail(ctx, FG_ERR_INVALID_ARGUMENT, "GEMM operand has too many rows");
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SPLIT, 4.0 * R * C * (1.0 + (saved ? 1.0 : 0.0) + (dz ? 1.0 : 0.0) + (pairs ? 1.0 : 0.0)));
    fg_launch(ctx, dz_pairs_kernel, grid, 128, 0, R, C, dy, saved, act, dz, pairs, plane_stride, colsum_part);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

// A dense row-major f32 tensor [R, C] and its pairs as an operand of the pair kernel.  `contract_cols`:
// the contraction runs over the columns (K-major), otherwise over the rows (MN-major).
PlaneSet paired_operand(const float* x, const void* pairs, uint64_t plane_stride, uint32_t C, bool contract_cols) {
    PlaneSet o{};
    o.p32 = const_cast<float*>(x);
    o.p16 = (__nv_bfloat16*)pairs;
    o.ld32 = o.ld16 = C;
    o.plane16 = plane_stride;
    o.mn = !contract_cols;
    return o;
}

// Can [M,N] = [M,K] x [K,N] run on the pair kernel straight from f32 tensors and their pairs?  Every
// tensor's row pitch must be a multiple of 16 bytes in both element sizes (columns % 8), and the tile
// shape must suit the pair kernel.
bool paired_shape_ok(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, uint32_t pitch_a, uint32_t pitch_b) {
    return ctx->opt_pairs && ctx->opt_tile_pair != 0 && ctx->tmap_encode && M > (uint32_t)BM && N > 128 && K >= 32 &&
           pitch_a % 8 == 0 && pitch_b % 8 == 0;
}

struct PairedOut {
    __nv_bfloat16* pairs;     // optional pairs of the result
    uint64_t stride;
    const float* mul_saved;   // optional: result = (acc + bias) * act'(mul_saved)
    int mul_act;
    float* colsum_part;       // optional [ceil(M/32)][N]
};

int32_t paired_gemm(fg_ctx* ctx, const PlaneSet& a, const PlaneSet& b, uint32_t M, uint32_t N, uint32_t K, float* C,
                    const float* bias, int act, float* preact, const PairedOut& o) {
    Epilogue ep{C, bias, preact, M, N, K, act, ctx->dev_status};
#ifdef FG_GEMM_PROFILE
    if (const char* e = getenv("FG_GEMM_DBG")) ep.dbg = (uint32_t)atoi(e);
#endif
    ep.c_pairs = o.pairs;
    ep.c_pairs_stride = o.stride;
    ep.mul_saved = o.mul_saved;
    ep.mul_act = o.mul_act;
    ep.colsum_part = o.colsum_part;
    return launch_tc_pair<32, 1>(ctx, a, b, ep);
}

// How one tensor-core product of f32 tensors [M,K] x [K,N] runs: operand planes written by a pre-pass (any shape), the pair
// kernel on tensors with their pairs, or the conversion kernel on the tensors alone.
enum { kRoutePlanes = 0, kRoutePair = 1, kRouteConv = 2 };
struct Route {
    int kind;
    ConvPlan conv;
};
// pair_ok: the pair kernel can read the operands as they lie.  missing / missing_n: elements and tensors whose pairs would
// have to be made for it.  copied / copied_n: the same for the padded copies the conversion kernel would need.
Route pick_route(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, bool pair_ok, double missing, int missing_n, double copied, int copied_n) {
    Route r{pair_ok ? (int)kRoutePair : (int)kRoutePlanes, ConvPlan{}};
    if (!conv_allowed(ctx)) return r;
    r.conv = plan_conv(ctx, M, N, K, 1);
    // (beside the pair kernel's, the time of several units on every SM is 8 % short: 8192 x 2048 x 512 76 us, by the pair kernel 70, dB of 1500 x 2048 x
    // 2048 60 and 49)
    const bool several = r.conv.split == 1 && (uint64_t)((M + BM - 1) / BM) * ((N + r.conv.bn - 1) / r.conv.bn) > (uint64_t)ctx->sm_count;
    const double conv = r.conv.cycles * (pair_ok && several ? 1.08 : 1.0) + copied * 8.0 / 2500.0 + 4000.0 * copied_n;
    // planes: both operands read and written twice over, transposed on the way, then 256 x 256 or 128-row tiles
    const double other = pair_ok ? pair_cycles(ctx, M, N, K, missing, missing_n)
                       : M > (uint32_t)BM && N > 128 ? pair_cycles(ctx, M, N, K, 2.0 * ((double)M * K + (double)N * K), 2) : 1e30;
    if (conv <= other || ctx->opt_conv_bn) r.kind = kRouteConv;
    return r;
}

// Which path a request takes: 0 = plain f32 FMAs (the exact path, or with FG_GEMM_AUTO the FMA kernel or the narrow layer's), otherwise the
// plane format + 1.
int pick_path(const fg_ctx* ctx, int mode, uint32_t M, uint32_t N, uint32_t K) {
    if (mode == FG_GEMM_SIMT) return 0;
    if (mode == FG_GEMM_3XTF32) return 1;
    if (mode == FG_GEMM_TF32_BF16X2) return 2;
    if (!ctx->tmap_encode) return 0;
    if (!(M >= 64 && (uint64_t)M * N * K >= (1ull << 22))) return 0;
    return 2;   // AUTO: tf32 main term + bf16 cross terms (same accuracy class, two thirds of the tensor work)
}

// Does FG_GEMM_AUTO take the FMA kernel for the forward product, or for one or both gradients?  (An option that names a tensor-core
// kernel keeps what those can run; gemm_fwd_core keeps the forward products of a short k for the exact path's kernel.)
bool takes_fma(const fg_ctx* ctx, int mode, uint32_t M, uint32_t N, uint32_t K, int products) {
    if (mode != FG_GEMM_AUTO) return false;
    if (pick_path(ctx, mode, M, N, K) == 0) return fg_gemm_fma_suits_small(M, N, K, products);
    return (conv_allowed(ctx) && !ctx->opt_conv_bn && fg_gemm_fma_suits(M, N, K, products & (kFgGradB | kFgGradA)));
}
// Are a layer's gradients the narrow layer's kernels'?  (Of small products with more rows than the pass over dZ always takes, 65535 tiles
// of 32, the FMA kernel's after all.)
bool takes_narrow(const fg_ctx* ctx, int mode, uint32_t M, uint32_t N, uint32_t K, int products) {
    if (mode != FG_GEMM_AUTO || N > 16) return false;
    return pick_path(ctx, mode, M, N, K) != 0 || (M <= 65535u * 32u && products && !fg_gemm_fma_suits_small(M, N, K, products));
}
int grad_products(const float* dA, const float* dB, const float* dbias, bool fuse) {
    return (dB ? kFgGradB : 0) | (dA ? kFgGradA : 0) | (dbias ? kFgBias : 0) | (fuse ? kFgFactor : 0);
}
// Scratch of the narrow layer's backward pass.  A small product that finds no room for it (a recording whose arena was sized for less) keeps
// to the kernels that need less.
uint64_t narrow_bwd_need(uint32_t M, uint32_t N, uint32_t K, bool dbias) {
    return 2048 + (uint64_t)M * N * 4 + 256 + fg_gemm_skinny_scratch_bytes(M, N, K) + (dbias ? (uint64_t)((M + 31) / 32) * N * 4 + 256 : 0);
}
bool runs_narrow(fg_ctx* ctx, int mode, uint32_t M, uint32_t N, uint32_t K, int products) {
    return takes_narrow(ctx, mode, M, N, K, products) &&
           (pick_path(ctx, mode, M, N, K) != 0 || fg_ws_try(ctx, narrow_bwd_need(M, N, K, (products & kFgBias) != 0)));
}

}  // namespace

namespace {

struct PairedArg {
    const float* x;
    const void* pairs;      // NULL: made on the fly in the scratch arena
    uint64_t stride;
};

// Forward product with every way of running it.  c_pairs (optional) receives the pairs of C.
int32_t gemm_fwd_core(fg_ctx* ctx, int32_t mode, int32_t transA, int32_t transB, uint32_t M, uint32_t N, uint32_t K,
                      PairedArg A, PairedArg B, float* C, const float* bias, int32_t act, float* preact_out,
                      __nv_bfloat16* c_pairs, uint64_t c_stride) {
    const uint64_t mn = (uint64_t)M * N;
    const int path = pick_path(ctx, mode, M, N, K);
    // The result's pairs, when no GEMM epilogue wrote them.
    auto pairs_after = [&]() -> int32_t { return c_pairs ? launch_pairs(ctx, C, mn, c_pairs, c_stride) : FG_OK; };
    const bool short_k = path == 0 && mode == FG_GEMM_AUTO && !c_pairs && fg_gemm_simt_suits(M, N, K);
    if (!short_k && takes_fma(ctx, mode, M, N, K, kFgForward)) {
        FgFmaOp o{};
        o.ta = transA; o.tb = transB; o.M = M; o.N = N; o.K = K; o.A = A.x; o.B = B.x; o.C = C;
        o.bias = bias; o.act = act; o.preact = preact_out; o.pairs = c_pairs; o.pairs_stride = c_stride;
        return fg_gemm_fma_launch(ctx, &o, 1, 1, false);
    }
    if (path == 0) {
        int32_t s = fg_gemm_simt_launch(ctx, transA, transB, M, N, K, A.x, B.x, C, bias, act, preact_out);
        return s != FG_OK ? s : pairs_after();
    }
    // A skinny output (say 10 classes) is bandwidth-bound on reading A once: no pre-pass, no tensor cores.
    if (mode == FG_GEMM_AUTO && N <= 16 && !transA && !transB) {
        const uint64_t need = fg_gemm_skinny_scratch_bytes(M, N, K) + 1024;
        { int32_t s0 = fg_ws_ensure(ctx, need); if (s0 != FG_OK) return s0; }
        int32_t s = fg_gemm_skinny_n_launch(ctx, M, N, K, A.x, B.x, C, bias, act, preact_out);
        return s != FG_OK ? s : pairs_after();
    }
    const int fmt = path - 1;
    const uint32_t pitch_a = transA ? M : K, pitch_b = transB ? K : N, rows_a = transA ? K : M, rows_b = transB ? N : K;
    const bool aligned = fg_aligned16(A.x) && fg_aligned16(B.x) && fg_aligned16(C) && (!preact_out || fg_aligned16(preact_out));
    const bool pair_ok = fmt == 1 && aligned && paired_shape_ok(ctx, M, N, K, pitch_a, pitch_b) && N % 4 == 0;
    if (fmt == 1) {
        const uint64_t ca = copy32_bytes(A.x, rows_a, pitch_a, 1, 0), cb = copy32_bytes(B.x, rows_b, pitch_b, 1, 0);
        const Route r = pick_route(ctx, M, N, K, pair_ok, (A.pairs ? 0.0 : (double)M * K) + (B.pairs ? 0.0 : (double)K * N), !A.pairs + !B.pairs,
                                   (ca ? (double)M * K : 0.0) + (cb ? (double)K * N : 0.0), (ca != 0) + (cb != 0));
        if (r.kind == kRouteConv) {
            int32_t s = fg_ws_ensure(ctx, ca + cb + 1024);
            if (s != FG_OK) return s;
            PlaneSet pa, pb;
            PrepBatch prep;
            if ((s = loadable32(ctx, A.x, rows_a, pitch_a, 1, 0, &pa, &prep)) != FG_OK) return s;
            if ((s = loadable32(ctx, B.x, rows_b, pitch_b, 1, 0, &pb, &prep)) != FG_OK) return s;
            if ((s = prep.launch(ctx)) != FG_OK) return s;
            Epilogue ep{C, bias, preact_out, M, N, K, act, ctx->dev_status};
            ep.c_pairs = c_pairs;
            ep.c_pairs_stride = c_stride;
            // A operand: rows = M, B operand: rows = N; the contraction runs along the columns of [M,K] and of [N,K]
            return launch_conv(ctx, as_operand(pa, transA != 0), as_operand(pb, transB == 0), ep, r.conv, 1);
        }
    }
    if (pair_ok) {
        // The tensors themselves are the operands; pairs the caller does not keep are made here (8 bytes
        // of traffic per element, no transposition).
        const uint64_t mk = (uint64_t)M * K, kn = (uint64_t)K * N;
        const uint64_t need = (A.pairs ? 0 : mk * 4 + 256) + (B.pairs ? 0 : kn * 4 + 256) + kPairPartialBytes + 1024;
        { int32_t s0 = fg_ws_ensure(ctx, need); if (s0 != FG_OK) return s0; }
        int32_t s;
        void* p;
        if (!A.pairs) {
            if ((s = fg_ws_alloc(ctx, mk * 4, &p)) != FG_OK) return s;
            if ((s = launch_pairs(ctx, A.x, mk, (__nv_bfloat16*)p, mk)) != FG_OK) return s;
            A.pairs = p; A.stride = mk;
        }
        if (!B.pairs) {
            if ((s = fg_ws_alloc(ctx, kn * 4, &p)) != FG_OK) return s;
            if ((s = launch_pairs(ctx, B.x, kn, (__nv_bfloat16*)p, kn)) != FG_OK) return s;
            B.pairs = p; B.stride = kn;
        }
        // A operand: rows = M; stored [M,K] (contraction along columns) or, transposed, [K,M].
        const PlaneSet pa = paired_operand(A.x, A.pairs, A.stride, pitch_a, !transA);
        // B operand: rows = N; stored [K,N] (contraction along rows) or, transposed, [N,K].
        const PlaneSet pb = paired_operand(B.x, B.pairs, B.stride, pitch_b, transB != 0);
        return paired_gemm(ctx, pa, pb, M, N, K, C, bias, act, preact_out, PairedOut{c_pairs, c_stride, nullptr, 0, nullptr});
    }
    // Operand planes written by a pre-pass (any shape and alignment; the strict 3xTF32 mode).
    const uint64_t need = planes_bytes(fmt, M, K) + planes_bytes(fmt, N, K) + kPairPartialBytes + 1024;
    { int32_t s0 = fg_ws_ensure(ctx, need); if (s0 != FG_OK) return s0; }
    PlaneSet pa{}, pb{};
    int32_t s;
    if ((s = alloc_planes(ctx, fmt, M, K, &pa)) != FG_OK) return s;
    if ((s = alloc_planes(ctx, fmt, N, K, &pb)) != FG_OK) return s;
    // A operand: [M, K] with K contiguous.
    SplitArgs sa{};
    sa.x = A.x;
    if (!transA) { sa.R = M; sa.C = K; sa.n = pa; }
    else         { sa.R = K; sa.C = M; sa.t = pa; }
    if ((s = launch_split(ctx, fmt, sa)) != FG_OK) return s;
    // B operand: [N, K] with K contiguous.
    SplitArgs sb{};
    sb.x = B.x;
    if (!transB) { sb.R = K; sb.C = N; sb.t = pb; }
    else         { sb.R = N; sb.C = K; sb.n = pb; }
    if ((s = launch_split(ctx, fmt, sb)) != FG_OK) return s;
    if ((s = tc_gemm(ctx, fmt, pa, pb, M, N, K, C, bias, act, preact_out)) != FG_OK) return s;
    return pairs_after();
}

}  // namespace

extern "C" {

int32_t fg_gemm_f32(fg_ctx* ctx, int32_t mode, int32_t transA, int32_t transB, uint32_t M, uint32_t N, uint32_t K,
                    const float* A, const float* B, float* C, const float* bias, int32_t act, float* preact_out) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, A && B && C, "fg_gemm_f32: NULL operand");
    FG_REQUIRE(ctx, M >= 1 && N >= 1 && K >= 1, "fg_gemm_f32: dimensions must be >= 1");
    FG_REQUIRE(ctx, mode >= FG_GEMM_AUTO && mode <= FG_GEMM_TF32_BF16X2, "fg_gemm_f32: unknown mode");
    FG_REQUIRE(ctx, act >= FG_ACT_NONE && act <= FG_ACT_GELU, "fg_gemm_f32: unknown activation");
    FG_REQUIRE(ctx, (uint64_t)M * N < (1ull << 40) && (uint64_t)M * K < (1ull << 40) && (uint64_t)N * K < (1ull << 40),
               "fg_gemm_f32: operand too large");
    return gemm_fwd_core(ctx, mode, transA, transB, M, N, K, PairedArg{A, nullptr, 0}, PairedArg{B, nullptr, 0}, C, bias, act,
                         preact_out, nullptr, 0);
}

int32_t fg_pairs_from_f32(fg_ctx* ctx, const float* x, uint64_t n, void* pairs, uint64_t plane_stride) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, x && pairs, "fg_pairs_from_f32: NULL pointer");
    FG_REQUIRE(ctx, fg_aligned16(x) && fg_aligned16(pairs) && plane_stride % 8 == 0 && plane_stride >= n,
               "fg_pairs_from_f32: pointers must be 16-byte aligned, the plane stride a multiple of 8 and at least n");
    if (n == 0) return FG_OK;
    return launch_pairs(ctx, x, n, (__nv_bfloat16*)pairs, plane_stride);
}

int32_t fg_gemm_paired_f32(fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, const float* A, const void* A_pairs,
                           uint64_t A_stride, const float* B, const void* B_pairs, uint64_t B_stride, float* C,
                           const float* bias, int32_t act, float* preact_out, void* C_pairs_out, uint64_t C_stride) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, A && B && C, "fg_gemm_paired_f32: NULL operand");
    FG_REQUIRE(ctx, M >= 1 && N >= 1 && K >= 1, "fg_gemm_paired_f32: dimensions must be >= 1");
    FG_REQUIRE(ctx, act >= FG_ACT_NONE && act <= FG_ACT_GELU, "fg_gemm_paired_f32: unknown activation");
    FG_REQUIRE(ctx, (uint64_t)M * N < (1ull << 40) && (uint64_t)M * K < (1ull << 40) && (uint64_t)N * K < (1ull << 40),
               "fg_gemm_paired_f32: operand too large");
    FG_REQUIRE(ctx, (!A_pairs || (fg_aligned16(A_pairs) && A_stride % 8 == 0 && A_stride >= (uint64_t)M * K)) &&
                        (!B_pairs || (fg_aligned16(B_pairs) && B_stride % 8 == 0 && B_stride >= (uint64_t)K * N)) &&
                        (!C_pairs_out || (fg_aligned16(C_pairs_out) && C_stride % 8 == 0 && C_stride >= (uint64_t)M * N)),
               "fg_gemm_paired_f32: pairs must be 16-byte aligned with a plane stride that is a multiple of 8 and covers the tensor");
    return gemm_fwd_core(ctx, FG_GEMM_AUTO, 0, 0, M, N, K, PairedArg{A, A_pairs, A_stride}, PairedArg{B, B_pairs, B_stride}, C,
                         bias, act, preact_out, (__nv_bfloat16*)C_pairs_out, C_stride);
}

}  // extern "C"

namespace {

// Backward of one layer through the SIMT kernels, the narrow-layer kernels or operand planes written by a
// pre-pass: any shape and alignment.  With exch_buf set, dB and dbias are finished first, the sum of exch_buf
// over the ranks is started on the exchange stream, and dA is computed while it runs.
int32_t gemm_bwd_planes(fg_ctx* ctx, int32_t mode, uint32_t M, uint32_t N, uint32_t K, const float* A, const float* B,
                        const float* dY, int32_t act, const float* saved, float* dA, float* dB, float* dbias,
                        float* dZ_out, float* exch_buf, uint64_t exch_count) {
    const bool fuse = act != FG_ACT_NONE;
    const bool skinny = runs_narrow(ctx, mode, M, N, K, grad_products(dA, dB, dbias, fuse));
    const int path = skinny ? 2 : pick_path(ctx, mode, M, N, K);
    const uint64_t mn = (uint64_t)M * N;

    if (path == 0) {
        const float* dz = dY;
        {
            uint64_t need = mn * 4 + (uint64_t)((M + 255) / 256) * N * 4 + 1024;
            { int32_t s0 = fg_ws_ensure(ctx, need); if (s0 != FG_OK) return s0; }
        }
        // Exact path: materialise dZ, then two SIMT GEMMs.
        if (fuse || dZ_out) {
            float* buf = dZ_out;
            if (!buf) {
                void* p;
                int32_t s = fg_ws_alloc(ctx, mn * 4, &p);
                if (s != FG_OK) return s;
                buf = (float*)p;
            }
            if (fuse) {
                int32_t s = fg_act_bwd_launch(ctx, mn, act, dY, saved, buf);
                if (s != FG_OK) return s;
            } else {
                FG_CUDA(ctx, FG_ERR_FAILED_BUFFER_COPY,
                        cudaMemcpyAsync(buf, dY, mn * 4, cudaMemcpyDeviceToDevice, ctx->stream));
            }
            dz = buf;
        }
        if (dB) { int32_t s = fg_gemm_simt_launch(ctx, 1, 0, K, N, M, A, dz, dB, nullptr, FG_ACT_NONE, nullptr); if (s) return s; }
        if (dbias) { int32_t s = fg_colsum_launch(ctx, M, N, dz, dbias); if (s) return s; }
        if (exch_buf) { int32_t s = fg_allreduce_sum_f32(ctx, exch_buf, exch_count); if (s) return s; }
        if (dA) { int32_t s = fg_gemm_simt_launch(ctx, 0, 1, M, K, N, dz, B, dA, nullptr, FG_ACT_NONE, nullptr); if (s) return s; }
        return FG_OK;
    }

    // Tensor-core path.  Scratch: dZ planes in both orientations, B planes, Aᵀ planes, dZ itself
    // when a bias gradient is wanted, and the column-sum partials.
    const int fmt = path - 1;
    // A skinny layer (N <= 16, say 10 classes): dA is bound by writing it once and dB by reading A once, so
    // both run as plain-FMA kernels on dZ itself; the operand pre-passes and a tensor-core GEMM that could
    // only fill M/128 CTAs would cost several times more.
    const bool tc_da = dA && !skinny, tc_db = dB && !skinny;
    uint64_t need = skinny ? narrow_bwd_need(M, N, K, dbias != nullptr) : 2048;
    if (tc_da) need += planes_bytes(fmt, M, N) + planes_bytes(fmt, K, N) + kPairPartialBytes;
    if (tc_db) need += planes_bytes(fmt, N, M) + planes_bytes(fmt, K, M) + kPairPartialBytes;
    if (dbias && !skinny) need += (uint64_t)((M + 31) / 32) * N * 4 + 256;   // per-tile column sums from the pre-pass
    { int32_t s0 = fg_ws_ensure(ctx, need); if (s0 != FG_OK) return s0; }
    PlaneSet dz_n{}, dz_t{}, b_n{}, a_t{};
    void* dz_val = dZ_out;
    int32_t s;
    if (tc_da) {
        if ((s = alloc_planes(ctx, fmt, M, N, &dz_n)) != FG_OK) return s;
        if ((s = alloc_planes(ctx, fmt, K, N, &b_n)) != FG_OK) return s;
    }
    if (tc_db) {
        if ((s = alloc_planes(ctx, fmt, N, M, &dz_t)) != FG_OK) return s;
        if ((s = alloc_planes(ctx, fmt, K, M, &a_t)) != FG_OK) return s;
    }
    if (skinny && fuse && !dz_val && (dA || dB)) {      // the skinny kernels read dZ itself
        if ((s = fg_ws_alloc(ctx, mn * 4, &dz_val)) != FG_OK) return s;
    }
    void* cs_part = nullptr;
    if (dbias && (s = fg_ws_alloc(ctx, (uint64_t)((M + 31) / 32) * N * 4, &cs_part)) != FG_OK) return s;
    SplitArgs sz{};
    sz.x = dY; sz.saved = fuse ? saved : nullptr; sz.act = act; sz.R = M; sz.C = N;
    sz.n = dz_n; sz.t = dz_t;
    sz.value_out = (float*)dz_val;
    sz.colsum_part = (float*)cs_part;
    uint32_t cs_chunks = 0;
    if (tc_da || tc_db || dz_val || dbias) {
        if ((s = launch_split(ctx, fmt, sz, &cs_chunks)) != FG_OK) return s;
    }
    const float* dz_src = dz_val ? (const float*)dz_val : dY;   // dZ == dY when there is no activation
    // weight and bias gradients first: with an exchange requested, it starts as soon as they are complete
    if (skinny && dB && (s = fg_gemm_skinny_tn_launch(ctx, M, K, N, A, dz_src, dB)) != FG_OK) return s;
    if (tc_db) {
        // dB[K,N] = Aᵀ · dZ: contraction over M; operands are Aᵀ [K,M] and dZᵀ [N,M].
        SplitArgs sa{};
        sa.x = A; sa.R = M; sa.C = K; sa.t = a_t;
        if ((s = launch_split(ctx, fmt, sa)) != FG_OK) return s;
        if ((s = tc_gemm(ctx, fmt, a_t, dz_t, K, N, M, dB, nullptr, FG_ACT_NONE, nullptr)) != FG_OK) return s;
    }
    if (dbias) {
        // the pre-pass left one row of column sums per row tile: fold them in a fixed order
        if ((s = fg_colsum_fold_launch(ctx, N, cs_chunks, (const float*)cs_part, dbias)) != FG_OK) return s;
    }
    if (exch_buf && (s = fg_allreduce_sum_f32(ctx, exch_buf, exch_count)) != FG_OK) return s;
    if (tc_da) {
        // dA[M,K] = dZ[M,N] · Bᵀ: contraction over N; B [K,N] is already "rows = K, contraction contiguous".
        SplitArgs sb{};
        sb.x = B; sb.R = K; sb.C = N; sb.n = b_n;
        if ((s = launch_split(ctx, fmt, sb)) != FG_OK) return s;
        if ((s = tc_gemm(ctx, fmt, dz_n, b_n, M, K, N, dA, nullptr, FG_ACT_NONE, nullptr)) != FG_OK) return s;
    }
    if (skinny && dA && (s = fg_gemm_skinny_nt_launch(ctx, M, K, N, dz_src, B, dA)) != FG_OK) return s;
    return FG_OK;
}

// Scratch gemm_bwd_planes may carve (an upper bound over its three routes).
uint64_t bwd_planes_need(uint32_t M, uint32_t N, uint32_t K) {
    const uint64_t mn = (uint64_t)M * N;
    uint64_t need = 4096 + mn * 4 + (uint64_t)((M + 31) / 32) * N * 4;
    need += planes_bytes(1, M, N) + planes_bytes(1, K, N) + planes_bytes(1, N, M) + planes_bytes(1, K, M) + 2 * kPairPartialBytes;
    need += fg_gemm_skinny_scratch_bytes(M, N, K);
    return need;
}

// Backward of Y = A·B given dZ = dL/dY (already multiplied by this layer's act'), on f32 tensors with pairs:
//   dB [K,N] = Aᵀ·dZ, then the exchange (if asked for), then
//   dA [M,K] = (dZ·Bᵀ) * act'(o.mul_saved) with its pairs (o.pairs) and its column sums (dbias_prev [K]) --
//   i.e. the dZ of the layer below and that layer's bias gradient come out of the dA epilogue.
// Pairs that are not supplied are made in the scratch arena.  The caller has reserved bwd_paired_need().
uint32_t colsum_room(uint32_t M, uint32_t N) { return N <= 16 ? fg_gemm_skinny_colsum_rows(M) : (M + 31) / 32; }
uint64_t bwd_paired_need(uint32_t M, uint32_t N, uint32_t K) {
    // (the conversion kernel's padded copies take less than the planes)
    return 4ull * ((uint64_t)M * K + (uint64_t)K * N + (uint64_t)M * N) + (uint64_t)colsum_room(M, N) * K * 4 +
           2 * kPairPartialBytes + 4096 + fg_gemm_skinny_scratch_bytes(M, N, K) + bwd_planes_need(M, N, K);
}

struct BwdRoutes {
    Route dB, dA;
    bool planes;      // every wanted product runs from operand planes
};
// Both wanted products may take the pair kernel or neither: its main term is truncated where the planes and the conversion
// kernel round it (dW of 128 x 4096 x 1024: 1.40e-6 against 0.87e-6 of the result's 2-norm), and a layer with one product that
// the pair kernel cannot run keeps the smaller error in both.  Between planes and conversion each product follows its
// estimate: 128 x 8192 x 8192 290 us, against 414 with both converted and 458 with both from planes.
BwdRoutes pick_bwd_routes(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, PairedArg A, PairedArg B, PairedArg dZ, const float* dB,
                          const float* dA, const float* mul_saved) {
    BwdRoutes r{};
    const double mk = (double)M * K, kn = (double)K * N, mn = (double)M * N;
    const bool n8 = N % 8 == 0 && K % 8 == 0 && fg_aligned16(dZ.x);
    const bool pair = (!dB || (n8 && fg_aligned16(A.x) && fg_aligned16(dB) && paired_shape_ok(ctx, K, N, M, K, N))) &&
                      (!dA || (n8 && fg_aligned16(B.x) && fg_aligned16(dA) && (!mul_saved || fg_aligned16(mul_saved)) &&
                               paired_shape_ok(ctx, M, K, N, N, N)));
    const bool tc = pick_path(ctx, FG_GEMM_AUTO, M, N, K) == 2;
    const bool cz = !in_place32(dZ.x, N, 1, 0);
    bool all = true, any = false;       // of the wanted products, from planes
    auto pick = [&](uint32_t m, uint32_t n, uint32_t k, double elems, bool pairs, bool copied) {
        const Route x = (tc || pair) ? pick_route(ctx, m, n, k, pair, (pairs ? 0.0 : elems) + (dZ.pairs ? 0.0 : mn), !pairs + !dZ.pairs,
                                                  (copied ? elems : 0.0) + (cz ? mn : 0.0), copied + cz) : Route{kRoutePlanes, ConvPlan{}};
        all &= x.kind == kRoutePlanes;
        any |= x.kind == kRoutePlanes;
        return x;
    };
    if (dB) r.dB = pick(K, N, M, mk, A.pairs != nullptr, !in_place32(A.x, K, 1, 0));
    if (dA) r.dA = pick(M, K, N, kn, B.pairs != nullptr, !in_place32(B.x, N, 1, 0));
    // a dZ of padded pitch, as the conversion kernel would have it, cannot be split into planes
    r.planes = all || (any && N % 4 != 0);
    return r;
}

// The two products of a backward step by their routes; dZ has row pitch ldz (N, or padded for the conversion kernel).  The
// caller has reserved what they carve.
int32_t gemm_bwd_products(fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, PairedArg A, PairedArg B, PairedArg dZ, uint32_t ldz,
                          const BwdRoutes& rt, float* dB, float* dA, const PairedOut& o, float* exch_buf, uint64_t exch_count, PrepBatch& prep,
                          uint32_t bias_rows, const float* bias_part, float* dbias) {
    int32_t s;
    const uint64_t mk = (uint64_t)M * K, kn = (uint64_t)K * N, mn = (uint64_t)M * N;
    const bool pair_b = dB && rt.dB.kind == kRoutePair, pair_a = dA && rt.dA.kind == kRoutePair;
    const bool conv_b = dB && rt.dB.kind == kRouteConv, conv_a = dA && rt.dA.kind == kRouteConv;
    auto make_pairs = [&](PairedArg& t, uint64_t n) -> int32_t {
        if (t.pairs) return FG_OK;
        void* q;
        int32_t e = fg_ws_alloc(ctx, n * 4, &q);
        if (e != FG_OK || (e = launch_pairs(ctx, t.x, n, (__nv_bfloat16*)q, n)) != FG_OK) return e;
        t.pairs = q; t.stride = n;
        return FG_OK;
    };
    // What the conversion kernel cannot read in place joins the passes that the caller has left; then the layer's bias gradient.
    PlaneSet z32, a32, b32;
    if (conv_b || conv_a) {
        if (ldz == N && (s = loadable32(ctx, dZ.x, M, N, 1, 0, &z32, &prep)) != FG_OK) return s;
        if (ldz != N) { z32 = PlaneSet{}; z32.p32 = const_cast<float*>(dZ.x); z32.ld32 = ldz; }
    }
    if (conv_b && (s = loadable32(ctx, A.x, M, K, 1, 0, &a32, &prep)) != FG_OK) return s;
    if (conv_a && (s = loadable32(ctx, B.x, K, N, 1, 0, &b32, &prep)) != FG_OK) return s;
    if ((s = prep.launch(ctx)) != FG_OK) return s;
    if (dbias && (s = fg_colsum_fold_launch(ctx, N, bias_rows, bias_part, dbias)) != FG_OK) return s;
    if ((pair_a || pair_b) && (s = make_pairs(dZ, mn)) != FG_OK) return s;
    const bool one = conv_b && conv_a && !exch_buf;      // both gradients in one launch
    ConvProduct both[2];
    if (pair_b) {
        if ((s = make_pairs(A, mk)) != FG_OK) return s;
        // operands Aᵀ (rows = K) and dZᵀ (rows = N), both read from [M, .] storage: contraction over the rows
        const PlaneSet pa = paired_operand(A.x, A.pairs, A.stride, K, false);
        const PlaneSet pz = paired_operand(dZ.x, dZ.pairs, dZ.stride, N, false);
        if ((s = paired_gemm(ctx, pa, pz, K, N, M, dB, nullptr, FG_ACT_NONE, nullptr, PairedOut{nullptr, 0, nullptr, 0, nullptr})) != FG_OK)
            return s;
    } else if (conv_b) {
        const Epilogue ep{dB, nullptr, nullptr, K, N, M, FG_ACT_NONE, ctx->dev_status};
        both[0] = ConvProduct{as_operand(a32, true), as_operand(z32, true), ep, 1};
        if (!one && (s = launch_conv(ctx, &both[0], 1, rt.dB.conv)) != FG_OK) return s;
    } else if (dB && (s = gemm_bwd_planes(ctx, FG_GEMM_AUTO, M, N, K, A.x, nullptr, dZ.x, FG_ACT_NONE, nullptr, nullptr, dB, nullptr,
                                          nullptr, nullptr, 0)) != FG_OK) return s;
    if (exch_buf && (s = fg_allreduce_sum_f32(ctx, exch_buf, exch_count)) != FG_OK) return s;
    if (pair_a) {
        if ((s = make_pairs(B, kn)) != FG_OK) return s;
        // operands dZ (rows = M) and B (rows = K), both with the contraction index N contiguous
        const PlaneSet pz = paired_operand(dZ.x, dZ.pairs, dZ.stride, N, true);
        const PlaneSet pb = paired_operand(B.x, B.pairs, B.stride, N, true);
        if ((s = paired_gemm(ctx, pz, pb, M, K, N, dA, nullptr, FG_ACT_NONE, nullptr, o)) != FG_OK) return s;
    } else if (conv_a) {
        Epilogue ep{dA, nullptr, nullptr, M, K, N, FG_ACT_NONE, ctx->dev_status};
        ep.c_pairs = o.pairs;
        ep.c_pairs_stride = o.stride;
        ep.mul_saved = o.mul_saved;
        ep.mul_act = o.mul_act;
        ep.colsum_part = o.colsum_part;
        both[1] = ConvProduct{as_operand(z32, false), as_operand(b32, false), ep, 1};
        if ((s = one ? launch_conv_both(ctx, both[0], both[1]) : launch_conv(ctx, &both[1], 1, rt.dA.conv)) != FG_OK) return s;
    } else if (dA) {        // (o is left to the caller)
        return gemm_bwd_planes(ctx, FG_GEMM_AUTO, M, N, K, nullptr, B.x, dZ.x, FG_ACT_NONE, nullptr, dA, nullptr, nullptr, nullptr, nullptr, 0);
    }
    return FG_OK;
}

int32_t gemm_bwd_paired_core(fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, PairedArg A, PairedArg B, PairedArg dZ, float* dB,
                             float* dA, PairedOut o, float* dbias, float* dbias_prev, float* exch_buf, uint64_t exch_count) {
    int32_t s;
    void* p;
    // Where dA lies over the saved tensor its factor comes from a copy on the routes that apply it elsewhere than they read it (in
    // the room of the pairs, which those routes do not make).
    auto saved_apart = [&]() -> int32_t {
        const uint64_t bytes = (uint64_t)M * K * 4;
        if (!o.mul_saved || !fg_ranges_meet(dA, bytes, o.mul_saved, bytes)) return FG_OK;
        if ((s = fg_ws_alloc(ctx, bytes, &p)) != FG_OK) return s;
        FG_CUDA(ctx, FG_ERR_FAILED_BUFFER_COPY, cudaMemcpyAsync(p, o.mul_saved, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        o.mul_saved = (const float*)p;
        return FG_OK;
    };
    const bool narrow = N <= 16;
    const int below = dA && (o.mul_saved || dbias_prev) ? kFgBelow : 0;
    if ((dA || dB) && takes_fma(ctx, FG_GEMM_AUTO, M, N, K, grad_products(dA, dB, dbias, false) | below)) {
        if (dA && o.mul_saved != dA && (s = saved_apart()) != FG_OK) return s;      // (an element is read and written by one thread)
        FgFmaBwd b{};
        b.M = M; b.N = N; b.K = K; b.A = A.x; b.B = B.x; b.dZ = dZ.x; b.dA = dA; b.dB = dB; b.dbias = dbias;
        b.mul_saved = o.mul_saved; b.mul_act = o.mul_act; b.pairs = o.pairs; b.pairs_stride = o.stride; b.below_dbias = dbias_prev;
        b.exch_buf = exch_buf; b.exch_count = exch_count;
        return fg_gemm_fma_bwd(ctx, b);
    }
    const BwdRoutes rt = narrow ? BwdRoutes{} : pick_bwd_routes(ctx, M, N, K, A, B, dZ, dB, dA, o.mul_saved);
    if (dbias && (s = fg_colsum_launch(ctx, M, N, dZ.x, dbias)) != FG_OK) return s;
    const uint32_t cs_chunks = (M + 31) / 32;
    float* cs_part = nullptr;
    if (dA && dbias_prev) {
        if ((s = fg_ws_alloc(ctx, (uint64_t)colsum_room(M, N) * K * 4, &p)) != FG_OK) return s;
        cs_part = (float*)p;
    }
    if (narrow) {
        // narrow layer: plain-FMA streaming kernels on the tensors themselves
        if (dB && (s = fg_gemm_skinny_tn_launch(ctx, M, K, N, A.x, dZ.x, dB)) != FG_OK) return s;
        if (exch_buf && (s = fg_allreduce_sum_f32(ctx, exch_buf, exch_count)) != FG_OK) return s;
        if (dA) {
            const fg_skinny_extras ex{o.mul_saved, o.mul_act, o.pairs, o.stride, cs_part};
            uint32_t cs_rows = 0;
            if ((s = fg_gemm_skinny_nt_launch(ctx, M, K, N, dZ.x, B.x, dA, &ex, &cs_rows)) != FG_OK) return s;
            if (cs_part && (s = fg_colsum_fold_launch(ctx, K, cs_rows, cs_part, dbias_prev)) != FG_OK) return s;
        }
        return FG_OK;
    }
    // There the factor is applied after the whole of dA has been written.
    if (dA && (rt.planes || rt.dA.kind == kRoutePlanes) && (s = saved_apart()) != FG_OK) return s;
    if (!rt.planes && (dA || dB)) {
        PairedOut po = o;
        po.colsum_part = cs_part;
        PrepBatch prep;
        if ((s = gemm_bwd_products(ctx, M, N, K, A, B, dZ, N, rt, dB, dA, po, exch_buf, exch_count, prep, 0, nullptr, nullptr)) != FG_OK) return s;
        if (!dA || rt.dA.kind != kRoutePlanes)
            return cs_part ? fg_colsum_fold_launch(ctx, K, cs_chunks, cs_part, dbias_prev) : FG_OK;
    } else if ((s = gemm_bwd_planes(ctx, FG_GEMM_AUTO, M, N, K, A.x, B.x, dZ.x, FG_ACT_NONE, nullptr, dA, dB, nullptr, nullptr, exch_buf,
                                    exch_count)) != FG_OK) {
        return s;
    }
    if (!dA) return FG_OK;
    // dA came from operand planes: what the other kernels' epilogues would have done, as passes of their own
    const uint64_t mk = (uint64_t)M * K;
    if (K % 4 == 0 && fg_aligned16(dA) && (!o.mul_saved || fg_aligned16(o.mul_saved))) {
        if (o.mul_saved || o.pairs || cs_part) {
            if ((s = launch_dz_pairs(ctx, M, K, dA, o.mul_saved, o.mul_act, o.mul_saved ? dA : nullptr, o.pairs, o.stride, cs_part)) != FG_OK)
                return s;
            if (cs_part && (s = fg_colsum_fold_launch(ctx, K, cs_chunks, cs_part, dbias_prev)) != FG_OK) return s;
        }
        return FG_OK;
    }
    if (o.mul_saved && (s = fg_act_bwd_launch(ctx, mk, o.mul_act, dA, o.mul_saved, dA)) != FG_OK) return s;
    if (o.pairs && (s = launch_pairs(ctx, dA, mk, o.pairs, o.stride)) != FG_OK) return s;
    if (dbias_prev && (s = fg_colsum_launch(ctx, M, K, dA, dbias_prev)) != FG_OK) return s;
    return FG_OK;
}

}  // namespace

bool fg_gemm_bwd_sums_bias(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, bool dA) {
    return takes_fma(ctx, FG_GEMM_AUTO, M, N, K, kFgGradB | (dA ? kFgGradA : 0));
}

uint32_t fg_gemm_reads_pairs(const fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K) {
    if (N <= 16) return 0;
    float* const any = reinterpret_cast<float*>(uintptr_t(256));      // only the alignment counts, and that pairs are there
    const PairedArg t{any, any, 0};
    uint32_t bits = 0;
    if (pick_path(ctx, FG_GEMM_AUTO, M, N, K) == 2 && !takes_fma(ctx, FG_GEMM_AUTO, M, N, K, kFgForward)) {
        const int ca = !in_place32(any, K, 1, 0), cb = !in_place32(any, N, 1, 0);
        const Route r = pick_route(ctx, M, N, K, paired_shape_ok(ctx, M, N, K, K, N) && N % 4 == 0, 0.0, 0, (ca ? (double)M * K : 0.0) + (cb ? (double)K * N : 0.0),
                                   ca + cb);
        if (r.kind == kRoutePair) bits |= 1 | 2;
    }
    for (int want = 1; want < 4; ++want) {      // dB, dA or both
        if (takes_fma(ctx, FG_GEMM_AUTO, M, N, K, want)) continue;
        const BwdRoutes r = pick_bwd_routes(ctx, M, N, K, t, t, t, want & 1 ? any : nullptr, want & 2 ? any : nullptr, nullptr);
        if ((want & 1) && !r.planes && r.dB.kind == kRoutePair) bits |= 1 | 4;
        if ((want & 2) && !r.planes && r.dA.kind == kRoutePair) bits |= 2 | 4;
    }
    return bits;
}

namespace {

// Backward of Y = act(A·B + bias) from dY: forms dZ = dY * act'(saved) first.
int32_t gemm_bwd_impl(fg_ctx* ctx, int32_t mode, uint32_t M, uint32_t N, uint32_t K, const float* A, const float* B,
                      const float* dY, int32_t act, const float* saved, float* dA, float* dB, float* dbias,
                      float* dZ_out, float* exch_buf, uint64_t exch_count) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, dY != nullptr, "fg_gemm_bwd_f32: dY is NULL");
    FG_REQUIRE(ctx, M >= 1 && N >= 1 && K >= 1, "fg_gemm_bwd_f32: dimensions must be >= 1");
    FG_REQUIRE(ctx, mode >= FG_GEMM_AUTO && mode <= FG_GEMM_TF32_BF16X2, "fg_gemm_bwd_f32: unknown mode");
    FG_REQUIRE(ctx, act >= FG_ACT_NONE && act <= FG_ACT_GELU, "fg_gemm_bwd_f32: unknown activation");
    FG_REQUIRE(ctx, act == FG_ACT_NONE || saved, "fg_gemm_bwd_f32: the activation backward needs the saved tensor");
    FG_REQUIRE(ctx, !dA || B, "fg_gemm_bwd_f32: dA needs B");
    FG_REQUIRE(ctx, !dB || A, "fg_gemm_bwd_f32: dB needs A");
    const bool fuse = act != FG_ACT_NONE;
    const int path = pick_path(ctx, mode, M, N, K);
    const bool fma = path == 0 ? mode == FG_GEMM_AUTO && !runs_narrow(ctx, mode, M, N, K, grad_products(dA, dB, dbias, fuse))
                               : (dA || dB) && takes_fma(ctx, mode, M, N, K, (dB ? kFgGradB : 0) | (dA ? kFgGradA : 0));
    if (!dZ_out && fma) {
        FgFmaBwd b{};
        b.M = M; b.N = N; b.K = K; b.A = A; b.B = B; b.dZ = dY; b.factor = fuse ? saved : nullptr; b.factor_act = act;
        b.dA = dA; b.dB = dB; b.dbias = dbias; b.exch_buf = exch_buf; b.exch_count = exch_count;
        const int32_t s = fg_ws_ensure(ctx, fg_gemm_fma_bwd_scratch(b));
        return s != FG_OK ? s : fg_gemm_fma_bwd(ctx, b);
    }
    // (prep_kernel takes up to 65535 * 32 rows, the planes twice as many)
    if (path == 2 && N > 16 && (dA || dB) && M <= 65535u * 32u) {
        // dZ (with its pairs, if a product needs them) and the bias gradient's partials in one pass, then both products
        // from the tensors themselves
        const uint64_t mn = (uint64_t)M * N;
        const uint32_t cs_chunks = (M + 31) / 32;
        const bool vec_z = N % 8 == 0 && fg_aligned16(dY) && (!fuse || fg_aligned16(saved)) && (!dZ_out || fg_aligned16(dZ_out));
        // dZ is new when there is an activation: it will lie in the scratch arena (or dZ_out) with a usable pitch
        const bool own_z = fuse || !in_place32(dY, N, 1, 0);
        const float* const z_like = own_z ? nullptr : dY;      // only its alignment counts
        const bool z_dense = N % 4 == 0;
        const BwdRoutes rt = pick_bwd_routes(ctx, M, N, K, PairedArg{A, nullptr, 0}, PairedArg{B, nullptr, 0}, PairedArg{z_like, nullptr, 0}, dB, dA, nullptr);
        const bool want_pairs = (dB && rt.dB.kind == kRoutePair) || (dA && rt.dA.kind == kRoutePair);
        if (!rt.planes && (!want_pairs || vec_z)) {
            uint64_t need = (uint64_t)cs_chunks * N * 4 + 2048;
            if (want_pairs) need += bwd_paired_need(M, N, K) + mn * 4;
            else {       // dZ and what each product carves: never more than the operand planes of both would take
                if (own_z) need += (uint64_t)M * round4(N) * 4 + 256;
                if (dB) need += rt.dB.kind == kRoutePlanes ? planes_bytes(1, N, M) + planes_bytes(1, K, M) + kPairPartialBytes + 4096
                                                           : copy32_bytes(A, M, K, 1, 0);
                if (dA) need += rt.dA.kind == kRoutePlanes ? planes_bytes(1, M, N) + planes_bytes(1, K, N) + kPairPartialBytes + 4096
                                                           : copy32_bytes(B, K, N, 1, 0);
            }
            { int32_t s0 = fg_ws_ensure(ctx, need); if (s0 != FG_OK) return s0; }
            int32_t s;
            PrepBatch prep;
            void *pz = nullptr, *dzb = nullptr, *csp = nullptr;
            if (dbias && (s = fg_ws_alloc(ctx, (uint64_t)cs_chunks * N * 4, &csp)) != FG_OK) return s;
            PairedArg z{dY, nullptr, 0};
            if (want_pairs) {
                dzb = dZ_out;
                if ((s = fg_ws_alloc(ctx, mn * 4, &pz)) != FG_OK) return s;
                if (fuse && !dzb && (s = fg_ws_alloc(ctx, mn * 4, &dzb)) != FG_OK) return s;
                if ((s = launch_dz_pairs(ctx, M, N, dY, fuse ? saved : nullptr, act, (float*)dzb, (__nv_bfloat16*)pz, mn, (float*)csp)) != FG_OK)
                    return s;
                if (dzb) z.x = (const float*)dzb;
                z.pairs = pz; z.stride = mn;
            } else if (own_z || csp || dZ_out) {
                PrepArgs a{};
                a.x = dY; a.saved = fuse ? saved : nullptr; a.act = act; a.R = M; a.C = N;
                a.colsum_part = (float*)csp;
                if (own_z && !(z_dense && dZ_out && fg_aligned16(dZ_out))) {
                    if ((s = fg_ws_alloc(ctx, (uint64_t)M * round4(N) * 4, &dzb)) != FG_OK) return s;
                    a.out = dzb; a.ld = round4(N);
                    a.copy = dZ_out;
                } else a.copy = dZ_out;
                if ((s = prep.add(ctx, FG_DTYPE_F32, a)) != FG_OK) return s;
                if (own_z) z.x = dzb ? (const float*)dzb : dZ_out;
            }
            return gemm_bwd_products(ctx, M, N, K, PairedArg{A, nullptr, 0}, PairedArg{B, nullptr, 0}, z, own_z && !z_dense && !want_pairs ? round4(N) : N, rt,
                                     dB, dA, PairedOut{nullptr, 0, nullptr, 0, nullptr}, exch_buf, exch_count, prep, cs_chunks, (const float*)csp, dbias);
        }
    }
    return gemm_bwd_planes(ctx, mode, M, N, K, A, B, dY, act, saved, dA, dB, dbias, dZ_out, exch_buf, exch_count);
}

}  // namespace

namespace {

// One launch of the conversion kernel for `batch` products, or a loop over them?  The loop's cost per matrix is the pair
// kernel's when the matrix suits it (its pairs are made for the whole batch at once), otherwise a pre-pass and a
// partly filled wave per matrix.
bool batch_converts(const fg_ctx* ctx, uint32_t batch, uint32_t M, uint32_t N, uint32_t K, bool pair_ok) {
    if (!conv_allowed(ctx) || batch > 65535) return false;
    const double elems = (double)M * K + (double)K * N;
    return plan_conv(ctx, M, N, K, batch).cycles <= (double)batch * pair_cycles(ctx, M, N, K, pair_ok ? elems : 2.0 * elems, 2);
}

// Arguments that the per-matrix entry points refuse (an unknown mode, K = 0) are left to the loop, which asks them.
bool batch_route_open(const fg_ctx* ctx, int32_t mode, uint32_t M, uint32_t N, uint32_t K) {
    return mode >= FG_GEMM_AUTO && mode <= FG_GEMM_TF32_BF16X2 && K >= 1 && pick_path(ctx, mode, M, N, K) == 2 &&
           (N > 16 || mode != FG_GEMM_AUTO);
}

// Small matrices: the sums of a batch come in the order of k, whichever kernel adds them and also one matrix at a time (more than 65535 of
// them, or no room for the dZ of matrices with room between them): the loops ask for the exact path.
int32_t batch_loop_mode(const fg_ctx* ctx, int32_t mode, uint32_t M, uint32_t N, uint32_t K) {
    return mode == FG_GEMM_AUTO && pick_path(ctx, mode, M, N, K) == 0 ? (int32_t)FG_GEMM_SIMT : mode;
}
// Where the exact path would take its large tiles the FMA
// kernel's are the faster ones forward and for both gradients together (31 x (60 x 500 x 500) 45 -> 34 and 92 -> 76 us), not for a
// gradient by itself (dB of 30 x (100 x 100 x 400) 17.7 us, 20.7 with it) nor for a short k (24 x (182 x 151 x 30) 6.2, 7.6 with it).
bool batch_large(const fg_ctx* ctx, int32_t mode, uint32_t batch, uint32_t M, uint32_t N) { return mode == FG_GEMM_AUTO && fg_gemm_simt_large(ctx, M, N, batch); }

// Matrices per launch: the whole batch if the scratch arena has room for it or can be grown (64 x (512 x 512 x 512) backward with
// an activation: 323 us, 360 in parts).  Otherwise (out of memory, a recording whose arena was sized for less) as many as find
// room in the arena or in what the loop over the matrices would make of it (`loop`).  need(t): bytes for t matrices.
template <typename Need>
uint32_t batch_part(fg_ctx* ctx, uint32_t batch, uint64_t loop, Need need) {
    if (fg_ws_try(ctx, need(batch))) return batch;
    const uint64_t room = ctx->capturing || loop < ctx->ws_bytes ? ctx->ws_bytes : loop;
    uint32_t t = batch;
    while (t > 1 && (need(t) > room || (batch % t && need(batch % t) > room))) t = (t + 1) / 2;      // (the last part may cut K)
    return t;
}

}  // namespace

extern "C" {

int32_t fg_gemm_bwd_f32(fg_ctx* ctx, int32_t mode, uint32_t M, uint32_t N, uint32_t K, const float* A, const float* B,
                        const float* dY, int32_t act, const float* saved, float* dA, float* dB, float* dbias,
                        float* dZ_out) {
    return gemm_bwd_impl(ctx, mode, M, N, K, A, B, dY, act, saved, dA, dB, dbias, dZ_out, nullptr, 0);
}

int32_t fg_gemm_bwd_exchange_f32(fg_ctx* ctx, int32_t mode, uint32_t M, uint32_t N, uint32_t K, const float* A,
                                 const float* B, const float* dY, int32_t act, const float* saved, float* dA, float* dB,
                                 float* dbias, float* exch_buf, uint64_t exch_count) {
    if (!ctx) return FG_ERR_NOT_INITIALIZED;
    FG_REQUIRE(ctx, exch_buf != nullptr && exch_count > 0, "fg_gemm_bwd_exchange_f32: nothing to exchange");
    if (!ctx->comm) return fg_fail(ctx, FG_ERR_NOT_INITIALIZED, "fg_gemm_bwd_exchange_f32: call fg_comm_init first");
    return gemm_bwd_impl(ctx, mode, M, N, K, A, B, dY, act, saved, dA, dB, dbias, nullptr, exch_buf, exch_count);
}

int32_t fg_gemm_bwd_paired_f32(fg_ctx* ctx, uint32_t M, uint32_t N, uint32_t K, const float* A, const void* A_pairs,
                               uint64_t A_stride, const float* B, const void* B_pairs, uint64_t B_stride, const float* dZ,
                               const void* dZ_pairs, uint64_t dZ_stride, float* dB, float* dbias, float* dA,
                               int32_t below_act, const float* below_saved, void* dA_pairs_out, uint64_t dA_stride,
                               float* below_dbias, float* exch_buf, uint64_t exch_count) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, dZ != nullptr, "fg_gemm_bwd_paired_f32: dZ is NULL");
    FG_REQUIRE(ctx, M >= 1 && N >= 1 && K >= 1, "fg_gemm_bwd_paired_f32: dimensions must be >= 1");
    FG_REQUIRE(ctx, below_act >= FG_ACT_NONE && below_act <= FG_ACT_GELU, "fg_gemm_bwd_paired_f32: unknown activation");
    FG_REQUIRE(ctx, below_act == FG_ACT_NONE || below_saved, "fg_gemm_bwd_paired_f32: the activation backward needs the saved tensor");
    FG_REQUIRE(ctx, !dA || B, "fg_gemm_bwd_paired_f32: dA needs B");
    FG_REQUIRE(ctx, !dB || A, "fg_gemm_bwd_paired_f32: dB needs A");
    FG_REQUIRE(ctx, dA || (!dA_pairs_out && !below_dbias), "fg_gemm_bwd_paired_f32: pairs and bias gradient of dA need dA");
    auto pairs_ok = [](const void* p, uint64_t stride, uint64_t n) { return !p || (fg_aligned16(p) && stride % 8 == 0 && stride >= n); };
    FG_REQUIRE(ctx, pairs_ok(A_pairs, A_stride, (uint64_t)M * K) && pairs_ok(B_pairs, B_stride, (uint64_t)K * N) &&
                        pairs_ok(dZ_pairs, dZ_stride, (uint64_t)M * N) && pairs_ok(dA_pairs_out, dA_stride, (uint64_t)M * K),
               "fg_gemm_bwd_paired_f32: pairs must be 16-byte aligned with a plane stride that is a multiple of 8 and covers the tensor");
    if (exch_buf && !ctx->comm) return fg_fail(ctx, FG_ERR_NOT_INITIALIZED, "fg_gemm_bwd_paired_f32: call fg_comm_init first");
    FG_REQUIRE(ctx, !exch_buf || exch_count > 0, "fg_gemm_bwd_paired_f32: nothing to exchange");
    { int32_t s0 = fg_ws_ensure(ctx, bwd_paired_need(M, N, K)); if (s0 != FG_OK) return s0; }
    const bool mul = below_act != FG_ACT_NONE;
    return gemm_bwd_paired_core(ctx, M, N, K, PairedArg{A, A_pairs, A_stride}, PairedArg{B, B_pairs, B_stride},
                                PairedArg{dZ, dZ_pairs, dZ_stride}, dB, dA,
                                PairedOut{(__nv_bfloat16*)dA_pairs_out, dA_stride, mul ? below_saved : nullptr, below_act, nullptr},
                                dbias, below_dbias, exch_buf, exch_count);
}

// Batched forms: `batch` independent products, operand t at base + t*stride (strides in elements).
// The reference steps A, B and C by one matrix per Z index of a rank-3 matmul (kernel/forward.rs:159-190).
// Rank-3 products.  Small matrices (below the tensor cores' sizes: the matrix index is the grid's z, as in the reference's generated
// kernel, kernel/forward.rs:159-190) and middling ones (the conversion kernel: it is part of the unit's number) run as ONE launch.  Large
// ones: the bf16 pairs of the whole batch are made by one pass per operand, then one GEMM launch per matrix reads its
// slice (batch + 2 launches, and a launch that fills the GPU gains nothing from being merged with its neighbours).
int32_t fg_gemm_batched_f32(fg_ctx* ctx, int32_t mode, uint32_t batch, uint32_t M, uint32_t N, uint32_t K, const float* A,
                            uint64_t strideA, const float* B, uint64_t strideB, float* C, uint64_t strideC,
                            const float* bias, int32_t act, float* preact_out) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, A && B && C, "fg_gemm_batched_f32: NULL pointer");
    FG_REQUIRE(ctx, act >= FG_ACT_NONE && act <= FG_ACT_GELU, "fg_gemm_batched_f32: unknown activation");
    FG_REQUIRE(ctx, strideA >= (uint64_t)M * K && strideB >= (uint64_t)K * N && strideC >= (uint64_t)M * N,
               "fg_gemm_batched_f32: a stride is smaller than its matrix (for one B shared by all products, "
               "call fg_gemm_f32 with batch*M rows)");
    if (batch == 0 || (uint64_t)M * N == 0) return FG_OK;
    if (pick_path(ctx, mode, M, N, K) == 0 && batch <= 65535 && K >= 64 && batch_large(ctx, mode, batch, M, N)) {
        FgFmaOp o{};
        o.M = M; o.N = N; o.K = K; o.A = A; o.B = B; o.C = C; o.bias = bias; o.act = act; o.preact = preact_out;
        o.sA = strideA; o.sB = strideB; o.sC = strideC;
        return fg_gemm_fma_launch(ctx, &o, 1, batch, true);
    }
    if (pick_path(ctx, mode, M, N, K) == 0 && batch <= 65535 && K > 0)
        return fg_gemm_simt_batched_launch(ctx, 0, 0, batch, M, N, K, A, strideA, B, strideB, C, strideC, bias, act, preact_out);
    if (batch_route_open(ctx, mode, M, N, K)) {
        if (batch_converts(ctx, batch, M, N, K, paired_shape_ok(ctx, M, N, K, K, N))) {
            auto need = [&](uint32_t t) {
                return copy32_bytes(A, M, K, t, strideA) + copy32_bytes(B, K, N, t, strideB) + 1024;
            };
            const uint32_t part = batch_part(ctx, batch, planes_bytes(1, M, K) + planes_bytes(1, N, K) + kPairPartialBytes + 1024, need);
            for (uint32_t t0 = 0; t0 < batch; t0 += part) {
                const uint32_t t = batch - t0 < part ? batch - t0 : part;
                PlaneSet pa, pb;
                ctx->ws_used = 0;
                int32_t s = fg_ws_ensure(ctx, need(t));
                if (s != FG_OK) return s;
                PrepBatch prep;
                if ((s = loadable32(ctx, A + t0 * strideA, M, K, t, strideA, &pa, &prep)) != FG_OK) return s;
                if ((s = loadable32(ctx, B + t0 * strideB, K, N, t, strideB, &pb, &prep)) != FG_OK) return s;
                if ((s = prep.launch(ctx)) != FG_OK) return s;
                Epilogue ep{C + t0 * strideC, bias, preact_out ? preact_out + t0 * strideC : nullptr, M, N, K, act, ctx->dev_status};
                ep.c_batch = t > 1 ? strideC : 0;
                if ((s = launch_conv(ctx, as_operand(pa, false), as_operand(pb, true), ep, plan_conv(ctx, M, N, K, t), t)) != FG_OK) return s;
            }
            return FG_OK;
        }
    }
    const bool dense = strideA == (uint64_t)M * K && strideB == (uint64_t)K * N;
    // the condition under which a per-matrix call below takes the path that reads pairs, if it takes the pair kernel
    const bool shared_pairs = dense && mode == FG_GEMM_AUTO && N > 16 && N % 4 == 0 && strideC % 4 == 0 && fg_aligned16(A) &&
                              fg_aligned16(B) && fg_aligned16(C) && (!preact_out || fg_aligned16(preact_out)) &&
                              paired_shape_ok(ctx, M, N, K, K, N);
    __nv_bfloat16 *pa = nullptr, *pb = nullptr;
    const uint64_t na = (uint64_t)batch * M * K, nb = (uint64_t)batch * K * N;
    if (shared_pairs) {
        void* p;
        int32_t s = fg_ws_ensure(ctx, (na + nb) * 4 + 2 * kPairPartialBytes + 8192);
        if (s != FG_OK) return s;
        if ((s = fg_ws_alloc(ctx, na * 4, &p)) != FG_OK) return s;
        pa = (__nv_bfloat16*)p;
        if ((s = fg_ws_alloc(ctx, nb * 4, &p)) != FG_OK) return s;
        pb = (__nv_bfloat16*)p;
        if ((s = launch_pairs(ctx, A, na, pa, na)) != FG_OK) return s;
        if ((s = launch_pairs(ctx, B, nb, pb, nb)) != FG_OK) return s;
    }
    for (uint32_t t = 0; t < batch; ++t) {
        int32_t s;
        if (shared_pairs) {
            // carve nothing more from the arena: the slices above stay valid for every matrix
            const uint64_t keep = ctx->ws_used;
            s = gemm_fwd_core(ctx, mode, 0, 0, M, N, K, PairedArg{A + t * strideA, pa + t * strideA, na},
                              PairedArg{B + t * strideB, pb + t * strideB, nb}, C + t * strideC, bias, act,
                              preact_out ? preact_out + t * strideC : nullptr, nullptr, 0);
            ctx->ws_used = keep;
        } else {
            s = fg_gemm_f32(ctx, batch_loop_mode(ctx, mode, M, N, K), 0, 0, M, N, K, A + t * strideA, B + t * strideB, C + t * strideC, bias, act,
                            preact_out ? preact_out + t * strideC : nullptr);
        }
        if (s != FG_OK) return s;
    }
    return FG_OK;
}

int32_t fg_gemm_batched_bwd_f32(fg_ctx* ctx, int32_t mode, uint32_t batch, uint32_t M, uint32_t N, uint32_t K,
                                const float* A, uint64_t strideA, const float* B, uint64_t strideB, const float* dY,
                                uint64_t strideC, int32_t act, const float* saved, float* dA, float* dB) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, dY != nullptr, "fg_gemm_batched_bwd_f32: dY is NULL");
    FG_REQUIRE(ctx, act >= FG_ACT_NONE && act <= FG_ACT_GELU, "fg_gemm_batched_bwd_f32: unknown activation");
    FG_REQUIRE(ctx, act == FG_ACT_NONE || saved, "fg_gemm_batched_bwd_f32: saved tensor required");
    FG_REQUIRE(ctx, (!dA || B) && (!dB || A), "fg_gemm_batched_bwd_f32: dA needs B, dB needs A");
    FG_REQUIRE(ctx, strideA >= (uint64_t)M * K && strideB >= (uint64_t)K * N && strideC >= (uint64_t)M * N,
               "fg_gemm_batched_bwd_f32: a stride is smaller than its matrix");
    if (batch == 0 || (uint64_t)M * N == 0 || (!dA && !dB)) return FG_OK;
    // (of matrices with room between them dZ is formed without it, if the arena has the room for that; the pass takes 65535 tiles of 32 rows)
    const bool dense_z = strideC == (uint64_t)M * N;
    auto apart_z = [&] { return K > 0 && M <= 65535u * 32u && fg_ws_try(ctx, (uint64_t)batch * M * N * 4 + 512); };
    if (pick_path(ctx, mode, M, N, K) == 0 && batch <= 65535 && (dense_z || (act == FG_ACT_NONE ? K > 0 : apart_z()))) {
        // dZ = dY * act'(saved) for the whole batch, then dB[t] = A[t]^T dZ[t] and dA[t] = dZ[t] B[t]^T: sums in the order of k
        const float* dz = dY;
        uint64_t sz = strideC;
        if (act != FG_ACT_NONE) {
            const uint64_t n = (uint64_t)batch * M * N;
            void* p;
            int32_t s = fg_ws_ensure(ctx, n * 4 + 512);
            if (s != FG_OK) return s;
            if ((s = fg_ws_alloc(ctx, n * 4, &p)) != FG_OK) return s;
            if (dense_z) s = fg_act_bwd_launch(ctx, n, act, dY, saved, (float*)p);
            else {
                PrepArgs a{};
                a.x = dY; a.saved = saved; a.act = act; a.R = M; a.C = N; a.x_batch = strideC; a.out = p; a.ld = N;
                PrepBatch prep;
                if ((s = prep.add(ctx, FG_DTYPE_F32, a, batch)) == FG_OK) s = prep.launch(ctx);
                sz = (uint64_t)M * N;
            }
            if (s != FG_OK) return s;
            dz = (const float*)p;
        }
        int32_t s;
        const bool large_b = batch_large(ctx, mode, batch, K, N), large_a = batch_large(ctx, mode, batch, M, K);
        FgFmaOp ops[2] = {};
        FgFmaOp &w = ops[0], &x = ops[1];
        w.ta = 1; w.M = K; w.N = N; w.K = M; w.A = A; w.B = dz; w.C = dB; w.sA = strideA; w.sB = sz; w.sC = strideB;
        x.tb = 1; x.M = M; x.N = K; x.K = N; x.A = dz; x.B = B; x.C = dA; x.sA = sz; x.sB = strideB; x.sC = strideA;
        // one launch for both where nothing was formed before, unless a gradient lies over what the other product reads
        const uint64_t na = ((batch - 1) * strideA + (uint64_t)M * K) * 4, nb = ((batch - 1) * strideB + (uint64_t)K * N) * 4,
                       nc = ((batch - 1) * sz + (uint64_t)M * N) * 4;
        auto over = [&](const void* p, uint64_t n) { return fg_ranges_meet(p, n, A, na) || fg_ranges_meet(p, n, B, nb) || fg_ranges_meet(p, n, dz, nc); };
        if (dA && dB && act == FG_ACT_NONE && mode == FG_GEMM_AUTO && large_a == large_b && !over(dA, na) && !over(dB, nb)) {
            return large_a ? fg_gemm_fma_launch(ctx, ops, 2, batch, true)
                           : fg_gemm_simt_batched_bwd_launch(ctx, batch, M, N, K, A, strideA, B, strideB, dz, sz, dA, dB);
        }
        if (dB && (s = fg_gemm_simt_batched_launch(ctx, 1, 0, batch, K, N, M, A, strideA, dz, sz, dB, strideB, nullptr, FG_ACT_NONE, nullptr)) != FG_OK) return s;
        return dA ? fg_gemm_simt_batched_launch(ctx, 0, 1, batch, M, K, N, dz, sz, B, strideB, dA, strideA, nullptr, FG_ACT_NONE, nullptr) : FG_OK;
    }
    if (batch_route_open(ctx, mode, M, N, K)) {
        const bool n8 = N % 8 == 0 && K % 8 == 0;
        const bool all = M <= 65535u * 32u && (!dB || batch_converts(ctx, batch, K, N, M, n8 && paired_shape_ok(ctx, K, N, M, K, N))) &&
                         (!dA || batch_converts(ctx, batch, M, K, N, n8 && paired_shape_ok(ctx, M, K, N, N, N)));
        const bool own_z = act != FG_ACT_NONE;
        auto need = [&](uint32_t t) {
            return (own_z ? (uint64_t)t * M * round4(N) * 4 + 256 : copy32_bytes(dY, M, N, t, strideC)) +
                   (dB ? copy32_bytes(A, M, K, t, strideA) : 0) +
                   (dA ? copy32_bytes(B, K, N, t, strideB) : 0) + 2048;
        };
        const uint64_t loop = 2048 + (dA ? planes_bytes(1, M, N) + planes_bytes(1, K, N) + kPairPartialBytes : 0) +
                              (dB ? planes_bytes(1, N, M) + planes_bytes(1, K, M) + kPairPartialBytes : 0);
        const uint32_t part = all ? batch_part(ctx, batch, loop, need) : 0;
        // dZ for a part of the batch in one pass, then one launch for the product or both
        for (uint32_t t0 = 0; t0 < batch && all; t0 += part) {
            const uint32_t t = batch - t0 < part ? batch - t0 : part;
            const float* const dy = dY + t0 * strideC;
            PlaneSet z, xa, xb;
            PrepBatch prep;
            ConvProduct both[2];
            ctx->ws_used = 0;
            int32_t s = fg_ws_ensure(ctx, need(t));
            if (s != FG_OK) return s;
            if (own_z) {
                void* p;
                if ((s = fg_ws_alloc(ctx, (uint64_t)t * M * round4(N) * 4, &p)) != FG_OK) return s;
                PrepArgs a{};
                a.x = dy; a.saved = saved + t0 * strideC; a.act = act; a.R = M; a.C = N; a.x_batch = strideC; a.out = p; a.ld = round4(N);
                if ((s = prep.add(ctx, FG_DTYPE_F32, a, t)) != FG_OK) return s;
                z = PlaneSet{};
                z.p32 = (float*)p;
                z.ld32 = round4(N);
                z.batch32 = (uint64_t)M * round4(N);
            } else if ((s = loadable32(ctx, dy, M, N, t, strideC, &z, &prep)) != FG_OK) return s;
            if (dB && (s = loadable32(ctx, A + t0 * strideA, M, K, t, strideA, &xa, &prep)) != FG_OK) return s;
            if (dA && (s = loadable32(ctx, B + t0 * strideB, K, N, t, strideB, &xb, &prep)) != FG_OK) return s;
            if ((s = prep.launch(ctx)) != FG_OK) return s;
            if (dB) {
                Epilogue ep{dB + t0 * strideB, nullptr, nullptr, K, N, M, FG_ACT_NONE, ctx->dev_status};
                ep.c_batch = t > 1 ? strideB : 0;
                both[0] = ConvProduct{as_operand(xa, true), as_operand(z, true), ep, t};
                if (!dA && (s = launch_conv(ctx, &both[0], 1, plan_conv(ctx, K, N, M, t))) != FG_OK) return s;
            }
            if (dA) {
                Epilogue ep{dA + t0 * strideA, nullptr, nullptr, M, K, N, FG_ACT_NONE, ctx->dev_status};
                ep.c_batch = t > 1 ? strideA : 0;
                both[1] = ConvProduct{as_operand(z, false), as_operand(xb, false), ep, t};
                if ((s = dB ? launch_conv_both(ctx, both[0], both[1]) : launch_conv(ctx, &both[1], 1, plan_conv(ctx, M, K, N, t))) != FG_OK) return s;
            }
        }
        if (all) return FG_OK;
    }
    for (uint32_t t = 0; t < batch; ++t) {
        int32_t s = fg_gemm_bwd_f32(ctx, batch_loop_mode(ctx, mode, M, N, K), M, N, K, A ? A + t * strideA : nullptr, B ? B + t * strideB : nullptr,
                                    dY + t * strideC, act, saved ? saved + t * strideC : nullptr,
                                    dA ? dA + t * strideA : nullptr, dB ? dB + t * strideB : nullptr, nullptr, nullptr);
        if (s != FG_OK) return s;
    }
    return FG_OK;
}

}  // extern "C"

// ------------------------------------------------------------------------------------
// 16-bit storage (f16 / bf16 tensors, f32 accumulation).  The operands are multiplied as they
// lie: one kind::f16 MMA per 16 values of k, read through K-major or MN-major descriptors, so
// nothing is transposed.  What the loads need is a 16-byte aligned base and row pitch; a tensor
// without them is copied once with its pitch padded, and dZ = dY * act'(saved) is formed once
// (both by prep_kernel, which also sums dZ's columns for the bias gradient).
// ------------------------------------------------------------------------------------
namespace {

inline uint32_t pad8(uint32_t x) { return (x + 7u) & ~7u; }
// A dense [rows, cols] tensor can be loaded in place when every row starts on a 16-byte boundary.
inline bool in_place16(const void* p, uint32_t cols) { return fg_aligned16(p) && cols % 8 == 0; }
inline uint64_t copy16_bytes(const void* p, uint32_t rows, uint32_t cols) { return in_place16(p, cols) ? 0 : (uint64_t)rows * pad8(cols) * 2 + 256; }

// x itself, or its copy with a padded pitch; *ld receives the pitch.
int32_t loadable16(fg_ctx* ctx, int dtype, const void* x, uint32_t rows, uint32_t cols, const void** out, uint32_t* ld, PrepBatch* prep) {
    *out = x;
    *ld = cols;
    if (in_place16(x, cols)) return FG_OK;
    void* p;
    int32_t s = fg_ws_alloc(ctx, (uint64_t)rows * pad8(cols) * 2, &p);
    if (s != FG_OK) return s;
    PrepArgs a{};
    a.x = x; a.R = rows; a.C = cols; a.out = p; a.ld = pad8(cols);
    *out = p;
    *ld = a.ld;
    return prep->add(ctx, dtype, a);
}

// An operand whose rows are the output's rows or columns; mn: the storage is [contraction][rows].
PlaneSet operand16(const void* p, uint32_t ld, bool mn) {
    PlaneSet o{};
    o.p16 = (__nv_bfloat16*)p;
    o.ld16 = ld;
    o.mn = mn;
    return o;
}

Epilogue epilogue16(const fg_ctx* ctx, int dtype, uint32_t M, uint32_t N, uint32_t K, void* C, const void* bias, int act, void* preact) {
    return Epilogue{(float*)C, (const float*)bias, (float*)preact, M, N, K, act, ctx->dev_status, nullptr, 0, 1, dtype};
}
// The pair kernel or the half kernel, whichever is estimated to end first (option gemm_tile: the pair kernel; gemm_conv: the other).
bool half_suits(const fg_ctx* ctx, const ConvShape& sh, ConvPlan* plan) {
    if (ctx->opt_tile_pair == 1) return false;
    *plan = plan_half(ctx, &sh, 1);
    return ctx->opt_conv_bn || plan->cycles <= pair16_cycles(ctx, sh);
}
int32_t launch_pair16(fg_ctx* ctx, const ConvProduct& p) {
    return p.ep.out_dtype == FG_DTYPE_BF16 ? launch_tc_pair<32, 2>(ctx, p.a, p.b, p.ep) : launch_tc_pair<32, 3>(ctx, p.a, p.b, p.ep);
}
// Two products in a launch of the pair kernel, the one with the longer k first.
template <int FMT>
int32_t launch_pair16_two(fg_ctx* ctx, const ConvProduct* pr, const PairRuns& r) {
    using Cfg = PairCfg<32, FMT>;
    CUtensorMap tm[4];
    PairArgs<true> pa{};
    double flop = 0.0;
    for (int j = 0; j < 2; ++j) {
        const ConvProduct& c = pr[j];
        int32_t s;
        if ((s = pair16_map<FMT>(ctx, &tm[2 * j], c.a, c.ep.M, c.ep.K, BM)) != FG_OK) return s;
        if ((s = pair16_map<FMT>(ctx, &tm[2 * j + 1], c.b, c.ep.N, c.ep.K, Cfg::kBN / 2)) != FG_OK) return s;
        pa.ep[j] = c.ep;
        pa.ep[j].a_mn = c.a.mn ? 1u : 0u;
        pa.ep[j].b_mn = c.b.mn ? 1u : 0u;
        pa.ep[j].group = pair_group(ctx, c.ep.K);
        pa.ep[j].t_full = (uint32_t)pair_tiles(conv_shape(c));
        flop += 2.0 * c.ep.M * c.ep.N * c.ep.K;
    }
    pa.extra = r.extra;
    pa.run[0] = r.run[0]; pa.run[1] = r.run[1];
    FG_CUDA(ctx, FG_ERR_INTERNAL, (pair_attr<32, FMT, true>(ctx)));
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_GEMM_TC, flop);
    gemm_tc_pair_kernel<32, FMT, true><<<(unsigned)(2 * r.pairs), kPairThreads, Cfg::kSmemBytes, ctx->stream>>>(tm[2], tm[3], tm[0], tm[1], pa);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}
int32_t lowp_gemm(fg_ctx* ctx, const ConvProduct& p) {
    ConvPlan plan;
    return half_suits(ctx, conv_shape(p), &plan) ? launch_half(ctx, &p, 1, plan) : launch_pair16(ctx, p);
}
// Both gradients of a layer, dB first: one launch where they are estimated to end sooner together and neither lies over what the
// other reads (layer of 2048 x 4096 x 4096: 122 -> 113 us for the two).
int32_t lowp_gemm_both(fg_ctx* ctx, const ConvProduct& dB, const ConvProduct& dA) {
    ConvPlan b, a;
    const bool hb = half_suits(ctx, conv_shape(dB), &b), ha = half_suits(ctx, conv_shape(dA), &a);
    auto over = [](const ConvProduct& w, const ConvProduct& r) {
        const uint64_t n = (uint64_t)w.ep.M * w.ep.N * 2;
        return fg_ranges_meet(w.ep.C, n, r.a.p16, (uint64_t)(r.a.mn ? r.ep.K : r.ep.M) * r.a.ld16 * 2) ||
               fg_ranges_meet(w.ep.C, n, r.b.p16, (uint64_t)(r.b.mn ? r.ep.K : r.ep.N) * r.b.ld16 * 2);
    };
    if (!over(dB, dA) && !over(dA, dB)) {
        const ConvProduct pr[2] = {dB.ep.K >= dA.ep.K ? dB : dA, dB.ep.K >= dA.ep.K ? dA : dB};      // the longer k first
        const ConvShape sh[2] = {conv_shape(pr[0]), conv_shape(pr[1])};
        // (a second launch costs 2500 more than the estimates know)
        const double apart = (hb ? b.cycles : pair16_cycles(ctx, conv_shape(dB))) + (ha ? a.cycles : pair16_cycles(ctx, conv_shape(dA))) + 2500.0;
        const uint64_t slots = ctx->opt_conv_bn ? 0 : dB.ep.out_dtype == FG_DTYPE_BF16 ? pair_slots<32, 2>(ctx) : pair_slots<32, 3>(ctx);
        const uint64_t n0 = pair_tiles(sh[0]), n1 = pair_tiles(sh[1]);
        PairRuns runs{};
        if (slots && n0 + n1 < (1ull << 24)) runs = pair_runs(slots, n0, pair16_tile(sh[0]), n1, pair16_tile(sh[1]));
        const double pairs = runs.pairs ? runs.cost + kPair16Around : 1e30;
        const ConvPlan half = ctx->opt_tile_pair == 1 ? ConvPlan{128, 1, 1e30} : plan_half(ctx, sh, 2);
        if (hb && ha && half.cycles <= apart && half.cycles <= pairs) return launch_half(ctx, pr, 2, half);
        if (pairs < apart) return dB.ep.out_dtype == FG_DTYPE_BF16 ? launch_pair16_two<2>(ctx, pr, runs) : launch_pair16_two<3>(ctx, pr, runs);
    }
    const int32_t s = hb ? launch_half(ctx, &dB, 1, b) : launch_pair16(ctx, dB);
    return s != FG_OK ? s : ha ? launch_half(ctx, &dA, 1, a) : launch_pair16(ctx, dA);
}

}  // namespace

extern "C" {

int32_t fg_gemm_lowp(fg_ctx* ctx, int32_t dtype, uint32_t M, uint32_t N, uint32_t K, const void* A, const void* B, void* C,
                     const void* bias, int32_t act, void* preact_out) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, dtype == FG_DTYPE_F16 || dtype == FG_DTYPE_BF16, "fg_gemm_lowp: dtype must be f16 or bf16");
    FG_REQUIRE(ctx, A && B && C, "fg_gemm_lowp: NULL operand");
    FG_REQUIRE(ctx, M >= 1 && N >= 1 && K >= 1, "fg_gemm_lowp: dimensions must be >= 1");
    FG_REQUIRE(ctx, act >= FG_ACT_NONE && act <= FG_ACT_GELU, "fg_gemm_lowp: unknown activation");
    FG_REQUIRE(ctx, fg_aligned16(C) && (!preact_out || fg_aligned16(preact_out)), "fg_gemm_lowp: outputs must be 16-byte aligned");
    if (!ctx->tmap_encode) return fg_fail(ctx, FG_ERR_UNSUPPORTED_FEATURE, "fg_gemm_lowp: tensor maps unavailable");
    const uint64_t need = copy16_bytes(A, M, K) + copy16_bytes(B, K, N) + kPairPartialBytes + 2048;
    { int32_t s0 = fg_ws_ensure(ctx, need); if (s0 != FG_OK) return s0; }
    int32_t s;
    const void *a, *b;
    uint32_t lda, ldb;
    PrepBatch prep;
    if ((s = loadable16(ctx, dtype, A, M, K, &a, &lda, &prep)) != FG_OK) return s;
    if ((s = loadable16(ctx, dtype, B, K, N, &b, &ldb, &prep)) != FG_OK) return s;
    if ((s = prep.launch(ctx)) != FG_OK) return s;
    // A [M][K] has the contraction index contiguous, B [K][N] its rows (the output's columns)
    return lowp_gemm(ctx, ConvProduct{operand16(a, lda, false), operand16(b, ldb, true), epilogue16(ctx, dtype, M, N, K, C, bias, act, preact_out), 1});
}

int32_t fg_gemm_bwd_lowp(fg_ctx* ctx, int32_t dtype, uint32_t M, uint32_t N, uint32_t K, const void* A, const void* B,
                         const void* dY, int32_t act, const void* saved, void* dA, void* dB, void* dbias) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, dtype == FG_DTYPE_F16 || dtype == FG_DTYPE_BF16, "fg_gemm_bwd_lowp: dtype must be f16 or bf16");
    FG_REQUIRE(ctx, dY != nullptr, "fg_gemm_bwd_lowp: dY is NULL");
    FG_REQUIRE(ctx, M >= 1 && N >= 1 && K >= 1, "fg_gemm_bwd_lowp: dimensions must be >= 1");
    FG_REQUIRE(ctx, act >= FG_ACT_NONE && act <= FG_ACT_GELU, "fg_gemm_bwd_lowp: unknown activation");
    FG_REQUIRE(ctx, act == FG_ACT_NONE || saved, "fg_gemm_bwd_lowp: the activation backward needs the saved tensor");
    FG_REQUIRE(ctx, !dA || B, "fg_gemm_bwd_lowp: dA needs B");
    FG_REQUIRE(ctx, !dB || A, "fg_gemm_bwd_lowp: dB needs A");
    FG_REQUIRE(ctx, (!dA || fg_aligned16(dA)) && (!dB || fg_aligned16(dB)), "fg_gemm_bwd_lowp: outputs must be 16-byte aligned");
    if (!ctx->tmap_encode) return fg_fail(ctx, FG_ERR_UNSUPPORTED_FEATURE, "fg_gemm_bwd_lowp: tensor maps unavailable");
    const bool fuse = act != FG_ACT_NONE;
    const bool dz_direct = !fuse && in_place16(dY, N);       // dZ == dY, loadable as it lies
    const uint32_t nchunk_rows = (M + 31) / 32;
    uint64_t need = 4096 + 2 * kPairPartialBytes;
    if ((dA || dB) && !dz_direct) need += (uint64_t)M * pad8(N) * 2 + 256;
    if (dA) need += copy16_bytes(B, K, N);
    if (dB) need += copy16_bytes(A, M, K);
    if (dbias) need += (uint64_t)nchunk_rows * N * 4 + 256;
    { int32_t s0 = fg_ws_ensure(ctx, need); if (s0 != FG_OK) return s0; }
    int32_t s;
    void *dz = const_cast<void*>(dY), *cs_part = nullptr;
    PrepArgs pz{};
    pz.x = dY; pz.saved = fuse ? saved : nullptr; pz.act = act; pz.R = M; pz.C = N;
    if ((dA || dB) && !dz_direct) {
        if ((s = fg_ws_alloc(ctx, (uint64_t)M * pad8(N) * 2, &dz)) != FG_OK) return s;
        pz.out = dz; pz.ld = pad8(N);
    }
    const uint32_t ldz = pz.out ? pz.ld : N;
    if (dbias) {
        if ((s = fg_ws_alloc(ctx, (uint64_t)nchunk_rows * N * 4, &cs_part)) != FG_OK) return s;
        pz.colsum_part = (float*)cs_part;
    }
    // dZ and the copies of what cannot be read in place: one launch
    PrepBatch prep;
    const void *xa = nullptr, *xb = nullptr;
    uint32_t lda = 0, ldb = 0;
    if ((pz.out || pz.colsum_part) && (s = prep.add(ctx, dtype, pz)) != FG_OK) return s;
    if (dB && (s = loadable16(ctx, dtype, A, M, K, &xa, &lda, &prep)) != FG_OK) return s;
    if (dA && (s = loadable16(ctx, dtype, B, K, N, &xb, &ldb, &prep)) != FG_OK) return s;
    if ((s = prep.launch(ctx)) != FG_OK) return s;
    if (dbias && (s = fg_colsum_fold_launch(ctx, N, nchunk_rows, (const float*)cs_part, dbias, dtype)) != FG_OK) return s;
    // dB[K,N] = A^T · dZ: contraction over M, the row index of both tensors; dA[M,K] = dZ · B^T: contraction over N, contiguous in both
    const ConvProduct w{operand16(xa, lda, true), operand16(dz, ldz, true), epilogue16(ctx, dtype, K, N, M, dB, nullptr, FG_ACT_NONE, nullptr), 1};
    const ConvProduct v{operand16(dz, ldz, false), operand16(xb, ldb, false), epilogue16(ctx, dtype, M, K, N, dA, nullptr, FG_ACT_NONE, nullptr), 1};
    if (dB && dA) return lowp_gemm_both(ctx, w, v);
    return dB ? lowp_gemm(ctx, w) : dA ? lowp_gemm(ctx, v) : FG_OK;
}

}  // extern "C"

// ---- self-test of the bounded waits ----
namespace {
__global__ void bounded_wait_selftest_kernel(int* dev_status, unsigned* arrivals, long long max_cycles) {
    __shared__ unsigned long long bar;
    if (threadIdx.x == 0) {
        atomicInc(arrivals, 1u);      // the first of two blocks of which the other gives up uncounted
        mbar_init(smem_u32(&bar), 1);
        fence_mbar_init();
        // nobody arrives on this barrier: the wait must give up after max_cycles and report it
        if (!mbar_wait_bounded(smem_u32(&bar), 0, max_cycles)) atomicOr(dev_status, FG_DEVERR_EPI_WAIT);
    }
}
}  // namespace

extern "C" int32_t fg_selftest_bounded_wait(fg_ctx* ctx, uint32_t max_cycles) {
    FG_ENTER(ctx);
    const long long limit = max_cycles > 1000000u ? 1000000ll : (long long)max_cycles;
    bounded_wait_selftest_kernel<<<1, 32, 0, ctx->stream>>>(ctx->dev_status, fg_arrivals(ctx), limit);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

#ifdef FG_GEMM_PROFILE
extern "C" int32_t fg_gemm_profile_read(unsigned long long out[8]) {
    unsigned long long zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (cudaDeviceSynchronize() != cudaSuccess) return FG_ERR_SYNC;
    if (cudaMemcpyFromSymbol(out, g_prof, sizeof(zero)) != cudaSuccess) return FG_ERR_INTERNAL;
    if (cudaMemcpyToSymbol(g_prof, zero, sizeof(zero)) != cudaSuccess) return FG_ERR_INTERNAL;
    return FG_OK;
}
#endif

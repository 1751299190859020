// f32 products with plain FMAs in shares of k: what FG_GEMM_AUTO runs where the tensor-core kernels' fixed costs, or their tiles of
// 128 rows, are the most of a product -- fewer than 64 samples, or up to some 20 to 45 million multiply-adds (fg_gemm_fma_suits) --
// forward and both gradients, but for forward products of a short k (fg_gemm_simt_suits) and narrow layers of many rows
// (fg_gemm_fma_suits_small).
//
// What it replaces: the reference's tiled matmul and its backward edges (crates/ferrograd-nn/src/op/matmul/mod.rs:17-188,
// generic.rs:13-325) with the elementwise work around them: bias and activation (kernel/forward.rs:373-457), the activation's
// derivative on dY (op/unary.rs:281-309, :453-472, :588-714), that of the layer below on dA, and the bias gradients.
//
// Bound by HBM for a few samples (the weights are read once), by shared memory's words into the FMAs above about twenty, and by
// launches and latencies for the smallest.  So: 16-byte asynchronous copies two or three stages ahead into shared memory, the
// tensors as they lie; a thread owns 4 to 8 rows x 4 or 8 columns; the k of a stage are dealt to groups of threads, of which a
// tile of few rows has more; the stages to the CTAs of a cluster, whose sums meet through distributed shared memory (no scratch,
// no second launch).  Both gradients of a layer, the activation's derivative on dZ and the bias gradient are one launch.
// Measured against one launch of sequential sums per product (us, on the device): 4096 x 4096 weights with 1 / 8 / 24 / 48 samples 72 /
// 73 / 127 / 163 -> 11 / 18 / 35 / 53, 8192 x 8192 with 16 samples 228 -> 68 (4.0 TB/s), 39 x 2016 x 288 38 -> 7; backward of
// 960 x 61 x 32 25 -> 8 and of 1544 x 37 x 12 36 -> 12; the steps of 2-16-2 (64 samples) 26.7 -> 22.7 and of
// 427-32-26-95 (128 samples) 69.8 -> 39.0.
#include <atomic>

#include "fg_internal.cuh"
#include "ptx_sm100.cuh"

namespace {

constexpr int kT = 256, kTN = 64;      // threads, columns of a tile

struct FmaArgs {
    const float *A, *B;
    const float* factor;      // dZ operand (B of a product with A transposed, A of one with B transposed) is x * act'(factor)
    const float *bias, *mul_saved;
    float *C, *preact;
    float* colsum_b;          // [N]: column sums of the B operand over k (the layer's bias gradient)
    float* colsum_c;          // [N] column sums of C, or, of several tiles down, [ceil(M / 32)][N] of 32 rows each
    __nv_bfloat16* pairs;
    uint64_t pairs_stride, sA, sB, sC;
    uint32_t M, N, K, tiles_m, tiles;      // tiles of one matrix
    int act, factor_act, mul_act;
    bool a16, b16, c16;                    // 16-byte accesses to A (and its factor), to B (and its), to what the epilogue touches
};
template <int N>
struct FmaLaunch {
    FmaArgs p[N];
    uint32_t units0, units, lg_split, batch;
};

// A tile of TM x 64: groups of TM * 64 / (RM * RN) threads take the k quads of a stage of TK in turn, a thread RM rows x RN columns.
template <int TM_, int RM_, int RN_, int TK_, int S_>
struct Tile {
    static constexpr int TM = TM_, RM = RM_, RN = RN_, TK = TK_, S = S_, TX = kTN / RN, TY = TM / RM, G = kT / (TX * TY);
    static constexpr int KS = RN == 4 ? 4 : 2, PK = TK + 4;      // k per step, pitch of a k-contiguous tile
    static_assert(TK / KS % G == 0 && TM * kTN * G * 4 <= 65536, "every group has its steps");
};
using Tile4 = Tile<4, 4, 4, 64, 4>;
using Tile16 = Tile<16, 8, 4, 64, 3>;
using Tile32 = Tile<32, 8, 4, 32, 4>;
using Tile64 = Tile<64, 8, 8, 32, 3>;
// One group and no shares: every sum is one chain of FMAs in the order of k (batches, which promise the exact path's results).
using TileOrdered = Tile<64, 4, 4, 32, 3>;

// Words of one stage: A, B and the factor's block.  Columns-contiguous operands lie as [k][cols], k-contiguous ones as [row][TK + 4],
// whose rows start four banks apart: the lanes' wide reads of eight rows meet no bank twice.
struct FmaStage { uint32_t a, b, f; };
template <typename T>
__host__ __device__ constexpr FmaStage fma_stage(bool ta, bool tb, bool factor) {
    const uint32_t a = ta ? T::TK * T::TM : T::TM * T::PK, b = tb ? kTN * T::PK : T::TK * kTN;
    return FmaStage{a, b, !factor ? 0u : ta ? b : a};
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(fgptx::smem_u32(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4(float* dst, const float* src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(fgptx::smem_u32(dst)), "l"(src), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The chunks of V words of a ROWS x COLS block that a thread copies (and multiplies): row r0 + i * STEP, column c.
template <int ROWS, int COLS, int V>
struct Chunks {
    static constexpr int PER_ROW = COLS / V, STEP = kT / PER_ROW, N = (ROWS + STEP - 1) / STEP;
    static_assert(PER_ROW <= kT && kT % PER_ROW == 0, "whole rows per pass");
    static __device__ __forceinline__ uint32_t row() { return threadIdx.x / PER_ROW; }
    static __device__ __forceinline__ uint32_t col() { return threadIdx.x % PER_ROW * V; }
    static __device__ __forceinline__ bool inside(uint32_t r) { return ROWS % STEP == 0 || r < ROWS; }
};
// src: the block's first element; zero behind `rows` and `cols` (with V = 4 `cols` is a multiple of four).
template <int ROWS, int COLS, int V>
__device__ __forceinline__ void copy_chunks(float* dst, uint32_t pitch, const float* src, uint32_t ld, uint32_t rows, uint32_t cols) {
    using C = Chunks<ROWS, COLS, V>;
    uint32_t r = C::row();
    const uint32_t c = C::col();
    const float* s = src + (size_t)r * ld + c;
    const size_t step = (size_t)C::STEP * ld;
#pragma unroll
    for (int i = 0; i < C::N; ++i, r += C::STEP, s += step) {
        if (!C::inside(r)) break;
        const bool live = r < rows && c < cols;
        if (V == 4) cp16(dst + r * pitch + c, live ? s : src, live);
        else cp4(dst + r * pitch + c, live ? s : src, live);
    }
}
template <int ROWS, int COLS>
__device__ __forceinline__ void copy_block(float* dst, uint32_t pitch, const float* src, uint32_t ld, uint32_t rows, uint32_t cols, bool v16) {
    if (v16) copy_chunks<ROWS, COLS, 4>(dst, pitch, src, ld, rows, cols);
    else copy_chunks<ROWS, COLS, 1>(dst, pitch, src, ld, rows, cols);
}
// dst *= act'(fac), the elements that this thread copied itself: no barrier between the copy and this.  The activation is chosen once
// and the chunks are unrolled, so that their chains run side by side (chosen for each element, backward of 1936 x 19 x 958 took
// twice as long).
template <int ROWS, int COLS, int V, int ACT>
__device__ __forceinline__ void factor_chunks(float* dst, const float* fac, uint32_t pitch) {
    using C = Chunks<ROWS, COLS, V>;
    const uint32_t r0 = C::row(), c = C::col();
#pragma unroll 4
    for (int i = 0; i < C::N; ++i) {
        const uint32_t r = r0 + i * C::STEP, o = r * pitch + c;
        if (!C::inside(r)) break;
        if constexpr (V == 4) {
            float4 v = *reinterpret_cast<float4*>(dst + o);
            const float4 s = *reinterpret_cast<const float4*>(fac + o);
            v.x *= fg_act_grad(ACT, s.x); v.y *= fg_act_grad(ACT, s.y); v.z *= fg_act_grad(ACT, s.z); v.w *= fg_act_grad(ACT, s.w);
            *reinterpret_cast<float4*>(dst + o) = v;
        } else {
            dst[o] *= fg_act_grad(ACT, fac[o]);
        }
    }
}
template <int ROWS, int COLS>
__device__ __forceinline__ void factor_block(float* dst, const float* fac, uint32_t pitch, bool v16, int act) {
    if (act == FG_ACT_GELU) {
        if (v16) factor_chunks<ROWS, COLS, 4, FG_ACT_GELU>(dst, fac, pitch);
        else factor_chunks<ROWS, COLS, 1, FG_ACT_GELU>(dst, fac, pitch);
    } else if (act == FG_ACT_TANH) {
        if (v16) factor_chunks<ROWS, COLS, 4, FG_ACT_TANH>(dst, fac, pitch);
        else factor_chunks<ROWS, COLS, 1, FG_ACT_TANH>(dst, fac, pitch);
    } else {
        if (v16) factor_chunks<ROWS, COLS, 4, FG_ACT_RELU>(dst, fac, pitch);
        else factor_chunks<ROWS, COLS, 1, FG_ACT_RELU>(dst, fac, pitch);
    }
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// Two FMAs in one instruction, each rounded as fmaf.  For the forward product alone, whose pairs of columns come from shared memory as
// they are used: 8192 x 8192 weights with 63 samples 244 -> 226 us; the gradients' operands would have to be put together (backward
// of 31 x (60 x 500 x 500) 84 -> 91 us).
__device__ __forceinline__ void fma2(float& c0, float& c1, float a, float b0, float b1) {
    asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %2};\n mov.b64 y, {%3, %4};\n mov.b64 z, {%0, %1};\n fma.rn.f32x2 z, x, y, z;\n mov.b64 {%0, %1}, z;\n}"
        : "+f"(c0), "+f"(c1) : "f"(a), "f"(b0), "f"(b1));
}
// One unit (a tile of one matrix), or this CTA's share of its k.  Thread: group g of k steps, rows ty, columns tx.
template <typename T, bool TA, bool TB>
__device__ __forceinline__ void fma_unit(const FmaArgs& p, uint32_t unit, uint32_t share, uint32_t lg_split, uint32_t batch, float* sm) {
    constexpr int TM = T::TM, RM = T::RM, RN = T::RN, TK = T::TK, PK = T::PK, S = T::S, G = T::G, TX = T::TX, TY = T::TY, KS = T::KS;
    constexpr bool kHasFactor = TA != TB;
    const uint32_t tid = threadIdx.x, tx = tid % TX, ty = tid / TX % TY, g = tid / (TX * TY), split = 1u << lg_split;
    const uint32_t bz = batch > 1 ? unit / p.tiles : 0u, tile = batch > 1 ? unit % p.tiles : unit;
    const uint32_t tm = p.tiles_m > 1 ? tile % p.tiles_m : 0u, m0 = tm * TM, n0 = (p.tiles_m > 1 ? tile / p.tiles_m : tile) * kTN;
    const bool factor = kHasFactor && p.factor;
    const FmaStage st = fma_stage<T>(TA, TB, factor);
    const uint32_t words = st.a + st.b + st.f;
    const uint32_t nk = (p.K + TK - 1) / TK, t0 = (uint32_t)((uint64_t)share * nk >> lg_split), t1 = (uint32_t)((uint64_t)(share + 1) * nk >> lg_split);
    const uint32_t lda = TA ? p.M : p.K, ldb = TB ? p.K : p.N, ra = p.M - m0, rb = p.N - n0;      // rows and columns from here on
    // the first k of this share; a stage further on is `step_a` and `step_b` words on
    const size_t at_a = TA ? (size_t)t0 * TK * lda + m0 : (size_t)m0 * lda + (size_t)t0 * TK;
    const size_t at_b = TB ? (size_t)n0 * ldb + (size_t)t0 * TK : (size_t)t0 * TK * ldb + n0;
    const size_t step_a = TA ? (size_t)TK * lda : TK, step_b = TB ? TK : (size_t)TK * ldb;
    const float *a_src = p.A + bz * p.sA + at_a, *b_src = p.B + bz * p.sB + at_b;
    const float* f_src = factor ? p.factor + (TA ? bz * p.sB + at_b : bz * p.sA + at_a) : nullptr;

    auto copy_a = [&](float* dst, const float* src, uint32_t left) {
        if (!TA) copy_block<TM, TK>(dst, PK, src, lda, ra, left, p.a16);
        else copy_block<TK, TM>(dst, TM, src, lda, left, ra, p.a16);
    };
    auto copy_b = [&](float* dst, const float* src, uint32_t left) {
        if (!TB) copy_block<TK, kTN>(dst, kTN, src, ldb, left, rb, p.b16);
        else copy_block<kTN, TK>(dst, PK, src, ldb, rb, left, p.b16);
    };
    uint32_t next = t0, slot_in = 0;
    auto load = [&]() {
        if (next < t1) {
            float* const s = sm + slot_in * words;
            const uint32_t left = p.K - next * TK;
            copy_a(s, a_src, left);
            copy_b(s + st.a, b_src, left);
            if constexpr (kHasFactor) {
                if (factor) {
                    if (TA) copy_b(s + st.a + st.b, f_src, left);
                    else copy_a(s + st.a + st.b, f_src, left);
                    f_src += TA ? step_b : step_a;
                }
            }
            a_src += step_a;
            b_src += step_b;
            ++next;
            slot_in = slot_in + 1 == S ? 0 : slot_in + 1;
        }
        cp_commit();      // a group per stage, empty behind the last one, so that the count below holds
    };
#pragma unroll 1
    for (int i = 0; i < S - 1; ++i) load();
    // This CTA finishes a range of column quads, all rows of it.
    const uint32_t lgq = 4 - lg_split, nq = 1u << lgq, q0 = share << lgq, col = n0 + (q0 + (tid & (nq - 1))) * 4;
    float bz4[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) bz4[j] = p.bias && col + j < p.N ? p.bias[col + j] : 0.0f;

    float acc[RM][RN];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = 0.0f;
    const bool sum_b = TA && !TB && p.colsum_b && tm == 0;
    float csb = 0.0f, stages = 0.0f;      // a thread's share of a column's sum, and of that the last few stages'
    uint32_t slot = 0;
#pragma unroll 1
    for (uint32_t t = t0; t < t1; ++t) {
        float* const As = sm + slot * words;
        float* const Bs = As + st.a;
        slot = slot + 1 == S ? 0 : slot + 1;
        cp_wait<S - 2>();
        if constexpr (kHasFactor) {
            if (factor) {
                if (TA) factor_block<TK, kTN>(Bs, Bs + st.b, kTN, p.b16, p.factor_act);
                else factor_block<TM, TK>(As, Bs + st.b, PK, p.a16, p.factor_act);
            }
        }
        __syncthreads();      // everybody's copies of this stage are here, and nobody reads the one that is filled next
        load();
        if (TA && !TB && sum_b) {
            // A stage's terms in pairs, eight stages and all of them in a chain each.  Error against 64 bits over 36 layers of 34 to 5700
            // rows: 0.6 to 1.2e-7 (column sums in a pass of their own: 0.8 to 1.5e-7; 4214 rows in one chain: 4.2e-7).
            float part[2] = {0.0f, 0.0f};
#pragma unroll 2
            for (int k = 0; k < TK / (kT / kTN); k += 4) {
                const float* const r = Bs + (k * (kT / kTN) + tid / kTN) * kTN + tid % kTN;
                part[0] += r[0] + r[kT];
                part[1] += r[2 * kT] + r[3 * kT];
            }
            stages += part[0] + part[1];
            if ((t & 7u) == 7u) {
                csb += stages;
                stages = 0.0f;
            }
        }
#pragma unroll
        for (int q = 0; q < TK / KS / G; ++q) {
            const uint32_t k0 = (q * G + g) * KS;
            float a[RM][KS], b[KS][RN];
            if (!TA) {
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    const float* const s = As + (ty + TY * i) * PK + k0;
                    if (KS == 4) {
                        const float4 v = *reinterpret_cast<const float4*>(s);
                        a[i][0] = v.x; a[i][1] = v.y; a[i][KS - 2] = v.z; a[i][KS - 1] = v.w;
                    } else {
                        const float2 v = *reinterpret_cast<const float2*>(s);
                        a[i][0] = v.x; a[i][1] = v.y;
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < KS; ++k)
#pragma unroll
                    for (int h = 0; h < RM; h += 4) {
                        const float4 v = *reinterpret_cast<const float4*>(As + (k0 + k) * TM + ty * RM + h);
                        a[h][k] = v.x; a[h + 1][k] = v.y; a[h + 2][k] = v.z; a[h + 3][k] = v.w;
                    }
            }
            if (!TB) {
#pragma unroll
                for (int k = 0; k < KS; ++k)
#pragma unroll
                    for (int h = 0; h < RN; h += 4) {
                        const float4 v = *reinterpret_cast<const float4*>(Bs + (k0 + k) * kTN + tx * 4 + h * TX);
                        b[k][h] = v.x; b[k][h + 1] = v.y; b[k][h + 2] = v.z; b[k][h + 3] = v.w;
                    }
            } else {
#pragma unroll
                for (int j = 0; j < RN; ++j) {
                    const float* const s = Bs + (tx + TX * j) * PK + k0;
                    if (KS == 4) {
                        const float4 v = *reinterpret_cast<const float4*>(s);
                        b[0][j] = v.x; b[1][j] = v.y; b[KS - 2][j] = v.z; b[KS - 1][j] = v.w;
                    } else {
                        const float2 v = *reinterpret_cast<const float2*>(s);
                        b[0][j] = v.x; b[1][j] = v.y;
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < KS; ++k)
#pragma unroll
                for (int i = 0; i < RM; ++i)
#pragma unroll
                    for (int j = 0; j < RN; j += 2) {
                        if (!TA && !TB) fma2(acc[i][j], acc[i][j + 1], a[i][k], b[k][j], b[k][j + 1]);
                        else {
                            acc[i][j] = fmaf(a[i][k], b[k][j], acc[i][j]);
                            acc[i][j + 1] = fmaf(a[i][k], b[k][j + 1], acc[i][j + 1]);
                        }
                    }
        }
    }
    // The groups' sums meet in the stages' room, [group][row][64], then the shares' in distributed shared memory.
    cp_wait<0>();
    __syncthreads();
    __shared__ float colb[kT / kTN][kTN];
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        float* const r = sm + (g * TM + (TA ? ty * RM + i : ty + TY * i)) * kTN;
#pragma unroll
        for (int h = 0; h < RN; h += 4) {
            if (!TB) *reinterpret_cast<float4*>(r + tx * 4 + h * TX) = make_float4(acc[i][h], acc[i][h + 1], acc[i][h + 2], acc[i][h + 3]);
            else
#pragma unroll
                for (int j = h; j < h + 4; ++j) r[tx + TX * j] = acc[i][j];
        }
    }
    if (TA && !TB && sum_b) colb[tid / kTN][tid % kTN] = csb + stages;
    __syncthreads();
    float4* const red = reinterpret_cast<float4*>(sm);
    auto group_sum = [&](uint32_t i) {
        float4 s = red[i];
#pragma unroll
        for (int k = 1; k < G; ++k) s = add4(s, red[k * TM * 16 + i]);
        return s;
    };
    if (split > 1) {
        for (uint32_t i = tid; i < TM * 16; i += kT) red[i] = group_sum(i);
        __syncwarp();
        fgptx::cluster_sync_all();
    }
    float4* const outs = red + TM * 16;      // (where the second group's sums were) what this CTA stores, for the column sums
    for (uint32_t e = tid; e < TM << lgq; e += kT) {
        const uint32_t m = e >> lgq, row = m0 + m, i = m * 16 + q0 + (e & (nq - 1));
        float4 z;
        if (split > 1) {
            const uint32_t at = fgptx::smem_u32(red + i);
            z = fgptx::ld_cluster_f4(fgptx::map_to_cta(at, 0));
            for (uint32_t r = 1; r < split; ++r) z = add4(z, fgptx::ld_cluster_f4(fgptx::map_to_cta(at, r)));
        } else z = group_sum(i);
        if (row >= p.M || col >= p.N) continue;
        const size_t off = bz * p.sC + (size_t)row * p.N + col;
        float zz[4] = {z.x + bz4[0], z.y + bz4[1], z.z + bz4[2], z.w + bz4[3]}, o[4];
        if (p.c16) {
            if (p.preact) *reinterpret_cast<float4*>(p.preact + off) = make_float4(zz[0], zz[1], zz[2], zz[3]);
            float4 sv = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p.mul_saved) sv = *reinterpret_cast<const float4*>(p.mul_saved + off);
            const float s4[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) o[j] = p.mul_saved ? zz[j] * fg_act_grad(p.mul_act, s4[j]) : fg_act_fwd(p.act, zz[j]);
            const float4 v = make_float4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<float4*>(p.C + off) = v;
            if (p.pairs) fg_store_pairs4(p.pairs, p.pairs_stride, off, v);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[j] = 0.0f;
                if (col + j >= p.N) continue;
                if (p.preact) p.preact[off + j] = zz[j];
                o[j] = p.mul_saved ? zz[j] * fg_act_grad(p.mul_act, p.mul_saved[off + j]) : fg_act_fwd(p.act, zz[j]);
                p.C[off + j] = o[j];
                if (p.pairs) fg_store_pairs1(p.pairs, p.pairs_stride, off + j, o[j]);
            }
        }
        if (G > 1 && p.colsum_c) outs[i] = make_float4(o[0], o[1], o[2], o[3]);
    }
    if (G > 1 && p.colsum_c) {
        // In the order of the tensor-core kernels' epilogues: a block of 32 rows in four chains (row r in chain r % 4), which are added
        // in pairs; then the blocks in order.
        __syncthreads();
        const uint32_t q = q0 + (tid >> 2), j = tid & 3u, c = n0 + q * 4 + j;
        if (tid < nq * 4 && c < p.N) {
            float total = 0.0f;
#pragma unroll 1
            for (uint32_t b = 0; b < TM && m0 + b < p.M; b += 32) {
                const uint32_t rows = min(min(32u, (uint32_t)TM), p.M - m0 - b);
                float ch[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
                for (uint32_t r = 0; r < rows; r += 4)
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (r + t < rows) ch[t] += reinterpret_cast<const float*>(outs + (b + r + t) * 16 + q)[j];
                const float sum = (ch[0] + ch[1]) + (ch[2] + ch[3]);
                if (p.tiles_m > 1) p.colsum_c[(size_t)((m0 + b) >> 5) * p.N + c] = sum;
                total += sum;
            }
            if (p.tiles_m == 1) p.colsum_c[c] = total;
        }
    }
    if (TA && !TB && sum_b && share == 0 && tid < kTN) {
        float s = 0.0f;
        for (uint32_t r = 0; r < split; ++r) {
            const uint32_t at = fgptx::smem_u32(&colb[0][tid]);
            float v[kT / kTN];
#pragma unroll
            for (int k = 0; k < kT / kTN; ++k) {
                const uint32_t w = at + k * kTN * 4;
                v[k] = split > 1 ? fgptx::ld_cluster_f(fgptx::map_to_cta(w, r)) : colb[k][tid];
            }
#pragma unroll
            for (int d = 1; d < kT / kTN; d *= 2)
#pragma unroll
                for (int k = 0; k < kT / kTN; k += 2 * d) v[k] += v[k + d];
            s += v[0];
        }
        if (n0 + tid < p.N) p.colsum_b[n0 + tid] = s;
    }
    __syncwarp();
    if (split > 1) fgptx::cluster_sync_all();      // no CTA leaves while another reads its sums
}

// One product.
template <typename T, bool TA, bool TB>
__global__ void __launch_bounds__(kT, 2) gemm_fma_kernel(const __grid_constant__ FmaLaunch<1> l) {
    extern __shared__ __align__(16) float sm[];
    fg_grid_enter();
    fma_unit<T, TA, TB>(l.p[0], blockIdx.x >> l.lg_split, blockIdx.x & ((1u << l.lg_split) - 1), l.lg_split, l.batch, sm);
}
// Both gradients of a layer: dB = Aᵀ·dZ, then dA = dZ·Bᵀ.
template <typename TB_, typename TA_>
__global__ void __launch_bounds__(kT, 2) gemm_fma_bwd_kernel(const __grid_constant__ FmaLaunch<2> l) {
    extern __shared__ __align__(16) float sm[];
    fg_grid_enter();
    const uint32_t u = blockIdx.x >> l.lg_split, share = blockIdx.x & ((1u << l.lg_split) - 1);
    if (u < l.units0) fma_unit<TB_, true, false>(l.p[0], u, share, l.lg_split, l.batch, sm);
    else fma_unit<TA_, false, true>(l.p[1], u - l.units0, share, l.lg_split, l.batch, sm);
}

// What the choice of a tile goes by: log2 of its rows and of a stage's k, SM cycles for a stage.
struct FmaTile { uint32_t lg_tm, lg_tk; float cycles; };
constexpr FmaTile kTiles[4] = {{2, 6, 45.0f}, {4, 6, 430.0f}, {5, 5, 790.0f}, {6, 5, 1530.0f}};

// Are the rows of A, and those of B, copied in 16-byte chunks (with the factor that goes with them)?
struct FmaRows { bool a16, b16; };
bool rows16(const float* x, uint32_t cols, uint64_t stride, uint32_t batch) { return fg_aligned16(x) && cols % 4 == 0 && (batch == 1 || stride % 4 == 0); }
FmaRows fma_rows(const FgFmaOp& o, uint32_t batch) {
    return {rows16(o.A, o.ta ? o.M : o.K, o.sA, batch) && (!o.factor || o.ta || fg_aligned16(o.factor)),
            rows16(o.B, o.tb ? o.K : o.N, o.sB, batch) && (!o.factor || o.tb || fg_aligned16(o.factor))};
}

struct FmaPlan { int tile[2]; uint32_t lg_split; float cycles; };
// Tile heights and K-shares by estimated cycles, fitted to 49 calls under every tile and split (2.2 % slower than the best of each in
// the geometric mean, 22 % at most): a stage takes a CTA no less than its copies' latency (270), the ends of a unit 1430, a meeting of
// shares 180 + 150 each.  The fit counts rounds at three CTAs an SM; two are resident (102 to 128 registers a thread).  For two products the
// rounds of all units times the longest unit of either only puts the plans in order: it is no time, least of all where one of them has many
// units and the other a long k.
// A word that is copied alone and one that is added to a column's sum take 0.05 more:
// with that, the gradients of 28 layers, 13 of them with odd rows, take 7 % more than under the best plan of each in the geometric mean
// and 12 % without (2000 x 100 x 30: 17.7 and 23.1 us); not with 16 columns or fewer, where most of a row's words are only zeroed
// (gradients of 1000 x 100 x 4 9.1 us with it, 7.6 without, 300 x 200 x 13 7.0 and 6.1, 500 x 300 x 10 8.1 and 8.9; by the narrow
// layer's own kernels 25, 12.3 and 17.4).  (The host spends this on every call: shifts, no division.)
FmaPlan fma_plan(const fg_ctx* ctx, const FgFmaOp* ops, int n, uint32_t batch) {
    FmaPlan best{{0, 0}, 0, 0.0f};
    const float sms = (float)fg_free_sms(ctx), per_round = 1.0f / (3.0f * sms), per_sm = 0.4f / sms;
    // a lower tile holds all rows; the caller has room for one row of column sums per 32 rows
    auto usable = [&](const FgFmaOp& o, int i) { return !(i > 0 && o.M <= 1u << kTiles[i - 1].lg_tm) && !(o.colsum_c && i < 2 && o.M > 1u << kTiles[i].lg_tm); };
    for (uint32_t lg = 0; lg <= 3; ++lg) {
        if (lg && (n > 1 ? (ops[0].K > ops[1].K ? ops[0].K : ops[1].K) : ops[0].K) <= 64u << (lg - 1)) break;      // shares without a stage
        float ctas[2][4], work[2][4], alone[2][4];
        for (int j = 0; j < n; ++j) {
            const float cols = (float)((ops[j].N + kTN - 1) / kTN) * batch * (float)(1u << lg);
            const FmaRows rows = fma_rows(ops[j], batch);
            const bool narrow = ops[j].N <= 16 || ops[j].K <= 16;
            const float by_a = rows.a16 || narrow ? 0.0f : ops[j].factor && !ops[j].ta ? 0.1f : 0.05f;
            const float by_b = (rows.b16 || narrow ? 0.0f : ops[j].factor && ops[j].ta ? 0.1f : 0.05f) + (ops[j].colsum_b && !narrow ? 0.05f : 0.0f);
            for (int i = 0; i < 4; ++i) {
                const FmaTile& t = kTiles[i];
                const float more = (by_a * (float)(1u << t.lg_tm) + by_b * kTN) * (float)(1u << t.lg_tk);
                const uint32_t nk = (ops[j].K + (1u << t.lg_tk) - 1) >> t.lg_tk;
                const float steps = (float)((nk + (1u << lg) - 1) >> lg), tail = 1430.0f + (1u << t.lg_tm);
                ctas[j][i] = (float)((ops[j].M + (1u << t.lg_tm) - 1) >> t.lg_tm) * cols;
                work[j][i] = ctas[j][i] * (steps * (t.cycles + more) + 5.3f * tail);
                alone[j][i] = steps * ((kTiles[i].cycles > 270.0f ? kTiles[i].cycles : 270.0f) + more) + tail;
            }
        }
        for (int i = 0; i < 4; ++i) {
            if (!usable(ops[0], i)) continue;
            for (int k = 0; k < (n > 1 ? 4 : 1); ++k) {
                float c = ctas[0][i], w = work[0][i], longest = alone[0][i];
                if (n > 1) {
                    if (!usable(ops[1], k)) continue;
                    c += ctas[1][k];
                    w += work[1][k];
                    if (alone[1][k] > longest) longest = alone[1][k];
                }
                float z = (float)(uint64_t)(c * per_round + 0.9999f) * longest;
                if (c > sms && z < w * per_sm) z = w * per_sm;
                if (lg) z += 180.0f + 150.0f * (float)(1u << lg);
                if (best.cycles == 0.0f || z < best.cycles) best = FmaPlan{{i, k}, lg, z};
            }
        }
    }
    return best;
}

// Shared memory for the ring (no more stages than a share has), no less than the groups' sums take.
template <typename T>
size_t fma_smem(const FgFmaOp& o, uint32_t lg_split) {
    const FmaStage st = fma_stage<T>(o.ta != 0, o.tb != 0, o.factor != nullptr);
    const uint32_t nk = ((o.K + T::TK - 1) / T::TK + (1u << lg_split) - 1) >> lg_split;
    const size_t ring = (size_t)(nk < (uint32_t)T::S ? nk : T::S) * (st.a + st.b + st.f) * 4, sums = (size_t)T::G * T::TM * kTN * 4;
    return ring > sums ? ring : sums;
}
constexpr int kFmaSmemMax = 180 * 1024;

template <int N>
int32_t fma_launch(fg_ctx* ctx, void (*kernel)(FmaLaunch<N>), std::atomic<uint64_t>& smem_set, const FmaLaunch<N>& l, size_t smem) {
    if (!(smem_set.load(std::memory_order_acquire) >> (ctx->device & 63) & 1ull)) {
        FG_CUDA(ctx, FG_ERR_INTERNAL, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFmaSmemMax));
        smem_set.fetch_or(1ull << (ctx->device & 63), std::memory_order_release);
    }
    fg_launch_cluster(ctx, kernel, l.units << l.lg_split, kT, smem, 1u << l.lg_split, l);
    FG_LAUNCHED(ctx);
    return FG_OK;
}
template <typename F>
auto with_tile(int i, F f) { return i == 0 ? f(Tile4{}) : i == 1 ? f(Tile16{}) : i == 2 ? f(Tile32{}) : f(Tile64{}); }

}  // namespace

bool fg_ranges_meet(const void* p, uint64_t np, const void* q, uint64_t nq) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(q);
    return p && q && a < b + nq && b < a + np;
}

namespace {
template <int n>
int32_t launch_products(fg_ctx* ctx, const FgFmaOp* ops, uint32_t batch, bool in_order) {
    const FmaPlan plan = in_order ? FmaPlan{} : fma_plan(ctx, ops, n, batch);
    FmaLaunch<n> l{};
    l.lg_split = plan.lg_split;
    l.batch = batch;
    size_t smem = 0;
    uint64_t units = 0;
    float *part = nullptr, *below = nullptr;
    uint32_t part_rows = 0, part_cols = 0;
    for (int j = 0; j < n; ++j) {
        const FgFmaOp& o = ops[j];
        const uint32_t tm = in_order ? TileOrdered::TM : 1u << kTiles[plan.tile[j]].lg_tm, tiles_m = (o.M + tm - 1) / tm;
        FmaArgs& a = l.p[j];
        a.A = o.A; a.B = o.B; a.factor = o.factor; a.bias = o.bias; a.mul_saved = o.mul_saved;
        a.C = o.C; a.preact = o.preact; a.colsum_b = o.colsum_b; a.colsum_c = o.colsum_c;
        a.pairs = o.pairs; a.pairs_stride = o.pairs_stride; a.sA = o.sA; a.sB = o.sB; a.sC = o.sC;
        a.M = o.M; a.N = o.N; a.K = o.K; a.tiles_m = tiles_m;
        const uint64_t tiles = (uint64_t)tiles_m * ((o.N + kTN - 1) / kTN);
        if ((tiles * batch + units) << plan.lg_split > 0x7fffffffull) return fg_fail(ctx, FG_ERR_INVALID_ARGUMENT, "GEMM: too many tiles");
        a.tiles = (uint32_t)tiles;
        a.act = o.act; a.factor_act = o.factor_act; a.mul_act = o.mul_act;
        const FmaRows rows = fma_rows(o, batch);
        a.a16 = rows.a16;
        a.b16 = rows.b16;
        a.c16 = rows16(o.C, o.N, o.sC, batch) && (!o.preact || fg_aligned16(o.preact)) && (!o.mul_saved || fg_aligned16(o.mul_saved)) &&
                (!o.pairs || (fg_aligned16(o.pairs) && o.pairs_stride % 4 == 0));
        if (o.colsum_c && tiles_m > 1) {
            void* p;
            part_rows = (o.M + 31) / 32;
            const int32_t s = fg_ws_alloc(ctx, (uint64_t)part_rows * o.N * 4, &p);
            if (s != FG_OK) return s;
            a.colsum_c = part = (float*)p;
            below = o.colsum_c; part_cols = o.N;
        }
        auto room = [&](auto t) { return fma_smem<decltype(t)>(o, plan.lg_split); };
        const size_t bytes = in_order ? room(TileOrdered{}) : with_tile(plan.tile[j], room);
        if (bytes > smem) smem = bytes;
        units += tiles * batch;
        if (j == 0) l.units0 = (uint32_t)units;
    }
    l.units = (uint32_t)units;
    auto launch = [&](auto kernel_of) -> int32_t {
        static std::atomic<uint64_t> set{0};      // one per instance of this lambda, that is per kernel
        return fma_launch(ctx, kernel_of(), set, l, smem);
    };
    int32_t s;
    if constexpr (n == 1) {
        auto one = [&](auto t) {
            using T = decltype(t);
            if (ops[0].ta) return ops[0].tb ? launch([] { return gemm_fma_kernel<T, true, true>; }) : launch([] { return gemm_fma_kernel<T, true, false>; });
            return ops[0].tb ? launch([] { return gemm_fma_kernel<T, false, true>; }) : launch([] { return gemm_fma_kernel<T, false, false>; });
        };
        s = in_order ? launch([] { return gemm_fma_kernel<TileOrdered, false, false>; }) : with_tile(plan.tile[0], one);      // (in order: forward alone)
    } else {
        auto both = [&](auto tb, auto ta) { return launch([] { return gemm_fma_bwd_kernel<decltype(tb), decltype(ta)>; }); };
        s = in_order ? both(TileOrdered{}, TileOrdered{})
                     : with_tile(plan.tile[0], [&](auto t) { return with_tile(plan.tile[1], [&](auto u) { return both(t, u); }); });
    }
    if (s != FG_OK || !part) return s;
    return fg_colsum_fold_launch(ctx, part_cols, part_rows, part, below);
}
}  // namespace

int32_t fg_gemm_fma_launch(fg_ctx* ctx, const FgFmaOp* ops, int n, uint32_t batch, bool in_order) {
    if (batch == 0) return FG_OK;
    if (in_order && n == 1 && (ops[0].ta || ops[0].tb)) return fg_fail(ctx, FG_ERR_INTERNAL, "FMA kernel: one gradient in order is the exact path's");
    return n > 1 ? launch_products<2>(ctx, ops, batch, in_order) : launch_products<1>(ctx, ops, batch, in_order);
}

// Multiply-adds of a launch with its tiles' padding, and up to how many of them this kernel is the faster one.  66 products of 1 to 130
// million multiply-adds, this kernel and the tensor-core routes (us): forward 384 x 256 x 200 4.6 / 8.3, 256 x 448 x 320 5.2 / 7.4,
// 512 x 800 x 128 7.2 / 7.0, 448 x 1024 x 200 10.2 / 8.4; dB with its bias gradient 384 x 256 x 200 6.0 / 9.4, 128 x 656 x 536 7.6 / 7.3; both
// gradients 128 x 256 x 256 6.8 / 11.5, 128 x 640 x 208 10.3 / 12.0, 384 x 256 x 200 9.9 / 8.9; of dZ rows that are copied word by word
// 1000 x 63 x 150 12.2 / 18.7, 2000 x 100 x 30 17.7 / 18.9, 2800 x 101 x 30 22.8 / 20.8.
bool fg_gemm_fma_suits(uint32_t M, uint32_t N, uint32_t K, int products) {
    if (products != kFgForward && N <= 16) return false;                // the narrow layer's own kernels
    auto padded = [](uint64_t m, uint64_t n, uint64_t k) { return (m + 15) / 16 * 16 * ((n + kTN - 1) / kTN * kTN) * ((k + 31) / 32 * 32); };
    // (where the conversion kernel needs no copies and its tiles wait for their stores alone it is ahead sooner: 6000 x 128 x 32 5.9 us, 5.1 by that
    // kernel, 2500 x 256 x 48 7.5 / 5.5, 1000 x 400 x 96 6.3 / 5.9; 2500 x 128 x 32 4.4 / 5.1, 240 x 2368 x 24 4.9 / 5.9, 256 x 2000 x 64 5.4 / 5.5)
    const uint64_t most = K % 4 || N % 4 || K > 128 ? 45000000ull : K <= 32 ? 19000000ull : K <= 64 ? 36000000ull : 40000000ull;
    if (products == kFgForward) return N > 16 && padded(M, N, K) <= most;
    const uint64_t work = (products & kFgGradB ? padded(K, N, M) : 0) + (products & kFgGradA ? padded(M, K, N) : 0);
    return work <= (products != (kFgGradA | kFgGradB) ? 40000000ull : N % 4 ? 24000000ull : 32000000ull);
}

// A narrow layer's dB is one tile across and a tile per 64 rows of B: its clusters go through all samples, where the narrow layer's own
// kernels (gemm_skinny_tn_partial_kernel) spread them over the GPU, taking longer with more columns; rows off 16 bytes are copied word
// by word here.  Device times of 300 layers, this kernel and those (us): all gradients with the factor of the layer below 1024 x 1 x 1 6.7 /
// 10.2, 1500 x 10 x 100 13.4 / 16.3, 3072 x 10 x 40 15.1 / 17.8, 4096 x 16 x 16 14.5 / 22.4, 4096 x 1 x 1 16.9 / 13.7, 1024 x 4 x 300 13.9 / 13.3,
// 64 x 4 x 4000 7.5 / 10.1, 128 x 4 x 4000 11.4 / 10.9, 65536 x 4 x 4 285 / 64; the gradients alone 1500 x 1 x 64 8.8 / 9.1, 3072 x 4 x 40
// 10.5 / 11.2, 496 x 16 x 496 (dB) 5.2 / 9.1, 3072 x 1 x 40 12.6 / 10.4; with an activation's factor on dZ 256 x 4 x 500 7.6 / 11.1,
// 512 x 4 x 200 10.4 / 10.7, 536 x 12 x 336 9.6 / 12.9, 1024 x 10 x 64 10.0 / 12.2, 2048 x 16 x 64 13.3 / 14.5, 1500 x 1 x 40 12.9 / 10.2; dA alone 1024 x 4 x 2 2.9 / 2.3.
bool fg_gemm_fma_suits_small(uint32_t M, uint32_t N, uint32_t K, int products) {
    if (N > 16 || products == kFgForward) return true;
    const bool quads = N % 4 == 0, wide = quads && N >= 12;
    const uint64_t mk = (uint64_t)M * K;
    if (!(products & kFgGradB)) return products & (kFgFactor | kFgBelow | kFgBias) ? M <= 4096 : M < 64;
    if (products & kFgFactor) return M <= (wide ? 2048u : 1024u) && mk <= (M <= (wide ? 600u : 256u) ? 250000u : wide ? 140000u : 100000u);
    return M <= (wide ? 4096u : quads || (products & kFgBelow) ? 3072u : 2048u) && mk + 55ull * M <= (wide ? 380000u : 260000u);
}

namespace {
// What a backward pass cannot do in one launch: an output lies over dZ or its factor, or over any operand; dZ is formed first, as it is
// read after the first output is written, or for a bias gradient without dB.
struct FmaBwdOverlap { bool over_z, over_in, forms_z; };
FmaBwdOverlap bwd_overlap(const FgFmaBwd& b) {
    const uint64_t mn = (uint64_t)b.M * b.N * 4, mk = (uint64_t)b.M * b.K * 4, kn = (uint64_t)b.K * b.N * 4;
    const struct { const void* p; uint64_t n; } outs[5] = {{b.dA, mk}, {b.dB, kn}, {b.dbias, b.N * 4ull}, {b.below_dbias, b.K * 4ull},
                                                           {b.pairs, (b.pairs_stride + (uint64_t)b.M * b.K) * 2}};
    FmaBwdOverlap r{};
    for (const auto& o : outs) {
        r.over_z |= fg_ranges_meet(o.p, o.n, b.dZ, mn) || fg_ranges_meet(o.p, o.n, b.factor, mn);
        r.over_in |= fg_ranges_meet(o.p, o.n, b.A, mk) || fg_ranges_meet(o.p, o.n, b.B, kn);
    }
    r.forms_z = b.factor && (r.over_z || (b.dbias && !b.dB));
    return r;
}
}  // namespace

uint64_t fg_gemm_fma_bwd_scratch(const FgFmaBwd& b) {
    return (bwd_overlap(b).forms_z ? (uint64_t)b.M * b.N * 4 + 256 : 0) + (b.dbias && !b.dB ? (uint64_t)((b.M + 255) / 256) * b.N * 4 + 256 : 0);
}

// The backward pass of one layer, see FgFmaBwd.  The caller has reserved fg_gemm_fma_bwd_scratch() and room for column sums of dA.
int32_t fg_gemm_fma_bwd(fg_ctx* ctx, const FgFmaBwd& b) {
    const FmaBwdOverlap lies = bwd_overlap(b);
    const float *dz = b.dZ, *factor = b.factor;
    int32_t s;
    if (lies.forms_z) {
        void* p;
        if ((s = fg_ws_alloc(ctx, (uint64_t)b.M * b.N * 4, &p)) != FG_OK ||
            (s = fg_act_bwd_launch(ctx, (uint64_t)b.M * b.N, b.factor_act, dz, factor, (float*)p)) != FG_OK) return s;
        dz = (const float*)p;
        factor = nullptr;
    }
    if (b.dbias && !b.dB && (s = fg_colsum_launch(ctx, b.M, b.N, dz, b.dbias)) != FG_OK) return s;
    FgFmaOp ops[2] = {};
    FgFmaOp &w = ops[0], &x = ops[1];
    w.ta = 1; w.M = b.K; w.N = b.N; w.K = b.M; w.A = b.A; w.B = dz; w.C = b.dB; w.factor = factor; w.factor_act = b.factor_act;
    w.colsum_b = b.dbias;
    x.tb = 1; x.M = b.M; x.N = b.K; x.K = b.N; x.A = dz; x.B = b.B; x.C = b.dA; x.factor = factor; x.factor_act = b.factor_act;
    x.mul_saved = b.mul_saved; x.mul_act = b.mul_act; x.pairs = b.pairs; x.pairs_stride = b.pairs_stride; x.colsum_c = b.below_dbias;
    if (b.dB && b.dA && !b.exch_buf && !lies.over_z && !lies.over_in) return fg_gemm_fma_launch(ctx, ops, 2, 1, false);
    if (b.dB && (s = fg_gemm_fma_launch(ctx, &w, 1, 1, false)) != FG_OK) return s;
    if (b.exch_buf && (s = fg_allreduce_sum_f32(ctx, b.exch_buf, b.exch_count)) != FG_OK) return s;
    return b.dA ? fg_gemm_fma_launch(ctx, &x, 1, 1, false) : FG_OK;
}

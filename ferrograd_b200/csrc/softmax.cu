// Row softmax, its backward, and the fused softmax + cross-entropy forward/backward.
//
// Semantics: softmax forward crates/ferrograd-nn/src/op/softmax.rs:112-446 (row max,
// e = exp(x - max), sum, y = e * (1/sum)); backward :448-688 (dx = y * (dy - sum(dy*y)));
// CROSS_ENTROPY crates/ferrograd-nn/src/loss/basic_loss.rs:91-133 (loss = -log p at the
// label column, grad = p - onehot).  The reference runs three kernels with about five
// passes over the matrix; the fused kernel here reads the logits from HBM once and
// writes dlogits once.
//
// Two kernels serve the fused path:
//   * rowreg: one persistent 1024-thread CTA per SM.  The row being worked on lives
//     in registers (8 x float4 per thread, up to 32768 columns) while the NEXT row is
//     already streaming into shared memory with bulk async copies (cp.async.bulk,
//     completion on an mbarrier), so HBM reads never wait for the exp/reduce/store
//     phases.  HBM traffic: rows*cols*4 B read + rows*cols*4 B written.
//   * stream: any shape and alignment; one CTA per row, re-reads the row (L1/L2 hits
//     for the row sizes it is used for).
#include <math_constants.h>

#include <atomic>

#include "fg_internal.cuh"

namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// Block-wide reductions over up to 32 warps; `red` is 32 floats of shared memory.
// Every thread gets the result.  Two barriers per call.
__device__ __forceinline__ float block_max(float v, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_max(v);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float r = lane < nw ? red[lane] : -CUDART_INF_F;
    r = warp_max(r);
    __syncthreads();
    return r;
}
__device__ __forceinline__ float block_sum(float v, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float r = lane < nw ? red[lane] : 0.0f;
    r = warp_sum(r);
    __syncthreads();
    return r;
}

// (value, index) argmax, first maximum wins.
__device__ __forceinline__ void argmax_merge(float& v, uint32_t& i, float ov, uint32_t oi) {
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}
__device__ __forceinline__ uint32_t block_argmax(float v, uint32_t i, float* redv, uint32_t* redi) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float ov = __shfl_xor_sync(kFull, v, o);
        uint32_t oi = __shfl_xor_sync(kFull, i, o);
        argmax_merge(v, i, ov, oi);
    }
    if (lane == 0) { redv[warp] = v; redi[warp] = i; }
    __syncthreads();
    v = lane < nw ? redv[lane] : -CUDART_INF_F;
    i = lane < nw ? redi[lane] : 0xffffffffu;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float ov = __shfl_xor_sync(kFull, v, o);
        uint32_t oi = __shfl_xor_sync(kFull, i, o);
        argmax_merge(v, i, ov, oi);
    }
    __syncthreads();
    return i;
}

// ------------------------------------------------------------------------------------
// General kernel: one CTA per row (grid-stride over rows), three reads of the row.
// MODE 0: softmax forward (y).  MODE 1: fused CE.
// ------------------------------------------------------------------------------------
struct CeArgs {
    const float* x;
    const uint32_t* labels;
    uint32_t rows, cols;
    float scale;
    float* loss_row;
    float* dlogits;
    float* probs;
    uint32_t* argmax;
    float* y;   // MODE 0 output
    float* mean;               // the mean of loss_row, by the block that arrives last (NULL: a launch of its own adds)
    unsigned* arrivals;
};

// The mean of the rows' losses, in a fixed order, in thread 0 of a block (L2: they come from other blocks of the same launch).
template <bool L2>
__device__ __forceinline__ void mean_of_rows(const float* x, uint32_t n, float* out, float* red) {
    float s = 0.0f, v[8];
    for (uint64_t i0 = threadIdx.x; i0 < n; i0 += 8 * blockDim.x) {      // eight loads in flight, added in order
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = i0 + j * blockDim.x < n ? (L2 ? __ldcg(x + i0 + j * blockDim.x) : x[i0 + j * blockDim.x]) : 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) s += v[j];
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) *out = s / (float)n;
}
// At the end of a kernel whose blocks have left their rows' losses.
__device__ __forceinline__ void leave_mean(const CeArgs& a, float* red) {
    if (a.mean && fg_last_block(a.arrivals, gridDim.x)) mean_of_rows<true>(a.loss_row, a.rows, a.mean, red);
}

template <int MODE, bool VEC>
__global__ void softmax_stream_kernel(CeArgs a) {
    fg_grid_enter();
    __shared__ float red[32];
    __shared__ uint32_t redi[32];
    const uint32_t cols = a.cols;
    for (uint32_t row = blockIdx.x; row < a.rows; row += gridDim.x) {
        const float* xr = a.x + (size_t)row * cols;
        float mx = -CUDART_INF_F;
        uint32_t mi = 0xffffffffu;
        if (VEC) {
            const float4* x4 = reinterpret_cast<const float4*>(xr);
            for (uint32_t i = threadIdx.x; i < (cols >> 2); i += blockDim.x) {
                float4 v = x4[i];
                if (MODE == 1 && a.argmax) {
                    argmax_merge(mx, mi, v.x, 4 * i);
                    argmax_merge(mx, mi, v.y, 4 * i + 1);
                    argmax_merge(mx, mi, v.z, 4 * i + 2);
                    argmax_merge(mx, mi, v.w, 4 * i + 3);
                } else {
                    mx = fmaxf(fmaxf(mx, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
                }
            }
        } else {
            for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
                if (MODE == 1 && a.argmax) argmax_merge(mx, mi, xr[c], c);
                else mx = fmaxf(mx, xr[c]);
            }
        }
        if (MODE == 1 && a.argmax) {
            uint32_t am = block_argmax(mx, mi, red, redi);
            if (threadIdx.x == 0) a.argmax[row] = am;
        }
        mx = block_max(mx, red);
        float s = 0.0f;
        if (VEC) {
            const float4* x4 = reinterpret_cast<const float4*>(xr);
            for (uint32_t i = threadIdx.x; i < (cols >> 2); i += blockDim.x) {
                float4 v = x4[i];
                s += (expf(v.x - mx) + expf(v.y - mx)) + (expf(v.z - mx) + expf(v.w - mx));
            }
        } else {
            for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) s += expf(xr[c] - mx);
        }
        s = block_sum(s, red);
        const float inv = 1.0f / s;
        uint32_t lab = 0xffffffffu;
        if (MODE == 1) {
            lab = a.labels[row];
            if (threadIdx.x == 0 && a.loss_row)
                a.loss_row[row] = lab < cols ? (logf(s) + mx) - xr[lab] : 0.0f;
        }
        float* o0 = MODE == 0 ? a.y + (size_t)row * cols : (a.dlogits ? a.dlogits + (size_t)row * cols : nullptr);
        float* o1 = (MODE == 1 && a.probs) ? a.probs + (size_t)row * cols : nullptr;
        if (VEC) {
            const float4* x4 = reinterpret_cast<const float4*>(xr);
            for (uint32_t i = threadIdx.x; i < (cols >> 2); i += blockDim.x) {
                float4 v = x4[i];
                float4 p = make_float4(expf(v.x - mx) * inv, expf(v.y - mx) * inv, expf(v.z - mx) * inv,
                                       expf(v.w - mx) * inv);
                if (MODE == 0) {
                    reinterpret_cast<float4*>(o0)[i] = p;
                } else {
                    if (o1) reinterpret_cast<float4*>(o1)[i] = p;
                    if (o0) {
                        uint32_t c = 4 * i;
                        float4 g = make_float4((p.x - (c == lab ? 1.f : 0.f)) * a.scale,
                                               (p.y - (c + 1 == lab ? 1.f : 0.f)) * a.scale,
                                               (p.z - (c + 2 == lab ? 1.f : 0.f)) * a.scale,
                                               (p.w - (c + 3 == lab ? 1.f : 0.f)) * a.scale);
                        reinterpret_cast<float4*>(o0)[i] = g;
                    }
                }
            }
        } else {
            for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
                float p = expf(xr[c] - mx) * inv;
                if (MODE == 0) o0[c] = p;
                else {
                    if (o1) o1[c] = p;
                    if (o0) o0[c] = (p - (c == lab ? 1.f : 0.f)) * a.scale;
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------
// rowreg kernel: persistent, row in registers, next row prefetched into shared memory.
// Requires cols % 4 == 0, 16-byte aligned base, cols <= 32768.
// ------------------------------------------------------------------------------------
constexpr int kRowT = 1024;   // threads per CTA
constexpr int kRowNV = 8;     // float4 per thread
constexpr long long kWaitCycles = 2000000000LL;  // about one second

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    long long t0 = clock64();
    for (uint32_t it = 0;; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((it & 63u) == 63u && clock64() - t0 > kWaitCycles) return false;
    }
}

// Issue the bulk copies that bring one row (bytes, a multiple of 16) into shared memory.
__device__ __forceinline__ void prefetch_row(uint32_t dst, const float* src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
    constexpr uint32_t kChunk = 16384;
    for (uint32_t off = 0; off < bytes; off += kChunk) {
        uint32_t n = bytes - off < kChunk ? bytes - off : kChunk;
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
            :: "r"(dst + off), "l"(reinterpret_cast<const char*>(src) + off), "r"(n), "r"(bar) : "memory");
    }
}

// Four elements of the outputs: e * inv, and for the loss (p - onehot) * scale.  Only the float4 that holds the label (i ==
// lab / 4) is looked at element by element.
template <int MODE>
__device__ __forceinline__ void softmax_put4(const CeArgs& a, float4* o0, float4* o1, uint32_t i, uint32_t lab, float4 e, float inv, bool stream) {
    const float4 p = make_float4(e.x * inv, e.y * inv, e.z * inv, e.w * inv);
    auto put = [&](float4* o, float4 v) { if (stream) __stcs(o + i, v); else o[i] = v; };
    if (MODE == 0) {
        put(o0, p);
    } else {
        if (o1) put(o1, p);
        if (o0) {
            float4 g = p;
            if (i == lab >> 2) {
                const uint32_t t = lab & 3u;
                g.x -= t == 0 ? 1.f : 0.f; g.y -= t == 1 ? 1.f : 0.f; g.z -= t == 2 ? 1.f : 0.f; g.w -= t == 3 ? 1.f : 0.f;
            }
            put(o0, make_float4(g.x * a.scale, g.y * a.scale, g.z * a.scale, g.w * a.scale));
        }
    }
}
// The lowest index among a thread's four elements that equal the row's maximum (fmaxf and == both pass over NaN).
__device__ __forceinline__ void first_equal4(uint32_t& mi, float4 v, float mx, uint32_t c) {
    if (v.w == mx) mi = min(mi, c + 3);
    if (v.z == mx) mi = min(mi, c + 2);
    if (v.y == mx) mi = min(mi, c + 1);
    if (v.x == mx) mi = min(mi, c);
}

// All 32 warps meet at every barrier, so what counts is the instructions and barriers of a row: 8192 x 32000 with loss,
// gradient and predicted class 419 -> 387 us with four barriers instead of eight, the label looked for in one float4 and the
// class found by comparing with the maximum afterwards (5.4 TB/s).
template <int MODE>
__global__ void __launch_bounds__(kRowT, 1) softmax_rowreg_kernel(CeArgs a, int* dev_status) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* stage = reinterpret_cast<float*>(smem_raw);             // cols floats
    // one array per reduction, so that each costs one barrier: an array is written again only after two more barriers
    __shared__ float red_max[32], red_sum[32];
    __shared__ uint32_t s_arg;
    __shared__ __align__(8) unsigned long long bar_storage;
    const uint32_t bar = smem_u32(&bar_storage);
    const uint32_t cols = a.cols, ncol4 = cols >> 2, row_bytes = cols * 4u;
    const int tid = threadIdx.x;

    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    fg_grid_enter();
    uint32_t row = blockIdx.x;
    if (tid == 0 && row < a.rows) prefetch_row(smem_u32(stage), a.x + (size_t)row * cols, row_bytes, bar);
    uint32_t parity = 0;

    const int lane = tid & 31, warp = tid >> 5;
    for (; row < a.rows; row += gridDim.x) {
        // the label and its value are fetched long before they are used: the label while the row is on its way, the value during
        // the reductions (asked for at once, it made thread 0 wait for the label first: 2048 x 8192 64 -> 70 us)
        uint32_t lab = 0xffffffffu;
        float xlab = 0.0f;
        if (MODE == 1) lab = a.labels[row];
        // 1. wait for this row in shared memory, move it to registers
        bool ok = mbar_wait_bounded(bar, parity);
        parity ^= 1u;
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicOr(dev_status, FG_DEVERR_TMA_WAIT);
            // give the copies in flight a bounded chance to land before the CTA retires
            if (!ok) mbar_wait_bounded(bar, parity ^ 1u);
            // counted like the others, so that the counter wraps to zero; no mean is left here
            if (MODE == 1 && a.mean && tid == 0) atomicInc(a.arrivals, gridDim.x - 1);
            return;
        }
        float4 v[kRowNV];
        const float4* s4 = reinterpret_cast<const float4*>(stage);
#pragma unroll
        for (int j = 0; j < kRowNV; ++j) {
            uint32_t i = tid + j * kRowT;
            v[j] = i < ncol4 ? s4[i] : make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
        }
        if (MODE == 1 && tid == 0) s_arg = 0xffffffffu;
        __syncthreads();   // everyone has read the staging buffer
        if (MODE == 1 && tid == 0 && lab < cols) xlab = a.x[(size_t)row * cols + lab];
        // 2. start streaming the next row while this one is processed
        const uint32_t next = row + gridDim.x;
        if (tid == 0 && next < a.rows) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            prefetch_row(smem_u32(stage), a.x + (size_t)next * cols, row_bytes, bar);
        }
        // 3. max, then the first column that has it
        float mx = -CUDART_INF_F;
#pragma unroll
        for (int j = 0; j < kRowNV; ++j)
            mx = fmaxf(fmaxf(mx, fmaxf(v[j].x, v[j].y)), fmaxf(v[j].z, v[j].w));
        mx = warp_max(mx);
        if (lane == 0) red_max[warp] = mx;
        __syncthreads();
        mx = warp_max(red_max[lane]);
        if (MODE == 1 && a.argmax) {
            uint32_t mi = 0xffffffffu;
#pragma unroll
            for (int j = 0; j < kRowNV; ++j)
                if (tid + j * kRowT < ncol4) first_equal4(mi, v[j], mx, 4u * (tid + j * kRowT));
            if (mi != 0xffffffffu) atomicMin(&s_arg, mi);
        }
        // 4. e = exp(x - max), sum
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < kRowNV; ++j) {
            v[j].x = expf(v[j].x - mx);
            v[j].y = expf(v[j].y - mx);
            v[j].z = expf(v[j].z - mx);
            v[j].w = expf(v[j].w - mx);
            s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
        }
        s = warp_sum(s);
        if (lane == 0) red_sum[warp] = s;
        __syncthreads();
        s = warp_sum(red_sum[lane]);
        const float inv = 1.0f / s;
        if (MODE == 1 && tid == 0) {
            if (a.argmax) a.argmax[row] = s_arg;
            if (a.loss_row) a.loss_row[row] = lab < cols ? (logf(s) + mx) - xlab : 0.0f;
        }
        // 5. write
        float4* o0 = MODE == 0 ? reinterpret_cast<float4*>(a.y + (size_t)row * cols)
                               : (a.dlogits ? reinterpret_cast<float4*>(a.dlogits + (size_t)row * cols) : nullptr);
        float4* o1 = (MODE == 1 && a.probs) ? reinterpret_cast<float4*>(a.probs + (size_t)row * cols) : nullptr;
#pragma unroll
        for (int j = 0; j < kRowNV; ++j)
            if (tid + j * kRowT < ncol4) softmax_put4<MODE>(a, o0, o1, tid + j * kRowT, lab, v[j], inv, true);
    }
    if constexpr (MODE == 1) leave_mean(a, red_max);
}

// ------------------------------------------------------------------------------------
// Rows of 512 to 8192 columns (a multiple of four, 16-byte aligned): the row is read ONCE into registers
// (thread t holds the float4s t, t + 256, ...: NV of them), the exponentials are computed once, and the row
// is written once.  The general kernel above reads such a row three times (the second and third time from the
// L1/L2) and evaluates every exponential twice; with its few loads in flight per thread it reached 49 % of the
// DRAM rate on 16384 x 4096.  MODE as above.
// ------------------------------------------------------------------------------------
template <int MODE, int NV, bool MEAN = false>
__global__ void __launch_bounds__(256) softmax_held_kernel(CeArgs a) {
    fg_grid_enter();
    __shared__ float red[32];
    __shared__ uint32_t redi[32];
    const uint32_t cols = a.cols, n4 = cols >> 2;
    for (uint32_t row = blockIdx.x; row < a.rows; row += gridDim.x) {
        const float* xr = a.x + (size_t)row * cols;
        const float4* x4 = reinterpret_cast<const float4*>(xr);
        float4 v[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const uint32_t i = threadIdx.x + 256u * j;
            v[j] = i < n4 ? __ldcs(x4 + i) : make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
        }
        float mx = -CUDART_INF_F;
        uint32_t mi = 0xffffffffu;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const uint32_t i = threadIdx.x + 256u * j;
            if (MODE == 1 && a.argmax) {
                if (i < n4) {
                    argmax_merge(mx, mi, v[j].x, 4 * i);
                    argmax_merge(mx, mi, v[j].y, 4 * i + 1);
                    argmax_merge(mx, mi, v[j].z, 4 * i + 2);
                    argmax_merge(mx, mi, v[j].w, 4 * i + 3);
                }
            } else {
                mx = fmaxf(fmaxf(mx, fmaxf(v[j].x, v[j].y)), fmaxf(v[j].z, v[j].w));
            }
        }
        if (MODE == 1 && a.argmax) {
            uint32_t am = block_argmax(mx, mi, red, redi);
            if (threadIdx.x == 0) a.argmax[row] = am;
        }
        mx = block_max(mx, red);
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < NV; ++j) {       // padding is -inf: its exponential is zero
            v[j] = make_float4(expf(v[j].x - mx), expf(v[j].y - mx), expf(v[j].z - mx), expf(v[j].w - mx));
            s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
        }
        s = block_sum(s, red);
        const float inv = 1.0f / s;
        uint32_t lab = 0xffffffffu;
        if (MODE == 1) {
            lab = a.labels[row];
            if (threadIdx.x == 0 && a.loss_row)
                a.loss_row[row] = lab < cols ? (logf(s) + mx) - xr[lab] : 0.0f;
        }
        float* o0 = MODE == 0 ? a.y + (size_t)row * cols : (a.dlogits ? a.dlogits + (size_t)row * cols : nullptr);
        float* o1 = (MODE == 1 && a.probs) ? a.probs + (size_t)row * cols : nullptr;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const uint32_t i = threadIdx.x + 256u * j;
            if (i >= n4) continue;
            const float4 p = make_float4(v[j].x * inv, v[j].y * inv, v[j].z * inv, v[j].w * inv);
            if (MODE == 0) {
                reinterpret_cast<float4*>(o0)[i] = p;
            } else {
                if (o1) reinterpret_cast<float4*>(o1)[i] = p;
                if (o0) {
                    const uint32_t c = 4 * i;
                    reinterpret_cast<float4*>(o0)[i] = make_float4((p.x - (c == lab ? 1.f : 0.f)) * a.scale,
                                                                   (p.y - (c + 1 == lab ? 1.f : 0.f)) * a.scale,
                                                                   (p.z - (c + 2 == lab ? 1.f : 0.f)) * a.scale,
                                                                   (p.w - (c + 3 == lab ? 1.f : 0.f)) * a.scale);
                }
            }
        }
    }
    if constexpr (MEAN) leave_mean(a, red);
}

// The same for the backward pass: y and dy of a row are read once.
template <int NV>
__global__ void __launch_bounds__(256) softmax_bwd_held_kernel(uint32_t rows, uint32_t cols, const float* __restrict__ y,
                                                               const float* __restrict__ dy, float* __restrict__ dx,
                                                               int accumulate) {
    fg_grid_enter();
    __shared__ float red[32];
    const uint32_t n4 = cols >> 2;
    for (uint32_t row = blockIdx.x; row < rows; row += gridDim.x) {
        const float4* y4 = reinterpret_cast<const float4*>(y + (size_t)row * cols);
        const float4* d4 = reinterpret_cast<const float4*>(dy + (size_t)row * cols);
        float4* x4 = reinterpret_cast<float4*>(dx + (size_t)row * cols);
        float4 a[NV], b[NV];
        float dot = 0.0f;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const uint32_t i = threadIdx.x + 256u * j;
            a[j] = i < n4 ? __ldcs(y4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            b[j] = i < n4 ? __ldcs(d4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < NV; ++j) dot += (a[j].x * b[j].x + a[j].y * b[j].y) + (a[j].z * b[j].z + a[j].w * b[j].w);
        dot = block_sum(dot, red);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const uint32_t i = threadIdx.x + 256u * j;
            if (i >= n4) continue;
            float4 g = make_float4(a[j].x * (b[j].x - dot), a[j].y * (b[j].y - dot), a[j].z * (b[j].z - dot), a[j].w * (b[j].w - dot));
            if (accumulate) {
                const float4 o = x4[i];
                g.x += o.x; g.y += o.y; g.z += o.z; g.w += o.w;
            }
            x4[i] = g;
        }
    }
}

// ------------------------------------------------------------------------------------
// Rows that the kernels above cannot take: short ones, and rows whose starts are not 16-byte aligned (any odd number of
// columns).  The row is held in registers like above: one read, one exponential per element, one write.
//   * a warp per row, up to 511 columns, any alignment: no barrier anywhere, eight rows per block;
//   * a block per row, up to 32768 columns (backward: 16384), when all tensors lie alike modulo 16 bytes: 16-byte accesses
//     from the first boundary in the row on, the up to six words before and after them singly.  NV groups of four per
//     thread and a block no larger than that asks for, so that several rows are in flight on an SM.
// The values of a row's label are fetched before the reductions, so that their latency is hidden behind them.
// 4096 x 10001: forward 155 -> 58 us, backward 134 -> 81 us against three and two scalar passes; held as scalars, 32 words a
// thread, the backward pass took 148 us (one block per SM).
// ------------------------------------------------------------------------------------
// A thread's partial sums, added in pairs: a chain over them is longer than the one that a block of more threads would have
// (rows of 511: 6.7e-8 of the result's 2-norm from 64 bits with a chain of 16, 6.2e-8 with the tree).
template <int N> __device__ __forceinline__ float tree_sum(float (&t)[N]) {
    static_assert((N & (N - 1)) == 0, "pairs all the way");
#pragma unroll
    for (int w = N / 2; w > 0; w /= 2)
#pragma unroll
        for (int j = 0; j < w; ++j) t[j] += t[j + w];
    return t[0];
}

// What happens to one element of a row once the row's maximum and sum are known.
template <int MODE>
__device__ __forceinline__ void softmax_put(const CeArgs& a, size_t off, uint32_t c, uint32_t lab, float e, float inv) {
    const float p = e * inv;
    if (MODE == 0) {
        a.y[off] = p;
    } else {
        if (a.probs) a.probs[off] = p;
        if (a.dlogits) a.dlogits[off] = (p - (c == lab ? 1.f : 0.f)) * a.scale;
    }
}

template <int MODE, int NV, bool MEAN = false>
__global__ void __launch_bounds__(256) softmax_warp_kernel(CeArgs a) {
    fg_grid_enter();
    const uint32_t cols = a.cols, lane = threadIdx.x & 31u, step = gridDim.x * 8;
    for (uint32_t row = blockIdx.x * 8 + (threadIdx.x >> 5); row < a.rows; row += step) {
        const size_t base = (size_t)row * cols;
        float v[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) v[j] = lane + 32u * j < cols ? a.x[base + lane + 32u * j] : -CUDART_INF_F;
        uint32_t lab = 0xffffffffu;
        float xlab = 0.0f;
        if (MODE == 1) {
            lab = a.labels[row];
            if (lab < cols) xlab = a.x[base + lab];
        }
        float mx = -CUDART_INF_F;
        if (MODE == 1 && a.argmax) {
            uint32_t mi = 0xffffffffu;
#pragma unroll
            for (int j = 0; j < NV; ++j)
                if (lane + 32u * j < cols) argmax_merge(mx, mi, v[j], lane + 32u * j);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(kFull, mx, o);
                const uint32_t oi = __shfl_xor_sync(kFull, mi, o);
                argmax_merge(mx, mi, ov, oi);
            }
            if (lane == 0) a.argmax[row] = mi;
        } else {
#pragma unroll
            for (int j = 0; j < NV; ++j) mx = fmaxf(mx, v[j]);
        }
        mx = warp_max(mx);
        float t[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) { v[j] = expf(v[j] - mx); t[j] = lane + 32u * j < cols ? v[j] : 0.0f; }
        const float s = warp_sum(tree_sum(t));
        const float inv = 1.0f / s;
        if (MODE == 1 && lane == 0 && a.loss_row) a.loss_row[row] = lab < cols ? (logf(s) + mx) - xlab : 0.0f;
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (lane + 32u * j < cols) softmax_put<MODE>(a, base + lane + 32u * j, lane + 32u * j, lab, v[j], inv);
    }
    if constexpr (MEAN) {
        __shared__ float red[32];
        leave_mean(a, red);
    }
}

// Where the 16-byte accesses of a row start: `head` words before them, n4 groups of four, and `extra`, the index of the one
// word before or after them that this thread takes (threads 0..2 and 4..6; cols when it takes none).
struct RowEdges {
    uint32_t head, n4, extra;
};
__device__ __forceinline__ RowEdges row_edges(const float* row, uint32_t cols) {
    RowEdges e;
    e.head = ((16u - (uint32_t)(reinterpret_cast<uintptr_t>(row) & 15u)) & 15u) >> 2;      // the host calls this for cols >= 4
    e.n4 = (cols - e.head) >> 2;
    const uint32_t tail0 = e.head + 4 * e.n4, t = threadIdx.x;
    e.extra = t < e.head ? t : (t >= 4 && t - 4 < cols - tail0) ? tail0 + t - 4 : cols;
    return e;
}

template <int MODE, int NV, bool MEAN = false>
__global__ void __launch_bounds__(1024) softmax_edge_kernel(CeArgs a) {
    fg_grid_enter();
    // one array per reduction, so that each costs one barrier: an array is written again only after another barrier
    __shared__ float red_max[32], red_sum[32];
    __shared__ uint32_t s_arg;
    const uint32_t cols = a.cols, t = threadIdx.x, nt = blockDim.x, lane = t & 31u, warp = t >> 5, nw = nt >> 5;
    for (uint32_t row = blockIdx.x; row < a.rows; row += gridDim.x) {
        const size_t base = (size_t)row * cols;
        const RowEdges ed = row_edges(a.x + base, cols);
        const float4* x4 = reinterpret_cast<const float4*>(a.x + base + ed.head);
        float4 v[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j)
            v[j] = t + nt * j < ed.n4 ? __ldcs(x4 + t + nt * j) : make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
        float ve = ed.extra < cols ? a.x[base + ed.extra] : -CUDART_INF_F;
        uint32_t lab = 0xffffffffu;
        float xlab = 0.0f;
        if (MODE == 1) {
            lab = a.labels[row];
            if (t == 0 && lab < cols) xlab = a.x[base + lab];
            if (t == 0) s_arg = 0xffffffffu;
        }
        float mx = ve;
#pragma unroll
        for (int j = 0; j < NV; ++j) mx = fmaxf(fmaxf(mx, fmaxf(v[j].x, v[j].y)), fmaxf(v[j].z, v[j].w));
        mx = warp_max(mx);
        if (lane == 0) red_max[warp] = mx;
        __syncthreads();
        mx = warp_max(lane < nw ? red_max[lane] : -CUDART_INF_F);
        if (MODE == 1 && a.argmax) {
            uint32_t mi = 0xffffffffu;
#pragma unroll
            for (int j = 0; j < NV; ++j)
                if (t + nt * j < ed.n4) first_equal4(mi, v[j], mx, ed.head + 4 * (t + nt * j));
            if (ed.extra < cols && ve == mx) mi = min(mi, ed.extra);
            if (mi != 0xffffffffu) atomicMin(&s_arg, mi);
        }
        // what lies outside the row is -inf: its exponential is zero (or NaN, when the whole row is)
        ve = expf(ve - mx);
        float part[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            v[j] = make_float4(expf(v[j].x - mx), expf(v[j].y - mx), expf(v[j].z - mx), expf(v[j].w - mx));
            part[j] = (v[j].x + v[j].y) + (v[j].z + v[j].w);
        }
        float s = warp_sum(ve + tree_sum(part));
        if (lane == 0) red_sum[warp] = s;
        __syncthreads();
        s = warp_sum(lane < nw ? red_sum[lane] : 0.0f);
        const float inv = 1.0f / s;
        if (MODE == 1 && t == 0) {
            if (a.argmax) a.argmax[row] = s_arg;
            if (a.loss_row) a.loss_row[row] = lab < cols ? (logf(s) + mx) - xlab : 0.0f;
        }
        auto at4 = [&](float* p) { return p ? reinterpret_cast<float4*>(p + base + ed.head) : nullptr; };
        float4* const o0 = at4(MODE == 0 ? a.y : a.dlogits);
        float4* const o1 = MODE == 1 ? at4(a.probs) : nullptr;
        const uint32_t lab4 = lab >= ed.head ? lab - ed.head : 0xffffffffu;      // past the last group: matches none
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (t + nt * j < ed.n4) softmax_put4<MODE>(a, o0, o1, t + nt * j, lab4, v[j], inv, true);
        if (ed.extra < cols) softmax_put<MODE>(a, base + ed.extra, ed.extra, lab, ve, inv);
    }
    if constexpr (MEAN) leave_mean(a, red_sum);
}

template <int NV>
__global__ void __launch_bounds__(256) softmax_bwd_warp_kernel(uint32_t rows, uint32_t cols, const float* __restrict__ y,
                                                               const float* __restrict__ dy, float* __restrict__ dx, int accumulate) {
    fg_grid_enter();
    const uint32_t lane = threadIdx.x & 31u, step = gridDim.x * 8;
    for (uint32_t row = blockIdx.x * 8 + (threadIdx.x >> 5); row < rows; row += step) {
        const size_t base = (size_t)row * cols + lane;
        float a[NV], b[NV], old[NV], part[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const bool in = lane + 32u * j < cols;
            a[j] = in ? y[base + 32u * j] : 0.0f;
            b[j] = in ? dy[base + 32u * j] : 0.0f;
            old[j] = in && accumulate ? dx[base + 32u * j] : 0.0f;      // on its way during the reduction
        }
#pragma unroll
        for (int j = 0; j < NV; ++j) part[j] = a[j] * b[j];
        const float dot = warp_sum(tree_sum(part));
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (lane + 32u * j < cols) {
                const float g = a[j] * (b[j] - dot);
                dx[base + 32u * j] = accumulate ? old[j] + g : g;
            }
    }
}

// ACC adds to dx: what it adds to is fetched with the rest (fetched after the reduction, 2000 x 12000 took 103 us; 79 with the
// two-pass kernel; 62 so), which needs more threads of fewer groups each.  Without it eight groups per thread are faster:
// 4096 x 10001 80 us against 88.  ONCE is the evict-first hint, which rows of more than 8192 columns go without: y has often just been
// written, and a tensor that the L2 holds stays there (500 x 12000 again and again: 16.4 -> 12.3 us, 4096 x 16384 149 -> 121);
// shorter rows keep it (2000 x 6001 accumulating: 25 us, 33 without).
template <int NV, bool ACC, bool ONCE>
__global__ void __launch_bounds__(4096 / NV) softmax_bwd_edge_kernel(uint32_t rows, uint32_t cols, const float* __restrict__ y,
                                                                 const float* __restrict__ dy, float* __restrict__ dx) {
    fg_grid_enter();
    __shared__ float red[2][32];        // rows take turns, so that the reduction costs one barrier
    auto fetch = [](const float4* p) { return ONCE ? __ldcs(p) : *p; };
    const uint32_t t = threadIdx.x, nt = blockDim.x, lane = t & 31u, nw = nt >> 5;
    int turn = 0;
    for (uint32_t row = blockIdx.x; row < rows; row += gridDim.x, turn ^= 1) {
        const size_t base = (size_t)row * cols;
        const RowEdges ed = row_edges(y + base, cols);
        const float4* y4 = reinterpret_cast<const float4*>(y + base + ed.head);
        const float4* d4 = reinterpret_cast<const float4*>(dy + base + ed.head);
        float4* x4 = reinterpret_cast<float4*>(dx + base + ed.head);
        float4 a[NV], b[NV], old[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const bool in = t + nt * j < ed.n4;
            a[j] = in ? fetch(y4 + t + nt * j) : make_float4(0.f, 0.f, 0.f, 0.f);
            b[j] = in ? fetch(d4 + t + nt * j) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (ACC) old[j] = in ? x4[t + nt * j] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const float ae = ed.extra < cols ? y[base + ed.extra] : 0.0f, be = ed.extra < cols ? dy[base + ed.extra] : 0.0f;
        float part[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) part[j] = (a[j].x * b[j].x + a[j].y * b[j].y) + (a[j].z * b[j].z + a[j].w * b[j].w);
        float dot = warp_sum(ae * be + tree_sum(part));
        if (lane == 0) red[turn][t >> 5] = dot;
        __syncthreads();
        dot = warp_sum(lane < nw ? red[turn][lane] : 0.0f);
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (t + nt * j < ed.n4) {
                float4 g = make_float4(a[j].x * (b[j].x - dot), a[j].y * (b[j].y - dot), a[j].z * (b[j].z - dot), a[j].w * (b[j].w - dot));
                if (ACC) { g.x += old[j].x; g.y += old[j].y; g.z += old[j].z; g.w += old[j].w; }
                x4[t + nt * j] = g;
            }
        if (ed.extra < cols) {
            const float g = ae * (be - dot);
            dx[base + ed.extra] = ACC ? dx[base + ed.extra] + g : g;
        }
    }
}

// Softmax backward: dx (+)= y * (dy - dot), dot = sum_row(dy * y).
template <bool VEC>
__global__ void softmax_bwd_kernel(uint32_t rows, uint32_t cols, const float* __restrict__ y,
                                   const float* __restrict__ dy, float* __restrict__ dx, int accumulate) {
    fg_grid_enter();
    __shared__ float red[32];
    for (uint32_t row = blockIdx.x; row < rows; row += gridDim.x) {
        const float* yr = y + (size_t)row * cols;
        const float* dr = dy + (size_t)row * cols;
        float* xr = dx + (size_t)row * cols;
        float dot = 0.0f;
        if (VEC) {
            for (uint32_t i = threadIdx.x; i < (cols >> 2); i += blockDim.x) {
                float4 a = reinterpret_cast<const float4*>(yr)[i], b = reinterpret_cast<const float4*>(dr)[i];
                dot += (a.x * b.x + a.y * b.y) + (a.z * b.z + a.w * b.w);
            }
        } else {
            for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) dot += yr[c] * dr[c];
        }
        dot = block_sum(dot, red);
        if (VEC) {
            for (uint32_t i = threadIdx.x; i < (cols >> 2); i += blockDim.x) {
                float4 a = reinterpret_cast<const float4*>(yr)[i], b = reinterpret_cast<const float4*>(dr)[i];
                float4 g = make_float4(a.x * (b.x - dot), a.y * (b.y - dot), a.z * (b.z - dot), a.w * (b.w - dot));
                if (accumulate) {
                    float4 o = reinterpret_cast<float4*>(xr)[i];
                    g.x += o.x; g.y += o.y; g.z += o.z; g.w += o.w;
                }
                reinterpret_cast<float4*>(xr)[i] = g;
            }
        } else {
            for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
                float g = yr[c] * (dr[c] - dot);
                xr[c] = accumulate ? xr[c] + g : g;
            }
        }
    }
}

// The reference's unfused per-element CE on probabilities; with `partials`, also the sum of the losses, one part per block.
__global__ void __launch_bounds__(256) ce_elem_kernel(const float* __restrict__ p, const uint32_t* __restrict__ labels, uint32_t rows,
                               uint32_t cols, float* __restrict__ loss, float* __restrict__ grad, float* partials, unsigned* arrivals,
                               float* sum) {
    fg_grid_enter();
    __shared__ float red[32];
    float s = 0.0f;
    const uint64_t n = (uint64_t)rows * cols;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t r = (uint32_t)(i / cols), c = (uint32_t)(i - (uint64_t)r * cols);
        float pv = p[i];
        bool hit = labels[r] == c;
        const float l = hit ? -logf(pv) : 0.0f;
        loss[i] = l;
        grad[i] = hit ? pv - 1.0f : pv;
        s += l;
    }
    if (partials) fg_leave_sum(block_sum(s, red), partials, arrivals, sum, red);
}

// Fixed-order mean of the per-row losses (one CTA).
__global__ void mean_kernel(const float* __restrict__ x, uint32_t n, float* __restrict__ out) {
    fg_grid_enter();
    __shared__ float red[32];
    mean_of_rows<false>(x, n, out, red);
}

// Algorithmic HBM bytes of the fused CE kernel: logits in, dlogits (and probs) out.
double ce_bytes(const CeArgs& a) {
    double mat = 4.0 * a.rows * a.cols;
    return mat * (1.0 + (a.dlogits ? 1.0 : 0.0) + (a.probs ? 1.0 : 0.0)) + 8.0 * a.rows;
}

// Threads of a block that holds a row of `cols` words at `nv` words per thread.
int held_threads(uint32_t cols, int nv) { return (int)(((cols + nv - 1) / nv + 31) / 32 * 32); }
// ... and of the kernels that stream a row several times, for what none of those take: rows whose tensors lie differently
// modulo 16 bytes, and longer ones.  Rows that the SMs hold at once at 1024 threads each get them (64 x 4096: 10 us, 16 with
// 256); of many rows a short one is done by fewer threads (50000 x 600 forward: 111 us with 128, 289 with 1024; 10000 x 3000:
// 109 with 256, 137; 3750 x 8000 backward: 145 with 256, 107).
int stream_threads(const fg_ctx* ctx, uint32_t rows, uint32_t cols) {
    if (rows <= 2u * (uint32_t)ctx->sm_count || cols > 4096) return 1024;
    return cols <= 2048 ? 128 : 256;
}
constexpr uint32_t kWarpRowCols = 511, kEdgeRowCols = 32768, kEdgeRowColsBwd = 16384;
inline bool lie_alike(const void* a, const void* b) {
    return !b || ((reinterpret_cast<uintptr_t>(a) ^ reinterpret_cast<uintptr_t>(b)) & 15u) == 0;
}
// Grid of the kernels above: what the SMs hold at once, at most one block per row (or per eight rows).
int rows_grid(const fg_ctx* ctx, uint64_t blocks, int threads) {
    const int fit = 2048 / threads;
    const uint64_t cap = (uint64_t)ctx->sm_count * (uint64_t)(fit > 32 ? 32 : fit);
    return (int)(blocks < cap ? blocks : cap);
}

// Called by the kernels that can add the mean themselves: do they (see fg_fold_in_launch)?  Otherwise a.mean stays for the caller.
// With that, and launches that start while the kernel before them ends, back to back (before that, plain launches): the loss of 712 x 768 takes
// 4.5 us (6.8), 2384 x 64 4.5 (6.1), 300 x 1001 4.6 (6.8), 600 x 32000 36.1 (37.4), 8192 x 32000 391 (391); softmax
// and its gradient on 1728 x 1285 9.6 (12.5), 4096 x 10001 132.6 (137.1).
template <int MODE>
CeArgs with_mean(fg_ctx* ctx, CeArgs& a, int grid) {
    CeArgs k = a;
    if (MODE == 1 && a.mean && fg_fold_in_launch(ctx, (uint64_t)grid)) {
        k.arrivals = fg_arrivals(ctx);
        a.mean = nullptr;
    } else k.mean = nullptr;
    return k;
}

template <int MODE>
int32_t launch_rows(fg_ctx* ctx, CeArgs& a) {
    const bool vec = (a.cols % 4 == 0) && fg_aligned16(a.x) &&
                     (MODE == 0 ? fg_aligned16(a.y)
                                : ((!a.dlogits || fg_aligned16(a.dlogits)) && (!a.probs || fg_aligned16(a.probs))));
    const size_t smem = (size_t)a.cols * 4;
    if (vec && a.cols >= 8192 && a.cols <= (uint32_t)(kRowT * kRowNV * 4) && smem <= 200 * 1024) {
        static std::atomic<uint64_t> attr_done{0};   // one bit per device (static per MODE instantiation)
        if (!(attr_done.load(std::memory_order_acquire) >> (ctx->device & 63) & 1ull)) {
            FG_CUDA(ctx, FG_ERR_INTERNAL,
                    cudaFuncSetAttribute(softmax_rowreg_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
            attr_done.fetch_or(1ull << (ctx->device & 63), std::memory_order_release);
        }
        int grid = (int)(a.rows < (uint32_t)ctx->sm_count ? a.rows : (uint32_t)ctx->sm_count);
        fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SOFTMAX_CE, MODE == 1 ? ce_bytes(a) : 8.0 * a.rows * a.cols);
        const CeArgs k = with_mean<MODE>(ctx, a, grid);
        fg_launch(ctx, softmax_rowreg_kernel<MODE>, grid, kRowT, smem, k, ctx->dev_status);
        fg_time_end(ctx, tr);
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
    if (vec && a.cols >= 512 && a.cols <= 8192) {
        const uint64_t cap = (uint64_t)ctx->sm_count * 8;
        const int grid = (int)(a.rows < cap ? a.rows : cap);
        const uint32_t nv = (a.cols / 4 + 255) / 256;      // float4s per thread: 1 .. 8
        fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SOFTMAX_CE, MODE == 1 ? ce_bytes(a) : 8.0 * a.rows * a.cols);
        const CeArgs k = with_mean<MODE>(ctx, a, grid);
        if (nv <= 1) fg_launch(ctx, k.mean ? softmax_held_kernel<MODE, 1, MODE == 1> : softmax_held_kernel<MODE, 1>, grid, 256, 0, k);
        else if (nv <= 2) fg_launch(ctx, k.mean ? softmax_held_kernel<MODE, 2, MODE == 1> : softmax_held_kernel<MODE, 2>, grid, 256, 0, k);
        else if (nv <= 4) fg_launch(ctx, k.mean ? softmax_held_kernel<MODE, 4, MODE == 1> : softmax_held_kernel<MODE, 4>, grid, 256, 0, k);
        else fg_launch(ctx, k.mean ? softmax_held_kernel<MODE, 8, MODE == 1> : softmax_held_kernel<MODE, 8>, grid, 256, 0, k);
        fg_time_end(ctx, tr);
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
    if (a.cols <= kWarpRowCols) {
        const int grid = rows_grid(ctx, ((uint64_t)a.rows + 7) / 8, 256);
        fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SOFTMAX_CE, MODE == 1 ? ce_bytes(a) : 8.0 * a.rows * a.cols);
        const CeArgs k = with_mean<MODE>(ctx, a, grid);
        if (a.cols <= 32) fg_launch(ctx, k.mean ? softmax_warp_kernel<MODE, 1, MODE == 1> : softmax_warp_kernel<MODE, 1>, grid, 256, 0, k);
        else if (a.cols <= 128) fg_launch(ctx, k.mean ? softmax_warp_kernel<MODE, 4, MODE == 1> : softmax_warp_kernel<MODE, 4>, grid, 256, 0, k);
        else fg_launch(ctx, k.mean ? softmax_warp_kernel<MODE, 16, MODE == 1> : softmax_warp_kernel<MODE, 16>, grid, 256, 0, k);
        fg_time_end(ctx, tr);
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
    const bool alike = MODE == 0 ? lie_alike(a.x, a.y) : lie_alike(a.x, a.dlogits) && lie_alike(a.x, a.probs);
    if (a.cols <= kEdgeRowCols && alike) {
        const int threads = held_threads(a.cols, 32);
        const int grid = rows_grid(ctx, a.rows, threads);
        fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SOFTMAX_CE, MODE == 1 ? ce_bytes(a) : 8.0 * a.rows * a.cols);
        const CeArgs k = with_mean<MODE>(ctx, a, grid);
        // (rows of up to 16384 columns take 1 to 3 % less with the instance that can add the mean, whether it does or not: 4096 x 1001 7.2 us and 7.5,
        // 4096 x 10001 55.9 and 56.5; 8192 x 20001 312 and 303)
        fg_launch(ctx, k.mean || a.cols <= 16384 ? softmax_edge_kernel<MODE, 8, MODE == 1> : softmax_edge_kernel<MODE, 8>, grid, threads, 0, k);
        fg_time_end(ctx, tr);
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
    const int threads = stream_threads(ctx, a.rows, a.cols);
    const int grid = rows_grid(ctx, a.rows, threads);
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SOFTMAX_CE, MODE == 1 ? ce_bytes(a) : 8.0 * a.rows * a.cols);
    CeArgs k = a;
    k.mean = nullptr;
    if (vec) fg_launch(ctx, softmax_stream_kernel<MODE, true>, grid, threads, 0, k);
    else fg_launch(ctx, softmax_stream_kernel<MODE, false>, grid, threads, 0, k);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

}  // namespace

static int32_t ce_elem_launch(fg_ctx* ctx, const float* probs, const uint32_t* labels, uint32_t rows, uint32_t cols, float* loss_out,
                              float* grad_out, float* loss_sum_out) {
    const int grid = fg_stream_grid(ctx, (uint64_t)rows * cols, 256, 8);
    FgBlockSums b;
    const int32_t s = fg_block_sums(ctx, grid, loss_sum_out, &b);
    if (s != FG_OK) return s;
    fg_launch(ctx, ce_elem_kernel, grid, 256, 0, probs, labels, rows, cols, loss_out, grad_out, b.partials, fg_arrivals(ctx), b.out);
    FG_LAUNCHED(ctx);
    return fg_block_sums_end(ctx, b);
}

extern "C" {

int32_t fg_softmax_fwd(fg_ctx* ctx, uint32_t rows, uint32_t cols, const float* x, float* y) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, x && y, "fg_softmax_fwd: NULL pointer");
    FG_REQUIRE(ctx, cols >= 1, "fg_softmax_fwd: cols must be >= 1");
    FG_REQUIRE(ctx, (uint64_t)rows * cols < (1ull << 40), "fg_softmax_fwd: tensor too large");
    if (rows == 0) return FG_OK;
    CeArgs a{};
    a.x = x; a.rows = rows; a.cols = cols; a.y = y;
    return launch_rows<0>(ctx, a);
}

int32_t fg_softmax_bwd(fg_ctx* ctx, uint32_t rows, uint32_t cols, const float* y, const float* dy, float* dx,
                       int32_t accumulate) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, y && dy && dx, "fg_softmax_bwd: NULL pointer");
    FG_REQUIRE(ctx, cols >= 1, "fg_softmax_bwd: cols must be >= 1");
    if (rows == 0) return FG_OK;
    const bool vec = (cols % 4 == 0) && fg_aligned16(y) && fg_aligned16(dy) && fg_aligned16(dx);
    if (vec && cols >= 512 && cols <= 8192) {
        const uint64_t cap8 = (uint64_t)ctx->sm_count * 8;
        const int grid8 = (int)(rows < cap8 ? rows : cap8);
        const uint32_t nv = (cols / 4 + 255) / 256;
        fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SOFTMAX_CE, (accumulate ? 16.0 : 12.0) * rows * cols);
        if (nv <= 1) fg_launch(ctx, softmax_bwd_held_kernel<1>, grid8, 256, 0, rows, cols, y, dy, dx, accumulate);
        else if (nv <= 2) fg_launch(ctx, softmax_bwd_held_kernel<2>, grid8, 256, 0, rows, cols, y, dy, dx, accumulate);
        else if (nv <= 4) fg_launch(ctx, softmax_bwd_held_kernel<4>, grid8, 256, 0, rows, cols, y, dy, dx, accumulate);
        else fg_launch(ctx, softmax_bwd_held_kernel<8>, grid8, 256, 0, rows, cols, y, dy, dx, accumulate);
        fg_time_end(ctx, tr);
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_SOFTMAX_CE, (accumulate ? 16.0 : 12.0) * rows * cols);
    if (cols <= kWarpRowCols) {
        const int grid = rows_grid(ctx, ((uint64_t)rows + 7) / 8, 256);
        if (cols <= 32) fg_launch(ctx, softmax_bwd_warp_kernel<1>, grid, 256, 0, rows, cols, y, dy, dx, accumulate);
        else if (cols <= 128) fg_launch(ctx, softmax_bwd_warp_kernel<4>, grid, 256, 0, rows, cols, y, dy, dx, accumulate);
        else fg_launch(ctx, softmax_bwd_warp_kernel<16>, grid, 256, 0, rows, cols, y, dy, dx, accumulate);
        fg_time_end(ctx, tr);
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
    if (cols <= kEdgeRowColsBwd && lie_alike(y, dy) && lie_alike(y, dx)) {
        const int threads = held_threads(cols, accumulate ? 16 : 32), grid = rows_grid(ctx, rows, threads);
        if (accumulate) {
            if (cols > 8192) fg_launch(ctx, softmax_bwd_edge_kernel<4, true, false>, grid, threads, 0, rows, cols, y, dy, dx);
            else fg_launch(ctx, softmax_bwd_edge_kernel<4, true, true>, grid, threads, 0, rows, cols, y, dy, dx);
        } else {
            if (cols > 8192) fg_launch(ctx, softmax_bwd_edge_kernel<8, false, false>, grid, threads, 0, rows, cols, y, dy, dx);
            else fg_launch(ctx, softmax_bwd_edge_kernel<8, false, true>, grid, threads, 0, rows, cols, y, dy, dx);
        }
        fg_time_end(ctx, tr);
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
    const int threads = stream_threads(ctx, rows, cols);
    const int grid = rows_grid(ctx, rows, threads);
    if (vec) fg_launch(ctx, softmax_bwd_kernel<true>, grid, threads, 0, rows, cols, y, dy, dx, accumulate);
    else fg_launch(ctx, softmax_bwd_kernel<false>, grid, threads, 0, rows, cols, y, dy, dx, accumulate);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

int32_t fg_softmax_ce_fwd_bwd(fg_ctx* ctx, const float* logits, const uint32_t* labels, uint32_t rows,
                              uint32_t cols, float grad_scale, float* loss_row_out, float* loss_mean_out,
                              float* dlogits_out, float* probs_out, uint32_t* argmax_out) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, logits && labels, "fg_softmax_ce_fwd_bwd: logits and labels are required");
    FG_REQUIRE(ctx, cols >= 1, "fg_softmax_ce_fwd_bwd: cols must be >= 1");
    FG_REQUIRE(ctx, !(loss_mean_out && !loss_row_out),
               "fg_softmax_ce_fwd_bwd: loss_mean_out needs loss_row_out (the mean is reduced from it)");
    if (rows == 0) return FG_OK;
    CeArgs a{};
    a.x = logits; a.labels = labels; a.rows = rows; a.cols = cols; a.scale = grad_scale;
    a.loss_row = loss_row_out; a.dlogits = dlogits_out; a.probs = probs_out; a.argmax = argmax_out;
    a.mean = loss_mean_out;
    int32_t s = launch_rows<1>(ctx, a);
    if (s != FG_OK) return s;
    if (a.mean) {
        fg_launch(ctx, mean_kernel, 1, 1024, 0, loss_row_out, rows, loss_mean_out);
        FG_LAUNCHED(ctx);
    }
    return FG_OK;
}

int32_t fg_ce_loss_grad(fg_ctx* ctx, const float* probs, const uint32_t* labels, uint32_t rows, uint32_t cols,
                        float* loss_out, float* grad_out) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, probs && labels && loss_out && grad_out, "fg_ce_loss_grad: NULL pointer");
    FG_REQUIRE(ctx, cols >= 1, "fg_ce_loss_grad: cols must be >= 1");
    if (rows == 0) return FG_OK;
    return ce_elem_launch(ctx, probs, labels, rows, cols, loss_out, grad_out, nullptr);
}

}  // extern "C"

int32_t fg_ce_loss_grad_sum(fg_ctx* ctx, const float* probs, const uint32_t* labels, uint32_t rows, uint32_t cols, float* loss_out,
                            float* grad_out, float* loss_sum_out) {
    FG_ENTER(ctx);
    if (rows == 0) return fg_sum_f32(ctx, loss_out, 0, loss_sum_out);
    return ce_elem_launch(ctx, probs, labels, rows, cols, loss_out, grad_out, loss_sum_out);
}

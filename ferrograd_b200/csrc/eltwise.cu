// Elementwise work: bias + activation, activation backward, MSE loss + gradient, column
// sums (bias gradient) and fused elementwise chains (one forward kernel, one backward
// kernel per chain).
//
// Semantics follow crates/ferrograd-nn/src/op/unary.rs (tanh :270-327, relu :436-490,
// gelu :492-733, elu :328-436, exp :741-756), crates/ferrograd-nn/src/op/binary.rs
// (add :74, mul :236, sub :449, div :644 and their backward forms) and
// MEAN_SQUARED_ERROR (crates/ferrograd-nn/src/loss/basic_loss.rs:3-27).  The reference
// inlines elementwise producers into their consumer kernel
// (crates/fused_gpu/src/dispatch/backend/kernel/forward.rs:298-464); a chain here is the
// same idea with the program interpreted per element: every input is read once, every
// output written once.
#include <atomic>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "fg_internal.cuh"

namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// The streaming kernels below move four consecutive floats per thread and access (128-bit loads and stores) when
// every pointer they are given is 16-byte aligned (VEC), one float otherwise; the last n % 4 elements always go
// singly.  `nv` is the number of whole groups of four.
__device__ __forceinline__ float4 ld4(const float* p, uint64_t i4) { return reinterpret_cast<const float4*>(p)[i4]; }
__device__ __forceinline__ void st4(float* p, uint64_t i4, float4 v) { reinterpret_cast<float4*>(p)[i4] = v; }
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// y = act(z + bias[col]); with VEC, cols is a multiple of four, so a group of four never straddles a row.
template <bool VEC>
__global__ void __launch_bounds__(256) bias_act_kernel(uint32_t rows, uint32_t cols, const float* __restrict__ z,
                                                       const float* __restrict__ bias, int act, float* __restrict__ y) {
    const uint64_t n = (uint64_t)rows * cols, stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nv = VEC ? n >> 2 : 0;
    const uint32_t cols4 = cols >> 2;
    if constexpr (VEC) for (uint64_t i = g; i < nv; i += stride) {
        float4 p = ld4(z, i);
        if (bias) {
            const float4 b = ld4(bias, i % cols4);
            p.x += b.x; p.y += b.y; p.z += b.z; p.w += b.w;
        }
        st4(y, i, make_float4(fg_act_fwd(act, p.x), fg_act_fwd(act, p.y), fg_act_fwd(act, p.z), fg_act_fwd(act, p.w)));
    }
    for (uint64_t i = (nv << 2) + g; i < n; i += stride) {
        float p = z[i];
        if (bias) p += bias[i % cols];
        y[i] = fg_act_fwd(act, p);
    }
}

template <bool VEC>
__global__ void __launch_bounds__(256) act_bwd_kernel(uint64_t n, int act, const float* __restrict__ dy,
                                                      const float* __restrict__ saved, float* __restrict__ dz) {
    fg_grid_enter();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nv = VEC ? n >> 2 : 0;
    if constexpr (VEC) for (uint64_t i = g; i < nv; i += stride) {
        float4 d = ld4(dy, i);
        if (act != FG_ACT_NONE) {
            const float4 s = ld4(saved, i);
            d.x *= fg_act_grad(act, s.x); d.y *= fg_act_grad(act, s.y);
            d.z *= fg_act_grad(act, s.z); d.w *= fg_act_grad(act, s.w);
        }
        st4(dz, i, d);
    }
    for (uint64_t i = (nv << 2) + g; i < n; i += stride)
        dz[i] = act == FG_ACT_NONE ? dy[i] : dy[i] * fg_act_grad(act, saved[i]);
}

struct MseTerm {   // loss = d*d, grad = 2*d*scale
    static __device__ __forceinline__ float loss(float p, float t) { const float d = p - t; return d * d; }
    static __device__ __forceinline__ float grad(float p, float t, float scale) { return (2.0f * (p - t)) * scale; }
};
struct BceTerm {   // on probabilities: loss = -(t*log(p) + (1-t)*log(1-p)), grad = (p - t)*scale
    static __device__ __forceinline__ float loss(float p, float t) { return -(t * logf(p) + (1.0f - t) * logf(1.0f - p)); }
    static __device__ __forceinline__ float grad(float p, float t, float scale) { return (p - t) * scale; }
};

// Per-element loss and gradient of MSE or BCE; with `partials`, the sum of the losses, one part per block (see fg_leave_sum).
template <class TERM, bool VEC>
__global__ void __launch_bounds__(256) loss_kernel(const float* __restrict__ pred, const float* __restrict__ target,
                                                   uint64_t n, float scale, float* __restrict__ loss_elem,
                                                   float* __restrict__ grad, float* partials, unsigned* arrivals, float* sum) {
    fg_grid_enter();
    __shared__ float red[8];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nv = VEC ? n >> 2 : 0;
    float s = 0.0f;
    if constexpr (VEC) for (uint64_t i = g; i < nv; i += stride) {
        const float4 p = ld4(pred, i), t = ld4(target, i);
        const float4 l = make_float4(TERM::loss(p.x, t.x), TERM::loss(p.y, t.y), TERM::loss(p.z, t.z), TERM::loss(p.w, t.w));
        if (loss_elem) st4(loss_elem, i, l);
        if (grad)
            st4(grad, i, make_float4(TERM::grad(p.x, t.x, scale), TERM::grad(p.y, t.y, scale), TERM::grad(p.z, t.z, scale),
                                     TERM::grad(p.w, t.w, scale)));
        s += (l.x + l.y) + (l.z + l.w);
    }
    for (uint64_t i = (nv << 2) + g; i < n; i += stride) {
        const float p = pred[i], t = target[i], l = TERM::loss(p, t);
        if (loss_elem) loss_elem[i] = l;
        if (grad) grad[i] = TERM::grad(p, t, scale);
        s += l;
    }
    if (partials) {
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
        __syncthreads();
        float t = 0.0f;
        if (threadIdx.x == 0)
            for (int w = 0; w < 8; ++w) t += red[w];
        fg_leave_sum(t, partials, arrivals, sum, red);
    }
}

// Sum of n values: one part per block (grid-stride over float4, fixed order inside a block), then the parts.
__global__ void __launch_bounds__(256) sum_kernel(const float* __restrict__ x, uint64_t n, float* partials, unsigned* arrivals, float* out) {
    fg_grid_enter();
    __shared__ float red[8];
    float s = 0.0f;
    const uint64_t nv = ((reinterpret_cast<uintptr_t>(x) & 15u) == 0) ? n >> 2 : 0, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += stride) {
        const float4 v = __ldcs(reinterpret_cast<const float4*>(x) + i);
        s += (v.x + v.y) + (v.z + v.w);
    }
    for (uint64_t i = (nv << 2) + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) s += x[i];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    float t = 0.0f;
    if (threadIdx.x == 0)
        for (int w = 0; w < 8; ++w) t += red[w];
    fg_leave_sum(t, partials, arrivals, out, red);
}

// The partial sums that a launch left, in the order of its last block.
__global__ void __launch_bounds__(256) fold_partials_kernel(const float* partials, uint32_t n, float* __restrict__ out) {
    fg_grid_enter();
    __shared__ float red[8];
    const float s = fg_sum_partials(partials, n, red);
    if (threadIdx.x == 0) *out = s;
}

// ---- storage types ----
// Elements of a type as f32, for conversions (to the nearest, ties to even).  ld4w / st4w move four consecutive elements starting
// at element i (one 128-bit access for f32, one 64-bit access for the 16-bit types; the caller has checked the alignment).
template <int DT> struct Stored;
template <> struct Stored<FG_DTYPE_F32> {
    static __device__ __forceinline__ float ld(const void* p, uint64_t i) { return static_cast<const float*>(p)[i]; }
    static __device__ __forceinline__ void st(void* p, uint64_t i, float v) { static_cast<float*>(p)[i] = v; }
    static __device__ __forceinline__ void ld4w(const void* p, uint64_t i, float* o) {
        const float4 v = *reinterpret_cast<const float4*>(static_cast<const float*>(p) + i);
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    }
    static __device__ __forceinline__ void st4w(void* p, uint64_t i, const float* v) {
        *reinterpret_cast<float4*>(static_cast<float*>(p) + i) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <> struct Stored<FG_DTYPE_F16> {
    static __device__ __forceinline__ float ld(const void* p, uint64_t i) { return __half2float(static_cast<const __half*>(p)[i]); }
    static __device__ __forceinline__ void st(void* p, uint64_t i, float v) { static_cast<__half*>(p)[i] = __float2half_rn(v); }
    static __device__ __forceinline__ void ld4w(const void* p, uint64_t i, float* o) {
        const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const __half*>(p) + i);
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
    }
    static __device__ __forceinline__ void st4w(void* p, uint64_t i, const float* v) {
        const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
        uint2 u;
        u.x = *reinterpret_cast<const uint32_t*>(&a); u.y = *reinterpret_cast<const uint32_t*>(&b);
        *reinterpret_cast<uint2*>(static_cast<__half*>(p) + i) = u;
    }
};
template <> struct Stored<FG_DTYPE_BF16> {
    static __device__ __forceinline__ float ld(const void* p, uint64_t i) { return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]); }
    static __device__ __forceinline__ void st(void* p, uint64_t i, float v) { static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v); }
    static __device__ __forceinline__ void ld4w(const void* p, uint64_t i, float* o) {
        const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p) + i);
        o[0] = __uint_as_float(u.x << 16); o[1] = __uint_as_float(u.x & 0xffff0000u);
        o[2] = __uint_as_float(u.y << 16); o[3] = __uint_as_float(u.y & 0xffff0000u);
    }
    static __device__ __forceinline__ void st4w(void* p, uint64_t i, const float* v) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
        uint2 u;
        u.x = *reinterpret_cast<const uint32_t*>(&a); u.y = *reinterpret_cast<const uint32_t*>(&b);
        *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p) + i) = u;
    }
};

// out[c] = sum over chunks of part[k][c], for 32 columns and 256 threads.  The eight warps each add every eighth chunk into eight
// sums in turn, which are added in pairs, then the warps' sums in order: 64 short chains of additions (50000 rows in 1563
// chunks: 3.0e-7 of the sums' 2-norm from 64 bits with eight long ones, 1.3e-7 so).  `out` is of storage type DT.
template <int DT>
__device__ __forceinline__ void fold_chunks_of_columns(uint32_t c, uint32_t gy, uint32_t cx, uint32_t cols, uint32_t nchunks, const float* part,
                                                       void* __restrict__ out, float (*red)[33]) {
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (c < cols)
        for (uint64_t k = gy; k < nchunks; k += 64) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (k + 8 * j < nchunks) s[j] += __ldcg(part + (size_t)(k + 8 * j) * cols + c);
        }
    red[gy][cx] = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
    __syncthreads();
    if (gy == 0 && c < cols) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += red[w][cx];
        Stored<DT>::st(out, c, t);
    }
}

// Column sums: block (32 x 8) covers 32 columns and `chunk` rows and leaves their sums in part[blockIdx.y]; with FOLD, the last
// block of those columns adds the chunks.
template <bool FOLD>
__global__ void __launch_bounds__(256) colsum_kernel(uint32_t rows, uint32_t cols, uint32_t chunk, const float* __restrict__ x, float* part,
                                                     unsigned* arrivals, float* __restrict__ out) {
    fg_grid_enter();
    __shared__ float red[8][33];
    const uint32_t c = blockIdx.x * 32 + threadIdx.x;
    const uint32_t r0 = blockIdx.y * chunk;
    const uint32_t r1 = min(rows, r0 + chunk);
    float s = 0.0f;
    if (c < cols)
        for (uint32_t r = r0 + threadIdx.y; r < r1; r += 8) s += x[(size_t)r * cols + c];
    red[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && c < cols) {
        float t = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += red[k][threadIdx.x];
        part[(size_t)blockIdx.y * cols + c] = t;
    }
    if constexpr (FOLD)
        if (fg_last_block(arrivals + blockIdx.x, gridDim.y))
            fold_chunks_of_columns<FG_DTYPE_F32>(c, threadIdx.y, threadIdx.x, cols, gridDim.y, part, out, red);
}
// The chunks of column sums that other kernels left; a block covers 32 columns.
template <int DT>
__global__ void __launch_bounds__(256) colsum_fold_kernel(uint32_t cols, uint32_t nchunks,
                                                          const float* __restrict__ part, void* __restrict__ out) {
    fg_grid_enter();
    __shared__ float red[8][33];
    const uint32_t cx = threadIdx.x & 31u;
    fold_chunks_of_columns<DT>(blockIdx.x * 32 + cx, threadIdx.x >> 5, cx, cols, nchunks, part, out, red);
}


// ---- chain programs as run by the kernel ----
// The host turns a chain (forward, or backward = the values it needs followed by the adjoints) into a list of
// single-result operations: instructions whose result nobody reads are dropped, an adjoint's first contribution is a
// plain result and only later ones add, and results live in a few slots that are reused once their last reader has run.
// The kernel keeps one set of values in registers, the result of the operation just before: an operation takes its first
// operand there (fetched from its slot if it is another value), its second one from a slot, and leaves its result there.
enum : uint32_t { VM_G_TANH = 14, VM_G_RELU, VM_G_GELU, VM_G_ELU, VM_G_ABS,      // after the fg_ew codes: result = op(x, y)
                  VM_RSUB, VM_RDIV,                                              // y - x, y / x
                  VM_LD, VM_LD2, VM_ST, VM_LDADD, VM_COPY };
static_assert(FG_EW_ELU + 1 == (int)VM_G_TANH, "the operation codes are dense: one jump table");
constexpr uint32_t kVmFetch = 0x100, kVmAdd = 0x200, kVmKeep = 0x400;       // first operand from slot x; + slot acc; result to slot dst
struct VmOp {                          // slots as offsets in units of 16 bytes
    uint8_t op, flags, ptr, ptr2;      // VM_LD2: ptr2 goes to slot y, ptr to the registers
    uint32_t y;                        // FG_EW_CONST: the constant's bits
    uint16_t x, acc;
    uint32_t dst;
};
static_assert(sizeof(VmOp) == 16, "one 128-bit constant load per operation");
constexpr int kVmMaxOps = 200;      // backward: 24 values, the seed, at most five operations per instruction, 24 + 2 * 8 for the input gradients
constexpr int kVmMaxPtrs = FG_EW_MAX_INPUTS + 1 + FG_EW_MAX_INSTR;
struct VmArgs {
    uint4 ops[kVmMaxOps];
    void* ptr[kVmMaxPtrs];
    int nops, vec;
    uint64_t n;
};
static_assert(sizeof(VmArgs) <= 4096, "kernel parameters");

constexpr int kVmThreads = 128;
// 32-bit words of a value that a thread holds (template parameter W): eight, that is eight f32 elements or sixteen 16-bit ones in
// pairs; four where the tensor is small (see launch_chain).
constexpr int kVmWords = 8;
constexpr int kVmSlotUnits = 2 * kVmThreads;

// A value's words: Lanes<DT> does arithmetic on them.  With 16-bit storage every operation's result is rounded to the type.  The
// words stay packed: + - * on two elements at once in the type's own arithmetic, functions and the quotient on f32 lanes and
// then rounded.  For + - * both ways give the same bits (f32 has at least two bits more than twice the type's, so its own
// rounding does no harm), but for bf16 products below f32's normal range (2^-126), where f32 rounds coarser and the packed product, which
// is rounded once, is the nearer one.
template <int DT> struct Lanes {
    typedef typename std::conditional<DT == FG_DTYPE_F16, __half2, __nv_bfloat162>::type P;
    static constexpr int kE = 2;
    static constexpr uint32_t kOne = DT == FG_DTYPE_F16 ? 0x3c00u : 0x3f80u;      // 1
    static __device__ __forceinline__ P p(uint32_t u) { return *reinterpret_cast<P*>(&u); }
    static __device__ __forceinline__ uint32_t u(P v) { return *reinterpret_cast<uint32_t*>(&v); }
    static __device__ __forceinline__ float2 f(uint32_t v) {
        if constexpr (DT == FG_DTYPE_F16) return __half22float2(p(v));
        else return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    }
    static __device__ __forceinline__ uint32_t pack(float a, float b) {
        if constexpr (DT == FG_DTYPE_F16) return u(__floats2half2_rn(a, b));
        else return u(__floats2bfloat162_rn(a, b));
    }
    static __device__ __forceinline__ uint32_t all(float v) { return pack(v, v); }
    static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) { return u(__hadd2_rn(p(a), p(b))); }
    static __device__ __forceinline__ uint32_t sub(uint32_t a, uint32_t b) { return u(__hsub2_rn(p(a), p(b))); }
    static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) { return u(__hmul2_rn(p(a), p(b))); }
    static __device__ __forceinline__ uint32_t neg(uint32_t a) { return a ^ 0x80008000u; }
    static __device__ __forceinline__ uint32_t abs(uint32_t a) { return a & 0x7fff7fffu; }
    static __device__ __forceinline__ uint32_t relu(uint32_t a) { return u(__hmax2(p(a), p(0u))); }          // max(NaN, 0) = 0
    static __device__ __forceinline__ uint32_t positive(uint32_t a) { return u(__hgt2(p(a), p(0u))); }       // 1 or 0
    static __device__ __forceinline__ uint32_t where_ge0(uint32_t c, uint32_t a, uint32_t b) {               // c >= 0 ? a : b
        const uint32_t m = __hge2_mask(p(c), p(0u));
        return (a & m) | (b & ~m);
    }
    template <class F> static __device__ __forceinline__ uint32_t map(uint32_t a, F fn) {
        const float2 x = f(a);
        return pack(fn(x.x), fn(x.y));
    }
    template <class F> static __device__ __forceinline__ uint32_t map(uint32_t a, uint32_t b, F fn) {
        const float2 x = f(a), y = f(b);
        return pack(fn(x.x, y.x), fn(x.y, y.y));
    }
    // Element h of a word, from or to a tensor
    static __device__ __forceinline__ uint32_t bits(const void* t, uint64_t i) { return static_cast<const uint16_t*>(t)[i]; }
    static __device__ __forceinline__ void put(void* t, uint64_t i, uint32_t v) { static_cast<uint16_t*>(t)[i] = (uint16_t)v; }
};
template <> struct Lanes<FG_DTYPE_F32> {
    static constexpr int kE = 1;
    static constexpr uint32_t kOne = 0x3f800000u;
    static __device__ __forceinline__ float f(uint32_t v) { return __uint_as_float(v); }
    static __device__ __forceinline__ uint32_t u(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ uint32_t all(float v) { return u(v); }
    static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) { return u(f(a) + f(b)); }
    static __device__ __forceinline__ uint32_t sub(uint32_t a, uint32_t b) { return u(f(a) - f(b)); }
    static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) { return u(f(a) * f(b)); }
    static __device__ __forceinline__ uint32_t neg(uint32_t a) { return a ^ 0x80000000u; }
    static __device__ __forceinline__ uint32_t abs(uint32_t a) { return a & 0x7fffffffu; }
    static __device__ __forceinline__ uint32_t relu(uint32_t a) { return u(f(a) > 0.0f ? f(a) : 0.0f); }
    static __device__ __forceinline__ uint32_t positive(uint32_t a) { return u(f(a) > 0.0f ? 1.0f : 0.0f); }
    static __device__ __forceinline__ uint32_t where_ge0(uint32_t c, uint32_t a, uint32_t b) { return f(c) >= 0.0f ? a : b; }
    template <class F> static __device__ __forceinline__ uint32_t map(uint32_t a, F fn) { return u(fn(f(a))); }
    template <class F> static __device__ __forceinline__ uint32_t map(uint32_t a, uint32_t b, F fn) { return u(fn(f(a), f(b))); }
};

// Slots are in shared memory (a program is only known at run time, so its values cannot be named registers): a slot holds
// the words of each thread as planes of one uint4 per thread, so that every access is a conflict-free 128-bit one.
template <int W> __device__ __forceinline__ void slot_ld(const uint4* sm, uint32_t off, uint32_t* o) {
#pragma unroll
    for (int j = 0; j < W / 4; ++j) {
        const uint4 a = sm[off + j * kVmThreads];
        o[4 * j] = a.x; o[4 * j + 1] = a.y; o[4 * j + 2] = a.z; o[4 * j + 3] = a.w;
    }
}
template <int W> __device__ __forceinline__ void slot_st(uint4* sm, uint32_t off, const uint32_t* v) {
#pragma unroll
    for (int j = 0; j < W / 4; ++j) sm[off + j * kVmThreads] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
}

// A thread's words of a tensor.  VEC: groups of four elements, kVmThreads groups apart, in a tile that is whole; otherwise
// single elements, kVmThreads apart, as far as the tensor goes, and ones beyond it (the quotient of zeros takes the long way
// round: x / (1 + exp(-x)) * y backward on 100 000 halves 9.2 us, 8.4 with ones).
template <int DT, bool VEC, int W>
__device__ __forceinline__ void words_ld(const void* t, uint64_t i, uint64_t n, uint32_t* o) {
    if constexpr (VEC && DT == FG_DTYPE_F32) {
        const uint4* p = reinterpret_cast<const uint4*>(static_cast<const float*>(t) + i);
        uint4 a[W / 4];
#pragma unroll
        for (int j = 0; j < W / 4; ++j) a[j] = p[j * kVmThreads];
#pragma unroll
        for (int j = 0; j < W / 4; ++j) { o[4 * j] = a[j].x; o[4 * j + 1] = a[j].y; o[4 * j + 2] = a[j].z; o[4 * j + 3] = a[j].w; }
    } else if constexpr (VEC) {
        const uint2* p = reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(t) + i);
#pragma unroll
        for (int j = 0; j < W / 2; ++j) { const uint2 a = p[j * kVmThreads]; o[2 * j] = a.x; o[2 * j + 1] = a.y; }
    } else if constexpr (DT == FG_DTYPE_F32) {
#pragma unroll
        for (int w = 0; w < W; ++w) o[w] = i + w * kVmThreads < n ? static_cast<const uint32_t*>(t)[i + w * kVmThreads] : Lanes<DT>::kOne;
    } else {
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint64_t e = i + 2 * w * kVmThreads;
            o[w] = (e < n ? Lanes<DT>::bits(t, e) : Lanes<DT>::kOne) | (e + kVmThreads < n ? Lanes<DT>::bits(t, e + kVmThreads) : Lanes<DT>::kOne) << 16;
        }
    }
}
template <int DT, bool VEC, int W>
__device__ __forceinline__ void words_st(void* t, uint64_t i, uint64_t n, const uint32_t* v) {
    if constexpr (VEC && DT == FG_DTYPE_F32) {
        uint4* p = reinterpret_cast<uint4*>(static_cast<float*>(t) + i);
#pragma unroll
        for (int j = 0; j < W / 4; ++j) p[j * kVmThreads] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    } else if constexpr (VEC) {
        uint2* p = reinterpret_cast<uint2*>(static_cast<uint16_t*>(t) + i);
#pragma unroll
        for (int j = 0; j < W / 2; ++j) p[j * kVmThreads] = make_uint2(v[2 * j], v[2 * j + 1]);
    } else if constexpr (DT == FG_DTYPE_F32) {
#pragma unroll
        for (int w = 0; w < W; ++w)
            if (i + w * kVmThreads < n) static_cast<uint32_t*>(t)[i + w * kVmThreads] = v[w];
    } else {
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint64_t e = i + 2 * w * kVmThreads;
            if (e < n) Lanes<DT>::put(t, e, v[w]);
            if (e + kVmThreads < n) Lanes<DT>::put(t, e + kVmThreads, v[w] >> 16);
        }
    }
}

// The program on a thread's elements of one tile, the first of them i.  The only values that live from one operation to the
// next are v[]; every second operand is fetched inside the case that reads it.
//
// What bounds it: instruction issue, on large f32 tensors together with HBM.  Fetching, decoding and keeping one operation
// takes about 35 instructions for the eight words (70 with both operands live across the loop, ncu's executed instructions).
// Forward and backward: gelu(x * y) + x on 32 Mi f32 257 -> 211 us (3.8 TB/s), x / (1 + exp(-x)) * y on 3 000 001 halves
// 42.3 -> 21.5 us, with both launches.  Requesting the next tile's words ahead through cp.async lost 6 % (the copies out of the
// staging cost more issue slots than the waits); sixteen words per thread gain 3 % in f32 and lose 30 % on halves.
template <int DT, bool VEC, int W>
__device__ __forceinline__ void vm_run(const VmArgs& a, uint64_t i, uint4* sm) {
    typedef Lanes<DT> L;
    uint32_t v[W];
#pragma unroll
    for (int w = 0; w < W; ++w) v[w] = 0u;
#define FG_VM_1(expr) _Pragma("unroll") for (int w = 0; w < W; ++w) { const uint32_t x = v[w]; v[w] = (expr); } break
#define FG_VM_2(expr)                                                                                       \
    {                                                                                                       \
        uint32_t yy[W];                                                                              \
        slot_ld<W>(sm, c.y, yy);                                                                            \
        _Pragma("unroll") for (int w = 0; w < W; ++w) { const uint32_t x = v[w], y = yy[w]; v[w] = (expr); } \
    } break
#pragma unroll 1
    for (int k = 0; k < a.nops; ++k) {
        const uint4 c = a.ops[k];
        const uint32_t flags = c.x;
        if (flags & kVmFetch) slot_ld<W>(sm, c.z & 0xffffu, v);
        switch (c.x & 255u) {
            case FG_EW_CONST: {
                const uint32_t k0 = L::all(__uint_as_float(c.y));
                FG_VM_1((void(x), k0));
            }
            case FG_EW_ADD: FG_VM_2(L::add(x, y));
            case FG_EW_SUB: FG_VM_2(L::sub(x, y));
            case VM_RSUB: FG_VM_2(L::sub(y, x));
            case FG_EW_MUL: FG_VM_2(L::mul(x, y));
            case FG_EW_DIV: FG_VM_2(L::map(x, y, [](float p, float q) { return __fdiv_rn(p, q); }));
            case VM_RDIV: FG_VM_2(L::map(y, x, [](float p, float q) { return __fdiv_rn(p, q); }));
            case FG_EW_NEG: FG_VM_1(L::neg(x));
            case FG_EW_ABS: FG_VM_1(L::abs(x));
            case FG_EW_EXP: FG_VM_1(L::map(x, [](float p) { return expf(p); }));
            case FG_EW_LOG: FG_VM_1(L::map(x, [](float p) { return logf(p); }));
            case FG_EW_TANH: FG_VM_1(L::map(x, [](float p) { return tanhf(p); }));
            case FG_EW_RELU: FG_VM_1(L::relu(x));
            case FG_EW_GELU: FG_VM_1(L::map(x, [](float p) { return fg_gelu_fwd(p); }));
            case FG_EW_ELU: FG_VM_1(L::map(x, [](float p) { return p >= 0.0f ? p : expf(p) - 1.0f; }));
            // adjoints: x is the adjoint of the result, y the value the derivative is taken at
            case VM_G_TANH: FG_VM_2(L::mul(x, L::sub(L::all(1.0f), L::mul(y, y))));
            case VM_G_RELU: FG_VM_2(L::mul(x, L::positive(y)));
            case VM_G_GELU: FG_VM_2(L::mul(x, L::map(y, [](float p) { return fg_gelu_grad(p); })));
            case VM_G_ELU: FG_VM_2(L::where_ge0(y, x, L::mul(x, L::add(y, L::all(1.0f)))));
            case VM_G_ABS: FG_VM_2(L::where_ge0(y, x, L::neg(x)));
            case VM_LD: words_ld<DT, VEC, W>(a.ptr[c.x >> 16 & 255u], i, a.n, v); break;
            case VM_LD2: {                                  // both on their way at once
                uint32_t yy[W];
                words_ld<DT, VEC, W>(a.ptr[c.x >> 24], i, a.n, yy);
                words_ld<DT, VEC, W>(a.ptr[c.x >> 16 & 255u], i, a.n, v);
                slot_st<W>(sm, c.y, yy);
                break;
            }
            case VM_ST: words_st<DT, VEC, W>(a.ptr[c.x >> 16 & 255u], i, a.n, v); break;
            case VM_LDADD: {
                uint32_t yy[W];
                words_ld<DT, VEC, W>(a.ptr[c.x >> 16 & 255u], i, a.n, yy);
#pragma unroll
                for (int w = 0; w < W; ++w) v[w] = L::add(yy[w], v[w]);
                break;
            }
            case VM_COPY: break;
            default: __builtin_unreachable();      // the host writes no other code: the jump needs no range check
        }
        if (flags & (kVmAdd | kVmKeep)) {
            if (flags & kVmAdd) {
                uint32_t yy[W];
                slot_ld<W>(sm, c.z >> 16, yy);
#pragma unroll
                for (int w = 0; w < W; ++w) v[w] = L::add(yy[w], v[w]);
            }
            if (flags & kVmKeep) slot_st<W>(sm, c.w, v);
        }
    }
#undef FG_VM_1
#undef FG_VM_2
}

// A block takes one tile of W words per thread at a time; block 0 of a vectorised launch has the incomplete last tile
// instead, element by element, so that no other tile needs bounds.
template <int DT, bool VEC, int W>
__global__ void __launch_bounds__(kVmThreads, 10) chain_kernel(const __grid_constant__ VmArgs a) {
    fg_grid_enter();
    extern __shared__ uint4 chain_smem[];
    uint4* const sm = chain_smem + threadIdx.x;
    constexpr uint32_t kTile = W * Lanes<DT>::kE * kVmThreads;
    if constexpr (VEC) {
        const uint64_t whole = a.n / kTile;
        const uint32_t rest = a.n % kTile != 0;
        if (rest && blockIdx.x == 0) {
            vm_run<DT, false, W>(a, whole * kTile + threadIdx.x, sm);
            return;
        }
        for (uint64_t t = blockIdx.x - rest; t < whole; t += gridDim.x - rest) vm_run<DT, true, W>(a, t * kTile + threadIdx.x * 4, sm);
    } else {
        for (uint64_t t = blockIdx.x; t * kTile < a.n; t += gridDim.x) vm_run<DT, false, W>(a, t * kTile + threadIdx.x, sm);
    }
}

// ---- host side: a chain as a list of operations ----
struct VmBuilder {
    struct Node { int op, x, y, acc, ptr; float imm; int id, ptr2, id2; };    // operands are result ids, -1 = none
    Node node[kVmMaxOps];
    int n = 0, ids = 0;
    int emit(int op, int x, int y, int acc, int ptr, float imm) {
        const int id = op == (int)VM_ST ? -1 : ids++;
        node[n++] = Node{op, x, y, acc, ptr, imm, id, -1, -1};
        return id;
    }
    // Loads before the first store move to the front (at most four: each holds a slot until it is used) and go two at a time.
    void gather_loads() {
        Node ld[4], rest[kVmMaxOps];
        int nl = 0, nr = 0;
        bool stored = false;
        for (int i = 0; i < n; ++i) {
            stored |= node[i].op == (int)VM_ST;
            if (node[i].op == (int)VM_LD && !stored && nl < 4) ld[nl++] = node[i];
            else rest[nr++] = node[i];
        }
        n = 0;
        int i = 0;
        for (; i + 1 < nl; i += 2) {
            node[n] = ld[i + 1];
            node[n].op = VM_LD2;
            node[n].ptr2 = ld[i].ptr;
            node[n++].id2 = ld[i].id;
        }
        if (i < nl) node[n++] = ld[i];
        for (int j = 0; j < nr; ++j) node[n++] = rest[j];
    }
    // Assigns slots by the results' life times and writes the kernel's operations; returns the number of slots.
    int finish(VmArgs* a) {
        gather_loads();
        int last_use[kVmMaxOps], slot[kVmMaxOps];
        bool stored[kVmMaxOps], taken[kVmMaxOps];
        for (int i = 0; i < ids; ++i) { last_use[i] = -1; slot[i] = -1; stored[i] = false; }
        for (int i = 0; i < kVmMaxOps; ++i) taken[i] = false;
        auto next_last = [](const Node& o, int prev) { return o.id >= 0 ? o.id : o.x >= 0 ? o.x : prev; };
        int prev = -1;      // the value that is in `last` before operation i
        for (int i = 0; i < n; ++i) {
            Node& o = node[i];
            // what is in the registers serves as the first operand
            if (o.y == prev && o.x != prev && o.op >= FG_EW_ADD && o.op <= FG_EW_DIV) {
                const int t = o.x; o.x = o.y; o.y = t;
                o.op = o.op == FG_EW_SUB ? (int)VM_RSUB : o.op == FG_EW_DIV ? (int)VM_RDIV : o.op;
            }
            if (o.x >= 0 && o.x != prev) { stored[o.x] = true; last_use[o.x] = i; }
            if (o.y >= 0) { stored[o.y] = true; last_use[o.y] = i; }
            if (o.acc >= 0) { stored[o.acc] = true; last_use[o.acc] = i; }
            if (o.id2 >= 0) { stored[o.id2] = true; if (last_use[o.id2] < i) last_use[o.id2] = i; }
            prev = next_last(o, prev);
        }
        int nslots = 0;
        auto take = [&](int id) {
            int f = 0;
            while (taken[f]) ++f;
            taken[f] = true;
            slot[id] = f;
            if (f + 1 > nslots) nslots = f + 1;
        };
        prev = -1;
        for (int i = 0; i < n; ++i) {
            const Node& o = node[i];
            auto at = [&](int u) -> uint16_t { return u < 0 ? (uint16_t)0 : (uint16_t)(slot[u] * kVmSlotUnits); };
            VmOp v{};
            v.op = (uint8_t)o.op;
            if (o.x >= 0 && o.x != prev) { v.flags |= kVmFetch >> 8; v.x = at(o.x); }
            v.y = at(o.y);
            if (o.acc >= 0) { v.flags |= kVmAdd >> 8; v.acc = at(o.acc); }
            v.ptr = (uint8_t)(o.ptr < 0 ? 0 : o.ptr);
            v.ptr2 = (uint8_t)(o.ptr2 < 0 ? 0 : o.ptr2);
            if (o.op == FG_EW_CONST) memcpy(&v.y, &o.imm, 4);
            if (o.id2 >= 0) { take(o.id2); v.y = at(o.id2); }
            // a slot whose last reader this is may receive the result: operands are read before it is written
            for (int u : {o.x, o.y, o.acc, o.id2})
                if (u >= 0 && slot[u] >= 0 && last_use[u] == i && !(u == o.id2 && o.op != (int)VM_LD2)) taken[slot[u]] = false;
            if (o.id >= 0 && stored[o.id]) { take(o.id); v.flags |= kVmKeep >> 8; v.dst = at(o.id); }
            prev = next_last(o, prev);
            memcpy(&a->ops[i], &v, sizeof(v));
        }
        a->nops = n;
        return nslots;
    }
};

inline bool ew_two_operands(int op) { return op >= FG_EW_ADD && op <= FG_EW_DIV; }

// The instructions marked in `need`, in order; id[k] becomes the result of instruction k.
void build_values(VmBuilder& b, const fg_ew_instr* prog, int ninstr, const bool* need, int* id, void* const* saved, int saved_ptr0) {
    for (int k = 0; k < ninstr; ++k) {
        if (!need[k]) continue;
        const fg_ew_instr& in = prog[k];
        if (in.op == FG_EW_INPUT) id[k] = b.emit(VM_LD, -1, -1, -1, in.a, 0.0f);
        else if (in.op == FG_EW_CONST) id[k] = b.emit(in.op, -1, -1, -1, -1, in.imm);
        else id[k] = b.emit(in.op, id[in.a], ew_two_operands(in.op) ? id[in.b] : -1, -1, -1, in.imm);
        if (saved && saved[k]) b.emit(VM_ST, id[k], -1, -1, saved_ptr0 + k, 0.0f);
    }
}
// Marks everything the marked instructions read.
void close_over(const fg_ew_instr* prog, int ninstr, bool* need) {
    for (int k = ninstr - 1; k >= 0; --k) {
        if (!need[k] || prog[k].op == FG_EW_INPUT || prog[k].op == FG_EW_CONST) continue;
        need[prog[k].a] = true;
        if (ew_two_operands(prog[k].op)) need[prog[k].b] = true;
    }
}

// Pointer table: inputs, then (forward) the output and the saved values, or (backward) the seed and the gradients.
constexpr int kPtrOut = FG_EW_MAX_INPUTS, kPtrSaved = FG_EW_MAX_INPUTS + 1;

void build_forward(VmBuilder& b, const fg_ew_instr* prog, int ninstr, void* const* saved) {
    bool need[FG_EW_MAX_INSTR] = {};
    int id[FG_EW_MAX_INSTR];
    for (int k = 0; k < ninstr; ++k) need[k] = k == ninstr - 1 || (saved && saved[k]);
    close_over(prog, ninstr, need);
    build_values(b, prog, ninstr, need, id, saved, kPtrSaved);
    b.emit(VM_ST, id[ninstr - 1], -1, -1, kPtrOut, 0.0f);
}

// Adjoints are added up in the order of the program walked backwards, operand a before operand b, and an input that is
// loaded several times sums its loads' adjoints from the last one down: the rounding of 16-bit storage depends on it.
void build_backward(VmBuilder& b, const fg_ew_instr* prog, int ninstr, int ninputs, void* const* grads, bool accumulate) {
    bool active[FG_EW_MAX_INSTR] = {}, touched[FG_EW_MAX_INSTR] = {}, need[FG_EW_MAX_INSTR] = {};
    int id[FG_EW_MAX_INSTR], adj[FG_EW_MAX_INSTR];
    for (int k = 0; k < ninstr; ++k) {          // does a wanted gradient lie below this instruction?
        const fg_ew_instr& in = prog[k];
        id[k] = adj[k] = -1;
        if (in.op == FG_EW_INPUT) active[k] = grads[in.a] != nullptr;
        else if (in.op != FG_EW_CONST) active[k] = active[in.a] || (ew_two_operands(in.op) && active[in.b]);
    }
    touched[ninstr - 1] = true;
    for (int k = ninstr - 1; k >= 0; --k) {     // which values do the derivatives read?
        const fg_ew_instr& in = prog[k];
        if (!touched[k] || !active[k] || in.op == FG_EW_INPUT || in.op == FG_EW_CONST) continue;
        const bool two = ew_two_operands(in.op), da = active[in.a], db = two && active[in.b];
        if (da) touched[in.a] = true;
        if (db) touched[in.b] = true;
        switch (in.op) {
            case FG_EW_MUL: if (da) need[in.b] = true; if (db) need[in.a] = true; break;
            case FG_EW_DIV: need[in.b] = true; if (db) need[in.a] = true; break;
            case FG_EW_ABS: case FG_EW_LOG: case FG_EW_GELU: need[in.a] = true; break;
            case FG_EW_EXP: case FG_EW_TANH: case FG_EW_RELU: case FG_EW_ELU: need[k] = true; break;
            default: break;
        }
    }
    close_over(prog, ninstr, need);
    build_values(b, prog, ninstr, need, id, nullptr, 0);
    bool flows = false;
    for (int k = 0; k < ninstr; ++k) flows |= prog[k].op == FG_EW_INPUT && active[k] && touched[k];
    if (flows) adj[ninstr - 1] = b.emit(VM_LD, -1, -1, -1, kPtrOut, 0.0f);
    for (int k = ninstr - 1; k >= 0 && flows; --k) {
        const fg_ew_instr& in = prog[k];
        if (!touched[k] || !active[k] || in.op == FG_EW_INPUT || in.op == FG_EW_CONST) continue;
        const int g = adj[k];
        auto add = [&](int to, int op, int x, int y) {
            if (adj[to] < 0 && op == (int)VM_COPY) adj[to] = x;              // a first contribution that is the adjoint itself
            else adj[to] = b.emit(op, x, y, adj[to], -1, 0.0f);
        };
        const bool da = active[in.a], db = ew_two_operands(in.op) && active[in.b];
        switch (in.op) {
            case FG_EW_ADD: if (da) add(in.a, VM_COPY, g, -1); if (db) add(in.b, VM_COPY, g, -1); break;
            case FG_EW_SUB: if (da) add(in.a, VM_COPY, g, -1); if (db) add(in.b, FG_EW_NEG, g, -1); break;
            case FG_EW_MUL: if (da) add(in.a, FG_EW_MUL, g, id[in.b]); if (db) add(in.b, FG_EW_MUL, g, id[in.a]); break;
            case FG_EW_DIV:
                if (da) add(in.a, FG_EW_DIV, g, id[in.b]);
                if (db) {       // - (g * a) / (b * b), every step rounded
                    const int den = b.emit(FG_EW_MUL, id[in.b], id[in.b], -1, -1, 0.0f), num = b.emit(FG_EW_MUL, g, id[in.a], -1, -1, 0.0f);
                    add(in.b, FG_EW_NEG, b.emit(FG_EW_DIV, num, den, -1, -1, 0.0f), -1);
                }
                break;
            case FG_EW_NEG: add(in.a, FG_EW_NEG, g, -1); break;
            case FG_EW_ABS: add(in.a, VM_G_ABS, g, id[in.a]); break;
            case FG_EW_EXP: add(in.a, FG_EW_MUL, g, id[k]); break;
            case FG_EW_LOG: add(in.a, FG_EW_DIV, g, id[in.a]); break;
            case FG_EW_TANH: add(in.a, VM_G_TANH, g, id[k]); break;
            case FG_EW_RELU: add(in.a, VM_G_RELU, g, id[k]); break;
            case FG_EW_GELU: add(in.a, VM_G_GELU, g, id[in.a]); break;
            case FG_EW_ELU: add(in.a, VM_G_ELU, g, id[k]); break;
            default: break;
        }
    }
    for (int j = 0; j < ninputs; ++j) {
        if (!grads[j]) continue;
        int sum = -1;
        for (int k = ninstr - 1; k >= 0; --k) {
            if (prog[k].op != FG_EW_INPUT || prog[k].a != j || adj[k] < 0) continue;
            sum = sum < 0 ? adj[k] : b.emit(FG_EW_ADD, sum, adj[k], -1, -1, 0.0f);
        }
        if (sum < 0) sum = b.emit(FG_EW_CONST, -1, -1, -1, -1, 0.0f);       // nothing flows into this input
        if (accumulate) sum = b.emit(VM_LDADD, sum, -1, -1, kPtrSaved + j, 0.0f);
        b.emit(VM_ST, sum, -1, -1, kPtrSaved + j, 0.0f);
    }
}

// dst[i] = (type of dst) src[i], round to nearest even; four elements per access when both ends allow it
template <int DS, int DD>
__global__ void __launch_bounds__(256) convert_kernel(const void* __restrict__ src, void* __restrict__ dst, uint64_t n, int vec) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nv = vec ? n >> 2 : 0;
    for (uint64_t i = g; i < nv; i += stride) {
        float v[4];
        Stored<DS>::ld4w(src, i << 2, v);
        Stored<DD>::st4w(dst, i << 2, v);
    }
    for (uint64_t i = (nv << 2) + g; i < n; i += stride) Stored<DD>::st(dst, i, Stored<DS>::ld(src, i));
}

// A program with many live values needs more than the default 48 KB of dynamic shared memory (4 KB per slot, and there
// are at most 24 values and 24 adjoints): the limit is raised once per device and kernel.
constexpr int kSlotBytes = kVmSlotUnits * (int)sizeof(uint4);
constexpr int kChainSmemMax = 2 * FG_EW_MAX_INSTR * kSlotBytes;
int32_t launch_chain(fg_ctx* ctx, int dtype, VmBuilder& b, VmArgs& a, double bytes) {
    static std::atomic<uint64_t> done[3][2][2];
    const uint64_t bit = 1ull << (ctx->device & 63);
    const size_t smem = (size_t)b.finish(&a) * kSlotBytes;
    if (smem > (size_t)kChainSmemMax) return fg_fail(ctx, FG_ERR_INTERNAL, "eltwise chain: too many live values");
    // As many blocks as an SM holds at once (ten by registers, fewer when the slots fill the shared memory), each with the same
    // number of tiles: a grid of sixteen per SM ran as one full wave and a second of three quarters.
    const size_t fit = (220u * 1024u) / (smem + 1024);
    const uint64_t per_sm = fit < 1 ? 1 : fit > 10 ? 10 : fit, cap_sm = (uint64_t)ctx->sm_count * per_sm;
    // Small tensors: a thread's elements come one after the other and the SMs are half empty, so four words each while that makes
    // five blocks per SM or fewer, two for a program of one operation, which waits for its loads.  Us with four words and with
    // eight: x / (1 + exp(-x)) * y backward 8.4 and 14.4 on 100 000 halves, 8.8 and 11.3 on 757 760 (five blocks per SM), 10.0 and 11.8
    // on 1 Mi, 27 and 24 on 3 M; x + y 1.9 and 2.1 on 300 001, 2.1 and 2.0 on 500 000; in f32 gelu(x * y) + x forward 2.2 and 2.4 on
    // 100 000, 2.6 and 2.6 on 300 001, 3.3 and 3.0 on 757 760.
    const uint64_t blocks = a.nops <= 4 ? 2 : per_sm < 5 ? per_sm : 5;
    const bool few = a.n <= (uint64_t)ctx->sm_count * blocks * (kVmWords / 2) * (dtype == FG_DTYPE_F32 ? 1 : 2) * kVmThreads;
    const int words = few ? kVmWords / 2 : kVmWords;
    auto of_type = [&](auto vec, auto small) {
        constexpr bool V = decltype(vec)::value;
        constexpr int W = decltype(small)::value ? kVmWords / 2 : kVmWords;
        return dtype == FG_DTYPE_F32 ? chain_kernel<FG_DTYPE_F32, V, W> : dtype == FG_DTYPE_F16 ? chain_kernel<FG_DTYPE_F16, V, W> : chain_kernel<FG_DTYPE_BF16, V, W>;
    };
    const std::true_type yes{};
    const std::false_type no{};
    auto kernel = a.vec ? (few ? of_type(yes, yes) : of_type(yes, no)) : few ? of_type(no, yes) : of_type(no, no);
    std::atomic<uint64_t>& set = done[dtype][a.vec ? 1 : 0][few ? 1 : 0];
    if (!(set.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kChainSmemMax);
        if (e != cudaSuccess) return fg_fail_cuda(ctx, FG_ERR_INTERNAL, "cudaFuncSetAttribute(chain kernel)", e);
        set.fetch_or(bit, std::memory_order_release);
    }
    const uint64_t tile = (uint64_t)words * (dtype == FG_DTYPE_F32 ? 1 : 2) * kVmThreads;
    const uint64_t rest = a.vec && a.n % tile ? 1 : 0, tiles = a.vec ? a.n / tile : (a.n + tile - 1) / tile;
    const uint64_t cap = cap_sm - rest;
    const uint64_t rounds = tiles ? (tiles + cap - 1) / cap : 1;
    const int grid = (int)((tiles + rounds - 1) / rounds + rest);
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_ELTWISE, bytes);
    fg_launch(ctx, kernel, grid, kVmThreads, smem, a);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

int32_t check_prog(fg_ctx* ctx, const fg_ew_instr* prog, int32_t ninstr, int32_t ninputs) {
    FG_REQUIRE(ctx, prog != nullptr, "eltwise chain: prog is NULL");
    FG_REQUIRE(ctx, ninstr >= 1 && ninstr <= FG_EW_MAX_INSTR, "eltwise chain: instruction count out of range");
    FG_REQUIRE(ctx, ninputs >= 1 && ninputs <= FG_EW_MAX_INPUTS, "eltwise chain: input count out of range");
    for (int k = 0; k < ninstr; ++k) {
        const fg_ew_instr& in = prog[k];
        FG_REQUIRE(ctx, in.op >= FG_EW_INPUT && in.op <= FG_EW_ELU, "eltwise chain: unknown op code");
        if (in.op == FG_EW_INPUT) {
            FG_REQUIRE(ctx, in.a >= 0 && in.a < ninputs, "eltwise chain: input index out of range");
        } else if (in.op != FG_EW_CONST) {
            FG_REQUIRE(ctx, in.a >= 0 && in.a < k, "eltwise chain: operand a must name an earlier value");
            if (in.op >= FG_EW_ADD && in.op <= FG_EW_DIV)
                FG_REQUIRE(ctx, in.b >= 0 && in.b < k, "eltwise chain: operand b must name an earlier value");
        }
    }
    return FG_OK;
}

}  // namespace

int32_t fg_act_bwd_launch(fg_ctx* ctx, uint64_t n, int act, const float* dy, const float* saved, float* dz) {
    const bool vec = aligned16(dy) && aligned16(saved) && aligned16(dz);
    const int grid = fg_stream_grid(ctx, vec ? (n + 3) / 4 : n, 256, 8);
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_ELTWISE, (act == FG_ACT_NONE ? 8.0 : 12.0) * n);
    if (vec) fg_launch(ctx, act_bwd_kernel<true>, grid, 256, 0, n, act, dy, saved, dz);
    else fg_launch(ctx, act_bwd_kernel<false>, grid, 256, 0, n, act, dy, saved, dz);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

int32_t fg_colsum_fold_launch(fg_ctx* ctx, uint32_t cols, uint32_t nchunks, const float* part, void* out, int out_dtype) {
    const uint32_t grid = (cols + 31) / 32;
    if (out_dtype == FG_DTYPE_F32) fg_launch(ctx, colsum_fold_kernel<FG_DTYPE_F32>, grid, 256, 0, cols, nchunks, part, out);
    else if (out_dtype == FG_DTYPE_F16) fg_launch(ctx, colsum_fold_kernel<FG_DTYPE_F16>, grid, 256, 0, cols, nchunks, part, out);
    else fg_launch(ctx, colsum_fold_kernel<FG_DTYPE_BF16>, grid, 256, 0, cols, nchunks, part, out);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

int32_t fg_block_sums(fg_ctx* ctx, int grid, float* sum, FgBlockSums* b) {
    *b = FgBlockSums{sum, nullptr, sum, grid};
    if (!sum || grid == 1) return FG_OK;
    void* p;
    const int32_t s = fg_ws_alloc(ctx, (uint64_t)grid * sizeof(float), &p);
    if (s != FG_OK) return s;
    b->partials = (float*)p;
    if (fg_fold_in_launch(ctx, (uint64_t)grid)) b->out = sum;
    return FG_OK;
}
int32_t fg_block_sums_end(fg_ctx* ctx, const FgBlockSums& b) {
    if (b.out || b.partials == b.sum) return FG_OK;
    fg_launch(ctx, fold_partials_kernel, 1, 256, 0, (const float*)b.partials, (uint32_t)b.grid, b.sum);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

int32_t fg_colsum_launch(fg_ctx* ctx, uint32_t rows, uint32_t cols, const float* x, float* out) {
    const uint32_t chunk = 256, groups = (cols + 31) / 32;
    const uint32_t nchunks = (rows + chunk - 1) / chunk;
    dim3 grid(groups, nchunks), block(32, 8);
    if (nchunks == 1) {      // the only partial is the sum
        fg_launch(ctx, colsum_kernel<false>, grid, block, 0, rows, cols, chunk, x, out, (unsigned*)nullptr, (float*)nullptr);
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
    void* part;
    int32_t s = fg_ws_alloc(ctx, (uint64_t)nchunks * cols * sizeof(float), &part);
    if (s != FG_OK) return s;
    if (groups <= kFgArrivals && fg_fold_in_launch(ctx, (uint64_t)groups * nchunks)) {      // a counter for each group of columns
        fg_launch(ctx, colsum_kernel<true>, grid, block, 0, rows, cols, chunk, x, (float*)part, fg_arrivals(ctx), out);
        FG_LAUNCHED(ctx);
        return FG_OK;
    }
    fg_launch(ctx, colsum_kernel<false>, grid, block, 0, rows, cols, chunk, x, (float*)part, (unsigned*)nullptr, (float*)nullptr);
    FG_LAUNCHED(ctx);
    return fg_colsum_fold_launch(ctx, cols, nchunks, (const float*)part, out);
}

extern "C" {

int32_t fg_bias_act_fwd(fg_ctx* ctx, uint32_t rows, uint32_t cols, const float* z, const float* bias, int32_t act,
                        float* y) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, z && y, "fg_bias_act_fwd: NULL pointer");
    FG_REQUIRE(ctx, act >= FG_ACT_NONE && act <= FG_ACT_GELU, "fg_bias_act_fwd: unknown activation");
    if ((uint64_t)rows * cols == 0) return FG_OK;
    const uint64_t n = (uint64_t)rows * cols;
    const bool vec = (cols & 3u) == 0 && aligned16(z) && aligned16(bias) && aligned16(y);
    const int grid = fg_stream_grid(ctx, vec ? n / 4 : n, 256, 8);
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_ELTWISE, 8.0 * n);
    if (vec) bias_act_kernel<true><<<grid, 256, 0, ctx->stream>>>(rows, cols, z, bias, act, y);
    else bias_act_kernel<false><<<grid, 256, 0, ctx->stream>>>(rows, cols, z, bias, act, y);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

int32_t fg_act_bwd(fg_ctx* ctx, uint64_t n, int32_t act, const float* dy, const float* saved, float* dz) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, dy && dz, "fg_act_bwd: NULL pointer");
    FG_REQUIRE(ctx, act >= FG_ACT_NONE && act <= FG_ACT_GELU, "fg_act_bwd: unknown activation");
    FG_REQUIRE(ctx, act == FG_ACT_NONE || saved, "fg_act_bwd: saved tensor required");
    if (n == 0) return FG_OK;
    return fg_act_bwd_launch(ctx, n, act, dy, saved, dz);
}

int32_t fg_sum_f32(fg_ctx* ctx, const float* x, uint64_t n, float* out) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, x && out, "fg_sum_f32: NULL pointer");
    if (n == 0) {
        FG_CUDA(ctx, FG_ERR_FAILED_BUFFER_COPY, cudaMemsetAsync(out, 0, 4, ctx->stream));
        return FG_OK;
    }
    const int grid = fg_stream_grid(ctx, (n + 3) / 4, 256, 4);
    FgBlockSums b;
    const int32_t s = fg_block_sums(ctx, grid, out, &b);
    if (s != FG_OK) return s;
    fg_launch(ctx, sum_kernel, grid, 256, 0, x, n, b.partials, fg_arrivals(ctx), b.out);
    FG_LAUNCHED(ctx);
    return fg_block_sums_end(ctx, b);
}

int32_t fg_mse_loss_grad(fg_ctx* ctx, const float* pred, const float* target, uint64_t n, float grad_scale,
                         float* loss_elem_out, float* loss_sum_out, float* grad_out) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, pred && target, "fg_mse_loss_grad: NULL pointer");
    FG_REQUIRE(ctx, loss_elem_out || loss_sum_out || grad_out, "fg_mse_loss_grad: no output requested");
    if (n == 0) {
        if (loss_sum_out) FG_CUDA(ctx, FG_ERR_FAILED_BUFFER_COPY, cudaMemsetAsync(loss_sum_out, 0, 4, ctx->stream));
        return FG_OK;
    }
    const bool vec = aligned16(pred) && aligned16(target) && aligned16(loss_elem_out) && aligned16(grad_out);
    const int grid = fg_stream_grid(ctx, vec ? (n + 3) / 4 : n, 256, 8);
    FgBlockSums b;
    const int32_t s = fg_block_sums(ctx, grid, loss_sum_out, &b);
    if (s != FG_OK) return s;
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_ELTWISE, (8.0 + (loss_elem_out ? 4.0 : 0.0) + (grad_out ? 4.0 : 0.0)) * n);
    if (vec) fg_launch(ctx, loss_kernel<MseTerm, true>, grid, 256, 0, pred, target, n, grad_scale, loss_elem_out, grad_out, b.partials, fg_arrivals(ctx), b.out);
    else fg_launch(ctx, loss_kernel<MseTerm, false>, grid, 256, 0, pred, target, n, grad_scale, loss_elem_out, grad_out, b.partials, fg_arrivals(ctx), b.out);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return fg_block_sums_end(ctx, b);
}

int32_t fg_bce_loss_grad(fg_ctx* ctx, const float* pred, const float* target, uint64_t n, float grad_scale,
                         float* loss_elem_out, float* loss_sum_out, float* grad_out) {
    FG_ENTER(ctx);
    FG_REQUIRE(ctx, pred && target, "fg_bce_loss_grad: NULL pointer");
    FG_REQUIRE(ctx, loss_elem_out || loss_sum_out || grad_out, "fg_bce_loss_grad: no output requested");
    if (n == 0) {
        if (loss_sum_out) FG_CUDA(ctx, FG_ERR_FAILED_BUFFER_COPY, cudaMemsetAsync(loss_sum_out, 0, 4, ctx->stream));
        return FG_OK;
    }
    const bool vec = aligned16(pred) && aligned16(target) && aligned16(loss_elem_out) && aligned16(grad_out);
    const int grid = fg_stream_grid(ctx, vec ? (n + 3) / 4 : n, 256, 8);
    FgBlockSums b;
    const int32_t s = fg_block_sums(ctx, grid, loss_sum_out, &b);
    if (s != FG_OK) return s;
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_ELTWISE, (8.0 + (loss_elem_out ? 4.0 : 0.0) + (grad_out ? 4.0 : 0.0)) * n);
    if (vec) fg_launch(ctx, loss_kernel<BceTerm, true>, grid, 256, 0, pred, target, n, grad_scale, loss_elem_out, grad_out, b.partials, fg_arrivals(ctx), b.out);
    else fg_launch(ctx, loss_kernel<BceTerm, false>, grid, 256, 0, pred, target, n, grad_scale, loss_elem_out, grad_out, b.partials, fg_arrivals(ctx), b.out);
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return fg_block_sums_end(ctx, b);
}

int32_t fg_eltwise_chain_fwd_dt(fg_ctx* ctx, int32_t dtype, uint64_t n, const fg_ew_instr* prog, int32_t ninstr,
                                const void* const* inputs, int32_t ninputs, void* out, void* const* saved_out) {
    FG_ENTER(ctx);
    int32_t s = check_prog(ctx, prog, ninstr, ninputs);
    if (s != FG_OK) return s;
    FG_REQUIRE(ctx, dtype >= FG_DTYPE_F32 && dtype <= FG_DTYPE_BF16, "fg_eltwise_chain_fwd: unknown dtype");
    FG_REQUIRE(ctx, inputs && out, "fg_eltwise_chain_fwd: NULL pointer");
    VmArgs a;
    memset(&a, 0, sizeof(a));
    for (int k = 0; k < ninputs; ++k) {
        FG_REQUIRE(ctx, inputs[k] != nullptr, "fg_eltwise_chain_fwd: NULL input");
        a.ptr[k] = const_cast<void*>(inputs[k]);
    }
    if (saved_out) for (int k = 0; k < ninstr; ++k) a.ptr[kPtrSaved + k] = saved_out[k];
    a.ptr[kPtrOut] = out;
    a.n = n;
    if (n == 0) return FG_OK;
    // four elements per access when every tensor starts on a boundary of four elements
    const uintptr_t mask = dtype == FG_DTYPE_F32 ? 15u : 7u;
    uintptr_t bits = 0;
    int tensors = 0;
    for (void* p : a.ptr) { bits |= reinterpret_cast<uintptr_t>(p); tensors += p != nullptr; }
    a.vec = (bits & mask) == 0;
    VmBuilder b;
    build_forward(b, prog, ninstr, saved_out);
    return launch_chain(ctx, dtype, b, a, (dtype == FG_DTYPE_F32 ? 4.0 : 2.0) * tensors * n);
}

int32_t fg_eltwise_chain_bwd_dt(fg_ctx* ctx, int32_t dtype, uint64_t n, const fg_ew_instr* prog, int32_t ninstr,
                                const void* const* inputs, int32_t ninputs, const void* seed, void* const* grads,
                                int32_t accumulate) {
    FG_ENTER(ctx);
    int32_t s = check_prog(ctx, prog, ninstr, ninputs);
    if (s != FG_OK) return s;
    FG_REQUIRE(ctx, dtype >= FG_DTYPE_F32 && dtype <= FG_DTYPE_BF16, "fg_eltwise_chain_bwd: unknown dtype");
    FG_REQUIRE(ctx, inputs && seed && grads, "fg_eltwise_chain_bwd: NULL pointer");
    VmArgs a;
    memset(&a, 0, sizeof(a));
    for (int k = 0; k < ninputs; ++k) {
        FG_REQUIRE(ctx, inputs[k] != nullptr, "fg_eltwise_chain_bwd: NULL input");
        a.ptr[k] = const_cast<void*>(inputs[k]);
        a.ptr[kPtrSaved + k] = grads[k];
    }
    a.ptr[kPtrOut] = const_cast<void*>(seed);
    a.n = n;
    if (n == 0) return FG_OK;
    const uintptr_t mask = dtype == FG_DTYPE_F32 ? 15u : 7u;
    uintptr_t bits = 0;
    for (void* p : a.ptr) bits |= reinterpret_cast<uintptr_t>(p);
    a.vec = (bits & mask) == 0;
    int tensors = ninputs + 1;
    for (int k = 0; k < ninputs; ++k) tensors += grads[k] ? 1 + (accumulate != 0) : 0;
    VmBuilder b;
    build_backward(b, prog, ninstr, ninputs, grads, accumulate != 0);
    return launch_chain(ctx, dtype, b, a, (dtype == FG_DTYPE_F32 ? 4.0 : 2.0) * tensors * n);
}

int32_t fg_eltwise_chain_fwd(fg_ctx* ctx, uint64_t n, const fg_ew_instr* prog, int32_t ninstr,
                             const float* const* inputs, int32_t ninputs, float* out, float* const* saved_out) {
    return fg_eltwise_chain_fwd_dt(ctx, FG_DTYPE_F32, n, prog, ninstr, reinterpret_cast<const void* const*>(inputs), ninputs,
                                   out, reinterpret_cast<void* const*>(saved_out));
}

int32_t fg_eltwise_chain_bwd(fg_ctx* ctx, uint64_t n, const fg_ew_instr* prog, int32_t ninstr,
                             const float* const* inputs, int32_t ninputs, const float* seed, float* const* grads,
                             int32_t accumulate) {
    return fg_eltwise_chain_bwd_dt(ctx, FG_DTYPE_F32, n, prog, ninstr, reinterpret_cast<const void* const*>(inputs), ninputs,
                                   seed, reinterpret_cast<void* const*>(grads), accumulate);
}

int32_t fg_convert(fg_ctx* ctx, const void* src, int32_t src_dtype, void* dst, int32_t dst_dtype, uint64_t n) {
    FG_ENTER(ctx);
    return fg_convert_launch(ctx, src, src_dtype, dst, dst_dtype, n);
}

}  // extern "C"

int32_t fg_convert_launch(fg_ctx* ctx, const void* src, int src_dtype, void* dst, int dst_dtype, uint64_t n) {
    FG_REQUIRE(ctx, src && dst, "fg_convert: NULL pointer");
    FG_REQUIRE(ctx, src_dtype >= FG_DTYPE_F32 && src_dtype <= FG_DTYPE_BF16 && dst_dtype >= FG_DTYPE_F32 &&
                        dst_dtype <= FG_DTYPE_BF16, "fg_convert: unknown dtype");
    if (n == 0) return FG_OK;
    const int vec = (reinterpret_cast<uintptr_t>(src) & (src_dtype == FG_DTYPE_F32 ? 15u : 7u)) == 0 &&
                    (reinterpret_cast<uintptr_t>(dst) & (dst_dtype == FG_DTYPE_F32 ? 15u : 7u)) == 0;
    const int grid = fg_stream_grid(ctx, vec ? (n + 3) / 4 : n, 256, 8);
    fg_time_rec* tr = fg_time_begin(ctx, FG_KERNEL_ELTWISE, ((src_dtype == FG_DTYPE_F32 ? 4.0 : 2.0) + (dst_dtype == FG_DTYPE_F32 ? 4.0 : 2.0)) * n);
#define FG_CONV(S, D) if (src_dtype == S && dst_dtype == D) convert_kernel<S, D><<<grid, 256, 0, ctx->stream>>>(src, dst, n, vec)
    FG_CONV(FG_DTYPE_F32, FG_DTYPE_F32); FG_CONV(FG_DTYPE_F32, FG_DTYPE_F16); FG_CONV(FG_DTYPE_F32, FG_DTYPE_BF16);
    FG_CONV(FG_DTYPE_F16, FG_DTYPE_F32); FG_CONV(FG_DTYPE_F16, FG_DTYPE_F16); FG_CONV(FG_DTYPE_F16, FG_DTYPE_BF16);
    FG_CONV(FG_DTYPE_BF16, FG_DTYPE_F32); FG_CONV(FG_DTYPE_BF16, FG_DTYPE_F16); FG_CONV(FG_DTYPE_BF16, FG_DTYPE_BF16);
#undef FG_CONV
    fg_time_end(ctx, tr);
    FG_LAUNCHED(ctx);
    return FG_OK;
}

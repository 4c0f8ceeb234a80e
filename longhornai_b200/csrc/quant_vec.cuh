// Vector forms of the storage-format passes: four columns a thread, 128 x 128 elements a CTA, every load of a
// thread in flight before the first is used.  They give the same bits as the scalar kernels beside them, which
// serve the sizes and alignments these do not take (vec_ok).
//
// What bounds them: memory, once division and rounding cost few enough instructions.  IEEE division (a branch and
// about ten operations) and a saturating rounding per weight, in two passes of single loads, kept int4 quantisation of
// 4096 x 14336 weights at 200 us; one pass with the division below (one multiplication except within 1e-4 of a
// rounding boundary) takes 72 us, 3.7 TB/s.  Floor at the copy rate: 41 us.
#pragma once
#include "common.cuh"

namespace lhb {

constexpr int QV_THREADS = 256, QV_COLS = 128, QV_ROWS = 128, QV_WARP_ROWS = 16;

// columns a multiple of 4, fp32 side 16-byte aligned, coded side 4-byte aligned, row blocks within grid.y
static inline bool vec_ok(const void* f32, const void* codes, int64_t rows, int64_t cols) {
    return (cols & 3) == 0 && (reinterpret_cast<uintptr_t>(f32) & 15) == 0 && (reinterpret_cast<uintptr_t>(codes) & 3) == 0 &&
           (rows + QV_ROWS - 1) / QV_ROWS <= 65535;
}
static inline dim3 vec_grid(int64_t rows, int64_t cols) {
    return dim3(static_cast<unsigned>((cols + QV_COLS - 1) / QV_COLS), static_cast<unsigned>((rows + QV_ROWS - 1) / QV_ROWS));
}

constexpr float QV_MAGIC = 12582912.0f;                     // 1.5 * 2^23: adding it rounds to an integer, half to even

// rint(x / s), s from the magnitudes of its own column or group (|x / s| below 2^8).  `inv` = 1 / s: x * inv is within
// 2^-14 of the IEEE quotient, so further than 1e-4 from a rounding boundary both round alike.  NaN, infinities and
// scales without a finite inverse fail the comparison and take the division.
__device__ __forceinline__ bool quick_rint(float x, float inv, int& q) {
    const float t = __fmul_rn(x, inv), m = __fadd_rn(t, QV_MAGIC);
    q = __float_as_int(m) - 0x4B400000;
    return fabsf(__fsub_rn(t, __fsub_rn(m, QV_MAGIC))) < 0.4999f;
}
__device__ __forceinline__ int div_code(float x, float s, float inv, int lim) {
    int q;
    return quick_rint(x, inv, q) ? q : sat_rne(__fdiv_rn(x, s), lim);
}
__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}
__device__ __forceinline__ float4 abs_max4(float4 m, float4 v) {
    return make_float4(fmaxf(m.x, fabsf(v.x)), fmaxf(m.y, fabsf(v.y)), fmaxf(m.z, fabsf(v.z)), fmaxf(m.w, fabsf(v.w)));
}
__device__ __forceinline__ float max4(float4 v) { return fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)); }

// ---- codecs: four values <-> four codes ------------------------------------------------------------

struct CodecQ8 {
    static constexpr float QMAX = 127.0f;
    // reciprocal multiply: q = sat(x * inv); the clamp takes a NaN to -127 as sat_rne does
    static __device__ __forceinline__ uint32_t mul(float4 v, float inv) {
        auto one = [&](float x) { return __float_as_int(__fadd_rn(fminf(fmaxf(__fmul_rn(x, inv), -127.0f), 127.0f), QV_MAGIC)); };
        return pack4(one(v.x), one(v.y), one(v.z), one(v.w));
    }
    static __device__ __forceinline__ uint32_t div(float4 v, float4 s, float4 inv) {
        return pack4(div_code(v.x, s.x, inv.x, 127), div_code(v.y, s.y, inv.y, 127), div_code(v.z, s.z, inv.z, 127),
                     div_code(v.w, s.w, inv.w, 127));
    }
    static __device__ __forceinline__ float4 decode(uint32_t w) {
        auto one = [&](int sh) { return static_cast<float>(static_cast<int8_t>(w >> sh)); };
        return make_float4(one(0), one(8), one(16), one(24));
    }
};

// ---- max|x| ------------------------------------------------------------------------------------------

// of everything (n4 float4s), merged with atomicMax on the bits of `out`
static __global__ void __launch_bounds__(QV_THREADS)
vec_absmax_kernel(const float4* __restrict__ src, unsigned* __restrict__ out, int64_t n4) {
    float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
    const int64_t step = static_cast<int64_t>(gridDim.x) * QV_THREADS;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(QV_THREADS) + threadIdx.x; i < n4; i += 4 * step) {
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = i + j * step < n4 ? __ldg(src + i + j * step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; ++j) m = abs_max4(m, v[j]);
    }
    __shared__ float red[QV_THREADS / 32];
    const float w = warp_max(max4(m));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = red[0];
        for (int i = 1; i < QV_THREADS / 32; ++i) b = fmaxf(b, red[i]);
        if (b > 0.0f) atomicMax(out, __float_as_uint(b));   // one per CTA
    }
}

// of every column
static __global__ void __launch_bounds__(QV_THREADS)
vec_col_absmax_kernel(const float* __restrict__ src, unsigned* __restrict__ colmax, int rows, int cols) {
    __shared__ float4 red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * QV_COLS + 4 * lane, r0 = blockIdx.y * QV_ROWS + warp * QV_WARP_ROWS;
    float4 v[QV_WARP_ROWS], m = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < QV_WARP_ROWS; ++i)
        v[i] = c < cols && r0 + i < rows ? __ldg(reinterpret_cast<const float4*>(src + static_cast<int64_t>(r0 + i) * cols + c))
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < QV_WARP_ROWS; ++i) m = abs_max4(m, v[i]);
    red[warp][lane] = m;
    __syncthreads();
    if (threadIdx.x < QV_COLS && blockIdx.x * QV_COLS + threadIdx.x < cols) {
        float b = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) b = fmaxf(b, reinterpret_cast<const float*>(red[w])[threadIdx.x]);
        if (b > 0.0f) atomicMax(colmax + blockIdx.x * QV_COLS + threadIdx.x, __float_as_uint(b));
    }
}

// ---- quantise --------------------------------------------------------------------------------------------

template <class Codec>
static __global__ void __launch_bounds__(QV_THREADS)
vec_quantize_tensor_kernel(const float4* __restrict__ src, uint32_t* __restrict__ dst, const float* __restrict__ scale, int64_t n4) {
    const float inv = __fdiv_rn(1.0f, *scale);
    const int64_t step = static_cast<int64_t>(gridDim.x) * QV_THREADS;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(QV_THREADS) + threadIdx.x; i < n4; i += 4 * step) {
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = i + j * step < n4 ? __ldg(src + i + j * step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i + j * step < n4) dst[i + j * step] = Codec::mul(v[j], inv);
    }
}

template <class Codec>
static __global__ void __launch_bounds__(QV_THREADS)
vec_quantize_cols_kernel(const float* __restrict__ src, uint8_t* __restrict__ dst, const float* __restrict__ scales, int rows, int cols) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * QV_COLS + 4 * lane, r0 = blockIdx.y * QV_ROWS + warp * QV_WARP_ROWS;
    if (c >= cols) return;
    const float4 s = make_float4(scales[c], scales[c + 1], scales[c + 2], scales[c + 3]);
    const float4 inv = make_float4(__fdiv_rn(1.0f, s.x), __fdiv_rn(1.0f, s.y), __fdiv_rn(1.0f, s.z), __fdiv_rn(1.0f, s.w));
#pragma unroll
    for (int h = 0; h < QV_WARP_ROWS; h += 8) {
        float4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = r0 + h + i < rows ? __ldg(reinterpret_cast<const float4*>(src + static_cast<int64_t>(r0 + h + i) * cols + c))
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (r0 + h + i < rows) *reinterpret_cast<uint32_t*>(dst + static_cast<int64_t>(r0 + h + i) * cols + c) = Codec::div(v[i], s, inv);
    }
}

// one CTA per row; rows of up to 8192 stay in registers between the two passes
template <class Codec>
static __global__ void __launch_bounds__(QV_THREADS)
vec_quantize_rows_kernel(const float* __restrict__ src, uint8_t* __restrict__ dst, float* __restrict__ scales, int dim) {
    __shared__ float red[QV_THREADS / 32];
    const float4* x = reinterpret_cast<const float4*>(src + static_cast<int64_t>(blockIdx.x) * dim);
    uint32_t* q = reinterpret_cast<uint32_t*>(dst + static_cast<int64_t>(blockIdx.x) * dim);
    const int n4 = dim >> 2;
    constexpr int KEEP = 8;
    float4 v[KEEP], m = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < KEEP; ++j) {
        const int i = threadIdx.x + j * QV_THREADS;
        v[j] = i < n4 ? __ldg(x + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < KEEP; ++j) m = abs_max4(m, v[j]);
    for (int i = threadIdx.x + KEEP * QV_THREADS; i < n4; i += QV_THREADS) m = abs_max4(m, __ldg(x + i));
    const float w = warp_max(max4(m));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = w;
    __syncthreads();
    float b = red[0];
#pragma unroll
    for (int i = 1; i < QV_THREADS / 32; ++i) b = fmaxf(b, red[i]);
    const float scale = (b > 0.0f) ? __fdiv_rn(b, Codec::QMAX) : 1.0f;
    const float inv = __fdiv_rn(1.0f, scale);
#pragma unroll
    for (int j = 0; j < KEEP; ++j) {
        const int i = threadIdx.x + j * QV_THREADS;
        if (i < n4) q[i] = Codec::mul(v[j], inv);
    }
    for (int i = threadIdx.x + KEEP * QV_THREADS; i < n4; i += QV_THREADS) q[i] = Codec::mul(__ldg(x + i), inv);
    if (threadIdx.x == 0) scales[blockIdx.x] = scale;
}

// ---- dequantise --------------------------------------------------------------------------------------------

// mode 0: scales[0] (or `one` where scales is null); 1: scales[row]; 2: scales[column]
template <class Codec>
static __global__ void __launch_bounds__(QV_THREADS)
vec_dequantize_kernel(const uint8_t* __restrict__ src, const float* __restrict__ scales, float one, float* __restrict__ dst, int rows,
                      int cols, int mode) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * QV_COLS + 4 * lane, r0 = blockIdx.y * QV_ROWS + warp * QV_WARP_ROWS;
    if (c >= cols) return;
    uint32_t w[QV_WARP_ROWS];
#pragma unroll
    for (int i = 0; i < QV_WARP_ROWS; ++i)
        w[i] = r0 + i < rows ? __ldg(reinterpret_cast<const uint32_t*>(src + static_cast<int64_t>(r0 + i) * cols + c)) : 0u;
    const float s0 = mode == 0 && scales ? scales[0] : one;
    const float4 s = mode == 2 ? make_float4(scales[c], scales[c + 1], scales[c + 2], scales[c + 3]) : make_float4(s0, s0, s0, s0);
#pragma unroll
    for (int i = 0; i < QV_WARP_ROWS; ++i) {
        if (r0 + i >= rows) break;
        const float4 x = Codec::decode(w[i]);
        const float sr = mode == 1 ? scales[r0 + i] : 0.0f;
        const float4 f = mode == 1 ? make_float4(sr, sr, sr, sr) : s;
        *reinterpret_cast<float4*>(dst + static_cast<int64_t>(r0 + i) * cols + c) =
            make_float4(__fmul_rn(x.x, f.x), __fmul_rn(x.y, f.y), __fmul_rn(x.z, f.z), __fmul_rn(x.w, f.w));
    }
}

}  // namespace lhb

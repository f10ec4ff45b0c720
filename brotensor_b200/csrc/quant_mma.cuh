// Pieces shared by the kernels that multiply raw quants on the warp-level tensor-core instructions (gemv_mb.cu: one to eight
// activation rows on integer MMA; gemm_mm.cu: a few dozen on FP16 MMA): how a 256-element piece of a weight row lies in
// shared memory, asynchronous 16-byte copies, activations as floats, and the plain FP32 loop for rows that they leave to it.
#pragma once

#include "common.cuh"

namespace b200q {

constexpr int kQmTile = 16;  // weight rows of an MMA

// A 256-element piece of a weight row in shared memory. `pair8`: a thread t of a quad multiplies elements 8t .. 8t+7 of a
// sub-block of 32, else 4t .. 4t+3 and 16+4t .. 16+4t+3. `stages`: ring depth of a warp in gemv_mb.cu.
template <int FMT>
struct QmFmt;
template <>
struct QmFmt<kQ4_K> {
    // stride = 32 (mod 128): the 8-byte loads of four neighbouring rows fall into different banks
    static constexpr int bytes = 144, chunks = 9, stride = 160, stages = 5;
    static constexpr bool pair8 = true, mins = true;
};
template <>
struct QmFmt<kQ5_K> {
    static constexpr int bytes = 176, chunks = 11, stride = 224, stages = 3;  // 96 (mod 128): likewise
    static constexpr bool pair8 = true, mins = true;
};
template <>
struct QmFmt<kQ8_0> {
    // stride = 16 (mod 128): the 4-byte loads of eight rows fall into different banks
    static constexpr int bytes = 272, chunks = 17, stride = 272, stages = 3;
    static constexpr bool pair8 = false, mins = false;
};
template <>
struct QmFmt<kQ4_0> {
    static constexpr int bytes = 144, chunks = 9, stride = 144, stages = 5;
    static constexpr bool pair8 = false, mins = false;
};
template <>
struct QmFmt<kQ6_K> {
    // 210 bytes from any even address: fourteen 16-byte chunks from the boundary before it
    static constexpr int bytes = 210, chunks = 14, stride = 240, stages = 3;
    static constexpr bool pair8 = false, mins = false;
};

// A row's block in shared memory. Q6_K blocks start on any even byte behind their 16-byte boundary: p is the aligned
// word that holds the first byte and sh the bits to shift it out by (0 or 16).
struct QmRow {
    const uint8_t* p;
    uint32_t sh;
};
template <int FMT>
__device__ __forceinline__ QmRow qm_row(const uint8_t* slot, const uint8_t* global) {
    if constexpr (FMT == kQ6_K) {
        const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(global) & 15u);
        return {slot + (off & 12u), (off & 2u) * 8u};
    } else {
        return {slot, 0u};
    }
}

__device__ __forceinline__ uint32_t ls16(const uint8_t* p) { return *reinterpret_cast<const unsigned short*>(p); }
__device__ __forceinline__ uint32_t ls32(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ uint2 ls64(const uint8_t* p) { return *reinterpret_cast<const uint2*>(p); }
__device__ __forceinline__ uint4 ls128(const uint8_t* p) { return *reinterpret_cast<const uint4*>(p); }
// 4 bytes at offset o (a multiple of 4) of a Q6_K block
__device__ __forceinline__ uint32_t qm_word(const QmRow& r, int o) { return __funnelshift_r(ls32(r.p + o), ls32(r.p + o + 4), r.sh); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The 16-byte chunks lt, lt + 4, ... of a row's block (four threads per row).
template <int FMT>
__device__ __forceinline__ void qm_copy_row(uint32_t dst, const uint8_t* src, int lt) {
    using F = QmFmt<FMT>;
    if constexpr (FMT == kQ6_K) src = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(src) & ~uintptr_t(15));
    src += 16 * lt;
    dst += 16u * lt;
#pragma unroll
    for (int c = 0; c < F::chunks; c += 4)
        if (c + 4 <= F::chunks || c + lt < F::chunks) cp_async16(dst + 16u * c, src + 16 * c);
}

// byte `idx` (0..3) of a word: as an integer, and as an exact float
__device__ __forceinline__ uint32_t byte_at(uint32_t w, int idx) { return __byte_perm(w, 0u, 0x4440u | idx); }
__device__ __forceinline__ float byte_to_f32(uint32_t w, uint32_t idx) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | idx)) - 8388608.0f;
}
// the 6-bit scales / mins of a Q4_K or Q5_K header, one per byte: sub-blocks 0..3 and 4..7
__device__ __forceinline__ uint32_t k_scales_lo(const uint4& h) { return h.y & 0x3f3f3f3fu; }
__device__ __forceinline__ uint32_t k_scales_hi(const uint4& h) { return (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u); }
__device__ __forceinline__ uint32_t k_mins_lo(const uint4& h) { return h.z & 0x3f3f3f3fu; }
__device__ __forceinline__ uint32_t k_mins_hi(const uint4& h) { return ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u); }

// D = A * B (+ D), 16 x 8 x 16, FP16 or BF16 operands and FP32 sums.
template <bool BF>
__device__ __forceinline__ void qm_mma_zero(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (BF)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
template <bool BF>
__device__ __forceinline__ void qm_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (BF)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Eight activations of row m from element k on: raw (the second word for FP32 only), and as floats.
__device__ __forceinline__ void qm_load_raw(const void* X, bool f32, int K, int m, int k, uint4 (&r)[2]) {
    const uint8_t* x = static_cast<const uint8_t*>(X) + ((size_t)m * K + k) * (f32 ? 4 : 2);
    r[0] = ld_dep_u4(x);
    if (f32) r[1] = ld_dep_u4(x + 16);
}
__device__ __forceinline__ void qm_to_f32(const uint4 (&r)[2], int x_dtype, float (&v)[8]) {
    const uint32_t w[8] = {r[0].x, r[0].y, r[0].z, r[0].w, r[1].x, r[1].y, r[1].z, r[1].w};
    if (x_dtype == B200Q_DT_F32) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(w[i]);
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (x_dtype == B200Q_DT_F16) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
            v[2 * i] = f.x;
            v[2 * i + 1] = f.y;
        } else {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
        }
    }
}
// Whether the bulk of some sub-block of 32 activations (f * s, eight per thread, four neighbouring threads) is lost in the error of its
// representation: `err2` is the thread's sum of squared errors, each times kErrUp (squares of what is left of activations 2^90 below the
// largest are subnormal). At least half of the elements that are not zero must stand 2^21 above the sub-block's root mean square
// of the error - so weights that are small in a few large channels leave a result with the accuracy of FP32 products (3e-7),
// whatever those channels hold. The answer is the warp's.
constexpr float kErrUp = 1073741824.0f;  // 2^30
__device__ __forceinline__ bool qm_sub_block_lost(const float (&f)[8], float s, float err2) {
    err2 += __shfl_xor_sync(0xffffffffu, err2, 1);
    err2 += __shfl_xor_sync(0xffffffffu, err2, 2);
    const float limit = err2 * 137438953472.0f;  // 2^42 / 32
    int count = 0;                               // elements below the limit, less those above
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float v = f[k] * s * kErrUp;
        count += f[k] == 0.f ? 0 : v * v <= limit ? 1 : -1;
    }
    count += __shfl_xor_sync(0xffffffffu, count, 1);
    count += __shfl_xor_sync(0xffffffffu, count, 2);
    return __any_sync(0xffffffffu, count > 0);
}
__device__ __forceinline__ float qm_bias(const void* bias, int dtype, int n) {
    if (!bias) return 0.f;
    if (dtype == B200Q_DT_F32) return static_cast<const float*>(bias)[n];
    if (dtype == B200Q_DT_F16) return __half2float(static_cast<const __half*>(bias)[n]);
    return __bfloat162float(static_cast<const __nv_bfloat16*>(bias)[n]);
}
__device__ __forceinline__ void qm_store(void* Y, int dtype, size_t at, float v) {
    if (dtype == B200Q_DT_F32) static_cast<float*>(Y)[at] = v;
    else if (dtype == B200Q_DT_F16) static_cast<__half*>(Y)[at] = __float2half_rn(v);
    else static_cast<__nv_bfloat16*>(Y)[at] = __float2bfloat16_rn(v);
}

// Y of weight rows [row_begin, row_begin + n_rows) and the activation rows m0 + i of the bits i of `rows`, in FP32 from memory, a
// warp per weight row: for activations that are not finite, where a result is what IEEE arithmetic makes of infinities and NaN, and for
// ones whose range the fixed-point forms do not hold.
template <int FMT>
__device__ __noinline__ void qm_plain_rows(const uint8_t* W, const void* X, int x_dtype, const void* bias, void* Y, int y_dtype, int m0, uint32_t rows,
                                              int N, int K, int row_bytes, int row_begin, int n_rows) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int r = warp; r < n_rows; r += nw) {
        const int n = row_begin + r;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int u = lane; u < (K >> 3); u += 32) {
            float w[8];
            decode8<FMT, LdDep>(W + (size_t)n * row_bytes, u, w);
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (rows >> i & 1u) {
                    float v[8];
                    uint4 raw[2];
                    qm_load_raw(X, x_dtype == B200Q_DT_F32, K, m0 + i, 8 * u, raw);
                    qm_to_f32(raw, x_dtype, v);
#pragma unroll
                    for (int k = 0; k < 8; ++k) acc[i] = fmaf(w[k], v[k], acc[i]);
                }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (rows >> i & 1u) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
                if (lane == 0) qm_store(Y, y_dtype, (size_t)(m0 + i) * N + n, acc[i] + qm_bias(bias, x_dtype, n));
            }
    }
}

}  // namespace b200q

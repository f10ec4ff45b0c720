// Block decode kernels: quantized rows -> FP16 / BF16 / FP32.
//
// One thread decodes eight consecutive elements (one 16-byte FP16 store), so a
// warp writes 512 contiguous bytes; the grid is a flat 1-D sweep over all
// eight-element groups, which has no 65535-row limit. Behaviour follows
// brotensor's dequant_q4k_to_fp16 (src/cuda/q4k.cu:53-96, 297-324),
// dequant_q6k_to_fp16 (q6k.cu:46-76) and dequant_q8_0_to_fp16 (q8_0.cu:40-54):
// FP32 decode, then round-to-nearest-even to the output type.
#include "common.cuh"

namespace b200q {

template <int FMT, typename OT>
__global__ void __launch_bounds__(256) dequant_kernel(const uint8_t* __restrict__ W, OT* __restrict__ out,
                                                      long long total_units, int units_per_row, int row_bytes) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x; id < total_units; id += stride) {
        const long long r = id / units_per_row;
        const int u = (int)(id - r * units_per_row);
        float w[8];
        decode8<FMT>(W + (size_t)r * row_bytes, u, w);
        OT* o = out + (size_t)id * 8;
        if constexpr (sizeof(OT) == 2) {
            union {
                OT h[8];
                uint4 v;
            } pk;
#pragma unroll
            for (int k = 0; k < 8; ++k) pk.h[k] = from_f32<OT>(w[k]);
            *reinterpret_cast<uint4*>(o) = pk.v;
        } else {
            reinterpret_cast<float4*>(o)[0] = make_float4(w[0], w[1], w[2], w[3]);
            reinterpret_cast<float4*>(o)[1] = make_float4(w[4], w[5], w[6], w[7]);
        }
    }
}

// Eight values, rounded once to the output type, to consecutive positions.
template <typename OT>
__device__ __forceinline__ void dq_store8(OT* o, const float (&f)[8]) {
    union {
        OT h[8];
        uint4 v;
    } pk;
#pragma unroll
    for (int k = 0; k < 8; ++k) pk.h[k] = from_f32<OT>(f[k]);
    *reinterpret_cast<uint4*>(o) = pk.v;
}

// Q4_K and Q5_K, one thread per eight positions of two neighbouring 64-element groups: the block header (one
// 16-byte load, shared through L1 by the block's eight threads), 8 quant bytes of each group (Q5_K: and
// its 8 bytes of fifth bits), and 32 values - eight consecutive ones in each of four sub-blocks - so four
// runs of stores, with neighbouring threads writing neighbouring pieces. The four sub-blocks' 6-bit scales
// and mins are unpacked four at a time. The value is the same exact FP32 number as the generic
// path's (d * sc * q and dmin * m are exact, one fused rounding), rounded once to the output type. Needs 16-byte
// aligned rows. (One thread per sub-block with 64 contiguous output bytes per thread: 11.1 us for
// 4096 x 4096 Q4_K -> FP16 against 7.4.)
template <int FMT, typename OT>
__global__ void __launch_bounds__(256) dequant_k_kernel(const uint8_t* W, OT* out, long long total_units, int units_per_row, int row_bytes, int K) {
    constexpr int kBytes = FMT == kQ4_K ? 144 : 176, kQs = FMT == kQ4_K ? 16 : 48;
    grid_dep_launch();
    grid_dep_wait();
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x; id < total_units; id += stride) {
        const long long r = id / units_per_row;
        const int u = (int)(id - r * units_per_row);  // eight units per block
        const int b = u >> 3, jp = (u >> 2) & 1, p = u & 3;
        const uint8_t* blk = W + (size_t)r * row_bytes + (size_t)b * kBytes;
        const uint4 h = ld_dep_u4(blk);
        const uint2 g0 = ld_dep_u2(blk + kQs + 64 * jp + 8 * p);
        const uint2 g1 = ld_dep_u2(blk + kQs + 32 + 64 * jp + 8 * p);
        uint2 fifth = make_uint2(0, 0);
        if constexpr (FMT == kQ5_K) fifth = ld_dep_u2(blk + 16 + 8 * p);
        // scales / mins of sub-blocks 4 jp .. 4 jp + 3, one per byte
        const uint32_t scw = jp ? ((h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u)) : (h.y & 0x3f3f3f3fu);
        const uint32_t mw = jp ? (((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u)) : (h.z & 0x3f3f3f3fu);
        const float d = h2f(h.x & 0xFFFFu), dmin = h2f(h.x >> 16);
        OT* o = out + (size_t)r * K + (size_t)b * 256 + 128 * jp + 8 * p;
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // sub-block 4 jp + q: low (q even) or high (q odd) nibbles of group 2 jp + q / 2
            const float ds = d * (float)((scw >> (8 * q)) & 0xFFu), dm = dmin * (float)((mw >> (8 * q)) & 0xFFu);
            const uint2 g = q < 2 ? g0 : g1;
            const uint32_t w[2] = {g.x, g.y}, hb[2] = {fifth.x, fifth.y};
            float f[8];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t v = ((q & 1) ? (w[k] >> 4) : w[k]) & 0x0F0F0F0Fu;
                if constexpr (FMT == kQ5_K) v |= ((hb[k] >> (4 * jp + q)) & 0x01010101u) << 4;
#pragma unroll
                for (int i = 0; i < 4; ++i) f[4 * k + i] = fmaf(ds, __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440 | i)) - 8388608.0f, -dm);
            }
            dq_store8<OT>(o + 32 * q, f);
        }
    }
}

// Q6_K, one thread per eight positions l0..l0+7 of one 128-element half block: its 8 low-nibble
// bytes for the quarters 0/2 and 1/3 and its 8 high-bit bytes give 32 values - eight consecutive ones in
// each of the half's four 32-element quarters - so four runs of stores, and the loads and the scale
// work of the generic path are shared by four times as many outputs. Blocks are 2-byte aligned only;
// all loads are 16-bit pairs. d * sc * (q - 32) is exact in FP32 (11 + 7 + 6 bits), one rounding to the output type.
template <bool RUNS, typename OT>  // RUNS: the layout regrouped by field in runs of eight blocks (16-byte aligned fields)
__global__ void __launch_bounds__(256) dequant_q6k_kernel(const uint8_t* W, OT* out, long long total_units, int units_per_row, int row_bytes, int K) {
    grid_dep_launch();
    grid_dep_wait();
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x; id < total_units; id += stride) {
        const long long r = id / units_per_row;
        const int u = (int)(id - r * units_per_row);  // eight units per block
        const int b = u >> 3, n = (u >> 2) & 1, l0 = (u & 3) * 8;
        uint32_t a[2][2], h[2], sc[4];  // sc: scale (l0 >> 4) + 2 q of the half's eight, for quarter q
        float d;
        if constexpr (RUNS) {
            const uint8_t* run = W + (size_t)r * row_bytes + (size_t)(b >> 3) * kQ6RunBytes;
            const int s = b & 7;
            const uint2 a0 = ld_dep_u2(run + s * 128 + n * 64 + l0);
            const uint2 a1 = ld_dep_u2(run + s * 128 + n * 64 + 32 + l0);
            const uint2 hh = ld_dep_u2(run + 1024 + s * 64 + n * 32 + l0);
            a[0][0] = a0.x; a[0][1] = a0.y; a[1][0] = a1.x; a[1][1] = a1.y;
            h[0] = hh.x; h[1] = hh.y;
            const uint2 sw = ld_dep_u2(run + 1536 + s * 16 + n * 8);
            const uint32_t sh = 8 * (l0 >> 4);
            sc[0] = sw.x >> sh; sc[1] = sw.x >> (16 + sh); sc[2] = sw.y >> sh; sc[3] = sw.y >> (16 + sh);
            d = h2f(ld_dep_u16(run + 1664 + 2 * s));
        } else {
            const uint8_t* blk = W + (size_t)r * row_bytes + (size_t)b * 210;
            const uint8_t* ql = blk + n * 64 + l0;
            const uint8_t* qh = blk + 128 + n * 32 + l0;
            a[0][0] = ld_u32_a2<LdDep>(ql); a[0][1] = ld_u32_a2<LdDep>(ql + 4);
            a[1][0] = ld_u32_a2<LdDep>(ql + 32); a[1][1] = ld_u32_a2<LdDep>(ql + 36);
            h[0] = ld_u32_a2<LdDep>(qh); h[1] = ld_u32_a2<LdDep>(qh + 4);
#pragma unroll
            for (int q = 0; q < 4; ++q) sc[q] = ld_dep_u16(blk + 192 + n * 8 + 2 * q) >> (8 * (l0 >> 4));
            d = h2f(ld_dep_u16(blk + 208));
        }
        OT* o = out + (size_t)r * K + (size_t)b * 256 + n * 128 + l0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float ds = d * (float)(int)(signed char)(sc[q] & 0xFFu);
            float f[8];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const uint32_t nib = (q < 2 ? a[q & 1][w] : (a[q & 1][w] >> 4)) & 0x0F0F0F0Fu;
                const uint32_t hb = ((h[w] >> (2 * q)) & 0x03030303u) << 4;
                const uint32_t six = nib | hb;  // four 6-bit values, one per byte
#pragma unroll
                for (int i = 0; i < 4; ++i) f[4 * w + i] = ds * (__uint_as_float(__byte_perm(six, 0x4B000000u, 0x7440 | i)) - 8388640.0f);  // byte - 32
            }
            dq_store8<OT>(o + 32 * q, f);
        }
    }
}

// Q8_0 and Q4_0, 32 values per thread as well: of Q8_0 eight consecutive ones in each of four neighbouring blocks, of Q4_0 eight
// bytes - a half block's low nibbles and the high ones sixteen positions on - in each of two. Blocks are 34 and 18 bytes, so every
// other one has its quants on a word boundary and the ones between two bytes behind one (a funnel shift). Needs rows of whole
// groups (K a multiple of 128 / 64) on a 4-byte boundary. d * q is exact in FP32, one rounding to the output type.
template <int FMT, typename OT>
__global__ void __launch_bounds__(256) dequant_32_kernel(const uint8_t* W, OT* out, long long total_units, int units_per_row, int row_bytes, int K) {
    constexpr int kBlock = FMT == kQ8_0 ? 34 : 18, kBlocks = FMT == kQ8_0 ? 4 : 2, kParts = FMT == kQ8_0 ? 4 : 2;
    grid_dep_launch();
    grid_dep_wait();
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x; id < total_units; id += stride) {
        const long long r = id / units_per_row;
        const int u = (int)(id - r * units_per_row), group = u / kParts, p = u % kParts;
        const uint8_t* g = W + (size_t)r * row_bytes + (size_t)group * (kBlocks * kBlock);
        uint32_t q[kBlocks][2];
        float d[kBlocks];
#pragma unroll
        for (int j = 0; j < kBlocks; ++j) {
            const uint8_t* b = g + kBlock * j + 8 * p;
            d[j] = h2f(ld_dep_u16(g + kBlock * j));
            if (j & 1) {
                q[j][0] = ld_dep_u32(b + 2);
                q[j][1] = ld_dep_u32(b + 6);
            } else {
                const uint32_t w0 = ld_dep_u32(b), w1 = ld_dep_u32(b + 4), w2 = ld_dep_u32(b + 8);
                q[j][0] = __funnelshift_r(w0, w1, 16);
                q[j][1] = __funnelshift_r(w1, w2, 16);
            }
        }
        OT* o = out + (size_t)r * K + (size_t)group * (32 * kBlocks) + 8 * p;
#pragma unroll
        for (int j = 0; j < kBlocks; ++j) {
#pragma unroll
            for (int h = 0; h < (FMT == kQ8_0 ? 1 : 2); ++h) {
                float f[8];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    // byte + 128 / nibble, as 2^23 + value
                    const uint32_t v = FMT == kQ8_0 ? q[j][k] ^ 0x80808080u : (q[j][k] >> (4 * h)) & 0x0F0F0F0Fu;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        f[4 * k + i] = d[j] * (__uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440 | i)) - (FMT == kQ8_0 ? 8388736.0f : 8388616.0f));
                }
                dq_store8<OT>(o + 32 * j + 16 * h, f);
            }
        }
    }
}

// The wide kernels' launch: 32 values per thread.
template <typename OT>
static int launch_dequant_wide(void (*kern)(const uint8_t*, OT*, long long, int, int, int), const uint8_t* W, void* out, int64_t rows, int K, int row_bytes,
                               long long cap, cudaStream_t st) {
    const long long units = (long long)rows * (K / 32);
    long long nb = (units + 255) / 256;
    if (nb > cap) nb = cap;
    B200Q_CUDA_TRY(launch_dep(pdl_option() >= 0, kern, dim3((unsigned)nb), dim3(256), 0, st, W, static_cast<OT*>(out), units, K / 32, row_bytes, K));
    return B200Q_OK;
}
template <int FMT, typename OT>
static int launch_dequant_wide_f(const uint8_t* W, void* out, int64_t rows, int K, int row_bytes, long long cap, cudaStream_t st) {
    if constexpr (FMT == kQ4_K || FMT == kQ5_K) return launch_dequant_wide<OT>(dequant_k_kernel<FMT, OT>, W, out, rows, K, row_bytes, cap, st);
    else if constexpr (FMT == kQ8_0 || FMT == kQ4_0) return launch_dequant_wide<OT>(dequant_32_kernel<FMT, OT>, W, out, rows, K, row_bytes, cap, st);
    else return launch_dequant_wide<OT>(dequant_q6k_kernel<FMT == kQ6_KP, OT>, W, out, rows, K, row_bytes, cap, st);
}

template <int FMT>
static int launch_dequant_fmt(const void* W, void* out, int out_dtype, int64_t rows, int K, cudaStream_t st) {
    const int upr = K / 8;
    const long long total = (long long)rows * upr;
    const int row_bytes = (K / Blk<FMT>::elems) * Blk<FMT>::bytes;
    long long blocks = (total + 255) / 256;
    const long long cap = 148LL * 8 * 16;
    if (blocks > cap) blocks = cap;
    const uint8_t* w = static_cast<const uint8_t*>(W);
    if (out_dtype == B200Q_DT_F16 || out_dtype == B200Q_DT_BF16) {
        // The wide kernels: 16-bit outputs. With FP32 a thread's 32-byte pieces lie apart and every store instruction of a warp leaves
        // half sectors; seven matrices of a 4096 / 14336 layer, wide against generic, us: FP16 Q8_0 134 / 163, Q4_0 110 / 165, BF16 Q4_K
        // and Q6_K 104 / 183, but FP32 Q8_0 242 / 223, Q4_0 342 / 212, Q4_K and Q6_K 240 / 234.
        // Q4_K and Q5_K load whole headers, Q8_0 and Q4_0 words of groups of blocks; Q6_K takes any block address.
        const uintptr_t at = reinterpret_cast<uintptr_t>(W);
        if (FMT == kQ6_K || FMT == kQ6_KP || ((FMT == kQ4_K || FMT == kQ5_K) && (at & 15) == 0) ||
            (FMT == kQ8_0 && K % 128 == 0 && (at & 3) == 0) || (FMT == kQ4_0 && K % 64 == 0 && (at & 3) == 0)) {
            if (out_dtype == B200Q_DT_F16) return launch_dequant_wide_f<FMT, __half>(w, out, rows, K, row_bytes, cap, st);
            return launch_dequant_wide_f<FMT, __nv_bfloat16>(w, out, rows, K, row_bytes, cap, st);
        }
    }
    switch (out_dtype) {
        case B200Q_DT_F16:
            dequant_kernel<FMT, __half><<<(unsigned)blocks, 256, 0, st>>>(w, (__half*)out, total, upr, row_bytes);
            break;
        case B200Q_DT_BF16:
            dequant_kernel<FMT, __nv_bfloat16>
                <<<(unsigned)blocks, 256, 0, st>>>(w, (__nv_bfloat16*)out, total, upr, row_bytes);
            break;
        case B200Q_DT_F32:
            dequant_kernel<FMT, float><<<(unsigned)blocks, 256, 0, st>>>(w, (float*)out, total, upr, row_bytes);
            break;
        default:
            return fail(B200Q_ERR_BAD_ARG, "dequant: unknown output dtype %d", out_dtype);
    }
    B200Q_CUDA_TRY(cudaGetLastError());
    return B200Q_OK;
}

int launch_dequant(int fmt, const void* W, void* out, int out_dtype, int64_t rows, int K, cudaStream_t st) {
    switch (fmt) {
        case kQ4_K: return launch_dequant_fmt<kQ4_K>(W, out, out_dtype, rows, K, st);
        case kQ6_K: return launch_dequant_fmt<kQ6_K>(W, out, out_dtype, rows, K, st);
        case kQ6_KP: return launch_dequant_fmt<kQ6_KP>(W, out, out_dtype, rows, K, st);
        case kQ8_0: return launch_dequant_fmt<kQ8_0>(W, out, out_dtype, rows, K, st);
        case kQ4_0: return launch_dequant_fmt<kQ4_0>(W, out, out_dtype, rows, K, st);
        case kQ5_K: return launch_dequant_fmt<kQ5_K>(W, out, out_dtype, rows, K, st);
    }
    return fail(B200Q_ERR_BAD_ARG, "dequant: unknown block format %d", fmt);
}

// Row gather with decode (a quantized embedding table): the dequant kernel with the row taken from
// an index vector. One thread decodes eight consecutive elements of one gathered row; an index
// outside the table writes zeros and reads nothing.
template <int FMT, typename OT>
__global__ void __launch_bounds__(256) gather_kernel(const uint8_t* __restrict__ W, const int32_t* __restrict__ idx, OT* __restrict__ out,
                                                     long long total_units, int units_per_row, int row_bytes, long long rows) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x; id < total_units; id += stride) {
        const long long b = id / units_per_row;
        const int u = (int)(id - b * units_per_row);
        const long long r = (long long)__ldg(idx + b);
        float w[8];
        if (r >= 0 && r < rows) {
            decode8<FMT>(W + (size_t)r * row_bytes, u, w);
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k] = 0.f;
        }
        OT* o = out + (size_t)id * 8;
        if constexpr (sizeof(OT) == 2) {
            union {
                OT h[8];
                uint4 v;
            } pk;
#pragma unroll
            for (int k = 0; k < 8; ++k) pk.h[k] = from_f32<OT>(w[k]);
            *reinterpret_cast<uint4*>(o) = pk.v;
        } else {
            reinterpret_cast<float4*>(o)[0] = make_float4(w[0], w[1], w[2], w[3]);
            reinterpret_cast<float4*>(o)[1] = make_float4(w[4], w[5], w[6], w[7]);
        }
    }
}

template <int FMT>
static int launch_gather_fmt(const void* W, const int32_t* idx, void* out, int out_dtype, int B, int64_t rows, int K, cudaStream_t st) {
    const int upr = K / 8;
    const long long total = (long long)B * upr;
    const int row_bytes = (K / Blk<FMT>::elems) * Blk<FMT>::bytes;
    long long blocks = (total + 255) / 256;
    const long long cap = 148LL * 8 * 16;
    if (blocks > cap) blocks = cap;
    const uint8_t* w = static_cast<const uint8_t*>(W);
    switch (out_dtype) {
        case B200Q_DT_F16: gather_kernel<FMT, __half><<<(unsigned)blocks, 256, 0, st>>>(w, idx, (__half*)out, total, upr, row_bytes, rows); break;
        case B200Q_DT_BF16: gather_kernel<FMT, __nv_bfloat16><<<(unsigned)blocks, 256, 0, st>>>(w, idx, (__nv_bfloat16*)out, total, upr, row_bytes, rows); break;
        case B200Q_DT_F32: gather_kernel<FMT, float><<<(unsigned)blocks, 256, 0, st>>>(w, idx, (float*)out, total, upr, row_bytes, rows); break;
        default: return fail(B200Q_ERR_BAD_ARG, "embedding_gather: unknown output dtype %d", out_dtype);
    }
    B200Q_CUDA_TRY(cudaGetLastError());
    return B200Q_OK;
}

int launch_gather(int fmt, const void* W, const int32_t* idx, void* out, int out_dtype, int B, int64_t rows, int K, cudaStream_t st) {
    switch (fmt) {
        case kQ4_K: return launch_gather_fmt<kQ4_K>(W, idx, out, out_dtype, B, rows, K, st);
        case kQ6_K: return launch_gather_fmt<kQ6_K>(W, idx, out, out_dtype, B, rows, K, st);
        case kQ6_KP: return launch_gather_fmt<kQ6_KP>(W, idx, out, out_dtype, B, rows, K, st);
        case kQ8_0: return launch_gather_fmt<kQ8_0>(W, idx, out, out_dtype, B, rows, K, st);
        case kQ4_0: return launch_gather_fmt<kQ4_0>(W, idx, out, out_dtype, B, rows, K, st);
        case kQ5_K: return launch_gather_fmt<kQ5_K>(W, idx, out, out_dtype, B, rows, K, st);
    }
    return fail(B200Q_ERR_BAD_ARG, "embedding_gather: unknown block format %d", fmt);
}

}  // namespace b200q

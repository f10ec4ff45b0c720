// GEMM of the formats without a tcgen05 form, Q5_K and Q4_0, on warp-level FP16 MMA (sm_100a): Y(M, N) = X(M, K) * decode(W(N, K))^T
// (+bias), K a multiple of 256, any M, in passes of up to 64 tokens.
//
// These formats are multiplied in FP32 for one row; an FP16 weight, as the tcgen05 GEMM makes one, would be less. Here no weight
// is ever rounded:
//   * A fragments are the quants as FP16 integers: masked into the mantissas of two halves that hold 1024 (one logic operation), from
//     which a packed subtraction takes the 1024 (and Q4_0's offset of 8) off, exactly. (Left as subnormals, q * 2^-24, they would save
//     the subtraction, but the tensor cores align products without normalising them first: 1e-6 against 1.2e-7 of error.)
//   * B fragments are the activations in FP16, scaled per token by a power of two to [2^14, 2^15) (FP16 inputs never down): FP16 inputs
//     are exact, BF16 ones down to 2^-31 of the token's largest, and FP32 inputs are split into two FP16 terms, each multiplied, that hold
//     them to 2^-22 of their own size down to 2^-17 of the largest. Where that range is not enough for the bulk of some sub-block
//     (qm_sub_block_lost, and likewise the sums below), the token is marked for the plain FP32 loop, as are infinities and NaN.
//   * Every sub-block's products are summed on the tensor cores in FP32 and then multiplied by its scale in FP32 (four
//     FMA per 16 x 8 x 32 products). The minimums' term of Q5_K is one more MMA per 256 k: A the 6-bit mins, B the sub-block
//     sums of the activations as two FP16 terms.
//   * The pre-pass writes the activations in the order in which the quants come out of their bytes (the two halves of a
//     register are bytes 0 and 2 of a word, or 1 and 3), rotated for conflict-free ldmatrix.
// A CTA owns an even share of the rows, up to eight 16-row tiles at a time, and its warps are tiles x k-groups (the k-groups share
// each 256-k stage by sub-blocks and add up at the end in a fixed order). Stages of 256 k - raw rows and activations - are fetched with
// cp.async two or three ahead, one CTA barrier per stage. What bounds it at 48 tokens: the latency of its instructions with three to
// four warps per scheduler (about 1.9 times the cycles that its MMAs and its reads of B take).
// 96 FP16 tokens, 14336 x 4096: Q5_K 106 us, Q4_0 82 (twelve passes of the plain-load GEMV before: 0.85 ms, 0.7 ms); 16 tokens 37 and 28
// (147, 126).
//
// Takes the place of what brotensor's fused-dequant WMMA kernels are for its formats (src/cuda/q4k_wmma.cu:56-310).
#include "quant_mma.cuh"

namespace b200q {

constexpr int kMmMaxWarps = 16;
constexpr int kMmMaxTokens = 64;  // per pass
constexpr int kMmMaxTiles = 8;    // 16-row tiles of a CTA at a time

struct MmParams {
    const uint8_t* W;
    const void* X;     // the caller's activations (only read for the marked tokens)
    const void* bias;
    void* Y;           // first token row of this pass
    // prepared activations, this pass's first token: [K/256][tok_stride] rows of 512 bytes (high and, FP32 only, low terms) and of
    // 32 bytes (sub-block sums), 2^-e per token, and a mark per token that goes to the plain loop
    const uint8_t *Xh, *Xl, *Xs;
    const float* inv;
    const int* plain;
    int tokens, tok_stride, N, K;
    int x_dtype, y_dtype;
    int row_bytes, nblk;
    int mt, kg;        // row tiles at a time, k-groups: the CTA has mt * kg warps
    int n_stages, stage_bytes, off_b, off_lo, off_s, off_red;
    int row_q, row_r;  // CTA b owns row_q + (b < row_r) rows
};

// ---- pre-pass -------------------------------------------------------------------------------------------
// One block per token. pair8: a thread of the GEMM holds elements 8t .. 8t+7 of a sub-block (Q4_K, Q5_K), else 4t .. 4t+3 and
// 16+4t .. 16+4t+3. Register i of its four per row multiplies two of them: image position 8 i + 2 t + j of the sub-block.
__global__ void __launch_bounds__(256) gemm_mm_prep_kernel(const void* X, int x_dtype, int K, int tok_stride, int pair8, uint8_t* Xh,
                                                           uint8_t* Xl, uint8_t* Xs, float* inv, int* plain) {
    __shared__ uint32_t warp_top[8];
    const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const bool f32 = x_dtype == B200Q_DT_F32;
    grid_dep_launch();
    grid_dep_wait();
    uint32_t top = 0;
    for (int c = tid; c < (K >> 3); c += 256) {
        uint4 raw[2];
        float f[8];
        qm_load_raw(X, f32, K, m, 8 * c, raw);
        qm_to_f32(raw, x_dtype, f);
#pragma unroll
        for (int k = 0; k < 8; ++k) top = max(top, __float_as_uint(f[k]) & 0x7FFFFFFFu);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) warp_top[tid >> 5] = top;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) top = max(top, warp_top[w]);
    const bool finite = top < 0x7F800000u;
    int e = 14 + 127 - (int)(top >> 23);
    bool lost = !finite || (top != 0 && e > 126);  // (below 2^-112 the scale ends)
    e = (top == 0 || !finite) ? 0 : max(x_dtype == B200Q_DT_F16 ? 0 : -126, min(126, e));
    const float s = __uint_as_float((uint32_t)(e + 127) << 23);
    if (tid == 0) inv[m] = __uint_as_float((uint32_t)(127 - e) << 23);
    for (int c = tid; c < (K >> 3); c += 256) {  // K % 256 == 0: whole warps are in or out
        uint4 raw[2];
        float f[8];
        qm_load_raw(X, f32, K, m, 8 * c, raw);
        qm_to_f32(raw, x_dtype, f);
        const int blk = c >> 5, sub = (c >> 2) & 7, t = c & 3;
        const size_t row = (size_t)blk * tok_stride + m;
        float sum = 0.f;
        uint32_t mine = 0;
        __half h[8], l[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float v = f[k] * s;
            sum += v;
            mine = max(mine, __float_as_uint(f[k]) & 0x7FFFFFFFu);
            h[k] = __float2half_rn(v);
            l[k] = __float2half_rn(v - __half2float(h[k]));
        }
        // Where every eight neighbours reach 2^-12 of the token's largest, the terms hold enough of them; elsewhere it is looked at closely.
        const bool uneven = __any_sync(0xffffffffu, mine + (12u << 23) < top);
        if (uneven) {
            float err2 = 0.f;  // where the subnormals cut bits off
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float v = f[k] * s, err = kErrUp * (v - __half2float(h[k]) - (f32 ? __half2float(l[k]) : 0.f));
                if (fabsf(v) < 0.125f) err2 = fmaf(err, err, err2);
            }
            lost |= qm_sub_block_lost(f, s, err2);
        }
        auto put = [&](uint8_t* img, const __half(&v)[8]) {
            uint8_t* base = img + row * 512;
            auto word = [&](int a, int b) { return (uint32_t)__half_as_ushort(v[a]) | ((uint32_t)__half_as_ushort(v[b]) << 16); };
            // 16-byte chunk i of the sub-block sits at chunk (4 sub + i) ^ (m & 7) of the row
            auto chunk = [&](int i) { return base + (((4 * sub + i) ^ (m & 7)) << 4); };
            if (pair8) {
                *reinterpret_cast<uint32_t*>(chunk(0) + 4 * t) = word(0, 2);
                *reinterpret_cast<uint32_t*>(chunk(1) + 4 * t) = word(1, 3);
                *reinterpret_cast<uint32_t*>(chunk(2) + 4 * t) = word(4, 6);
                *reinterpret_cast<uint32_t*>(chunk(3) + 4 * t) = word(5, 7);
            } else {
                const int i = 2 * (t >> 1), o = 8 * (t & 1);  // run t / 2, threads 2 (t % 2) and the next
                *reinterpret_cast<uint2*>(chunk(i) + o) = make_uint2(word(0, 2), word(4, 6));
                *reinterpret_cast<uint2*>(chunk(i + 1) + o) = make_uint2(word(1, 3), word(5, 7));
            }
        };
        put(Xh, h);
        if (f32) put(Xl, l);
        if (pair8) {  // sub-block sums / 64 as two FP16 terms: [t2][high 2 t2, 2 t2 + 1, low 2 t2, 2 t2 + 1]
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum *= 0.015625f;
            const __half a = __float2half_rn(sum), b = __float2half_rn(sum - __half2float(a));
            if (t == 0) {
                __half* d = reinterpret_cast<__half*>(Xs + row * 32) + 4 * (sub >> 1) + (sub & 1);
                d[0] = a;
                d[2] = b;
            }
            if (uneven) {
                float size = 0.f;
#pragma unroll
                for (int k = 0; k < 8; ++k) size += fabsf(f[k] * s);
                size += __shfl_xor_sync(0xffffffffu, size, 1);
                size += __shfl_xor_sync(0xffffffffu, size, 2);
                lost |= fabsf(sum - __half2float(a) - __half2float(b)) * 2097152.0f > size * 0.015625f;
            }
        }
    }
    lost = __syncthreads_or(lost) != 0;
    if (tid == 0) plain[m] = lost ? 1 : 0;
}

// ---- the GEMM -------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// Quants of sub-block s (32 k) of one row as FP16 numbers: a[i], i = 0..3 (k16 step i / 2).
template <int FMT>
__device__ __forceinline__ void mm_quants(const QmRow& r, int s, int t, uint32_t (&a)[4]) {
    constexpr uint32_t kOne = 0x64006400u;  // 1024 in both halves: its lowest mantissa bit counts one
    if constexpr (FMT == kQ5_K) {
        const uint2 w = ls64(r.p + 48 + 32 * (s >> 1) + 8 * t), h = ls64(r.p + 16 + 8 * t);
        if (s & 1) {  // 16 q: nibble at bits 4..7, fifth bit at bit 8
            a[0] = hsub2_u32(lop3_and_or(w.x, 0x00F000F0u, kOne) | ((h.x << (8 - s)) & 0x01000100u), kOne);
            a[1] = hsub2_u32(lop3_and_or(w.x >> 8, 0x00F000F0u, kOne) | ((h.x >> s) & 0x01000100u), kOne);
            a[2] = hsub2_u32(lop3_and_or(w.y, 0x00F000F0u, kOne) | ((h.y << (8 - s)) & 0x01000100u), kOne);
            a[3] = hsub2_u32(lop3_and_or(w.y >> 8, 0x00F000F0u, kOne) | ((h.y >> s) & 0x01000100u), kOne);
        } else {
            const uint32_t x = s <= 4 ? h.x << (4 - s) : h.x >> (s - 4), y = s <= 4 ? h.y << (4 - s) : h.y >> (s - 4);
            a[0] = hsub2_u32(lop3_and_or(w.x, 0x000F000Fu, kOne) | (x & 0x00100010u), kOne);
            a[1] = hsub2_u32(lop3_and_or(w.x >> 8, 0x000F000Fu, kOne) | ((x >> 8) & 0x00100010u), kOne);
            a[2] = hsub2_u32(lop3_and_or(w.y, 0x000F000Fu, kOne) | (y & 0x00100010u), kOne);
            a[3] = hsub2_u32(lop3_and_or(w.y >> 8, 0x000F000Fu, kOne) | ((y >> 8) & 0x00100010u), kOne);
        }
    } else {
        const uint8_t* p = r.p + 18 * s + 4 * t;
        const uint32_t w = (s & 1) ? ls32(p + 2) : __funnelshift_r(ls32(p), ls32(p + 4), 16);
        a[0] = hsub2_u32(lop3_and_or(w, 0x000F000Fu, kOne), 0x64086408u);
        a[1] = hsub2_u32(lop3_and_or(w >> 8, 0x000F000Fu, kOne), 0x64086408u);
        a[2] = hsub2_u32(lop3_and_or(w >> 4, 0x000F000Fu, kOne), 0x64086408u);
        a[3] = hsub2_u32(lop3_and_or(w >> 12, 0x000F000Fu, kOne), 0x64086408u);
    }
}

// Scale of sub-block s of one row (Q5_K: over 16 where the quants come as 16 q). h: the row's header (Q5_K).
template <int FMT>
__device__ __forceinline__ float mm_scale(const QmRow& r, const uint4& h, int s) {
    if constexpr (FMT == kQ5_K) return h2f(h.x & 0xFFFFu) * ((s & 1) ? 0.0625f : 1.f) * byte_to_f32(s < 4 ? k_scales_lo(h) : k_scales_hi(h), s & 3);
    else return h2f(ls16(r.p + 18 * s));
}

template <int FMT, int NT, bool SPLIT, int KG>
__global__ void __launch_bounds__(kMmMaxWarps * 32, 1) gemm_mm_kernel(const __grid_constant__ MmParams p) {
    using F = QmFmt<FMT>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 127u) & ~127u;
    const uint8_t* smem = smem_raw + (sbase - smem_u32(smem_raw));
    __shared__ uint32_t plain[kMmMaxTokens / 32];  // bits of the tokens for the plain loop
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int nthreads = 32 * p.mt * KG;
    const int ki = warp / p.mt, mi = warp - ki * p.mt;
    const int cta = (int)blockIdx.x;
    const int row_begin = cta * p.row_q + min(cta, p.row_r), n_rows = p.row_q + (cta < p.row_r ? 1 : 0);
    const int rows_it = kQmTile * p.mt, iters = (n_rows + rows_it - 1) / rows_it, steps = iters * p.nblk;
    if (tid < kMmMaxTokens / 32) plain[tid] = 0;
    grid_dep_launch();

    // Next stage to fetch: rows of iteration ii, block ib, into ring slot islot.
    int ii = 0, ib = 0, islot = 0;
    const int lrow = tid >> 2, lt = tid & 3;
    auto issue = [&] {
        if (ii < iters) {
            const uint32_t st = sbase + (uint32_t)(islot * p.stage_bytes);
            for (int r = lrow; r < rows_it; r += nthreads >> 2)
                if (ii * rows_it + r < n_rows)
                    qm_copy_row<FMT>(st + (uint32_t)(r * F::stride), p.W + (size_t)(row_begin + ii * rows_it + r) * p.row_bytes + (size_t)ib * F::bytes, lt);
            const size_t row = (size_t)ib * p.tok_stride;
            for (int c = tid; c < p.tokens * 32; c += nthreads) cp_async16(st + (uint32_t)p.off_b + 16u * c, p.Xh + row * 512 + 16 * c);
            if constexpr (SPLIT)
                for (int c = tid; c < p.tokens * 32; c += nthreads) cp_async16(st + (uint32_t)p.off_lo + 16u * c, p.Xl + row * 512 + 16 * c);
            if constexpr (F::mins)
                for (int c = tid; c < p.tokens * 2; c += nthreads) cp_async16(st + (uint32_t)p.off_s + 16u * c, p.Xs + row * 32 + 16 * c);
            if (++ib == p.nblk) { ib = 0; ++ii; }
        }
        cp_async_commit();
        if (++islot == p.n_stages) islot = 0;
    };
    // Until the predecessor is done only the L2 is told about the first blocks of this CTA's rows.
    for (int r = lrow; r < min(rows_it, n_rows); r += nthreads >> 2) prefetch_l2_line(p.W + (size_t)(row_begin + r) * p.row_bytes + min(128 * lt, p.row_bytes - 1));
    grid_dep_wait();
    for (int s = 0; s < p.n_stages - 1; ++s) issue();

    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
    constexpr int kSubs = 8 / KG;
    const int s_first = ki * kSubs;
    const uint32_t b_lane = (uint32_t)((lane & 7) * 512);
    int slot = 0, it = 0, blk = 0;
    float odd = 0.f;  // not zero once one of the thread's results is not finite (an infinite scale)
    for (int step = 0; step < steps; ++step) {
        if (p.n_stages == 4) cp_async_wait<2>();
        else if (p.n_stages == 3) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();  // the stage has landed for everybody, and everybody is done with the slot filled next
        issue();
        const uint32_t st = sbase + (uint32_t)(slot * p.stage_bytes), sb = st + (uint32_t)p.off_b;
        const int r0 = it * rows_it + mi * kQmTile;
        if (r0 < n_rows) {
            const uint8_t* slot_a = smem + slot * p.stage_bytes + (mi * kQmTile + g) * F::stride;
            const QmRow ra = {slot_a, 0u}, rb = {slot_a + 8 * F::stride, 0u};
            uint4 hA = make_uint4(0, 0, 0, 0), hB = hA;
            if constexpr (F::mins) {
                hA = ls128(ra.p);
                hB = ls128(rb.p);
            }
#pragma unroll
            for (int si = 0; si < kSubs; ++si) {
                const int s = s_first + si;
                uint32_t a[4], b[4];
                mm_quants<FMT>(ra, s, t, a);
                mm_quants<FMT>(rb, s, t, b);
                const float fA = mm_scale<FMT>(ra, hA, s), fB = mm_scale<FMT>(rb, hB, s);
                const uint32_t baddr = sb + b_lane + ((((uint32_t)(4 * s) + (uint32_t)(lane >> 3)) ^ (uint32_t)(lane & 7)) << 4);
                // three or four token groups together: their loads, then their MMAs - a group's second MMA waits for its
                // first - then their FMAs (one after the other a group cost the sum of those latencies)
                constexpr int GN = NT % 4 == 0 ? 4 : NT % 3 == 0 ? 3 : 2;
#pragma unroll
                for (int n0 = 0; n0 < NT; n0 += GN) {
                    uint32_t x[GN][4], y[SPLIT ? GN : 1][4];
                    float c[GN][4];
#pragma unroll
                    for (int n = 0; n < GN; ++n) {
                        ldsm4(baddr + (uint32_t)(n0 + n) * 4096u, x[n]);
                        if constexpr (SPLIT) ldsm4(baddr + (uint32_t)(p.off_lo - p.off_b) + (uint32_t)(n0 + n) * 4096u, y[n]);
                    }
#pragma unroll
                    for (int n = 0; n < GN; ++n) qm_mma_zero<false>(c[n], a[0], b[0], a[1], b[1], x[n][0], x[n][1]);
                    if constexpr (SPLIT) {
#pragma unroll
                        for (int n = 0; n < GN; ++n) qm_mma<false>(c[n], a[0], b[0], a[1], b[1], y[n][0], y[n][1]);
                    }
#pragma unroll
                    for (int n = 0; n < GN; ++n) qm_mma<false>(c[n], a[2], b[2], a[3], b[3], x[n][2], x[n][3]);
                    if constexpr (SPLIT) {
#pragma unroll
                        for (int n = 0; n < GN; ++n) qm_mma<false>(c[n], a[2], b[2], a[3], b[3], y[n][2], y[n][3]);
                    }
#pragma unroll
                    for (int n = 0; n < GN; ++n) {
                        acc[n0 + n][0] = fmaf(fA, c[n][0], acc[n0 + n][0]);
                        acc[n0 + n][1] = fmaf(fA, c[n][1], acc[n0 + n][1]);
                        acc[n0 + n][2] = fmaf(fB, c[n][2], acc[n0 + n][2]);
                        acc[n0 + n][3] = fmaf(fB, c[n][3], acc[n0 + n][3]);
                    }
                }
            }
            if constexpr (F::mins) {
                if (blk % KG == ki) {  // the k-groups take turns with the blocks' minimums
                    // A: mins of sub-blocks 2t, 2t + 1, once against the sums' high terms and once against the low
                    auto mins = [&](const uint4& h) {
                        return hsub2_u32(__byte_perm(t < 2 ? k_mins_lo(h) : k_mins_hi(h), 0x64u, (t & 1) ? 0x4342 : 0x4140), 0x64006400u);
                    };
                    const uint32_t m0 = mins(hA), m1 = mins(hB);
                    const float fA = -64.f * h2f(hA.x >> 16), fB = -64.f * h2f(hB.x >> 16);
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        const uint2 x = ls64(smem + slot * p.stage_bytes + p.off_s + (8 * n + g) * 32 + 8 * t);
                        float c[4];
                        qm_mma_zero<false>(c, m0, m1, m0, m1, x.x, x.y);
                        acc[n][0] = fmaf(fA, c[0], acc[n][0]);
                        acc[n][1] = fmaf(fA, c[1], acc[n][1]);
                        acc[n][2] = fmaf(fB, c[2], acc[n][2]);
                        acc[n][3] = fmaf(fB, c[3], acc[n][3]);
                    }
                }
            }
        }
        if (++slot == p.n_stages) slot = 0;
        if (++blk < p.nblk) continue;
        // ---- these rows are done: add up the k-groups (in order), store
        blk = 0;
        {
            const uint32_t red = sbase + (uint32_t)p.off_red + (uint32_t)(lane * 16);
            if (ki > 0)
#pragma unroll
                for (int n = 0; n < NT; ++n)
                    sts128(red + (uint32_t)((((ki - 1) * p.mt + mi) * NT + n) * 512),
                           make_uint4(__float_as_uint(acc[n][0]), __float_as_uint(acc[n][1]), __float_as_uint(acc[n][2]), __float_as_uint(acc[n][3])));
            __syncthreads();
            if (ki == 0)
                for (int k = 1; k < KG; ++k)
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        const uint4 v = lds128i<0>(red + (uint32_t)((((k - 1) * p.mt + mi) * NT + n) * 512));
                        acc[n][0] += __uint_as_float(v.x);
                        acc[n][1] += __uint_as_float(v.y);
                        acc[n][2] += __uint_as_float(v.z);
                        acc[n][3] += __uint_as_float(v.w);
                    }
        }
        if (ki == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + g + 8 * h;
                if (r < n_rows) {
                    const int row = row_begin + r;
                    const float bv = qm_bias(p.bias, p.x_dtype, row);
#pragma unroll
                    for (int n = 0; n < NT; ++n)
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const int m = 8 * n + 2 * t + j;
                            if (m < p.tokens) {
                                odd = fmaf(acc[n][2 * h + j], 0.f, odd);
                                qm_store(p.Y, p.y_dtype, (size_t)m * p.N + row, fmaf(acc[n][2 * h + j], p.inv[m], bv));
                            }
                        }
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
        ++it;
    }
    // The marked tokens, and all of them where a result is not finite: their results in FP32 arithmetic.
    if (!(odd == 0.f)) atomicOr(&plain[0], ~0u), atomicOr(&plain[1], ~0u);
    if (tid < p.tokens && p.plain[tid]) atomicOr(&plain[tid >> 5], 1u << (tid & 31));
    __syncthreads();  // (and the stores above come first)
    for (int m = 0; m < p.tokens; m += 8)
        if (const uint32_t rows = plain[m >> 5] >> (m & 31) & 0xFFu & ((1u << min(8, p.tokens - m)) - 1u))
            qm_plain_rows<FMT>(p.W, p.X, p.x_dtype, p.bias, p.Y, p.y_dtype, m, rows, p.N, p.K, p.row_bytes, row_begin, n_rows);
}

// ---- host side ------------------------------------------------------------------------------------------

static int g_opt_mm = 1;
void mm_set_enabled(int v) { g_opt_mm = v ? 1 : 0; }
int mm_get_enabled() { return g_opt_mm; }

// The workspace: images of the high and (FP32) low terms, the sub-block sums, 2^-e and the marks.
static int mm_tok_stride(int M) { return (M + 7) & ~7; }
static size_t mm_image_bytes(int M, int K) { return (size_t)(K / 256) * mm_tok_stride(M) * 512; }
static size_t mm_sums_bytes(int M, int K) { return (size_t)(K / 256) * mm_tok_stride(M) * 32; }
size_t gemm_mm_workspace_bytes(int fmt, int x_dtype, int M, int N, int K) {
    (void)N;
    if (K % 256 != 0 || (fmt != kQ5_K && fmt != kQ4_0)) return 0;
    return mm_image_bytes(M, K) * (x_dtype == B200Q_DT_F32 ? 2 : 1) + mm_sums_bytes(M, K) + (size_t)mm_tok_stride(M) * 8;
}

template <int FMT, int NT, bool SPLIT, int KG>
static int launch_mm_k(const MmParams& p, int grid, size_t smem, cudaStream_t st) {
    auto kern = gemm_mm_kernel<FMT, NT, SPLIT, KG>;
    static bool configured[64] = {};
    int dev = 0;
    B200Q_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        B200Q_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    B200Q_CUDA_TRY(launch_dep(pdl_option() >= 0, kern, dim3((unsigned)grid), dim3((unsigned)(32 * p.mt * p.kg)), smem, st, p));
    return B200Q_OK;
}

template <int FMT, int NT, bool SPLIT>
static int launch_mm(const MmParams& p, int grid, size_t smem, cudaStream_t st) {
    if (p.kg == 8) return launch_mm_k<FMT, NT, SPLIT, 8>(p, grid, smem, st);
    if (p.kg == 4) return launch_mm_k<FMT, NT, SPLIT, 4>(p, grid, smem, st);
    return launch_mm_k<FMT, NT, SPLIT, 2>(p, grid, smem, st);
}

template <int FMT, bool SPLIT>
static int launch_mm_f(MmParams& p, int sms, cudaStream_t st, bool* taken) {
    using F = QmFmt<FMT>;
    p.row_bytes = p.nblk * F::bytes;
    int grid = sms;
    if (grid > p.N) grid = p.N;
    p.row_q = p.N / grid;
    p.row_r = p.N % grid;
    const int rows = p.row_q + (p.row_r ? 1 : 0), tiles = (rows + kQmTile - 1) / kQmTile;
    const int iters = (tiles + kMmMaxTiles - 1) / kMmMaxTiles;
    p.mt = (tiles + iters - 1) / iters;
    p.kg = p.mt <= 2 ? 8 : p.mt <= 4 ? 4 : 2;  // at most sixteen warps
    const int nt = p.tokens <= 16 ? 2 : p.tokens <= 32 ? 4 : p.tokens <= 48 ? 6 : 8;
    p.off_b = p.mt * kQmTile * F::stride;
    p.off_lo = p.off_b + nt * 8 * 512;
    p.off_s = p.off_lo + (SPLIT ? nt * 8 * 512 : 0);
    p.stage_bytes = (p.off_s + (F::mins ? nt * 8 * 32 : 0) + 127) & ~127;
    const size_t red = (size_t)(p.kg - 1) * p.mt * nt * 512, budget = 227 * 1024 - 1024 - 128;
    p.n_stages = 4;
    while (p.n_stages > 2 && (size_t)p.n_stages * p.stage_bytes + red > budget) --p.n_stages;
    if ((size_t)p.n_stages * p.stage_bytes + red > budget) return B200Q_OK;
    p.off_red = p.n_stages * p.stage_bytes;
    const size_t smem = (size_t)p.off_red + red + 128;
    *taken = true;
    switch (nt) {
        case 2: return launch_mm<FMT, 2, SPLIT>(p, grid, smem, st);
        case 4: return launch_mm<FMT, 4, SPLIT>(p, grid, smem, st);
        case 6: return launch_mm<FMT, 6, SPLIT>(p, grid, smem, st);
        default: return launch_mm<FMT, 8, SPLIT>(p, grid, smem, st);
    }
}
template <int FMT>
static int launch_mm_x(MmParams& p, int sms, cudaStream_t st, bool* taken) {
    return p.x_dtype == B200Q_DT_F32 ? launch_mm_f<FMT, true>(p, sms, st, taken) : launch_mm_f<FMT, false>(p, sms, st, taken);
}

// Runs the call when it can (*taken = true): Q5_K or Q4_0, K a multiple of 256, weights on a 16-byte boundary, a 16-byte aligned workspace of gemm_mm_workspace_bytes.
int launch_gemm_mm(int fmt, const void* W, const void* X, int x_dtype, const void* bias, void* Y, int y_dtype, int M, int N, int K,
                   void* ws, size_t ws_bytes, int sms, cudaStream_t st, bool* taken) {
    *taken = false;
    const size_t need = gemm_mm_workspace_bytes(fmt, x_dtype, M, N, K);
    if (!g_opt_mm || !need || !ws || ws_bytes < need || (reinterpret_cast<uintptr_t>(ws) & 15) != 0) return B200Q_OK;
    if ((reinterpret_cast<uintptr_t>(W) & 15) != 0) return B200Q_OK;
    const int stride = mm_tok_stride(M);
    uint8_t* base = static_cast<uint8_t*>(ws);
    uint8_t* xh = base;
    uint8_t* xl = xh + mm_image_bytes(M, K);
    uint8_t* xs = xl + (x_dtype == B200Q_DT_F32 ? mm_image_bytes(M, K) : 0);
    float* inv = reinterpret_cast<float*>(xs + mm_sums_bytes(M, K));
    int* plain = reinterpret_cast<int*>(inv + stride);
    const int passes = (M + kMmMaxTokens - 1) / kMmMaxTokens, per = ((M + passes - 1) / passes + 7) & ~7;
    bool prepared = false;
    for (int t0 = 0; t0 < M; t0 += per) {
        MmParams p = {};
        p.W = static_cast<const uint8_t*>(W);
        p.X = static_cast<const uint8_t*>(X) + (size_t)t0 * K * (x_dtype == B200Q_DT_F32 ? 4 : 2);
        p.bias = bias;
        p.Y = static_cast<uint8_t*>(Y) + (size_t)t0 * N * (y_dtype == B200Q_DT_F32 ? 4 : 2);
        p.Xh = xh + (size_t)t0 * 512;
        p.Xl = xl + (size_t)t0 * 512;
        p.Xs = xs + (size_t)t0 * 32;
        p.inv = inv + t0;
        p.plain = plain + t0;
        p.tokens = M - t0 < per ? M - t0 : per;
        p.tok_stride = stride;
        p.N = N;
        p.K = K;
        p.x_dtype = x_dtype;
        p.y_dtype = y_dtype;
        p.nblk = K / 256;
        if (!prepared) {
            prepared = true;
            B200Q_CUDA_TRY(launch_dep(pdl_option() >= 0, gemm_mm_prep_kernel, dim3((unsigned)M), dim3(256), 0, st, X, x_dtype, K, stride,
                                      (int)(fmt == kQ5_K), xh, xl, xs, inv, plain));
        }
        bool ok = false;
        int rc = B200Q_OK;
        if (fmt == kQ5_K) rc = launch_mm_x<kQ5_K>(p, sms, st, &ok);
        else rc = launch_mm_x<kQ4_0>(p, sms, st, &ok);
        if (rc) return rc;
        if (!ok) return B200Q_OK;  // every pass has the same plan or a smaller one: the first declines or none does
    }
    *taken = true;
    return B200Q_OK;
}

}  // namespace b200q

// Decode GEMV on the integer tensor cores for the calls that gemv_hm.cu does not take and that had only the plain-load kernel -
// Q5_K and Q4_0, and Q6_K rows that are not whole runs of eight blocks - 1..8 activation rows of any type, K a multiple of 256
// (sm_100a): Y(M, N) = X(M, K) * decode(W(N, K))^T with FP32-class accuracy.
//
// What bounds a decode GEMV is the weight stream; what kept the other kernels from it outside their home shapes
// is listed with each choice:
//   * Weights stay integers. A 16-row x 32-k piece of the blocks is the A operand of mma.sync.m16n8k32 (Q6_K, whose
//     scales cover 16 elements: m16n8k16), unpacked with one to four logic operations per four weights; block and
//     sub-block scales are applied to the integer sums.
//   * Activations are fixed point with one power-of-two scale per 256 elements and row, cut into signed bytes ("planes"). The
//     MMA's eight columns are (plane, row) pairs: eight planes of one FP32 row (62 bits, in which a value above 2^-36 of the block's
//     largest is exact), four planes of two rows (30 bits: FP32 values are exact down to 2^-6 of the largest, FP16 ones to 2^-19, BF16
//     ones to 2^-22), two of four or one of eight. So one to two rows need ONE MMA per k-step, three to four two, five to eight
//     four. Integer sums are exact; a result's error is that of a few hundred FP32 additions, as long as what the planes leave out is
//     small beside the bulk of a sub-block's activations and not only beside the largest (qm_sub_block_lost); a row where it is not (a
//     channel some thousand times the others, in FP32), or of magnitudes outside 2^-90 .. 2^97, takes the plain loop below.
//   * A warp owns one 256-element block column of the weight rows ("its block") for a whole phase of the launch: the B
//     fragments of that block stay in registers (16 per MMA column set). Up to sixteen warps cover K = 4096; longer rows run in
//     phases over the CTA's rows, shorter ones with several row groups side by side.
//   * A warp loads what it multiplies itself: cp.async, 16 bytes per lane, into a private ring of three to five tiles of
//     16 rows x 1 block. No producer warp, no bulk copies (one costs an SM 45-70 ns whatever its size), no alignment demand on
//     rows: a Q6_K row of K = 2560 is 2100 bytes, so its pieces are fetched from the 16-byte boundary before them.
//   * The warps' partial sums meet in shared memory one tile late: a warp leaves its sums of tile i after everybody
//     has arrived for tile i - 1, adds up its share of tile i - 1 and arrives, so nobody waits for the slowest
//     warp of the current tile. The order of the additions is fixed (reproducible results).
//   * The minimums' term of Q5_K, sum over sub-blocks of dmin * m * sum(x), is one TF32 MMA per column set: the
//     6-bit mins are exact in TF32 and the FP32 sums of x are split over the planes' columns in pieces of 11 bits.
// Measured (one FP32 row, us, plain-load kernel -> this one): Q5_K 14336 x 4096 39.8 -> 18.3, 4096 x 4096 16.9 -> 8.3, 4096 x 14336 50.6 -> 21.9; Q4_0 29.5 -> 19.0,
// 13.1 -> 7.6, 40.4 -> 21.4; Q6_K 2560 x 6912 20.8 -> 13.2. 14336 x 4096 is 2.2 TB/s of Q5_K and 1.7 of Q4_0, 34 and 27 % of the memory's rate: 58
// instructions per k-step of 16 x 32, of which the kernel's own work is about 25 and the rest is waiting for the others at a tile's end.
// Three and more rows spill (128 registers, 60 .. 840 bytes): staging, not the loop.
// Rows of activations that are not finite or not held, and all rows where a result is not finite, take a plain FP32 loop at the end of the
// launch (qm_plain_rows): an integer sum of zero times an infinite scale is not what the decoded weights give.
//
// Takes the place of brotensor's decode GEMVs (src/cuda/q4k.cu:159-224, q6k.cu:117-176, q8_0.cu:75-138) and of the
// per-row loop of its batched ops for small B (q4k.cu:413-418).
#include "quant_mma.cuh"
#include "stream_common.cuh"

namespace b200q {

constexpr int kMbMaxWarps = 16;

struct MbParams {
    const uint8_t* W;
    const void* X;
    const void* bias;
    void* Y;
    int* status;
    int M, N, K;
    int x_dtype, y_dtype;
    int row_bytes, nblk;     // bytes and 256-element blocks of a weight row
    int nwk, rg;             // warps along K per phase, row groups: the CTA has nwk * rg warps
    int phases;              // ceil(nblk / nwk)
    int tpo;                 // threads that add up one output's partial sums (a power of two)
    int row_q, row_r;        // CTA b owns row_q + (b < row_r) rows
    int off_part, off_yacc;  // shared-memory offsets behind the rings
    int early_w;             // 1: weights are read ahead of griddepcontrol.wait
    unsigned int wait_limit_us;
};

// D = A * B + c, 16 x 8 x 32, all four accumulators starting at c
__device__ __forceinline__ void mma_s8s8(int (&d)[4], const uint32_t (&a)[4], uint2 b, int c) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y), "r"(c));
}
__device__ __forceinline__ void mma_s8s8_k16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(b), "r"(0));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const float (&a)[4], float b0, float b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
                   "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)), "f"(0.f));
}
__device__ __forceinline__ int s8_at(uint32_t w, int idx) { return (int)(w << (24 - 8 * idx)) >> 24; }

// The activations of a warp's block as it multiplies them.
template <int NB>
struct MbX {
    uint2 b[8][NB];   // B fragments of the eight k-steps
    float mn[NB][2];  // B fragments of the mins' MMA: pieces of the sub-block sums t and t + 4 of the lane's column
    float cs[2];      // what the accumulator columns 2t and 2t + 1 count: 2^-e, with eight planes the highest plane's 2^(24-e)
};

// One block column of a 16-row tile (FP32 factors are applied in an order that keeps products of sums and block scales in range): v = this warp's share of (row g, columns 2t, 2t + 1), (row g + 8, same), the
// planes that sit in different column sets already combined. ra, rb: rows g and g + 8.
template <int FMT, int MC, int NB>
__device__ __forceinline__ void mb_block(const QmRow& ra, const QmRow& rb, int t, const MbX<NB>& x, float (&v)[4]) {
    // weight of column set nb: planes run over the sets in steps of 8 / MC
    constexpr float kStep = MC == 8 ? 256.f : 65536.f;
    if constexpr (FMT == kQ5_K) {
        const uint4 hA = ls128(ra.p), hB = ls128(rb.p);
        const uint32_t sc[2][2] = {{k_scales_lo(hA), k_scales_hi(hA)}, {k_scales_lo(hB), k_scales_hi(hB)}};
        const uint8_t *pa = ra.p + 8 * t, *pb = rb.p + 8 * t;
        const uint2 hbA = ls64(pa + 16), hbB = ls64(pb + 16);
        int is[NB][4];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
            for (int i = 0; i < 4; ++i) is[nb][i] = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint2 qA = ls64(pa + 48 + 32 * c), qB = ls64(pb + 48 + 32 * c);
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int s = 2 * c + o;  // sub-block
                auto quants = [&](uint32_t q, uint32_t hb) {
                    return ((q >> (4 * o)) & 0x0F0F0F0Fu) | ((s < 4 ? hb << (4 - s) : hb >> (s - 4)) & 0x10101010u);
                };
                const uint32_t a[4] = {quants(qA.x, hbA.x), quants(qB.x, hbB.x), quants(qA.y, hbA.y), quants(qB.y, hbB.y)};
                const int scA = (int)byte_at(sc[0][s >> 2], s & 3), scB = (int)byte_at(sc[1][s >> 2], s & 3);
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    int d[4];
                    mma_s8s8(d, a, x.b[s][nb], 0);
                    // 63 * 32 * 31 * 128 * 8 sub-blocks = 6.4e7
                    is[nb][0] += scA * d[0];
                    is[nb][1] += scA * d[1];
                    is[nb][2] += scB * d[2];
                    is[nb][3] += scB * d[3];
                }
            }
        }
        // mins: A(16 x 8) = m of the eight sub-blocks, B(8 x 8) = pieces of the sums of x
        const float am[4] = {byte_to_f32(k_mins_lo(hA), t), byte_to_f32(k_mins_lo(hB), t), byte_to_f32(k_mins_hi(hA), t), byte_to_f32(k_mins_hi(hB), t)};
        float f[4] = {0.f, 0.f, 0.f, 0.f}, fm[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int nb = NB - 1; nb >= 0; --nb) {
            float dm[4];
            mma_tf32(dm, am, x.mn[nb][0], x.mn[nb][1]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                f[i] = fmaf(f[i], kStep, (float)is[nb][i]);
                fm[i] = fmaf(fm[i], kStep, dm[i]);
            }
        }
        const float dA = h2f(hA.x & 0xFFFFu), dB = h2f(hB.x & 0xFFFFu), mA = h2f(hA.x >> 16), mB = h2f(hB.x >> 16);
        v[0] = fmaf(dA * f[0], x.cs[0], -(mA * fm[0]));
        v[1] = fmaf(dA * f[1], x.cs[1], -(mA * fm[1]));
        v[2] = fmaf(dB * f[2], x.cs[0], -(mB * fm[2]));
        v[3] = fmaf(dB * f[3], x.cs[1], -(mB * fm[3]));
    } else if constexpr (FMT == kQ6_K) {
        int is[NB][4];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
            for (int i = 0; i < 4; ++i) is[nb][i] = 0;
#pragma unroll
        for (int G = 0; G < 2; ++G) {
            uint32_t ql[2][4], qh[2][2], sc[2][2];  // [row][2 j + h] / [row][h] / [row][word]
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const QmRow& row = r ? rb : ra;
                const QmRow mine = {row.p + 4 * t, row.sh};
#pragma unroll
                for (int jh = 0; jh < 4; ++jh) ql[r][jh] = qm_word(mine, 64 * G + 32 * (jh >> 1) + 16 * (jh & 1));
#pragma unroll
                for (int h = 0; h < 2; ++h) qh[r][h] = qm_word(mine, 128 + 32 * G + 16 * h);
                sc[r][0] = qm_word(row, 192 + 8 * G);
                sc[r][1] = qm_word(row, 196 + 8 * G);
            }
#pragma unroll
            for (int Q = 0; Q < 4; ++Q)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t a[2];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {  // bytes 4 * (raw6 - 32), -128 .. 124
                        const uint32_t w = ql[r][2 * (Q & 1) + h];
                        const uint32_t lo = (Q < 2 ? w << 2 : w >> 2) & 0x3C3C3C3Cu;
                        a[r] = (lo | ((qh[r][h] << (6 - 2 * Q)) & 0xC0C0C0C0u)) ^ 0x80808080u;
                    }
                    const int s = 2 * Q + h;  // scale of the half
                    const int scA = s8_at(sc[0][s >> 2], s & 3), scB = s8_at(sc[1][s >> 2], s & 3);
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) {
                        int d[4];
                        const uint2 b = x.b[4 * G + Q][nb];
                        mma_s8s8_k16(d, a[0], a[1], h ? b.y : b.x);
                        // 128 * 16 * 128 * 128 * 16 sub-blocks = 5.4e8
                        is[nb][0] += scA * d[0];
                        is[nb][1] += scA * d[1];
                        is[nb][2] += scB * d[2];
                        is[nb][3] += scB * d[3];
                    }
                }
        }
        float f[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int nb = NB - 1; nb >= 0; --nb)
#pragma unroll
            for (int i = 0; i < 4; ++i) f[i] = fmaf(f[i], kStep, (float)is[nb][i]);
        const float dA = h2f((ls32(ra.p + 208) >> ra.sh) & 0xFFFFu) * 0.25f, dB = h2f((ls32(rb.p + 208) >> rb.sh) & 0xFFFFu) * 0.25f;
        v[0] = dA * f[0] * x.cs[0];
        v[1] = dA * f[1] * x.cs[1];
        v[2] = dB * f[2] * x.cs[0];
        v[3] = dB * f[3] * x.cs[1];
    } else {
        // Q4_0: a scale per 32 elements. The MMA starts from the bits of 1.5 * 2^23, so its integer result (at most
        // 2^19) read as a float is that number plus the sum: one subtraction instead of a conversion.
        float f[NB][4];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
            for (int i = 0; i < 4; ++i) f[nb][i] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            uint32_t a[4];
            const uint8_t *pa = ra.p + 18 * j + 4 * t, *pb = rb.p + 18 * j + 4 * t;
            // quants two bytes behind a word boundary in even blocks
            const uint32_t wa = (j & 1) ? ls32(pa + 2) : __funnelshift_r(ls32(pa), ls32(pa + 4), 16);
            const uint32_t wb = (j & 1) ? ls32(pb + 2) : __funnelshift_r(ls32(pb), ls32(pb + 4), 16);
            // bytes 16 * (nibble - 8); the low nibbles are elements 0..15, the high ones 16..31
            a[0] = ((wa << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
            a[1] = ((wb << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
            a[2] = (wa & 0xF0F0F0F0u) ^ 0x80808080u;
            a[3] = (wb & 0xF0F0F0F0u) ^ 0x80808080u;
            const float dA = h2f(ls16(ra.p + 18 * j)) * 0.0625f, dB = h2f(ls16(rb.p + 18 * j)) * 0.0625f;
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
                int d[4];
                mma_s8s8(d, a, x.b[j][nb], 0x4B400000);
                f[nb][0] = fmaf(dA, __int_as_float(d[0]) - 12582912.0f, f[nb][0]);
                f[nb][1] = fmaf(dA, __int_as_float(d[1]) - 12582912.0f, f[nb][1]);
                f[nb][2] = fmaf(dB, __int_as_float(d[2]) - 12582912.0f, f[nb][2]);
                f[nb][3] = fmaf(dB, __int_as_float(d[3]) - 12582912.0f, f[nb][3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float s = f[NB - 1][i];
#pragma unroll
            for (int nb = NB - 2; nb >= 0; --nb) s = fmaf(s, kStep, f[nb][i]);
            v[i] = s * x.cs[i & 1];
        }
    }
}

// Fixed point and byte planes of the warp's block: x rows 0 .. M-1, elements [256 blk, 256 blk + 256), into fragments.
// `scratch`: 2304 bytes of shared memory of the warp's own. Returns the rows (bits) that are not finite or not held closely enough.
template <int FMT, int MC, int NB>
__device__ __forceinline__ uint32_t mb_stage_x(const MbParams& p, int blk, uint32_t scratch, int lane, MbX<NB>& x) {
    constexpr int kPlanes = 8 * NB / MC;
    static_assert(kPlanes == 4 || kPlanes == 8, "planes");
    const int g = lane >> 2, t = lane & 3;
    const bool f32 = p.x_dtype == B200Q_DT_F32;
    constexpr int kBatch = MC == 8 ? 4 : MC;  // rows whose loads are in flight together (registers)
    uint32_t w[MC][kPlanes][2];               // byte planes of the lane's eight elements
    float s0 = 0.f, s1 = 0.f;  // sums of x over sub-blocks t and t + 4, row of this lane's column
    uint32_t left = 0;
    x.cs[0] = x.cs[1] = 0.f;
#pragma unroll
    for (int m0 = 0; m0 < MC; m0 += kBatch) {
        uint4 raw[kBatch][2];
#pragma unroll
        for (int i = 0; i < kBatch; ++i)
            if (m0 + i < p.M) qm_load_raw(p.X, f32, p.K, m0 + i, 256 * blk + 8 * lane, raw[i]);
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const int m = m0 + i;
            if (m < p.M) {
                float f[8];
                qm_to_f32(raw[i], p.x_dtype, f);
                uint32_t mine = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) mine = max(mine, __float_as_uint(f[k]) & 0x7FFFFFFFu);
                const uint32_t top = __reduce_max_sync(0xffffffffu, mine);
                // 2^-90 .. 2^97: scales, sums of x and their pieces stay in FP32's range
                const bool in_range = top - 0x12800000u < 0x70000000u - 0x12800000u;
                // the largest value lies in [2^29, 2^30)
                const int e = in_range ? 29 + 127 - (int)(top >> 23) : 0;
                const float s = __uint_as_float((uint32_t)(e + 127) << 23), inv = __uint_as_float((uint32_t)(127 - e + (kPlanes == 8 ? 24 : 0)) << 23);
                uint32_t u[kPlanes / 4][8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float v = f[k] * s;
                    const int hi = __float2int_rn(v);
                    if constexpr (kPlanes == 8) {
                        const int lo = __float2int_rn((v - (float)hi) * 2147483648.0f);
                        const unsigned long long b = ((unsigned long long)(unsigned int)hi << 32) + (unsigned long long)(2LL * lo) + 0x8080808080808080ull;
                        u[0][k] = (uint32_t)b;
                        u[1][k] = (uint32_t)(b >> 32);
                    } else {
                        u[0][k] = (uint32_t)hi + 0x80808080u;
                    }
                }
                // Where every eight neighbours reach 2^-6 of the block's largest (eight planes: 2^-30), the planes hold enough of them; elsewhere it
                // is looked at closely.
                if (__any_sync(0xffffffffu, mine + ((kPlanes == 8 ? 30u : 6u) << 23) < top)) {
                    float err2 = 0.f;  // of eight planes at most 2^-32 each
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float err = kErrUp * (kPlanes == 8 ? 2.3283064365386963e-10f : f[k] * s - (float)__float2int_rn(f[k] * s));
                        err2 = fmaf(err, err, err2);
                    }
                    if (qm_sub_block_lost(f, s, err2)) left |= 1u << m;
                }
                if (top != 0 && !in_range) left |= 1u << m;
#pragma unroll
                for (int pl = 0; pl < kPlanes; ++pl)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t* q = &u[pl / 4][4 * h];
                        const uint32_t sel = (pl & 3) | ((4 + (pl & 3)) << 4);
                        w[m][pl][h] = __byte_perm(__byte_perm(q[0], q[1], sel), __byte_perm(q[2], q[3], sel), 0x5410) ^ 0x80808080u;
                    }
                if (((2 * t) & (MC - 1)) == m) x.cs[0] = inv;
                if (((2 * t + 1) & (MC - 1)) == m) x.cs[1] = inv;
                if constexpr (QmFmt<FMT>::mins) {
                    float sum = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
                    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                    const float a = __shfl_sync(0xffffffffu, sum, 4 * t), b = __shfl_sync(0xffffffffu, sum, 4 * t + 16);
                    if ((g & (MC - 1)) == m) {
                        s0 = a;
                        s1 = b;
                    }
                }
            }
        }
    }
    if constexpr (QmFmt<FMT>::mins) {
        // three pieces of 11 bits; plane i of four counts 256^i times (of eight: the highest once, the next 1 / 256), so a piece is divided by that
        float pc[4][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float s = h ? s1 : s0;
            const float a = __uint_as_float(__float_as_uint(s) & 0xFFFFE000u), r = s - a;
            const float b = __uint_as_float(__float_as_uint(r) & 0xFFFFE000u);
            pc[0][h] = a;
            pc[1][h] = b * (kPlanes == 8 ? 256.f : 0.00390625f);
            pc[2][h] = (r - b) * (kPlanes == 8 ? 65536.f : 1.52587890625e-5f);
            pc[3][h] = 0.f;
        }
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if constexpr (MC == 8) x.mn[nb][h] = pc[nb][h];
                else if constexpr (MC == 4) x.mn[nb][h] = (g & 4) ? pc[2 * nb + 1][h] : pc[2 * nb][h];
                else if constexpr (MC == 2) x.mn[nb][h] = (g & 4) ? ((g & 2) ? pc[3][h] : pc[2][h]) : ((g & 2) ? pc[1][h] : pc[0][h]);
                else x.mn[nb][h] = g == 7 ? pc[0][h] : g == 6 ? pc[1][h] : g == 5 ? pc[2][h] : 0.f;
            }
    }
    // k-steps per pass through the scratch memory: [k-step][set][column][t] of 8 bytes, k-steps 32 bytes apart in banks
    constexpr int KC = NB == 1 ? 8 : NB == 2 ? 4 : 2;
    constexpr uint32_t kStepBytes = NB * 256 + 32;
    static_assert(KC * kStepBytes <= 2304, "scratch");
    const int j = lane >> 2;  // this lane's eight elements belong to k-step j
#pragma unroll
    for (int ch = 0; ch < 8 / KC; ++ch) {
        __syncwarp();
        if (j / KC == ch) {
            const uint32_t base = scratch + (uint32_t)(j - ch * KC) * kStepBytes;
#pragma unroll
            for (int m = 0; m < MC; ++m) {
                if (m < p.M) {
#pragma unroll
                    for (int pl = 0; pl < kPlanes; ++pl) {
                        const int col = pl * MC + m;  // column set col / 8, column col % 8
                        const uint32_t at = base + (uint32_t)(col >> 3) * 256u + (uint32_t)(col & 7) * 32u;
                        if constexpr (QmFmt<FMT>::pair8) {  // thread t multiplies k 8t .. 8t+7
                            asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(at + 8u * t), "r"(w[m][pl][0]), "r"(w[m][pl][1]) : "memory");
                        } else {  // thread t multiplies k 4t .. 4t+3 and 16+4t .. 16+4t+3
                            const uint32_t o = at + 16u * (uint32_t)(t & 1) + 4u * (uint32_t)(t >> 1);
                            sts32(o, w[m][pl][0]);
                            sts32(o + 8u, w[m][pl][1]);
                        }
                    }
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int jc = 0; jc < KC; ++jc)
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) x.b[ch * KC + jc][nb] = lds64(scratch + (uint32_t)jc * kStepBytes + (uint32_t)nb * 256u + 8u * (uint32_t)lane);
    }
    __syncwarp();
    return left;
}

template <int FMT, int MC, int NB>
__global__ void __launch_bounds__(kMbMaxWarps * 32, 1) gemv_mb_kernel(const __grid_constant__ MbParams p) {
    using F = QmFmt<FMT>;
    constexpr int NS = F::stages;
    constexpr uint32_t kStage = kQmTile * F::stride;
    static_assert(kStage >= 2304, "a ring stage doubles as the activations' scratch memory");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 127u) & ~127u;
    __shared__ uint64_t bar_part[2];
    __shared__ int abort_flag;
    __shared__ uint32_t left;  // activation rows for the plain loop

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int nw = p.nwk * p.rg, rgi = warp / p.nwk, wk = warp - rgi * p.nwk;
    const int cta = (int)blockIdx.x;
    const int row_begin = cta * p.row_q + min(cta, p.row_r), n_rows = p.row_q + (cta < p.row_r ? 1 : 0);
    const int iters = (n_rows + kQmTile * p.rg - 1) / (kQmTile * p.rg), steps = iters * p.phases;
    const uint32_t ring = sbase + (uint32_t)(warp * NS) * kStage;
    const uint8_t* ring_p = smem_raw + (ring - smem_u32(smem_raw));
    const uint64_t wait_limit = p.wait_limit_us ? (uint64_t)p.wait_limit_us * 1000ull : kWaitLimitNs;

    if (tid == 0) {
        abort_flag = 0;
        left = 0;
        mbar_init(smem_u32(&bar_part[0]), nw);
        mbar_init(smem_u32(&bar_part[1]), nw);
        fence_mbar_init();
    }
    grid_dep_launch();

    // The next tile to fetch: phase ip, iteration ii, the ring's slot islot; isrc: this lane's row g of it.
    int ip = 0, ii = 0, islot = 0;
    const size_t tile_step = (size_t)(kQmTile * p.rg) * p.row_bytes, row8 = (size_t)8 * p.row_bytes;
    const uint8_t* const src0 = p.W + (size_t)(row_begin + rgi * kQmTile + g) * p.row_bytes + (size_t)wk * F::bytes;
    const uint8_t* isrc = src0;
    auto issue = [&] {
        if (ip < p.phases) {
            if (ip * p.nwk + wk < p.nblk) {
                const uint32_t dst = ring + (uint32_t)islot * kStage + (uint32_t)(g * F::stride);
                const int r = (ii * p.rg + rgi) * kQmTile + g;
                if (r < n_rows) qm_copy_row<FMT>(dst, isrc, t);
                if (r + 8 < n_rows) qm_copy_row<FMT>(dst + 8u * F::stride, isrc + row8, t);
            }
            isrc += tile_step;
            if (++ii == iters) {
                ii = 0;
                ++ip;
                isrc = src0 + (size_t)(ip * p.nwk) * F::bytes;
            }
        }
        cp_async_commit();
        if (++islot == NS) islot = 0;
    };
    if (!p.early_w) {
        // The predecessor may be what writes the weights: until it is done only the L2 is told about the first tiles.
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ((i >> 1) * p.rg + rgi) * kQmTile + g + 8 * (i & 1);
            if (r < n_rows && 64 * t < F::bytes) prefetch_l2_line(p.W + (size_t)(row_begin + r) * p.row_bytes + (size_t)wk * F::bytes + 64 * t);
        }
        grid_dep_wait();
    }
#pragma unroll
    for (int s = 0; s < NS - 1; ++s) issue();
    if (p.early_w) grid_dep_wait();
    __syncthreads();  // the barriers exist

    const uint32_t part = sbase + (uint32_t)p.off_part, yacc = sbase + (uint32_t)p.off_yacc;
    // Adds up the partial sums of step (phase rp, iteration ri): `tpo` threads per output, fixed order. Which outputs a
    // thread takes part in - row `o_row` of row group `o_g`, activation row `o_m` - is the same in every step.
    int rp = 0, ri = 0;
    const int tpo_log = 31 - __clz(p.tpo), sub = tid & (p.tpo - 1), per_pass = (nw * 32) >> tpo_log, n_out = kQmTile * p.rg * p.M;
    const int o_first = tid >> tpo_log, o_gm = o_first >> 4;
    const int g_first = o_gm / p.M, m_first = o_gm - g_first * p.M;
    float odd = 0.f;  // not zero once one of the thread's results is not finite: an infinite scale, or more than FP32 holds on the way
    auto reduce = [&](uint32_t buf) {
        int gr = g_first, m = m_first;
        for (int base = 0; base < n_out; base += per_pass) {
            const int o = base + o_first, row = o & (kQmTile - 1);
            if (base > 0) {
                gr = (o >> 4) / p.M;
                m = (o >> 4) - gr * p.M;
            }
            const bool mine = o < n_out;
            float s = 0.f;
            if (mine) {
                uint32_t at = buf + (uint32_t)(((gr * p.nwk + sub) * kQmTile + row) * 8 + m) * 4u;
                for (int w = sub; w < p.nwk; w += p.tpo, at += (uint32_t)p.tpo * 512u) {
                    float c = __uint_as_float(lds32i<0>(at));
                    if constexpr (MC == 4) c = fmaf(256.f, __uint_as_float(lds32i<16>(at)), c);
                    if constexpr (MC == 1) {
                        const uint4 q = lds128i<0>(at), h = lds128i<16>(at);
                        const uint32_t col[8] = {q.x, q.y, q.z, q.w, h.x, h.y, h.z, h.w};
#pragma unroll
                        for (int i = 1; i < 8; ++i) c = fmaf(c, 0.00390625f, __uint_as_float(col[i]));
                    }
                    if constexpr (MC == 2) {
                        const float c1 = __uint_as_float(lds32i<8>(at)), c2 = __uint_as_float(lds32i<16>(at)), c3 = __uint_as_float(lds32i<24>(at));
                        c = fmaf(256.f, fmaf(256.f, fmaf(256.f, c3, c2), c1), c);
                    }
                    s += c;
                }
            }
            for (int d = p.tpo >> 1; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
            const int r = (ri * p.rg + gr) * kQmTile + row;
            if (mine && sub == 0 && r < n_rows) {
                const uint32_t ya = yacc + (uint32_t)(r * p.M + m) * 4u;
                if (rp > 0) s += __uint_as_float(lds32i<0>(ya));
                if (rp + 1 < p.phases) sts32(ya, __float_as_uint(s));  // read by this thread alone
                else {
                    odd = fmaf(s, 0.f, odd);
                    qm_store(p.Y, p.y_dtype, (size_t)m * p.N + row_begin + r, s + qm_bias(p.bias, p.x_dtype, row_begin + r));
                }
            }
        }
        if (++ri == iters) { ri = 0; ++rp; }
    };

    MbX<NB> x;
    int ph = 0, it = 0, slot = 0;
    bool live = true;
    for (int step = 0; step < steps; ++step) {
        const int blk = ph * p.nwk + wk;
        if (it == 0 && blk < p.nblk) {
            // the slot of the tile before (at the start: the ring's last) is free until the next issue
            const uint32_t rows = mb_stage_x<FMT, MC, NB>(p, blk, ring + (uint32_t)islot * kStage, lane, x);
            if (rows && lane == 0) atomicOr(&left, rows);
        }
        issue();
        cp_async_wait<NS - 1>();
        __syncwarp();
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (blk < p.nblk && (it * p.rg + rgi) * kQmTile < n_rows) {
            const uint8_t* slot_a = ring_p + slot * kStage + g * F::stride;
            const uint8_t* row_a = src0 + (size_t)it * tile_step + (size_t)(ph * p.nwk) * F::bytes;
            const QmRow ra = qm_row<FMT>(slot_a, row_a), rb = qm_row<FMT>(slot_a + 8 * F::stride, row_a + row8);
            mb_block<FMT, MC, NB>(ra, rb, t, x, v);
        }
        const int b = step & 1;
        if (step > 0 && live)
            live = wait_or_abort(smem_u32(&bar_part[b ^ 1]), ((step - 1) >> 1) & 1, &abort_flag, p.status, kDevTimeoutFull, wait_limit);
        const uint32_t mine = part + (uint32_t)(b * nw + warp) * 512u + (uint32_t)(g * 32 + t * 8);
        asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(mine), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])) : "memory");
        asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(mine + 256u), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])) : "memory");
        __syncwarp();
        if (step > 0) reduce(part + (uint32_t)((b ^ 1) * nw) * 512u);
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_part[b]));
        if (++slot == NS) slot = 0;
        if (++it == iters) { it = 0; ++ph; }
    }
    if (steps > 0) {
        const int b = (steps - 1) & 1;
        if (live) live = wait_or_abort(smem_u32(&bar_part[b]), ((steps - 1) >> 1) & 1, &abort_flag, p.status, kDevTimeoutFull, wait_limit);
        __syncwarp();
        reduce(part + (uint32_t)(b * nw) * 512u);
    }
    if (!(odd == 0.f)) atomicOr(&left, (1u << p.M) - 1u);
    __syncthreads();
    if (left) qm_plain_rows<FMT>(p.W, p.X, p.x_dtype, p.bias, p.Y, p.y_dtype, 0, left, p.N, p.K, p.row_bytes, row_begin, n_rows);
}

// ---- host side ------------------------------------------------------------------------

// 1: the calls that gain by it (mb_wanted), 2: every call it can run, 0: none
static int g_opt_mb = 1;
void mb_set_enabled(int v) { g_opt_mb = v < 0 ? 0 : (v > 2 ? 2 : v); }
int mb_get_enabled() { return g_opt_mb; }
int dp_get_wait_limit_us();

template <int FMT, int MC, int NB>
static int launch_mb(const MbParams& p, int grid, size_t smem, cudaStream_t st) {
    auto kern = gemv_mb_kernel<FMT, MC, NB>;
    static bool configured[64] = {};
    int dev = 0;
    B200Q_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        B200Q_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 512));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    B200Q_CUDA_TRY(launch_dep(pdl_option() >= 0, kern, dim3((unsigned)grid), dim3((unsigned)(32 * p.nwk * p.rg)), smem, st, p));
    return B200Q_OK;
}

template <int FMT>
static int launch_mb_f(MbParams& p, int sms, cudaStream_t st, bool* taken) {
    using F = QmFmt<FMT>;
    p.nblk = p.K / 256;
    p.row_bytes = p.nblk * F::bytes;
    int grid = stream_get_option(3) > 0 ? stream_get_option(3) : sms;
    if (grid > p.N) grid = p.N;
    p.row_q = p.N / grid;
    p.row_r = p.N % grid;
    const int rows = p.row_q + (p.row_r ? 1 : 0);
    // How the CTA's warps are laid out over K and rows: the fewest tile steps per warp, where staging a phase's
    // activations counts as two, then the most warps.
    constexpr size_t kSmem = 227 * 1024 - 1024;
    size_t smem = 0;
    int best = 0;
    for (int nwk = 1; nwk <= kMbMaxWarps && nwk <= p.nblk; ++nwk) {
        const int phases = (p.nblk + nwk - 1) / nwk;
        for (int rg = kMbMaxWarps / nwk; rg >= 1; --rg) {
            const int iters = (rows + kQmTile * rg - 1) / (kQmTile * rg), nw = nwk * rg;
            if (rg > 1 && kQmTile * (rg - 1) >= rows) continue;  // a row group without rows
            const size_t off_part = (size_t)nw * F::stages * kQmTile * F::stride, off_yacc = off_part + 2 * (size_t)nw * 512;
            const size_t need = 128 + off_yacc + (phases > 1 ? (size_t)rows * p.M * 4 : 0);
            if (need > kSmem) continue;
            const int cost = (phases * (iters + 2)) * 64 - nw;
            if (best && cost >= best) continue;
            best = cost;
            p.nwk = nwk;
            p.rg = rg;
            p.phases = phases;
            p.off_part = (int)off_part;
            p.off_yacc = (int)off_yacc;
            smem = need;
        }
    }
    if (!best) return B200Q_OK;
    const int threads = 32 * p.nwk * p.rg, n_out = kQmTile * p.rg * p.M;
    p.tpo = 1;
    while (p.tpo < 32 && p.tpo < p.nwk && 2 * p.tpo * n_out <= threads) p.tpo *= 2;
    *taken = true;
    // One row of FP32: eight planes, whose cost is their staging (Q5_K 14336 x 4096 18.2 us, with four planes 18.1; 1024 x 4096 5.2, with four
    // 4.4); four would send a token with one channel a thousand times the others to the plain loop. 16-bit values hardly need more than four.
    if (p.M == 1 && p.x_dtype == B200Q_DT_F32) return launch_mb<FMT, 1, 1>(p, grid, smem, st);
    if (p.M <= 2) return launch_mb<FMT, 2, 1>(p, grid, smem, st);
    if (p.M <= 4) return launch_mb<FMT, 4, 2>(p, grid, smem, st);
    return launch_mb<FMT, 8, 4>(p, grid, smem, st);
}

// Launches the kernel when it takes the call (*taken = true): whole 256-element pieces, weights on a 16-byte
// boundary (Q6_K: any even address).
int launch_gemv_mb(int fmt, const void* W, const void* X, int x_dtype, const void* bias, void* Y, int y_dtype, int M, int N, int K,
                   int sms, int* status, cudaStream_t st, bool* taken) {
    *taken = false;
    if (!g_opt_mb || M < 1 || M > 8 || N < 1 || K < 256 || K % 256 != 0) return B200Q_OK;
    if (fmt != kQ6_K && (reinterpret_cast<uintptr_t>(W) & 15) != 0) return B200Q_OK;
    MbParams p = {};
    p.W = static_cast<const uint8_t*>(W);
    p.X = X;
    p.bias = bias;
    p.Y = Y;
    p.status = status;
    p.M = M;
    p.N = N;
    p.K = K;
    p.x_dtype = x_dtype;
    p.y_dtype = y_dtype;
    p.early_w = pdl_option() > 0;
    p.wait_limit_us = (unsigned int)dp_get_wait_limit_us();
    switch (fmt) {
        case kQ5_K: return launch_mb_f<kQ5_K>(p, sms, st, taken);
        case kQ6_K: return launch_mb_f<kQ6_K>(p, sms, st, taken);
        case kQ4_0: return launch_mb_f<kQ4_0>(p, sms, st, taken);
    }
    return B200Q_OK;
}

}  // namespace b200q

// Decode GEMV on warp-level FP16 / BF16 MMA for activations of these types, 1..8 rows, every block format, K a multiple of 256 (sm_100a):
// Y(M, N) = X(M, K) * decode(W(N, K))^T with FP32-class accuracy, at nearly the same time for any M.
//
// The activations are multiplied as they lie in memory: an FP16 or BF16 value is an MMA operand, so there is no staging pass, no scale and
// no rounding. The weights' quants become integers of the same type in a mask, a byte permute and a packed subtraction per two (their offsets -
// 32 in Q6_K, 128 in Q8_0, 8 in Q4_0 - come off in the same subtraction), all exact. (Q8_0's eight bits do not fit BF16's seven of mantissa: they go as two operands, the high nibble times 16
// less 128 and the low one, into the same sums.)
// Each sub-block's products are summed on the tensor cores in FP32 and multiplied by its scale in FP32 (four FMA per 16 x 8 x 32
// products). The minimums of Q4_K / Q5_K go through the same B fragments: an MMA whose A operand is the sub-block's 6-bit min in
// every lane accumulates sum(m * x) over a block, one FMA with dmin per block.
// A k-step of 16 rows x 32 k is two (with mins four) MMAs and some eighty instructions whatever M is, half of them on the half-rate integer
// pipe, against the 12 cycles that its bytes take from memory. Six rows of 14336 x 4096 Q4_K: 18.1 us, 28 % of the memory's rate, IPC 2.05, no pipe
// above 40 %; 32000 x 4096 32.7 us, 35 %. So a call of few rows per SM costs little more than a launch, and long matrices stay with the
// kernels that have fewer instructions per weight where there are any; 20 and 24 warps instead of 14 are no faster.
//
// A CTA owns an even share of the rows, up to eight 16-row tiles at a time, and its warps are tiles x blocks: a stage holds as many
// neighbouring 256-element blocks of the rows (and of X) as there are warps per tile, each warp multiplies one of them, and the tile's
// warps add up at the end of the rows in a fixed order. So every warp has eight k-steps of independent work between two CTA
// barriers (the staged form's largest stall) however few rows there are (with stages of one block, shared by sub-blocks, 4096 x 14336 took 33 us instead of 17.6). Stages
// are fetched with cp.async up to five ahead. Where the rows take many steps and the activations are short they are kept in shared memory
// whole, every warp has a ring of its own and no barrier is left in the loop.
// Results that are not finite are computed again in plain FP32 (qm_plain_rows): 0 * inf on a masked quant is not what the
// dequantised weight gives.
//
// Takes the place of brotensor's decode GEMVs (src/cuda/q4k.cu:159-224, q6k.cu:117-176, q8_0.cu:75-138) and of the per-row loop of its
// batched ops for small B (q4k.cu:413-418).
#include "quant_mma.cuh"

namespace b200q {

constexpr int kHmMaxWarps = 16;
constexpr int kHmMaxTiles = 8;  // 16-row tiles of a CTA at a time
constexpr int kHmMaxStages = 6;
constexpr int kHmResident = 32768;  // activations (M * K) that are kept in shared memory for the whole launch

struct HmParams {
    const uint8_t* W;
    const uint8_t* X;
    const void* bias;
    void* Y;
    int M, N, K, y_dtype;
    int row_bytes, nblk;
    int mt, kg;       // row tiles at a time, blocks per stage: the CTA has mt * kg warps, one per (tile, block)
    int k_stages;     // ceil(nblk / kg)
    int n_stages, stage_bytes, off_x, off_red;
    int row_q, row_r;  // CTA b owns row_q + (b < row_r) rows
};

__device__ __forceinline__ uint32_t sub_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// Two bytes of a word (`sel`: where they go) as integers of the activations' type less `off`: they go into the mantissas of two
// halves that hold 1024 (FP16) or 128 (BF16; bytes below 128), which come off together with the offset, exactly.
template <bool BF>
__device__ __forceinline__ uint32_t hm_halves(uint32_t w, uint32_t sel, uint32_t off) {
    if constexpr (BF) {
        return sub_bf16x2(__byte_perm(w, 0x43u, sel), 0x43004300u + off * 0x10001u);
    } else {
        return hsub2_u32(__byte_perm(w, 0x64u, sel), 0x64006400u + off * 0x10001u);
    }
}
template <bool BF>
__device__ __forceinline__ uint32_t halves_lo(uint32_t w, uint32_t off) { return hm_halves<BF>(w, 0x4140, off); }
template <bool BF>
__device__ __forceinline__ uint32_t halves_hi(uint32_t w, uint32_t off) { return hm_halves<BF>(w, 0x4342, off); }

// Quants of sub-block s of one row as FP16 integers, two neighbouring elements per register. Q4_K's odd sub-blocks: 16 q (FP16). HIGH: the second operand of Q8_0 in BF16.
template <int FMT, bool BF, bool HIGH = false>
__device__ __forceinline__ void hm_quants(const QmRow& r, int s, int t, uint32_t (&a)[4]) {
    if constexpr (FMT == kQ4_K) {
        const uint2 w = ls64(r.p + 16 + 32 * (s >> 1) + 8 * t);
        const uint32_t mask = (!BF && (s & 1)) ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
        const uint32_t x = ((BF && (s & 1)) ? w.x >> 4 : w.x) & mask, y = ((BF && (s & 1)) ? w.y >> 4 : w.y) & mask;
        a[0] = halves_lo<BF>(x, 0);
        a[1] = halves_hi<BF>(x, 0);
        a[2] = halves_lo<BF>(y, 0);
        a[3] = halves_hi<BF>(y, 0);
    } else if constexpr (FMT == kQ5_K) {
        const uint2 w = ls64(r.p + 48 + 32 * (s >> 1) + 8 * t), h = ls64(r.p + 16 + 8 * t);
        const uint32_t x = ((w.x >> (4 * (s & 1))) & 0x0F0F0F0Fu) | (((h.x >> s) & 0x01010101u) << 4);
        const uint32_t y = ((w.y >> (4 * (s & 1))) & 0x0F0F0F0Fu) | (((h.y >> s) & 0x01010101u) << 4);
        a[0] = halves_lo<BF>(x, 0);
        a[1] = halves_hi<BF>(x, 0);
        a[2] = halves_lo<BF>(y, 0);
        a[3] = halves_hi<BF>(y, 0);
    } else if constexpr (FMT == kQ6_K) {
        const int G = s >> 2, Q = s & 3;  // half block, quad
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t w = qm_word(r, 64 * G + 32 * (Q & 1) + 16 * h + 4 * t), b = qm_word(r, 128 + 32 * G + 16 * h + 4 * t);
            const uint32_t six = ((w >> (4 * (Q >> 1))) & 0x0F0F0F0Fu) | (((b >> (2 * Q)) & 0x03030303u) << 4);
            a[2 * h] = halves_lo<BF>(six, 32);
            a[2 * h + 1] = halves_hi<BF>(six, 32);
        }
    } else if constexpr (FMT == kQ8_0) {
        const uint8_t* p = r.p + 34 * s + 4 * t;
        uint32_t w[2];
        if (s & 1) {
            w[0] = ls32(p + 2);
            w[1] = ls32(p + 18);
        } else {  // quants two bytes behind a word boundary
            w[0] = __funnelshift_r(ls32(p), ls32(p + 4), 16);
            w[1] = __funnelshift_r(ls32(p + 16), ls32(p + 20), 16);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t u = w[h] ^ 0x80808080u;  // q + 128
            if constexpr (BF && HIGH) {  // halves that hold 2048 count sixteens
                const uint32_t n = (u >> 4) & 0x0F0F0F0Fu;
                a[2 * h] = sub_bf16x2(__byte_perm(n, 0x45u, 0x4140), 0x45084508u);
                a[2 * h + 1] = sub_bf16x2(__byte_perm(n, 0x45u, 0x4342), 0x45084508u);
            } else if constexpr (BF) {
                a[2 * h] = halves_lo<BF>(u & 0x0F0F0F0Fu, 0);
                a[2 * h + 1] = halves_hi<BF>(u & 0x0F0F0F0Fu, 0);
            } else {
                a[2 * h] = halves_lo<BF>(u, 128);
                a[2 * h + 1] = halves_hi<BF>(u, 128);
            }
        }
    } else {  // Q4_0: low nibbles are elements 0..15, high ones 16..31
        const uint8_t* p = r.p + 18 * s + 4 * t;
        const uint32_t w = (s & 1) ? ls32(p + 2) : __funnelshift_r(ls32(p), ls32(p + 4), 16);
        const uint32_t lo = w & 0x0F0F0F0Fu, hi = (w >> 4) & 0x0F0F0F0Fu;
        a[0] = halves_lo<BF>(lo, 8);
        a[1] = halves_hi<BF>(lo, 8);
        a[2] = halves_lo<BF>(hi, 8);
        a[3] = halves_hi<BF>(hi, 8);
    }
}

// Scales of sub-block s of one row (over 16 for 16 q): f[0] for the first sixteen k, f[1] for the others (Q6_K).
template <int FMT, bool BF>
__device__ __forceinline__ void hm_scales(const QmRow& r, float d, uint32_t sc_lo, uint32_t sc_hi, int s, float (&f)[2]) {
    if constexpr (FMT == kQ4_K || FMT == kQ5_K) {
        f[0] = f[1] = d * byte_to_f32(s < 4 ? sc_lo : sc_hi, s & 3) * ((FMT == kQ4_K && !BF && (s & 1)) ? 0.0625f : 1.f);
    } else if constexpr (FMT == kQ6_K) {
        const uint32_t w = qm_word(r, 192 + 4 * (s >> 1)) ^ 0x80808080u;  // int8 + 128
        f[0] = d * (byte_to_f32(w, 2 * (s & 1)) - 128.f);
        f[1] = d * (byte_to_f32(w, 2 * (s & 1) + 1) - 128.f);
    } else {
        f[0] = f[1] = h2f(ls16(r.p + (FMT == kQ8_0 ? 34 : 18) * s));
    }
}

// XRES: the activations are short enough to lie in shared memory whole (M * K <= kHmResident). Then a warp needs nothing but its own copies
// and the warps run without a barrier until the rows are done.
template <int FMT, bool BF, bool XRES>
__global__ void __launch_bounds__(kHmMaxWarps * 32, 1) gemv_hm_kernel(const __grid_constant__ HmParams p) {
    using F = QmFmt<FMT>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int nonfinite;
    const uint32_t sbase = (smem_u32(smem_raw) + 127u) & ~127u;
    const uint8_t* smem = smem_raw + (sbase - smem_u32(smem_raw));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int ki = warp / p.mt, mi = warp - ki * p.mt;
    const int cta = (int)blockIdx.x;
    const int row_begin = cta * p.row_q + min(cta, p.row_r), n_rows = p.row_q + (cta < p.row_r ? 1 : 0);
    const int rows_it = kQmTile * p.mt, iters = (n_rows + rows_it - 1) / rows_it, steps = iters * p.k_stages;
    if (tid == 0) nonfinite = 0;
    grid_dep_launch();

    // A warp copies what it multiplies - rows g and g + 8 of its tile, four threads each, of its block - and the first tile's warps
    // the activations of their block, a row of X per instruction. The 16-byte chunks of X are rotated so that the threads that read
    // together - 16 bytes each from two rows, or 8 bytes each from four - find them in different banks.
    constexpr uint32_t kTileBytes = kQmTile * F::stride;
    // a slot's bytes of this lane's row g: with XRES in the warp's own ring, else in the CTA's
    const uint32_t slot_bytes = XRES ? kTileBytes : (uint32_t)p.stage_bytes;
    const uint32_t my_rows = (XRES ? (uint32_t)(warp * p.n_stages) : (uint32_t)(ki * p.mt + mi)) * kTileBytes + (uint32_t)(g * F::stride), my_x = (uint32_t)p.off_x + (uint32_t)(ki * p.M * 512);
    const size_t row8 = (size_t)8 * p.row_bytes, k_step = (size_t)p.kg * F::bytes, it_step = (size_t)rows_it * p.row_bytes;
    const uint8_t* const src0 = p.W + (size_t)(row_begin + mi * kQmTile + g) * p.row_bytes + (size_t)ki * F::bytes;
    const uint8_t* const x0 = p.X + 512 * (size_t)ki + 16 * lane;
    int ii = 0, is = 0, islot = 0;
    const uint8_t *isrc = src0, *xsrc = x0;
    auto issue = [&] {
        if (ii < iters) {
            if (is * p.kg + ki < p.nblk) {
                const uint32_t st = sbase + (uint32_t)islot * slot_bytes;
                const int r = ii * rows_it + mi * kQmTile + g;
                if (r < n_rows) qm_copy_row<FMT>(st + my_rows, isrc, t);
                if (r + 8 < n_rows) qm_copy_row<FMT>(st + my_rows + 8u * F::stride, isrc + row8, t);
                if (!XRES && mi == 0) {
                    const uint8_t* x = xsrc;
                    for (int m = 0; m < p.M; ++m, x += 2 * (size_t)p.K) {
                        const uint32_t sw = F::pair8 ? (uint32_t)(m & 1) << 2 : (uint32_t)(m & 3) << 1;
                        cp_async16(st + my_x + (uint32_t)(m * 512) + (((uint32_t)lane ^ sw) << 4), x);
                    }
                }
            }
            isrc += k_step;
            xsrc += 512 * (size_t)p.kg;
            if (++is == p.k_stages) {
                is = 0;
                ++ii;
                isrc = src0 + (size_t)ii * it_step;
                xsrc = x0;
            }
        }
        cp_async_commit();
        if (++islot == p.n_stages) islot = 0;
    };
    // Until the predecessor is done only the L2 is told about the first stage.
    if (ki < p.nblk && 64 * t < F::bytes) {
        if (mi * kQmTile + g < n_rows) prefetch_l2_line(src0 + 64 * t);
        if (mi * kQmTile + g + 8 < n_rows) prefetch_l2_line(src0 + row8 + 64 * t);
    }
    grid_dep_wait();
    for (int s = 0; s < p.n_stages - 1; ++s) issue();
    if constexpr (XRES) {
        for (int i = warp; i < p.nblk * p.M; i += p.mt * p.kg) {  // row m of block b
            const int b = i / p.M, m = i - b * p.M;
            const uint32_t sw = F::pair8 ? (uint32_t)(m & 1) << 2 : (uint32_t)(m & 3) << 1;
            cp_async16(sbase + (uint32_t)p.off_x + (uint32_t)(i * 512) + (((uint32_t)lane ^ sw) << 4), p.X + ((size_t)m * p.K + 256 * (size_t)b) * 2 + 16 * lane);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
    }

    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    int slot = 0, it = 0, ks = 0;
    const uint8_t* rsrc = src0;  // the warp's row g in memory (Q6_K: its alignment)
    for (int step = 0; step < steps; ++step) {
        switch (p.n_stages) {
            case 6: cp_async_wait<4>(); break;
            case 5: cp_async_wait<3>(); break;
            case 4: cp_async_wait<2>(); break;
            case 3: cp_async_wait<1>(); break;
            default: cp_async_wait<0>(); break;
        }
        // the stage has landed for everybody who reads it, and everybody is done with the slot filled next
        if constexpr (XRES) __syncwarp();
        else __syncthreads();
        issue();
        const int r0 = it * rows_it + mi * kQmTile;
        if (r0 < n_rows && ks * p.kg + ki < p.nblk) {
            const uint8_t* st = smem + slot * slot_bytes;
            const QmRow ra = qm_row<FMT>(st + my_rows, rsrc), rb = qm_row<FMT>(st + my_rows + 8 * F::stride, rsrc + row8);
            float dA = 0.f, dB = 0.f, mA = 0.f, mB = 0.f;
            uint32_t sc[2][2] = {{0, 0}, {0, 0}}, mn[2][2] = {{0, 0}, {0, 0}};
            if constexpr (F::mins) {
                const uint4 hA = ls128(ra.p), hB = ls128(rb.p);
                sc[0][0] = k_scales_lo(hA); sc[0][1] = k_scales_hi(hA); sc[1][0] = k_scales_lo(hB); sc[1][1] = k_scales_hi(hB);
                mn[0][0] = k_mins_lo(hA); mn[0][1] = k_mins_hi(hA); mn[1][0] = k_mins_lo(hB); mn[1][1] = k_mins_hi(hB);
                dA = h2f(hA.x & 0xFFFFu); dB = h2f(hB.x & 0xFFFFu);
                mA = h2f(hA.x >> 16); mB = h2f(hB.x >> 16);
            } else if constexpr (FMT == kQ6_K) {
                dA = h2f((ls32(ra.p + 208) >> ra.sh) & 0xFFFFu);
                dB = h2f((ls32(rb.p + 208) >> rb.sh) & 0xFFFFu);
            }
            const uint8_t* xrow = XRES ? smem + p.off_x + ((ks * p.kg + ki) * p.M + g) * 512 : st + my_x + g * 512;
            float cm[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                uint32_t x[4];
                if constexpr (F::pair8) {
                    const uint4 v = ls128(xrow + (((4 * s + t) ^ ((g & 1) << 2)) << 4));
                    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
                } else {
                    const uint2 v = ls64(xrow + (((4 * s + (t >> 1)) ^ ((g & 3) << 1)) << 4) + 8 * (t & 1));
                    const uint2 w = ls64(xrow + (((4 * s + 2 + (t >> 1)) ^ ((g & 3) << 1)) << 4) + 8 * (t & 1));
                    x[0] = v.x; x[1] = v.y; x[2] = w.x; x[3] = w.y;
                }
                uint32_t a[4], b[4];
                float fA[2], fB[2], c[4];
                hm_quants<FMT, BF>(ra, s, t, a);
                hm_quants<FMT, BF>(rb, s, t, b);
                hm_scales<FMT, BF>(ra, dA, sc[0][0], sc[0][1], s, fA);
                hm_scales<FMT, BF>(rb, dB, sc[1][0], sc[1][1], s, fB);
                qm_mma_zero<BF>(c, a[0], b[0], a[1], b[1], x[0], x[1]);
                if constexpr (FMT == kQ6_K) {
                    float c2[4];
                    qm_mma_zero<BF>(c2, a[2], b[2], a[3], b[3], x[2], x[3]);
                    acc[0] = fmaf(fA[1], c2[0], acc[0]);
                    acc[1] = fmaf(fA[1], c2[1], acc[1]);
                    acc[2] = fmaf(fB[1], c2[2], acc[2]);
                    acc[3] = fmaf(fB[1], c2[3], acc[3]);
                } else {
                    qm_mma<BF>(c, a[2], b[2], a[3], b[3], x[2], x[3]);
                }
                if constexpr (FMT == kQ8_0 && BF) {
                    hm_quants<FMT, BF, true>(ra, s, t, a);
                    hm_quants<FMT, BF, true>(rb, s, t, b);
                    qm_mma<BF>(c, a[0], b[0], a[1], b[1], x[0], x[1]);
                    qm_mma<BF>(c, a[2], b[2], a[3], b[3], x[2], x[3]);
                }
                acc[0] = fmaf(fA[0], c[0], acc[0]);
                acc[1] = fmaf(fA[0], c[1], acc[1]);
                acc[2] = fmaf(fB[0], c[2], acc[2]);
                acc[3] = fmaf(fB[0], c[3], acc[3]);
                if constexpr (F::mins) {
                    const uint32_t sel = 0x4040u | (uint32_t)((s & 3) * 0x101);
                    const uint32_t m0 = hm_halves<BF>(s < 4 ? mn[0][0] : mn[0][1], sel, 0);
                    const uint32_t m1 = hm_halves<BF>(s < 4 ? mn[1][0] : mn[1][1], sel, 0);
                    qm_mma<BF>(cm, m0, m1, m0, m1, x[0], x[1]);
                    qm_mma<BF>(cm, m0, m1, m0, m1, x[2], x[3]);
                }
            }
            if constexpr (F::mins) {
                acc[0] = fmaf(-mA, cm[0], acc[0]);
                acc[1] = fmaf(-mA, cm[1], acc[1]);
                acc[2] = fmaf(-mB, cm[2], acc[2]);
                acc[3] = fmaf(-mB, cm[3], acc[3]);
            }
        }
        if (FMT == kQ6_K) rsrc += k_step;
        if (++slot == p.n_stages) slot = 0;
        if (++ks < p.k_stages) continue;
        // ---- these rows are done: add up the tile's warps (in order), store
        ks = 0;
        if (p.kg > 1) {
            // (two buffers in turn where no stage barrier keeps the next rows' sums from overtaking the reads of these)
            const uint32_t red = sbase + (uint32_t)p.off_red + (uint32_t)(lane * 16) + (XRES && (it & 1) ? (uint32_t)((p.kg - 1) * p.mt * 512) : 0u);
            if (ki > 0)
                sts128(red + (uint32_t)(((ki - 1) * p.mt + mi) * 512),
                       make_uint4(__float_as_uint(acc[0]), __float_as_uint(acc[1]), __float_as_uint(acc[2]), __float_as_uint(acc[3])));
            __syncthreads();
            if (ki == 0)
                for (int k = 1; k < p.kg; ++k) {
                    const uint4 v = lds128i<0>(red + (uint32_t)(((k - 1) * p.mt + mi) * 512));
                    acc[0] += __uint_as_float(v.x);
                    acc[1] += __uint_as_float(v.y);
                    acc[2] += __uint_as_float(v.z);
                    acc[3] += __uint_as_float(v.w);
                }
        }
        if (ki == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + g + 8 * h;
                if (r < n_rows) {
                    const float bv = qm_bias(p.bias, BF ? B200Q_DT_BF16 : B200Q_DT_F16, row_begin + r);
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        if (2 * t + j < p.M) {
                            const float v = acc[2 * h + j];
                            if (!(fabsf(v) <= 3.402823466e38f)) nonfinite = 1;
                            qm_store(p.Y, p.y_dtype, (size_t)(2 * t + j) * p.N + row_begin + r, v + bv);
                        }
                }
            }
        }
        acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
        ++it;
        rsrc = src0 + (size_t)it * it_step;
    }
    __syncthreads();
    if (nonfinite)
        qm_plain_rows<FMT>(p.W, p.X, BF ? B200Q_DT_BF16 : B200Q_DT_F16, p.bias, p.Y, p.y_dtype, 0, (1u << p.M) - 1u, p.N, p.K, p.row_bytes, row_begin, n_rows);
}

// ---- host side ------------------------------------------------------------------------------------------

static int g_opt_hm = 1;
void hm_set_enabled(int v) { g_opt_hm = v < 0 ? 0 : (v > 2 ? 2 : v); }
int hm_get_enabled() { return g_opt_hm; }

template <int FMT, bool BF, bool XRES>
static int launch_hm(const HmParams& p, int grid, size_t smem, cudaStream_t st) {
    auto kern = gemv_hm_kernel<FMT, BF, XRES>;
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

template <int FMT>
static int launch_hm_f(HmParams& p, bool bf, int sms, cudaStream_t st) {
    using F = QmFmt<FMT>;
    p.row_bytes = p.nblk * F::bytes;
    int grid = stream_get_option(3) > 0 ? stream_get_option(3) : sms;
    if (grid > p.N) grid = p.N;
    p.row_q = p.N / grid;
    p.row_r = p.N % grid;
    const int rows = p.row_q + (p.row_r ? 1 : 0), tiles = (rows + kQmTile - 1) / kQmTile;
    const int iters = (tiles + kHmMaxTiles - 1) / kHmMaxTiles;
    p.mt = (tiles + iters - 1) / iters;
    // As many blocks per stage as there are warps left for a tile and as leave room for two stages, the stages of a row as even as they
    // come. (Eight rows of 1024 x 12288 Q8_0 have room for 12 blocks, not 16: 9.0 us, and 16 to 25 on the kernels that took such calls before;
    // holding out for three stages instead costs 2 to 24 % on K = 2560 .. 14336 and gains 2 to 6 % on a few shapes.)
    const size_t budget = 227 * 1024 - 1024 - 256;
    for (int most = kHmMaxWarps / p.mt;; --most) {
        p.k_stages = (p.nblk + most - 1) / most;
        p.kg = (p.nblk + p.k_stages - 1) / p.k_stages;
        // sums of the tile's warps; rows past M of the last block's activations are read, not used: up to 7 x 512 bytes past the stage
        const size_t red = (size_t)(p.kg - 1) * p.mt * 512, tile = (size_t)p.mt * p.kg * kQmTile * F::stride;
        // Activations resident, no stage barrier: 14336 x 4096 Q4_K (8 steps) 18.9 -> 17.2 us, 32000 x 4096 (16) 37.5 -> 31.5, 4096 x 14336 one row (7)
        // 17.5 -> 16.9; but the start waits for all of X, so short runs lose: 4096 x 4096 (2 steps) 6.5 -> 7.2, 2560 x 6912 (4) 8.8 -> 9.3.
        if ((long long)p.M * p.K <= kHmResident && iters * p.k_stages >= 6) {
            const size_t x = (size_t)p.nblk * p.M * 512, tail = 2 * red > 3584 ? 2 * red : 3584;
            p.n_stages = kHmMaxStages;
            while (p.n_stages > 2 && p.n_stages * tile + x + tail > budget) --p.n_stages;
            if (p.n_stages * tile + x + tail <= budget) {
                p.off_x = (int)(p.n_stages * tile);
                p.off_red = p.off_x + (int)x;
                const size_t smem = (size_t)p.off_red + tail + 128;
                return bf ? launch_hm<FMT, true, true>(p, grid, smem, st) : launch_hm<FMT, false, true>(p, grid, smem, st);
            }
        }
        const size_t tail = red > 3584 ? red : 3584;
        p.off_x = (int)tile;
        p.stage_bytes = (p.off_x + p.kg * p.M * 512 + 127) & ~127;
        p.n_stages = kHmMaxStages;
        while (p.n_stages > 2 && (size_t)p.n_stages * p.stage_bytes + tail > budget) --p.n_stages;
        if ((size_t)p.n_stages * p.stage_bytes + tail > budget && most > 1) continue;  // (one block per stage fits: 2 x 39 KB at most)
        p.off_red = p.n_stages * p.stage_bytes;
        const size_t smem = (size_t)p.off_red + tail + 128;
        return bf ? launch_hm<FMT, true, false>(p, grid, smem, st) : launch_hm<FMT, false, false>(p, grid, smem, st);
    }
}

// The calls it takes, and takes in every case: FP16 or BF16 activations, 1..8 rows, K a multiple of 256, weights on a 16-byte boundary
// (Q6_K: any even address).
bool gemv_hm_takes(int fmt, const void* W, int x_dtype, int M, int N, int K) {
    if (!g_opt_hm || x_dtype == B200Q_DT_F32 || M < 1 || M > 8 || N < 1 || K < 256 || K % 256 != 0) return false;
    if (fmt == kQ6_K) return true;
    return (fmt == kQ4_K || fmt == kQ5_K || fmt == kQ8_0 || fmt == kQ4_0) && (reinterpret_cast<uintptr_t>(W) & 15) == 0;
}

int launch_gemv_hm(int fmt, const void* W, const void* X, int x_dtype, const void* bias, void* Y, int y_dtype, int M, int N, int K,
                   int sms, cudaStream_t st, bool* taken) {
    *taken = gemv_hm_takes(fmt, W, x_dtype, M, N, K);
    if (!*taken) return B200Q_OK;
    const bool bf = x_dtype == B200Q_DT_BF16;
    HmParams p = {};
    p.W = static_cast<const uint8_t*>(W);
    p.X = static_cast<const uint8_t*>(X);
    p.bias = bias;
    p.Y = Y;
    p.M = M;
    p.N = N;
    p.K = K;
    p.y_dtype = y_dtype;
    p.nblk = K / 256;
    switch (fmt) {
        case kQ4_K: return launch_hm_f<kQ4_K>(p, bf, sms, st);
        case kQ5_K: return launch_hm_f<kQ5_K>(p, bf, sms, st);
        case kQ6_K: return launch_hm_f<kQ6_K>(p, bf, sms, st);
        case kQ8_0: return launch_hm_f<kQ8_0>(p, bf, sms, st);
        default: return launch_hm_f<kQ4_0>(p, bf, sms, st);
    }
}

}  // namespace b200q

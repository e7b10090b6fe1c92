// The i-quants (IQ2_XXS, IQ2_XS, IQ2_S, IQ3_XXS; block layouts in iquant.cuh) at several activation rows, on the skeleton of row_stream.cuh. Two tables in
// shared memory make a unit of 32 weights:
//   * a 2-bit grid has three magnitudes, so the eight bytes of an entry fit the eight nibbles of one word, each nibble a selector of `prmt` over the
//     magnitudes (selectors 0..2) and their negatives (4..6);
//   * the eight signs of a group are a word with bit 2 of every nibble set where the sign is negative: one XOR with the entry, and two `prmt` give
//     the eight int8 weights;
//   * IQ3_XXS (eight magnitudes, four to an entry) keeps the grid's bytes, and its signs are byte masks m: (g ^ m) + (m & 0x01010101) negates
//     (a grid byte is never 0: no carry).
// The tables are stored once for each of 32 (16, 8) lanes, side by side, so that lanes with different indices read different banks.
#include "common.cuh"
#include "iquant.cuh"
#include "kernels.h"
#include "row_stream.cuh"

namespace lb {
namespace iqr {

// bit j of `s8` -> bit 4 j + 2
__device__ __forceinline__ uint32_t spread_signs(uint32_t s8) {
    uint32_t x = (s8 | s8 << 12) & 0x000F000Fu;
    x = (x | x << 6) & 0x03030303u;
    x = (x | x << 3) & 0x11111111u;
    return x << 2;
}
template <int FMT> struct Format {
    static constexpr int GRID_WORDS = 8192;
    static constexpr int M_MIN = 3, M_MAX = 8;
    static constexpr bool DIRECT = false, AHEAD = true, CHUNKS = false;
    static constexpr bool IQ3 = FMT == FMT_IQ3XXS;
    static constexpr int ENTRIES = iq_grid_bytes(FMT) / (IQ3 ? 4 : 8), COPIES = GRID_WORDS / ENTRIES;  // 32 KB of grid words: 32, 16 (IQ2_XS), 8 (IQ2_S) copies
    static constexpr int SIGNS = FMT == FMT_IQ2S ? 256 : 128, SIGN_COPIES = GRID_WORDS / 2 / SIGNS / (IQ3 ? 2 : 1);
    static constexpr size_t TABLE_BYTES = 6 * GRID_WORDS;
    static constexpr int BB = iq_block_bytes(FMT);
    static __host__ __device__ uint64_t row_bytes(uint32_t k) { return (uint64_t)(k / QK) * BB; }

    static __device__ __forceinline__ void fill(uint8_t *smem, const uint8_t *grid, int tid, int threads) {
        uint32_t *t = (uint32_t *)smem;
        for (int i = tid; i < ENTRIES; i += threads) {
            uint32_t e;
            if constexpr (IQ3) {
                e = ((const uint32_t *)grid)[i];
            } else {  // magnitudes 8, 25, 43: their high nibbles 0, 1, 2 are the selectors
                const uint2 g = ((const uint2 *)grid)[i];
                auto nibbles = [](uint32_t w) {
                    w = (w >> 4) & 0x0F0F0F0Fu;
                    w = (w | w >> 4) & 0x00FF00FFu;
                    return (w | w >> 8) & 0xFFFFu;
                };
                e = nibbles(g.x) | nibbles(g.y) << 16;
            }
#pragma unroll
            for (int c = 0; c < COPIES; c += 4) *(uint4 *)(t + i * COPIES + ((c + 4 * i) & (COPIES - 1))) = make_uint4(e, e, e, e);
        }
        uint32_t *s = (uint32_t *)(smem + 4 * GRID_WORDS);
        for (int i = tid; i < SIGNS; i += threads) {
            const uint32_t s8 = FMT == FMT_IQ2S ? (uint32_t)i : iq_ksign((uint32_t)i);
            if constexpr (IQ3) {
                uint32_t m[2];
#pragma unroll
                for (int h = 0; h < 2; h++) m[h] = prmt(((s8 >> (4 * h)) & 15u) * 0x10204080u, 0u, 0xBA98u);  // sign bit j in the top bit of byte j, replicated
#pragma unroll
                for (int c = 0; c < SIGN_COPIES; c += 2) *(uint4 *)(s + 2 * (i * SIGN_COPIES + ((c + 2 * i) & (SIGN_COPIES - 1)))) = make_uint4(m[0], m[1], m[0], m[1]);
            } else {
                const uint32_t e = spread_signs(s8);
#pragma unroll
                for (int c = 0; c < SIGN_COPIES; c += 4) *(uint4 *)(s + i * SIGN_COPIES + ((c + 4 * i) & (SIGN_COPIES - 1))) = make_uint4(e, e, e, e);
            }
        }
    }

    // Where a lane reads the tables
    struct Tables {
        const uint8_t *grid, *signs;
        __device__ __forceinline__ Tables(const uint8_t *smem, int lane) : grid(smem + (lane & (COPIES - 1)) * 4), signs(smem + 4 * GRID_WORDS + (lane & (SIGN_COPIES - 1)) * (IQ3 ? 8 : 4)) {}
        __device__ __forceinline__ uint32_t entry(uint32_t i) const { return *(const uint32_t *)(grid + i * (COPIES * 4)); }
        __device__ __forceinline__ uint32_t sign(uint32_t i) const { return *(const uint32_t *)(signs + i * (SIGN_COPIES * 4)); }
        __device__ __forceinline__ uint2 masks(uint32_t i) const { return *(const uint2 *)(signs + i * (SIGN_COPIES * 8)); }
    };

    // Lane l takes sub-block l % 8 of every fourth block; its indices lie at `lane_offset` in the row, eight bytes a sub-block (IQ2_S: four).
    static constexpr uint32_t STEP_BYTES = 4 * BB;
    static constexpr int UNIT = FMT == FMT_IQ2S ? 4 : 8;
    static __device__ __forceinline__ uint32_t lane_offset(int lane) { return (lane >> 3) * BB + 2 + UNIT * (lane & 7); }
    struct Raw {
        uint32_t w0, w1, w2;  // XXS, XS, IQ3_XXS: the aligned words around eight bytes of indices (IQ2_XXS: and signs); IQ2_S: index bytes, sign bytes
        uint32_t x, d, sh;    // what else there is; f16 d; how far into w0 the eight bytes start
    };
    static __device__ __forceinline__ Raw none() { return Raw{0u, 0u, 0u, 0u, 0u, 0u}; }
    static __device__ __forceinline__ Raw load(const uint8_t *base, uint32_t at, int lane) {  // base: on a 4-byte boundary
        const uint32_t ib = lane & 7, b = at - 2 - UNIT * ib;
        Raw r = none();
        if constexpr (FMT == FMT_IQ2S) {
            r.w0 = ld32_by16(base + at), r.w1 = ld32_by16(base + (at + 32));
            r.x = (uint32_t)base[b + 66 + ib] | (uint32_t)base[b + 74 + ib] << 8;
        } else {  // (the third word only where it holds any of the eight bytes: a matrix may end behind the second)
            const uint32_t *a = (const uint32_t *)(base + (at & ~3u));
            r.sh = (at & 2u) << 3;
            r.w0 = __ldg(a), r.w1 = __ldg(a + 1);
            if (r.sh) r.w2 = __ldg(a + 2);
            if constexpr (FMT == FMT_IQ2XS) r.x = base[b + 66 + ib];
            if constexpr (IQ3) r.x = ld32_by16(base + (b + 66 + 4 * ib));
        }
        r.d = ld16(base + b);
        return r;
    }

    struct W {
        uint32_t w[8];
        float d;     // the reference's scale: block scale times (0.5 + scale) / 4 (IQ3_XXS: / 2); IQ2_XS, IQ2_S: block scale / 8
        int m0, m1;  // IQ2_XS, IQ2_S: 2 scale + 1 of each half
    };
    // (0.5 + the top four bits of x) / 4 (IQ3_XXS: / 2), exactly: as the low bits of 2^21 (2^22), whose last place is 1/4 (1/2). The whole scale goes into every term:
    // a power of two taken out of the sum would let it overflow where the reference's does not.
    static __device__ __forceinline__ float half_more(uint32_t x) {
        return IQ3 ? xsub(__uint_as_float(x >> 28 | 0x4A800000u), 4194303.75f) : xsub(__uint_as_float(x >> 28 | 0x4A000000u), 2097151.875f);
    }
    static __device__ __forceinline__ W unpack(const Raw &r, const Tables &t) {
        W o;
        const float d = half_bits_to_float(r.d);
        const uint32_t q0 = FMT == FMT_IQ2S ? r.w0 : __funnelshift_r(r.w0, r.w1, r.sh), q1 = FMT == FMT_IQ2S ? r.w1 : __funnelshift_r(r.w1, r.w2, r.sh);
        o.m0 = o.m1 = 0;
        if constexpr (IQ3) {
#pragma unroll
            for (int l = 0; l < 4; l++) {
                const uint32_t q = (l < 2 ? q0 : q1) >> (16 * (l & 1));
                const uint2 m = t.masks((r.x >> (7 * l)) & 127u);
                o.w[2 * l] = (t.entry(q & 255u) ^ m.x) + (m.x & 0x01010101u);
                o.w[2 * l + 1] = (t.entry((q >> 8) & 255u) ^ m.y) + (m.y & 0x01010101u);
            }
            o.d = xmul(d, half_more(r.x));  // (exact: 5 bits times 11)
        } else {
            uint32_t idx[4], sg[4];
            if constexpr (FMT == FMT_IQ2XXS) {
#pragma unroll
                for (int l = 0; l < 4; l++) idx[l] = (q0 >> (8 * l)) & 255u, sg[l] = (q1 >> (7 * l)) & 127u;
                o.d = xmul(d, half_more(q1));
            } else if constexpr (FMT == FMT_IQ2XS) {
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    const uint32_t q = (l < 2 ? q0 : q1) >> (16 * (l & 1));
                    idx[l] = q & 511u, sg[l] = (q >> 9) & 127u;
                }
                o.m0 = 2 * (int)(r.x & 15u) + 1, o.m1 = 2 * (int)(r.x >> 4) + 1;
                o.d = xmul(d, 0.125f);
            } else {
#pragma unroll
                for (int l = 0; l < 4; l++) idx[l] = ((q0 >> (8 * l)) & 255u) | (((r.x >> (2 * l)) & 3u) << 8), sg[l] = (q1 >> (8 * l)) & 255u;
                o.m0 = 2 * (int)((r.x >> 8) & 15u) + 1, o.m1 = 2 * (int)(r.x >> 12) + 1;
                o.d = xmul(d, 0.125f);
            }
#pragma unroll
            for (int l = 0; l < 4; l++) {
                const uint32_t sel = t.entry(idx[l]) ^ t.sign(sg[l]);
                o.w[2 * l] = prmt(0x002B1908u, 0x00D5E7F8u, sel);  // 8, 25, 43; -8, -25, -43
                o.w[2 * l + 1] = prmt(0x002B1908u, 0x00D5E7F8u, sel >> 16);
            }
        }
        return o;
    }
    static __device__ __forceinline__ float dot(const W &w, const uint32_t (&a)[8]) {
        // |sum| <= 32 * 127 * 62 < 2^22: added to the bit pattern of 1.5 * 2^23 it lands in the mantissa, and one exact subtraction makes it a float
        int d0 = FMT == FMT_IQ2XXS || IQ3 ? 0x4B400000 : 0, d1 = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) d0 = __dp4a((int)w.w[i], (int)a[i], d0), d1 = __dp4a((int)w.w[4 + i], (int)a[4 + i], d1);
        if constexpr (FMT == FMT_IQ2XXS || IQ3) return __int_as_float(d0 + d1) - 12582912.0f;
        else return (float)(d0 * w.m0 + d1 * w.m1);  // |sum| <= 32 * 127 * 43 * 31 < 2^24: exact
    }
    static __device__ __forceinline__ void order(uint4 &, uint4 &) {}
};

}  // namespace iqr

bool qgemv_iq_rows_fits(uint32_t rows, uint32_t k) { return rows >= 3 && rows <= 8 && rs::smem_bytes<iqr::Format<FMT_IQ2XXS>>(rows, k, 2, true) <= rs::ACT_SMEM_MAX; }
// Where this kernel beats qgemv_iq.cu's, us there / here. The activations are copied once instead of being read from L1 for every one or two matrix rows; its tables
// cost a CTA some 2 us to fill, which the pre-pass hides. Three rows and K below 2048 do too little to win it back (IQ2_XS 1024 x 1024 3.5 / 4.0, 14336 x 1024
// 8.3 / 8.9; IQ2_XXS 1024 x 2048 5.2 / 4.2; IQ2_XS, whose other kernel is the quickest, 3000 x 2048 5.5 / 5.8, 4096 x 2048 6.3 / 5.8). IQ2_XXS and IQ2_XS else always: 256 x 1024, 4 rows 4.1 / 4.0, 8 rows 6.4 / 5.2; 2048 x 4096, 3 rows 6.6 / 5.4, 4096 x 14336
// 29.6 / 14.0, 14336 x 4096, 8 rows 35.7 / 26.8. IQ2_S and IQ3_XXS unpack in more instructions and lose at three to five rows to the other kernel's two matrix
// rows a warp (28672 x 4096, 3 rows 33.6 / 37.9, 5 rows 45.5 / 46.7; 4096 x 4096, 5 rows 14.4 / 10.5; 28672 x 4096, 6 rows 54.7 / 49.8), IQ3_XXS at five and six also
// where few columns of many steps leave warps idle here (1536 x 4096, 6 rows 7.2 / 7.6, 512 x 8192, 5 rows 6.1 / 6.7; 2048 x 4096, 5 rows 7.7 / 7.4).
bool qgemv_iq_rows_pays(int fmt, uint32_t rows, uint64_t n, uint32_t k, int sm_count) {
    if (rows == 3 && (k < 2048 || (fmt == FMT_IQ2XS && n * k < (8u << 20)))) return false;
    if (fmt == FMT_IQ2XXS || fmt == FMT_IQ2XS) return true;
    if (rows <= 5 && n >= 2 * 32 * (uint64_t)sm_count) return false;
    if (fmt == FMT_IQ3XXS) return !((rows == 5 || rows == 6) && k >= 4096 && n < 12 * (uint64_t)sm_count);
    return rows != 4 || k >= 2048;
}

cudaError_t launch_qgemv_iq_rows(int fmt, const GemvGroup &group, const uint8_t *grid, int force_ks, int sm_count, bool pdl, cudaStream_t stream) {
    switch (fmt) {
        case FMT_IQ2XXS: return rs::launch_group<iqr::Format<FMT_IQ2XXS>>(group, grid, force_ks, sm_count, pdl, stream);
        case FMT_IQ2XS: return rs::launch_group<iqr::Format<FMT_IQ2XS>>(group, grid, force_ks, sm_count, pdl, stream);
        case FMT_IQ2S: return rs::launch_group<iqr::Format<FMT_IQ2S>>(group, grid, force_ks, sm_count, pdl, stream);
        default: return rs::launch_group<iqr::Format<FMT_IQ3XXS>>(group, grid, force_ks, sm_count, pdl, stream);
    }
}

}  // namespace lb

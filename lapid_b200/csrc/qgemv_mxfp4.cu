// Decode GEMV over MXFP4 blocks (ggml `block_mxfp4`, crates/lapid-quant/src/mxfp4.rs: 32 elements in 17 bytes --
// one e8m0 scale byte, then 16 bytes whose low nibbles are elements 0..15 and high nibbles elements 16..31;
// x = KV[nibble] * 2^(e - 128) with KV the doubled e2m1 values) with lapid-cpu's int8-activation arithmetic
// (crates/lapid-cpu/src/mxfp4.rs:38-58):
//
//     acc += d * da_g * f32(sum_32 qa * KV[q])          one activation group per weight block
//
// on the skeleton of row_stream.cuh (its unit is a block). Blocks are 17 bytes long, so they start on any byte boundary: they are fetched as the aligned
// 32-bit words around them and funnel-shifted into place. The four nibbles of a 16-bit half are the codes of elements j, j + 16, j + 1, j + 17 and exactly
// a `prmt` selector over the table of magnitudes; the activations are put into that order once, when they are copied to shared memory.
// One and two rows: bit 3 of a selector nibble replicates the chosen byte's top bit, which no magnitude has, so one `prmt` gives the magnitudes of the positive
// codes and 0 elsewhere, a second, on the word with all the sign bits turned round, those of the negative codes: the sum is the difference of two `dp4a`
// chains, and nothing is spent on signs. From three rows on (K no multiple of 512; the others go to qgemv_mxfp4_mma.cu) the signed values are made once (mxfp4_kv4).
// Before (a row at a time per warp, activations read from L1 for every row, seven operations for four signed values, rows staged through shared memory by 16-byte
// copies where K allowed) -> now, us: 14336 x 4096 17.0 -> 13.3, 28672 x 4096 29.5 -> 20.7, 4096 x 14336 18.9 -> 13.9, 4096 x 4096 6.7 -> 6.3, two rows on 14336 x 4096
// 19.2 -> 16.1, six experts of 2304 x 5120 22.1 -> 15.7, of 5120 x 2304 25.7 -> 18.6, five rows on 4096 x 2880 14.4 -> 10.2. The six experts' 37.6 MB need 5.8 us.
#include "common.cuh"
#include "kernels.h"
#include "row_stream.cuh"

namespace lb {
namespace mx {

template <bool SPLIT> struct Format {  // SPLIT: positive and negative codes apart
    static constexpr int M_MIN = SPLIT ? 1 : 3, M_MAX = SPLIT ? 2 : 8;
    static constexpr bool DIRECT = true, AHEAD = false, CHUNKS = true;
    static constexpr size_t TABLE_BYTES = 0;  // no lookups
    static __device__ __forceinline__ void fill(uint8_t *, const uint8_t *, int, int) {}
    struct Tables {
        __device__ __forceinline__ Tables(const uint8_t *, int) {}
    };
    static constexpr uint32_t STEP_BYTES = 32 * MXFP4_BYTES;
    static __host__ __device__ uint64_t row_bytes(uint32_t k) { return (uint64_t)(k / GROUP) * MXFP4_BYTES; }
    static __device__ __forceinline__ uint32_t lane_offset(int lane) { return lane * MXFP4_BYTES; }
    struct Raw {
        uint32_t w[5], sh;  // the aligned words that hold the block's 17 bytes, each of them some of them; bits before the first
    };
    static __device__ __forceinline__ Raw none() { return Raw{{0u, 0u, 0u, 0u, 0u}, 0u}; }
    static __device__ __forceinline__ Raw load(const uint8_t *base, uint32_t at, int) {
        const uint32_t *a = (const uint32_t *)(base + (at & ~3u));
        Raw r;
#pragma unroll
        for (int i = 0; i < 5; i++) r.w[i] = __ldg(a + i);
        r.sh = (at & 3u) * 8;
        return r;
    }
    struct W {
        uint32_t q[8];  // SPLIT: q[i] the nibbles of four elements (low half) of each kind; else the values
        float d;
    };
    static __device__ __forceinline__ W unpack(const Raw &r, const Tables &) {
        W o;
        o.d = e8m0_half((r.w[0] >> r.sh) & 255u);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t w = __funnelshift_rc(r.w[i], r.w[i + 1], r.sh + 8);  // elements 4i.. (low nibbles), 16 + 4i.. (high nibbles)
            if constexpr (SPLIT) o.q[i] = w, o.q[4 + i] = 0;
            else o.q[2 * i] = mxfp4_kv4(w), o.q[2 * i + 1] = mxfp4_kv4(w >> 16);
        }
        return o;
    }
    static __device__ __forceinline__ float dot(const W &w, const uint32_t (&a)[8]) {
        // |sum| <= 32 * 127 * 12 < 2^22: added to the bit pattern of 1.5 * 2^23 it lands in the mantissa, and one exact subtraction makes it a float
        int pos = 0x4B400000, neg = 0;
        if constexpr (SPLIT) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t p = w.q[i], n = p ^ 0x88888888u;
                pos = __dp4a((int)prmt(0x03020100u, 0x0C080604u, p), (int)a[2 * i], pos);
                neg = __dp4a((int)prmt(0x03020100u, 0x0C080604u, n), (int)a[2 * i], neg);
                pos = __dp4a((int)prmt(0x03020100u, 0x0C080604u, p >> 16), (int)a[2 * i + 1], pos);
                neg = __dp4a((int)prmt(0x03020100u, 0x0C080604u, n >> 16), (int)a[2 * i + 1], neg);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) pos = __dp4a((int)w.q[i], (int)a[i], pos), neg = __dp4a((int)w.q[4 + i], (int)a[4 + i], neg);
        }
        return __int_as_float(SPLIT ? pos - neg : pos + neg) - 12582912.0f;
    }
    // bytes of a group in the order of the nibbles: (0, 16, 1, 17), (2, 18, 3, 19), ...
    static __device__ __forceinline__ void order(uint4 &lo, uint4 &hi) {
        const uint4 l = lo, h = hi;
        lo = make_uint4(prmt(l.x, h.x, 0x5140u), prmt(l.x, h.x, 0x7362u), prmt(l.y, h.y, 0x5140u), prmt(l.y, h.y, 0x7362u));
        hi = make_uint4(prmt(l.z, h.z, 0x5140u), prmt(l.z, h.z, 0x7362u), prmt(l.w, h.w, 0x5140u), prmt(l.w, h.w, 0x7362u));
    }
};

static int g_k_split = 0;  // warps per row: 0: chosen per launch; 1, 2, 4: forced

}  // namespace mx

void qgemv_mxfp4_set_k_split(int ways) { mx::g_k_split = ways == 1 || ways == 2 || ways == 4 ? ways : 0; }

cudaError_t launch_qgemv_mxfp4(const GemvGroup &group, int sm_count, bool pdl, cudaStream_t stream) {
    if (group.count < 1 || group.count > GEMV_GROUP_MAX) return cudaErrorInvalidValue;
    for (int i = 0; i < group.count; i++) {  // members: same rows, k, ids and activations, none of them empty
        const GemvArgs &a = group.item[i];
        if (group.count == 1 && (a.n == 0 || a.rows == 0)) return cudaSuccess;
        if (a.n == 0 || a.k % GROUP != 0 || ((uintptr_t)a.w & 3) != 0 || (a.ids && (a.id_stride & 3))) return cudaErrorInvalidValue;
    }
    if (group.item[0].ids || group.item[0].rows <= 2) return rs::launch_group<mx::Format<true>>(group, nullptr, mx::g_k_split, sm_count, pdl, stream);
    return rs::launch_group<mx::Format<false>>(group, nullptr, mx::g_k_split, sm_count, pdl, stream);
}

}  // namespace lb

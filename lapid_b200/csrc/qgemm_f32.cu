// Exact-f32 quantized GEMM: f32 activations x weights dequantized to f32 with lapid-quant's
// arithmetic, every output accumulated over k = 0..K-1 in order with one fused multiply-add per
// term from a zero accumulator. That is the arithmetic of lapid-cpu's `qdeq` path on x86-64 with
// AVX2+FMA (crates/lapid-cpu/src/matmul/qdeq.rs:57-123, kernels.rs:95-119), so results are
// bit-identical to it. This is the reference-exact path for more than 8 activation rows; the
// tensor-core kernel is the fast one.
//
// Expert-indexed launches (Kernel::MatMulId above decode sizes) run through the same kernel: the
// activation tiles are runs of (token, slot) pairs grouped by expert (moe.cu), a tile looks up its
// expert's matrix, rows are gathered and scattered through the pair table. Every output is still
// the in-order FMA sum over k, i.e. what lapid-cpu's per-expert matmul gives
// (crates/lapid-cpu/src/moe.rs:80-118 with float_act, :109).
//
// CUDA-core kernel: the order of the sum is fixed (one chain of fused multiply-adds over k per output), so neither the tensor
// cores nor a split of K can be used; what bounds it is FMA issue (128 a clock and SM: 74 TFLOP/s at 1.96 GHz). Two neighbouring
// activation rows share one packed fma.rn.f32x2 (two independent, separately rounded FMAs in one instruction): half the issue
// slots of scalar FMAs, which leaves room for the shared-memory loads and for expanding the weights (64 x 64 tiles, scalar: 33.4 against
// 40.6 TFLOP/s at 512 rows on 14336 x 4096). k runs in steps of BK; while a step is multiplied the next one's activations and packed
// weights are on their way into registers, and two shared-memory buffers leave one barrier per step. Both operands
// lie as [k][row] in shared memory with an XOR on the row that keeps the transposing stores and the wide reads of a warp free of bank
// conflicts. Tiles of 64 x 64, 32 x 128 and 16 x 32 outputs; launches with work for 128 rows x 64 columns or more on every SM take the
// producer / consumer kernel further down.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "iquant.cuh"
#include "kernels.h"
#include "pipe.cuh"

namespace lb {

// What one thread fetches for eight consecutive weights of a row, before anything waits for it: the values as they are loaded, since a shift or
// a table lookup here would wait for a load. With those in expand8 (lookups: Entry8), us before -> after: 12 rows on 4096 x 2048: MXFP4 69 -> 47, Q6_K 69 -> 53,
// Int4 as before.
template <int FMT> struct Raw8 {
    uint32_t w[FMT == FMT_Q5K ? 8 : FMT == FMT_Q4K ? 6 : FMT == FMT_Q6K ? 10 : FMT == FMT_MXFP4 ? 5 : is_iq(FMT) ? 5 : 3];
};
template <int FMT> __device__ __forceinline__ void load_raw8(const GemmF32Args &p, uint32_t row, uint32_t k0, Raw8<FMT> &r) {
    if constexpr (FMT == FMT_Q4K || FMT == FMT_Q5K) {  // header (d, dmin, scales), then the eight bytes that hold the nibbles (and the fifth bits)
        const uint8_t *b = p.w + ((uint64_t)row * (p.k / QK) + k0 / QK) * (FMT == FMT_Q4K ? Q4K_BYTES : Q5K_BYTES);
        const uint32_t e = k0 % QK, l0 = e & 31;
        const uint4 h = *(const uint4 *)b;
        const uint2 q = *(const uint2 *)(b + (FMT == FMT_Q4K ? 16 : 48) + 32 * (e >> 6) + l0);
        r.w[0] = h.x, r.w[1] = h.y, r.w[2] = h.z, r.w[3] = h.w, r.w[4] = q.x, r.w[5] = q.y;
        if constexpr (FMT == FMT_Q5K) {
            const uint2 f = *(const uint2 *)(b + 16 + l0);
            r.w[6] = f.x, r.w[7] = f.y;
        }
    } else if constexpr (FMT == FMT_Q6K) {  // 2-byte aligned blocks
        const uint8_t *b = p.w + ((uint64_t)row * (p.k / QK) + k0 / QK) * Q6K_BYTES;
        const uint32_t e = k0 % QK, nh = e >> 7, w = (e >> 5) & 3, l0 = e & 31;
        const uint8_t *ql = b + 64 * nh + 32 * (w & 1) + l0, *qh = b + 128 + 32 * nh + l0;
#pragma unroll
        for (int i = 0; i < 4; i++) r.w[i] = ld16(ql + 2 * i), r.w[4 + i] = ld16(qh + 2 * i);
        r.w[8] = ld16(b + 208);
        r.w[9] = b[192 + 8 * nh + 2 * w + (l0 >> 4)];
    } else if constexpr (FMT == FMT_MXFP4) {  // unaligned blocks: the aligned words around the eight bytes
        const uint8_t *b = p.w + (((uint64_t)row * p.k + k0) / GROUP) * MXFP4_BYTES;
        const uintptr_t at = (uintptr_t)(b + 1 + (k0 & 15));
        const uint32_t *a = (const uint32_t *)(at & ~(uintptr_t)3);
        r.w[0] = b[0], r.w[1] = a[0], r.w[2] = a[1], r.w[3] = 0;
        r.w[4] = 8 * (uint32_t)(at & 3);
        if (r.w[4]) r.w[3] = a[2];
    } else if constexpr (is_iq(FMT)) {  // index, signs, scales, d of 8-group j (iquant.cuh has the layouts)
        const uint8_t *b = p.w + ((uint64_t)row * (p.k / QK) + k0 / QK) * iq_block_bytes(FMT);
        const uint32_t j = (k0 % QK) >> 3, ib = j >> 2, l = j & 3;
        r.w[3] = ld16(b);
        if constexpr (FMT == FMT_IQ2XXS) {
            r.w[0] = b[2 + 8 * ib + l], r.w[1] = ld16(b + 6 + 8 * ib), r.w[2] = ld16(b + 8 + 8 * ib);
        } else if constexpr (FMT == FMT_IQ2XS) {
            r.w[0] = ld16(b + 2 + 2 * j), r.w[1] = b[66 + ib];
        } else if constexpr (FMT == FMT_IQ2S) {
            r.w[0] = b[2 + j], r.w[1] = b[66 + ib], r.w[2] = b[34 + j], r.w[4] = b[74 + ib];
        } else {
            r.w[0] = ld16(b + 2 + 8 * ib + 2 * l), r.w[1] = ld16(b + 66 + 4 * ib), r.w[2] = ld16(b + 68 + 4 * ib);
        }
    } else {
        const uint64_t g = ((uint64_t)row * p.k + k0) / GROUP;
        const uint2 q = FMT == FMT_INT4 ? *(const uint2 *)(p.w + g * 16 + (k0 & 15)) : *(const uint2 *)(p.w + (uint64_t)row * p.k + k0);
        r.w[0] = q.x, r.w[1] = q.y, r.w[2] = ((const uint16_t *)(p.w + p.scales_offset))[g];
    }
}
// Byte i of w minus `bias`, as a float: the byte becomes the low mantissa bits of 2^23 (exact; I2F runs at a sixteenth of the rate)
__device__ __forceinline__ float byte_float(uint32_t w, int i, float bias) {
    return xsub(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u | (uint32_t)i)), 8388608.0f + bias);
}
// i-quants: the grid's bytes. Their address is in what was loaded, so they are a load behind a load: asked for when the raw values have arrived (a step after they
// were asked for), a step before they are expanded. us, looked up with the raw values / when they are expanded / in between: IQ2_S, 64 rows on 4096 x 4096
// 172 / 201 / 170, 16 rows on 14336 x 4096 177 / 200 / 171, 600 rows on 4096 x 14336 2033 / 2185 / 1987.
template <int FMT> struct Entry8 {
    uint32_t g[is_iq(FMT) ? 2 : 1];
};
template <int FMT> __device__ __forceinline__ void look8(const Raw8<FMT> &r, uint32_t k0, const uint8_t *grid, Entry8<FMT> &e) {
    if constexpr (FMT == FMT_IQ3XXS) {
        e.g[0] = *(const uint32_t *)(grid + 4 * (r.w[0] & 255u)), e.g[1] = *(const uint32_t *)(grid + 4 * (r.w[0] >> 8));
    } else if constexpr (is_iq(FMT)) {
        const uint32_t l = ((k0 % QK) >> 3) & 3;
        const uint32_t idx = FMT == FMT_IQ2XXS ? r.w[0] : FMT == FMT_IQ2XS ? r.w[0] & 511u : r.w[0] | ((r.w[1] << (8 - 2 * l)) & 0x300u);
        const uint2 v = *(const uint2 *)(grid + 8 * idx);
        e.g[0] = v.x, e.g[1] = v.y;
    }
}
// ... and the weights themselves, bit-exact dequant (each operation rounded on its own, as the reference rounds it).
template <int FMT> __device__ __forceinline__ void expand8(const Raw8<FMT> &r, const Entry8<FMT> &en, uint32_t k0, float (&y)[8]) {
    if constexpr (FMT == FMT_Q4K || FMT == FMT_Q5K) {
        const uint32_t e = k0 % QK, j = e >> 6, h = (e >> 5) & 1;
        const float d = half_bits_to_float(r.w[0] & 0xffffu), dmin = half_bits_to_float(r.w[0] >> 16);
        int sc0, mn0, sc1, mn1;
        scale_min_pair(j, r.w[1], r.w[2], r.w[3], sc0, mn0, sc1, mn1);
        const float d1 = xmul(d, (float)(h ? sc1 : sc0)), m1 = xmul(dmin, (float)(h ? mn1 : mn0));
#pragma unroll
        for (int i = 0; i < 8; i++) {
            int q = (r.w[4 + (i >> 2)] >> (8 * (i & 3) + 4 * h)) & 15;
            if constexpr (FMT == FMT_Q5K) q += ((r.w[6 + (i >> 2)] >> (8 * (i & 3) + 2 * j + h)) & 1) << 4;
            y[i] = xsub(xmul(d1, (float)q), m1);
        }
    } else if constexpr (FMT == FMT_Q6K) {
        const uint32_t w = ((k0 % QK) >> 5) & 3;
        const float t = xmul(half_bits_to_float(r.w[8]), (float)(int8_t)r.w[9]);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int lo = (r.w[i >> 1] >> (8 * (i & 1) + 4 * (w >> 1))) & 15, hi = (r.w[4 + (i >> 1)] >> (8 * (i & 1) + 2 * w)) & 3;
            y[i] = xmul(t, (float)((lo | (hi << 4)) - 32));
        }
    } else if constexpr (FMT == FMT_MXFP4) {
        const float d = e8m0_half(r.w[0]);
        const int sh = (k0 & 16) ? 4 : 0;
        const uint32_t q[2] = {__funnelshift_r(r.w[1], r.w[2], r.w[4]), __funnelshift_r(r.w[2], r.w[3], r.w[4])};
#pragma unroll
        for (int i = 0; i < 8; i++) y[i] = xmul((float)mxfp4_kv((q[i >> 2] >> (8 * (i & 3) + sh)) & 15u), d);
    } else if constexpr (is_iq(FMT)) {  // y = db * grid byte * sign (crates/lapid-quant/src/iq2.rs:38-90, iq3.rs:18-39)
        const uint32_t j = (k0 % QK) >> 3, l = j & 3, a = r.w[1] | r.w[2] << 16;
        uint32_t s, signs;
        if constexpr (FMT == FMT_IQ3XXS) {
            signs = iq_ksign((a >> (7 * l)) & 127u), s = a >> 28;
        } else {
            signs = FMT == FMT_IQ2XXS ? iq_ksign((a >> (7 * l)) & 127u) : FMT == FMT_IQ2XS ? iq_ksign(r.w[0] >> 9) : r.w[2];
            const uint32_t sc = FMT == FMT_IQ2XS ? r.w[1] : r.w[4];
            s = FMT == FMT_IQ2XXS ? a >> 28 : (j & 2) ? sc >> 4 : sc & 15u;  // (a half of 16 weights is two groups)
        }
        const float db = xmul(xmul(half_bits_to_float(r.w[3]), xadd(0.5f, (float)s)), FMT == FMT_IQ3XXS ? 0.5f : 0.25f);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float v = xmul(db, (float)((en.g[i >> 2] >> (8 * (i & 3))) & 255u));
            y[i] = (signs >> i) & 1u ? -v : v;
        }
    } else if constexpr (FMT == FMT_INT4) {
        const float d = half_bits_to_float(r.w[2]);
        const int sh = (k0 & 16) ? 4 : 0;  // elements 16.. of a group are the high nibbles of the same bytes
#pragma unroll
        for (int i = 0; i < 8; i++) y[i] = xmul((float)((int)((r.w[i >> 2] >> (8 * (i & 3) + sh)) & 15u) - 8), d);
    } else {
        const float d = half_bits_to_float(r.w[2]);
#pragma unroll
        for (int i = 0; i < 8; i++) y[i] = xmul(byte_float(r.w[i >> 2] ^ 0x80808080u, i & 3, 128.0f), d);
    }
}

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t &c, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }

// TM x TN outputs per thread, TM in pairs of rows; both in runs of four (16-byte shared loads), the runs of a thread BM / 2 (BN / 2) apart
// when there are two of them.
template <int FMT, int BM, int BN, int BK, int TM, int TN> __global__ void __launch_bounds__((BM / TM) * (BN / TN), 512 / ((BM / TM) * (BN / TN)))
qgemm_f32_kernel(GemmF32Args p) {
    constexpr int THREADS = (BM / TM) * (BN / TN), TX = BN / TN, TR = TN % 4 ? 2 : 4;  // TR: columns per run
    constexpr int AU = BM * BK / 4, WU = BN * BK / 8, WP = BK / 8;  // loads per step: four activations, eight weights each
    constexpr int AN = (AU + THREADS - 1) / THREADS, WN = (WU + THREADS - 1) / THREADS;
    static_assert(AU % THREADS == 0 && WU % THREADS == 0 && BM % 16 == 0 && BN % 32 == 0 && TM % 4 == 0 && TN % 2 == 0 && (BK == 16 || BK == 64), "tile");
    // BK = 16: four lanes fetch a row's 16 activations, two its 16 weights; BK = 64: a warp fetches four activations of each of its
    // rows, eight lanes a row's 64 weights. The XOR that keeps the transposing stores of a warp apart:
    auto swz_a = [](int k) { return BK == 16 ? 8 * (k >> 2) : 0; };
    auto swz_b = [](int k) { return BK == 16 ? 8 * (k >> 2) : 4 * (k >> 3); };
    auto a_row = [](int u) { return BK == 16 ? u >> 2 : u % BM; };
    auto a_k = [](int u) { return 4 * (BK == 16 ? u & 3 : u / BM); };
    static_assert(BK == 64 || BM >= 32, "the XOR stays inside the tile's rows");
    __shared__ __align__(16) float As[2][BK][BM];
    __shared__ __align__(16) float Bs[2][BK][BN];
    const int tid = threadIdx.x;
    const uint32_t row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    if (p.tile_expert) {  // expert-indexed launch (moe.cu): this activation tile multiplies one expert's matrix
        const int32_t e = p.tile_expert[blockIdx.y];
        if (e < 0) return;
        p.w += (uint64_t)e * p.id_stride;
    }
    const int ty = tid / TX, tx = tid % TX;
    uint64_t acc[TM / 2][TN];
#pragma unroll
    for (int i = 0; i < TM / 2; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0;

    const void *aptr[AN];
#pragma unroll
    for (int t = 0; t < AN; t++) {
        const int u = tid + t * THREADS;
        const uint32_t arow = row0 + (uint32_t)a_row(u);
        aptr[t] = nullptr;
        if (p.tile_expert) {
            const int32_t pair = p.row_pair[arow];
            if (pair >= 0) aptr[t] = (const char *)p.a + (p.a_off + (uint64_t)((uint32_t)pair / p.id_r) * p.a_rs) * act_elem_bytes(p.a_type);
        } else if (arow < p.rows) {
            aptr[t] = act_row(p.a, p.a_type, p.a_off, p.a_bs, p.a_rs, arow, p.m);
        }
    }

    float av[AN][4];
    Raw8<FMT> wv[WN], wv2[WN];  // (the second one: i-quants)
    Entry8<FMT> entry[WN];
    auto fetch = [&](uint32_t k0) {
#pragma unroll
        for (int t = 0; t < AN; t++) {
            const uint32_t k = k0 + (uint32_t)a_k(tid + t * THREADS);
            if (!aptr[t] || (BK == 64 && k >= p.k)) {
#pragma unroll
                for (int i = 0; i < 4; i++) av[t][i] = 0.0f;
            } else if (p.a_vec && p.a_type == ACT_F32) {
                const float4 v = *(const float4 *)((const float *)aptr[t] + k);
                av[t][0] = v.x, av[t][1] = v.y, av[t][2] = v.z, av[t][3] = v.w;
            } else if (p.a_vec) {
                const uint2 v = *(const uint2 *)((const uint16_t *)aptr[t] + k);
#pragma unroll
                for (int i = 0; i < 4; i++) av[t][i] = widen_act(((i < 2 ? v.x : v.y) >> (16 * (i & 1))) & 0xffffu, p.a_type);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) av[t][i] = load_act(aptr[t], k + i, p.a_type);
            }
        }
    };
    auto fetch_weights = [&](uint32_t k0, Raw8<FMT> (&to)[WN]) {
#pragma unroll
        for (int t = 0; t < WN; t++) {
            const int u = tid + t * THREADS;
            const uint32_t wrow = col0 + (uint32_t)(u / WP);
            const uint32_t k = k0 + 8 * (uint32_t)(u % WP);
            if (BK == 16 || k < p.k) load_raw8<FMT>(p, wrow < p.n ? wrow : p.n - 1, k, to[t]);  // columns past the matrix are not stored
        }
    };
    auto look_up = [&](uint32_t k0, const Raw8<FMT> (&wv)[WN]) {
#pragma unroll
        for (int t = 0; t < WN; t++) {
            const uint32_t k = k0 + 8 * (uint32_t)((tid + t * THREADS) % WP);
            if (BK == 16 || k < p.k) look8<FMT>(wv[t], k, p.iq_grid, entry[t]);
        }
    };
    auto stage = [&](int buf, uint32_t k0, const Raw8<FMT> (&wv)[WN]) {
#pragma unroll
        for (int t = 0; t < AN; t++) {
            const int u = tid + t * THREADS, k = a_k(u);
#pragma unroll
            for (int i = 0; i < 4; i++) As[buf][k + i][a_row(u) ^ swz_a(k)] = av[t][i];
        }
#pragma unroll
        for (int t = 0; t < WN; t++) {
            const int u = tid + t * THREADS, k = 8 * (u % WP);
            if (BK == 64 && k0 + (uint32_t)k >= p.k) continue;
            float y[8];
            expand8<FMT>(wv[t], entry[t], k0 + (uint32_t)k, y);
#pragma unroll
            for (int i = 0; i < 8; i++) Bs[buf][k + i][(u / WP) ^ swz_b(k + i)] = y[i];
        }
    };

    // k is a multiple of 32: the last step of BK = 64 may be half full and then ends there (a term 0 * 0 more would turn an accumulator
    // of -0, which a negative product that underflows leaves, into +0).
    fetch(0);
    fetch_weights(0, wv);
    look_up(0, wv);
    stage(0, 0, wv);
    if (is_iq(FMT) && BK < p.k) fetch_weights(BK, wv);
    __syncthreads();
    auto step = [&](uint32_t k0, int buf, Raw8<FMT> (&next)[WN], Raw8<FMT> (&after)[WN]) {  // `after`: i-quants, whose raw values come two steps ahead
        const bool more = k0 + BK < p.k;
        if (more) {
            fetch(k0 + BK);
            if constexpr (is_iq(FMT)) {
                look_up(k0 + BK, next);
                if (k0 + 2 * BK < p.k) fetch_weights(k0 + 2 * BK, after);
            } else {
                fetch_weights(k0 + BK, next);
            }
        }
        // operands of step kk + 1 are on their way while kk is multiplied
        uint64_t a2[2][TM / 2];
        float b[2][TN];
        auto operands = [&](int kk) {
#pragma unroll
            for (int i = 0; i < TM / 4; i++) {
                const ulonglong2 v = *(const ulonglong2 *)&As[buf][kk][(4 * ty + i * (BM / (TM / 4))) ^ swz_a(kk)];
                a2[kk & 1][2 * i] = v.x, a2[kk & 1][2 * i + 1] = v.y;
            }
#pragma unroll
            for (int j = 0; j < TN / TR; j++) {
                const float *src = &Bs[buf][kk][(TR * tx + j * (BN / (TN / TR))) ^ swz_b(kk)];
                if constexpr (TR == 4) *(float4 *)&b[kk & 1][4 * j] = *(const float4 *)src;
                else *(float2 *)&b[kk & 1][2 * j] = *(const float2 *)src;
            }
        };
        auto multiply = [&](auto steps) {
            operands(0);
#pragma unroll 16
            for (int kk = 0; kk < steps.value; kk++) {
                if (kk + 1 < steps.value) operands(kk + 1);
#pragma unroll
                for (int j = 0; j < TN; j++) {
                    const uint64_t b2 = pack2(b[kk & 1][j], b[kk & 1][j]);
#pragma unroll
                    for (int i = 0; i < TM / 2; i++) fma2(acc[i][j], a2[kk & 1][i], b2);
                }
            }
        };
        if (BK == 64 && p.k - k0 < BK) multiply(std::integral_constant<int, BK / 2>());
        else multiply(std::integral_constant<int, BK>());
        if (more) {
            stage(buf ^ 1, k0 + BK, next);  // the other buffer's readers passed the barrier of the step before
            __syncthreads();
        }
    };
    if constexpr (is_iq(FMT)) {
        for (uint32_t k0 = 0; k0 < p.k; k0 += 2 * BK) {
            step(k0, 0, wv, wv2);
            if (k0 + BK < p.k) step(k0 + BK, 1, wv2, wv);
        }
    } else {
        int buf = 0;
        for (uint32_t k0 = 0; k0 < p.k; k0 += BK, buf ^= 1) step(k0, buf, wv, wv);
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const uint32_t r = row0 + 4 * ty + (i >> 2) * (BM / (TM / 4)) + (i & 3);
        if (r >= p.rows) continue;
        float *o;
        const float *ex = nullptr;
        if (p.tile_expert) {
            const int32_t pair = p.row_pair[r];
            if (pair < 0) continue;
            o = p.out + p.out_off + (uint64_t)pair * p.n;
        } else {
            const uint32_t bt = r / p.m, ii = r % p.m;
            o = p.out + p.out_off + (uint64_t)bt * p.out_bs + (uint64_t)ii * p.out_rs;
            if (p.extra) ex = p.extra + (p.ex_off + (int64_t)bt * p.ex_s0 + (int64_t)ii * p.ex_s1);
        }
#pragma unroll
        for (int jr = 0; jr < TN / TR; jr++) {
            const uint32_t col = col0 + TR * tx + jr * (BN / (TN / TR));
            float v[TR];
#pragma unroll
            for (int j = 0; j < TR; j++) {
                const uint64_t c = acc[i >> 1][TR * jr + j];
                v[j] = __uint_as_float((uint32_t)((i & 1) ? c >> 32 : c));
                if (ex && col + j < p.n) v[j] += ex[(int64_t)(col + j) * p.ex_s2];
            }
            if constexpr (TR == 4) {
                if (col + 3 < p.n && ((uintptr_t)(o + col) & 15) == 0) {
                    *(float4 *)(o + col) = make_float4(v[0], v[1], v[2], v[3]);
                    continue;
                }
            }
#pragma unroll
            for (int j = 0; j < TR; j++)
                if (col + j < p.n) o[col + j] = v[j];
        }
    }
}

// ---- many outputs: producer and consumer warps ------------------------------------------------------------------
// The same sums with the roles of a CTA's warps split: four producer warps fetch activations and packed weights and write both operands
// into a ring of shared-memory stages, eight consumer warps do nothing but shared loads and packed FMAs, 8 rows x W columns each thread,
// and never wait for a barrier of the whole CTA. A tile is 128 rows x 16 W columns, W = 4..8 chosen per tile: a launch's columns are cut
// into nearly equal tiles so that every SM gets the same number of them, where tiles of a fixed width leave the last round mostly empty
// (512 rows on 4096 columns: 128 x 128 tiles use 128 of 148 SMs, tiles of 112 columns all of them). One CTA per SM walks its tiles; the
// producers run ahead into the next one. int8 weights, us, 128 x 128 or 64 x 64 tiles of the kernel above -> this one: 512 rows on 14336 x 4096
// 1432 -> 1191 (50.5 TFLOP/s), on 4096 x 4096 424 -> 353, 128 rows on 14336 x 4096 425 -> 353, 2048 rows on 9600 x 2880 2203 -> 2140 (52.9).
// FMA pipe busy 70 %, shared loads 56 % (a load of 16 bytes a lane takes the 128-byte return path four cycles whoever shares it); the rest
// is latency of two consumer warps a scheduler, and the producers (without their stores and expansion: 56 TFLOP/s). Measured and not better:
// one consumer warp a scheduler with 16 x 8 outputs a thread (44 TFLOP/s), two with 16 x 8 (48.5), columns up to 12 a thread (49.8),
// operands fetched over the edge of a stage (46), pairs of rows turned round instead of columns written twice (46).
namespace ws {

constexpr int BK = 16, STAGES = 4, CONSUMERS = 256, PRODUCERS = 128, W_MIN = 4, W_MAX = 8;
constexpr int BM = 128, TX = 16, BN = W_MAX * TX;  // BN: the widest tile
constexpr int A_FLOATS = BK * BM, STAGE_FLOATS = A_FLOATS + BK * BN;
constexpr size_t SMEM = (size_t)STAGES * STAGE_FLOATS * 4 + 2 * STAGES * 8;
constexpr uint32_t WAIT_LIMIT = 1u << 19;  // a failed attempt sleeps some 4 us: two seconds

struct Cut {  // how the launch is cut: `per_block` tiles for each block of BM rows, each of whole units of TX columns
    uint32_t row_blocks, per_block, units, turn;
    uint64_t tiles;
};
struct Tile {
    uint32_t rb, col0, w;  // w: units of TX columns (0: nothing to do)
};
__device__ __forceinline__ Tile tile_at(const GemmF32Args &p, const Cut &c, uint64_t t) {
    // every block of rows starts at another tile: the wider ones do not all meet on the same CTAs
    const uint32_t rb = (uint32_t)(t / c.per_block), i = (uint32_t)((t % c.per_block + (uint64_t)rb * c.turn) % c.per_block);
    const uint32_t u0 = (uint32_t)((uint64_t)i * c.units / c.per_block), u1 = (uint32_t)((uint64_t)(i + 1) * c.units / c.per_block);
    return Tile{rb, u0 * TX, (p.tile_expert && p.tile_expert[rb] < 0) ? 0u : u1 - u0};
}

// 8 rows x W columns of a thread: rows 4 ty + 0..3 and BM / 2 further, columns in runs of four, two and one (16-, 8- and 4-byte shared loads).
template <int W>
__device__ __forceinline__ bool consume(const GemmF32Args &p, const Tile &tile, const float *ring, uint64_t *full, uint64_t *empty, uint32_t &stage, uint32_t &phase) {
    constexpr int NQ = W / 4, NP = (W % 4) / 2, N1 = W % 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ty = (lane & 3) + 4 * (warp & 3), tx = (lane >> 2) + 8 * (warp >> 2);
    uint64_t acc[4][W];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < W; j++) acc[i][j] = 0;
    for (uint32_t k0 = 0; k0 < p.k; k0 += BK) {
        if (!pipe::mbar_wait(full + stage, phase, WAIT_LIMIT)) return false;
        const float *As = ring + stage * STAGE_FLOATS, *Bs = As + A_FLOATS;
        uint64_t a2[2][4];
        float b[2][W];
        auto operands = [&](int kk) {
            const int q = 8 * (kk >> 2);  // (the XOR of the producers' transposing stores)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const ulonglong2 v = *(const ulonglong2 *)(As + kk * BM + ((4 * ty) ^ q) + i * (BM / 2));
                a2[kk & 1][2 * i] = v.x, a2[kk & 1][2 * i + 1] = v.y;
            }
            const float *row = Bs + kk * BN;
#pragma unroll
            for (int j = 0; j < NQ; j++) *(float4 *)&b[kk & 1][4 * j] = *(const float4 *)(row + 4 * TX * j + ((4 * tx) ^ q));
            if constexpr (NP) {
                const float2 v = *(const float2 *)(row + 4 * TX * NQ + ((2 * tx) ^ q));
                b[kk & 1][4 * NQ] = v.x, b[kk & 1][4 * NQ + 1] = v.y;
            }
            if constexpr (N1) b[kk & 1][W - 1] = row[TX * (W - 1) + (tx ^ q)];
        };
        operands(0);
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {  // the operands of the next step are on their way
            if (kk + 1 < BK) operands(kk + 1);
#pragma unroll
            for (int j = 0; j < W; j++) {
                const uint64_t b2 = pack2(b[kk & 1][j], b[kk & 1][j]);
#pragma unroll
                for (int i = 0; i < 4; i++) fma2(acc[i][j], a2[kk & 1][i], b2);
            }
        }
        __syncwarp();
        if (lane == 0) pipe::mbar_arrive(empty + stage);  // (behind the last products: what was read has been used)
        if (++stage == STAGES) stage = 0, phase ^= 1;
    }
    const uint32_t row0 = tile.rb * BM, end = min(p.n, tile.col0 + tile.w * TX);  // (columns past a narrow tile belong to the next one)
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t r = row0 + 4 * ty + (i >> 2) * (BM / 2) + (i & 3);
        if (r >= p.rows) continue;
        float *o;
        const float *ex = nullptr;
        if (p.tile_expert) {
            const int32_t pair = p.row_pair[r];
            if (pair < 0) continue;
            o = p.out + p.out_off + (uint64_t)pair * p.n;
        } else {
            const uint32_t bt = r / p.m, ii = r % p.m;
            o = p.out + p.out_off + (uint64_t)bt * p.out_bs + (uint64_t)ii * p.out_rs;
            if (p.extra) ex = p.extra + (p.ex_off + (int64_t)bt * p.ex_s0 + (int64_t)ii * p.ex_s1);
        }
        float v[W];
#pragma unroll
        for (int j = 0; j < W; j++) v[j] = __uint_as_float((uint32_t)((i & 1) ? acc[i >> 1][j] >> 32 : acc[i >> 1][j]));
#pragma unroll
        for (int j = 0; j < NQ; j++) {
            const uint32_t col = tile.col0 + 4 * TX * j + 4 * tx;
            if (!ex && col + 3 < end && ((uintptr_t)(o + col) & 15) == 0) {
                *(float4 *)(o + col) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                continue;
            }
#pragma unroll
            for (int l = 0; l < 4; l++)
                if (col + l < end) o[col + l] = ex ? v[4 * j + l] + ex[(int64_t)(col + l) * p.ex_s2] : v[4 * j + l];
        }
#pragma unroll
        for (int j = 4 * NQ; j < W; j++) {
            const uint32_t col = tile.col0 + (j < 4 * NQ + 2 * NP ? 4 * TX * NQ + 2 * tx + (j & 1) : TX * (W - 1) + tx);
            if (col < end) o[col] = ex ? v[j] + ex[(int64_t)col * p.ex_s2] : v[j];
        }
    }
    return true;
}

template <int FMT> __global__ void __launch_bounds__(CONSUMERS + PRODUCERS, 1) qgemm_f32_ws_kernel(GemmF32Args p, Cut cut) {
    extern __shared__ __align__(16) float ring[];
    uint64_t *full = (uint64_t *)(ring + STAGES * STAGE_FLOATS), *empty = full + STAGES;
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; i++) pipe::mbar_init(full + i, PRODUCERS / 32), pipe::mbar_init(empty + i, CONSUMERS / 32);
        pipe::mbar_fence_init();
    }
    __syncthreads();
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    if (threadIdx.x < CONSUMERS) {
        for (uint64_t t = blockIdx.x; t < cut.tiles && ok; t += gridDim.x) {
            const Tile tile = tile_at(p, cut, t);
            switch (tile.w) {
                case 0: break;
                case 8: ok = consume<8>(p, tile, ring, full, empty, stage, phase); break;
                case 7: ok = consume<7>(p, tile, ring, full, empty, stage, phase); break;
                case 6: ok = consume<6>(p, tile, ring, full, empty, stage, phase); break;
                case 5: ok = consume<5>(p, tile, ring, full, empty, stage, phase); break;
                default: ok = consume<4>(p, tile, ring, full, empty, stage, phase); break;
            }
        }
    } else {
        constexpr int AN = BM * BK / 4 / PRODUCERS, WN = W_MAX * TX * 2 / PRODUCERS;  // loads per step: four activations, eight weights each
        static_assert(BM * BK / 4 % PRODUCERS == 0 && W_MAX * TX * 2 % PRODUCERS == 0, "producers");
        const int tid = threadIdx.x - CONSUMERS;
        const uint8_t *stack = p.w;
        for (uint64_t t = blockIdx.x; t < cut.tiles && ok; t += gridDim.x) {
            const Tile tile = tile_at(p, cut, t);
            if (tile.w == 0) continue;
            const uint32_t row0 = tile.rb * BM, cols = max(tile.w, (uint32_t)W_MIN) * TX;
            if (p.tile_expert) p.w = stack + (uint64_t)p.tile_expert[tile.rb] * p.id_stride;
            const void *aptr[AN];
#pragma unroll
            for (int i = 0; i < AN; i++) {
                const uint32_t arow = row0 + (uint32_t)((tid + i * PRODUCERS) >> 2);
                aptr[i] = nullptr;
                if (p.tile_expert) {
                    const int32_t pair = p.row_pair[arow];
                    if (pair >= 0) aptr[i] = (const char *)p.a + (p.a_off + (uint64_t)((uint32_t)pair / p.id_r) * p.a_rs) * act_elem_bytes(p.a_type);
                } else if (arow < p.rows) {
                    aptr[i] = act_row(p.a, p.a_type, p.a_off, p.a_bs, p.a_rs, arow, p.m);
                }
            }
            const int ak = 4 * (tid & 3), arow = tid >> 2, wk = 8 * (tid & 1), wcol = tid >> 1;
            uint32_t av[2][AN][4];  // four activations as they lie: f32 bits, or halves in pairs (a_vec) or one by one, widened when they are written
            Raw8<FMT> wv[2][WN];    // (widening them here would wait for the load: IQ2_XS, 200 bf16 rows on 13306 x 5632 1278 us, so 886)
            auto fetch = [&](int set, uint32_t k0) {
#pragma unroll
                for (int i = 0; i < AN; i++) {
                    const uint32_t k = k0 + ak;
                    uint32_t (&a)[4] = av[set][i];
                    if (!aptr[i]) {
                        a[0] = a[1] = a[2] = a[3] = 0;
                    } else if (p.a_vec && p.a_type == ACT_F32) {
                        const uint4 v = *(const uint4 *)((const float *)aptr[i] + k);
                        a[0] = v.x, a[1] = v.y, a[2] = v.z, a[3] = v.w;
                    } else if (p.a_vec) {
                        const uint2 v = *(const uint2 *)((const uint16_t *)aptr[i] + k);
                        a[0] = v.x, a[1] = v.y;
                    } else if (p.a_type == ACT_F32) {
#pragma unroll
                        for (int l = 0; l < 4; l++) a[l] = ((const uint32_t *)aptr[i])[k + l];
                    } else {
#pragma unroll
                        for (int l = 0; l < 4; l++) a[l] = ((const uint16_t *)aptr[i])[k + l];
                    }
                }
#pragma unroll
                for (int i = 0; i < WN; i++) {
                    const uint32_t c = (uint32_t)wcol + i * (PRODUCERS / 2), row = tile.col0 + c;
                    if (c < cols) load_raw8<FMT>(p, row < p.n ? row : p.n - 1, k0 + wk, wv[set][i]);  // columns past the matrix are not stored
                }
            };
            Entry8<FMT> entry[2][WN];
            auto look_up = [&](int set, uint32_t k0) {  // (i-quants; the raw values were asked for a step ago)
#pragma unroll
                for (int i = 0; i < WN; i++)
                    if ((uint32_t)wcol + i * (PRODUCERS / 2) < cols) look8<FMT>(wv[set][i], k0 + wk, p.iq_grid, entry[set][i]);
            };
            auto put = [&](int set, uint32_t k0) {
                if (!pipe::mbar_wait(empty + stage, phase ^ 1, WAIT_LIMIT)) return false;
                float *As = ring + stage * STAGE_FLOATS, *Bs = As + A_FLOATS;
#pragma unroll
                for (int i = 0; i < AN; i++) {
                    const uint32_t (&a)[4] = av[set][i];
                    float x[4];
                    if (p.a_type == ACT_F32) {
#pragma unroll
                        for (int l = 0; l < 4; l++) x[l] = __uint_as_float(a[l]);
                    } else {
#pragma unroll
                        for (int l = 0; l < 4; l++) x[l] = widen_act(p.a_vec ? (a[l >> 1] >> (16 * (l & 1))) & 0xffffu : a[l], p.a_type);
                    }
#pragma unroll
                    for (int l = 0; l < 4; l++) As[(ak + l) * BM + ((arow + i * (PRODUCERS / 4)) ^ (2 * ak))] = x[l];
                }
#pragma unroll
                for (int i = 0; i < WN; i++) {
                    const uint32_t c = (uint32_t)wcol + i * (PRODUCERS / 2);
                    if (c >= cols) continue;
                    float y[8];
                    expand8<FMT>(wv[set][i], entry[set][i], k0 + wk, y);
#pragma unroll
                    for (int l = 0; l < 8; l++) Bs[(wk + l) * BN + (c ^ (2 * wk + 8 * (l >> 2)))] = y[l];
                }
                __syncwarp();
                if ((tid & 31) == 0) pipe::mbar_arrive(full + stage);
                if (++stage == STAGES) stage = 0, phase ^= 1;
                return true;
            };
            // the operands of the step after the one being written are on their way (k is a multiple of 32: steps come in pairs)
            fetch(0, 0);
            for (uint32_t k0 = 0; k0 < p.k && ok; k0 += 2 * BK) {
                look_up(0, k0);
                fetch(1, k0 + BK);
                ok = put(0, k0);
                if (!ok) break;
                look_up(1, k0 + BK);
                if (k0 + 2 * BK < p.k) fetch(0, k0 + 2 * BK);
                ok = put(1, k0 + BK);
            }
        }
    }
    if (!ok && p.status) atomicOr(p.status, 256);
}

}  // namespace ws

constexpr uint32_t GRID_Y_MAX = 65535;
template <int FMT, int BM, int BN, int BK, int TM, int TN> static cudaError_t launch_tile(const GemmF32Args &a, cudaStream_t stream) {
    const dim3 grid((a.n + BN - 1) / BN, (a.rows + BM - 1) / BM);
    if (grid.y > GRID_Y_MAX) return cudaErrorInvalidValue;
    qgemm_f32_kernel<FMT, BM, BN, BK, TM, TN><<<grid, (BM / TM) * (BN / TN), 0, stream>>>(a);
    return cudaGetLastError();
}

// Time of a tile of W units of 16 columns on a CTA of the producer / consumer kernel, us, K = 4096 (int8 weights; the other formats within a tenth; W below 4 costs
// what 4 costs). On long rows narrow tiles take more than their share (4 units, K = 14336: 960 us, 14336 / 4096 of 241 is 844), and of i-quants, whose
// expansion the producers then wait for (IQ3_XXS 279).
static double ws_tile_us(double w, uint32_t k, bool iq) {
    static const double SHORT[] = {241, 268, 305, 330, 390}, LONG[] = {262, 278, 305, 330, 390}, IQ[] = {280, 290, 305, 330, 390};  // W = 4..8
    const double *us = iq ? IQ : k < 8192 ? SHORT : LONG;
    if (w <= 4) return us[0];
    if (w >= ws::W_MAX) return us[4];
    const int i = (int)w - 4;
    return us[i] + (us[i + 1] - us[i]) * (w - 4 - i);
}
// Tiles per block of 128 rows: of the numbers that fill whole rounds of CTAs, the one whose tiles cost least. Few rounds of wide tiles win until a round more
// makes them fit: 512 rows on 4096 columns, one round of 7 units 353 us, two of 4 466; on 14336, four rounds of 6 1191 us, five of 5 1310.
static ws::Cut ws_cut(bool iq, uint64_t row_blocks, uint64_t n, uint32_t k, int sm_count, double &cost) {
    ws::Cut c{};
    c.row_blocks = (uint32_t)row_blocks;
    c.units = (uint32_t)((n + ws::TX - 1) / ws::TX);
    cost = 1e30;
    for (int w = ws::W_MAX; w >= 1; w--) {
        uint64_t per = (c.units + w - 1) / w;
        const uint64_t rounds = (row_blocks * per + sm_count - 1) / sm_count;
        if (rounds * sm_count / row_blocks > per) per = rounds * sm_count / row_blocks;  // more tiles in as many rounds
        if (per > c.units) per = c.units;
        const double widest = ceil((double)c.units / (double)per), mean = (double)c.units / (double)per;
        // (with several rounds the wider tiles spread over the CTAs)
        const double us = (double)rounds * ws_tile_us(rounds == 1 ? widest : mean + (widest - mean) / (double)rounds, k, iq);
        if (us < cost) cost = us, c.per_block = (uint32_t)per;
    }
    c.tiles = (uint64_t)c.per_block * row_blocks;
    c.turn = c.per_block / 3 + 1;
    return c;
}
template <int FMT> static cudaError_t launch_ws(const GemmF32Args &a, int sm_count, cudaStream_t stream) {
    const uint64_t row_blocks = ((uint64_t)a.rows + ws::BM - 1) / ws::BM;
    if (row_blocks > GRID_Y_MAX) return cudaErrorInvalidValue;
    double cost;
    const ws::Cut c = ws_cut(is_iq(FMT), row_blocks, a.n, a.k, sm_count, cost);
    static DynamicSmemOptIn optin;
    cudaError_t e = optin.raise((const void *)ws::qgemm_f32_ws_kernel<FMT>, ws::SMEM);
    if (e != cudaSuccess) return e;
    ws::qgemm_f32_ws_kernel<FMT><<<c.tiles < (uint64_t)sm_count ? (uint32_t)c.tiles : sm_count, ws::CONSUMERS + ws::PRODUCERS, ws::SMEM, stream>>>(a, c);
    return cudaGetLastError();
}

// The tiles, and what a launch on them takes: us at K = 4096 for an SM with 1, 2, .. of them (several run side by side), then `more` for each further one, all but
// `start` in proportion to K (int8 weights, every SM with that many; measured at 9 to 600 rows on 512 to 14336 columns and K 1024, 4096 and 14336: of 250 shapes the choice
// is the fastest or within 1 % of it). The last round costs a tenth of a tile less where it reaches part of the SMs. Activation rows that lie a multiple of 4096 bytes apart
// share cache sets, which the kernel above feels (`uneven`: where they don't). Examples, us, 16 x 32 / 32 x 128 / 64 x 64 / 128 rows: 64 rows on 4096 x 4096 150 / 171 / 155 /
// 231, 300 on 3000 x 4096 - / 283 / 245 / 237, on 3000 x 1024 - / 69 / 60 / 65, 86 on 9728 x 4096 - / 282 / 350 / 269, 86 on 9728 x 2560 - / 164 / 210 / 169.
struct F32Tile {
    uint32_t bm, bn;
    double start, more, uneven;
    int counted;
    double us[7];
};
static const F32Tile F32_TILES[] = {{128, 0, 10, 0, 1, 0, {}},  // ws_tile_us
                                    {64, 64, 2, 105, 0.95, 4, {152, 246, 358, 462}},
                                    {32, 128, 0, 125, 0.93, 4, {168, 280, 410, 532}},
                                    {16, 32, 4, 29.5, 1, 7, {75, 92, 121, 146, 185, 206, 238}}};
static int pick_tile(bool iq, uint64_t matrices, double rows, uint64_t n, uint32_t k, int sm_count) {  // `matrices` products of `rows` rows each
    int best = 0;
    double cost = 1e30;
    for (int i = 0; i < 4; i++) {
        const F32Tile &t = F32_TILES[i];
        const uint64_t blocks = matrices * (uint64_t)ceil(rows / t.bm);
        double us;
        if (t.bn) {
            const uint64_t tiles = blocks * ((n + t.bn - 1) / t.bn), per = (tiles + sm_count - 1) / sm_count;
            us = per <= (uint64_t)t.counted ? t.us[per - 1] : t.us[t.counted - 1] + t.more * (double)(per - t.counted);
            if (t.bm > 16 && per > 1) us -= 0.1 * t.more * ((double)per - (double)tiles / sm_count);
        } else {
            ws_cut(iq, blocks, n, k, sm_count, us);
        }
        us = t.start + (us - t.start) * (double)k / 4096.0 * (k % 1024 ? t.uneven : 1.0);
        if (us < cost) cost = us, best = i;
    }
    return best;
}
// Expert-indexed launches: the tile for the experts' expected rows plus the spread of a random routing.
uint32_t qgemm_f32_moe_tile(int fmt, uint64_t pairs, uint64_t experts, uint64_t n, uint32_t k, int sm_count) {
    const uint64_t used = experts < pairs ? experts : pairs;
    if (!used) return 64;
    const double avg = (double)pairs / (double)used;
    int i = pick_tile(is_iq(fmt), used, avg + (avg > 1 ? sqrt(avg) : 0), n, k, sm_count);
    while (i > 0 && moe_max_tiles(pairs, experts, F32_TILES[i].bm) > GRID_Y_MAX) i--;  // tens of thousands of experts: taller tiles, fewer of them
    return F32_TILES[i].bm;
}

template <int FMT> static cudaError_t launch_fmt(const GemmF32Args &a, int sm_count, cudaStream_t stream) {
    switch (a.tile_expert ? a.mt : a.tile ? a.tile : F32_TILES[pick_tile(is_iq(FMT), 1, a.rows, a.n, a.k, sm_count)].bm) {
        case 128: return launch_ws<FMT>(a, sm_count, stream);
        case 64: return launch_tile<FMT, 64, 64, 16, 8, 4>(a, stream);
        case 32: return launch_tile<FMT, 32, 128, 16, 8, 4>(a, stream);
        case 16: return launch_tile<FMT, 16, 32, 64, 4, 2>(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_qgemm_f32(int fmt, const GemmF32Args &args, int sm_count, cudaStream_t stream) {
    if (args.rows == 0 || args.n == 0) return cudaSuccess;
    GemmF32Args a = args;
    const uint64_t quad = a.a_type == ACT_F32 ? 16 : 8;  // four activations in one load
    a.a_vec = ((uintptr_t)a.a + a.a_off * act_elem_bytes(a.a_type)) % quad == 0 && a.a_rs % 4 == 0 && a.a_bs % 4 == 0;
    switch (fmt) {
        case FMT_Q4K: return launch_fmt<FMT_Q4K>(a, sm_count, stream);
        case FMT_Q5K: return launch_fmt<FMT_Q5K>(a, sm_count, stream);
        case FMT_Q6K: return launch_fmt<FMT_Q6K>(a, sm_count, stream);
        case FMT_INT8: return launch_fmt<FMT_INT8>(a, sm_count, stream);
        case FMT_INT4: return launch_fmt<FMT_INT4>(a, sm_count, stream);
        case FMT_MXFP4: return launch_fmt<FMT_MXFP4>(a, sm_count, stream);
        case FMT_IQ2XXS:
        case FMT_IQ2XS:
        case FMT_IQ2S:
        case FMT_IQ3XXS: {
            const uint8_t *grids = iq_grids();
            if (!grids) return cudaErrorNotReady;
            a.iq_grid = grids + iq_grid_offset(fmt);
            if (fmt == FMT_IQ2XXS) return launch_fmt<FMT_IQ2XXS>(a, sm_count, stream);
            if (fmt == FMT_IQ2XS) return launch_fmt<FMT_IQ2XS>(a, sm_count, stream);
            if (fmt == FMT_IQ2S) return launch_fmt<FMT_IQ2S>(a, sm_count, stream);
            return launch_fmt<FMT_IQ3XXS>(a, sm_count, stream);
        }
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace lb

// Weight quantizers on the device, byte-identical to lapid-quant's reference quantizers.
//
//   Q4_K  crates/lapid-quant/src/kquant.rs:42-121 (make_qkx2_quants), :188-260
//   Q5_K  the same search with 5-bit levels (nmax 31, rmin -0.5, 15 steps), :263-287
//   Q6_K  crates/lapid-quant/src/kquant.rs:124-174 (make_qx_quants, rmse_type 1), :290-334
//   Int8  crates/lapid-quant/src/imp.rs:24-40, :95-115
//
// The searches are sequential f32 recurrences whose rounding order defines the output bytes, so
// the parallelism is across sub-blocks, never inside one: one thread owns one sub-block (32
// values for Q4_K, 16 for Q6_K) and runs the reference's loops in the reference's order with
// separately rounded operations; the 8 / 16 threads of a super-block then agree on the block
// scale through warp shuffles, and the quants are packed through shared memory, four bytes at a time.
// Compile this file with -fmad=false as a second guard against contraction.
//
// What bounds the searches is instruction issue (a Q4_K weight goes through 21 candidate scales, each two passes of about ten
// operations), so the loops are written for few instructions: element pairs in packed f32x2 operations
// (two separately rounded results in one instruction; only the running sums, whose order is fixed, stay scalar), the
// level of an element as a float that never leaves the 2^23 offset domain (no integer conversions, which run at a quarter of the rate), everything in
// registers. The levels of the best candidate are not kept: they are rarely needed, and the scale they came from gives them again.
// 14336 x 4096: 880 us (Q4_K; scalar operations with the levels in local memory: 1336)
#include "common.cuh"
#include "kernels.h"

namespace lb {

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// ---- pairs of f32 in one register pair. A product that a packed addition takes goes through scalar additions instead (xadd2): the
// assembler contracts mul.rn.f32x2 + add.rn.f32x2 to one rounding, whatever -fmad says; scalar .rn additions it leaves alone.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t both(float a) { return pack2(a, a); }
__device__ __forceinline__ float lo2(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t xadd2(uint64_t a, float b) { return pack2(xadd(lo2(a), b), xadd(hi2(a), b)); }
// clampi(nearest_int(v), LO, HI) as a float, for both halves: nearest_int's offset form keeps the low 23 bits (they wrap for
// values out of its range, NaN included, and so they do here), planted as the mantissa of 2^23 they order like
// the integers, and taking 2^23 + 2^22 off again is exact.
template <int LO, int HI> __device__ __forceinline__ float clamp_offset(float f) {
    const float r = __uint_as_float((__float_as_uint(f) & 0x007fffffu) | 0x4B000000u);
    return fminf(fmaxf(r, 12582912.0f + LO), 12582912.0f + HI);
}
template <int LO, int HI> __device__ __forceinline__ uint64_t level2(uint64_t v) {
    const float a = clamp_offset<LO, HI>(xadd(lo2(v), 12582912.0f)), b = clamp_offset<LO, HI>(xadd(hi2(v), 12582912.0f));
    return add2(pack2(a, b), both(-12582912.0f));
}

// What the search for a sub-block returns: the scale, and how the levels of the best candidate were made.
struct Best32 {
    float scale, the_min, iscale, from;  // level of x = nearest(iscale * (x - from)), clamped
    bool flat;                           // all values the same: every level is 0
};

// Asymmetric (scale, min) search for one 32-value sub-block.
template <int FMT> __device__ __forceinline__ Best32 make_qkx2_32(const uint64_t (&x)[16], const uint64_t (&w)[16]) {
    constexpr int nmax = FMT == FMT_Q5K ? 31 : 15, nstep = FMT == FMT_Q5K ? 15 : 20;
    const float rmin = FMT == FMT_Q5K ? -0.5f : -1.0f, rdelta = 0.1f;
    Best32 r{0.0f, 0.0f, 0.0f, 0.0f, false};
    float mn = lo2(x[0]), mx = lo2(x[0]);
    float sum_w = lo2(w[0]), sum_x = xmul(lo2(w[0]), lo2(x[0]));
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const uint64_t wx = mul2(w[i], x[i]);
#pragma unroll
        for (int h = i == 0 ? 1 : 0; h < 2; h++) {
            const float xi = h ? hi2(x[i]) : lo2(x[i]);
            if (xi < mn) mn = xi;
            if (xi > mx) mx = xi;
            sum_w = xadd(sum_w, h ? hi2(w[i]) : lo2(w[i]));
            sum_x = xadd(sum_x, h ? hi2(wx) : lo2(wx));
        }
    }
    if (mn > 0.0f) mn = 0.0f;
    if (mx == mn) {
        r.the_min = -mn;
        r.flat = true;
        return r;
    }
    float iscale = xdiv((float)nmax, xsub(mx, mn));
    r.scale = xdiv(1.0f, iscale);
    r.iscale = iscale, r.from = mn;
    // sum of w (scale l + mn - x)^2; the difference is taken the other way round, which squares to the same bits
    auto error_of = [&](const uint64_t (&l)[16], float scale, float min) {
        const uint64_t ns = both(-scale);
        float e = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const uint64_t d = add2(x[i], xadd2(mul2(ns, l[i]), -min)), t = mul2(w[i], mul2(d, d));
            e = xadd(e, lo2(t));
            e = xadd(e, hi2(t));
        }
        return e;
    };
    uint64_t l[16];
#pragma unroll
    for (int i = 0; i < 16; i++) l[i] = level2<0, nmax>(mul2(both(iscale), add2(x[i], both(-mn))));
    float best = error_of(l, r.scale, mn);
#pragma unroll 1
    for (int is = 0; is <= nstep; is++) {
        iscale = xdiv(xadd(xadd(rmin, xmul(rdelta, (float)is)), (float)nmax), xsub(mx, mn));
        const uint64_t is2 = both(iscale), nm2 = both(-mn);
        float sum_l = 0.0f, sum_l2 = 0.0f, sum_xl = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            l[i] = level2<0, nmax>(mul2(is2, add2(x[i], nm2)));
            const uint64_t wl = mul2(w[i], l[i]), wll = mul2(wl, l[i]), wlx = mul2(wl, x[i]);
            sum_l = xadd(sum_l, lo2(wl)), sum_l2 = xadd(sum_l2, lo2(wll)), sum_xl = xadd(sum_xl, lo2(wlx));
            sum_l = xadd(sum_l, hi2(wl)), sum_l2 = xadd(sum_l2, hi2(wll)), sum_xl = xadd(sum_xl, hi2(wlx));
        }
        const float D = xsub(xmul(sum_w, sum_l2), xmul(sum_l, sum_l));
        if (D > 0.0f) {
            float this_scale = xdiv(xsub(xmul(sum_w, sum_xl), xmul(sum_x, sum_l)), D);
            float this_min = xdiv(xsub(xmul(sum_l2, sum_x), xmul(sum_l, sum_xl)), D);
            if (this_min > 0.0f) {
                this_min = 0.0f;
                this_scale = xdiv(sum_xl, sum_l2);
            }
            const float cur = error_of(l, this_scale, this_min);
            if (cur < best) {
                best = cur;
                r.scale = this_scale;
                r.iscale = iscale, r.from = mn;
                mn = this_min;
            }
        }
    }
    r.the_min = -mn;
    return r;
}

constexpr int Q4_BLOCKS_PER_CTA = 32;  // 8 threads per super-block, 256 threads

template <int FMT>
__global__ void __launch_bounds__(256, 2) quantize_q4k_kernel(const float *__restrict__ src, uint8_t *__restrict__ dst,
                                                              uint64_t n_blocks) {
    constexpr int BB = FMT == FMT_Q5K ? Q5K_BYTES : Q4K_BYTES, NMAX = FMT == FMT_Q5K ? 31 : 15;
    __shared__ __align__(16) uint32_t sL[Q4_BLOCKS_PER_CTA][QK / 4];  // the levels, four to a word
    const int tid = threadIdx.x;
    const int lb_ = tid >> 3;  // super-block within the CTA
    const int j = tid & 7;     // sub-block within the super-block
    for (uint64_t base = (uint64_t)blockIdx.x * Q4_BLOCKS_PER_CTA; base < n_blocks;
         base += (uint64_t)gridDim.x * Q4_BLOCKS_PER_CTA) {
        uint64_t blk = base + lb_;
        bool live = blk < n_blocks;
        uint64_t x[16], w[16];
        Best32 b{0.0f, 0.0f, 0.0f, 0.0f, false};
        if (live) {
            const ulonglong2 *xp = (const ulonglong2 *)(src + blk * QK + 32 * j);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const ulonglong2 v = xp[i];
                x[2 * i] = v.x, x[2 * i + 1] = v.y;
            }
            float sum_x2 = 0.0f;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const uint64_t xx = mul2(x[i], x[i]);
                sum_x2 = xadd(sum_x2, lo2(xx));
                sum_x2 = xadd(sum_x2, hi2(xx));
            }
            const uint64_t av_x = both(__fsqrt_rn(xdiv(sum_x2, 32.0f)));
#pragma unroll
            for (int i = 0; i < 16; i++) w[i] = add2(av_x, x[i] & 0x7fffffff7fffffffull);
            b = make_qkx2_32<FMT>(x, w);
        }
        // the eight threads of a super-block are eight consecutive lanes: exchange by shuffle
        float scales[8], mins[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
            scales[t] = __shfl_sync(0xffffffffu, b.scale, (tid & 24) + t);
            mins[t] = __shfl_sync(0xffffffffu, b.the_min, (tid & 24) + t);
        }
        float max_scale = 0.0f, max_min = 0.0f;
#pragma unroll
        for (int t = 0; t < 8; t++) {
            if (scales[t] > max_scale) max_scale = scales[t];
            if (mins[t] > max_min) max_min = mins[t];
        }
        float inv_scale = max_scale > 0.0f ? xdiv(63.0f, max_scale) : 0.0f;
        float inv_min = max_min > 0.0f ? xdiv(63.0f, max_min) : 0.0f;
        uint32_t ls[8], lm[8], lsj = 0, lmj = 0;
#pragma unroll
        for (int t = 0; t < 8; t++) {
            // the C original stores nearest_int() in a uint8_t (wraps) before MIN(63, .)
            const uint32_t a = (uint8_t)nearest_int(xmul(inv_scale, scales[t])), c = (uint8_t)nearest_int(xmul(inv_min, mins[t]));
            ls[t] = a > 63 ? 63 : a;
            lm[t] = c > 63 ? 63 : c;
            if (t == j) lsj = ls[t], lmj = lm[t];
        }
        __half dh = __float2half_rn(xdiv(max_scale, 63.0f));
        __half mh = __float2half_rn(xdiv(max_min, 63.0f));
        if (live) {
            const float d = xmul(__half2float(dh), (float)lsj);
            uint32_t lw[8];
            if (d != 0.0f) {
                const float dm = xmul(__half2float(mh), (float)lmj);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const uint64_t a = xadd2(x[2 * i], dm), c = xadd2(x[2 * i + 1], dm);
                    const float v[4] = {lo2(a), hi2(a), lo2(c), hi2(c)};
                    lw[i] = 0;
#pragma unroll
                    for (int h = 0; h < 4; h++) lw[i] |= (uint32_t)clampi(nearest_int(xdiv(v[h], d)), 0, NMAX) << (8 * h);
                }
            } else {  // the levels the search ended with
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    lw[i] = 0;
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        const uint64_t pair = x[2 * i + (h >> 1)];
                        const float v = xmul(b.iscale, xsub(h & 1 ? hi2(pair) : lo2(pair), b.from));
                        lw[i] |= (uint32_t)(b.flat ? 0 : clampi(nearest_int(v), 0, NMAX)) << (8 * h);
                    }
                }
            }
            uint4 *row = (uint4 *)&sL[lb_][8 * j];
            row[0] = make_uint4(lw[0], lw[1], lw[2], lw[3]);
            row[1] = make_uint4(lw[4], lw[5], lw[6], lw[7]);
            if (j == 0) {
                uint8_t *out = dst + blk * BB;
                uint32_t sc[3] = {0, 0, 0};
#pragma unroll
                for (int t = 0; t < 4; t++) {  // bytes t, 4 + t and 8 + t of the twelve
                    sc[0] |= (ls[t] | ((ls[t + 4] >> 4) << 6)) << (8 * t);
                    sc[1] |= (lm[t] | ((lm[t + 4] >> 4) << 6)) << (8 * t);
                    sc[2] |= ((ls[t + 4] & 0xF) | ((lm[t + 4] & 0xF) << 4)) << (8 * t);
                }
                *(uint4 *)out = make_uint4((uint32_t)__half_as_ushort(dh) | ((uint32_t)__half_as_ushort(mh) << 16), sc[0], sc[1], sc[2]);
            }
        }
        __syncthreads();
        // pack nibbles: byte i of pair k = L[64k + i] | L[64k + 32 + i] << 4; 32 words per block
        for (int o = tid; o < Q4_BLOCKS_PER_CTA * 32; o += 256) {
            const int bl = o >> 5, t = o & 31, k = t >> 3, i = t & 7;
            const uint64_t gb = base + bl;
            if (gb < n_blocks)
                *(uint32_t *)(dst + gb * BB + (FMT == FMT_Q5K ? 48 : 16) + 4 * t) = ((sL[bl][16 * k + i] & 0x0F0F0F0Fu) | ((sL[bl][16 * k + 8 + i] & 0x0F0F0F0Fu) << 4));
        }
        if constexpr (FMT == FMT_Q5K) {  // the fifth bits: bit s of qh[i] belongs to element 32 s + i
            const int bl = tid >> 3, i = tid & 7;
            const uint64_t gb = base + bl;
            if (gb < n_blocks) {
                uint32_t h = 0;
#pragma unroll
                for (int sblk = 0; sblk < 8; sblk++) h |= ((sL[bl][8 * sblk + i] >> 4) & 0x01010101u) << sblk;
                *(uint32_t *)(dst + gb * BB + 16 + 4 * i) = h;
            }
        }
        __syncthreads();
    }
}

// Symmetric search for one 16-value sub-block (nmax 32); `iscale_best` receives the factor its levels came from.
__device__ __forceinline__ float make_qx_rmse1_16(const uint64_t (&x)[8], float &iscale_best, bool &zero) {
    constexpr int nmax = 32;
    float mx = 0.0f, amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const float xi = i & 1 ? hi2(x[i >> 1]) : lo2(x[i >> 1]), ax = fabsf(xi);
        if (ax > amax) {
            amax = ax;
            mx = xi;
        }
    }
    zero = amax < 1e-15f;
    if (zero) return 0.0f;
    uint64_t w[8], wx[8];  // the weight x^2 and x^2 x of every element
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = mul2(x[i], x[i]), wx[i] = mul2(w[i], x[i]);
    auto sums = [&](float iscale, float &sumlx, float &suml2) {
        const uint64_t is2 = both(iscale);
        sumlx = 0.0f, suml2 = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint64_t l = level2<-nmax, nmax - 1>(mul2(is2, x[i])), a = mul2(wx[i], l), b = mul2(mul2(w[i], l), l);
            sumlx = xadd(sumlx, lo2(a)), suml2 = xadd(suml2, lo2(b));
            sumlx = xadd(sumlx, hi2(a)), suml2 = xadd(suml2, hi2(b));
        }
    };
    float iscale = xdiv(-(float)nmax, mx), sumlx, suml2;
    sums(iscale, sumlx, suml2);
    iscale_best = iscale;
    float scale = suml2 != 0.0f ? xdiv(sumlx, suml2) : 0.0f;
    float best = xmul(scale, sumlx);
#pragma unroll 1
    for (int is = -9; is <= 9; is++) {
        if (is == 0) continue;
        iscale = xdiv(-xadd((float)nmax, xmul(0.1f, (float)is)), mx);
        sums(iscale, sumlx, suml2);
        if (suml2 > 0.0f && xmul(sumlx, sumlx) > xmul(best, suml2)) {
            iscale_best = iscale;
            scale = xdiv(sumlx, suml2);
            best = xmul(scale, sumlx);
        }
    }
    return scale;
}

constexpr int Q6_BLOCKS_PER_CTA = 16;  // 16 threads per super-block

__global__ void __launch_bounds__(256) quantize_q6k_kernel(const float *__restrict__ src, uint8_t *__restrict__ dst,
                                                           uint64_t n_blocks) {
    __shared__ __align__(16) uint32_t sL[Q6_BLOCKS_PER_CTA][QK / 4];  // levels + 32, four to a word
    const int tid = threadIdx.x;
    const int lb_ = tid >> 4;
    const int j = tid & 15;
    for (uint64_t base = (uint64_t)blockIdx.x * Q6_BLOCKS_PER_CTA; base < n_blocks;
         base += (uint64_t)gridDim.x * Q6_BLOCKS_PER_CTA) {
        uint64_t blk = base + lb_;
        bool live = blk < n_blocks, zero = true;
        uint64_t x[8];
        float scale = 0.0f, iscale_best = 0.0f;
        if (live) {
            const ulonglong2 *xp = (const ulonglong2 *)(src + blk * QK + 16 * j);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const ulonglong2 v = xp[i];
                x[2 * i] = v.x, x[2 * i + 1] = v.y;
            }
            scale = make_qx_rmse1_16(x, iscale_best, zero);
        }
        // first sub-block with the largest |scale| decides the block scale (kquant.rs:296-303)
        float max_scale = 0.0f, max_abs = 0.0f;
#pragma unroll
        for (int t = 0; t < 16; t++) {
            float s = __shfl_sync(0xffffffffu, scale, (tid & 16) + t);
            float as = fabsf(s);
            if (as > max_abs) {
                max_abs = as;
                max_scale = s;
            }
        }
        bool zero_block = max_abs < 1e-15f;
        float iscale = zero_block ? 0.0f : xdiv(-128.0f, max_scale);
        __half dh = zero_block ? __float2half_rn(0.0f) : __float2half_rn(xdiv(1.0f, iscale));
        int sc = nearest_int(xmul(iscale, scale));
        if (sc > 127) sc = 127;
        int8_t sc8 = (int8_t)sc;
        if (live) {
            uint8_t *out = dst + blk * Q6K_BYTES;
            uint32_t lw[4] = {0, 0, 0, 0};
            if (!zero_block) {
                const float d = xmul(__half2float(dh), (float)sc8);
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float xi = i & 1 ? hi2(x[i >> 1]) : lo2(x[i >> 1]);
                    // (d == 0: the levels the search ended with; 0 for a sub-block of zeros)
                    int q = d != 0.0f ? clampi(nearest_int(xdiv(xi, d)), -32, 31) + 32
                                      : zero ? 0 : clampi(nearest_int(xmul(iscale_best, xi)), -32, 31) + 32;
                    lw[i >> 2] |= (uint32_t)q << (8 * (i & 3));
                }
            }
            *(uint4 *)&sL[lb_][4 * j] = make_uint4(lw[0], lw[1], lw[2], lw[3]);
            out[192 + j] = zero_block ? 0 : (uint8_t)sc8;
            if (j == 0) {
                unsigned short dbits = zero_block ? 0 : __half_as_ushort(dh);
                out[208] = dbits & 0xff;
                out[209] = dbits >> 8;
            }
        }
        __syncthreads();
        // ql (128 bytes) and qh (64 bytes) per block, interleaved over the two 128-halves; 48 words
        for (int o = tid; o < Q6_BLOCKS_PER_CTA * 48; o += 256) {
            const int b = o / 48, t = o % 48;
            const uint64_t gb = base + b;
            if (gb >= n_blocks) continue;
            const uint32_t *l = sL[b];
            uint32_t v;
            if (t < 32) {
                const int e0 = 32 * (t >> 4) + (t & 15);  // ql[64k + r]: elements 128k + r and 128k + r + 64
                v = (l[e0] & 0x0F0F0F0Fu) | ((l[e0 + 16] & 0x0F0F0F0Fu) << 4);
            } else {
                const int e0 = 32 * ((t - 32) >> 3) + (t & 7);
                v = ((l[e0] >> 4) & 0x03030303u) | (((l[e0 + 8] >> 4) & 0x03030303u) << 2) | (((l[e0 + 16] >> 4) & 0x03030303u) << 4) |
                    (((l[e0 + 24] >> 4) & 0x03030303u) << 6);
            }
            uint16_t *out = (uint16_t *)(dst + gb * Q6K_BYTES + 4 * t);  // (210-byte blocks: 2-byte aligned)
            out[0] = (uint16_t)v, out[1] = (uint16_t)(v >> 16);
        }
        __syncthreads();
    }
}

// One thread per 32-value group: d = amax/127, q = clamp(round_half_away(x * (1/d)), +-127).
__global__ void __launch_bounds__(256) quantize_int8_kernel(const float *__restrict__ src, int8_t *__restrict__ qs,
                                                            uint16_t *__restrict__ scales, uint64_t n_groups) {
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n_groups; g += stride) {
        const float4 *xp = (const float4 *)(src + g * 32);
        float x[32];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            float4 v = xp[i];
            x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
        }
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            float a = fabsf(x[i]);
            if (a > amax) amax = a;
        }
        float d = xdiv(amax, 127.0f);
        float id = d != 0.0f ? xdiv(1.0f, d) : 0.0f;
        uint32_t packed[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            uint32_t wv = 0;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                float pr = xmul(x[4 * i + t], id);
                float r = fminf(fmaxf(roundf(pr), -127.0f), 127.0f);
                int q = (pr != pr) ? 0 : (int)r;  // a NaN product quantizes to 0 (imp.rs:36-37)
                wv |= (uint32_t)(uint8_t)(int8_t)q << (8 * t);
            }
            packed[i] = wv;
        }
        uint4 *qp = (uint4 *)(qs + g * 32);
        qp[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        qp[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
        scales[g] = __half_as_ushort(__float2half_rn(d));
    }
}

// Int4 (crates/lapid-quant/src/imp.rs:47-71): d = (the value of largest magnitude) / -8, q = trunc(x / d + 8.5)
// clamped to 0..15, byte j = element j | element j + 16 << 4. One thread per 32-group.
__global__ void __launch_bounds__(256) quantize_int4_kernel(const float *__restrict__ src, uint8_t *__restrict__ qs,
                                                            uint16_t *__restrict__ scales, uint64_t n_groups) {
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n_groups; g += stride) {
        const float4 *xp = (const float4 *)(src + g * 32);
        float x[32];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            float4 v = xp[i];
            x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
        }
        float amax = 0.0f, mx = 0.0f;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            float a = fabsf(x[i]);
            if (amax < a) {
                amax = a;
                mx = x[i];
            }
        }
        float d = mx == 0.0f ? 0.0f : xdiv(mx, -8.0f);
        float id = d != 0.0f ? xdiv(1.0f, d) : 0.0f;
        auto nib = [&](float v) -> uint32_t {
            float t = xadd(xmul(v, id), 8.5f);
            int q = (t != t) ? 0 : (t >= 2147483648.0f ? 2147483647 : (t <= -2147483648.0f ? (-2147483647 - 1) : (int)t));
            return (uint32_t)clampi(q, 0, 15);
        };
        uint32_t packed[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t wv = 0;
#pragma unroll
            for (int t = 0; t < 4; t++) wv |= (nib(x[4 * i + t]) | (nib(x[4 * i + t + 16]) << 4)) << (8 * t);
            packed[i] = wv;
        }
        *(uint4 *)(qs + g * 16) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        scales[g] = __half_as_ushort(__float2half_rn(d));
    }
}

// MXFP4 (crates/lapid-quant/src/mxfp4.rs:27-49): one warp per 32-element block, lane = element.
//   e = u8(floor(log2(amax)) - 2 + 127) (0 for an all-zero block), d = 2^(e - 128),
//   code = the first of the 16 values KV * d closest to x.
// The reference takes log2 in f32 from its maths library; here it is taken in f64 and rounded to f32, which
// gives the correctly rounded f32 logarithm (the cases where the two could differ need a logarithm within
// 2^-29 of a rounding boundary; inputs just below a power of two, whose logarithm rounds up to the integer,
// come out the same).
__global__ void __launch_bounds__(256) quantize_mxfp4_kernel(const float *__restrict__ src, uint8_t *__restrict__ dst, uint64_t n_blocks) {
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t blk = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); blk < n_blocks; blk += warps) {
        const float x = src[blk * GROUP + lane];
        float amax = fabsf(x);
        if (!(amax == amax)) amax = 0.0f;  // f32::max ignores a NaN operand
#pragma unroll
        for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        uint32_t e = 0;
        if (amax > 0.0f) {
            const float l = (float)log2((double)amax);
            const float v = xadd(xsub(floorf(l), 2.0f), 127.0f);
            e = v <= 0.0f ? 0u : (v >= 255.0f ? 255u : (uint32_t)v);  // `as u8` saturates
        }
        const float d = e8m0_half(e);
        uint32_t best = 0;
        float best_err = fabsf(xsub(xmul(0.0f, d), x));
#pragma unroll
        for (uint32_t i = 1; i < 16; i++) {
            const float err = fabsf(xsub(xmul((float)mxfp4_kv(i), d), x));
            if (err < best_err) {
                best = i;
                best_err = err;
            }
        }
        const uint32_t hi = __shfl_down_sync(0xffffffffu, best, 16);
        uint8_t *out = dst + blk * MXFP4_BYTES;
        if (lane < 16) out[1 + lane] = (uint8_t)(best | (hi << 4));
        if (lane == 0) out[0] = (uint8_t)e;
    }
}

cudaError_t zero_gaps(void *dst, uint64_t payload, uint64_t scales_offset, uint64_t scales_bytes, uint64_t total, cudaStream_t stream) {
    uint8_t *d = (uint8_t *)dst;
    if (payload < scales_offset)
        if (cudaError_t e = cudaMemsetAsync(d + payload, 0, scales_offset - payload, stream); e != cudaSuccess) return e;
    if (scales_offset + scales_bytes < total) return cudaMemsetAsync(d + scales_offset + scales_bytes, 0, total - scales_offset - scales_bytes, stream);
    return cudaSuccess;
}

cudaError_t launch_quantize(int fmt, const float *src, uint64_t rows, uint64_t cols, uint64_t scales_offset,
                            uint64_t total_bytes, void *dst, int sm_count, cudaStream_t stream) {
    uint64_t n = rows * cols;
    // padding and gaps are zero; everything else the kernels write
    const bool planes = fmt == FMT_INT8 || fmt == FMT_INT4;  // (other formats: scales_offset is the end of the blocks)
    const uint64_t payload = fmt == FMT_INT8 ? n : fmt == FMT_INT4 ? n / 2 : scales_offset;
    cudaError_t e = zero_gaps(dst, payload, scales_offset, planes ? n / GROUP * 2 : 0, total_bytes, stream);
    if (e != cudaSuccess) return e;
    if (n == 0) return cudaSuccess;
    uint64_t cap = (uint64_t)sm_count * 8;
    if (fmt == FMT_Q4K) {
        uint64_t nb = n / QK, ctas = (nb + Q4_BLOCKS_PER_CTA - 1) / Q4_BLOCKS_PER_CTA;
        quantize_q4k_kernel<FMT_Q4K><<<(int)(ctas < cap ? ctas : cap), 256, 0, stream>>>(src, (uint8_t *)dst, nb);
    } else if (fmt == FMT_Q5K) {
        uint64_t nb = n / QK, ctas = (nb + Q4_BLOCKS_PER_CTA - 1) / Q4_BLOCKS_PER_CTA;
        quantize_q4k_kernel<FMT_Q5K><<<(int)(ctas < cap ? ctas : cap), 256, 0, stream>>>(src, (uint8_t *)dst, nb);
    } else if (fmt == FMT_Q6K) {
        uint64_t nb = n / QK, ctas = (nb + Q6_BLOCKS_PER_CTA - 1) / Q6_BLOCKS_PER_CTA;
        quantize_q6k_kernel<<<(int)(ctas < cap ? ctas : cap), 256, 0, stream>>>(src, (uint8_t *)dst, nb);
    } else if (fmt == FMT_MXFP4) {
        uint64_t nb = n / GROUP, ctas = (nb + 7) / 8;
        quantize_mxfp4_kernel<<<(int)(ctas < cap ? ctas : cap), 256, 0, stream>>>(src, (uint8_t *)dst, nb);
    } else if (fmt == FMT_INT4) {
        uint64_t ng = n / GROUP, ctas = (ng + 255) / 256;
        uint8_t *d = (uint8_t *)dst;
        quantize_int4_kernel<<<(int)(ctas < cap ? ctas : cap), 256, 0, stream>>>(src, d, (uint16_t *)(d + scales_offset), ng);
    } else {
        uint64_t ng = n / GROUP, ctas = (ng + 255) / 256;
        uint8_t *d = (uint8_t *)dst;
        quantize_int8_kernel<<<(int)(ctas < cap ? ctas : cap), 256, 0, stream>>>(src, (int8_t *)d,
                                                                                (uint16_t *)(d + scales_offset), ng);
    }
    return cudaGetLastError();
}

}  // namespace lb

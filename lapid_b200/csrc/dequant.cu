// Dequantization to f32, bit-identical to lapid-quant, and the GGUF -> lapid layout conversion.
//
//   dequantize_q4k   crates/lapid-quant/src/kquant.rs:337-352   y = (d*sc)*q - (dmin*m)
//   dequantize_q5k   crates/lapid-quant/src/kquant.rs:355-373   y = (d*sc)*(q + 16*h) - (dmin*m)
//   dequantize_q6k   crates/lapid-quant/src/kquant.rs:376-396   y = (d*sc)*(q-32)
//   Int8 rows        crates/lapid-quant/src/imp.rs:143-148      y = f32(q) * f32(d)
//   Int4 rows        crates/lapid-quant/src/imp.rs:148-156      y = f32(nibble - 8) * f32(d)
//   from_ggml_blocks crates/lapid-quant/src/imp.rs:171-200
//
// The kernels are bound by the 4 bytes written per element (HBM store bandwidth), as long as expanding costs few
// instructions: a thread takes four consecutive elements, which share the header reads and go out as one 16-byte store
// (14336 x 4096 Q4_K: 63 us, 4.2 TB/s; one element per thread, which this replaces, 148 us).
#include <type_traits>

#include "common.cuh"
#include "iquant.cuh"
#include "kernels.h"

namespace lb {

// A row-major matrix of any format (cols a multiple of the format's block, so blocks follow each other in the order of the elements; FMT < 0:
// plain f32). Buffers start at multiples of 16 bytes.
struct Matrix {
    const uint8_t *p, *iq_grid;
    uint64_t scales_offset;
};
// Elements pos .. pos + 3, pos = r * cols + c a multiple of 4.
template <int FMT> __device__ __forceinline__ float4 element4(const Matrix &t, uint64_t pos) {
    float y[4] = {};
    if constexpr (FMT == FMT_Q4K || FMT == FMT_Q5K) {
        const uint8_t *b = t.p + pos / QK * (FMT == FMT_Q4K ? Q4K_BYTES : Q5K_BYTES);
        const int e = (int)(pos % QK), j = e >> 6, h = (e >> 5) & 1, l = e & 31;
        const uint4 hd = *(const uint4 *)b;
        const uint32_t q4 = *(const uint32_t *)(b + (FMT == FMT_Q4K ? 16 : 48) + 32 * j + l);
        const uint32_t q5 = FMT == FMT_Q5K ? *(const uint32_t *)(b + 16 + l) : 0;
        int sc0, mn0, sc1, mn1;
        scale_min_pair(j, hd.y, hd.z, hd.w, sc0, mn0, sc1, mn1);
        const float d1 = xmul(half_bits_to_float(hd.x & 0xffffu), (float)(h ? sc1 : sc0));
        const float m1 = xmul(half_bits_to_float(hd.x >> 16), (float)(h ? mn1 : mn0));
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int q = ((q4 >> (8 * i + 4 * h)) & 15) + (FMT == FMT_Q5K ? ((q5 >> (8 * i + 2 * j + h)) & 1) << 4 : 0);
            y[i] = xsub(xmul(d1, (float)q), m1);
        }
    } else if constexpr (FMT == FMT_Q6K) {  // 2-byte aligned blocks
        const uint8_t *b = t.p + pos / QK * Q6K_BYTES;
        const int e = (int)(pos % QK), n = e >> 7, w = (e >> 5) & 3, l = e & 31;
        const uint32_t ql = ld32_by16(b + 64 * n + 32 * (w & 1) + l), qh = ld32_by16(b + 128 + 32 * n + l);
        const float dsc = xmul(half_bits_to_float(ld16(b + 208)), (float)(int8_t)b[192 + 8 * n + 2 * w + (l >> 4)]);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int q = ((ql >> (8 * i + 4 * (w >> 1))) & 15) | (((qh >> (8 * i + 2 * w)) & 3) << 4);
            y[i] = xmul(dsc, (float)(q - 32));
        }
    } else if constexpr (is_iq(FMT)) {  // (crates/lapid-quant/src/iq2.rs:38-90, iq3.rs:18-39)
        const uint8_t *b = t.p + pos / QK * iq_block_bytes(FMT);
        const int e = (int)(pos % QK);
        uint32_t lo, hi, signs;
        iq_group8<FMT>(b, e >> 3, t.iq_grid, lo, hi, signs);
        const float db = iq_half_scale<FMT>(b, e >> 4);
        const uint32_t gr = (e & 4) ? hi : lo;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float v = xmul(db, (float)((gr >> (8 * i)) & 255u));
            y[i] = (signs >> ((e & 4) + i)) & 1u ? -v : v;
        }
    } else if constexpr (FMT == FMT_INT4) {  // (crates/lapid-quant/src/imp.rs:148-156)
        const uint64_t g = pos >> 5;
        const uint32_t e = (uint32_t)(pos & 31), w = *(const uint32_t *)(t.p + g * 16 + (e & 15));
        const float d = half_bits_to_float(((const uint16_t *)(t.p + t.scales_offset))[g]);
#pragma unroll
        for (int i = 0; i < 4; i++) y[i] = xmul((float)((int)((w >> (8 * i + (e < 16 ? 0 : 4))) & 15) - 8), d);
    } else if constexpr (FMT == FMT_INT8) {
        const char4 q = *(const char4 *)(t.p + pos);
        const float d = half_bits_to_float(((const uint16_t *)(t.p + t.scales_offset))[pos >> 5]);
        y[0] = xmul((float)q.x, d), y[1] = xmul((float)q.y, d), y[2] = xmul((float)q.z, d), y[3] = xmul((float)q.w, d);
    } else if constexpr (FMT == FMT_MXFP4) {  // unaligned blocks: byte by byte
        const uint8_t *b = t.p + (pos >> 5) * MXFP4_BYTES;
#pragma unroll
        for (int i = 0; i < 4; i++) y[i] = mxfp4_element(b, (uint32_t)((pos + i) & 31));
    } else {
        return *(const float4 *)((const float *)t.p + pos);
    }
    return make_float4(y[0], y[1], y[2], y[3]);
}

template <int FMT> __global__ void __launch_bounds__(256) dequant_kernel(Matrix t, float *__restrict__ dst, uint64_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * 1024;
    for (uint64_t i = ((uint64_t)blockIdx.x * 256 + threadIdx.x) * 4; i < n; i += stride) *(float4 *)(dst + i) = element4<FMT>(t, i);
}

// Gather: out[i, :] = dequant(table[ids[i], :]) (lapid's Kernel::Gather, crates/lapid-compiler/src/ir.rs:284-300;
// CPU: crates/lapid-cpu/src/rows.rs:164-215 -- the embedding lookup from a quantized table). One CTA
// per (output row, 256 threads' columns); an index outside [0, rows) is not read: the row is skipped and bit
// 128 of the host-visible status word reports it ("index_out_of_range" after the launch sequence).
template <int FMT, int VEC>
__global__ void __launch_bounds__(256) gather_kernel(Matrix t, const int32_t *__restrict__ ids, uint64_t rows, uint64_t cols, uint64_t count,
                                                     float *__restrict__ out, int *status) {
    const uint64_t per_row = (cols + 256 * VEC - 1) / (256 * VEC);
    for (uint64_t u = blockIdx.x; u < count * per_row; u += gridDim.x) {
        const uint64_t i = u / per_row, c = ((u % per_row) * 256 + threadIdx.x) * VEC;
        const int64_t r = ids[i];
        if (r < 0 || (uint64_t)r >= rows) {
            if (threadIdx.x == 0 && status) atomicOr(status, 128);
            continue;
        }
        if (c >= cols) continue;
        if constexpr (VEC == 4) *(float4 *)(out + i * cols + c) = element4<FMT>(t, (uint64_t)r * cols + c);
        else out[i * cols + c] = ((const float *)t.p)[(uint64_t)r * cols + c];  // (an f32 table of any width)
    }
}

// GGUF block_q8_0 (f16 d + 32 x i8, 34 bytes) -> quants plane + scales plane, and block_q4_0 (f16 d + 16 nibble bytes, 18 bytes;
// the same nibble order) -> nibble plane + scales plane. A thread moves 16 bytes of payload: one store of the plane, read as
// 16-bit halves, which is how the blocks are aligned; the first of a group also moves the scale. Bound by HBM.
template <int PAYLOAD> __global__ void __launch_bounds__(256) blocks_to_planes_kernel(const uint8_t *__restrict__ blocks, uint8_t *__restrict__ qs,
                                                                                      uint8_t *__restrict__ scales, uint64_t n_groups) {
    constexpr int PER = PAYLOAD / 16;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_groups * PER; i += stride) {
        const uint64_t g = i / PER;
        const int t = (int)(i % PER);
        const uint8_t *b = blocks + g * (PAYLOAD + 2), *q = b + 2 + 16 * t;
        *(uint4 *)(qs + 16 * i) = make_uint4(ld32_by16(q), ld32_by16(q + 4), ld32_by16(q + 8), ld32_by16(q + 12));
        if (t == 0) *(uint16_t *)(scales + 2 * g) = (uint16_t)ld16(b);
    }
}

static int grid_for(uint64_t work_items, int sm_count) {
    uint64_t want = work_items;
    uint64_t cap = (uint64_t)sm_count * 8;  // 8 resident CTAs of 256 threads per SM
    return (int)(want < cap ? (want ? want : 1) : cap);
}

// Calls f(std::integral_constant<int, FMT>) for the format; f32 tables are FMT -1.
template <class F> static cudaError_t with_format(int fmt, F f) {
    switch (fmt) {
        case FMT_Q4K: return f(std::integral_constant<int, FMT_Q4K>());
        case FMT_Q5K: return f(std::integral_constant<int, FMT_Q5K>());
        case FMT_Q6K: return f(std::integral_constant<int, FMT_Q6K>());
        case FMT_MXFP4: return f(std::integral_constant<int, FMT_MXFP4>());
        case FMT_INT8: return f(std::integral_constant<int, FMT_INT8>());
        case FMT_INT4: return f(std::integral_constant<int, FMT_INT4>());
        case FMT_IQ2XXS: return f(std::integral_constant<int, FMT_IQ2XXS>());
        case FMT_IQ2XS: return f(std::integral_constant<int, FMT_IQ2XS>());
        case FMT_IQ2S: return f(std::integral_constant<int, FMT_IQ2S>());
        case FMT_IQ3XXS: return f(std::integral_constant<int, FMT_IQ3XXS>());
        default: return f(std::integral_constant<int, -1>());
    }
}
static cudaError_t matrix_of(int fmt, const void *p, uint64_t scales_offset, Matrix &t) {
    t = Matrix{(const uint8_t *)p, nullptr, scales_offset};
    if (is_iq(fmt)) {
        const uint8_t *grids = iq_grids();
        if (!grids) return cudaErrorNotReady;
        t.iq_grid = grids + iq_grid_offset(fmt);
    }
    return cudaSuccess;
}

cudaError_t launch_dequantize(int fmt, const void *src, uint64_t rows, uint64_t cols, uint64_t scales_offset,
                              float *dst, int sm_count, cudaStream_t stream) {
    const uint64_t n = rows * cols;
    if (n == 0) return cudaSuccess;
    Matrix t;
    if (cudaError_t e = matrix_of(fmt, src, scales_offset, t); e != cudaSuccess) return e;
    return with_format(fmt, [&](auto f) {  // (n is a multiple of 32)
        dequant_kernel<f.value><<<grid_for((n + 1023) / 1024, sm_count), 256, 0, stream>>>(t, dst, n);
        return cudaGetLastError();
    });
}

// fmt < 0: plain f32 table
cudaError_t launch_gather(int fmt, const void *table, uint64_t scales_offset, const int32_t *ids, uint64_t rows, uint64_t cols,
                          uint64_t count, float *out, int *status, int sm_count, cudaStream_t stream) {
    if (count == 0 || cols == 0) return cudaSuccess;
    Matrix t;
    if (cudaError_t e = matrix_of(fmt, table, scales_offset, t); e != cudaSuccess) return e;
    if (cols % 4) {
        gather_kernel<-1, 1><<<grid_for(count * ((cols + 255) / 256), sm_count), 256, 0, stream>>>(t, ids, rows, cols, count, out, status);
        return cudaGetLastError();
    }
    return with_format(fmt, [&](auto f) {
        gather_kernel<f.value, 4><<<grid_for(count * ((cols + 1023) / 1024), sm_count), 256, 0, stream>>>(t, ids, rows, cols, count, out, status);
        return cudaGetLastError();
    });
}

template <int PAYLOAD> static cudaError_t launch_planes(const void *blocks, void *dst, uint64_t scales_offset, uint64_t n_groups, int sm_count, cudaStream_t stream) {
    if (n_groups == 0) return cudaSuccess;
    const uint8_t *b = (const uint8_t *)blocks;
    uint8_t *d = (uint8_t *)dst;
    blocks_to_planes_kernel<PAYLOAD><<<grid_for((n_groups * (PAYLOAD / 16) + 255) / 256, sm_count), 256, 0, stream>>>(b, d, d + scales_offset, n_groups);
    return cudaGetLastError();
}
cudaError_t launch_q4_0_to_planes(const void *blocks, void *dst, uint64_t scales_offset, uint64_t n_groups, int sm_count, cudaStream_t stream) {
    return launch_planes<16>(blocks, dst, scales_offset, n_groups, sm_count, stream);
}
cudaError_t launch_q8_0_to_planes(const void *blocks, void *dst, uint64_t scales_offset, uint64_t n_groups, int sm_count, cudaStream_t stream) {
    return launch_planes<32>(blocks, dst, scales_offset, n_groups, sm_count, stream);
}

}  // namespace lb

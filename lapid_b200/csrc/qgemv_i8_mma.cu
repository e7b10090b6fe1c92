// Int8 planes (GGUF Q8_0 in lapid's plane layout) and Int4 nibble planes: decode GEMV for 1..8 activation rows on the
// warp-level int8 tensor-core instruction. Arithmetic as in qgemv_i8.cu / qgemv_i4.cu: exact integer dot products per
// 32-element group, one f32 step per group, f32(dot) * da * db (crates/lapid-cpu/src/matmul/
// qkernels.rs:60-84; the order of the two scale multiplications and of the f32 sums differs).
//
// Int8 weights are plain signed bytes, so they are the MMA's A operand as they lie in memory: one
// `mma.sync.m16n8k32.s8.s8` covers 16 weight rows x one 32-element group x 8 activation rows, and
// nothing has to be unpacked. Int4: a nibble q (weight q - 8) becomes the int8 value 16 (q - 8) with two logic operations
// per register, the exact factor 1/16 goes into the group scale. A CTA takes a share of the 16-row tiles, cut along K into chunks of 512
// (RAGGED: 256) quants; these (tile, chunk) units are dealt out to its warps in order, whatever tile they belong to (a tile of 2880 has six
// chunks of 512: dealt out tile by tile, two of eight warps had nothing to do). The warps' partial 16x8 tiles are summed in shared memory in
// the order of the chunks, up to four tiles between two barriers. A warp's stage is 16 rows x one chunk plus their f16 scales, brought in by
// `cp.async` (16 bytes per lane and instruction) into a layout of the kernel's choosing: 16-byte
// chunk c of row r sits at chunk position c ^ 2 (r & 3) (Int4: c ^ (r & 7)), which makes the fragment loads (64 bits per
// lane: within a group the k order is free, lane t takes quants 8t..8t+7 of both operands; Int4: elements 0..15 are
// the low nibbles of the group's 16 bytes, 16..31 the high ones) bank-conflict free. Stages of the next chunks are in flight
// while one is consumed (two per warp, cp.async groups), and the first ones are issued before the
// programmatic-dependent-launch wait. Activations: the same shared-memory tiles as the K-quant tensor-core kernels.
//
// RAGGED: K any multiple of 32. The last chunk of a row is partly there (the copies past it are zero-filled, its missing groups
// skipped), and a row's scales start at any even byte: the two aligned 16-byte pieces around a chunk's 16 bytes of scales
// are staged and read with 16-bit loads. Widths that are no multiple of 512 are common (2880, shards of 7680). So that the f32 sums are no further
// off than those of the generic dp4a kernel, the even and odd groups of a chunk are summed apart, the chunks behind that, the warps as a balanced
// tree (against f64, three rows, K 2880: 7.5e-8; 14368: 8.4e-8, with chunks of 512 8.9e-8).
// What bounds it is latency: 8-16 warps an SM wait for their copies, then for each other. Sixteen warps with chunks of 256 keep as many bytes in flight as
// eight with 512. Tile by tile with eight warps -> units in order with sixteen, us: three rows int8 15360 x 2880 16.8 -> 14.7, seven rows 4096 x 11008 19.6 -> 14.7,
// three rows Int4 15360 x 2880 22.4 -> 13.4; a token of three rows through 12 layers of 2880 / 7680 606 -> 574. Where K is a multiple of 512, eight warps stay
// (sixteen with 256: 14336 x 4096 15.6 -> 17.2), units in order: eight rows int8 8192 x 1024 6.2 -> 5.5, four rows Int4 4096 x 4096 7.5 -> 6.4; EVEN as before.
// Less than a tile for every CTA pays 0.1 us for the order (eight rows int8 512 x 1024 3.66 -> 3.77, 3.89 while the warps' places were found by subtracting in a loop).
//
// Several projections over the same activations (q, k, v; gate, up) run as one launch over the concatenated tiles. Early
// mode (GemvArgs::early): activations are read and tiles computed before the dependency wait, which comes before the first store.
#include "common.cuh"
#include "kernels.h"
#include "tp_ll.cuh"

namespace lb {
namespace i8m {

// Quants per row and stage. RAGGED: 256, for sixteen warps; else 512, for eight (the rings are as large either way): see launch_k.
__host__ __device__ constexpr int chunk_of(bool ragged) { return ragged ? 256 : 512; }
constexpr int STAGES = 2;
constexpr float MAGIC = 12582912.0f;
__host__ __device__ constexpr uint32_t row_bytes(bool i4, bool ragged) { return chunk_of(ragged) / (i4 ? 2 : 1); }  // of a row's quants in a stage
__host__ __device__ constexpr uint32_t scale_bytes() { return 32; }  // (RAGGED: eight scales on any even byte)
__host__ __device__ constexpr uint32_t stage_bytes(bool i4, bool ragged) { return 16 * (row_bytes(i4, ragged) + scale_bytes()); }

__device__ __forceinline__ uint32_t s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16 weight rows x 32 k x 8 activation rows, signed bytes; the accumulators start at the bit
// pattern of 1.5 * 2^23, so the result reinterpreted as f32 is 12582912 + dot (|dot| < 2^22)
__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0x4B400000));
}
// 16 bytes; only the first `bytes` (0 or 16) are read, the rest is zero
__device__ __forceinline__ void copy16(uint8_t *dst, const uint8_t *src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s32(dst)), "l"(src), "r"(bytes) : "memory");
}

__host__ __device__ constexpr uint32_t act_block_bytes(uint32_t rows) { return 256 * rows + 512; }  // per 256 k, as the K-quant kernels' tiles

// EVEN: a tile's chunks divide evenly over the warps, which then keep their places from tile to tile.
template <bool I4, bool RAGGED, bool EVEN, int WARPS, int NG>
__global__ void __launch_bounds__(WARPS * 32, 1) qgemv_i8_mma_kernel(const __grid_constant__ GemvGroupT<NG> grp, uint32_t round_in, uint32_t buffers_in, uint32_t inverse) {
    const uint32_t round_tiles = EVEN ? 1 : round_in, buffers = EVEN ? 2 : buffers_in;
    constexpr int THREADS = WARPS * 32;
    constexpr int KC = chunk_of(RAGGED), CPR = KC / (I4 ? 32 : 16), RPI = 32 / CPR;  // 16-byte copies a row, rows an instruction
    constexpr uint32_t ROWB = row_bytes(I4, RAGGED), Q_BYTES = 16 * ROWB, SCB = scale_bytes(), STAGE = stage_bytes(I4, RAGGED);
    extern __shared__ __align__(128) uint8_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gq = lane >> 2, t4 = lane & 3;
    const uint32_t M = grp.item[0].rows, k = grp.item[0].k, kg = k / GROUP, rowb = I4 ? k / 2 : k;
    const uint32_t iters = (k + KC - 1) / KC;
    const uint32_t ABLK = act_block_bytes(M);
    const uint32_t tasks = grp.task_end[NG == 1 ? 0 : grp.count - 1];
    const uint32_t t_lo = (uint32_t)(((uint64_t)tasks * blockIdx.x) / gridDim.x);
    const uint32_t t_hi = (uint32_t)(((uint64_t)tasks * (blockIdx.x + 1)) / gridDim.x);
    // the member a 16-row tile belongs to, and the tile's number inside it
    auto locate = [&](uint32_t t, uint32_t &local) -> int {
        int i = 0;
        if constexpr (NG > 1)
            while (t >= grp.task_end[i]) i++;
        local = i ? t - grp.task_end[i - 1] : t;
        return i;
    };

    uint8_t *ring = smem + (size_t)warp * (STAGES * STAGE);
    float *red = (float *)(smem + (size_t)WARPS * STAGES * STAGE);  // [buffers][round_tiles][WARPS][128]
    uint8_t *acts = (uint8_t *)(red + buffers * round_tiles * WARPS * 128);

    // A CTA's work is its (tile, chunk) units in order, dealt out to the warps one by one. Producer cursor: unit, as tile and chunk, and ring slot. One
    // stage = 512 (RAGGED or Int4: half of that) + 32 sixteen-byte copies.
    // `inverse` divides numbers up to WARPS by `iters`: subtracting in a loop takes longer than the smallest launches' products.
    const uint32_t first_tile = EVEN ? 0 : warp * inverse >> 16, step_tiles = EVEN ? 0 : WARPS * inverse >> 16, step = WARPS - step_tiles * iters;
    uint32_t pt = t_lo + first_tile, pit = warp - first_tile * iters, pslot = 0;
    uint32_t ct = pt, it = pit;  // the unit being multiplied
    auto issue = [&]() {
        if (pt < t_hi) {
            uint32_t local;
            const GemvArgs &p = grp.item[locate(pt, local)];
            uint8_t *dst = ring + (size_t)pslot * STAGE;
            const uint32_t row0 = local * 16;
            // rows past the end repeat the last one; their outputs are dropped
#pragma unroll
            for (int i = 0; i < 16 / RPI; i++) {  // lane -> 16-byte chunk lane % CPR of row RPI i + lane / CPR
                const uint32_t r = RPI * i + lane / CPR, c = lane % CPR;
                const uint8_t *src = p.w + (size_t)min(row0 + r, p.n - 1) * rowb;
                const uint32_t at = pit * ROWB + 16 * c;
                const bool there = !RAGGED || at < rowb;
                copy16(dst + r * ROWB + 16 * (c ^ (I4 ? r & 7 : 2 * (r & 3))), src + (there ? at : 0), there ? 16 : 0);
            }
            if constexpr (RAGGED) {  // scales: piece (lane & 1) of row lane / 2 of the two aligned ones; the readable bytes end with the matrix's last line
                const uint64_t end = (p.scales_offset + (uint64_t)p.n * kg * 2 + 15) & ~(uint64_t)15;
                const uint64_t at = ((p.scales_offset + ((uint64_t)min(row0 + (lane >> 1), p.n - 1) * kg + pit * (KC / GROUP)) * 2) & ~(uint64_t)15) + 16 * (lane & 1);
                copy16(dst + Q_BYTES + 16 * lane, p.w + (at < end ? at : 0), at < end ? 16 : 0);
            } else {  // scales: lane -> half (lane & 1) of row lane / 2
                const uint32_t row = min(row0 + (lane >> 1), p.n - 1);
                copy16(dst + Q_BYTES + 16 * lane, p.w + p.scales_offset + ((size_t)row * kg + (size_t)pit * (KC / GROUP)) * 2 + 16 * (lane & 1), 16);
            }
            pslot ^= 1;
            if constexpr (EVEN) {
                pit += WARPS;
                if (pit >= iters) pit = warp, pt++;
            } else {
                pit += step, pt += step_tiles;
                if (pit >= iters) pit -= iters, pt++;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");  // an empty group keeps the count in step
    };
    issue();
    issue();

    bool waited = grp.item[0].early == 0;
    if (waited) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    __shared__ TpPushCtx tp_ctx;  // (a launch that pushes is never early and has one member)
    if (grp.item[0].tp && threadIdx.x == 0) tp_push_ctx_load(&tp_ctx, grp.item[0].tp);
    {   // the activation tiles, once per CTA (their own cp.async group, waited for with the first stage)
        const uint32_t chunks = ((k + QK - 1) / QK) * ABLK / 16;
        const uint8_t *src = (const uint8_t *)grp.item[0].qa;
        for (uint32_t c = threadIdx.x; c < chunks; c += THREADS) copy16(acts + 16 * c, src + 16 * (size_t)c, 16);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }

    const uint32_t colq = (uint32_t)gq < M ? gq : 0;      // activation row of this lane's B fragment
    const uint32_t cp = (uint32_t)(2 * t4) < M ? t4 : 0;  // activation row pair of this lane's C fragment
    uint32_t cslot = 0, par = 0;
    for (uint32_t t0 = t_lo; t0 < t_hi; t0 += round_tiles) {
        const uint32_t t1 = min(t0 + round_tiles, t_hi);
        while (ct < t1) {
            const uint32_t tile = ct;
            uint32_t local;
            const GemvArgs &p = grp.item[locate(tile, local)];
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            do {
                asm volatile("cp.async.wait_group 1;" ::: "memory");  // all but the newest group: this stage has landed
                __syncwarp();
                const uint8_t *stage = ring + (size_t)cslot * STAGE;
                const uint16_t *sr0 = nullptr, *sr1 = nullptr;  // RAGGED: the scales of this lane's two weight rows
                if constexpr (RAGGED) {
                    auto skew = [&](uint32_t r) { return (uint32_t)((min(local * 16 + r, p.n - 1) * kg + it * (KC / GROUP)) * 2) & 15u; };  // (scales_offset is a multiple of 16)
                    sr0 = (const uint16_t *)(stage + Q_BYTES + gq * SCB + skew(gq));
                    sr1 = (const uint16_t *)(stage + Q_BYTES + (gq + 8) * SCB + skew(gq + 8));
                }
#pragma unroll
                for (int blk = 0; blk < KC / QK; blk++) {  // the chunk's 256-wide activation tiles
                const uint8_t *ab = acts + (size_t)(KC / QK * it + blk) * ABLK;
                const float2 *dsp = (const float2 *)(ab + 256 * M) + 2 * cp;  // {da[c0], da[c1]} of group s at [8 * (s >> 1) + (s & 1)]
                // the f16 scales of this lane's two weight rows for the tile's eight groups
                uint4 sw0 = make_uint4(0, 0, 0, 0), sw1 = sw0;
                if constexpr (!RAGGED) {
                    sw0 = *(const uint4 *)(stage + Q_BYTES + gq * SCB + 16 * blk);
                    sw1 = *(const uint4 *)(stage + Q_BYTES + (gq + 8) * SCB + 16 * blk);
                }
                const uint32_t s0[4] = {sw0.x, sw0.y, sw0.z, sw0.w}, s1[4] = {sw1.x, sw1.y, sw1.z, sw1.w};
                float part[2][4] = {};  // RAGGED: the tile's even and odd groups
#pragma unroll
                for (int s = 0; s < 8; s++) {
                    if (RAGGED && it * (KC / GROUP) + s >= kg) break;
                    float (&sum)[4] = RAGGED ? part[s & 1] : acc;
                    uint32_t a0, a1, a2, a3;
                    if constexpr (I4) {
                        const int c16 = 8 * blk + s;  // the group's 16 bytes are one chunk of the row
                        const uint2 w_lo = *(const uint2 *)(stage + gq * ROWB + 16 * (c16 ^ (gq & 7)) + 8 * (t4 & 1));
                        const uint2 w_hi = *(const uint2 *)(stage + (gq + 8) * ROWB + 16 * (c16 ^ (gq & 7)) + 8 * (t4 & 1));
                        const int sh = t4 < 2 ? 4 : 0;  // low nibbles (elements 0..15 of the group) for t4 < 2, high nibbles above
                        a0 = ((w_lo.x << sh) & 0xF0F0F0F0u) ^ 0x80808080u, a2 = ((w_lo.y << sh) & 0xF0F0F0F0u) ^ 0x80808080u;
                        a1 = ((w_hi.x << sh) & 0xF0F0F0F0u) ^ 0x80808080u, a3 = ((w_hi.y << sh) & 0xF0F0F0F0u) ^ 0x80808080u;
                    } else {
                        const int c16 = 2 * (8 * blk + s) + (t4 >> 1);  // 16-byte chunk of the row that holds quants 8 t4 .. 8 t4 + 7 of the group
                        const uint2 w_lo = *(const uint2 *)(stage + gq * ROWB + 16 * (c16 ^ (2 * (gq & 3))) + 8 * (t4 & 1));
                        const uint2 w_hi = *(const uint2 *)(stage + (gq + 8) * ROWB + 16 * (c16 ^ (2 * (gq & 3))) + 8 * (t4 & 1));
                        a0 = w_lo.x, a1 = w_hi.x, a2 = w_lo.y, a3 = w_hi.y;
                    }
                    const uint2 b = *(const uint2 *)(ab + s * (M * 32) + colq * 32 + 8 * t4);
                    int c[4];
                    mma_s8(c, a0, a1, a2, a3, b.x, b.y);
                    const float2 da = dsp[8 * (s >> 1) + (s & 1)];
                    const uint32_t h0 = RAGGED ? sr0[s] : (s0[s >> 1] >> (16 * (s & 1))) & 0xffff;
                    const uint32_t h1 = RAGGED ? sr1[s] : (s1[s >> 1] >> (16 * (s & 1))) & 0xffff;
                    const float w0 = half_bits_to_float(h0) * (I4 ? 0.0625f : 1.0f), w1 = half_bits_to_float(h1) * (I4 ? 0.0625f : 1.0f);  // (Int4: the dot is 16 times too large)
                    sum[0] = fmaf((__int_as_float(c[0]) - MAGIC) * da.x, w0, sum[0]);
                    sum[1] = fmaf((__int_as_float(c[1]) - MAGIC) * da.y, w0, sum[1]);
                    sum[2] = fmaf((__int_as_float(c[2]) - MAGIC) * da.x, w1, sum[2]);
                    sum[3] = fmaf((__int_as_float(c[3]) - MAGIC) * da.y, w1, sum[3]);
                }
                if constexpr (RAGGED)
#pragma unroll
                    for (int i = 0; i < 4; i++) acc[i] += part[0][i] + part[1][i];
                }
                __syncwarp();  // every lane is done reading the slot before it is refilled
                issue();
                cslot ^= 1;
                if constexpr (EVEN) {
                    it += WARPS;
                    if (it >= iters) it = warp, ct++;
                } else {
                    it += step, ct += step_tiles;
                    if (it >= iters) it -= iters, ct++;
                }
            } while (ct == tile);
            float *mine = red + ((size_t)(par * round_tiles + tile - t0) * WARPS + warp) * 128;
#pragma unroll
            for (int i = 0; i < 4; i++) mine[i * 32 + lane] = acc[i];
        }

        // ---- sum the warps' partial tiles and store: one output per thread and step. Unit c of a tile is warp (first + c) % WARPS's, and so are
        // c + WARPS, ...: the partial sums are added as a balanced tree in the order of c
        __syncthreads();  // with two buffers: the other one is free again once every warp got here
        if (!waited) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            waited = true;
        }
        const uint32_t e = threadIdx.x % 128;
        for (uint32_t tile = t0 + threadIdx.x / 128; tile < t1; tile += THREADS / 128) {
            uint32_t local;
            const GemvArgs &p = grp.item[locate(tile, local)];
            const float *src = red + (par * round_tiles + tile - t0) * (WARPS * 128) + e;
            float q[WARPS];
            if constexpr (EVEN) {
#pragma unroll
                for (int c = 0; c < WARPS; c++) q[c] = src[c * 128];
            } else {
                const uint32_t first = (tile - t_lo) * iters;  // (the warps are a power of two: it may wrap)
#pragma unroll
                for (int c = 0; c < WARPS; c++) q[c] = (uint32_t)c < iters ? src[((first + c) % WARPS) * 128] : 0.0f;
            }
#pragma unroll
            for (int n = WARPS / 2; n; n /= 2)
#pragma unroll
                for (int c = 0; c < n; c++) q[c] = q[2 * c] + q[2 * c + 1];
            float v = q[0];
            const uint32_t el = e & 31, i = e >> 5;
            const uint32_t row = local * 16 + (el >> 2) + ((i & 2) ? 8 : 0);
            const uint32_t r = 2 * (el & 3) + (i & 1);
            if (row < p.n && r < M) {
                const uint32_t bt = r / p.m, ri = r % p.m;
                if (p.extra && !p.epi.n) v += p.extra[p.ex_off + (int64_t)bt * p.ex_s0 + (int64_t)ri * p.ex_s1 + (int64_t)row * p.ex_s2];
                if (p.tp) tp_push_value(&tp_ctx, (uint64_t)r * p.n + row, v);  // row-parallel partial: to every rank
                else p.out[p.out_off + (uint64_t)bt * p.out_bs + (uint64_t)ri * p.out_rs + row] = v;
            }
        }
        if (buffers > 1) par ^= 1;
        else if (t1 < t_hi) __syncthreads();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

static bool ragged(uint32_t k) { return k % chunk_of(false) != 0; }
constexpr size_t SMEM_MAX = 227 * 1024 - 256;
static size_t smem_bytes(bool i4, int warps, uint32_t rows, uint32_t k, uint32_t parts = 1) {  // parts: tiles whose partial sums there is room for
    return (size_t)warps * (STAGES * stage_bytes(i4, ragged(k)) + parts * 128 * 4) + (size_t)((k + QK - 1) / QK) * act_block_bytes(rows);
}

template <bool I4, bool RAGGED, bool EVEN, int WARPS, int NG> static cudaError_t launch_e(const GemvGroup &group, int sm_count, bool pdl, cudaStream_t stream) {
    auto kern = qgemv_i8_mma_kernel<I4, RAGGED, EVEN, WARPS, NG>;
    GemvGroupT<NG> g{};
    g.count = group.count;
    uint32_t tasks = 0;
    for (int i = 0; i < group.count; i++) {
        g.item[i] = group.item[i];
        g.task_end[i] = tasks += (group.item[i].n + 15) / 16;
    }
    // Tiles between two barriers: one where a tile's units divide evenly over the warps, else up to four; two buffers for their partial sums save a
    // second barrier. As far as it fits.
    const uint32_t rows = g.item[0].rows, k = g.item[0].k;
    auto fits = [&](uint32_t parts) { return smem_bytes(I4, WARPS, rows, k, parts) <= SMEM_MAX; };
    const uint32_t buffers = EVEN || fits(2) ? 2 : 1;
    uint32_t round = 1;
    while (!EVEN && round < 4 && fits(2 * buffers * round)) round *= 2;
    const size_t smem = smem_bytes(I4, WARPS, rows, k, buffers * round);
    static DynamicSmemOptIn opted;
    if (cudaError_t e = opted.raise((const void *)kern, smem); e != cudaSuccess) return e;
    uint32_t fit = (uint32_t)((227 * 1024) / (smem + 1024));
    const uint32_t by_registers = WARPS == 16 ? 1 : WARPS == 8 ? 2 : 4;  // (at most 105 a thread)
    if (fit > by_registers) fit = by_registers;
    if (fit < 1) fit = 1;
    // CTAs per SM: the count whose equal shares of the 16-row tiles are the most even (896 tiles over 296 CTAs are
    // rounds of 4 and 3: a quarter of the time half the GPU idles; over 148 they are 7 and 6); more CTAs on a tie
    uint32_t grid = 1;
    double best = 0.0;
    for (uint32_t c = 1; c <= fit && c <= 4; c++) {
        uint32_t gr = (uint32_t)sm_count * c;
        if (gr > tasks) gr = tasks;
        const double eff = (double)tasks / ((double)gr * ((tasks + gr - 1) / gr));
        if (eff >= best) best = eff, grid = gr;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    const uint32_t iters = (k + chunk_of(RAGGED) - 1) / chunk_of(RAGGED);
    return cudaLaunchKernelEx(&cfg, kern, g, round, buffers, 65536 / iters + 1);
}
template <bool I4, bool RAGGED, int WARPS, int NG> static cudaError_t launch_w(const GemvGroup &g, int sm_count, bool pdl, cudaStream_t stream) {
    const uint32_t iters = g.item[0].k / chunk_of(RAGGED);
    if constexpr (!RAGGED)
        if (iters % WARPS == 0 && smem_bytes(I4, WARPS, g.item[0].rows, g.item[0].k, 2) <= SMEM_MAX) return launch_e<I4, RAGGED, true, WARPS, NG>(g, sm_count, pdl, stream);
    return launch_e<I4, RAGGED, false, WARPS, NG>(g, sm_count, pdl, stream);
}
template <bool I4, bool RAGGED> static cudaError_t launch_k(const GemvGroup &g, int sm_count, bool pdl, cudaStream_t stream) {
    const uint32_t rows = g.item[0].rows, k = g.item[0].k;
    constexpr int MOST = RAGGED ? 16 : 8;
    if (smem_bytes(I4, MOST, rows, k) <= SMEM_MAX)
        return g.count == 1 ? launch_w<I4, RAGGED, MOST, 1>(g, sm_count, pdl, stream) : launch_w<I4, RAGGED, MOST, GEMV_GROUP_MAX>(g, sm_count, pdl, stream);
    if (RAGGED && smem_bytes(I4, 8, rows, k) <= SMEM_MAX)
        return g.count == 1 ? launch_w<I4, RAGGED, 8, 1>(g, sm_count, pdl, stream) : launch_w<I4, RAGGED, 8, GEMV_GROUP_MAX>(g, sm_count, pdl, stream);
    return g.count == 1 ? launch_w<I4, RAGGED, 4, 1>(g, sm_count, pdl, stream) : launch_w<I4, RAGGED, 4, GEMV_GROUP_MAX>(g, sm_count, pdl, stream);
}

}  // namespace i8m

// Any K (a multiple of 32) whose activation tiles leave room for 70 KB of rings (beyond that the streaming kernels take over).
bool qgemv_i8_mma_shape_ok(int fmt, uint32_t rows, uint32_t k) {
    const bool i4 = fmt == FMT_INT4;
    const size_t rings = 4 * (2 * 16 * (i4 ? 256 : 512) + 2 * 16 * (i8m::ragged(k) ? 48 : 32) + 1024);
    return rows >= 1 && rows <= 8 && k >= GROUP && k % GROUP == 0 && rings + (size_t)((k + QK - 1) / QK) * i8m::act_block_bytes(rows) <= i8m::SMEM_MAX;
}

cudaError_t launch_qgemv_i8_mma(int fmt, const GemvGroup &g, int sm_count, bool pdl, cudaStream_t stream) {
    if (g.count < 1 || !qgemv_i8_mma_shape_ok(fmt, g.item[0].rows, g.item[0].k)) return cudaErrorInvalidValue;
    for (int i = 0; i < g.count; i++) {
        const GemvArgs &a = g.item[i];
        if (a.qa != g.item[0].qa || a.k != g.item[0].k || a.rows != g.item[0].rows || ((uintptr_t)a.w & 15) != 0 || (a.scales_offset & 15) != 0)
            return cudaErrorInvalidValue;
    }
    const bool rag = i8m::ragged(g.item[0].k);
    if (fmt == FMT_INT4) return rag ? i8m::launch_k<true, true>(g, sm_count, pdl, stream) : i8m::launch_k<true, false>(g, sm_count, pdl, stream);
    return rag ? i8m::launch_k<false, true>(g, sm_count, pdl, stream) : i8m::launch_k<false, false>(g, sm_count, pdl, stream);
}

}  // namespace lb

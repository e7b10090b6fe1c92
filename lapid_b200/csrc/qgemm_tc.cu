// Prefill GEMM on the 5th-generation tensor cores: out[m, n] = sum_k A[m, k] * dequant(W)[n, k] for
// Q4_K, Q5_K and Q6_K weights, bf16 operands, f32 accumulation in tensor memory.
//
// Reference semantics: lapid-cpu's path for more than 8 rows multiplies f32 activations by the
// dequantized f32 weights (crates/lapid-cpu/src/matmul/qdeq.rs:57-123); lapid-cuda's tensor-core
// kernel rounds both operands to f16 (crates/lapid-cuda/src/codegen/kquant.rs:335-519). Here both
// operands are rounded to bf16 (weights: bf16 of lapid-quant's f32 value -- Q4_K d1*q - m1 computed
// with one fused multiply-add, Q6_K d*sc*(q-32), exact in f32), products are exact and sums are
// f32, so the result differs from the f32 reference by the operand rounding only (2^-9 relative
// per operand).
//
// The weights are the M side of the instruction, the activations the N side, so a tile has as many columns as the launch
// has rows (in steps of 16) and nothing is padded to 128. What bounds the kernel is the expansion of the packed weights
// (integer instructions, about 1.7 a weight for Q4_K) against the tensor pipe, so:
//   - an expanded weight goes from registers straight into tensor memory (`tcgen05.st`, the A operand of the instruction may
//     lie there): lane = weight row, 64 k = 32 columns. Shared memory then only carries the activations and the packed
//     blocks; as bf16 in shared memory the weights were written and read through the same 128 bytes a cycle that the
//     activations need.
//   - a thread owns one row and 64 of a super-block's 256 k: one look at the header's scales for 64 weights, no partner.
//   - above 128 rows two CTAs of a cluster are one `cta_group::2` unit (where single CTAs do not hold the tiles as well, qgemm_tc_plan()): 256
//     weight rows (each CTA expands its own 128) by up to 256 activation rows, of which each CTA loads half: an expanded weight
//     feeds 256 columns, an activation 256 rows.
//
// Roles of a CTA's 19 warps:
//   warps 0-15 expand: warp (quarter of the rows, j) writes the 64 k at 64 j of every super-block into its half of a stage of tensor
//              memory. They are also the epilogue: the accumulator is given back once its columns are in registers, and
//              the stores run beside the next tile's first products.
//   warp 16    one lane drives TMA for the activations: a 128-byte swizzled copy of the tile's rows for two k-steps of 64 at a time
//   warp 17    allocates tensor memory; one lane issues `tcgen05.mma` (A in tensor memory, B by shared-memory descriptor; four
//              K=16 steps per k-step) and commits to mbarriers
//   warp 18    one lane drives TMA for the weights: per super-block a 2-D tensor-map copy of the 128 rows' packed blocks
//              (144 / 176 bytes; Q6_K: 240 bytes from the 16-byte boundary below the 2-byte aligned 210); Q6_K rows
//              that are not 16-byte multiples come in eight copies of every eighth row
// A CTA (pair) takes every gridDim-th unit of the launch: no CTA start and no first trip to HBM per tile, and the first two
// super-blocks of a tile are expanded before the results of the one before are stored. Tensor memory: 256 columns of accumulators
// (one 256-column set for a pair, two of 128 for a single CTA), 4 stages of 64 columns (two k-steps) of weights.
// Units: whole tiles as long as they fill every CTA, and where the last round would leave SMs idle its tiles are split over K
// (cut() below); the partial tiles of those go to a scratch area and a second kernel sums them in order.
//
// Measured (B200, before: weights through shared memory, one CTA per tile): 77 rows on 14336 x 4096 Q4_K 42.0 -> 25.8 us (1 % more since, the waits at a
// CTA's end; instruction issue: 474 warp instructions for 64 weights of 32 rows); 2048 rows on 28672 x 8192 Q4_K 936 -> 681 us (1400 TFLOP/s, above the sustained rate of
// cuBLAS under the power cap), on 8192 x 28672 Q6_K 1121 -> 800, on 8192 x 3584 Q6_K 172 -> 114. All instantiations sit at the cap of 96
// registers and spill 24 to 80 bytes. Without pairs above 128 rows each CTA would expand every weight for half as many columns.
//
// Programmatic dependent launch: barriers, tensor memory and the packed weights come before `griddepcontrol.wait`; only what
// the kernel in front may have written (activations, expert tables, epilogue terms) and all stores come behind it.
// Every mbarrier wait is bounded: a wait that gives up sets a bit in the host-visible status
// word, the roles fall through to the end, tensor memory is released and the kernel returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include <cstring>

#include "common.cuh"
#include "kernels.h"

namespace lb {

namespace tc {

constexpr int TN = 128;            // weight rows per CTA
constexpr int KS = 64;             // k per k-step: 128 bytes of bf16, the width of a swizzled row
constexpr int STAGE_KS = 2;        // k-steps per stage: half a super-block (one k-step per stage: the waits and commits of the issuing warp took as long as the products)
constexpr int STAGES = 4;          // two super-blocks in flight
constexpr int Q6K_BOX = 240;       // Q6_K: bytes staged per row and super-block (210 from a 2-byte aligned start; an odd number of 16-byte chunks keeps 128-bit row loads free of bank conflicts)
constexpr int DEQ_WARPS = 16;
constexpr int ACT_WARP = DEQ_WARPS, MMA_WARP = DEQ_WARPS + 1, RAW_WARP = DEQ_WARPS + 2;
constexpr int THREADS = 32 * (DEQ_WARPS + 3);
constexpr int A_COL = 256;         // tensor-memory column of the first weight stage
constexpr uint32_t WAIT_NS = 8000, SPIN_LIMIT = 1u << 19;  // a wait gives up after this many attempts of at most this long: 2.1 s measured, at most 4.2

template <int FMT, bool PAIR> struct Cfg {
    static constexpr int MT = PAIR ? 256 : 128;  // most activation rows of a tile
    static constexpr int ACCS = PAIR ? 1 : 2;    // accumulator sets of MT columns
    static constexpr int A_BYTES = STAGE_KS * 128 * 128;  // activations of one stage in this CTA: up to 128 rows of 64 bf16, twice
    static constexpr int ROW_BYTES = FMT == FMT_Q4K ? Q4K_BYTES : FMT == FMT_Q5K ? Q5K_BYTES : Q6K_BOX;  // packed bytes staged per row and super-block
    static constexpr int RAW = (TN + (FMT == FMT_Q6K ? 8 : 0)) * ROW_BYTES;  // (Q6_K: and room for rows copied one by one)
    // Super-blocks of packed weights in flight or in use: as many as the shared memory has room for (5 / 4 / 3)
    static constexpr int RAWS = (227 * 1024 - 512 - 1024 - STAGES * A_BYTES) / RAW;
    static_assert(RAWS >= 3 && 3 * STAGES + 2 * RAWS + 5 <= 64, "shared memory");
    static constexpr int SMEM = STAGES * A_BYTES + RAWS * RAW + 512 /*barriers*/ + 1024 /*alignment slack*/;
};

__device__ __forceinline__ uint32_t s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(bar)) : "memory");
}
// Bounded wait. A failed attempt sleeps in hardware until the phase completes or a time is over that the hardware chooses (4 us measured, also where
// WAIT_NS allows more): waiters that come back at once took as many issue slots as the expansion. The bound covers the kernel in front as
// well, behind whose end the activations come. (Elapsed time read from the clock as the bound: 77 rows 1265 -> 1297 us, 2048 rows 6803 -> 7074.)
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    for (uint32_t spin = 0; spin < SPIN_LIMIT; spin++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(s32(bar)), "r"(parity), "r"(WAIT_NS)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// A producer's last waits: for the copies it has issued into a ring of COUNT slots; (slot, phase) are its next ones, so the slots below were last filled
// in this lap and the others in the lap before (in the first lap: never, and the wait returns at once).
template <int COUNT> __device__ __forceinline__ void wait_for_copies(uint64_t *full, uint32_t slot, uint32_t phase) {
#pragma unroll 1
    for (uint32_t i = 0; i < COUNT; i++) mbar_wait(full + i, i < slot ? phase ^ 1 : phase);
}
// A whole warp waits: all lanes or none give up.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); }

// Two f32 lanes in one 64-bit register pair: Blackwell's packed f32 pipe halves the instruction
// count of the dequantization.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
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
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// {lo, hi} f32 -> packed bf16x2 with lo in the low half
__device__ __forceinline__ uint32_t to_bf16x2(uint64_t v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     s32(dst)),
                 "l"((uint64_t)map), "r"(x), "r"(y), "r"(s32(bar))
                 : "memory");
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                     s32(dst)),
                 "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(s32(bar))
                 : "memory");
}

// K-major operand, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// D[tmem] (+)= A[tmem] * B[smem]: PAIR: the unit of both CTAs, each holding its own 128 rows of A and D and half the rows of B
template <bool PAIR> __device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    if constexpr (PAIR)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
            "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
            "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
            : "memory");
}
// arrival on the barrier (PAIR: on the barrier at the same place of both CTAs) when the products issued so far are done
template <bool PAIR> __device__ __forceinline__ void mma_commit(uint64_t *bar) {
    if constexpr (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(s32(bar)), "h"((uint16_t)3) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(bar)) : "memory");
}
// the shared::cluster address of `p` in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t cluster_addr_of(const void *p, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(s32(p)), "r"(rank));
    return r;
}
// Arrival on a barrier of either CTA. What it reports was complete before (tensor-memory stores that `tcgen05.wait::st` has waited for,
// copies whose barrier has completed), so it carries no cluster-wide release: that one waits for every store of the thread and
// took 1100 to 1500 cycles an arrival. Likewise the waits acquire at CTA scope: at cluster scope each one drops the SM's L1.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// 16 consecutive columns of this warp's 32 lanes of tensor memory (not waited for: tmem_ld_wait)
__device__ __forceinline__ void tmem_ld16(uint32_t *r, uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 16 columns of this warp's 32 lanes (not waited for: tmem_st_wait)
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::"r"(r[0]), "r"(r[1]),
        "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15]), "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// f32 bits of (2^23 + byte `sel` of w): the byte planted in the mantissa by one PRMT
__device__ __forceinline__ float biased(uint32_t w, uint32_t sel) { return __uint_as_float(__byte_perm(w, 0x4B000000u, sel)); }
// 2^23 + (w & mask): a nibble planted where it lies (mask within the 23 bits of the mantissa): 2^p times its value, p = its lowest bit
// (one three-input logic operation: the exponent comes in a register, since of two constants the instruction encodes one)
template <uint32_t MASK> __device__ __forceinline__ float planted(uint32_t w, uint32_t exponent) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "n"(MASK), "r"(exponent));
    return __uint_as_float(r);
}
__device__ __forceinline__ uint32_t planted_exponent() {
    uint32_t r;
    asm volatile("mov.b32 %0, 0x4B000000;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint64_t unbias2(float a, float b) { return add2(pack2(a, b), pack2(-8388608.0f, -8388608.0f)); }
__device__ __forceinline__ uint32_t rot(uint32_t v, uint32_t by) { return __funnelshift_l(v, v, by); }

// ---- expansion of one thread's share of a super-block: row = its lane, k = 64 j .. 64 j + 63, in two halves of 32 weights (16 registers of
// two bf16 each, k ascending). The words it needs are loaded a super-block ahead.
//
// Q4_K / Q5_K (crates/lapid-quant/src/kquant.rs:337-373): byte l of the 32 bytes at 32 j holds element 64 j + l in its low and 64 j + 32 + l
// in its high nibble; scales and mins of sub-blocks 2 j and 2 j + 1. Q5_K: bit s of qh[l] belongs to element 32 s + l.
// Q6_K (:375-396): ql[128] | qh[64] | int8 sc[16] | f16 d. k-step j: half nh = j >> 1 of the 256, nibble hi = j & 1; the first 32 weights from
// ql[64 nh + l], the second 32 from ql[64 nh + 32 + l]; the two high bits from qh[32 nh + l] >> 2 (2 hi + h); scale
// sc[8 nh + 2 (2 hi + h) + l / 16].
template <int FMT> struct Packed {
    uint4 h;
    uint32_t w[8], x[FMT == FMT_Q5K ? 8 : 1];
};
template <> struct Packed<FMT_Q6K> {
    uint32_t wl[8], wh[8], sc, d;  // (wl: of one half at a time)
};
template <int FMT> __device__ __forceinline__ void load_packed(Packed<FMT> &r, const uint8_t *blk, uint32_t j) {
    constexpr int QS = FMT == FMT_Q5K ? 48 : 16;
    r.h = *(const uint4 *)blk;
    *(uint4 *)r.w = *(const uint4 *)(blk + QS + 32 * j);
    *(uint4 *)(r.w + 4) = *(const uint4 *)(blk + QS + 16 + 32 * j);
    if constexpr (FMT == FMT_Q5K) {
        *(uint4 *)r.x = *(const uint4 *)(blk + 16);
        *(uint4 *)(r.x + 4) = *(const uint4 *)(blk + 32);
    }
}
// Eight words at byte `at` (a multiple of 16) of a Q6_K block, from 128-bit chunks of its staged row; the block starts 4 WS (+ 2: sh = 16) bytes behind
// a chunk boundary
template <int WS> __device__ __forceinline__ void q6k_words(const uint8_t *row, uint32_t at, uint32_t sh, uint32_t (&w)[8]) {
    uint32_t t[12];
#pragma unroll
    for (int c = 0; c < 3; c++) *(uint4 *)(t + 4 * c) = *(const uint4 *)(row + at + 16 * c);
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = __funnelshift_r(t[i + WS], t[i + WS + 1], sh);
}
// `skew`: where the block starts in its staged row; `uniform`: the same for every row of the matrix
__device__ __forceinline__ void q6k_run(const uint8_t *row, uint32_t skew, bool uniform, uint32_t at, uint32_t (&w)[8]) {
    const uint32_t sh = 8 * (skew & 2);
    if (uniform) {
        switch (skew >> 2) {
            case 0: q6k_words<0>(row, at, sh, w); break;
            case 1: q6k_words<1>(row, at, sh, w); break;
            case 2: q6k_words<2>(row, at, sh, w); break;
            default: q6k_words<3>(row, at, sh, w); break;
        }
    } else {
        const uint32_t *a = (const uint32_t *)(row + (skew & ~3u) + at);
        uint32_t prev = a[0];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t next = a[i + 1];
            w[i] = __funnelshift_r(prev, next, sh);
            prev = next;
        }
    }
}
template <int H> __device__ __forceinline__ void load_packed_q6(Packed<FMT_Q6K> &r, const uint8_t *row, uint32_t skew, bool uniform, uint32_t j) {
    const uint32_t nh = j >> 1, hi = j & 1;
    q6k_run(row, skew, uniform, 64 * nh + 32 * H, r.wl);
    if (H == 0) {
        q6k_run(row, skew, uniform, 128 + 32 * nh, r.wh);
        const uint16_t *scp = (const uint16_t *)(row + skew + 192 + 8 * nh + 4 * hi);
        r.sc = (uint32_t)scp[0] | ((uint32_t)scp[1] << 16);
        r.d = *(const uint16_t *)(row + skew + 208);
    }
}
// d * byte `sel` of w, exactly: d (2^23 + b) - d 2^23 has one rounding, and d b (11 x 8 bits) needs none
__device__ __forceinline__ float scaled(float d, uint32_t w, uint32_t sel, float neg_d23) { return fmaf(d, biased(w, sel), neg_d23); }
// half H (0: the first 32 weights) of the share
template <int FMT, int H> __device__ __forceinline__ void expand(const Packed<FMT> &r, uint32_t j, uint32_t e23, uint32_t (&o)[16]) {
    if constexpr (FMT == FMT_Q6K) {
        const float d = half_bits_to_float(r.d);
        const uint32_t hi = j & 1, up = (4 - 4 * hi - 2 * H) & 31;  // rotation that brings the two high bits of every byte to bits 4 and 5
        const uint32_t sb = r.sc ^ 0x80808080u;                      // scales + 128
        // d * sc (11 x 8 bits) and d * sc * (q - 32) are exact in f32; d = inf stays inf (removed behind the product, the bias would make it NaN)
        const float sd[2] = {d * (biased(sb, 0x7440u + 2 * H) - 8388736.0f), d * (biased(sb, 0x7441u + 2 * H) - 8388736.0f)};  // 2^23 + 128
        const uint64_t unbias32 = pack2(-8388640.0f, -8388640.0f);   // -(2^23 + 32)
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t q = ((r.wl[i] >> (4 * hi)) & 0x0F0F0F0Fu) | (rot(r.wh[i], up) & 0x30303030u);
            const uint64_t s2 = pack2(sd[i >> 2], sd[i >> 2]);
            o[2 * i] = to_bf16x2(mul2(s2, add2(pack2(biased(q, 0x7440u), biased(q, 0x7441u)), unbias32)));
            o[2 * i + 1] = to_bf16x2(mul2(s2, add2(pack2(biased(q, 0x7442u), biased(q, 0x7443u)), unbias32)));
        }
    } else {
        // the two 6-bit scales in bytes 0 and 1 of sc, the mins in mn (scale_min_pair's layout)
        const uint32_t sh = 16 * (j & 1);
        const uint32_t w0 = r.h.y >> sh, w1 = r.h.z >> sh, w2 = r.h.w >> sh;
        const uint32_t sc = j < 2 ? w0 & 0x3F3Fu : (w2 & 0x0F0Fu) | ((w0 >> 2) & 0x3030u);
        const uint32_t mn = j < 2 ? w1 & 0x3F3Fu : ((w2 >> 4) & 0x0F0Fu) | ((w1 >> 2) & 0x3030u);
        const float d = half_bits_to_float(r.h.x & 0xffff), dmin = half_bits_to_float(r.h.x >> 16);
        const float s = scaled(d, sc, 0x7440u + H, d * -8388608.0f), m = -scaled(dmin, mn, 0x7440u + H, dmin * -8388608.0f);
        const uint64_t nm = pack2(m, m);
        if constexpr (FMT == FMT_Q4K) {
            // Each nibble is planted where it lies, which costs one logic operation a weight and one shift for four; its power of two
            // goes into the multiplier, so y = sc q - m still has one rounding and the bits of the plain form.
            constexpr float P4 = 0x1p-4f, P8 = 0x1p-8f, P12 = 0x1p-12f, P16 = 0x1p-16f;
            const uint64_t s01 = H ? pack2(s * P4, s * P12) : pack2(s, s * P8), s23 = H ? pack2(s * P8, s * P16) : pack2(s * P16, s * P12);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t v = r.w[i] >> 12;  // byte 2's high nibble at bit 8, byte 3's at 12 and 16
                o[2 * i] = to_bf16x2(fma2(s01, unbias2(planted<H ? 0xF0u : 0xFu>(r.w[i], e23), planted<H ? 0xF000u : 0xF00u>(r.w[i], e23)), nm));
                o[2 * i + 1] = to_bf16x2(fma2(s23, unbias2(planted<H ? 0xF00u : 0xF0000u>(H ? v : r.w[i], e23), planted<H ? 0xF0000u : 0xF000u>(v, e23)), nm));
            }
        } else {
            const uint64_t s2 = pack2(s, s);
            const uint32_t up = (4 - 2 * j - H) & 31;  // rotation that brings bit 2 j + H of every byte to bit 4
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t a = ((H ? r.w[i] >> 4 : r.w[i]) & 0x0F0F0F0Fu) | (rot(r.x[i], up) & 0x10101010u);
                o[2 * i] = to_bf16x2(fma2(s2, unbias2(biased(a, 0x7440u), biased(a, 0x7441u)), nm));
                o[2 * i + 1] = to_bf16x2(fma2(s2, unbias2(biased(a, 0x7442u), biased(a, 0x7443u)), nm));
            }
        }
    }
}

// One unit of work: a tile of 128 (PAIR: 256) weight rows x mt activation rows and the super-blocks [kb0, kb0 + nblk) of K.
struct Tile {
    uint32_t n0, m0, wrow0, kb0, nblk;
    int32_t part;  // -1: the tile's results; else which partial tile
};

template <int FMT, bool PAIR>
__global__ void __launch_bounds__(THREADS, 1)
qgemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, GemmTcArgs p) {
    using C = Cfg<FMT, PAIR>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((0u - s32(smem_raw)) & 1023u);  // (an offset, not a cast: the loads below stay shared-memory loads)
    uint8_t *stage0 = smem;
    uint8_t *raw0 = smem + STAGES * C::A_BYTES;
    uint64_t *bars = (uint64_t *)(raw0 + C::RAWS * C::RAW);
    uint64_t *full_a = bars, *full_w = bars + STAGES, *empty = bars + 2 * STAGES;  // activations, weights in place; stage read by the tensor cores
    uint64_t *raw_full = bars + 3 * STAGES, *raw_empty = raw_full + C::RAWS;
    uint64_t *acc_full = raw_empty + C::RAWS, *acc_empty = acc_full + 2;
    uint32_t *tmem_slot = (uint32_t *)(acc_empty + 2);
    uint32_t rank = 0;
    if constexpr (PAIR) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Units [0, full) are whole tiles, those behind are `splits` to a tile. Within `group` activation tiles the tile order
    // walks the activation tiles first, so that the CTAs that run side by side share packed weights in L2.
    const uint32_t nx = p.tiles_x, ny = p.tiles_y, units = p.units, step = PAIR ? gridDim.x >> 1 : gridDim.x, first = PAIR ? blockIdx.x >> 1 : blockIdx.x;
    const uint32_t nblk_total = p.k / QK;
    auto tile_at = [&](uint32_t u, Tile &o) -> bool {
        uint32_t t = u, z = 0;
        o.part = -1;
        o.kb0 = 0, o.nblk = nblk_total;
        if (u >= p.full) {
            const uint32_t v = u - p.full, per = (nblk_total + p.splits - 1) / p.splits;
            t = v / p.splits, z = v - t * p.splits;
            o.part = (int32_t)v;
            t += p.full;
            o.kb0 = z * per;
            o.nblk = min(per, nblk_total - o.kb0);
        }
        const uint32_t g = t / (nx * p.group), r = t - g * nx * p.group, gy = min(p.group, ny - g * p.group);
        const uint32_t x = r / gy, y = g * p.group + (r - x * gy);
        o.wrow0 = 0;
        if (p.tile_expert) {
            // Expert-indexed launch (Kernel::MatMulId, moe.cu): the activation tiles are runs of (token, slot)
            // pairs grouped by expert; the weights are the dense stack [experts * n, k], so a tile's weight
            // rows start at expert * n; tiles past the last used one have no expert.
            const int32_t e = p.tile_expert[y];
            if (e < 0) return false;
            o.wrow0 = (uint32_t)e * p.n;
        }
        o.n0 = x * (PAIR ? 2 * TN : TN) + rank * TN;
        o.m0 = y * p.mt;
        return true;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(full_a + s, 1);
            mbar_init(full_w + s, PAIR ? 17 : 8);  // the eight warps of a stage; PAIR: of both CTAs, and the other CTA's activations
            mbar_init(empty + s, 1);
        }
        for (int r = 0; r < C::RAWS; r++) {
            mbar_init(raw_full + r, 1);
            mbar_init(raw_empty + r, DEQ_WARPS);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(acc_full + a, 1);
            mbar_init(acc_empty + a, PAIR ? 2 * DEQ_WARPS : DEQ_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        if constexpr (PAIR) {  // the same warp of both CTAs: a pair-wide allocation of the same columns
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (PAIR) cluster_sync_all();  // both CTAs' barriers exist before either one signals the other
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    bool healthy = true;
    if (p.tile_expert || !p.w_early) grid_dep_wait();  // every role looks the tiles' experts up; weights the kernel in front may write

    if (warp == ACT_WARP) {
        // ---------------- TMA producer, activations: two k-steps of 128-byte-swizzled rows per copy (PAIR: this CTA's half of the rows)
        if (lane == 0) {
            grid_dep_wait();
            grid_dep_launch();
            const uint32_t rows = PAIR ? p.mt / 2 : p.mt;
            uint32_t s = 0, ph = 1;
            Tile o;
            for (uint32_t u = first; u < units && healthy; u += step) {
                if (!tile_at(u, o)) continue;
                for (uint32_t h = 0; h < 2 * o.nblk; h++) {  // halves of super-blocks
                    if (!mbar_wait(empty + s, ph)) { healthy = false; break; }
                    mbar_expect_tx(full_a + s, rows * 128 * STAGE_KS);
                    tma_load_3d(stage0 + s * C::A_BYTES, &map_a, 0, (int)(o.m0 + rows * rank), (int)(o.kb0 * (QK / KS) + h * STAGE_KS), full_a + s);
                    if (++s == STAGES) s = 0, ph ^= 1;
                }
            }
            // Nothing may arrive in this CTA's shared memory or use its tensor memory once it leaves: the products have read every stage that was
            // filled (a pair's second CTA hears that from the first), and when a role gave up, the copies into the others are done.
            const uint32_t s_next = s, ph_next = ph;
            for (int i = 0; i < STAGES && healthy; i++) {
                healthy = mbar_wait(empty + s, ph);
                if (++s == STAGES) s = 0, ph ^= 1;
            }
            if (!healthy) {
                wait_for_copies<STAGES>(full_a, s_next, ph_next);
                if (p.status) atomicOr(p.status, 2);
            }
        }
    } else if (warp == RAW_WARP && FMT == FMT_Q6K && ((nblk_total * Q6K_BYTES) & 15u) != 0) {
        // ---------------- TMA producer, packed Q6_K weights whose rows are not a multiple of 16 bytes (K not a multiple of 2048, e.g. the K/8 shard of a
        // row-parallel projection). Eight rows are: a row of the tensor map is a group of eight, and copy number g brings row g of the
        // tile's 16 groups, from the 16-byte boundary below its block (the consumers compute the same offset), to the 16 places from 16 g on.
        // Rows behind the last whole group are copied one by one, to the places behind the tile's.
        // What bounds it is the number of copies: with one of each row (128 in place of 8) a super-block took 6 us, 2048 rows on 8192 x 3584 275 us (now
        // 118), 77 rows 45 (21).
        if (lane == 0) {
            const uint64_t pitch = (uint64_t)nblk_total * Q6K_BYTES;
            const uint64_t end16 = ((uint64_t)(uintptr_t)p.w + (uint64_t)p.n * pitch + 15) & ~(uint64_t)15;  // never read past the matrix's last 16-byte line
            const uint32_t grouped = p.n & ~7u;
            uint32_t r = 0, ph = 1;
            Tile o;
            for (uint32_t u = first; u < units && healthy; u += step) {
                if (!tile_at(u, o)) continue;
                const uint32_t single = grouped >= o.n0 && grouped < o.n0 + TN ? p.n - grouped : 0;
                auto copy_of = [&](uint32_t i, uint32_t b, uint64_t &src) -> uint32_t {
                    src = ((uint64_t)(uintptr_t)p.w + (uint64_t)(grouped + i) * pitch + (uint64_t)(o.kb0 + b) * Q6K_BYTES) & ~(uint64_t)15;
                    return (uint32_t)min((uint64_t)224, end16 - src);
                };
                for (uint32_t b = 0; b < o.nblk; b++) {
                    if (!mbar_wait(raw_empty + r, ph)) { healthy = false; break; }
                    uint8_t *dst = raw0 + r * C::RAW;
                    uint64_t src;
                    uint32_t bytes = grouped ? TN * Q6K_BOX : 0;
                    for (uint32_t i = 0; i < single; i++) bytes += copy_of(i, b, src);
                    if (bytes) mbar_expect_tx(raw_full + r, bytes);
                    else mbar_arrive(raw_full + r);  // (fewer than eight rows: the second CTA of a pair has none)
                    if (grouped)
                        for (uint32_t g = 0; g < 8; g++)
                            tma_load_2d(dst + g * (TN / 8) * Q6K_BOX, &map_w, (int)((g * pitch + (uint64_t)(o.kb0 + b) * Q6K_BYTES) & ~(uint64_t)15), (int)(o.n0 / 8), raw_full + r);
                    for (uint32_t i = 0; i < single; i++) {
                        const uint32_t n = copy_of(i, b, src);
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(s32(dst + (TN + i) * Q6K_BOX)),
                                     "l"(src), "r"(n), "r"(s32(raw_full + r))
                                     : "memory");
                    }
                    if (++r == C::RAWS) r = 0, ph ^= 1;
                }
            }
            wait_for_copies<C::RAWS>(raw_full, r, ph);  // (done already unless the expanding warps gave up)
            if (!healthy && p.status) atomicOr(p.status, 32);
        }
    } else if (warp == RAW_WARP) {
        // ---------------- TMA producer, packed weights: one super-block of every row of the tile
        // per copy, up to RAWS super-blocks (of four k-steps) ahead of the expanding warps
        if (lane == 0) {
            uint32_t r = 0, ph = 1;
            Tile o;
            for (uint32_t u = first; u < units && healthy; u += step) {
                if (!tile_at(u, o)) continue;
                for (uint32_t b = 0; b < o.nblk; b++) {
                    if (!mbar_wait(raw_empty + r, ph)) { healthy = false; break; }
                    mbar_expect_tx(raw_full + r, TN * C::ROW_BYTES);
                    tma_load_2d(raw0 + r * C::RAW, &map_w, FMT == FMT_Q6K ? (int)(((o.kb0 + b) * Q6K_BYTES) & ~15u) : (int)((o.kb0 + b) * C::ROW_BYTES),
                                (int)(o.wrow0 + o.n0), raw_full + r);
                    if (++r == C::RAWS) r = 0, ph ^= 1;
                }
            }
            wait_for_copies<C::RAWS>(raw_full, r, ph);  // (done already unless the expanding warps gave up)
            if (!healthy && p.status) atomicOr(p.status, 32);
        }
    } else if (warp == MMA_WARP && PAIR && rank == 1) {
        // ---------------- the pair's second CTA: its activations of a stage are in place
        if (lane == 0) {
            const uint32_t to = cluster_addr_of(full_w, 0);
            uint32_t s = 0, ph = 0;
            Tile o;
            for (uint32_t u = first; u < units && healthy; u += step) {
                if (!tile_at(u, o)) continue;
                for (uint32_t h = 0; h < 2 * o.nblk; h++) {
                    if (!mbar_wait(full_a + s, ph)) { healthy = false; break; }
                    mbar_arrive_cluster(to + 8 * s);
                    if (++s == STAGES) s = 0, ph ^= 1;
                }
            }
            if (!healthy && p.status) atomicOr(p.status, 4);
        }
    } else if (warp == MMA_WARP) {
        // ---------------- MMA issuer (PAIR: the first CTA's, for both). The whole warp walks the loop and one elected lane issues, so that the
        // operands stay in uniform registers (issued by one lane of a diverged warp: 80 cycles a product instead of 28).
        // D f32, A and B bf16, both K-major, M = 128 (PAIR: 256), N = mt
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((p.mt >> 3) << 17) | ((uint32_t)((PAIR ? 2 * TN : TN) >> 4) << 24);
        const uint32_t half_rows = (PAIR ? p.mt / 2 : p.mt) * 8;  // rows * 128 bytes between a stage's two k-steps, in the descriptor's units of 16
        uint32_t s = 0, ph = 0, ti = 0;  // stage, its phase, tiles so far
        Tile o;
        for (uint32_t u = first; u < units && healthy; u += step) {
            if (!tile_at(u, o)) continue;
            const uint32_t acc = ti % C::ACCS, tmem_d = tmem_base + acc * C::MT, halves = 2 * o.nblk;
            if (!warp_wait(acc_empty + acc, ((ti / C::ACCS) & 1) ^ 1)) { healthy = false; break; }  // its last results have been read
            ti++;
            for (uint32_t h = 0; h < halves; h++) {
                if (!__all_sync(0xffffffffu, mbar_wait(full_a + s, ph) && mbar_wait(full_w + s, ph))) { healthy = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t wt = tmem_base + A_COL + s * (STAGE_KS * KS / 2);
                const uint64_t at = smem_desc(s32(stage0) + s * C::A_BYTES);
                if (elect_one()) {
#pragma unroll
                    for (int q = 0; q < STAGE_KS; q++)
#pragma unroll
                        for (int kk = 0; kk < KS / 16; kk++)
                            mma_bf16<PAIR>(tmem_d, wt + q * (KS / 2) + 8 * kk, at + q * half_rows + 2 * kk, idesc, (h | q | kk) ? 1u : 0u);
                    mma_commit<PAIR>(empty + s);  // the stage may be refilled once these have read it
                    if (h + 1 == halves) mma_commit<PAIR>(acc_full + acc);
                }
                __syncwarp();
                if (++s == STAGES) s = 0, ph ^= 1;
            }
        }
        if (!healthy && lane == 0 && p.status) atomicOr(p.status, 4);
    } else {
        // ---------------- expand and store
        const uint32_t quarter = warp & 3, j = (uint32_t)warp >> 2;  // the tensor-memory lanes this warp may touch; which 64 k of a super-block
        const uint32_t row = 32 * quarter + lane;
        const uint32_t lanes = (32 * quarter) << 16;
        const uint32_t e23 = planted_exponent();
        uint32_t sb = 0, ti = 0;         // super-blocks and tiles so far
        uint32_t r = 0, rph = 0;         // ring slot and phase

        // ---------------- epilogue: tensor-memory lane = weight row, column = activation row
        auto store_tile = [&](uint32_t unit, uint32_t index) {
            constexpr int ROUNDS = C::MT / 128;  // rounds of two chunks of 16 columns: this warp has every fourth chunk
            const uint32_t acc = index % C::ACCS;
            if (!warp_wait(acc_full + acc, (index / C::ACCS) & 1)) {
                if (lane == 0 && p.status) atomicOr(p.status, 16);
                healthy = false;
                return;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            grid_dep_wait();  // (returns at once after the first time)
            Tile t;
            tile_at(unit, t);
            const uint32_t n = t.n0 + row;
#pragma unroll 1
            for (int round = 0; round < ROUNDS; round++) {
                uint32_t v[32];
#pragma unroll
                for (int i = 0; i < 2; i++)
                    if (16 * (j + 4 * (2 * round + i)) < p.mt) tmem_ld16(v + 16 * i, tmem_base + acc * C::MT + lanes + 16 * (j + 4 * (2 * round + i)));
                tmem_ld_wait();
                if (round == ROUNDS - 1) {  // the accumulator may be overwritten
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        if constexpr (PAIR) mbar_arrive_cluster(cluster_addr_of(acc_empty + acc, 0));
                        else mbar_arrive(acc_empty + acc);
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const uint32_t col = 16 * (j + 4 * (2 * round + i)), mfirst = t.m0 + col;
                    if (col >= p.mt) break;
                    if (t.part >= 0) {  // partial sums, [unit][activation row][weight row]; summed by a second kernel
                        constexpr uint32_t W = PAIR ? 2 * TN : TN;
                        float *prow = p.partial + ((size_t)t.part * p.mt + col) * W + rank * TN + row;
#pragma unroll
                        for (int c = 0; c < 16; c++) prow[(size_t)c * W] = __uint_as_float(v[16 * i + c]);
                    } else if (p.row_pair) {  // expert-indexed: tile-space row -> (token, slot) pair = output row; padding rows have none
                        if (n < p.n) {
#pragma unroll
                            for (int c = 0; c < 16; c++) {
                                const int32_t pair = p.row_pair[mfirst + c];
                                if (pair >= 0) p.out[p.out_off + (uint64_t)pair * p.n + n] = __uint_as_float(v[16 * i + c]);
                            }
                        }
                    } else if (n < p.n && mfirst < p.rows) {
                        // (batch, row) of the chunk's first activation row by one division, then by stepping
                        uint32_t bt = mfirst / p.m, ir = mfirst % p.m;
                        float *orow = p.out + p.out_off + (uint64_t)bt * p.out_bs + (uint64_t)ir * p.out_rs + n;
                        const float *erow = p.extra ? p.extra + p.ex_off + (int64_t)bt * p.ex_s0 + (int64_t)ir * p.ex_s1 + (int64_t)n * p.ex_s2 : nullptr;
                        const uint32_t cnt = min(16u, p.rows - mfirst);
                        if (!erow && ir + cnt <= p.m) {  // the common case: rows of one batch entry, no epilogue term
#pragma unroll
                            for (uint32_t c = 0; c < 16; c++)
                                if (c < cnt) orow[(uint64_t)c * p.out_rs] = __uint_as_float(v[16 * i + c]);
                        } else {
#pragma unroll
                            for (int c = 0; c < 16; c++) {
                                if (mfirst + c < p.rows) {
                                    float x = __uint_as_float(v[16 * i + c]);
                                    if (erow) x += *erow;
                                    *orow = x;
                                }
                                if (++ir == p.m) {  // next batch entry
                                    ir = 0;
                                    bt++;
                                    orow = p.out + p.out_off + (uint64_t)bt * p.out_bs + n;
                                    if (erow) erow = p.extra + p.ex_off + (int64_t)bt * p.ex_s0 + (int64_t)n * p.ex_s2;
                                } else {
                                    orow += p.out_rs;
                                    if (erow) erow += p.ex_s1;
                                }
                            }
                        }
                    }
                }
            }
        };
        // The packed words of the next super-block are loaded before this one's are expanded. A ring slot goes back behind the tensor-memory
        // stores of what was expanded from it: not behind the loads, which may be carried out late (hundreds of cycles behind an
        // arrival while the load / store unit is busy) and would then read the first rows of the block that follows.
        const uint32_t to_mma = PAIR ? cluster_addr_of(full_w, 0) : 0;
        Tile o;
        auto valid = [&](uint32_t u) -> uint32_t {  // the first unit from u on that has work
            while (u < units && !tile_at(u, o)) u += step;
            return u;
        };
        // Q6_K: where a block starts inside its staged bytes: the distance of its address from the 16-byte boundary below it
        const uint32_t pitch = nblk_total * Q6K_BYTES;
        const bool uniform = (pitch & 15u) == 0;
        auto skew_of = [&](uint32_t kb, uint32_t first_row) { return (kb * Q6K_BYTES + (first_row + row) * pitch) & 15u; };  // (p.w is 16-byte aligned; only the low bits matter)
        uint32_t place = row;  // which staged row is this thread's (of the current tile; see the producer)
        auto load = [&](Packed<FMT> &w, uint32_t kb, uint32_t first_row) {  // (the place of the block matters for Q6_K only)
            if (!warp_wait(raw_full + r, rph)) {
                healthy = false;
                return;
            }
            const uint8_t *blk = raw0 + r * C::RAW + place * C::ROW_BYTES;
            if constexpr (FMT == FMT_Q6K) load_packed_q6<0>(w, blk, skew_of(kb, first_row), uniform, j);
            else load_packed<FMT>(w, blk, j);
        };
        constexpr bool AHEAD = FMT == FMT_Q4K;    // (Q5_K, Q6_K: too many words a share to hold twice)
        uint32_t u = valid(first), done = 0;      // the current unit; the one whose results are to be stored
        uint32_t kb0 = 0, n0 = 0, nblk = 0;
        auto enter = [&]() {
            nblk = u < units ? o.nblk : 0, kb0 = o.kb0, n0 = o.n0;
            if (FMT == FMT_Q6K && !uniform) place = n0 + row < (p.n & ~7u) ? (row & 7) * (TN / 8) + (row >> 3) : TN + (row & 7);
        };
        enter();
        Packed<FMT> cur;
        if (AHEAD && nblk) load(cur, 0, 0);
        while (healthy) {
            // Results of the tile before are stored behind the super-blocks that fit the stages: one more would wait for products
            // that wait for the accumulator.
            const uint32_t store_behind = min(nblk, (uint32_t)(STAGES / 2));
            uint32_t un = u;
            for (uint32_t b = 0;; b++) {
                if (b == store_behind && ti > 0) store_tile(done, ti - 1);
                if (b == nblk || !healthy) break;
                if constexpr (!AHEAD) load(cur, kb0 + b, n0);
                const uint32_t slot = r;
                if (++r == C::RAWS) r = 0, rph ^= 1;
                Packed<FMT> next;
                if (b + 1 == nblk) un = valid(u + step);
                if constexpr (AHEAD)
                    if (un < units) load(next, 0, 0);
                const uint32_t s = 2 * (sb & 1) + (j >> 1), col = tmem_base + A_COL + lanes + s * (STAGE_KS * KS / 2) + (j & 1) * (KS / 2);
                uint32_t w[16];
                expand<FMT, 0>(cur, j, e23, w);
                if (!healthy || !warp_wait(empty + s, ((sb >> 1) & 1) ^ 1)) { healthy = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                tmem_st16(col, w);
                if constexpr (FMT == FMT_Q6K) load_packed_q6<1>(cur, raw0 + slot * C::RAW + place * C::ROW_BYTES, skew_of(kb0 + b, n0), uniform, j);
                expand<FMT, 1>(cur, j, e23, w);
                tmem_st16(col + 16, w);
                tmem_st_wait();
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if constexpr (PAIR) mbar_arrive_cluster(to_mma + 8 * s);
                    else mbar_arrive(full_w + s);
                    mbar_arrive(raw_empty + slot);
                }
                sb++;
                if constexpr (AHEAD) cur = next;
            }
            if (nblk == 0) break;
            ti++;
            done = u;
            u = un;
            enter();
        }
        if (!healthy && lane == 0 && p.status) atomicOr(p.status, 8);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (PAIR) cluster_sync_all();  // neither CTA releases the pair's tensor memory (or exits) while the other still uses it
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if constexpr (PAIR)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// Second pass of the tiles split over K: out[m, n] = sum over the splits (in order) of their partial tiles (+ extra). A thread takes
// four consecutive weight rows of one activation row.
template <int W> __global__ void __launch_bounds__(256) splitk_sum_kernel(GemmTcArgs p) {
    grid_dep_wait();
    grid_dep_launch();
    const uint32_t tiles = (p.units - p.full) / p.splits, per_tile = p.mt * (W / 4);
    const size_t part = (size_t)p.mt * W;
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < (uint64_t)tiles * per_tile; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t ts = (uint32_t)(e / per_tile), q = (uint32_t)(e - (uint64_t)ts * per_tile), col = q / (W / 4), w4 = q % (W / 4);
        const uint32_t t = p.full + ts, g = t / (p.tiles_x * p.group), rr = t - g * p.tiles_x * p.group, gy = min(p.group, p.tiles_y - g * p.group);
        const uint32_t x = rr / gy, y = g * p.group + (rr - x * gy);
        const uint32_t m = y * p.mt + col, n = x * W + 4 * w4;
        if (m >= p.rows || n >= p.n) continue;
        const float4 *src = (const float4 *)(p.partial + ts * (size_t)p.splits * part + (size_t)col * W) + w4;
        float4 v = *src;
        for (uint32_t z = 1; z < p.splits; z++) {
            const float4 a = src[z * (part / 4)];
            v.x += a.x, v.y += a.y, v.z += a.z, v.w += a.w;
        }
        const uint32_t bt = m / p.m, i = m % p.m;
        float r[4] = {v.x, v.y, v.z, v.w};
        float *out = p.out + p.out_off + (uint64_t)bt * p.out_bs + (uint64_t)i * p.out_rs + n;
        if (p.extra) {
            const float *ex = p.extra + p.ex_off + (int64_t)bt * p.ex_s0 + (int64_t)i * p.ex_s1;
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (n + c < p.n) r[c] += ex[(int64_t)(n + c) * p.ex_s2];
        }
        if (n + 4 <= p.n && ((uintptr_t)out & 15) == 0) {
            *(float4 *)out = make_float4(r[0], r[1], r[2], r[3]);
        } else {
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (n + c < p.n) out[c] = r[c];
        }
    }
}

// Activation rows (any row stride) -> bf16 [k / 64][rows][64]: what a k-step of the GEMM loads is one contiguous piece instead of a line from
// every row. blockIdx.y = row (one division per thread, not per element), a thread converts eight consecutive elements (k is a multiple of 256);
// VEC: the rows are 16-byte aligned, so the loads are 128-bit.
template <bool VEC> __global__ void __launch_bounds__(256) a_to_bf16_kernel(GemmTcArgs p, __nv_bfloat16 *dst) {
    grid_dep_wait();
    grid_dep_launch();
    for (uint32_t r = blockIdx.y; r < p.rows; r += gridDim.y) {
        const void *srow = act_row(p.a, p.a_type, p.a_off, p.a_bs, p.a_rs, r, p.m);
        const float *src = (const float *)srow;  // (VEC: f32 rows only)
        for (uint32_t c8 = blockIdx.x * blockDim.x + threadIdx.x; c8 < p.k / 8; c8 += gridDim.x * blockDim.x) {
            float v[8];
            if constexpr (VEC) {
                const float4 lo = ((const float4 *)src)[2 * c8], hi = ((const float4 *)src)[2 * c8 + 1];
                v[0] = lo.x, v[1] = lo.y, v[2] = lo.z, v[3] = lo.w, v[4] = hi.x, v[5] = hi.y, v[6] = hi.z, v[7] = hi.w;
            } else {
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = load_act(srow, 8 * c8 + i, p.a_type);
            }
            __nv_bfloat162 o[4];
#pragma unroll
            for (int i = 0; i < 4; i++) o[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            ((uint4 *)dst)[((size_t)(c8 / 8) * p.rows + r) * 8 + c8 % 8] = *(const uint4 *)o;
        }
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)ptr;
    }
    return fn;
}

// A launch with (optionally) the programmatic-dependent and the pair attribute.
struct LaunchCfg {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    LaunchCfg(dim3 grid, unsigned threads, size_t smem, bool pdl, bool pair, cudaStream_t stream) {
        cfg.gridDim = grid;
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = attr;
        if (pdl) {
            attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
        }
        if (pair) {
            attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
            attr[cfg.numAttrs].val.clusterDim.x = 2;
            attr[cfg.numAttrs].val.clusterDim.y = 1;
            attr[cfg.numAttrs++].val.clusterDim.z = 1;
        }
    }
};

using Plan = GemmTcPlan;

template <int FMT, bool PAIR>
static cudaError_t launch_tiles(const GemmTcArgs &a, const Plan &pl, const CUtensorMap &mw, const CUtensorMap &ma, int sm_count, bool pdl, cudaStream_t stream) {
    auto kern = qgemm_tc_kernel<FMT, PAIR>;
    using C = Cfg<FMT, PAIR>;
    static DynamicSmemOptIn opted;
    if (cudaError_t e = opted.raise((const void *)kern, C::SMEM); e != cudaSuccess) return e;
    const uint32_t workers = PAIR ? (uint32_t)sm_count / 2 : (uint32_t)sm_count;
    const uint32_t n = pl.units < workers ? pl.units : workers;
    LaunchCfg l(dim3(PAIR ? 2 * n : n), THREADS, C::SMEM, pdl, PAIR, stream);
    return cudaLaunchKernelEx(&l.cfg, kern, mw, ma, a);
}
static cudaError_t launch_plan(int fmt, const GemmTcArgs &a, const Plan &pl, const CUtensorMap &mw, const CUtensorMap &ma, int sm_count, bool pdl, cudaStream_t stream) {
    if (pl.pair)
        return fmt == FMT_Q4K ? launch_tiles<FMT_Q4K, true>(a, pl, mw, ma, sm_count, pdl, stream)
             : fmt == FMT_Q5K ? launch_tiles<FMT_Q5K, true>(a, pl, mw, ma, sm_count, pdl, stream) : launch_tiles<FMT_Q6K, true>(a, pl, mw, ma, sm_count, pdl, stream);
    return fmt == FMT_Q4K ? launch_tiles<FMT_Q4K, false>(a, pl, mw, ma, sm_count, pdl, stream)
         : fmt == FMT_Q5K ? launch_tiles<FMT_Q5K, false>(a, pl, mw, ma, sm_count, pdl, stream) : launch_tiles<FMT_Q6K, false>(a, pl, mw, ma, sm_count, pdl, stream);
}

}  // namespace tc

bool qgemm_tc_supported(int fmt, const GemmTcArgs &a) {
    if (a.k % QK != 0 || a.k < QK || a.rows < 1 || ((uintptr_t)a.w & 15) != 0 || tc::encode_fn() == nullptr) return false;
    // (Q6_K rows that are not 16-byte multiples are copied by byte offsets inside groups of eight: a 32-bit coordinate)
    if (fmt == FMT_Q6K && a.k / QK * Q6K_BYTES % 16 != 0 && 8 * (uint64_t)(a.k / QK) * Q6K_BYTES >= (1ull << 31)) return false;
    return fmt == FMT_Q4K || fmt == FMT_Q5K || fmt == FMT_Q6K;
}

static uint32_t tc_block_bytes(int fmt) { return fmt == FMT_Q4K ? Q4K_BYTES : fmt == FMT_Q5K ? Q5K_BYTES : Q6K_BYTES; }
static uint32_t tc_box_bytes(int fmt) { return fmt == FMT_Q6K ? (uint32_t)tc::Q6K_BOX : tc_block_bytes(fmt); }

// Tiles and K splits of a launch on single CTAs or on pairs. The activation rows are divided evenly over as few tiles as hold them. Whole tiles run in rounds over the CTAs (pairs); K is split for the tiles of the last round when that round would be less than
// half full: `ways` units to a tile, as many as fit the round, never below two super-blocks each, never more than
// SPLITK_SCRATCH_MAX of partial sums. Half full is where two ways stop fitting one round, and then they cost more than they give (77 rows of
// Q4_K, K = 4096, on 148 SMs, not split / two / three ways: 64 tiles 27.3 / 20.2 / 26.1 us, 74 tiles 27.2 / 20.7 / 26.3, 75 tiles 27.3 / 30.7 / 26.4,
// 112 tiles 27.5 / 32.2 / 33.8; 256 rows in pairs, 43 tiles on 74 pairs: 32.0 / 41.5 / 37.5).
constexpr size_t SPLITK_SCRATCH_MAX = (size_t)256 << 20;
static GemmTcPlan cut(bool pair, uint32_t rows, uint32_t n, uint32_t k, int sm_count, int splitk, uint64_t &walk) {
    tc::Plan p{};
    p.pair = pair;
    const uint32_t cap = p.pair ? 256 : 128, gran = p.pair ? 32 : 16, width = p.pair ? 2 * tc::TN : tc::TN;
    p.ny = (rows + cap - 1) / cap;
    p.mt = ((rows + p.ny - 1) / p.ny + gran - 1) / gran * gran;
    p.nx = (n + width - 1) / width;
    const uint64_t tiles = (uint64_t)p.nx * p.ny;
    const uint32_t workers = (uint32_t)(p.pair ? sm_count / 2 : sm_count), nblk = k / QK;
    uint64_t tail = 0;
    uint32_t ways = 1;
    if (splitk > 1) {
        tail = tiles;
        ways = (uint32_t)splitk;
    } else if (splitk < 0 && workers > 0) {
        tail = tiles % workers;
        if (tail * 2 > workers) tail = 0;
        if (tail) ways = (uint32_t)(workers / tail);
    }
    if (ways > nblk / 2) ways = nblk / 2;
    if (ways > 16) ways = 16;
    while (ways > 1 && tail * ways * p.mt * width * 4 > SPLITK_SCRATCH_MAX) ways--;
    // every split must own at least one super-block
    while (ways > 1 && (uint64_t)(ways - 1) * ((nblk + ways - 1) / ways) >= nblk) ways--;
    if (ways <= 1) ways = 1, tail = 0;
    p.splits = ways;
    p.full = (uint32_t)(tiles - tail);
    p.units = (uint32_t)(tiles - tail + tail * ways);
    // the super-blocks that the CTA (pair) with the most to do walks
    walk = workers ? (tiles - tail + workers - 1) / workers * nblk + (tail * ways + workers - 1) / workers * ((nblk + ways - 1) / ways) : 0;
    return p;
}
// Above 128 rows pairs of CTAs: an expanded weight feeds twice the activation rows. A pair takes some 2 us longer to start and end, though, so launches
// whose tiles fit the single CTAs as well (no CTA walks more super-blocks) stay on those: few rows of weights, or K too short to be split. Single CTAs
// against pairs: 2048 rows on 300 x 256 Q4_K 10.3 / 12.9 us (the kernel before pairs 11.4), 1024 rows on 768 x 512 10.4 / 12.8 (12.1), 4096 rows on
// 128 x 2048 17.9 / 21.5 (19.9); where they walk more: 4096 rows on 1024 x 1024 (8 super-blocks against 4) 24.6 / 20.2.
GemmTcPlan qgemm_tc_plan(uint32_t rows, uint32_t n, uint32_t k, int sm_count, const GemmTcTuning &tuning) {
    uint64_t single, pairs;
    const GemmTcPlan one = cut(false, rows, n, k, sm_count, tuning.splitk, single);
    if (rows <= 128 || tuning.pair == 0) return one;
    const GemmTcPlan two = cut(true, rows, n, k, sm_count, tuning.splitk, pairs);
    return tuning.pair < 0 && single <= pairs ? one : two;
}

// the bf16 copy of the activations, and the partial sums of a split-K launch
size_t qgemm_tc_copy_bytes(uint32_t rows, uint32_t k) { return ((size_t)rows * k * 2 + 255) & ~(size_t)255; }
size_t qgemm_tc_partial_bytes(const GemmTcPlan &p) { return (size_t)p.split_units() * p.mt * (p.pair ? 2 * tc::TN : tc::TN) * 4; }

bool qgemm_tc_moe_supported(int fmt, uint64_t experts, uint64_t n, uint64_t k, const void *w) {
    if (fmt != FMT_Q4K && fmt != FMT_Q5K && fmt != FMT_Q6K) return false;
    if (k % QK != 0 || k < QK || ((uintptr_t)w & 15) != 0 || tc::encode_fn() == nullptr) return false;
    const uint64_t pitch = k / QK * tc_block_bytes(fmt);
    // one tensor map over all experts' rows: rows of 16-byte multiples, no padding between the matrices
    return pitch % 16 == 0 && (n * pitch) % 256 == 0 && experts * n < (1ull << 31);
}

// Tensor maps: packed weights as bytes [weight rows][row bytes], box = one block (Q6_K: the 240 bytes around one) of 128 rows (Q6_K rows that are not
// 16-byte multiples: [groups of eight rows][their bytes], box = 240 bytes of 16 groups); bf16 activations
// [k / 64][rows][64], box = 64 k (128 bytes, swizzled) x the rows a CTA loads x the k-steps of a stage.
static cudaError_t tc_maps(int fmt, const GemmTcArgs &a, uint64_t weight_rows, const tc::Plan &pl, void *a_bf16, CUtensorMap &mw, CUtensorMap &ma) {
    const tc::EncodeTiledFn enc = tc::encode_fn();
    if (!enc) return cudaErrorNotSupported;
    const uint32_t blk_bytes = tc_block_bytes(fmt);
    cuuint32_t es[3] = {1, 1, 1};
    {
        cuuint64_t dims[2] = {(cuuint64_t)(a.k / QK) * blk_bytes, weight_rows};
        cuuint64_t strides[1] = {(cuuint64_t)(a.k / QK) * blk_bytes};
        cuuint32_t box[2] = {(cuuint32_t)tc_box_bytes(fmt), tc::TN};
        if (strides[0] % 16 != 0) {  // Q6_K with K not a multiple of 2048: a row of the map is a group of eight, a copy takes one row of 16 groups
            dims[0] *= 8, strides[0] *= 8, dims[1] /= 8;
            box[1] = tc::TN / 8;
        }
        if (dims[1] == 0) std::memset(&mw, 0, sizeof(mw));  // (no whole group: not used)
        else if (enc(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void *)a.w, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    {
        cuuint64_t dims[3] = {tc::KS, a.rows, a.k / tc::KS};
        cuuint64_t strides[2] = {tc::KS * 2, (cuuint64_t)a.rows * tc::KS * 2};
        cuuint32_t box[3] = {tc::KS, pl.pair ? pl.mt / 2 : pl.mt, tc::STAGE_KS};
        if (enc(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, a_bf16, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}
static void tc_fill(GemmTcArgs &a, const tc::Plan &pl, uint32_t group) {
    a.tiles_x = pl.nx, a.tiles_y = pl.ny, a.splits = pl.splits, a.full = pl.full, a.units = pl.units, a.mt = pl.mt, a.group = group;
}

cudaError_t launch_qgemm_tc_moe(int fmt, const GemmTcArgs &a, uint32_t experts, uint32_t mt, void *a_bf16, int sm_count, bool pdl, cudaStream_t stream) {
    if (a.rows == 0 || a.n == 0) return cudaSuccess;
    if (!a.tile_expert || !a.row_pair || a.rows % mt != 0 || mt % 32 != 0 || mt > 256) return cudaErrorInvalidValue;
    tc::Plan pl{};
    pl.pair = mt > 128;
    pl.mt = mt;
    pl.nx = (a.n + (pl.pair ? 2 : 1) * tc::TN - 1) / ((pl.pair ? 2 : 1) * tc::TN);
    pl.ny = a.rows / mt;
    if ((uint64_t)pl.nx * pl.ny >= (1u << 31)) return cudaErrorInvalidValue;
    pl.splits = 1;
    pl.full = pl.units = pl.nx * pl.ny;
    CUtensorMap mw, ma;
    if (cudaError_t e = tc_maps(fmt, a, (uint64_t)experts * a.n, pl, a_bf16, mw, ma); e != cudaSuccess) return e;
    GemmTcArgs b = a;
    tc_fill(b, pl, 1);
    return tc::launch_plan(fmt, b, pl, mw, ma, sm_count, pdl, stream);
}

cudaError_t launch_qgemm_tc(int fmt, const GemmTcArgs &a, const GemmTcPlan &pl, void *a_bf16_scratch, bool copy, void *partial, int sm_count, bool pdl,
                            cudaStream_t stream, int *launched) {
    using namespace tc;
    *launched = 0;
    if (a.rows == 0 || a.n == 0) return cudaSuccess;
    if ((uint64_t)pl.nx * pl.ny * pl.splits >= (1u << 31)) return cudaErrorInvalidValue;
    CUtensorMap mw, ma;
    if (cudaError_t e = tc_maps(fmt, a, a.n, pl, a_bf16_scratch, mw, ma); e != cudaSuccess) return e;

    if (copy) {
        const dim3 cgrid((a.k / 8 + 255) / 256, a.rows < 65535u ? a.rows : 65535u);
        const bool vec = a.a_type == ACT_F32 && ((uintptr_t)a.a & 15) == 0 && a.a_off % 4 == 0 && a.a_bs % 4 == 0 && a.a_rs % 4 == 0;
        LaunchCfg l(cgrid, 256, 0, pdl, false, stream);
        if (cudaError_t e = cudaLaunchKernelEx(&l.cfg, vec ? a_to_bf16_kernel<true> : a_to_bf16_kernel<false>, a, (__nv_bfloat16 *)a_bf16_scratch);
            e != cudaSuccess)
            return e;
        ++*launched;
    }
    GemmTcArgs b = a;
    b.partial = (float *)partial;
    tc_fill(b, pl, 8);
    if (cudaError_t e = launch_plan(fmt, b, pl, mw, ma, sm_count, pdl, stream); e != cudaSuccess) return e;
    ++*launched;
    if (pl.split_units()) {
        const uint64_t threads = (uint64_t)(pl.split_units() / pl.splits) * pl.mt * (pl.pair ? 64 : 32), blocks = (threads + 255) / 256;
        LaunchCfg l(dim3((unsigned)(blocks > (uint64_t)sm_count * 8 ? (uint64_t)sm_count * 8 : blocks)), 256, 0, pdl, false, stream);
        if (cudaError_t e = pl.pair ? cudaLaunchKernelEx(&l.cfg, splitk_sum_kernel<256>, b) : cudaLaunchKernelEx(&l.cfg, splitk_sum_kernel<128>, b); e != cudaSuccess) return e;
        ++*launched;
    }
    return cudaSuccess;
}

}  // namespace lb

// Decode GEMV skeleton for formats whose weights become int8 by byte permutes or lookups (MXFP4; the i-quants at several rows), 1..8 activation rows.
// A unit is 32 weights of one matrix row: one lane's work, multiplied with one activation group. A warp step is 32 consecutive units of a row.
//
// What bounds these formats is instruction issue and the load / store unit, not HBM (2 to 4 bits a weight), so the kernel is laid out to spend
// little of either beside the unpacking itself:
//   * every CTA owns an equal share of the matrix rows (of all members of a grouped launch, concatenated), its warps are G groups of rows x KS
//     slices of k, and a warp takes RB rows at a time: the activations of a step are read once for RB rows, their packed bytes are requested one
//     step ahead, and RB sums are reduced by one transposing shuffle tree;
//   * the quantized activations are copied to shared memory once, in two planes of 16 bytes a group (conflict-free wide loads), zeros behind the
//     end of k, so that the last step of a row needs no masks beside its loads.
// The first packed bytes do not depend on the kernel in front and are fetched before the dependency wait. One CTA of sixteen warps an SM: more and smaller ones
// copy the activations more often (three of eight warps: 4096 x 4096 6.8 against 6.3 us, six experts of 5120 x 2304 19.1 against 18.6). ROOM: a CTA takes
// three quarters of the registers (launch bounds of 640 threads: 96 each): with all of them the small kernel in front or behind (the activations' quantization)
// finds no room beside it and cannot overlap (IQ2_XXS, four rows on 2048 x 4096 8.9 -> 7.3 us, MXFP4, two rows on 2304 x 1024 4.9 -> 4.3).
//
// The integer sums of a group are exact and the products those of the reference; only the order in which the groups' f32 terms are added differs. It keeps the error no
// larger than that of the kernels before, which gave a row to up to four warps: every four steps by themselves (F::CHUNKS: MXFP4), the warps of a row, each with one
// rounding less, without roundings in between (against f64, MXFP4, one row on 4096 x 14336: before 8.3e-8, here 8.2e-8, as one chain 9.2e-8, on 1500 x 14336
// 8.2e-8, 6.5e-8, 8.8e-8). The i-quants' two halves of a unit are one
// exact sum here, two terms there.
//
// A format F gives: M_MIN and M_MAX (activation rows), DIRECT (activations that do not fit shared memory are read where they lie), TABLE_BYTES, fill() and
// Tables (lookup tables in shared memory, and where a lane reads them), AHEAD (packed bytes requested before the present ones are unpacked), CHUNKS (see above), STEP_BYTES and lane_offset() (where a lane's unit of a row
// lies), Raw and load() (its packed bytes, as they lie), W and unpack() (int8 weights and scale), dot() (a unit's integer sum as a float), order() (the activation group's bytes in the order of the weights).
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace lb {
namespace rs {

constexpr int WARPS = 16, THREADS = WARPS * 32, PARTS = 2048;

// Lane l gets the warp's sum of v[row_of(l)]: RB - 1 exchanges halve the rows, the rest is a plain tree, the last addition left to the caller.
template <int RB> __device__ __forceinline__ float2 reduce_rows(float (&v)[RB], int lane) {
    static_assert(RB == 1 || RB == 2 || RB == 4, "rows");
    int o = 16;
    float x[RB];
#pragma unroll
    for (int j = 0; j < RB; j++) x[j] = v[j];
#pragma unroll
    for (int n = RB; n > 1; n /= 2, o /= 2) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < n / 2; j++) {
            const float keep = up ? x[2 * j + 1] : x[2 * j], send = up ? x[2 * j] : x[2 * j + 1];
            x[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    float s = x[0];
#pragma unroll
    for (int p = 16 / RB; p > 1; p /= 2) s += __shfl_xor_sync(0xffffffffu, s, p);
    return make_float2(s, __shfl_xor_sync(0xffffffffu, s, 1));
}
template <int RB> __device__ __forceinline__ int row_of(int lane) {
    return RB == 4 ? 2 * ((lane >> 3) & 1) + ((lane >> 4) & 1) : RB == 2 ? (lane >> 4) & 1 : 0;
}

// The sum of n (up to WARPS) numbers that lie `STRIDE` apart.
template <int STRIDE> __device__ __forceinline__ float sum_parts(const double *x, uint32_t n) {
    double v[WARPS];
#pragma unroll
    for (int i = 0; i < WARPS; i++) v[i] = (uint32_t)i < n ? x[i * STRIDE] : 0.0;
#pragma unroll
    for (int w = 1; w < WARPS; w *= 2)
#pragma unroll
        for (int i = 0; i < WARPS; i += 2 * w) v[i] += v[i + w];
    return (float)v[0];
}

// ks_log: log2 of the warps that share a row; pass_rows: matrix rows of a CTA between two exchanges of their partial sums
template <class F, int M, int RB, bool ACT_SMEM, int NG, bool ROOM>
__global__ void __launch_bounds__(ROOM ? THREADS + 128 : THREADS, 1)
row_stream_kernel(const __grid_constant__ GemvGroupT<NG> grp, const uint8_t *__restrict__ table, uint32_t ks_log, uint32_t pass_rows) {
    extern __shared__ __align__(16) uint8_t smem[];
    // the member of the launch this CTA works for (task_end: CTAs), and its share of the rows
    int it = 0;
    if constexpr (NG > 1) {
#pragma unroll
        for (int i = 1; i < NG; i++)
            if (i < grp.count && blockIdx.x >= grp.task_end[i - 1]) it = i;
    }
    const GemvArgs &p = grp.item[it];
    const uint32_t cta = NG > 1 && it ? blockIdx.x - grp.task_end[it - 1] : blockIdx.x, ctas = NG > 1 ? grp.task_end[it] - (it ? grp.task_end[it - 1] : 0u) : gridDim.x;
    const uint32_t each = p.n / ctas, more = p.n - each * ctas;  // (the first `more` CTAs take one row more; 64-bit divisions would take longer than the smallest launches' sums)
    const uint32_t c0 = cta * each + min(cta, more), rows = each + (cta < more ? 1 : 0);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t ks_count = 1u << ks_log;
    const uint32_t k = p.k, units = k / GROUP, steps = (units + 31) / 32, whole = units / 32, sg = steps * 32;  // sg: groups of the padded planes
    double *part = (double *)(smem + F::TABLE_BYTES);
    uint8_t *acts = smem + F::TABLE_BYTES + (ks_count > 1 ? PARTS * 8 : 0);
    float *act_d = (float *)(acts + (size_t)M * sg * GROUP);
    constexpr int WARPS_LOG = 4;
    static_assert(1 << WARPS_LOG == WARPS, "warps");
    const uint32_t ks = warp & (ks_count - 1), group = warp >> ks_log;
    const int8_t *qa = p.qa;
    const float *da = p.da;
    float *out = p.out + p.out_off;
    const uint8_t *w = p.w + (uint64_t)c0 * F::row_bytes(k);
    const uint32_t row_bytes = (uint32_t)F::row_bytes(k);

    // this warp's rows of a pass that starts at p0: [r0, r1), counted from c0
    auto slice = [&](uint32_t p0, uint32_t &r0, uint32_t &r1) {
        const uint32_t n = min(pass_rows, rows - p0);
        r0 = p0 + (n * group >> (WARPS_LOG - ks_log)), r1 = p0 + (n * (group + 1) >> (WARPS_LOG - ks_log));
    };
    // The packed bytes are requested one step ahead: of this warp's next step, rows or pass. A CTA's rows lie within 4 GB of their first byte.
    typename F::Raw raw[RB];
    const uint8_t *base = (const uint8_t *)((uintptr_t)w & ~(uintptr_t)3);
    uint32_t at[RB];     // this lane's unit of the rows being requested, from `base`
    uint32_t ahead = 0;  // their step
    auto rows_at = [&](uint32_t row, uint32_t end) {
        ahead = ks;
        const uint32_t first = (uint32_t)((uintptr_t)w & 3) + F::lane_offset(lane) + ks * F::STEP_BYTES;
#pragma unroll
        for (int j = 0; j < RB; j++) at[j] = (row + j < end ? row + j : row) * row_bytes + first;
    };
    auto request = [&]() {
        if (ahead < whole || 32 * ahead + lane < units) {
#pragma unroll
            for (int j = 0; j < RB; j++) raw[j] = F::load(base, at[j], lane);
        } else {
#pragma unroll
            for (int j = 0; j < RB; j++) raw[j] = F::none();
        }
#pragma unroll
        for (int j = 0; j < RB; j++) at[j] += ks_count * F::STEP_BYTES;
        ahead += ks_count;
    };
    uint32_t r0, r1;
    slice(0, r0, r1);
    if (!p.ids && r0 < r1) rows_at(r0, r1), request();
    F::fill(smem, table, threadIdx.x, THREADS);
    // The arguments that the end of the kernel reads are fetched before the wait: a launch's arguments are in no cache yet.
    asm volatile("" ::"r"(p.m), "l"(p.out_bs), "l"(p.out_rs), "l"(p.extra), "r"(p.epi.n), "l"(p.ex_off), "l"(p.ex_s2));
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (p.ids) {
        // Expert-indexed launch (Kernel::MatMulId at decode sizes): grid row y is one (token, slot) pair
        const uint32_t pair = blockIdx.y, token = pair / p.id_r;
        const int32_t id = p.ids[pair];
        const bool bad = id < 0 || (uint32_t)id >= p.id_e;
        if (bad && p.status && threadIdx.x == 0) atomicOr(p.status, 128);
        w += bad ? 0 : (uint64_t)id * p.id_stride;
        base = (const uint8_t *)((uintptr_t)w & ~(uintptr_t)3);
        qa += (uint64_t)token * k;
        da += (uint64_t)token * units;
        out += (uint64_t)pair * p.n;
        if (r0 < r1) rows_at(r0, r1), request();
    }
    if constexpr (ACT_SMEM) {
        for (uint32_t i = threadIdx.x; i < M * sg; i += THREADS) {
            uint32_t r = 0, g = i;
#pragma unroll
            for (int j = 1; j < M; j++)
                if (g >= sg) g -= sg, r++;
            uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
            float d = 0.0f;
            if (g < units) {
                const uint4 *src = (const uint4 *)(qa + (uint64_t)r * k + (uint64_t)g * GROUP);
                lo = src[0], hi = src[1];
                d = da[(uint64_t)r * units + g];
                F::order(lo, hi);
            }
            *(uint4 *)(acts + ((size_t)(2 * r) * sg + g) * 16) = lo;
            *(uint4 *)(acts + ((size_t)(2 * r + 1) * sg + g) * 16) = hi;
            act_d[(size_t)r * sg + g] = d;
        }
    }
    __syncthreads();
    const typename F::Tables tables(smem, lane);
    auto store = [&](uint32_t row, uint32_t r, float v) {
        const uint32_t col = c0 + row;
        uint32_t bt = 0, i = r;
        if (M > 1 && r >= p.m) bt = r / p.m, i = r % p.m;
        if (p.extra && !p.epi.n) v += p.extra[p.ex_off + (int64_t)bt * p.ex_s0 + (int64_t)i * p.ex_s1 + (int64_t)col * p.ex_s2];
        out[(uint64_t)bt * p.out_bs + (uint64_t)i * p.out_rs + col] = v;
    };
    for (uint32_t p0 = 0; p0 < rows; p0 += pass_rows) {
        for (uint32_t row = r0; row < r1; row += RB) {
            const uint32_t left = r1 - row;
            // Every four steps are summed by themselves. More activation rows have no registers to spare (pick() splits k instead), and where a CTA has matrix rows for
            // four a warp, a row had one warp before, too.
            constexpr bool CHUNKS = F::CHUNKS && M <= 2 && RB <= 2;
            float acc[M][RB], total[M][RB];
            uint32_t left_in_chunk = 4;
#pragma unroll
            for (int r = 0; r < M; r++)
#pragma unroll
                for (int j = 0; j < RB; j++) acc[r][j] = total[r][j] = 0.0f;
            for (uint32_t step = ks; step < steps; step += ks_count) {
                typename F::W wv[RB];
                // the packed bytes of what comes next are on their way while this is unpacked and multiplied (F::AHEAD; else while it is multiplied, which
                // saves the copies)
                auto next = [&]() {
                    if (ahead < steps) request();
                    else if (row + RB < r1) rows_at(row + RB, r1), request();
                };
                typename F::Raw cur[RB];
#pragma unroll
                for (int j = 0; j < RB; j++) cur[j] = raw[j];
                if (F::AHEAD) next();
                if (left >= RB) {
#pragma unroll
                    for (int j = 0; j < RB; j++) wv[j] = F::unpack(cur[j], tables);
                } else {  // (the rows that are missing cost their loads alone)
#pragma unroll
                    for (int j = 0; j < RB; j++)
                        if (j == 0 || j < left) wv[j] = F::unpack(cur[j], tables);
                        else wv[j] = wv[0];
                }
                if (!F::AHEAD) next();
                const uint32_t g = 32 * step + lane;
#pragma unroll
                for (int r = 0; r < M; r++) {
                    uint4 lo, hi;
                    float d;
                    if constexpr (ACT_SMEM) {
                        lo = *(const uint4 *)(acts + ((size_t)(2 * r) * sg + g) * 16), hi = *(const uint4 *)(acts + ((size_t)(2 * r + 1) * sg + g) * 16);
                        d = act_d[(size_t)r * sg + g];
                    } else {
                        lo = make_uint4(0, 0, 0, 0), hi = lo, d = 0.0f;
                        if (g < units) {
                            const uint4 *src = (const uint4 *)(qa + (uint64_t)r * k + (uint64_t)g * GROUP);
                            lo = __ldg(src), hi = __ldg(src + 1);
                            d = __ldg(da + (uint64_t)r * units + g);
                            F::order(lo, hi);
                        }
                    }
                    const uint32_t a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                    for (int j = 0; j < RB; j++) acc[r][j] = fmaf(wv[j].d * d, F::dot(wv[j], a), acc[r][j]);
                }
                if (CHUNKS && --left_in_chunk == 0) {
                    left_in_chunk = 4;
#pragma unroll
                    for (int r = 0; r < M; r++)
#pragma unroll
                        for (int j = 0; j < RB; j++) total[r][j] += acc[r][j], acc[r][j] = 0.0f;
                }
            }
            float2 v[M];
#pragma unroll
            for (int r = 0; r < M; r++) {
#pragma unroll
                for (int j = 0; CHUNKS && j < RB; j++) acc[r][j] += total[r][j];
                v[r] = reduce_rows<RB>(acc[r], lane);
            }
            const uint32_t mine = row + row_of<RB>(lane);
            if (lane % (32 / RB) == 0 && mine < r1) {
                if (ks_count > 1) {
#pragma unroll
                    for (int r = 0; r < M; r++) part[(((mine - p0) << ks_log) + ks) * M + r] = (double)v[r].x + (double)v[r].y;
                } else {
#pragma unroll
                    for (int r = 0; r < M; r++) store(mine, r, v[r].x + v[r].y);
                }
            }
        }
        const uint32_t n = min(pass_rows, rows - p0);
        if (n < rows - p0) {
            slice(p0 + pass_rows, r0, r1);
            if (r0 < r1) rows_at(r0, r1), request();
        }
        if (ks_count > 1) {
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < n * M; i += THREADS) {
                const uint32_t row = i / M, r = i % M;
                store(p0 + row, r, sum_parts<M>(part + (row << ks_log) * M + r, ks_count));
            }
            __syncthreads();  // the partial sums are read: the next pass may overwrite them
        }
    }
}

// Shared memory of a launch.
template <class F> static size_t smem_bytes(uint32_t rows, uint32_t k, uint32_t ks, bool acts) {
    const size_t sg = ((size_t)k / GROUP + 31) / 32 * 32;
    return F::TABLE_BYTES + (ks > 1 ? PARTS * 8 : 0) + (acts ? (size_t)rows * sg * (GROUP + 4) : 0);
}

// How a launch is cut.
struct Cut {
    uint32_t grid, end[GEMV_GROUP_MAX];  // CTAs in all (for each pair), and up to each member's end
    uint64_t mine;                       // matrix rows of the busiest CTA
};
// A launch has one CTA per SM. Its members get as many of them as their rows are worth. Each pair of an expert-indexed launch gets the same number, rounded down, so that
// up to a third of the SMs stay without a CTA (56 pairs: 112 CTAs).
template <class F> static Cut cut_rows(const GemvGroup &g, uint32_t pairs, int sm_count) {
    Cut c{};
    uint64_t rows = 0, seen = 0;
    for (int i = 0; i < g.count; i++) rows += g.item[i].n;
    uint32_t ctas = (uint32_t)sm_count / pairs;
    const uint64_t least = (rows * F::row_bytes(g.item[0].k) >> 31) + g.count;  // (offsets inside a CTA's share have 32 bits)
    if (ctas < least) ctas = (uint32_t)least;
    for (int i = 0; i < g.count; i++) {
        const uint64_t n = g.item[i].n;
        seen += n;
        uint64_t to = (seen * ctas + rows / 2) / rows;
        if (to <= c.grid) to = c.grid + 1;
        if (to - c.grid > n) to = c.grid + n;
        const uint64_t each = (n + (to - c.grid) - 1) / (to - c.grid);
        if (each > c.mine) c.mine = each;
        c.end[i] = c.grid = (uint32_t)to;
    }
    return c;
}
// Matrix rows that a warp takes at a time (RB: 1, 2) and warps per row (KS): the least time of the slowest warp, in steps of one row. A step of two rows
// takes 1.4 (one activation row) to 1.9 (eight) steps of one, and as much when the second row is missing; a reduction about a sixth of a step, an exchange as
// much again. One row at a time only where a warp has no second one: else the activations' loads are what two rows share (eight rows, IQ2_XXS, 14336 x 4096 26.8
// against 35.0 us). At least `least` warps. MXFP4, one activation row: 2304 x 1024 one row, one warp 3.52, two rows 3.80; 1024 x 14336 one row, two warps 7.9, two rows, four warps 6.7.
static void pick(uint32_t m, uint64_t mine, uint32_t steps, uint32_t least, int force_ks, int &rb, uint32_t &ks) {
    double best = 1e30;
    for (uint32_t c = least; c <= WARPS && c <= steps; c *= 2) {
        if (force_ks && (uint32_t)force_ks <= steps && c != (uint32_t)force_ks) continue;
        const uint64_t r = (mine * c + WARPS - 1) / WARPS;
        const double row = (double)((steps + c - 1) / c) + (c > 1 ? 0.33 : 0.17), pair = row * (double)((r + 1) / 2) * (1.35 + 0.07 * m);
        if (r == 1 && row < best) best = row, rb = 1, ks = c;
        if (pair < best) best = pair, rb = 2, ks = c;
    }
}

template <class F, int M, int RB, bool ACT_SMEM, int NG, bool ROOM = true>
static cudaError_t launch(const GemvGroup &all, const uint8_t *table, const Cut &cut, uint32_t ks, uint32_t pairs, bool pdl, cudaStream_t stream) {
    GemvGroupT<NG> g{};
    g.count = all.count;
    for (int i = 0; i < all.count; i++) g.item[i] = all.item[i], g.task_end[i] = cut.end[i];
    const uint32_t k = g.item[0].k;
    if ((cut.mine + 1) * F::row_bytes(k) >> 32) return cudaErrorInvalidValue;
    uint32_t ks_log = 0;
    while (2u << ks_log <= ks) ks_log++;
    const uint32_t pass = ks > 1 ? PARTS / (ks * M) : (uint32_t)cut.mine;  // (one pass where nothing is exchanged)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cut.grid, pairs);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem_bytes<F>(M, k, ks, ACT_SMEM);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    static DynamicSmemOptIn optin;
    cudaError_t e = optin.raise((const void *)row_stream_kernel<F, M, RB, ACT_SMEM, NG, ROOM>, cfg.dynamicSmemBytes);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, row_stream_kernel<F, M, RB, ACT_SMEM, NG, ROOM>, g, table, ks_log, pass);
}

// One activation row over many matrix rows: four of them share the activation loads and give the schedulers more independent work, two leave fewer warps idle at the
// end of a CTA's share: MXFP4, 14336 x 4096 12.2 against 14.6 us, 28672 x 4096 19.5 against 23.3, but 4096 x 4096 8.9 against 6.3 and 4096 x 14336 18.1 against
// 13.9. Two activation rows have no registers for four (14336 x 4096 17.2, with spills, against 15.5). Long launches of that kind and those of several expert pairs
// gain more from all registers than from what runs beside them: us, 96 / 128 registers, 11008 x 4096 10.6 / 11.5, 28672 x 4096 19.5 / 20.0, 128256 x 2048 36.1 /
// 35.3, six experts of 2304 x 5120, gate and up, 21.7 / 20.9, 64 of 1408 x 2048 54.7 / 51.5.
// One activation row and at most one step for each warp: the activations are read where they lie, once, instead of copied (256 x 1024 3.29 -> 3.24, 2304 x 1024
// 3.52 -> 3.34; 2304 x 2048, two steps, 3.91 -> 3.93; two activation rows 256 x 1024 3.90 -> 4.04).
constexpr uint32_t FOUR_ROWS_FROM = 64, SHORT_STEPS = 800;  // matrix rows of a CTA; times the steps of a row
constexpr size_t ACT_SMEM_MAX = 200 * 1024;
template <class F, int M, int NG> static cudaError_t launch_rows(const GemvGroup &g, const uint8_t *table, uint32_t pairs, int force_ks, int sm_count, bool pdl, cudaStream_t stream) {
    const uint32_t k = g.item[0].k, steps = (k / GROUP + 31) / 32;
    const bool acts = smem_bytes<F>(M, k, 2, true) <= ACT_SMEM_MAX;
    const Cut cut = cut_rows<F>(g, pairs, sm_count);
    int rb = 2;
    uint32_t ks = 1;
    // (three MXFP4 rows and more: few matrix rows had two warps each before, too)
    pick(M, cut.mine, steps, F::CHUNKS && M > 2 && cut.mine < 32 && steps > 4 && !force_ks ? 2 : 1, force_ks, rb, ks);
    if constexpr (M == 1) {
        if (F::DIRECT && cut.mine * steps <= WARPS) return launch<F, M, 1, false, NG>(g, table, cut, ks, pairs, pdl, stream);
        if (acts && cut.mine >= FOUR_ROWS_FROM)
            return pairs == 1 && cut.mine * steps <= SHORT_STEPS ? launch<F, M, 4, true, NG>(g, table, cut, ks, pairs, pdl, stream)
                                                                 : launch<F, M, 4, true, NG, false>(g, table, cut, ks, pairs, pdl, stream);
    }
    if (acts && rb == 1) return launch<F, M, 1, true, NG>(g, table, cut, ks, pairs, pdl, stream);
    if (acts) return launch<F, M, 2, true, NG>(g, table, cut, ks, pairs, pdl, stream);
    if constexpr (F::DIRECT) return launch<F, M, 2, false, NG>(g, table, cut, ks, pairs, pdl, stream);
    return cudaErrorInvalidValue;
}

// F::M_MIN..F::M_MAX activation rows
template <class F, int NG, int M = F::M_MIN> static cudaError_t launch_m(const GemvGroup &g, const uint8_t *table, int force_ks, int sm_count, bool pdl, cudaStream_t stream) {
    if (g.item[0].rows == M) return launch_rows<F, M, NG>(g, table, 1, force_ks, sm_count, pdl, stream);
    if constexpr (M < F::M_MAX) return launch_m<F, NG, M + 1>(g, table, force_ks, sm_count, pdl, stream);
    else return cudaErrorInvalidValue;
}

// One launch for the members of `g` (same format, rows, k and activations). Expert-indexed (same ids too): one-row work for each pair.
template <class F> static cudaError_t launch_group(const GemvGroup &g, const uint8_t *table, int force_ks, int sm_count, bool pdl, cudaStream_t stream) {
    if (g.count < 1 || g.count > GEMV_GROUP_MAX) return cudaErrorInvalidValue;
    const GemvArgs &a = g.item[0];
    if (F::M_MIN == 1 && a.ids) {
        if (a.id_r == 0 || a.id_e == 0 || a.rows > 8 || (uint64_t)a.rows * a.id_r > 65535) return cudaErrorInvalidValue;
        GemvGroup one = g;
        for (int i = 0; i < g.count; i++) one.item[i].rows = one.item[i].m = 1;
        return g.count == 1 ? launch_rows<F, F::M_MIN, 1>(one, table, a.rows * a.id_r, force_ks, sm_count, pdl, stream)
                            : launch_rows<F, F::M_MIN, GEMV_GROUP_MAX>(one, table, a.rows * a.id_r, force_ks, sm_count, pdl, stream);
    }
    return g.count == 1 ? launch_m<F, 1>(g, table, force_ks, sm_count, pdl, stream) : launch_m<F, GEMV_GROUP_MAX>(g, table, force_ks, sm_count, pdl, stream);
}

}  // namespace rs
}  // namespace lb

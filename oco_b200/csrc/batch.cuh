// Expert products for a few tokens (about two routes per expert, e.g. a decode batch of 64 over
// 128 experts). The work is still memory-bound, and a 32-route tile would decode every weight
// block for two live columns, so the rows are streamed as in the single-token kernels
// (decode.cuh) with the eight columns of the MMA's B operand holding up to eight routes of the
// same expert. Numerics are the tile kernels': half operands, fp32 accumulation, the same
// epilogues (reference expert_up_tensor / expert_down_tensor, shaders/experts/projections.metal:
// 185-420, taken at a tile height of eight).
//
//   route_plan_kernel (tile_rows = 8)  ->  groups of up to 8 routes of one expert
//   batch_fragments_kernel             ->  each group's token rows as B fragments
//   batch_rows_kernel, up epilogue     ->  activations (half, expert-sorted) + the down stage's fragments
//   batch_rows_kernel, down epilogue   ->  bf16 expert outputs in route order
#pragma once
#include "decode.cuh"
#include "gemm.cuh"

namespace oco {

constexpr int kBatchWarps = 16;                     // one CTA per SM; the group's fragments take 512 bytes a block
constexpr int kBatchThreads = kBatchWarps * 32;
constexpr int kBatchCols = 8;
constexpr int kBatchFragBlock = kBatchCols * 64;    // bytes of one block's B fragments

__host__ __device__ inline size_t batch_smem_bytes(int fmt, int nkb) {
    return (size_t)nkb * kBatchFragBlock + kMiscBytes + (size_t)kBatchWarps * scale_table_bytes(fmt) +
           (size_t)kBatchWarps * 2 * kStageBytes + 16;
}

// Position (in halves) of element k of column `col` in a group's fragments: frag_place within the block, but for Q4_K
// neighbours (RowStream::chunk_kh).
__host__ __device__ inline size_t batch_frag_pos(int fmt, int k, int col) {
    int tig, slot, sel;
    if (fmt == OCO_FMT_Q4_K) {
        tig = (k & 31) >> 3; slot = (k & 7) >> 1; sel = k & 1;
    } else {
        frag_place(fmt, k & 31, tig, slot, sel);
    }
    return ((((size_t)(k >> 5) * kBatchCols + col) * 4 + tig) * 4 + slot) * 2 + sel;
}

// The token rows of every route group as B fragments (bf16 -> half, zero in unused columns).
// grid: max groups; one thread per 16-byte fragment piece (block, column, tig).
template <int FMT>
__global__ void __launch_bounds__(256) batch_fragments_kernel(const uint16_t* __restrict__ x,
                                                              const uint32_t* __restrict__ tiles,
                                                              const uint32_t* __restrict__ tile_count,
                                                              const uint32_t* __restrict__ offsets,
                                                              const uint32_t* __restrict__ route_of_row, int per_row,
                                                              int H, uint4* __restrict__ frag) {
    pdl_launch_dependents();
    pdl_wait();
    if (blockIdx.x >= *tile_count) return;
    const uint32_t expert = tiles[2 * blockIdx.x], begin = tiles[2 * blockIdx.x + 1];
    const uint32_t row0 = offsets[expert] + begin, count = offsets[expert + 1] - offsets[expert];
    const int n = (int)min((uint32_t)kBatchCols, count - begin);
    const int nkb = H / 32;
    uint4* out = frag + (size_t)blockIdx.x * nkb * (kBatchFragBlock / 16);
    for (int i = threadIdx.x; i < nkb * 32; i += 256) {
        const int kb = i >> 5, col = (i >> 2) & 7, tig = i & 3;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (col < n) {
            const uint32_t token = route_of_row[row0 + col] / (uint32_t)per_row;
            // elements 4 tig .. 4 tig + 3 and the same of the elements 16 further; Q4_K: 8 tig .. 8 tig + 7
            const uint16_t* src = x + (size_t)token * H + kb * 32 + (FMT == OCO_FMT_Q4_K ? 8 : 4) * tig;
            const uint2 lo = *reinterpret_cast<const uint2*>(src), hi = *reinterpret_cast<const uint2*>(src + (FMT == OCO_FMT_Q4_K ? 4 : 16));
            auto pair = [](uint32_t a, uint32_t b) {          // (bf16 a, bf16 b) -> half2
                __half2 h = __floats2half2_rn(__uint_as_float(a << 16), __uint_as_float(b << 16));
                return *reinterpret_cast<uint32_t*>(&h);
            };
            if (FMT == OCO_FMT_Q4_K) {                        // neighbours (batch_frag_pos)
                v.x = pair(lo.x & 0xffffu, lo.x >> 16);
                v.y = pair(lo.y & 0xffffu, lo.y >> 16);
                v.z = pair(hi.x & 0xffffu, hi.x >> 16);
                v.w = pair(hi.y & 0xffffu, hi.y >> 16);
            } else if (FMT == OCO_FMT_Q4_0) {                 // elements two apart (frag_place)
                v.x = pair(lo.x & 0xffffu, lo.y & 0xffffu);
                v.y = pair(lo.x >> 16, lo.y >> 16);
                v.z = pair(hi.x & 0xffffu, hi.y & 0xffffu);
                v.w = pair(hi.x >> 16, hi.y >> 16);
            } else {
                v.x = pair(lo.x & 0xffffu, hi.x & 0xffffu);
                v.y = pair(lo.x >> 16, hi.x >> 16);
                v.z = pair(lo.y & 0xffffu, hi.y & 0xffffu);
                v.w = pair(lo.y >> 16, hi.y >> 16);
            }
        }
        out[i] = v;
    }
}

struct BatchParams {
    const uint8_t* w0;        // expand: gate rows (up rows when not gated); down: the down rows
    const uint8_t* w1;        // expand, gated: up rows
    const float* b0;
    const float* b1;
    const uint32_t* tiles;    // (expert, first row within the expert) per route group
    const uint32_t* tile_count;
    const uint32_t* offsets;
    const uint32_t* route_of_row;
    const __half* frag_in;    // [group][n_in / 32] blocks of 512 bytes
    __half* frag_out;         // expand: the down stage's fragments, [group][n_out / 32] blocks
    uint16_t* out;            // expand: half [R, n_out] expert-sorted, operand order; down: bf16 [R, n_out] route order
    int n_in, n_out;          // contraction length, output features
    uint32_t row_bytes;       // bytes from one weight row of a matrix to its next row
    int bias_stride;          // floats from one feature's bias to the next
    uint32_t* status;
};

// EPI as in gemm.cuh. Persistent: the work is a list of rounds, a round being sixteen units (16 weight rows each)
// of one group, one per warp, and every CTA takes an equal run of the list. With a CTA for each eighth of a group
// (or fewer) the last wave decided: 19 groups made 152 CTAs of three rounds on 148 SMs, six rounds where three
// suffice. Within its run a warp starts the next unit's first stage under the last stage of the one before, across
// groups too, so that its rows never stop; only the group's fragments are waited for when the group changes.
// Up to 18 groups (eight CTAs and more each) whole rounds are too coarse: 15 groups of 180 units are 32 CTAs of two
// rounds beside 116 of one. There the CTAs are dealt out to the groups and take equal shares of a group's units, unless
// the longest share exceeds the longest run of whole rounds. With fewer CTAs to a group the equal runs are the better
// deal: 8 to 20 tokens took 1 to 2 % longer with shares.
// gpt-oss-20b-shaped layer, a CTA for each eighth | equal runs | this: 2 tokens 109.5 | 85.5 | 78.1 us, 5 tokens 113.4 | 118.8
// | 112.7, 6 tokens 114.6 | 120.2 | 116.0, 8 tokens 187.6 | 136.2 | 136.1, 40 tokens 198 | 186 | 187; 7 tokens, norm
// included, 130 or 153 by the routes | 131.6 | 128.7; 120b-shaped of 64 tokens 560 | 490 | 491 (519 | 487 on other routes).
// Qwen3 (Q4_K), which took 256-route tiles for any batch: 2 rows 136 -> 66 us, 8 rows 351 -> 130, 32 rows 280 -> 210,
// 96 rows 327 -> 259.
template <int FMT, int EPI>
__global__ void __launch_bounds__(kBatchThreads, 1) batch_rows_kernel(const BatchParams p) {
    constexpr bool GATED = epi_gated(EPI);
    constexpr bool DOWN = EPI == kEpiDownBf16;
    constexpr int ROWS = GATED ? 8 : 16;              // output features per unit
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, tig = lane & 3;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nkb = p.n_in / 32;
    const uint32_t part_off = (uint32_t)nkb * kBatchFragBlock;
    float* misc = reinterpret_cast<float*>(smem + part_off);
    volatile uint32_t* give_up = reinterpret_cast<volatile uint32_t*>(misc) + 496;
    const uint32_t xbar = smem_u32(smem) + part_off + 1920u;
    const uint32_t stab = part_off + kMiscBytes + (uint32_t)warp * scale_table_bytes(FMT);
    const uint32_t ring = part_off + kMiscBytes + (uint32_t)kBatchWarps * scale_table_bytes(FMT) + (uint32_t)warp * 2 * kStageBytes;
    pdl_launch_dependents();
    RowStream<FMT, 2, kBatchCols> rs;
    rs.init(smem, ring, stab, part_off + 1280u + (uint32_t)warp * 16u, give_up, p.status, lane);
    if (tid == 0) {
        *give_up = 0u;
        mbar_init(xbar, 1);
        fence_barrier_init();
    }
    pdl_wait();               // the route plan and the group fragments are complete
    __syncthreads();          // the mbarriers exist

    const int units = p.n_out / ROWS, rounds = (units + kBatchWarps - 1) / kBatchWarps;
    const int groups = (int)*p.tile_count, ctas = (int)gridDim.x, cta = (int)blockIdx.x, total = groups * rounds;   // total * ctas: well below 2^31
    int r_begin = total * cta / ctas, r_end = total * (cta + 1) / ctas, first = warp, last = units;
    const int per = groups ? ctas / groups : 0;
    if (per >= 8 && (units + per - 1) / per <= kBatchWarps * ((total + ctas - 1) / ctas)) {
        const int group = cta / per, k = cta - group * per;
        r_begin = r_end = group * rounds;
        if (group < groups) {                         // (the last CTAs may have no group)
            first = units * k / per;
            last = units * (k + 1) / per;
            r_end += (last - first + kBatchWarps - 1) / kBatchWarps;
            first += warp;
        }
    }
    // the spans of this warp's unit in a round; null where the group's last round has none for it
    auto spans = [&](int round, const uint8_t*& a, const uint8_t*& b) {
        a = b = nullptr;
        const int group = round / rounds, u = (round - group * rounds) * kBatchWarps + first;
        if (u >= last) return;
        const size_t off = ((size_t)__ldg(p.tiles + 2 * group) * p.n_out + (size_t)u * ROWS) * p.row_bytes;
        a = p.w0 + off;
        b = GATED ? p.w1 + off : a + (size_t)8 * p.row_bytes;
    };
    const uint32_t xlane = (uint32_t)((g * 4 + tig) * 16);
    const int c0 = 2 * tig, c1 = 2 * tig + 1;
    const uint8_t *na = nullptr, *nb = nullptr;       // this warp's unit of the round to come
    auto find = [&](int from) {
        na = nb = nullptr;
        for (int next = from; next < r_end && !na; next++) spans(next, na, nb);
    };
    find(r_begin);
    uint32_t phase = 0;
    for (int r0 = r_begin; r0 < r_end;) {
        const int group = r0 / rounds, seg_end = min(r_end, (group + 1) * rounds);
        if (r0 != r_begin) __syncthreads();           // nobody still reads the fragments of the group before
        if (tid == 0) {
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(xbar, part_off);
            bulk_copy(smem_u32(smem), p.frag_in + (size_t)group * nkb * (kBatchFragBlock / 2), part_off, xbar);
        }
        const uint32_t expert = __ldg(p.tiles + 2 * group), begin = __ldg(p.tiles + 2 * group + 1);
        const uint32_t row0 = __ldg(p.offsets + expert) + begin, count = __ldg(p.offsets + expert + 1) - __ldg(p.offsets + expert);
        const int n = (int)min((uint32_t)kBatchCols, count - begin);
        rs.ncols = n;
        // the routes of this lane's two columns
        uint32_t orow0 = 0, orow1 = 0;
        if (c0 < n) orow0 = DOWN ? p.route_of_row[row0 + c0] : row0 + c0;
        if (c1 < n) orow1 = DOWN ? p.route_of_row[row0 + c1] : row0 + c1;
        __half* fout = DOWN ? nullptr : p.frag_out + (size_t)group * (p.n_out / 32) * (kBatchFragBlock / 2);
        bool fetched = false;
        for (int round = r0; round < seg_end; round++) {
            const int u = (round - group * rounds) * kBatchWarps + first;
            if (u >= last) continue;                 // na, nb stay: the unit of a later round
            const uint8_t *a = na, *b = nb;
            find(round + 1);
            const int f0 = u * ROWS;
            rs.begin(a, b, p.row_bytes, 0, nkb);
            // biases travel while the rows stream: accumulator rows g (span A) and g (span B)
            const int fa = f0 + g, fb = GATED ? fa : fa + 8;
            float bias_a = 0.f, bias_b = 0.f;
            if (p.b0) bias_a = bf16_round(__ldg(p.b0 + ((size_t)expert * p.n_out + fa) * p.bias_stride));
            if (GATED) {
                if (EPI == kEpiSwigluF16) bias_b = bf16_round(__fadd_rn(__ldg(p.b1 + ((size_t)expert * p.n_out + fa) * p.bias_stride), 1.0f));
            } else if (p.b0) {
                bias_b = bf16_round(__ldg(p.b0 + ((size_t)expert * p.n_out + fb) * p.bias_stride));
            }
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
            if (!fetched) { mbar_wait(xbar, phase, give_up, p.status); fetched = true; }
            rs.run(xlane, sum, na, nb);
            // sum[0..1]: row g of span A x columns c0, c1; sum[2..3]: row g of span B
            auto put = [&](int col, uint32_t orow, int f, uint16_t h) {
                if (DOWN) {
                    p.out[(size_t)orow * p.n_out + f] = h;
                } else {
                    p.out[(size_t)orow * p.n_out + operand_pos(FMT, f)] = h;
                    reinterpret_cast<uint16_t*>(fout)[batch_frag_pos(FMT, f, col)] = h;
                }
            };
            if (GATED) {
                if (c0 < n) put(c0, orow0, fa, epilogue_value<EPI>(__fadd_rn(sum[0], bias_a), __fadd_rn(sum[2], bias_b)));
                if (c1 < n) put(c1, orow1, fa, epilogue_value<EPI>(__fadd_rn(sum[1], bias_a), __fadd_rn(sum[3], bias_b)));
            } else {
                if (c0 < n) {
                    put(c0, orow0, fa, epilogue_value<EPI>(__fadd_rn(sum[0], bias_a), 0.f));
                    put(c0, orow0, fb, epilogue_value<EPI>(__fadd_rn(sum[2], bias_b), 0.f));
                }
                if (c1 < n) {
                    put(c1, orow1, fa, epilogue_value<EPI>(__fadd_rn(sum[1], bias_a), 0.f));
                    put(c1, orow1, fb, epilogue_value<EPI>(__fadd_rn(sum[3], bias_b), 0.f));
                }
            }
        }
        if (!fetched) mbar_wait(xbar, phase, give_up, p.status);   // the copy has landed before the next one, or the exit
        phase ^= 1u;
        r0 = seg_end;
    }
}

}  // namespace oco

// Q3G64_F16S linears of many rows on sm_100a as one launch: the 3-bit codes are turned into BF16 operands on their way into the
// tensor core's shared-memory tiles. Stands behind the reference's Q3 prefill entries (native/include/euhedral_cuda.h:173-197).
//
// Exactness: code * f32(scale) is the sum of two BF16 numbers, code * hi + code * lo, where hi is the FP16 scale cut to 6
// significant bits and lo the other 5: a code has at most 2, so both products have at most 8. Both multiply the unchanged BF16
// activations; products are exact in FP32, an output is one FP32 sum in K order (64 values of hi terms, the same 64 of lo terms),
// rounded once to BF16. Nothing in that order depends on the rows of a call or of the tensor.
//
// Bound: shared memory (profiles/q3_prefill_kernel_600_rows.md), then the tensor pipe, 4 M N K FLOP. A separate launch that wrote both terms to memory (4 bytes a weight), which this replaces,
// took most of a call of few rows (a layer's four fused linears, 5120 wide, at 40 / 300 / 600 / 1024 / 4096 rows: 745 / 853 / 1093 / 1467 / 4332 us before,
// 284 / 430 / 662 / 1083 / 3997 now, 250 / 383 / 634 / 1010 / 3843 without the release at cluster scope that passes the odd CTA's word on).
// Here the terms of a weight are made once per tile of up to 256 activation rows, beside the MMAs:
// 2.6 instructions a code (16-bit windows of the code stream, so that two neighbouring codes land in the two halves of a
// BF16 pair: one mask, one packed FMA, two packed multiplies), 190 issue slots per 64 values of K where the MMAs of a full tile take
// 1024 cycles.
//
// The weights are the M operand (256 rows on a CTA pair, tcgen05 cta_group::2, 128 in each CTA), the activation rows the N operand, so
// that a call of any row count is cut into equal tiles of up to 256 rows (a multiple of 16) with next to no padding.
//   * warp 2: raw codes of 128 values (48 bytes a row) by TMA, their two scales a row by cp.async, three slots. Tensor maps address
//     device memory only: codes that lie elsewhere (host-mapped, managed) come by cp.async as the scales do.
//   * warps 4..19: codes -> the two BF16 tiles of 64 values (128-byte swizzle), four stages
//   * warp 0: the activation tile of a stage by TMA, half in each CTA, counted on the even CTA's barrier
//   * warp 1 of the even CTA: eight MMAs a stage; two accumulators of up to 256 columns
//   * warps 1, 3, 24 and 25 of the odd CTA: pass on to the even one that the odd half of a stage is made
//   * warps 20..23: a thread has one output column and walks the tile's rows; in the paired region (a tile holds 64 gate rows and the
//     64 up rows that match them) the up half meets the gate half in shared memory
// Every wait is bounded.
#pragma once

#include <algorithm>

#include "bf16_gemm.cuh"
#include "q3_gemv.cuh"

namespace q3p {

constexpr uint32_t kThreads = 832, kStages = 4, kRawSlots = 3;
constexpr uint32_t kATile = 128u * 128u, kBTile = 128u * 128u, kStageBytes = 2u * kATile + kBTile;   // hi, lo, half of the activation tile
constexpr uint32_t kRawCodes = 128u * 48u, kRawBytes = kRawCodes + 128u * 4u;
constexpr uint32_t kOffRaw = kStages * kStageBytes, kOffUp = kOffRaw + kRawSlots * kRawBytes, kUpPitch = 17u;
constexpr uint32_t kOffBars = kOffUp + 64u * kUpPitch * 4u, kSharedBytes = kOffBars + 256u + 1024u;
constexpr uint32_t kWaitFailed = bf16n::kWaitFailed;

// Two neighbouring codes sit in 6 bits of both halves of `w` (from bit 0 on): the first is read from the low half at bits 0..2, the
// second from the high half at bits 3..5. As BF16 mantissa bits over 0x4300 they read 128 + (code ^ 4) and 128 + 8 (code ^ 4).
__device__ __forceinline__ uint32_t code_pair(uint32_t w, uint32_t mask, uint32_t magic) {
    return eb::bf16x2_fma(eb::lop3<eb::kLutAndXor>(w, mask, magic), 0x3E003F80u, 0xC1A0C304u);   // * (1, 1/8) - (132, 20)
}
// The eight codes of 24 bits as four pairs.
__device__ __forceinline__ void codes8(uint32_t bits, uint32_t mask, uint32_t magic, uint32_t (&pair)[4]) {
    const uint32_t low = __byte_perm(bits, 0u, 0x1010), high = __byte_perm(bits, 0u, 0x2121);   // bits 0..15 and 8..23, twice each
    pair[0] = code_pair(low, mask, magic);
    pair[1] = code_pair(low >> 6, mask, magic);
    pair[2] = code_pair(high >> 4, mask, magic);
    pair[3] = code_pair(high >> 10, mask, magic);
}

__device__ __forceinline__ void sts_v4(uint32_t to, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

//   grid 2 x pairs, cluster 2, block kThreads, dynamic shared kSharedBytes. map_x: activations [rows][k] BF16, box 64 x tile / 2;
//   map_w: codes [weight_rows][k * 3 / 32] 32-bit, box 12 x 64, used when `codes` (the same plane) is null. tile: activation rows of an item. gate_rows != 0: the paired region
//   (the output has gate_rows columns), else the output has weight_rows columns.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) kernel(const __grid_constant__ CUtensorMap map_x,
        const __grid_constant__ CUtensorMap map_w, const uint8_t* __restrict__ codes, const uint8_t* __restrict__ scales, uint16_t* __restrict__ out, uint32_t rows, uint32_t weight_rows,
        uint32_t k, uint32_t tile, uint32_t gate_rows, uint32_t* __restrict__ error) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~(uintptr_t)1023u);
    uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + kOffBars);
    uint64_t *raw_empty = raw_full + kRawSlots, *rows_full = raw_empty + kRawSlots, *made = rows_full + kStages, *empty = made + kStages,
             *acc_full = empty + kStages, *acc_empty = acc_full + 2;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
    uint32_t* failed = tmem_holder + 1;
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;
    const uint32_t rank = eb::cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const bool paired = gate_rows != 0u;
    const uint32_t columns = paired ? gate_rows : weight_rows;                 // of the output
    const uint32_t span = paired ? 64u : 128u;                                 // output columns of a CTA's tile
    const uint32_t weight_tiles = (columns + 2u * span - 1u) / (2u * span), items = weight_tiles * ((rows + tile - 1u) / tile);
    const uint32_t chunks = k / 128u, stages_item = k / 64u;
    auto wait = [&](uint64_t* bar, uint32_t parity) { eb::mbar_wait_or_fail(bar, parity, failed); };
    // Weight tiles run fastest: the pairs of a wave share one tile of activation rows.
    auto first_column = [&](uint32_t item) { return (item % weight_tiles * 2u + rank) * span; };   // of this CTA
    auto first_row = [&](uint32_t item) { return item / weight_tiles * tile; };

    if (warp == 0) {
        if (lane < kRawSlots) {
            eb::mbar_init(&raw_full[lane], 33);    // the TMA request and the lanes' cp.async
            eb::mbar_init(&raw_empty[lane], 16);
        } else if (lane >= 8u && lane < 8u + kStages) {
            eb::mbar_init(&rows_full[lane - 8u], 1);
            eb::mbar_init(&made[lane - 8u], rank == 0u ? 9 : 8);   // eight converting warps, and word from the odd CTA
            eb::mbar_init(&empty[lane - 8u], 1);
        } else if (lane >= 16u && lane < 18u) {
            eb::mbar_init(&acc_full[lane - 16u], 1);
            eb::mbar_init(&acc_empty[lane - 16u], 8);
        } else if (lane == 18u) {
            *failed = 0u;
        }
        eb::mbar_fence_init();
    } else if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(eb::smem_u32(tmem_holder)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    nvfp4n::tcgen05_fence_before();
    __syncthreads();
    eb::cluster_sync();   // both CTAs' barriers exist before anything arrives on them from the other CTA
    nvfp4n::tcgen05_fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_holder, 0);
    eb::pdl_launch_dependents();

    // Odd CTA: tells the even one whenever the terms of this stage are made. An arrive that releases memory to another CTA takes a
    // microsecond or more: by the converting warps themselves a layer's linears took 1.4 to 1.8 times as long, by one warp for every two
    // stages 4096 x 14336 at 600 rows took 123 us, by one for each 120 (107 without the release).
    auto pass_on = [&](uint32_t stage) {
        const uint32_t total = (items - pair + pairs - 1u) / pairs * stages_item;   // stages of all items
        uint32_t parity = 0u;
        for (uint32_t i = stage; i < total; i += kStages, parity ^= 1u) {
            wait(&made[stage], parity);
            if (lane == 0u) nvfp4n::signal_rank(&made[stage], 0u);
            __syncwarp();
        }
    };

    if (warp == 0) {
        const bool leader = eb::elect_one();
        const uint32_t bytes = tile / 2u * 128u;
        eb::Ring ring;
        bool first_round = true;
        eb::pdl_wait();   // the activations may come from the launch before
        for (uint32_t item = pair; item < items; item += pairs) {
            const int row = (int)(first_row(item) + rank * (tile / 2u));
            for (uint32_t ks = 0; ks < stages_item; ++ks) {
                if (!first_round) wait(&empty[ring.stage], ring.parity ^ 1u);
                if (leader) {
                    if (rank == 0u) eb::mbar_arrive_expect_tx(&rows_full[ring.stage], 2u * bytes);
                    nvfp4n::pair_tma_load_2d(smem + ring.stage * kStageBytes + 2u * kATile, &map_x, (int)(ks * 64u), row,
                            eb::map_to_rank(eb::smem_u32(&rows_full[ring.stage]), 0u));
                }
                __syncwarp();
                ring.advance(kStages);
                first_round = first_round && ring.stage != 0u;
            }
        }
    } else if (warp == 1) {
        if (rank == 0u) {   // the odd CTA issues nothing: its tiles are read by the even CTA's MMAs
            const bool leader = eb::elect_one();
            const uint32_t instruction = (1u << 4) | (1u << 7) | (1u << 10) | ((tile >> 3) << 17) | ((256u >> 4) << 24);
            const uint64_t first = nvfp4n::tile_descriptor(smem);
            eb::Ring ring, accumulator;
            bool used = false;   // both accumulators have been used once
            for (uint32_t item = pair; item < items; item += pairs) {
                if (used) wait(&acc_empty[accumulator.stage], accumulator.parity ^ 1u);
                nvfp4n::tcgen05_fence_after();
                const uint32_t d = tmem + accumulator.stage * 256u;
                for (uint32_t ks = 0; ks < stages_item; ++ks) {
                    wait(&rows_full[ring.stage], ring.parity);
                    eb::mbar_wait_cluster_or_fail(&made[ring.stage], ring.parity, failed);   // half of the terms are in the other CTA
                    nvfp4n::tcgen05_fence_after();
                    const uint64_t hi = first + (uint64_t)(ring.stage * kStageBytes >> 4), lo = hi + (uint64_t)(kATile >> 4), x = lo + (uint64_t)(kATile >> 4);
                    if (leader) {
#pragma unroll
                        for (uint32_t j = 0; j < 4u; ++j) bf16n::pair_mma_bf16(d, hi + 2u * j, x + 2u * j, instruction, (uint32_t)((ks | j) != 0u));
#pragma unroll
                        for (uint32_t j = 0; j < 4u; ++j) bf16n::pair_mma_bf16(d, lo + 2u * j, x + 2u * j, instruction, 1u);
                        nvfp4n::pair_commit(&empty[ring.stage]);
                    }
                    __syncwarp();
                    ring.advance(kStages);
                }
                if (leader) nvfp4n::pair_commit(&acc_full[accumulator.stage]);
                __syncwarp();
                accumulator.advance(2u);
                used = used || accumulator.stage == 0u;
            }
        } else {
            pass_on(0u);
        }
    } else if (warp == 3 || warp >= 24u) {
        if (rank != 0u) pass_on(warp == 3u ? 1u : warp - 22u);
    } else if (warp == 2) {
        const bool leader = eb::elect_one();
        eb::Ring ring;
        bool first_round = true;
        const uint32_t pitch = chunks * 4u;   // scale bytes of a row
        for (uint32_t item = pair; item < items; item += pairs) {
            const uint32_t low = first_column(item), high = paired ? gate_rows + low : low + 64u;   // first weight rows of the tile's halves
            const uint8_t* from[4];
            bool live[4];
            auto weight_row = [&](uint32_t j) { return (j < 2u ? low : high - 64u) + j * 32u + lane; };
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {
                live[j] = weight_row(j) < weight_rows;
                from[j] = scales + (uint64_t)(live[j] ? weight_row(j) : 0u) * pitch;
            }
            for (uint32_t c = 0; c < chunks; ++c) {
                if (!first_round) wait(&raw_empty[ring.stage], ring.parity ^ 1u);
                uint8_t* slot = smem + kOffRaw + ring.stage * kRawBytes;
                if (codes != nullptr) {
#pragma unroll 1
                    for (uint32_t j = 0; j < 4u; ++j) {
                        const uint8_t* row = codes + (uint64_t)(live[j] ? weight_row(j) : 0u) * (chunks * 48u) + c * 48u;
                        for (uint32_t i = 0; i < 48u; i += 16u)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(eb::smem_u32(slot) + (j * 32u + lane) * 48u + i), "l"(row + i),
                                    "r"(live[j] ? 16 : 0)
                                    : "memory");
                    }
                    if (leader) eb::mbar_arrive(&raw_full[ring.stage]);
                } else if (leader) {
                    eb::mbar_arrive_expect_tx(&raw_full[ring.stage], kRawCodes);
                    eb::tma_load_2d(slot, &map_w, (int)(c * 12u), (int)low, &raw_full[ring.stage]);
                    eb::tma_load_2d(slot + kRawCodes / 2u, &map_w, (int)(c * 12u), (int)high, &raw_full[ring.stage]);
                }
                const uint32_t to = eb::smem_u32(slot + kRawCodes) + lane * 4u;
#pragma unroll
                for (uint32_t j = 0; j < 4u; ++j) {
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + j * 128u), "l"(from[j]), "r"(live[j] ? 4 : 0) : "memory");
                    from[j] += 4;
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(eb::smem_u32(&raw_full[ring.stage])) : "memory");
                __syncwarp();
                ring.advance(kRawSlots);
                first_round = first_round && ring.stage != 0u;
            }
        }
        eb::cp_async_wait_all();
    } else if (warp >= 4u && warp < 20u) {
        // A thread makes 32 values (half a group) of one weight row of every other stage: warps 4..11 the even stages, 12..19 the odd
        // ones, so that the latencies of two stages overlap.
        const uint32_t odd = warp >= 12u ? 1u : 0u, row = ((warp - 4u) & 7u) * 16u + (lane >> 1), half = lane & 1u;
        const uint32_t mask = eb::pinned(0x00380007u), magic = eb::pinned(0x43204304u);
        uint32_t at[4];   // this thread's four 16-byte pieces of a tile row under the 128-byte swizzle
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) at[i] = eb::smem_u32(smem) + row * 128u + (((half * 4u + i) ^ (row & 7u)) << 4);
        eb::Ring ring, raw;   // ring: of pairs of stages
        bool first_round = true;
        for (uint32_t item = pair; item < items; item += pairs) {
            for (uint32_t c = 0; c < chunks; ++c) {
                wait(&raw_full[raw.stage], raw.parity);
                const uint8_t* slot = smem + kOffRaw + raw.stage * kRawBytes;
                const uint32_t* words = reinterpret_cast<const uint32_t*>(slot + row * 48u + odd * 24u + half * 12u);
                const uint32_t w0 = words[0], w1 = words[1], w2 = words[2];
                const float scale = __half2float(*reinterpret_cast<const __half*>(slot + kRawCodes + row * 4u + odd * 2u));
                __syncwarp();
                if (lane == 0u) eb::mbar_arrive(&raw_empty[raw.stage]);
                raw.advance(kRawSlots);
                const float scale_hi = __uint_as_float(__float_as_uint(scale) & 0xFFFC0000u), scale_lo = __fsub_rn(scale, scale_hi);   // exact
                const uint32_t hi2 = eb::bf16_pair(scale_hi, scale_hi), lo2 = eb::bf16_pair(scale_lo, scale_lo);
                const uint32_t bits[4] = {w0, __funnelshift_r(w0, w1, 24), __funnelshift_r(w1, w2, 16), w2 >> 8};
                uint32_t p[4][4];
#pragma unroll
                for (uint32_t i = 0; i < 4u; ++i) codes8(bits[i], mask, magic, p[i]);
                const uint32_t stage = 2u * ring.stage + odd, to = stage * kStageBytes;
                if (!first_round) wait(&empty[stage], ring.parity ^ 1u);
#pragma unroll
                for (uint32_t i = 0; i < 4u; ++i) {
                    sts_v4(at[i] + to, eb::bf16x2_mul(p[i][0], hi2), eb::bf16x2_mul(p[i][1], hi2), eb::bf16x2_mul(p[i][2], hi2), eb::bf16x2_mul(p[i][3], hi2));
                    sts_v4(at[i] + to + kATile, eb::bf16x2_mul(p[i][0], lo2), eb::bf16x2_mul(p[i][1], lo2), eb::bf16x2_mul(p[i][2], lo2), eb::bf16x2_mul(p[i][3], lo2));
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // what was written is for the tensor core to read
                __syncwarp();
                if (lane == 0u) eb::mbar_arrive(&made[stage]);
                ring.advance(kStages / 2u);
                first_round = first_round && ring.stage != 0u;
            }
        }
    } else if (warp >= 20u) {
        const uint32_t quarter = warp & 3u, local = quarter * 32u + lane;        // this thread's weight row of the CTA's 128
        float* up_sums = reinterpret_cast<float*>(smem + kOffUp) + (local & 63u) * kUpPitch;
        eb::Ring accumulator;
        eb::pdl_wait();   // the output may be what the launch before reads
        for (uint32_t item = pair; item < items; item += pairs) {
            const uint32_t column = first_column(item) + (paired ? local & 63u : local), row0 = first_row(item);
            wait(&acc_full[accumulator.stage], accumulator.parity);
            nvfp4n::tcgen05_fence_after();
            const uint32_t d = tmem + ((quarter * 32u) << 16) + accumulator.stage * 256u;
            uint16_t* to = out + (uint64_t)row0 * columns + column;
            const bool live = column < columns;
#pragma unroll 1
            for (uint32_t h = 0; h < tile; h += 16u) {
                uint32_t r[16];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                        : "r"(d + h));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (paired) {
                    if (local >= 64u)
#pragma unroll
                        for (uint32_t i = 0; i < 16u; ++i) up_sums[i] = __uint_as_float(r[i]);
                    epilogue_sync();
                }
                if (!paired || local < 64u) {
#pragma unroll
                    for (uint32_t i = 0; i < 16u; ++i) {   // a warp writes 32 neighbouring values of a row
                        float value = __uint_as_float(r[i]);
                        if (paired) {   // gate and up rounded to BF16 before the SwiGLU (the reference's paired kernel)
                            const float gate = eb::bf16_bits_to_float(eb::float_to_bf16_bits(value)), up = eb::bf16_bits_to_float(eb::float_to_bf16_bits(up_sums[i]));
                            value = __fmul_rn(__fdiv_rn(gate, __fadd_rn(1.0f, expf(-gate))), up);
                        }
                        if (live && row0 + h + i < rows) to[(uint64_t)(h + i) * columns] = eb::float_to_bf16_bits(value);
                    }
                }
                if (paired) epilogue_sync();   // the up sums have been read
            }
            nvfp4n::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0u) nvfp4n::signal_rank_relaxed(&acc_empty[accumulator.stage], 0u);
            accumulator.advance(2u);
        }
    }
    nvfp4n::tcgen05_fence_before();
    __syncthreads();
    if (*failed != 0u && threadIdx.x == 0) atomicOr(error, kWaitFailed);
    eb::cluster_sync();   // neither CTA leaves while the other may still read its shared memory or arrive on its barriers
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

inline cudaError_t initialize() { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSharedBytes); }

// Activation rows of an item: the fewest waves of pairs times what a stage of 64 values of K costs, and a little for every item's
// epilogue. A stage measured 466 / 545 / 589 / 645 ns at 48 / 128 / 160 / 208 rows (the difference of K = 10240 and 5120 on 18,944 weight
// rows), in which shared memory moves 32 KB of terms in and out and the activations in once and out twice; at 256 rows, where the
// MMAs take 1024 cycles, 709 ns in a call of 4096 rows under the power cap.
inline uint32_t tile_of(uint32_t rows, uint32_t weight_tiles, uint32_t pairs) {
    uint32_t best = 256u;
    uint64_t best_cost = ~0ull;
    for (uint32_t count = (rows + 255u) / 256u; count <= (rows + 31u) / 32u; ++count) {
        const uint32_t tile = ((rows + count - 1u) / count + 15u) / 16u * 16u, tiles = (rows + tile - 1u) / tile;
        const uint64_t cost = (((uint64_t)weight_tiles * tiles + pairs - 1u) / pairs) * (std::max(44000u + 85u * tile, 310u * tile) + 2000u);   // 1/100 ns
        if (cost < best_cost) {
            best_cost = cost;
            best = tile;
        }
        if ((uint64_t)weight_tiles * tiles > 64ull * pairs) break;
    }
    return best;
}

// x [rows][k] BF16, w a Q3G64_F16S tensor of weight_rows rows; all 16-byte aligned, k % 128 == 0, weight_rows % 128 == 0. x and out are
// device memory, w any memory that the device can read.
// paired: w is a gate/up object (gate rows first), the output [rows][weight_rows / 2] SwiGLU values.
inline cudaError_t linear(const void* x, const void* w, void* out, uint32_t rows, uint32_t k, uint32_t weight_rows, bool paired, int sms, cudaStream_t stream,
        bool pdl, uint32_t* error) {
    const eb::EncodeTiled encode = eb::encoder();
    if (encode == nullptr) return cudaErrorNotSupported;
    const q3::Geometry geo(weight_rows, k);
    const uint32_t gate_rows = paired ? weight_rows / 2u : 0u, columns = paired ? gate_rows : weight_rows, span = paired ? 128u : 256u;
    const uint32_t weight_tiles = (columns + span - 1u) / span, most = (uint32_t)sms / 2u, tile = tile_of(rows, weight_tiles, most);
    cudaPointerAttributes attributes;
    const bool device_memory = cudaPointerGetAttributes(&attributes, w) == cudaSuccess && attributes.type == cudaMemoryTypeDevice;
    (void)cudaGetLastError();
    CUtensorMap map_x, map_w;
    const cuuint32_t ones[2] = {1u, 1u}, x_box[2] = {64u, tile / 2u}, w_box[2] = {12u, 64u};
    const cuuint64_t x_dims[2] = {k, rows}, x_strides[1] = {(cuuint64_t)k * 2u}, w_dims[2] = {geo.row_bytes / 4u, weight_rows}, w_strides[1] = {geo.row_bytes};
    if (encode(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), x_dims, x_strides, x_box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                    != CUDA_SUCCESS
            || (device_memory && encode(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(w), w_dims, w_strides, w_box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                    != CUDA_SUCCESS))
        return cudaErrorInvalidValue;
    if (!device_memory) map_w = map_x;
    const uint32_t items = weight_tiles * ((rows + tile - 1u) / tile);
    return eb::launch_on(stream, pdl, 1u, kernel, dim3(2u * std::min(most, items)), dim3(kThreads), kSharedBytes, map_x, map_w,
            device_memory ? nullptr : static_cast<const uint8_t*>(w), static_cast<const uint8_t*>(w) + geo.scale_offset, static_cast<uint16_t*>(out), rows, weight_rows, k, tile, gate_rows, error);
}

}  // namespace q3p

// BF16 x BF16 -> BF16 linear on tcgen05 (kind::f16, FP32 accumulators in tensor memory) for the trellis prefill route:
// out[r][j] = bf16(sum_k a[r][k] * b[j][k]) for a [rows][k] and b [n][k], both BF16 and K-major. It stands where the
// reference's trellis prefill calls its row-exact BF16 linear on the decoded weights
// (core/.../artifact/format/TrellisFormat.java:560-604, RowExactBf16.java:52-84): every output is one FP32 sum over K in
// K order whatever the row count, so a row's bits do not depend on the rows beside it.
//
// The engine is the NVFP4 prefill kernel's (nvfp4_native.cuh) without scales: a persistent CTA per SM walks 128 x 256
// output tiles; warp 0 requests the stages by TMA (64 K of the 128 activation rows and of the 256 weight rows: 48 KB,
// 128-byte swizzle, four stages), one thread of warp 1 issues four K = 16 MMAs per stage and commits the stage back, eight
// epilogue warps drain a 128 x 256 accumulator into registers, hand it back and round and store, while the MMAs of the next
// tile fill the other accumulator (two of 256 columns: all of tensor memory). Every wait is bounded.
#pragma once

#include <atomic>

#include "nvfp4_native.cuh"
#include "trellis_codebook.cuh"

namespace bf16n {

using nvfp4n::kTileM;
using nvfp4n::kTileN;
using nvfp4n::kTmemColumns;

constexpr uint32_t kThreads = 384;                                // TMA warp, MMA warp, two that idle, eight epilogue warps
constexpr uint32_t kStepK = 64;                                   // BF16 values of K per stage: 128 bytes a row
constexpr uint32_t kATile = kTileM * 128u, kBTile = kTileN * 128u;
constexpr uint32_t kStageBytes = kATile + kBTile;
constexpr uint32_t kStages = 4;
constexpr uint32_t kSharedBytes = kStages * kStageBytes + 128u + 1024u;   // + barriers + slack to align to 1024
constexpr uint32_t kWaitFailed = 16u;                             // error bit: a bounded wait of this kernel gave up

// Registers: the launch's 168 a thread are shared out as 64 for the control warps and 208 for the epilogue, which holds 128 sums.
// kind::f16 instruction descriptor: FP32 accumulator, BF16 x BF16, both operands K-major, M 128, N 256.
constexpr uint32_t kInstruction = (1u << 4) | (1u << 7) | (1u << 10) | ((kTileN >> 3) << 17) | ((kTileM >> 4) << 24);

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate) {
    asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
            "l"(a_desc), "l"(b_desc), "r"(kInstruction), "r"(accumulate)
            : "memory");
}

// A thread's 128 consecutive sums of one row (one 128-column block of the trellis output) -> the block's final values:
// the sums rounded to BF16 as the plan's BF16 linear stores them, the block's Hadamard transform in FP32 by the format's
// butterflies (stage h pairs i with i + h; every a + b and a - b as trellis::hadamard128_warp forms them, so the bits are
// those of the plan's epilogue kernel), times 1/sqrt(128), times svh, BF16. No other thread is needed.
__device__ __forceinline__ void store_rotated(uint32_t (&r)[4][32], uint16_t* __restrict__ out, const uint16_t* __restrict__ svh) {
    float* v = reinterpret_cast<float*>(&r[0][0]);
    const bool wide = (reinterpret_cast<uintptr_t>(out) & 31u) == 0;
#pragma unroll
    for (int i = 0; i < 128; i += 2) {
        const uint32_t pair = eb::bf16_pair(v[i], v[i + 1]);
        v[i] = eb::bf16_bits_to_float(pair & 0xFFFFu);
        v[i + 1] = __uint_as_float(pair & 0xFFFF0000u);
    }
#pragma unroll
    for (int h = 1; h < 128; h <<= 1) {
#pragma unroll
        for (int p = 0; p < 64; ++p) {
            const int i = (p / h) * 2 * h + (p % h);
            const float a = v[i], b = v[i + h];
            v[i] = __fadd_rn(a, b);
            v[i + h] = __fsub_rn(a, b);
        }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        uint32_t packed[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 scales = *reinterpret_cast<const uint4*>(svh + 16 * c + 8 * h);
            const uint32_t sw[4] = {scales.x, scales.y, scales.z, scales.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 scale = __half22float2(*reinterpret_cast<const __half2*>(&sw[i]));
                const float* at = v + 16 * c + 8 * h + 2 * i;
                packed[4 * h + i] = eb::bf16_pair(__fmul_rn(scale.x, __fmul_rn(at[0], trellis::kInvSqrt128)),
                        __fmul_rn(scale.y, __fmul_rn(at[1], trellis::kInvSqrt128)));
            }
        }
        nvfp4n::store_16(out + 16 * c, packed, wide);
    }
}

// The columns of a call as segments that each have activations of their own (a fused trellis object rotates its input once per
// segment): segment g is columns [begin[g], begin[g + 1]) and multiplies rows [g * rows, (g + 1) * rows) of map_a. An output tile
// lies in one segment; tile_begin[g] is the number of tile columns before it.
constexpr uint32_t kMaxSegments = 8;
struct Segments {
    uint32_t count, begin[kMaxSegments + 1], tile_begin[kMaxSegments + 1];
    // Segment of tile column tn.
    __device__ __forceinline__ uint32_t of(uint32_t tn) const {
        uint32_t g = 0;
        while (g + 1u < count && tn >= tile_begin[g + 1u]) ++g;
        return g;
    }
};

//   grid: min(tiles, SMs), block kThreads, dynamic shared kSharedBytes. map_a: [rows][k] BF16, box 64 x 128;
//   map_b: [n][k] BF16, box 64 x 128 (a B tile is two boxes). n a multiple of 128. out: row stride `stride` elements.
//   svh null: out[r][j] = bf16(sum); else out[r][j] = the trellis output of the 128-column block j belongs to (svh [n]).
__global__ void __launch_bounds__(kThreads, 1) bf16_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
        uint16_t* __restrict__ out, const uint16_t* __restrict__ svh, uint32_t stride, uint32_t rows, uint32_t n, uint32_t k,
        const __grid_constant__ Segments segments, uint32_t* __restrict__ error) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~(uintptr_t)1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
    uint64_t* empty = full + kStages;
    uint64_t* acc_full = empty + kStages;    // two accumulators of 256 columns: the MMAs of a tile run while the tile before is drained
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const nvfp4n::TileWalk walk(rows, segments.tile_begin[segments.count]);
    const uint32_t k_steps = k / kStepK;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            eb::mbar_init(&full[s], 1);
            eb::mbar_init(&empty[s], 1);
        }
        for (uint32_t b = 0; b < 2u; ++b) {
            eb::mbar_init(&acc_full[b], 1);
            eb::mbar_init(&acc_empty[b], 8);
        }
        eb::mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(eb::smem_u32(tmem_holder)), "r"(kTmemColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    nvfp4n::tcgen05_fence_before();
    __syncthreads();
    nvfp4n::tcgen05_fence_after();
    const uint32_t tmem = *tmem_holder;
    eb::pdl_launch_dependents();
    eb::pdl_wait();   // both operands come from the launches before this one

    if (warp < 4u) {
      nvfp4n::registers_give_back<64>();
      if (warp == 0) {
        if (lane == 0) {
            uint32_t step = 0;
            bool ok = true;
            for (uint32_t tile = blockIdx.x; tile < walk.total && ok; tile += gridDim.x) {
                uint32_t tm, tn;
                walk.at(tile, &tm, &tn);
                const uint32_t g = segments.of(tn), column = segments.begin[g] + (tn - segments.tile_begin[g]) * kTileN;
                for (uint32_t ks = 0; ks < k_steps; ++ks, ++step) {
                    const uint32_t s = step % kStages, round = step / kStages;
                    if (round > 0 && !eb::mbar_wait(&empty[s], (round - 1u) & 1u)) {
                        atomicOr(error, kWaitFailed);
                        ok = false;
                        break;
                    }
                    uint8_t* stage = smem + s * kStageBytes;
                    eb::mbar_arrive_expect_tx(&full[s], kStageBytes);
                    // rows past the end of a matrix read as zeros (and the transaction still counts the whole box)
                    eb::tma_load_2d(stage, &map_a, (int)(ks * kStepK), (int)(g * rows + tm * kTileM), &full[s]);
                    eb::tma_load_2d(stage + kATile, &map_b, (int)(ks * kStepK), (int)column, &full[s]);
                    eb::tma_load_2d(stage + kATile + kBTile / 2u, &map_b, (int)(ks * kStepK), (int)column + 128, &full[s]);
                }
            }
        }
      } else if (warp == 1) {
        if (lane == 0) {
            uint32_t step = 0, local = 0;
            bool ok = true;
            for (uint32_t tile = blockIdx.x; tile < walk.total && ok; tile += gridDim.x, ++local) {
                const uint32_t buffer = local & 1u, use = local >> 1;
                if (use > 0 && !eb::mbar_wait(&acc_empty[buffer], (use - 1u) & 1u)) {
                    atomicOr(error, kWaitFailed);
                    break;
                }
                nvfp4n::tcgen05_fence_after();
                const uint32_t accumulator = tmem + buffer * kTileN;
                for (uint32_t ks = 0; ks < k_steps; ++ks, ++step) {
                    const uint32_t s = step % kStages, round = step / kStages;
                    if (!eb::mbar_wait(&full[s], round & 1u)) {
                        atomicOr(error, kWaitFailed);
                        ok = false;
                        break;
                    }
                    nvfp4n::tcgen05_fence_after();
                    const uint8_t* stage = smem + s * kStageBytes;
                    const uint64_t a = nvfp4n::tile_descriptor(stage), b = nvfp4n::tile_descriptor(stage + kATile);
#pragma unroll
                    for (uint32_t j = 0; j < 4u; ++j) mma_bf16(accumulator, a + 2u * j, b + 2u * j, (uint32_t)((ks | j) != 0u));   // 32 bytes of K further
                    nvfp4n::mma_commit(&empty[s]);
                }
                if (ok) nvfp4n::mma_commit(&acc_full[buffer]);
            }
        }
      }
    } else {
        // warp w reads the 32 accumulator rows of lane quarter w % 4; warps 4..7 take columns 0..127, warps 8..11 128..255
        nvfp4n::registers_take<208>();
        const uint32_t quarter = warp & 3u, half = (warp - 4u) >> 2;
        uint32_t local = 0;
        for (uint32_t tile = blockIdx.x; tile < walk.total; tile += gridDim.x, ++local) {
            uint32_t tm, tn;
            walk.at(tile, &tm, &tn);
            const uint32_t buffer = local & 1u;
            if (!eb::mbar_wait(&acc_full[buffer], (local >> 1) & 1u)) {
                if (lane == 0) atomicOr(error, kWaitFailed);
                break;
            }
            nvfp4n::tcgen05_fence_after();
            uint32_t r[4][32];
            const uint32_t from = tmem + ((quarter * 32u) << 16) + buffer * kTileN + half * 128u;
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) nvfp4n::tmem_load_32(r[i], from + 32u * i);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            nvfp4n::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) eb::mbar_arrive(&acc_empty[buffer]);
            const uint32_t g = segments.of(tn), end = segments.begin[g + 1u];
            const uint32_t row = tm * kTileM + quarter * 32u + lane;
            const uint32_t col = segments.begin[g] + (tn - segments.tile_begin[g]) * kTileN + half * 128u;
            if (svh == nullptr) {
                nvfp4n::store_block(r, out, row, rows, n, col, 1.0f, false);   // row stride n
            } else if (row < rows && col < end) {
                store_rotated(r, out + (uint64_t)row * stride + col, svh + col);
            }
        }
    }
    nvfp4n::tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns) : "memory");
    }
}

// ---- the same GEMM on CTA pairs -----------------------------------------------------------------------------------------
// Two CTAs of a cluster share an output tile of 256 rows x 256 columns: each holds its own 128 activation rows and HALF of
// the weight tile (128 weight rows); one thread of the even CTA issues tcgen05.mma.cta_group::2 (M 256, N 256, K 16), which
// reads both CTAs' shared memory and accumulates each CTA's 128 rows in its own tensor memory. A stage is 32 KB per CTA
// instead of 48 KB for the same FLOP: a third fewer operand bytes from L2 per FLOP and six stages in flight instead of four.
// No multicast loads: each CTA requests its own tiles, and both CTAs' loads are counted on the even CTA's stage barrier
// (the pair form of the TMA load may signal a barrier of the peer), so no thread relays arrivals between the CTAs. Used for calls of kPairRows rows and more.
// A last wave with fewer tiles than half of the pairs runs them as halves of 128 columns: 5120 columns at 2048 rows are 160 tiles on
// 74 pairs, 2 waves and 12 tiles, which took a third whole wave. The segments of a trellis object share one launch for the same
// reason (query_key_value at 2048 rows: 160 + 32 + 32 tiles were 3 + 1 + 1 waves). A trellis layer of 512 / 1024 / 2048 rows, with
// its rotate and decode side by side (w = 64): 703 / 985 / 1518 -> 580 / 872 / 1426 us.
constexpr uint32_t kPairStages = 6;
constexpr uint32_t kPairStageBytes = kATile + 128u * 128u;
constexpr uint32_t kPairShared = kPairStages * kPairStageBytes + 256u + 1024u;
constexpr uint32_t kPairInstruction = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((256u >> 4) << 24);
constexpr uint32_t kPairInstructionHalf = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((256u >> 4) << 24);   // N 128
constexpr uint32_t kPairRows = 512;

__device__ __forceinline__ void pair_mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t instruction, uint32_t accumulate) {
    asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
            "l"(a_desc), "l"(b_desc), "r"(instruction), "r"(accumulate)
            : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) bf16_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a,
        const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_half, uint16_t* __restrict__ out, const uint16_t* __restrict__ svh,
        uint32_t stride, uint32_t rows, uint32_t n, uint32_t k, const __grid_constant__ Segments segments, uint32_t* __restrict__ error) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~(uintptr_t)1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kPairStages * kPairStageBytes);
    uint64_t* empty = full + kPairStages;
    uint64_t* acc_full = empty + kPairStages;    // two accumulators of 256 columns: a tile's MMAs run while the tile before is drained
    uint64_t* acc_empty = acc_full + 2;          // even CTA: both CTAs' epilogue warps have drained the accumulator
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t rank = eb::cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const uint32_t tiles_m = (rows + 255u) / 256u, tiles_n = segments.tile_begin[segments.count], tiles = tiles_m * tiles_n;
    const uint32_t k_steps = k / kStepK;
    // The tiles of a last wave that would leave more than half of the pairs idle are cut into two items of 128 columns each.
    const uint32_t rest = tiles % pairs, whole = 2u * rest <= pairs ? tiles - rest : tiles, items = whole + 2u * (tiles - whole);
    struct Place {
        uint32_t tm, segment;
        uint32_t out, end;               // first output column, end of the output columns that may be written
    };
    // Panels of kPanel tile columns; inside a panel the row index runs fastest across the panel's columns.
    auto place = [&](uint32_t item) {
        const bool cut = item >= whole;
        const uint32_t tile = cut ? whole + ((item - whole) >> 1) : item, part = cut ? (item - whole) & 1u : 0u;
        const uint32_t per_panel = tiles_m * nvfp4n::kPanel, panel = tile / per_panel, in_panel = tile - panel * per_panel;
        const uint32_t width = min(nvfp4n::kPanel, tiles_n - panel * nvfp4n::kPanel), tn = panel * nvfp4n::kPanel + in_panel % width;
        Place at;
        at.tm = in_panel / width;
        at.segment = segments.of(tn);
        at.out = segments.begin[at.segment] + (tn - segments.tile_begin[at.segment]) * 256u + part * 128u;
        at.end = segments.begin[at.segment + 1u];
        return at;
    };

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kPairStages; ++s) {
            eb::mbar_init(&full[s], 1);
            eb::mbar_init(&empty[s], 1);
        }
        for (uint32_t b = 0; b < 2u; ++b) {
            eb::mbar_init(&acc_full[b], 1);
            eb::mbar_init(&acc_empty[b], 16);
        }
        eb::mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(eb::smem_u32(tmem_holder)), "r"(kTmemColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    nvfp4n::tcgen05_fence_before();
    __syncthreads();
    eb::cluster_sync();   // both CTAs' barriers exist before anything arrives on them from the other CTA
    nvfp4n::tcgen05_fence_after();
    const uint32_t tmem = *tmem_holder;
    eb::pdl_launch_dependents();
    eb::pdl_wait();   // both operands come from the launches before this one

    if (warp < 4u) {
      nvfp4n::registers_give_back<64>();
      if (warp == 0) {
        if (lane == 0) {
            uint32_t step = 0;
            bool ok = true;
            for (uint32_t item = pair; item < items && ok; item += pairs) {
                const Place at = place(item);
                const uint32_t row = at.segment * rows + (2u * at.tm + rank) * kTileM;   // this CTA's 128 rows
                const uint32_t weight = at.out + rank * (item < whole ? 128u : 64u);     // its half of the weight rows
                const CUtensorMap* map_weights = item < whole ? &map_b : &map_half;
                const uint32_t bytes = kATile + (item < whole ? 128u : 64u) * 128u;
                for (uint32_t ks = 0; ks < k_steps; ++ks, ++step) {
                    const uint32_t s = step % kPairStages, round = step / kPairStages;
                    if (round > 0 && !eb::mbar_wait(&empty[s], (round - 1u) & 1u)) {
                        atomicOr(error, kWaitFailed);
                        ok = false;
                        break;
                    }
                    uint8_t* stage = smem + s * kPairStageBytes;
                    // both CTAs' boxes are counted on the even CTA's barrier, where the thread that issues the MMAs waits
                    if (rank == 0u) eb::mbar_arrive_expect_tx(&full[s], 2u * bytes);
                    const uint32_t bar = eb::map_to_rank(eb::smem_u32(&full[s]), 0u);
                    nvfp4n::pair_tma_load_2d(stage, &map_a, (int)(ks * kStepK), (int)row, bar);
                    nvfp4n::pair_tma_load_2d(stage + kATile, map_weights, (int)(ks * kStepK), (int)weight, bar);
                }
            }
        }
      } else if (warp == 1) {
        if (rank == 0u) {   // the odd CTA issues nothing: its tiles are read by the even CTA's MMAs
            const bool leader = eb::elect_one();   // in a loop of the whole warp: see eb::elect_one
            eb::Ring ring;
            uint32_t local = 0;
            bool ok = true;
            for (uint32_t item = pair; item < items && ok; item += pairs, ++local) {
                const uint32_t buffer = local & 1u, use = local >> 1;
                if (use > 0 && !__all_sync(0xFFFFFFFFu, eb::mbar_wait(&acc_empty[buffer], (use - 1u) & 1u))) {
                    if (lane == 0) atomicOr(error, kWaitFailed);
                    break;
                }
                nvfp4n::tcgen05_fence_after();
                const uint32_t accumulator = tmem + buffer * kTileN;
                const uint32_t instruction = item < whole ? kPairInstruction : kPairInstructionHalf;
                for (uint32_t ks = 0; ks < k_steps; ++ks) {
                    if (!__all_sync(0xFFFFFFFFu, eb::mbar_wait(&full[ring.stage], ring.parity))) {
                        if (lane == 0) atomicOr(error, kWaitFailed);
                        ok = false;
                        break;
                    }
                    nvfp4n::tcgen05_fence_after();
                    const uint8_t* stage = smem + ring.stage * kPairStageBytes;
                    const uint64_t a = nvfp4n::tile_descriptor(stage), b = nvfp4n::tile_descriptor(stage + kATile);
                    if (leader) {
#pragma unroll
                        for (uint32_t j = 0; j < 4u; ++j) pair_mma_bf16(accumulator, a + 2u * j, b + 2u * j, instruction, (uint32_t)((ks | j) != 0u));
                        nvfp4n::pair_commit(&empty[ring.stage]);
                    }
                    __syncwarp();
                    ring.advance(kPairStages);
                }
                if (ok && leader) nvfp4n::pair_commit(&acc_full[buffer]);
                __syncwarp();
            }
        }
      }
    } else {
        // Epilogue, in both CTAs, each over its own 128 rows: as in bf16_gemm_kernel.
        nvfp4n::registers_take<208>();
        const uint32_t quarter = warp & 3u, half = (warp - 4u) >> 2;
        uint32_t local = 0;
        for (uint32_t item = pair; item < items; item += pairs, ++local) {
            const bool cut = item >= whole, works = !cut || half == 0u;   // a cut item's 128 accumulator columns are one warp's
            const uint32_t buffer = local & 1u;
            if (!eb::mbar_wait(&acc_full[buffer], (local >> 1) & 1u)) {
                if (lane == 0) atomicOr(error, kWaitFailed);
                break;
            }
            nvfp4n::tcgen05_fence_after();
            uint32_t r[4][32];
            const uint32_t from = tmem + ((quarter * 32u) << 16) + buffer * kTileN + half * 128u;
            if (works) {
#pragma unroll
                for (uint32_t i = 0; i < 4u; ++i) nvfp4n::tmem_load_32(r[i], from + 32u * i);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            }
            nvfp4n::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) nvfp4n::signal_rank_relaxed(&acc_empty[buffer], 0u);   // what it orders are tensor-memory reads
            if (!works) continue;
            const Place at = place(item);
            const uint32_t row = (2u * at.tm + rank) * kTileM + quarter * 32u + lane, col = at.out + half * 128u;
            if (svh == nullptr) {
                nvfp4n::store_block(r, out, row, rows, n, col, 1.0f, false);   // row stride n
            } else if (row < rows && col < at.end) {
                store_rotated(r, out + (uint64_t)row * stride + col, svh + col);
            }
        }
    }
    nvfp4n::tcgen05_fence_before();
    __syncthreads();
    eb::cluster_sync();   // neither CTA leaves while the other may still read its shared memory or arrive on its barriers
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns) : "memory");
    }
}

inline cudaError_t initialize() {
    const cudaError_t e = cudaFuncSetAttribute(bf16_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSharedBytes);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(bf16_gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairShared);
}

// Whether calls of kPairRows rows and more run on CTA pairs (process-wide; same bits either way).
inline std::atomic<bool> g_pairs{true};

// a [rows][k], b [n][k] -> out [rows][n] at row stride `stride`, all BF16 in device memory, 16-byte aligned; k % 64 == 0,
// n % 128 == 0. svh (FP16 [n], may be null): finish the trellis output in the epilogue instead of storing the sums.
// ends: the exclusive column ends of `count` (at most
// kMaxSegments) segments, for which a is [count][rows][k]; null: one segment.
inline cudaError_t linear(const void* a, const void* b, void* out, const void* svh, uint32_t stride, uint32_t rows, uint32_t k, uint32_t n, int sms,
        cudaStream_t stream, bool pdl, uint32_t* error, const int32_t* ends = nullptr, uint32_t count = 1) {
    const eb::EncodeTiled encode = eb::encoder();
    if (encode == nullptr) return cudaErrorNotSupported;
    const bool pairs = rows >= kPairRows && g_pairs.load();
    CUtensorMap map_a, map_b, map_half;   // boxes of 128 rows, and of 64 for the cut tiles of the pair kernel
    const cuuint32_t ones[2] = {1u, 1u}, box[2] = {kStepK, 128u}, half_box[2] = {kStepK, 64u};
    const cuuint64_t a_dims[2] = {k, (cuuint64_t)rows * count}, b_dims[2] = {k, n}, strides[1] = {(cuuint64_t)k * 2u};
    auto encode_bf16 = [&](CUtensorMap* map, const void* at, const cuuint64_t* dims, const cuuint64_t* pitch, const cuuint32_t* of) {
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(at), dims, pitch, of, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                == CUDA_SUCCESS;
    };
    if (!encode_bf16(&map_a, a, a_dims, strides, box) || !encode_bf16(&map_b, b, b_dims, strides, box)
            || (pairs && !encode_bf16(&map_half, b, b_dims, strides, half_box)))
        return cudaErrorInvalidValue;
    Segments segments = {};
    segments.count = count;
    for (uint32_t g = 0; g < count; ++g) {
        segments.begin[g + 1u] = ends != nullptr ? (uint32_t)ends[g] : n;
        segments.tile_begin[g + 1u] = segments.tile_begin[g] + (segments.begin[g + 1u] - segments.begin[g] + kTileN - 1u) / kTileN;
    }
    const uint32_t tiles_n = segments.tile_begin[count];
    if (pairs) {
        const uint32_t most = (uint32_t)sms / 2u, tiles = ((rows + 255u) / 256u) * tiles_n;   // a short call's tiles are cut in two (see the kernel)
        const uint32_t ctas = 2u * std::max(1u, 2u * tiles <= most ? 2u * tiles : std::min(most, tiles));
        return nvfp4n::launch_on(stream, pdl, bf16_gemm_pair_kernel, dim3(ctas), dim3(kThreads), kPairShared, map_a, map_b, map_half,
                static_cast<uint16_t*>(out), static_cast<const uint16_t*>(svh), stride, rows, n, k, segments, error);
    }
    const uint32_t tiles = ((rows + kTileM - 1u) / kTileM) * tiles_n;
    return nvfp4n::launch_on(stream, pdl, bf16_gemm_kernel, dim3(tiles < (uint32_t)sms ? tiles : (uint32_t)sms), dim3(kThreads), kSharedBytes, map_a, map_b,
            static_cast<uint16_t*>(out), static_cast<const uint16_t*>(svh), stride, rows, n, k, segments, error);
}

}  // namespace bf16n

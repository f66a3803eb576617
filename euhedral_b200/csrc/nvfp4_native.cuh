// NVFP4 prefill GEMM on sm_100a: both operands NVFP4, tcgen05 block-scaled MMA (kind::mxf4nvf4, one UE4M3 scale per 16
// values) with the accumulator in tensor memory.
//
// Replaces the reference's native route behind euhedral_cuda_linear_nvfp4_native_bf16
// (native/src/host/nvfp4_linear.c:299-361): its activation quantizer native/src/nvfp4_native/native.cuh:105-168 and its
// 128x128 warp-MMA tile native/src/nvfp4_native/native.cuh:265-432. Same arithmetic contract: each BF16 activation row
// becomes two NVFP4 terms (the value and the quantized residual) under one FP32 scale per row; per output the K steps
// run in increasing order with one MMA per term into the same FP32 accumulator; the result is
// bf16(acc * row scale * tensor scale).
//
// Two launches per call, all on the selected stream, no allocation (everything lives in the caller's scratch):
//   1. quantize_rows: BF16 rows -> code planes [term][row][K/2], block scales already in the layout tcgen05 wants
//      (512-byte atoms of 128 rows x 4 scales, byte (r % 32) * 16 + (r / 32) * 4 + s), one FP32 scale per row. One CTA
//      per row.
//   2. gemm: persistent CTAs, one per SM, 128 x 256 output tiles, K in steps of 256 through a 3-stage ring.
//      warp 0 (one lane) issues the TMA loads (codes as 128-byte-swizzled tiles, the weights' scale bytes as they lie in the
//      tensor, the activations' scale atoms as bulk copies), warps 4..7 move the stage's scales from shared memory through
//      registers into tensor memory (tcgen05.st), warp 1 (one lane) issues the MMAs (M 128, N 256, K 64; two terms x four K
//      blocks per stage) and commits to the ring's and the accumulator's mbarriers, warps 8..15 drain the accumulator into
//      registers (tcgen05.ld), hand it back at once, then scale, round and store BF16 while the next tile's MMAs already run.
//      Calls of kPairRows rows and more run the same on CTA pairs (gemm_pair_kernel).
// What bounds it: the tensor pipe under the power cap. Copying the scales with tcgen05.cp, as this kernel did before, queues in
// order with the MMAs (16 copies of about 37 cycles beside 8 MMAs of 135 per stage) and wants the weights' scales re-laid-out by
// a launch of its own; the registers' way runs beside the MMAs and reads the tensor's plane. What then limited the single-CTA
// kernel was the epilogue's 16-byte stores (every sector written in halves) and shared-memory bandwidth (12 KB read per MMA
// and 9 KB filled per 135 cycles at 128 bytes a cycle; the pairs read 8 and fill 7). 4096 x 17408 x 5120, activations quantized
// before, back to back under the power cap: 245 to 276 us on pairs, 261 to 299 on single CTAs (the clock moves between runs).
// Tiles are walked in panels of eight tile columns with the row index fastest, so that CTAs running together share
// weight tiles and re-read activation tiles from L2. Every CTA issues its own loads.
#pragma once

#include <cuda.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>

#include <algorithm>

#include "common.cuh"

namespace nvfp4d {   // nvfp4_decode.cuh: the kernel that takes few rows
inline cudaError_t quantized(const void* weights, void* output, const CUtensorMap& activations, const uint8_t* atoms, const float* row_globals, uint32_t rows,
        uint32_t k, uint32_t out_features, bool paired, bool table, int sms, cudaStream_t stream, bool pdl, uint32_t* error);
inline bool better_for(uint32_t rows, uint32_t k, uint32_t out_features, bool paired, uint32_t sms);
inline uint32_t columns_of(uint32_t rows);
}  // namespace nvfp4d

namespace nvfp4n {

constexpr uint32_t kTerms = 2;
constexpr uint32_t kTileM = 128, kTileN = 256, kStepK = 256, kBlockK = 64;
constexpr uint32_t kStages = 3;
constexpr uint32_t kATile = kTileM * 128u;                 // one term's codes of a stage: 128 rows x 128 bytes
constexpr uint32_t kBTile = kTileN * 128u;
constexpr uint32_t kAtom = 512u;                           // 128 rows x 4 scales
constexpr uint32_t kSfaStage = (kStepK / kBlockK) * kTerms * kAtom;
constexpr uint32_t kSfbStage = (kStepK / kBlockK) * (kTileN / 128u) * kAtom;
constexpr uint32_t kStageBytes = kTerms * kATile + kBTile + kSfaStage + kSfbStage;
constexpr uint32_t kBarrierBytes = 128u;
constexpr uint32_t kSharedBytes = kStages * kStageBytes + kBarrierBytes + 1024u;   // + slack to align to 1024
constexpr uint32_t kScaledThreads = 512u;                   // TMA and MMA warps (and two that idle), four scale warps, eight epilogue warps
constexpr uint32_t kTmemColumns = 512u;
constexpr uint32_t kTmemScales = 256u, kScaleColumns = 64u; // behind the 256 accumulator columns: 64 columns of scales per ring stage
constexpr uint32_t kPanel = 8u;                            // tile columns per panel of the tile walk

__host__ __device__ inline uint64_t align256(uint64_t v) { return (v + 255ull) & ~255ull; }

// Caller scratch of one native linear.
struct ActivationLayout {
    uint64_t sfa_offset, global_offset, sfb_offset, bytes;
    uint32_t row_tiles, k_blocks;
    __host__ __device__ ActivationLayout(uint32_t rows, uint32_t k, uint32_t out_features = 0) {
        const uint64_t kp = ((uint64_t)k + 127u) / 128u * 128u;
        row_tiles = (rows + kTileM - 1u) / kTileM;
        k_blocks = (uint32_t)(kp / kBlockK);
        sfa_offset = align256((uint64_t)kTerms * rows * (kp / 2u));
        global_offset = align256(sfa_offset + (uint64_t)row_tiles * k_blocks * kTerms * kAtom);
        sfb_offset = align256(global_offset + 4ull * rows);
        const uint64_t n128 = ((uint64_t)out_features + 255u) / 256u * 2u;
        bytes = align256(sfb_offset + n128 * k_blocks * kAtom);
    }
};

__host__ __device__ inline uint32_t atom_byte(uint32_t row_in_tile, uint32_t scale) {
    return (row_in_tile & 31u) * 16u + (row_in_tile >> 5) * 4u + scale;
}

// ---- 1. activation quantizer -----------------------------------------------------------------------------------------
// The arithmetic is the reference's, operation for operation (native/src/nvfp4_native/native.cuh:105-127, pinned bit for
// bit against that kernel compiled for this GPU): global = amax / (6 * 448) (1 for a zero row); per block of 16:
// scale = e4m3_satfinite(amax * (1/6) * (1/global)); codes = e2m1_rn(v * ((1/global) / scale)), saturating; the next term
// quantizes fma(-decoded, scale * global, v). All in FP32 with the hardware conversions.
// The work split is this kernel's own: one CTA per row, a 16-value block per thread and turn, held in registers from the pass
// that finds the row's largest magnitude to the pass that quantizes it (kHeld turns; what a longer row has beyond is read again).
// Four neighbouring lanes share a K block of 64 values; their four scale bytes meet by two shuffles
// and leave as ONE 4-byte store, which is exactly one row's entry of the 512-byte atom tcgen05 reads; their codes leave as 32
// contiguous bytes per term. A warp per row, which this replaces, read every row twice and left all but a few SMs idle on
// calls of few rows.
// Bound: no single pipe was profiled; fewer instructions and more rows resident on an SM both measured faster; spilled registers, a CTA that walks several rows and
// loads a row ahead all measured slower. Alone, us at 512 / 4096 / 32768 rows, warp per row -> now: 5120 values 8.2 / 20.6 / 113 -> 4.6 /
// 15.7 / 119; 17,408 values 25.2 / 86.3 / 473 -> 8.8 / 57.7 / 429; 25,600 values (partly read twice) 36.2 / 123 / 698 -> 13.2 / 97.9 / 731.
__host__ __device__ constexpr uint32_t quantize_threads(uint32_t held) { return held == 2u ? 512u : 384u; }   // the most of a row: two CTAs per SM without spills

// One block of 16 values with its largest magnitude: its scale code, its 8 code bytes, and v replaced by the residual.
__device__ __forceinline__ uint32_t quantize_block(float (&v)[16], float block_max, float global, float inverse_global, uint2* codes) {
    const __nv_fp8_storage_t scale = __nv_cvt_float_to_fp8(__fmul_rn(__fmul_rn(block_max, 1.0f / 6.0f), inverse_global), __NV_SATFINITE, __NV_E4M3);
    const float decoded = __half2float(__half(__nv_cvt_fp8_to_halfraw(scale, __NV_E4M3)));
    const float inverse = decoded > 0.0f ? __fdiv_rn(inverse_global, decoded) : 0.0f;
    const float step = __fmul_rn(decoded, global);
    uint32_t packed[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const __nv_fp4x2_storage_t pair = __nv_cvt_float2_to_fp4x2(
                make_float2(__fmul_rn(v[2 * i], inverse), __fmul_rn(v[2 * i + 1], inverse)), __NV_E2M1, cudaRoundNearest);
        packed[i >> 2] |= (uint32_t)pair << (8 * (i & 3));
        const __half2_raw back = __nv_cvt_fp4x2_to_halfraw2(pair, __NV_E2M1);
        const float2 q = __half22float2(*reinterpret_cast<const __half2*>(&back));
        v[2 * i] = __fmaf_rn(-q.x, step, v[2 * i]);       // the residual in one rounding, as the reference's build contracts it
        v[2 * i + 1] = __fmaf_rn(-q.y, step, v[2 * i + 1]);
    }
    *codes = make_uint2(packed[0], packed[1]);
    return (uint32_t)scale;
}

// Largest magnitude of 16 BF16 values, two at a time (a NaN loses against any number, as with fmaxf).
__device__ __forceinline__ float largest_of(const uint4& lo, const uint4& hi) {
    const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    __nv_bfloat162 most = __float2bfloat162_rn(0.0f);
#pragma unroll
    for (int j = 0; j < 8; ++j) most = __hmax2(most, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[j])));
    return fmaxf(__low2float(most), __high2float(most));
}

//   grid rows, block: the fewest whole warps that hold the row in kHeld turns, at most quantize_threads. k a multiple of 64.
template <uint32_t kHeld>
__global__ void __launch_bounds__(quantize_threads(kHeld), 2) quantize_rows(const __nv_bfloat16* __restrict__ input, uint8_t* __restrict__ scratch,
        uint32_t rows, uint32_t k) {
    const uint32_t t = threadIdx.x, threads = blockDim.x, row = blockIdx.x;
    __shared__ float warp_most[quantize_threads(kHeld) / 32u];
    const ActivationLayout layout(rows, k);
    eb::pdl_launch_dependents();
    eb::pdl_wait();
    const uint4* x = reinterpret_cast<const uint4*>(input + (uint64_t)row * k);   // 8 values per element
    const uint32_t blocks = k / 16u;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 lo[kHeld], hi[kHeld];
#pragma unroll
    for (uint32_t i = 0; i < kHeld; ++i) {
        const uint32_t b = i * threads + t;
        lo[i] = b < blocks ? x[2u * b] : zero;
        hi[i] = b < blocks ? x[2u * b + 1u] : zero;
    }
    float amax = 0.0f, block_max[kHeld];
#pragma unroll
    for (uint32_t i = 0; i < kHeld; ++i) amax = fmaxf(amax, block_max[i] = largest_of(lo[i], hi[i]));
    for (uint32_t b = kHeld * threads + t; b < blocks; b += threads) amax = fmaxf(amax, largest_of(x[2u * b], x[2u * b + 1u]));
    // magnitudes are non-negative floats, whose bits order as integers
    const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
    if ((t & 31u) == 0u) warp_most[t >> 5] = __uint_as_float(most);
    __syncthreads();
    amax = 0.0f;
    for (uint32_t w = 0; w < threads / 32u; ++w) amax = fmaxf(amax, warp_most[w]);
    const float global = amax > 0.0f ? __fdiv_rn(amax, 6.0f * 448.0f) : 1.0f;
    const float inverse_global = __fdiv_rn(1.0f, global);
    uint8_t* sfa = scratch + layout.sfa_offset + (uint64_t)(row / kTileM) * layout.k_blocks * kTerms * kAtom + atom_byte(row % kTileM, 0);
    const uint64_t plane = (uint64_t)rows * (k / 2u);
    uint8_t* codes_row = scratch + (uint64_t)row * (k / 2u);
    auto quantize = [&](uint32_t b, const uint4& first, const uint4& second, float most_of_block) {   // whole quartets of lanes come here together
        const uint32_t words[8] = {first.x, first.y, first.z, first.w, second.x, second.y, second.z, second.w};
        const uint32_t sub = b & 3u, members = 0xFu << (t & 28u);
        float v[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[2 * i] = eb::bf16_bits_to_float(words[i] & 0xFFFFu);
            v[2 * i + 1] = __uint_as_float(words[i] & 0xFFFF0000u);
        }
#pragma unroll
        for (uint32_t term = 0; term < kTerms; ++term) {
            uint2 codes;
            if (term != 0u) {
                most_of_block = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; ++i) most_of_block = fmaxf(most_of_block, fabsf(v[i]));
            }
            uint32_t scales = quantize_block(v, most_of_block, global, inverse_global, &codes) << (8u * sub);
            scales |= __shfl_xor_sync(members, scales, 1);   // the K block's four scale bytes, in every one of the four lanes
            scales |= __shfl_xor_sync(members, scales, 2);
            *reinterpret_cast<uint2*>(codes_row + term * plane + 8u * b) = codes;
            if (sub == 0u) *reinterpret_cast<uint32_t*>(sfa + ((uint64_t)(b >> 2) * kTerms + term) * kAtom) = scales;
        }
    };
#pragma unroll
    for (uint32_t i = 0; i < kHeld; ++i)
        if (i * threads + t < blocks) quantize(i * threads + t, lo[i], hi[i], block_max[i]);
    for (uint32_t b = kHeld * threads + t; b < blocks; b += threads) {
        const uint4 first = x[2u * b], second = x[2u * b + 1u];
        quantize(b, first, second, largest_of(first, second));
    }
    if (t == 0u) reinterpret_cast<float*>(scratch + layout.global_offset)[row] = global;
}

// ---- 2. table-indexed weight scales ---------------------------------------------------------------------------------------
// Layout row-split-k128-sd4-v1 only: 4-bit indices, two per byte with the even block in the low nibble, into the tensor's 16
// E4M3 codes at `table` -> the scale bytes [n][K/16] a plain tensor has, so that the GEMM is the same for both layouts. A
// thread writes 16 bytes. grid ceil(n * K / 256 / 256).
__global__ void __launch_bounds__(256) expand_table_scales(const uint8_t* __restrict__ indices, const uint8_t* __restrict__ table,
        uint8_t* __restrict__ scales, uint32_t count) {
    const uint32_t index = blockIdx.x * 256u + threadIdx.x;
    eb::pdl_launch_dependents();
    eb::pdl_wait();   // the GEMM of the call before this one may still be reading these bytes
    if (index >= count) return;
    const uint4 t = *reinterpret_cast<const uint4*>(table);
    const uint2 pairs = reinterpret_cast<const uint2*>(indices)[index];
    uint32_t words[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t four = ((i & 2) ? pairs.y : pairs.x) >> (16 * (i & 1));   // four indices; the upper half is ignored
        const uint32_t within = four & 0x7777u;
        const uint32_t low = __byte_perm(t.x, t.y, within), high = __byte_perm(t.z, t.w, within);
        const uint32_t upper = __byte_perm(0u, 0xFFFFFFFFu, (four >> 1) & 0x4444u);   // a byte of ones where the index is 8 or more
        words[i] = eb::lop3<eb::kLutSelect>(high, low, upper);
    }
    reinterpret_cast<uint4*>(scales)[index] = make_uint4(words[0], words[1], words[2], words[3]);
}

// ---- 3. the GEMM ----------------------------------------------------------------------------------------------------------

using eb::tma_load_2d;
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                         eb::smem_u32(dst)),
            "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(eb::smem_u32(bar))
            : "memory");
}

// Shared-memory matrix descriptor of a K-major tile with 128-byte rows under the 128-byte swizzle: 8-row groups are
// 1024 bytes apart, descriptor version 1 (sm_100), layout type 2.
__device__ __forceinline__ uint64_t tile_descriptor(const void* smem_tile) {
    uint64_t d = 0;
    d |= (uint64_t)((eb::smem_u32(smem_tile) & 0x3FFFFu) >> 4);
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// kind::mxf4nvf4 instruction descriptor: E2M1 x E2M1, UE4M3 scales, both operands K-major, M 128, N 256.
constexpr uint32_t kInstruction = (1u << 7) | (1u << 10) | ((kTileN >> 3) << 17) | (0u << 23) | ((kTileM >> 4) << 24);

__device__ __forceinline__ void mma_block_scaled(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t sfa_tmem, uint32_t sfb_tmem,
        uint32_t accumulate) {
    asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %6, 0;\n"
            "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%4], [%5], p;\n}" ::"r"(d_tmem),
            "l"(a_desc), "l"(b_desc), "r"(kInstruction), "r"(sfa_tmem), "r"(sfb_tmem), "r"(accumulate)
            : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(eb::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive accumulator columns of the calling warp's 32 lanes (one row per thread) into registers.
__device__ __forceinline__ void tmem_load_32(uint32_t (&r)[32], uint32_t address) {
    asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
            "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
              "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
              "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
              "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(address));
}

// 32 consecutive 32-bit columns of the calling warp's 32 lanes from registers into tensor memory.
__device__ __forceinline__ void tmem_store_32(uint32_t address, const uint32_t (&r)[32]) {
    asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
            "%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(address),
            "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
            "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
            "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
            : "memory");
}
// Register limit of the calling warpgroup (all of its four warps execute it). The kernels' splits stay within the launch's registers.
template <int COUNT>
__device__ __forceinline__ void registers_give_back() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(COUNT)); }
template <int COUNT>
__device__ __forceinline__ void registers_take() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(COUNT)); }

// 16 BF16 values (eight registers) to global memory. A thread's 32 bytes lie in a row of their own, so one 32-byte store per
// thread writes whole sectors where two of 16 bytes would write each sector in halves. `wide`: dst is 32-byte aligned.
__device__ __forceinline__ void store_16(uint16_t* dst, const uint32_t (&v)[8], bool wide) {
    if (wide) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
                "r"(v[5]), "r"(v[6]), "r"(v[7])
                : "memory");
    } else {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    }
}

// A thread's row of an epilogue block, scaled, rounded to BF16 and stored 32 bytes at a time from column col0 (n and col0 are
// multiples of 64, out is 16-byte aligned).
// plain: r holds 4 x 32 consecutive columns. paired (the gate/up region): r[0], r[1] are 64 gate columns, r[2], r[3] the 64
// up columns that match them; out[row][col] = bf16(silu(gate) * up) with gate and up rounded to BF16 first (the reference's
// region, native/src/nvfp4_native/native.cuh:390-413: the same expression, expf and division).
__device__ __forceinline__ void store_block(const uint32_t (&r)[4][32], uint16_t* __restrict__ out, uint32_t row, uint32_t rows, uint32_t n,
        uint32_t col0, float scale, bool paired) {
    if (row >= rows) return;
    const bool wide = (reinterpret_cast<uintptr_t>(out) & 31u) == 0;
#pragma unroll
    for (uint32_t cb = 0; cb < 4u; ++cb) {
        if (paired && cb >= 2u) break;
        const uint32_t col = col0 + cb * 32u;
        if (col >= n) continue;
        uint16_t* dst = out + (uint64_t)row * n + col;
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            uint32_t packed[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float value[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = 16 * v + 2 * i + e;
                    const float first = __fmul_rn(__uint_as_float(r[cb][c]), scale);
                    if (paired) {
                        const float gate = eb::bf16_bits_to_float(eb::float_to_bf16_bits(first));
                        const float up = eb::bf16_bits_to_float(eb::float_to_bf16_bits(__fmul_rn(__uint_as_float(r[(cb + 2u) & 3u][c]), scale)));
                        value[e] = __fmul_rn(__fdiv_rn(gate, __fadd_rn(1.0f, expf(-gate))), up);
                    } else {
                        value[e] = first;
                    }
                }
                packed[i] = eb::bf16_pair(value[0], value[1]);
            }
            store_16(dst + 16 * v, packed, wide);
        }
    }
}

// One scale warp, one stage: the stage's scales from shared memory into the warp's quarter of tensor memory (every quarter
// holds all of them). `sf`: this lane's 16 bytes of the first atom; `to`: the stage's columns in the warp's quarter.
// Columns 8 j + 4 t + i: the four scales of K block j, term t, of activation row 32 i + lane (the atom's 16 bytes of this
// lane). Columns 32 + 8 j + i: of weight row 32 i + lane of the tile's 256 (word j of that row's 16 scale bytes).
__device__ __forceinline__ void scales_to_tmem(const uint4* sf, uint32_t to) {
    uint32_t a[32], b[32];
#pragma unroll
    for (uint32_t i = 0; i < 8u; ++i) {
        const uint4 v = sf[i * 32u], w = sf[kSfaStage / 16u + i * 32u];
        a[4 * i] = v.x, a[4 * i + 1] = v.y, a[4 * i + 2] = v.z, a[4 * i + 3] = v.w;
        b[i] = w.x, b[8 + i] = w.y, b[16 + i] = w.z, b[24 + i] = w.w;
    }
    tmem_store_32(to, a);
    tmem_store_32(to + 32u, b);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tcgen05_fence_before();
    __syncwarp();
}

struct TileWalk {
    uint32_t tiles_m, tiles_n, total;
    __device__ TileWalk(uint32_t rows, uint32_t tile_columns) : tiles_m((rows + kTileM - 1u) / kTileM), tiles_n(tile_columns) { total = tiles_m * tiles_n; }
    // Panels of kPanel tile columns; inside a panel the row index runs fastest across the panel's columns.
    __device__ void at(uint32_t tile, uint32_t* tm, uint32_t* tn) const {
        const uint32_t per_panel = tiles_m * kPanel;
        const uint32_t panel = tile / per_panel, rest = tile - panel * per_panel;
        const uint32_t width = min(kPanel, tiles_n - panel * kPanel);
        *tm = rest / width;
        *tn = panel * kPanel + rest % width;
    }
};

__global__ void __launch_bounds__(kScaledThreads, 1) gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
        const __grid_constant__ CUtensorMap map_s, const uint8_t* __restrict__ sfa, const float* __restrict__ row_globals,
        const float* __restrict__ tensor_global, uint16_t* __restrict__ out, uint32_t rows, uint32_t n, uint32_t k,
        uint32_t pair_tiles, uint32_t* __restrict__ error) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~(uintptr_t)1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
    uint64_t* empty = full + kStages;
    uint64_t* scaled = empty + kStages;      // the stage's scales are in tensor memory
    uint64_t* acc_full = scaled + kStages;
    uint64_t* acc_empty = acc_full + 1;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 1);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    // pair_tiles != 0: the gate/up region. `n` is the output width (half of the weight rows); an output tile of 128 columns
    // takes the 128 gate rows at its own place and the 128 up rows pair_tiles * 128 further down as the halves of its B tile.
    const bool paired = pair_tiles != 0u;
    const TileWalk walk(rows, paired ? n / 128u : (n + kTileN - 1u) / kTileN);
    const uint32_t k_steps = k / kStepK, k_blocks = k / kBlockK;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            eb::mbar_init(&full[s], 1);
            eb::mbar_init(&empty[s], 1);
            eb::mbar_init(&scaled[s], 4);
        }
        eb::mbar_init(acc_full, 1);
        eb::mbar_init(acc_empty, 8);
        eb::mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(eb::smem_u32(tmem_holder)), "r"(kTmemColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = *tmem_holder;
    eb::pdl_launch_dependents();
    eb::pdl_wait();   // the scratch comes from the launches before this one

    if (warp < 4u) {
      registers_give_back<56>();
      if (warp == 0) {
        if (lane == 0) {
            uint32_t step = 0;
            bool ok = true;
            for (uint32_t item = blockIdx.x; item < walk.total && ok; item += gridDim.x) {
                uint32_t tm, tn;
                walk.at(item, &tm, &tn);
                for (uint32_t ks = 0; ks < k_steps; ++ks, ++step) {
                    const uint32_t s = step % kStages, round = step / kStages;
                    if (round > 0 && !eb::mbar_wait(&empty[s], (round - 1u) & 1u)) {
                        atomicOr(error, 8u);
                        ok = false;
                        break;
                    }
                    uint8_t* stage = smem + s * kStageBytes;
                    eb::mbar_arrive_expect_tx(&full[s], kStageBytes);
                    tma_load_3d(stage, &map_a, (int)(ks * 128u), (int)(tm * kTileM), 0, &full[s]);
                    tma_load_3d(stage + kATile, &map_a, (int)(ks * 128u), (int)(tm * kTileM), 1, &full[s]);
                    // the B tile's two halves of 128 weight rows, as 128-row tiles of the weight matrix
                    const uint32_t low = paired ? tn : 2u * tn, high = paired ? pair_tiles + tn : 2u * tn + 1u;
                    tma_load_2d(stage + kTerms * kATile, &map_b, (int)(ks * 128u), (int)(low * 128u), &full[s]);
                    tma_load_2d(stage + kTerms * kATile + kBTile / 2u, &map_b, (int)(ks * 128u), (int)(high * 128u), &full[s]);
                    uint8_t* sf = stage + kTerms * kATile + kBTile;
                    eb::bulk_g2s(sf, sfa + ((uint64_t)tm * k_blocks + ks * 4u) * kTerms * kAtom, kSfaStage, &full[s]);
                    tma_load_2d(sf + kSfaStage, &map_s, (int)(ks * 16u), (int)(low * 128u), &full[s]);
                    tma_load_2d(sf + kSfaStage + kSfbStage / 2u, &map_s, (int)(ks * 16u), (int)(high * 128u), &full[s]);
                }
            }
        }
      } else if (warp == 1) {
        {
            const bool leader = eb::elect_one();   // in a loop of the whole warp: see eb::elect_one
            eb::Ring ring;
            uint32_t local = 0;
            bool ok = true;
            for (uint32_t item = blockIdx.x; item < walk.total && ok; item += gridDim.x, ++local) {
                if (local > 0 && !__all_sync(0xFFFFFFFFu, eb::mbar_wait(acc_empty, (local - 1u) & 1u))) {
                    if (lane == 0) atomicOr(error, 8u);
                    break;
                }
                tcgen05_fence_after();
                for (uint32_t ks = 0; ks < k_steps; ++ks) {
                    const uint32_t s = ring.stage;
                    if (!__all_sync(0xFFFFFFFFu, eb::mbar_wait(&full[s], ring.parity) && eb::mbar_wait(&scaled[s], ring.parity))) {
                        if (lane == 0) atomicOr(error, 8u);
                        ok = false;
                        break;
                    }
                    tcgen05_fence_after();
                    const uint8_t* stage = smem + s * kStageBytes;
                    const uint64_t a0 = tile_descriptor(stage), a1 = tile_descriptor(stage + kATile), b = tile_descriptor(stage + kTerms * kATile);
                    const uint32_t scales = tmem + kTmemScales + s * kScaleColumns;
                    if (leader) {
#pragma unroll
                        for (uint32_t j = 0; j < 4u; ++j) {
                            mma_block_scaled(tmem, a0 + 2u * j, b + 2u * j, scales + j * 8u, scales + 32u + j * 8u, (uint32_t)((ks | j) != 0u));
                            mma_block_scaled(tmem, a1 + 2u * j, b + 2u * j, scales + j * 8u + 4u, scales + 32u + j * 8u, 1u);
                        }
                        mma_commit(&empty[s]);
                    }
                    __syncwarp();
                    ring.advance(kStages);
                }
                if (ok && leader) mma_commit(acc_full);
                __syncwarp();
            }
        }
      }
    } else if (warp < 8u) {
        registers_give_back<96>();
        uint32_t step = 0;
        bool ok = true;
        for (uint32_t item = blockIdx.x; item < walk.total && ok; item += gridDim.x) {
            for (uint32_t ks = 0; ks < k_steps; ++ks, ++step) {
                const uint32_t s = step % kStages, round = step / kStages;
                if (!eb::mbar_wait(&full[s], round & 1u)) {
                    if (lane == 0) atomicOr(error, 8u);
                    ok = false;
                    break;
                }
                scales_to_tmem(reinterpret_cast<const uint4*>(smem + s * kStageBytes + kTerms * kATile + kBTile) + lane,
                        tmem + (((warp & 3u) * 32u) << 16) + kTmemScales + s * kScaleColumns);
                if (lane == 0) eb::mbar_arrive(&scaled[s]);
            }
        }
    } else {
        // Epilogue: warp w may read the 32 accumulator rows of lane quarter w % 4 only; warps 8..11 take columns 0..127 of
        // their quarter, warps 12..15 columns 128..255. A warp first drains its 32 x 128 block into registers and hands the
        // accumulator back (the MMA warp starts the next tile while this one is scaled, rounded and stored).
        registers_take<176>();
        const uint32_t quarter = warp & 3u, half = (warp - 8u) >> 2;
        const float scale_w = *tensor_global;
        uint32_t local = 0;
        for (uint32_t item = blockIdx.x; item < walk.total; item += gridDim.x, ++local) {
            uint32_t tm, tn;
            walk.at(item, &tm, &tn);
            if (!eb::mbar_wait(acc_full, local & 1u)) {
                if (lane == 0) atomicOr(error, 8u);
                break;
            }
            tcgen05_fence_after();
            uint32_t r[4][32];
            // plain: 128 consecutive columns; paired: 64 gate columns (r[0], r[1]) and the 64 up columns that match them (r[2], r[3])
            const uint32_t from = tmem + ((quarter * 32u) << 16) + (paired ? half * 64u : half * 128u);
            const uint32_t other = paired ? from + 128u : from + 64u;
            tmem_load_32(r[0], from);
            tmem_load_32(r[1], from + 32u);
            tmem_load_32(r[2], other);
            tmem_load_32(r[3], other + 32u);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) eb::mbar_arrive(acc_empty);
            const uint32_t row = tm * kTileM + quarter * 32u + lane;
            const float scale = row < rows ? __fmul_rn(row_globals[row], scale_w) : 0.0f;
            store_block(r, out, row, rows, n, paired ? tn * 128u + half * 64u : tn * kTileN + half * 128u, scale, paired);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns) : "memory");
    }
}

// ---- the same GEMM on CTA pairs -----------------------------------------------------------------------------------------
// Two CTAs of a cluster share an output tile of 256 rows x 256 columns: each holds its own 128 activation rows (both
// terms) and HALF of the weight tile (128 weight rows), and one thread of the even CTA issues tcgen05.mma.cta_group::2
// (M 256, N 256, K 64), which reads both CTAs' shared memory and accumulates each CTA's 128 rows in its own tensor
// memory. A stage is 56 KB per CTA instead of 72 KB for the same FLOP, so four stages fit and the ring carries 22 % fewer
// bytes per MMA. Every CTA issues its own loads into its own shared memory (no multicast); both CTAs' code tiles are counted
// on the even CTA's stage barrier, where the thread that issues the MMAs waits, and each CTA's scale warps - its own 128
// activation rows, all 256 weight rows of the tile - wait for their own CTA's scales and arrive on the even CTA's barrier.
constexpr uint32_t kPairStages = 4;
constexpr uint32_t kPairBTile = 128u * 128u;
constexpr uint32_t kPairCodes = kTerms * kATile + kPairBTile;
constexpr uint32_t kPairStageBytes = kPairCodes + kSfaStage + kSfbStage;
constexpr uint32_t kPairShared = kPairStages * kPairStageBytes + 256u + 1024u;
constexpr uint32_t kPairInstruction = (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | (0u << 23) | ((256u >> 4) << 24);

// Tiled TMA loads of a CTA of a pair whose completion is counted on a barrier of either CTA of the pair (`bar`: a
// shared::cluster address). No multicast: the box lands in the executing CTA's shared memory only.
__device__ __forceinline__ void pair_tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                         eb::smem_u32(dst)),
            "l"(map), "r"(c0), "r"(c1), "r"(bar)
            : "memory");
}
__device__ __forceinline__ void pair_tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                         eb::smem_u32(dst)),
            "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
            : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
    asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %6, 0;\n"
            "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%4], [%5], p;\n}" ::"r"(d_tmem),
            "l"(a_desc), "l"(b_desc), "r"(kPairInstruction), "r"(sfa_tmem), "r"(sfb_tmem), "r"(accumulate)
            : "memory");
}
// Arrives (once the MMAs issued so far are done) on the barrier at this shared address in both CTAs of the pair.
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(eb::smem_u32(bar)),
            "h"((uint16_t)3)
            : "memory");
}
// Arrives on the barrier at this shared address in CTA `rank`; what the thread (and those it has synchronized with) read and wrote
// before is ordered before what follows a wait for it (eb::mbar_wait_cluster_or_fail).
__device__ __forceinline__ void signal_rank(uint64_t* bar, uint32_t rank) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(eb::map_to_rank(eb::smem_u32(bar), rank)) : "memory");
}
// The same without a release of ordinary memory, for the barriers `scaled` and `acc_empty` only: what they signal are completed
// tensor-memory operations of the thread, which tcgen05.fence::before_thread_sync has ordered. (An arrive with release waits for the
// global stores that the epilogue's threads have in flight, about a microsecond: 420 us instead of 315 us for the GEMM of 4096 x
// 17408 x 5120.)
__device__ __forceinline__ void signal_rank_relaxed(uint64_t* bar, uint32_t rank) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(eb::map_to_rank(eb::smem_u32(bar), rank)) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kScaledThreads, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a,
        const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_s, const uint8_t* __restrict__ sfa,
        const float* __restrict__ row_globals, const float* __restrict__ tensor_global, uint16_t* __restrict__ out, uint32_t rows, uint32_t n,
        uint32_t k, uint32_t pair_tiles, uint32_t* __restrict__ error) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~(uintptr_t)1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kPairStages * kPairStageBytes);   // even CTA: both CTAs' codes have landed
    uint64_t* landed = full + kPairStages;       // this CTA's scales have landed
    uint64_t* empty = landed + kPairStages;
    uint64_t* scaled = empty + kPairStages;      // even CTA: both CTAs' scales are in tensor memory
    uint64_t* acc_full = scaled + kPairStages;
    uint64_t* acc_empty = acc_full + 1;          // even CTA: both CTAs' epilogue warps have drained the accumulator
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 1);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t rank = eb::cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    // pair_tiles != 0: the gate/up region; the even CTA's half of the weight tile is the gate rows, the odd CTA's the up rows.
    const bool paired = pair_tiles != 0u;
    const uint32_t tiles_m = (rows + 255u) / 256u, tiles_n = paired ? pair_tiles : (n + 255u) / 256u, items = tiles_m * tiles_n;
    const uint32_t row_tiles = (rows + kTileM - 1u) / kTileM;
    const uint32_t k_steps = k / kStepK, k_blocks = k / kBlockK;
    // Panels of kPanel tile columns; inside a panel the row index runs fastest across the panel's columns.
    auto place = [&](uint32_t item, uint32_t* tm, uint32_t* tn) {
        const uint32_t per_panel = tiles_m * kPanel, panel = item / per_panel, rest = item - panel * per_panel;
        const uint32_t width = min(kPanel, tiles_n - panel * kPanel);
        *tm = rest / width;
        *tn = panel * kPanel + rest % width;
    };

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kPairStages; ++s) {
            eb::mbar_init(&full[s], 1);
            eb::mbar_init(&landed[s], 1);
            eb::mbar_init(&empty[s], 1);
            eb::mbar_init(&scaled[s], 8);
        }
        eb::mbar_init(acc_full, 1);
        eb::mbar_init(acc_empty, 16);
        eb::mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(eb::smem_u32(tmem_holder)), "r"(kTmemColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    eb::cluster_sync();   // both CTAs' barriers exist before anything arrives on them from the other CTA
    tcgen05_fence_after();
    const uint32_t tmem = *tmem_holder;
    eb::pdl_launch_dependents();
    eb::pdl_wait();   // the scratch comes from the launches before this one

    if (warp < 4u) {
      registers_give_back<56>();
      if (warp == 0) {
        if (lane == 0) {
            uint32_t step = 0;
            bool ok = true;
            for (uint32_t item = pair; item < items && ok; item += pairs) {
                uint32_t tm, tn;
                place(item, &tm, &tn);
                const uint32_t row_tile = 2u * tm + rank;                      // this CTA's 128 rows
                const uint32_t low = paired ? tn : 2u * tn, high = paired ? pair_tiles + tn : 2u * tn + 1u;
                const uint32_t weight_tile = rank == 0u ? low : high;          // its 128 weight rows
                const uint32_t scale_tile = min(row_tile, row_tiles - 1u);     // a CTA without rows multiplies zeros by some tile's scales
                for (uint32_t ks = 0; ks < k_steps; ++ks, ++step) {
                    const uint32_t s = step % kPairStages, round = step / kPairStages;
                    if (round > 0 && !eb::mbar_wait(&empty[s], (round - 1u) & 1u)) {
                        atomicOr(error, 8u);
                        ok = false;
                        break;
                    }
                    uint8_t* stage = smem + s * kPairStageBytes;
                    if (rank == 0u) eb::mbar_arrive_expect_tx(&full[s], 2u * kPairCodes);
                    const uint32_t bar = eb::map_to_rank(eb::smem_u32(&full[s]), 0u);
                    eb::mbar_arrive_expect_tx(&landed[s], kSfaStage + kSfbStage);
                    uint8_t* sf = stage + kPairCodes;
                    eb::bulk_g2s(sf, sfa + ((uint64_t)scale_tile * k_blocks + ks * 4u) * kTerms * kAtom, kSfaStage, &landed[s]);
                    tma_load_2d(sf + kSfaStage, &map_s, (int)(ks * 16u), (int)(low * 128u), &landed[s]);
                    tma_load_2d(sf + kSfaStage + kSfbStage / 2u, &map_s, (int)(ks * 16u), (int)(high * 128u), &landed[s]);
                    pair_tma_load_3d(stage, &map_a, (int)(ks * 128u), (int)(row_tile * kTileM), 0, bar);
                    pair_tma_load_3d(stage + kATile, &map_a, (int)(ks * 128u), (int)(row_tile * kTileM), 1, bar);
                    pair_tma_load_2d(stage + kTerms * kATile, &map_b, (int)(ks * 128u), (int)(weight_tile * 128u), bar);
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
                if (local > 0 && !__all_sync(0xFFFFFFFFu, eb::mbar_wait(acc_empty, (local - 1u) & 1u))) {
                    if (lane == 0) atomicOr(error, 8u);
                    break;
                }
                tcgen05_fence_after();
                for (uint32_t ks = 0; ks < k_steps; ++ks) {
                    const uint32_t s = ring.stage;
                    if (!__all_sync(0xFFFFFFFFu, eb::mbar_wait(&full[s], ring.parity) && eb::mbar_wait(&scaled[s], ring.parity))) {
                        if (lane == 0) atomicOr(error, 8u);
                        ok = false;
                        break;
                    }
                    tcgen05_fence_after();
                    const uint8_t* stage = smem + s * kPairStageBytes;
                    const uint64_t a0 = tile_descriptor(stage), a1 = tile_descriptor(stage + kATile), b = tile_descriptor(stage + kTerms * kATile);
                    const uint32_t scales = tmem + kTmemScales + s * kScaleColumns;
                    if (leader) {
#pragma unroll
                        for (uint32_t j = 0; j < 4u; ++j) {
                            pair_mma(tmem, a0 + 2u * j, b + 2u * j, scales + j * 8u, scales + 32u + j * 8u, (uint32_t)((ks | j) != 0u));
                            pair_mma(tmem, a1 + 2u * j, b + 2u * j, scales + j * 8u + 4u, scales + 32u + j * 8u, 1u);
                        }
                        pair_commit(&empty[s]);
                    }
                    __syncwarp();
                    ring.advance(kPairStages);
                }
                if (ok && leader) pair_commit(acc_full);
                __syncwarp();
            }
        }
      }
    } else if (warp < 8u) {
        registers_give_back<96>();
        uint32_t step = 0;
        bool ok = true;
        for (uint32_t item = pair; item < items && ok; item += pairs)
            for (uint32_t ks = 0; ks < k_steps; ++ks, ++step) {
                const uint32_t s = step % kPairStages, round = step / kPairStages;
                if (!eb::mbar_wait(&landed[s], round & 1u)) {
                    if (lane == 0) atomicOr(error, 8u);
                    ok = false;
                    break;
                }
                scales_to_tmem(reinterpret_cast<const uint4*>(smem + s * kPairStageBytes + kPairCodes) + lane,
                        tmem + (((warp & 3u) * 32u) << 16) + kTmemScales + s * kScaleColumns);
                if (lane == 0) signal_rank_relaxed(&scaled[s], 0u);
            }
    } else {
        // Epilogue, in both CTAs, each over its own 128 rows: as in gemm_kernel.
        registers_take<176>();
        const uint32_t quarter = warp & 3u, half = (warp - 8u) >> 2;
        const float scale_w = *tensor_global;
        uint32_t local = 0;
        for (uint32_t item = pair; item < items; item += pairs, ++local) {
            uint32_t tm, tn;
            place(item, &tm, &tn);
            if (!eb::mbar_wait(acc_full, local & 1u)) {
                if (lane == 0) atomicOr(error, 8u);
                break;
            }
            tcgen05_fence_after();
            uint32_t r[4][32];
            const uint32_t from = tmem + ((quarter * 32u) << 16) + (paired ? half * 64u : half * 128u);
            const uint32_t other = paired ? from + 128u : from + 64u;
            tmem_load_32(r[0], from);
            tmem_load_32(r[1], from + 32u);
            tmem_load_32(r[2], other);
            tmem_load_32(r[3], other + 32u);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) signal_rank_relaxed(acc_empty, 0u);   // what it orders are tensor-memory reads
            const uint32_t row = (2u * tm + rank) * kTileM + quarter * 32u + lane;
            const float scale = row < rows ? __fmul_rn(row_globals[row], scale_w) : 0.0f;
            store_block(r, out, row, rows, n, paired ? tn * 128u + half * 64u : tn * kTileN + half * 128u, scale, paired);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    eb::cluster_sync();   // neither CTA leaves while the other may still read its shared memory or arrive on its barriers
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns) : "memory");
    }
}

// ---- host side ------------------------------------------------------------------------------------------------------------

using eb::EncodeTiled;
using eb::encoder;

inline cudaError_t initialize() {
    const cudaError_t e = cudaFuncSetAttribute(gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSharedBytes);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairShared);
}

// Fewer rows than this run on single CTAs. us on pairs / single CTAs, in turn, rows x 17408 x 5120 and rows x 5120 x 17408: 256 rows
// 20.4 / 20.3 and 46.0 / 47.9, 384 rows 33.2 / 34.5 and 49.2 / 48.4, 512 rows 33.5 / 35.4 and 49.1 / 50.0, 1024 rows 66.4 / 71.0 and
// 92.2 / 99.5, 4096 rows 260 / 281 and 277 / 298: from 512 rows on both shapes are faster on pairs, below that one of them is not.
constexpr uint32_t kPairRows = 512;

template <typename... Params, typename... Args>
inline cudaError_t launch_on(cudaStream_t stream, bool pdl, void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared, Args... args) {
    return eb::launch_on(stream, pdl, 1u, kernel, grid, block, shared, args...);
}

// The launches of a native linear. Shapes are pre-checked by the caller: k % 256 == 0, out_features % 128 == 0,
// scratch aligned to 16 bytes and at least ActivationLayout(rows, k, out_features).bytes long.
// quantize: BF16 rows -> the activation part of the scratch (code planes, scale atoms, row scales).
inline cudaError_t quantize(const void* input, void* scratch, uint32_t rows, uint32_t k, cudaStream_t stream, bool pdl) {
    const uint32_t blocks = k / 16u;
    auto threads_of = [&](uint32_t held) { return std::min(quantize_threads(held), ((blocks + held - 1u) / held + 31u) / 32u * 32u); };
    auto run = [&](auto kernel, uint32_t held) {
        return launch_on(stream, pdl, kernel, dim3(rows), dim3(threads_of(held)), 0, static_cast<const __nv_bfloat16*>(input), static_cast<uint8_t*>(scratch), rows, k);
    };
    // rows an SM holds at once, by registers; three turns measured no better where they hold no more (rows of 8192 and 16,384 values)
    auto resident = [&](uint32_t held, uint32_t registers) { return 65536u / (threads_of(held) * registers); };
    return resident(3u, 80u) > resident(2u, 64u) || blocks > 2u * quantize_threads(2u) ? run(quantize_rows<3>, 3u) : run(quantize_rows<2>, 2u);
}

// multiply: the GEMM over the quantized activations found in the scratch (table-indexed weight scales are expanded there first).
// paired: the weights are a gate/up object (gate rows first); the output is [rows][out_features / 2] SwiGLU values.
// pairs: calls of kPairRows rows and more run on CTA pairs (gemm_pair_kernel).
inline cudaError_t multiply(const void* weights, void* output, void* scratch, uint32_t rows, uint32_t k, uint32_t out_features, int sms,
        cudaStream_t stream, bool pdl, uint32_t* error, bool paired = false, bool pairs = false, bool table_scales = false) {
    const EncodeTiled encode = encoder();
    if (encode == nullptr) return cudaErrorNotSupported;
    const ActivationLayout layout(rows, k, out_features);
    uint8_t* base = static_cast<uint8_t*>(scratch);
    const uint8_t* w = static_cast<const uint8_t*>(weights);
    const uint64_t row_bytes = k / 2u;
    // plain: scale bytes, then the FP32 tensor scale; table-indexed: index bytes, then 16 table codes and the tensor scale
    const uint64_t scale_offset = align256((uint64_t)out_features * row_bytes);
    const uint64_t table_offset = align256(scale_offset + (uint64_t)out_features * (k / (table_scales ? 32u : 16u)));
    const uint64_t global_offset = table_scales ? table_offset + 16u : table_offset;
    CUtensorMap map_a, map_b, map_s;
    const cuuint32_t ones[3] = {1u, 1u, 1u};
    const cuuint64_t a_dims[3] = {row_bytes, rows, kTerms}, a_strides[2] = {row_bytes, row_bytes * rows};
    // few rows: one kernel with the weights as the 128-row operand (nvfp4_decode.cuh), the rows as columns of a narrower box
    const bool few = nvfp4d::better_for(rows, k, out_features, paired, (uint32_t)sms);
    const cuuint32_t a_box[3] = {128u, few ? nvfp4d::columns_of(rows) : kTileM, 1u};
    const cuuint64_t b_dims[2] = {row_bytes, out_features}, b_strides[1] = {row_bytes};
    const cuuint32_t b_box[2] = {128u, 128u};   // half a B tile: the kernel places the two halves itself
    CUresult r = encode(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, a_dims, a_strides, a_box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    const float* row_globals = reinterpret_cast<const float*>(base + layout.global_offset);
    if (few && r == CUDA_SUCCESS) {
        const cudaError_t e = nvfp4d::quantized(weights, output, map_a, base + layout.sfa_offset, row_globals, rows, k, out_features, paired, table_scales, sms, stream,
                pdl, error);
        if (e != cudaErrorNotSupported) return e;
        return cudaErrorInvalidValue;
    }
    if (r == CUDA_SUCCESS)
        r = encode(&map_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(w), b_dims, b_strides, b_box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    // the scale bytes [n][K/16]: the tensor's own plane, or the plane a table-indexed tensor's indices are expanded to
    const uint64_t scale_row = k / 16u;
    uint8_t* scales = table_scales ? base + layout.sfb_offset : const_cast<uint8_t*>(w + scale_offset);
    const cuuint64_t s_dims[2] = {scale_row, out_features}, s_strides[1] = {scale_row};
    const cuuint32_t s_box[2] = {kStepK / 16u, 128u};
    if (r == CUDA_SUCCESS)
        r = encode(&map_s, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, scales, s_dims, s_strides, s_box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    cudaError_t e = cudaSuccess;
    if (table_scales) {
        const uint32_t vectors = (uint32_t)((uint64_t)out_features * scale_row / 16u);
        e = launch_on(stream, pdl, expand_table_scales, dim3((vectors + 255u) / 256u), dim3(256), 0, w + scale_offset, w + table_offset, scales, vectors);
        if (e != cudaSuccess) return e;
    }
    const uint32_t pair_tiles = paired ? out_features / 256u : 0u, width = paired ? out_features / 2u : out_features;
    const uint32_t tiles = ((rows + kTileM - 1u) / kTileM) * (paired ? pair_tiles : (out_features + kTileN - 1u) / kTileN);
    const uint32_t grid = tiles < (uint32_t)sms ? tiles : (uint32_t)sms;
    const float* tensor_global = reinterpret_cast<const float*>(w + global_offset);
    if (pairs && rows >= kPairRows) {
        const uint32_t pair_items = ((rows + 255u) / 256u) * (paired ? pair_tiles : (out_features + 255u) / 256u);
        const uint32_t ctas = 2u * std::max(1u, std::min((uint32_t)sms / 2u, pair_items));
        return launch_on(stream, pdl, gemm_pair_kernel, dim3(ctas), dim3(kScaledThreads), kPairShared, map_a, map_b, map_s,
                base + layout.sfa_offset, row_globals, tensor_global, static_cast<uint16_t*>(output), rows, width, k, pair_tiles, error);
    }
    return launch_on(stream, pdl, gemm_kernel, dim3(grid), dim3(kScaledThreads), kSharedBytes, map_a, map_b, map_s, base + layout.sfa_offset, row_globals,
            tensor_global, static_cast<uint16_t*>(output), rows, width, k, pair_tiles, error);
}

inline cudaError_t run(const void* input, const void* weights, void* output, void* scratch, uint32_t rows, uint32_t k, uint32_t out_features,
        int sms, cudaStream_t stream, bool pdl, uint32_t* error, bool paired = false, bool pairs = false, bool table_scales = false) {
    const cudaError_t e = quantize(input, scratch, rows, k, stream, pdl);
    return e != cudaSuccess ? e : multiply(weights, output, scratch, rows, k, out_features, sms, stream, pdl, error, paired, pairs, table_scales);
}

}  // namespace nvfp4n

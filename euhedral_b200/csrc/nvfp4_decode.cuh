// NVFP4 linears of few rows on sm_100a as one tcgen05 kernel: the weights are the 128-row operand, the activation rows the
// columns, so that a call streams the weights once and everything else hides behind that stream.
//
// Two sources of activations (template parameter):
//   * BF16 rows (euhedral_cuda_linear_nvfp4_bf16 and the grouped calls, up to kMaxRows). kind::mxf4nvf4 multiplies E2M1 by E2M1, so
//     a CTA writes its K slice of every activation row as EIGHT E2M1 terms of three bits each - the octal digits, -4 to 3, of
//     the value as an integer of 24 bits, in units of 2^-21 of the power of two of the row's largest value of the slice - and a
//     row becomes eight columns. Products are exact; column t of a row counts 8^-t and the eight sums are added in FP32 once per K
//     slice. Every value counts in full. Eight digits hold a BF16 value exactly down to 2^-14 of the power of two of the slice's largest;
//     where a row has smaller ones, four more columns hold the next four digits, down to 2^-24; what is smaller still (or is below
//     2^-103 whatever the largest, or not finite) is left out of the digits, and the draining warps add its products in FP32 from the
//     weights in memory (about 0.5 us a tile and 32 values: 34816 x 5120 at 5 rows 24 us, 36 where four values of a row are 1000 times
//     larger, 731 where the values spread evenly over 40 powers of two). So an infinity gives every output what IEEE arithmetic gives it. The choice is a row's and slice's own and
//     changes no bit of the rows beside it. Of 1280 normally distributed values, one slice in eight takes more digits, one in ten
//     thousand leaves a value out.
//   * two NVFP4 terms per row, quantized into the scratch before (the native route): a row is one column, both terms accumulate
//     into it, as in the large GEMM (nvfp4_native.cuh), and more than kMaxColumns rows take a tile of weights several times.
//     With `pair_rows` a tile is 64 gate rows and the 64 up rows that match them, finished as SwiGLU (the paired region).
// The reference's counterparts: native/src/nvfp4/kernels.cu:8-36 (decode) and native/src/nvfp4_native/native.cuh:435-585 (the
// 9- to 64-row kernel).
//
// Bound: HBM, with about 5 us of launch, staging and exchange around the stream. Per 128 rows x 64 values the weights are 4.6 KB =
// 200 cycles of an SM's share of the bandwidth; an MMA takes about 110 of them, whatever its columns up to 64. The decode
// through registers and mma.sync that this replaces was bound by its instruction issue at 0.4 of the bandwidth. Measured, NVFP4,
// replayed back to back with programmatic dependent launch, before -> now (us at 1 / 5 / 8 rows): 34816 x 5120 33.6 / 35.7 / 68.3 -> 21.0 /
// 23.8 / 25.8 (4.8 TB/s at one row); 17408 x 5120 19.6 / 21.5 / 41.0 -> 13.3 / 15.6 / 17.1; 5120 x 17408 22.3 / 25.4 / 46.5 -> 13.7 / 17.4 / 21.2;
// 5120 x 5120 9.6 / 11.5 / 21.7 -> 8.4 / 10.5 / 11.4. Tensors of a few MB, where the fixed part is not hidden, lose about 1 us up to 5
// rows (1024 x 5120: 4.1 / 6.2 / 11.0 -> 5.3 / 7.2 / 8.2): a choice by the number of rows of the weights would give shards and group
// members other bits than the whole. The native route's few rows: a layer's four fused linears at 40 rows 176 -> 90 us, quantizers included.
// The fixed part is a chain of short pieces of code that every launch fetches anew, so what is rarely needed stands after the loops,
// a loop runs one copy of its body over values held in registers, and an item's fields are copied before they are needed: together
// with the digits by table (octal_digits) 1024 x 5120 at 1 / 5 / 8 rows went from 6.0 / 8.6 / 9.8 to 5.3 / 7.2 / 8.2 us.
// Instructions that one thread issues for the tensor core sit in a loop of the whole warp under an elected predicate (eb::elect_one):
// 757 -> 453 cycles per unit of 256 values.
//
// Execution:
//   * K is cut into units of 256 and these over the CTAs of a cluster. For BF16 rows the cut (split_of) is a function of K only, as is
//     every order of summation, so that rows, N-shards and members of a group give the bits of the single call. A cluster walks
//     a contiguous run of the 128-row tiles of all tensors of the launch. One CTA per SM.
//   * warp 0: the ring - codes by TMA (a stage: 128 rows x 256 values, 128-byte swizzle) [and the quantized activations], scale bytes
//     by cp.async, any pitch; warps 4..7: scale bytes (or table indices) to tensor memory; warp 1: four MMAs a stage; warps 8..11:
//     drain the tile's sums, send each row's to the CTA of the cluster that owns it (st.async into its shared memory, counted on
//     its barrier), and add the cluster's slices in rank order there; warps 2, 3 and 8..15 write the digits; warp 2 also tells the
//     cluster when this CTA's exchange buffers have been read.
//   * Weights do not depend on the launch before: their ring fills before griddepcontrol.wait and while the rows are staged.
// Every wait is bounded.
#pragma once

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "exact_kernels.cuh"
#include "nvfp4_native.cuh"

namespace nvfp4d {

constexpr uint32_t kTile = 128, kUnit = 256, kDigits = 8, kMoreDigits = 4;
constexpr uint32_t kMaxRows = 16;         // BF16 activation rows of a launch
constexpr uint32_t kMaxColumns = 64;      // quantized activation rows of an item
constexpr uint32_t kMaxGroup = 8;         // tensors of a launch
constexpr uint32_t kThreads = 512, kStagers = 320;   // staging warps: 2, 3 and 8 to 15
constexpr uint32_t kCodeBytes = kTile * kUnit / 2u, kScaleBytes = kTile * kUnit / 16u;
constexpr uint32_t kMaxStages = 8;
constexpr uint32_t kTmemColumns = 512;
constexpr uint32_t kHeldByEight = 14, kHeldByTwelve = 24;   // powers of two below the largest value that the digits hold exactly (see above)
// Exchange buffers of a CTA. The word that one may be filled again reaches the other CTAs a microsecond or two after it was read;
// with two buffers for BF16 rows the draining warps waited for it (34816 x 5120 at one row 26.4 us, with four 22.1).
// Two remain for quantized rows, whose buffers are large and whose calls exchange few tiles, and where four leave no room for the digits.
constexpr uint32_t kMostSlots = 4, kFewSlots = 2;
constexpr uint32_t kLeftWords = 128;      // rows times units of a CTA: more than its shared memory has room for digits of
constexpr uint32_t kLeastExponent = 48;   // of a row's slice: the grid does not get finer than that of 2^-79

__host__ __device__ inline uint32_t units_of(uint32_t k) { return (k + kUnit - 1u) / kUnit; }
// BF16 rows: CTAs of a cluster that share a tile's K, and so the slices that are added in order: a function of K only. More of them
// keep more SMs busy on short tensors and need less shared memory for the digits each; fewer exchange fewer sums. Never 1: the
// exchange (st.async) needs a launch in clusters. A CTA may be left without a unit (K up to 256), it sends zeros.
__host__ __device__ inline uint32_t split_of(uint32_t units) { return units < 4u ? 2u : units <= 48u ? 4u : 8u; }

struct alignas(64) Tensor {
    CUtensorMap codes;         // bytes [n][K/2], box 128 x 64 rows (half a tile)
    const uint16_t* x;         // BF16 [rows][K] (decode)
    const uint8_t* weights;    // the code plane
    const uint8_t* scales;     // the scale (or index) plane
    const uint8_t* table;      // the 16 E4M3 codes of a table-indexed tensor, else null
    const float* global;
    uint16_t* y;
    uint32_t n, tile_end;      // end of this tensor's tiles in the launch's list
};

struct alignas(64) Group {
    uint32_t count, rows, k, tiles, stages, scale_row_bytes;
    uint32_t split;            // CTAs of a cluster, each with a slice of K; 1 (quantized rows only): no cluster, no exchange
    uint32_t tmem_columns;     // allocated: a power of two
    uint32_t buffers;          // accumulators of consecutive items: 2, or 1 where tensor memory is short
    uint32_t slots;            // exchange buffers
    uint32_t row_groups;       // quantized rows: groups of kMaxColumns; an item of the launch is a tile and a group
    uint32_t pair_rows;        // the paired region: gate rows of the tensor (0: a plain linear)
    const uint8_t* atoms;      // quantized rows: their block scales (nvfp4n::ActivationLayout)
    const float* row_globals;
    Tensor tensor[kMaxGroup];
    CUtensorMap activations;   // quantized rows: bytes [term][rows][K/2], box 128 x columns x 1
};

// What a CTA of a launch keeps in shared memory.
//   columns: of an item (resident: the digits of the rows; else the rows, to a multiple of 32). n: of the MMA - quantized rows
//   bring their two terms as columns of their own.
struct Layout {
    uint32_t columns, n, plain_n, width, pitch, stage_bytes, off_rows, off_gather, gather_bytes, off_bars, bytes;
    __host__ __device__ Layout(bool resident, uint32_t rows, uint32_t units_cta, uint32_t stages, uint32_t split, bool paired, uint32_t slots) {
        columns = resident ? (rows * (kDigits + kMoreDigits) + 15u) / 16u * 16u : rows >= kMaxColumns ? kMaxColumns : (rows + 7u) / 8u * 8u;
        n = resident ? columns : nvfp4n::kTerms * columns;
        plain_n = resident ? (rows * kDigits + 15u) / 16u * 16u : n;   // of rows without outliers: the first eight digits come first
        width = resident ? rows : columns;                           // sums of a weight row and slice that travel together
        pitch = columns + 4u;                                        // quantized rows: floats from row to row of an exchange buffer
        gather_bytes = resident ? kTile * width * 4u : kTile * pitch * 4u;   // one of the exchange buffers
        stage_bytes = kCodeBytes + kScaleBytes + (resident ? 0u : nvfp4n::kTerms * columns * 128u + nvfp4n::kSfaStage);
        stage_bytes = (stage_bytes + 1023u) & ~1023u;
        off_rows = stages * stage_bytes;                             // resident digits: a tile of `columns` x 128 bytes per unit
        off_gather = off_rows + (resident ? units_cta * columns * 128u : 0u);
        off_bars = off_gather + (split > 1u ? slots * gather_bytes : paired ? gather_bytes / 2u : 0u);
        bytes = off_bars + 1024u + 1024u;                            // barriers, the rows' exponents and left-out values or scales; slack to align to 1024
    }
};

__device__ __forceinline__ void stagers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kStagers) : "memory"); }
__device__ __forceinline__ void drainers_sync() { asm volatile("bar.sync 2, 128;" ::: "memory"); }
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void send_f32(uint32_t to, float value, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(to), "r"(__float_as_uint(value)), "r"(bar) : "memory");
}
__device__ __forceinline__ void send_f32x4(uint32_t to, float a, float b, float c, float d, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to), "r"(__float_as_uint(a)),
            "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(__float_as_uint(d)), "r"(bar)
            : "memory");
}
// cp.async of BYTES bytes, zeros when `live` is false.
template <int BYTES>
__device__ __forceinline__ void copy_or_zero(uint32_t to, const void* from, bool live) {
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(live ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(to), "l"(from), "n"(BYTES), "r"(live ? BYTES : 0) : "memory");
}

template <int N>
__device__ __forceinline__ void tmem_store(uint32_t to, const uint32_t* r) {
    static_assert(N == 16 || N == 32, "");
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(to), "r"(r[0]), "r"(r[1]),
            "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
            "r"(r[15])
            : "memory");
    if constexpr (N == 32) tmem_store<16>(to + 16u, r + 16);
}
__device__ __forceinline__ void tmem_load_4(uint32_t (&r)[4], uint32_t from) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(from));
}
__device__ __forceinline__ void tmem_load_8(uint32_t (&r)[8], uint32_t from) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
            : "r"(from));
}
__device__ __forceinline__ void tmem_load_16(uint32_t (&r)[16], uint32_t from) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
              "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(from));
}
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t instruction, uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
    asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %6, 0;\n"
            "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%4], [%5], p;\n}" ::"r"(d),
            "l"(a), "l"(b), "r"(instruction), "r"(sfa), "r"(sfb), "r"(accumulate)
            : "memory");
}

// Eight values as eight octal digits each, transposed: word t holds digit t (the highest first) of the eight values as E2M1 codes,
// value i in nibble i. The values are counted in units of 1 / `per`; kMore: what that count cuts off, in units of 2^-22 / `per`.
template <bool kMore>
__device__ __forceinline__ void octal_digits(const uint4& v, float per, uint32_t (&word)[8]) {
    const uint32_t pairs[4] = {v.x, v.y, v.z, v.w};
    const float unit = __uint_as_float(0x7F000000u - __float_as_uint(per)), count = kMore ? __uint_as_float(__float_as_uint(per) + (22u << 23)) : per;
    uint32_t low[4], high[4];   // of a pair of neighbouring values, digits 0 to 3 and 4 to 7 (0: the lowest), a byte each
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float x = (i & 1) ? __uint_as_float(pairs[i >> 1] & 0xFFFF0000u) : __uint_as_float(pairs[i >> 1] << 16);
        if (kMore) x = __fmaf_rn(-__fsub_rn(__fmaf_rn(x, per, 12582912.0f), 12582912.0f), unit, x);   // exact
        // 1.5 * 2^23 + the integer, then + 4 in every octal digit: each digit less 4 is the signed digit
        uint32_t s = __float_as_uint(__fmaf_rn(x, count, 12582912.0f)) - 0x4B400000u + 9586980u;
        s += (s & 0x00FFF000u) * 15u;   // 24 bits of octal digits to eight nibbles
        s += (s & 0x0FC00FC0u) * 3u;
        s += s & 0x38383838u;
        // Each nibble selects its E2M1 code from eight bytes: -4 to -1 and 0 to 3 halves, of odd values in the byte's upper half.
        const uint32_t below = (i & 1) ? 0x90A0B0C0u : 0x090A0B0Cu, above = (i & 1) ? 0x30201000u : 0x03020100u;
        const uint32_t four = __byte_perm(below, above, s), next = __byte_perm(below, above, s >> 16);
        low[i >> 1] = (i & 1) ? low[i >> 1] | four : four;
        high[i >> 1] = (i & 1) ? high[i >> 1] | next : next;
    }
    auto transposed = [&](const uint32_t (&c)[4], uint32_t* highest) {   // 4 x 4 bytes; the highest digit first
        const uint32_t a = __byte_perm(c[0], c[1], 0x5140), b = __byte_perm(c[2], c[3], 0x5140);
        const uint32_t d = __byte_perm(c[0], c[1], 0x7362), e = __byte_perm(c[2], c[3], 0x7362);
        highest[3] = __byte_perm(a, b, 0x5410), highest[2] = __byte_perm(a, b, 0x7632);
        highest[1] = __byte_perm(d, e, 0x5410), highest[0] = __byte_perm(d, e, 0x7632);
    };
    transposed(high, word);
    transposed(low, word + 4);
}

// The largest exponent of eight BF16 values. 0: nothing but zeros (or subnormal values); 255: not all of them are finite.
__device__ __forceinline__ uint32_t largest_exponent(const uint4& v) {
    const uint32_t most = __vmaxu2(__vmaxu2(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu), __vmaxu2(v.z & 0x7FFF7FFFu, v.w & 0x7FFF7FFFu));
    return max(most & 0xFFFFu, most >> 16) >> 7;
}
// The least exponent of the eight, zeros aside (subnormal values: 0). More than 255: nothing but zeros.
__device__ __forceinline__ uint32_t least_exponent(const uint4& v) {
    auto less_one = [](uint32_t w) { return ((w & 0x7FFF7FFFu) + 0x7FFF7FFFu) ^ 0x80008000u; };   // both halves' magnitudes; of a zero 65535
    const uint32_t low = __vminu2(__vminu2(less_one(v.x), less_one(v.y)), __vminu2(less_one(v.z), less_one(v.w)));
    return (min(low & 0xFFFFu, low >> 16) + 1u) >> 7;
}
// What the digits of a BF16 value leave out of it. `per`: 1 / the unit of its row; more: the row has the further digits.
__device__ __forceinline__ float not_held(uint32_t bits, float per, bool more) {
    const float x = eb::bf16_bits_to_float(bits), unit = __uint_as_float(0x7F000000u - __float_as_uint(per));
    const float behind = __fmaf_rn(-__fsub_rn(__fmaf_rn(x, per, 12582912.0f), 12582912.0f), unit, x);
    // The further digits count that in units of 2^-22 / `per`; of eight digits, the last four (-2340 to 1755) are not kept.
    const int count = (int)(__float_as_uint(__fmaf_rn(behind, __uint_as_float(__float_as_uint(per) + (22u << 23)), 12582912.0f)) - 0x4B400000u);
    const float last = __fmaf_rn(-(float)((count + 2340) & ~4095), __uint_as_float(__float_as_uint(unit) - (22u << 23)), behind);
    return (bits & 0x7F80u) == 0x7F80u ? x : more ? last : behind;
}
// Eight BF16 values with zeros in the place of those that are not finite.
__device__ __forceinline__ uint4 finite_only(const uint4& v) {
    auto word = [](uint32_t w) {
        return w & (((w & 0x7F80u) == 0x7F80u ? 0u : 0xFFFFu) | ((w & 0x7F800000u) == 0x7F800000u ? 0u : 0xFFFF0000u));
    };
    return make_uint4(word(v.x), word(v.y), word(v.z), word(v.w));
}

// What the staging warps of a CTA share about its slice of the rows.
struct Slice {
    const uint16_t* x;
    uint32_t rows, k, unit_begin, units;
    uint32_t stager, lane;                  // the staging warp among them
    uint32_t *exponents, *least, *left;
    uint8_t* digits;
    uint32_t columns;
    __device__ __forceinline__ uint4 load(uint32_t row, uint32_t unit) const {   // this lane's eight values of a unit
        const uint32_t at = (unit_begin + unit) * kUnit + lane * 8u;
        return row < rows && at < k ? *reinterpret_cast<const uint4*>(x + (uint64_t)row * k + at) : make_uint4(0u, 0u, 0u, 0u);
    }
    __device__ __forceinline__ bool has_more(uint32_t row) const { return least[row] + kHeldByEight < exponents[row]; }
    __device__ __forceinline__ void find(uint32_t row, const uint4& v) const {
        const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, largest_exponent(v)), low = __reduce_min_sync(0xFFFFFFFFu, least_exponent(v));
        if (row < rows && lane == 0) {
            atomicMax(&exponents[row], most);
            atomicMin(&least[row], low);
        }
    }
    __device__ __forceinline__ float per(uint32_t row) const { return __uint_as_float((275u - exponents[row]) << 23); }   // 1 / the row's unit
    // Whether the digits of the row leave values out: there are some that are not finite, or too small.
    __device__ __forceinline__ bool leaves_out(uint32_t row) const { return exponents[row] == 255u || least[row] + kHeldByTwelve < exponents[row]; }
    __device__ __forceinline__ void write(uint32_t row, uint32_t unit, const uint4& values) const {
        write_digits<false>(row * kDigits, row, unit, values);
        if (has_more(row)) write_digits<true>(rows * kDigits + row * kMoreDigits, row, unit, values);
    }
    // `column`: of digit 0; rows of 128 bytes, swizzled.
    template <bool kMore>
    __device__ __forceinline__ void write_digits(uint32_t column, uint32_t row, uint32_t unit, const uint4& values) const {
        uint32_t word[8];
        octal_digits<kMore>(values, per(row), word);
        uint8_t* to = digits + unit * columns * 128u + (column >> 3) * 1024u + (lane & 3u) * 4u;
        const uint32_t first = kMore ? column & 7u : 0u;   // 4 for every other row's further digits
#pragma unroll
        for (uint32_t t = 0; t < (kMore ? kMoreDigits : kDigits); ++t)
            *reinterpret_cast<uint32_t*>(to + (first + t) * 128u + (((lane >> 2) ^ (first + t)) << 4)) = word[t];
    }
};

// For the rows of a mask, whose digits leave values out: the words that say where those are. Rows with values that are not finite first
// get their exponents over the others, and their digits again. Taken by every staging warp when all digits have been written.
__device__ __forceinline__ void stage_again(const Slice& slice, const uint32_t odd_rows) {
    auto for_units = [&](uint32_t mask, auto&& body) {
#pragma unroll 1
        for (; mask != 0u; mask &= mask - 1u)
#pragma unroll 1
            for (uint32_t u = slice.stager; u < slice.units; u += kStagers / 32u) body((uint32_t)__ffs((int)mask) - 1u, u);
    };
    const bool mine = ((odd_rows >> slice.lane) & 1u) && slice.exponents[slice.lane & (kMaxRows - 1u)] == 255u;
    const uint32_t again = __ballot_sync(0xFFFFFFFFu, mine);
    if (again != 0u) {
        stagers_sync();   // nobody needs the exponents that led here any more
        if (slice.stager == 0u && mine) slice.exponents[slice.lane] = kLeastExponent, slice.least[slice.lane] = 255u;
        stagers_sync();
        for_units(again, [&](uint32_t row, uint32_t u) { slice.find(row, finite_only(slice.load(row, u))); });
        stagers_sync();
        for_units(again, [&](uint32_t row, uint32_t u) { slice.write(row, u, finite_only(slice.load(row, u))); });
    }
    for_units(odd_rows, [&](uint32_t row, uint32_t u) {
        const uint4 values = slice.load(row, u);
        const uint32_t pairs[4] = {values.x, values.y, values.z, values.w};
        bool some = false;
#pragma unroll
        for (uint32_t i = 0; i < 8u; ++i) some = some || not_held((pairs[i >> 1] >> (16u * (i & 1u))) & 0xFFFFu, slice.per(row), slice.has_more(row)) != 0.0f;
        const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, some);
        if (slice.lane == 0u) slice.left[row * slice.units + u] = lanes;
    });
    stagers_sync();   // the words are there for the draining warps
}

// What the digits of the odd rows leave out of a slice, summed against one weight row per lane in FP32 in K order: beside[m] of every
// odd row m. The weights are read where they lie (the ring has moved on), 32 values of K at a time: a lane finds what is left of one
// of them and all take it from there. The loads of a part are in flight while the part before it is summed. Taken by
// whole warps.
template <bool kTable>
__device__ __forceinline__ void left_out(const Tensor& t, const Slice& slice, uint32_t row, uint32_t odd_rows, float (&beside)[kMaxRows]) {
    row = min(row, t.n - 1u);
    const uint32_t code_pitch = slice.k / 2u, scale_pitch = slice.k / (kTable ? 32u : 16u);
    const uint8_t* codes = t.weights + (uint64_t)row * code_pitch;
    const uint8_t* scale_codes = t.scales + (uint64_t)row * scale_pitch;
    struct Part {
        uint32_t m, scale, value;   // activation row (kMaxRows: there are no more), the weight row's scale codes, the lane's value
        uint4 code;
    } now = {kMaxRows, 0u, 0u, make_uint4(0u, 0u, 0u, 0u)}, ahead = now;
    const uint16_t* x = t.x;
    const uint8_t* table = t.table;
    uint32_t m = 0u, base = slice.units, word = 0u, units = 0u, u = 0u, lanes = 0u;   // a lane looks at every 32nd unit's word
    float sum = 0.0f;
#pragma unroll 1
    while (true) {
        ahead.m = kMaxRows;
#pragma unroll 1
        while (lanes == 0u) {
            if (units != 0u) {
                const uint32_t at = (uint32_t)__ffs((int)units) - 1u;
                units &= units - 1u;
                u = base + at;
                lanes = __shfl_sync(0xFFFFFFFFu, word, (int)at);
                break;
            }
            base += 32u;
            if (base >= slice.units) {
                if (odd_rows == 0u) break;
                m = (uint32_t)__ffs((int)odd_rows) - 1u;
                odd_rows &= odd_rows - 1u;
                base = 0u;
                beside[m] = 0.0f;
            }
            word = base + slice.lane < slice.units ? slice.left[m * slice.units + base + slice.lane] : 0u;
            units = __ballot_sync(0xFFFFFFFFu, word != 0u);
        }
        if (lanes != 0u) {
            const uint32_t shift = ((uint32_t)__ffs((int)lanes) - 1u) & ~3u, eighths = (lanes >> shift) & 15u;
            lanes &= ~(15u << shift);
            const uint32_t first = ((slice.unit_begin + u) * 32u + shift) * 8u;   // of its 32 values
            ahead.m = m;
            ahead.code = *reinterpret_cast<const uint4*>(codes + first / 2u);
            ahead.scale = kTable ? scale_codes[first / 32u] : *reinterpret_cast<const uint16_t*>(scale_codes + first / 16u);
            ahead.value = (eighths >> (slice.lane >> 3)) & 1u ? x[(uint64_t)m * slice.k + first + slice.lane] : 0u;
        }
        if (now.m != kMaxRows) {
            const uint32_t scale = kTable ? table[now.scale & 15u] | (uint32_t)table[now.scale >> 4] << 8 : now.scale;
            const float rest = not_held(now.value, slice.per(now.m), slice.has_more(now.m));
            const uint32_t words[4] = {now.code.x, now.code.y, now.code.z, now.code.w};
            const float blocks[2] = {exact::e4m3(scale & 0xFFu), exact::e4m3(scale >> 8)};
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const uint32_t code4 = words[i >> 3] >> (4 * (i & 7));
                // sign and magnitude where an FP32 number reads them as e2m1 * 2^-126
                const float weight = __fmul_rn(__uint_as_float((code4 & 8u) << 28 | (code4 & 7u) << 22), 8.507059173023462e37f);
                sum = __fmaf_rn(__shfl_sync(0xFFFFFFFFu, rest, i), __fmul_rn(weight, blocks[i >> 4]), sum);
            }
            if (ahead.m != now.m) {   // the row's last part
                beside[now.m] = sum;
                sum = 0.0f;
            }
        }
        if (ahead.m == kMaxRows) break;
        now = ahead;
    }
}

// One lane's four words of scales (K blocks 0..3 of a unit) of a row, from its bytes in the stage.
template <bool kTable>
__device__ __forceinline__ uint4 row_scales(const uint8_t* at, const uint4& table) {
    if (!kTable) return *reinterpret_cast<const uint4*>(at);
    const uint2 pairs = *reinterpret_cast<const uint2*>(at);
    uint32_t words[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t four = ((i & 2) ? pairs.y : pairs.x) >> (16 * (i & 1)), within = four & 0x7777u;
        const uint32_t low = __byte_perm(table.x, table.y, within), high = __byte_perm(table.z, table.w, within);
        words[i] = eb::lop3<eb::kLutSelect>(high, low, __byte_perm(0u, 0xFFFFFFFFu, (four >> 1) & 0x4444u));
    }
    return make_uint4(words[0], words[1], words[2], words[3]);
}

//   grid: clusters x split CTAs, cluster split, block kThreads, dynamic shared Layout(...).bytes.
//   kResident: BF16 rows, whose digits stay in shared memory; else quantized rows through the ring.
template <bool kResident, bool kTable>
__global__ void __launch_bounds__(kThreads, 1) kernel(const __grid_constant__ Group group, uint32_t* __restrict__ error) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~(uintptr_t)1023u);
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31u;   // the same in all lanes, and known to be
    const uint32_t rows = group.rows, k = group.k, stages = group.stages;
    const uint32_t units = units_of(k), split = group.split;
    const bool exchange = split > 1u;
    const uint32_t rank = exchange ? eb::cluster_rank() : 0u, clusters = gridDim.x / split, cluster = blockIdx.x / split;
    const uint32_t run_begin = (uint32_t)((uint64_t)cluster * group.tiles / clusters), run_end = (uint32_t)((uint64_t)(cluster + 1u) * group.tiles / clusters);
    const uint32_t unit_begin = rank * units / split, unit_end = (rank + 1u) * units / split, mine = unit_end - unit_begin;
    const uint32_t slots = group.slots, slots_log = slots >> 1;   // 4 or 2
    const bool paired = !kResident && group.pair_rows != 0u;
    const Layout layout(kResident, rows, (units + split - 1u) / split, stages, split, paired, slots);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + layout.off_bars);
    uint64_t *full = bars, *empty = full + kMaxStages, *scaled = empty + kMaxStages, *acc_full = scaled + kMaxStages, *acc_empty = acc_full + 2,
             *staged = acc_empty + 2, *gather_full = staged + 1, *gather_empty = gather_full + kMostSlots, *gather_read = gather_empty + kMostSlots;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(gather_read + kMostSlots);
    uint32_t* failed = tmem_holder + 1;
    uint32_t* exponents = failed + 1;        // per row: the largest exponent of the slice
    uint32_t* least = exponents + kMaxRows;  // per row: the least exponent of the slice, zeros aside
    uint32_t* left = least + kMaxRows;       // of a row whose digits leave values out, [row][unit of the slice]: bit i: of values 8 i .. 8 i + 7 of the unit
    auto has_more = [&](uint32_t row) { return least[row] + kHeldByEight < exponents[row]; };   // four more digits
    const uint32_t kBoxColumns = layout.columns;

    if (warp == 0) {
        if (lane < stages) {
            eb::mbar_init(&full[lane], 33);     // the TMA request and the lanes' cp.async
            eb::mbar_init(&empty[lane], 1);
            eb::mbar_init(&scaled[lane], 4);
        } else if (lane >= 16u && lane < 18u) {
            const uint32_t b = lane - 16u;
            eb::mbar_init(&acc_full[b], 1);
            eb::mbar_init(&acc_empty[b], 4);
        } else if (lane >= 20u && lane < 20u + slots) {
            const uint32_t b = lane - 20u;
            eb::mbar_init(&gather_full[b], 1);
            eb::mbar_init(&gather_empty[b], split);
            eb::mbar_init(&gather_read[b], 4);
        } else if (lane == 18u) {
            eb::mbar_init(staged, kStagers / 32u);
            *failed = 0u;
        }
        eb::mbar_fence_init();
        __syncwarp();
    } else if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(eb::smem_u32(tmem_holder)), "r"(group.tmem_columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else if (warp == 2) {
        if (kResident && lane < kMaxRows) exponents[lane] = kLeastExponent, least[lane] = 255u;
    }
    nvfp4n::tcgen05_fence_before();
    __syncthreads();
    if (exchange) eb::cluster_arrive();    // waited for by the warps that touch another CTA
    nvfp4n::tcgen05_fence_after();
    eb::pdl_launch_dependents();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_holder, 0);
    auto wait = [&](uint64_t* bar, uint32_t parity) { eb::mbar_wait_or_fail(bar, parity, failed); };

    // Calls body(t, tile in the tensor, items before it in this run, row group) for the run's items in order.
    auto for_tiles = [&](auto&& body) {
        if (kResident) {
            uint32_t first = 0, at = run_begin;
            for (uint32_t ti = 0; ti < group.count && at < run_end; ++ti) {
                const Tensor& t = group.tensor[ti];
                for (; at < min(run_end, t.tile_end); ++at) body(t, at - first, at - run_begin, 0u);
                first = t.tile_end;
            }
        } else {
            for (uint32_t at = run_begin; at < run_end; ++at) body(group.tensor[0], at / group.row_groups, at - run_begin, at % group.row_groups);
        }
    };
    // First weight row of the lower and the upper half of a tile.
    auto lower = [&](uint32_t tile) { return paired ? tile * 64u : tile * kTile; };
    auto upper = [&](uint32_t tile) { return paired ? group.pair_rows + tile * 64u : tile * kTile + 64u; };

    if (warp == 0) {
        // ---- the ring: codes [and quantized activations] by TMA, scale bytes by cp.async ----
        // The scale bytes of a stage: lane l takes rows l, l + 32, ... of the tile. Past the tensor's rows or K: zeros.
        if (!kResident) eb::pdl_wait();
        bool first_round = true;
        eb::Ring ring;
        const bool leader = eb::elect_one();
        const uint32_t pitch = group.scale_row_bytes;
        constexpr uint32_t kRowBytes = kTable ? 8u : 16u;   // of a unit
        const uint32_t off = layout.stage_bytes - kScaleBytes;
        for_tiles([&](const Tensor& t, uint32_t tile, uint32_t, uint32_t row_group) {
            const int low = (int)lower(tile), high = (int)upper(tile);
            // this lane's four rows of scale bytes, at the slice's first unit
            const uint8_t* from[4];
            bool live[4];
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {
                const uint32_t row = (uint32_t)(j < 2u ? low : high - 64) + j * 32u + lane;
                live[j] = row < t.n;
                from[j] = t.scales + (uint64_t)(live[j] ? row : 0u) * pitch + unit_begin * kRowBytes;
            }
            for (uint32_t u = unit_begin; u < unit_end; ++u) {
                const uint32_t s = ring.stage;
                if (!first_round) wait(&empty[s], ring.parity ^ 1u);
                uint8_t* stage = smem + s * layout.stage_bytes;
                if (leader) {
                    eb::mbar_arrive_expect_tx(&full[s], kCodeBytes + (kResident ? 0u : nvfp4n::kTerms * kBoxColumns * 128u + nvfp4n::kSfaStage));
                    eb::tma_load_2d(stage, &t.codes, (int)(u * 128u), low, &full[s]);
                    eb::tma_load_2d(stage + kCodeBytes / 2u, &t.codes, (int)(u * 128u), high, &full[s]);
                    if (!kResident) {
                        uint8_t* to = stage + kCodeBytes;
                        nvfp4n::tma_load_3d(to, &group.activations, (int)(u * 128u), (int)(row_group * kMaxColumns), 0, &full[s]);
                        nvfp4n::tma_load_3d(to + kBoxColumns * 128u, &group.activations, (int)(u * 128u), (int)(row_group * kMaxColumns), 1, &full[s]);
                        to += nvfp4n::kTerms * kBoxColumns * 128u;
                        eb::bulk_g2s(to, group.atoms + ((uint64_t)(row_group * kMaxColumns / nvfp4n::kTileM) * units + u) * nvfp4n::kSfaStage, nvfp4n::kSfaStage, &full[s]);
                    }
                }
                const uint32_t to = eb::smem_u32(stage + off) + lane * 16u;
                const bool whole = (u + 1u) * kRowBytes <= pitch;   // the unit's second half exists
#pragma unroll
                for (uint32_t j = 0; j < 4u; ++j) {
                    const uint32_t into = to + j * 512u;
                    const bool tail = live[j] && whole;
                    if (!kTable) {
                        if ((pitch & 15u) == 0u) {
                            copy_or_zero<16>(into, from[j], live[j]);
                        } else {
                            copy_or_zero<8>(into, from[j], live[j]);
                            copy_or_zero<8>(into + 8u, tail ? from[j] + 8u : from[j], tail);
                        }
                    } else if ((pitch & 7u) == 0u) {
                        copy_or_zero<8>(into, from[j], live[j]);
                    } else {
                        copy_or_zero<4>(into, from[j], live[j]);
                        copy_or_zero<4>(into + 4u, tail ? from[j] + 4u : from[j], tail);
                    }
                    from[j] += kRowBytes;
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(eb::smem_u32(&full[s])) : "memory");
                ring.advance(stages);
                first_round = first_round && ring.stage != 0u;
            }
        });
        eb::cp_async_wait_all();
    }
    // tensor memory: the accumulators, the stages' weight scales [and activation scales], the resident rows' scales
    const uint32_t buffers = group.buffers, acc_columns = layout.n;
    const uint32_t tm_scales = tmem + buffers * acc_columns;
    constexpr uint32_t kStageColumns = 16u + (kResident ? 0u : 16u);
    const uint32_t tm_rows = tm_scales + stages * kStageColumns;

    if (warp == 1) {
        const bool leader = eb::elect_one();
        auto instruction_of = [](uint32_t n) { return (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((kTile >> 4) << 24); };
        uint32_t instruction = instruction_of(layout.n);
        const uint64_t first_a = nvfp4n::tile_descriptor(smem), first_b = nvfp4n::tile_descriptor(smem + (kResident ? layout.off_rows : kCodeBytes));
        const uint16_t* held = nullptr;
        eb::Ring ring, accumulator;
        uint32_t stagings = 0;
        bool used = false;   // every accumulator has been used once
        for_tiles([&](const Tensor& t, uint32_t, uint32_t, uint32_t) {
            if (kResident && t.x != held) {
                held = t.x;
                wait(staged, stagings++ & 1u);
                const bool more = __any_sync(0xFFFFFFFFu, lane < rows && has_more(min(lane, rows - 1u)));
                instruction = instruction_of(more ? layout.n : layout.plain_n);
            }
            const uint32_t buffer = accumulator.stage;
            if (used) wait(&acc_empty[buffer], accumulator.parity ^ 1u);
            nvfp4n::tcgen05_fence_after();
            const uint32_t d = tmem + buffer * acc_columns;
            uint64_t b = first_b;
            for (uint32_t u = 0; u < mine; ++u) {
                const uint32_t s = ring.stage;
                wait(&scaled[s], ring.parity);   // the scale warps have seen the stage land
                nvfp4n::tcgen05_fence_after();
                const uint64_t a = first_a + (uint64_t)(s * layout.stage_bytes >> 4);
                const uint32_t sfa = tm_scales + s * kStageColumns;
                if (!kResident) b = first_b + (uint64_t)(s * layout.stage_bytes >> 4);
                if (leader) {
#pragma unroll
                    for (uint32_t j = 0; j < 4u; ++j) mma(d, a + 2u * j, b + 2u * j, instruction, sfa + 4u * j, kResident ? tm_rows : sfa + 16u + 4u * j, (uint32_t)((u | j) != 0u));
                    nvfp4n::mma_commit(&empty[s]);
                }
                __syncwarp();
                if (kResident) b += (uint64_t)(layout.columns * 128u >> 4);
                ring.advance(stages);
            }
            if (leader) nvfp4n::mma_commit(&acc_full[buffer]);
            __syncwarp();
            accumulator.advance(buffers);
            used = used || accumulator.stage == 0u;
        });
    } else if (warp >= 2u) {
        const uint32_t quarter = warp & 3u;
        const bool drains = warp >= 8u && warp < 12u, scales = warp >= 4u && warp < 8u;
        const uint32_t lanes = (quarter * 32u) << 16;
        const uint16_t* held = nullptr;
        const uint32_t stager = warp < 4u ? warp - 2u : warp - 6u;    // 0 .. 9 among the staging warps

        // A task of the staging: one unit of one row. A staging warp takes every kStagers / 32nd of them, row by row.
        struct Task {
            uint32_t row, unit;
        };
        const uint32_t divisor = max(mine, 1u), step_rows = kStagers / 32u / divisor, step_units = kStagers / 32u % divisor;
        const Task first_task = {stager / divisor, stager % divisor};

        auto slice_of = [&](const uint16_t* x) {
            return Slice{x, rows, k, unit_begin, mine, stager, lane, exponents, least, left, smem + layout.off_rows, layout.columns};
        };
        uint32_t odd_rows = 0u;   // bit m: the digits of row m leave values of the slice out
        uint32_t more_rows = 0u;  // or there are further ones

        // The digits of every row of the slice, by the staging warps. Taken by all of them at the same points of the tile list; the
        // draining warps come when every MMA that reads the digits held before is done.
        auto stage_rows = [&](const uint16_t* x, bool again) {
            // 8 values per lane. The first kHold loads of a warp are in flight together while it finds the rows' exponents; the pass
            // that writes the digits finds the values in L1.
            constexpr uint32_t kHold = 4;
            const Slice slice = slice_of(x);
            Task at = first_task;
            auto next = [&]() {
                at.row += step_rows;
                at.unit += step_units;
                if (at.unit >= mine) {
                    at.unit -= mine;
                    ++at.row;
                }
            };
            if (mine != 0u) {
                uint4 v[kHold];
#pragma unroll
                for (uint32_t i = 0; i < kHold; ++i, next()) v[i] = slice.load(at.row, at.unit);
                // Task i in v[0] when its turn comes: one copy of the code for all of them.
                auto turn = [&](const uint4& done) { v[0] = v[1], v[1] = v[2], v[2] = v[3], v[3] = done; };
                if (again) {
                    stagers_sync();
                    if (stager == 0u && lane < rows) exponents[lane] = kLeastExponent, least[lane] = 255u;
                    stagers_sync();
                }
                uint32_t i = 0;
#pragma unroll 1
                for (at = first_task; at.row < rows; next(), ++i) {
                    const uint4 values = i < kHold ? v[0] : slice.load(at.row, at.unit);
                    slice.find(at.row, values);
                    turn(values);
                }
                const bool held = i <= kHold;
#pragma unroll 1
                for (; i < kHold; ++i) turn(v[0]);
                stagers_sync();
                odd_rows = __ballot_sync(0xFFFFFFFFu, lane < rows && slice.leaves_out(lane & (kMaxRows - 1u)));
#pragma unroll 1
                for (at = first_task; at.row < rows; next()) {
                    const uint4 values = held ? v[0] : slice.load(at.row, at.unit);
                    slice.write(at.row, at.unit, values);
                    turn(values);
                }
                if (odd_rows != 0u) stage_again(slice, odd_rows);
                more_rows = odd_rows | __ballot_sync(0xFFFFFFFFu, lane < rows && has_more(lane & (kMaxRows - 1u)));
            }
            fence_async_proxy();
            __syncwarp();
            if (lane == 0) eb::mbar_arrive(staged);
        };

        if (!scales || !kResident) eb::pdl_wait();   // the weights' scales do not depend on the launch before
        if (scales) {
            if (kResident) {   // the scales of the digits' columns: ones, whatever the K block
                uint32_t ones[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) ones[i] = 0x38383838u;
                tmem_store<16>(tm_rows + lanes, ones);   // (of up to 192 columns: six words)
            }
            // ---- weight scales (and activation scales) of every stage to tensor memory ----
            eb::Ring ring;
            const uint32_t off = layout.stage_bytes - kScaleBytes;
            uint4 table = make_uint4(0u, 0u, 0u, 0u);
            const uint8_t* table_of = nullptr;
            int column_from[4] = {-1, -1, -1, -1};   // where this lane's columns' scales lie in a K block's two atoms
            for_tiles([&](const Tensor& t, uint32_t, uint32_t, uint32_t row_group) {
                if (!kResident) {
#pragma unroll
                    for (uint32_t c = 0; c < 4u; ++c) {
                        const uint32_t column = 32u * c + lane, term = column >= layout.columns ? 1u : 0u, row = column - term * layout.columns;
                        const uint32_t in_tile = row_group * kMaxColumns % nvfp4n::kTileM + row;
                        column_from[c] = column < layout.n ? (int)(term * nvfp4n::kAtom + nvfp4n::atom_byte(in_tile, 0)) : -1;
                    }
                }
                if (kTable && t.table != table_of) {
                    table_of = t.table;
                    table = *reinterpret_cast<const uint4*>(t.table);
                }
                for (uint32_t u = 0; u < mine; ++u, ring.advance(stages)) {
                    const uint32_t s = ring.stage;
                    wait(&full[s], ring.parity);
                    const uint8_t* at = smem + s * layout.stage_bytes + off + lane * 16u;
                    uint32_t r[kStageColumns];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {   // row 32 j + lane of the tile
                        const uint4 w = row_scales<kTable>(at + j * 512, table);
                        r[j] = w.x, r[4 + j] = w.y, r[8 + j] = w.z, r[12 + j] = w.w;
                    }
                    if (!kResident) {
                        // column 32 c + lane of K block j: a row of the first term, then (from layout.columns on) of the second
                        const uint8_t* atoms = smem + s * layout.stage_bytes + kCodeBytes + nvfp4n::kTerms * kBoxColumns * 128u;
#pragma unroll
                        for (int j = 0; j < 4; ++j)
#pragma unroll
                            for (int c = 0; c < 4; ++c) r[16 + 4 * j + c] = column_from[c] >= 0 ? *reinterpret_cast<const uint32_t*>(atoms + j * 1024 + column_from[c]) : 0u;
                    }
                    tmem_store<kStageColumns>(tm_scales + lanes + s * kStageColumns, r);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    nvfp4n::tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) eb::mbar_arrive(&scaled[s]);
                }
            });
        } else if (drains) {
            // ---- the sums: drain, send to the owners, add the slices ----
            // A CTA owns `owned` rows of a tile: where it finishes the sums of all slices. In the paired region half of them are
            // gate rows and the other half the up rows that match them.
            const uint32_t owned = kTile / split, half_owned = owned / 2u;
            const uint32_t local = quarter * 32u + lane;                        // this thread's row of the tile
            const uint32_t owner = paired ? (local & 63u) / half_owned : local / owned;
            const uint32_t place = paired ? (local >> 6) * half_owned + (local & 63u) % half_owned : local % owned;
            const uint32_t gather = eb::smem_u32(smem + layout.off_gather), width = layout.width, dt = tid - 256u;   // dt: 0 .. 127
            const uint32_t slot_bytes = layout.gather_bytes;
            if (exchange) eb::cluster_wait();                                   // the other CTAs' barriers exist
            // Exchange buffers. BF16 rows: [slice][activation row][owned row], one word at a time, neighbouring threads neighbouring
            // words. Quantized rows: [slice][owned row][pitch], 16 bytes at a time.
            const uint32_t peer_gather = (exchange ? eb::map_to_rank(gather, owner) : gather)
                    + (kResident ? rank * width * owned + place : (rank * owned + place) * layout.pitch) * 4u;
            const uint32_t peer_full = exchange ? eb::map_to_rank(eb::smem_u32(gather_full), owner) : 0u;
            const uint32_t exchanges = run_end - run_begin;                     // one per item
            const uint32_t outputs = paired ? half_owned : owned;               // output rows of a tile that this CTA writes: a power of two
            const uint32_t outputs_log = 31u - (uint32_t)__clz((int)outputs);
            const uint32_t out_stride = paired ? group.pair_rows : group.tensor[0].n;   // (quantized rows)
            float* row_scales = reinterpret_cast<float*>(exponents);            // quantized rows: of the item's activation rows
            // The item of exchange e, and the one whose slices are added while it is on its way.
            struct Place {
                uint16_t* y;
                uint32_t n, tile, first;   // the item's tile and first activation row
                float global;
            } now = {nullptr, 0u, 0u, 0u, 0.0f}, before = now;   // by value: read through a pointer, they arrive late
            uint32_t ti = 0, tile_first = 0;
            // bf16(silu(gate) * up) of two sums: the reference's expression (native/src/nvfp4_native/native.cuh:390-413)
            auto swiglu = [](float gate_sum, float up_sum) {
                const float gate = eb::bf16_bits_to_float(eb::float_to_bf16_bits(gate_sum)), up = eb::bf16_bits_to_float(eb::float_to_bf16_bits(up_sum));
                return eb::float_to_bf16_bits(__fmul_rn(__fdiv_rn(gate, __fadd_rn(1.0f, expf(-gate))), up));
            };
            for (uint32_t e = 0; e < exchanges + (exchange ? 1u : 0u); ++e) {
                before = now;
                if (e < exchanges) {
                    const uint32_t item = run_begin + e;
                    if (kResident)
                        while (item >= group.tensor[ti].tile_end) tile_first = group.tensor[ti++].tile_end;
                    const Tensor& t = group.tensor[ti];
                    now.y = t.y, now.n = t.n;
                    now.tile = kResident ? item - tile_first : item / group.row_groups;
                    now.first = kResident ? 0u : item % group.row_groups * kMaxColumns;
                    now.global = *t.global;   // requested before the wait for the sums
                    if (kResident && t.x != held) {
                        stage_rows(t.x, held != nullptr);
                        held = t.x;
                    }
                    const uint32_t buffer = buffers == 2u ? e & 1u : 0u, use = buffers == 2u ? e >> 1 : e, slot = e & (slots - 1u);
                    if (!kResident && !exchange) {   // the scales of the item's activation rows
                        drainers_sync();   // those of the item before have been read
                        if (dt < width) row_scales[dt] = now.first + dt < rows ? __fmul_rn(group.row_globals[now.first + dt], now.global) : 0.0f;
                        drainers_sync();
                    }
                    float beside[kMaxRows];   // of the odd rows: what their digits leave out, summed while the tensor core works
                    if (kResident && odd_rows != 0u) left_out<kTable>(t, slice_of(t.x), now.tile * kTile + local, odd_rows, beside);
                    wait(&acc_full[buffer], use & 1u);
                    nvfp4n::tcgen05_fence_after();
                    const uint32_t d = tmem + lanes + buffer * acc_columns;
                    if (exchange && e >= slots) eb::mbar_wait_cluster_or_fail(&gather_empty[slot], ((e >> slots_log) - 1u) & 1u, failed);
                    const uint32_t to = peer_gather + slot * slot_bytes, bar = peer_full + slot * 8u;
                    if constexpr (kResident) {
                        // This thread's sum of a row of the slice from the sums of its eight digits, in units of half the largest value's.
                        auto joined = [&](const uint32_t* r) {
                            float sum = __uint_as_float(r[7]);
#pragma unroll
                            for (int i = 6; i >= 0; --i) sum = __fmaf_rn(sum, 0.125f, __uint_as_float(r[i]));
                            return mine == 0u ? 0.0f : sum;
                        };
                        auto scaled_up = [&](uint32_t m, float sum) { return __fmul_rn(__fadd_rn(sum, sum), __uint_as_float(exponents[m] << 23)); };
#pragma unroll 1
                        for (uint32_t m = 0; m < rows; m += 2u) {   // two rows at a time (the columns of an odd last one's neighbour exist)
                            uint32_t r[16];
                            tmem_load_16(r, d + m * 8u);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                            const float one = scaled_up(m, joined(r)), two = scaled_up(min(m + 1u, kMaxRows - 1u), joined(r + 8));
                            if (((more_rows >> m) & 1u) == 0u) send_f32(to + m * owned * 4u, one, bar);
                            if (m + 1u < rows && ((more_rows >> m) & 2u) == 0u) send_f32(to + (m + 1u) * owned * 4u, two, bar);
                        }
#pragma unroll 1
                        for (uint32_t more = more_rows; more != 0u; more &= more - 1u) {   // rows with further digits, or values that those leave out
                            const uint32_t m = (uint32_t)__ffs((int)more) - 1u;
                            uint32_t r[8], q[4];
                            tmem_load_8(r, d + m * 8u);
                            tmem_load_4(q, d + rows * kDigits + m * kMoreDigits);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                            float sum = joined(r), rest = __uint_as_float(q[3]);
#pragma unroll
                            for (int i = 2; i >= 0; --i) rest = __fmaf_rn(rest, 0.125f, __uint_as_float(q[i]));
                            if (mine != 0u && has_more(m)) sum = __fmaf_rn(rest, 2.384185791015625e-07f, sum);   // 2^-22
                            const float value = scaled_up(m, sum);
                            send_f32(to + m * owned * 4u, (odd_rows >> m) & 1u ? __fadd_rn(value, beside[m]) : value, bar);
                        }
                    } else {
                        // eight columns of this thread's weight row: both terms' sums added
                        auto sums = [&](uint32_t h, float (&sum)[8]) {
                            uint32_t r[8], q[8];
                            tmem_load_8(r, d + h);
                            tmem_load_8(q, d + layout.columns + h);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int i = 0; i < 8; ++i) sum[i] = mine == 0u ? 0.0f : __fadd_rn(__uint_as_float(r[i]), __uint_as_float(q[i]));
                        };
                        if (exchange) {
#pragma unroll 2
                            for (uint32_t h = 0; h < width; h += 8u) {
                                float sum[8];
                                sums(h, sum);
                                send_f32x4(to + h * 4u, sum[0], sum[1], sum[2], sum[3], bar);
                                send_f32x4(to + h * 4u + 16u, sum[4], sum[5], sum[6], sum[7], bar);
                            }
                        } else {
                            // The whole sums. In the paired region the up rows (the upper two quarters) go to shared memory first.
                            float* mine_up = reinterpret_cast<float*>(smem + layout.off_gather) + (local & 63u) * layout.pitch;
                            if (paired) {
                                if (local >= 64u)
                                    for (uint32_t h = 0; h < width; h += 8u) {
                                        float sum[8];
                                        sums(h, sum);
                                        *reinterpret_cast<float4*>(mine_up + h) = make_float4(sum[0], sum[1], sum[2], sum[3]);
                                        *reinterpret_cast<float4*>(mine_up + h + 4u) = make_float4(sum[4], sum[5], sum[6], sum[7]);
                                    }
                                drainers_sync();
                            }
                            const uint32_t at = now.tile * (paired ? 64u : kTile) + local;
                            if (!paired || local < 64u) {
                                uint16_t* y = t.y + (uint64_t)now.first * out_stride + at;
#pragma unroll 2
                                for (uint32_t h = 0; h < width; h += 8u) {
                                    float sum[8];
                                    sums(h, sum);
#pragma unroll
                                    for (uint32_t i = 0; i < 8u; ++i) {   // a warp writes 32 neighbouring values
                                        const float scale = row_scales[h + i], value = __fmul_rn(sum[i], scale);
                                        const uint16_t bits = paired ? swiglu(value, __fmul_rn(mine_up[h + i], scale)) : eb::float_to_bf16_bits(value);
                                        if (now.first + h + i < rows && at < out_stride) y[(uint64_t)(h + i) * out_stride] = bits;
                                    }
                                }
                            }
                            if (paired) drainers_sync();   // the up sums have been read
                        }
                    }
                    nvfp4n::tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) eb::mbar_arrive(&acc_empty[buffer]);
                }
                if (exchange && e > 0u) {
                    // The slices of the exchange before, added in order; this CTA's share of the outputs.
                    const uint32_t last = e - 1u, slot = last & (slots - 1u);
                    if (dt == 0u) eb::mbar_arrive_expect_tx(&gather_full[slot], kResident ? slot_bytes : kTile * width * 4u);
                    eb::mbar_wait_cluster_or_fail(&gather_full[slot], (last >> slots_log) & 1u, failed);   // st.async of all CTAs of the cluster
                    const float* from = reinterpret_cast<const float*>(smem + layout.off_gather + slot * slot_bytes);
                    const uint32_t row0 = before.tile * (paired ? 64u : kTile) + rank * outputs;
                    if constexpr (kResident) {
#pragma unroll 1
                        for (uint32_t o = dt; o < outputs * width; o += 128u) {
                            const uint32_t row = o & (outputs - 1u), i = o >> outputs_log, at = row0 + row;
                            const float* p = from + i * owned + row;
                            float sum = p[0];
                            for (uint32_t q = 1; q < split; ++q) sum = __fadd_rn(sum, p[q * width * owned]);
                            if (at < before.n) before.y[(uint64_t)i * before.n + at] = (uint16_t)eb::bf16_pair(__fmul_rn(sum, before.global), 0.0f);   // keeps a NaN one
                        }
                    } else {
                        const uint32_t quads = width / 4u;
                        auto total = [&](uint32_t row, uint32_t quad) {
                            const float* p = from + row * layout.pitch + 4u * quad;
                            float4 sum = *reinterpret_cast<const float4*>(p);
                            for (uint32_t q = 1; q < split; ++q) {
                                const float4 part = *reinterpret_cast<const float4*>(p + q * owned * layout.pitch);
                                sum.x = __fadd_rn(sum.x, part.x), sum.y = __fadd_rn(sum.y, part.y), sum.z = __fadd_rn(sum.z, part.z), sum.w = __fadd_rn(sum.w, part.w);
                            }
                            return sum;
                        };
#pragma unroll 2
                        for (uint32_t o = dt; o < outputs * quads; o += 128u) {   // four columns of a row; neighbouring threads neighbouring rows
                            const uint32_t row = o & (outputs - 1u), quad = o >> outputs_log, at = row0 + row;
                            const float4 sum = total(row, quad), up = paired ? total(half_owned + row, quad) : sum;
                            const float sums[4] = {sum.x, sum.y, sum.z, sum.w}, ups[4] = {up.x, up.y, up.z, up.w};
#pragma unroll
                            for (uint32_t i = 0; i < 4u; ++i) {
                                const uint32_t column = before.first + 4u * quad + i;
                                if (column >= rows || at >= out_stride) continue;
                                const float scale = __fmul_rn(group.row_globals[column], before.global), value = __fmul_rn(sums[i], scale);
                                before.y[(uint64_t)column * out_stride + at] = paired ? swiglu(value, __fmul_rn(ups[i], scale)) : eb::float_to_bf16_bits(value);
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0 && last + slots < exchanges) eb::mbar_arrive(&gather_read[slot]);   // warp 2 passes it on
                }
            }
        } else if (kResident || (warp == 2u && exchange)) {
            // Warp 2 also tells the cluster which exchange buffers of this CTA may be filled again: the draining warps have read them. An
            // arrive that releases memory to another CTA waits for the thread's global stores, and the draining warps have some in
            // flight: by them, 34816 x 5120 at one row took 26.8 us instead of 21.4 without the release. Nobody waits for the last signals, so they
            // are not sent: what a CTA is sent it waits for, and no CTA needs to outlive its own last wait.
            const bool passes = warp == 2u && exchange;
            const uint32_t exchanges = run_end - run_begin;
            if (passes) eb::cluster_wait();   // the other CTAs' barriers exist
            for_tiles([&](const Tensor& t, uint32_t, uint32_t e, uint32_t) {
                if (kResident && t.x != held) {
                    stage_rows(t.x, held != nullptr);
                    held = t.x;
                }
                if (passes && e > 0u && e - 1u + slots < exchanges) {
                    const uint32_t last = e - 1u;
                    wait(&gather_read[last & (slots - 1u)], (last >> slots_log) & 1u);
                    if (lane < split) nvfp4n::signal_rank(&gather_empty[last & (slots - 1u)], lane);
                    __syncwarp();
                }
            });
        }
    }
    nvfp4n::tcgen05_fence_before();
    __syncthreads();
    if (*failed != 0u) {   // a wait gave up: stay until the other CTAs of the cluster, which may still write here, are done too
        if (tid == 0) atomicOr(error, 1u);
        if (exchange) {
            if (warp != 2u && (warp < 8u || warp >= 12u)) eb::cluster_wait();   // warp 2 and the draining warps have taken this phase already
            __syncwarp();
            eb::cluster_sync();
        }
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(group.tmem_columns) : "memory");
}

// ---- host side ------------------------------------------------------------------------------------------------------------

using Kernel = void (*)(const Group, uint32_t*);
inline Kernel kernel_of(bool resident, bool table) {
    return resident ? (table ? kernel<true, true> : kernel<true, false>) : (table ? kernel<false, true> : kernel<false, false>);
}

constexpr uint32_t kSharedLimit = 227u * 1024u;

inline cudaError_t initialize() {
    for (int i = 0; i < 4; ++i) {
        const cudaError_t e = cudaFuncSetAttribute(kernel_of(i & 1, i & 2), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSharedLimit);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

struct Plan {
    uint32_t split, stages, shared, tmem, buffers, slots;
};

// Whether a launch of `rows` rows over clusters of `split` fits, and how deep its ring is: as many stages as an SM's shared and tensor
// memory hold, at least three. One CTA per SM: two with half the ring each measured 5 to 30 % slower on every shape but the
// smallest (34816 x 5120, 1 row: 24.7 us against 22.6).
inline bool plan(bool resident, uint32_t rows, uint32_t k, uint32_t split, bool paired, Plan* out) {
    const uint32_t units = units_of(k), units_cta = (units + split - 1u) / split;
    if (rows == 0u || (resident && (rows > kMaxRows || rows * units_cta > kLeftWords))) return false;
    for (uint32_t slots = resident ? kMostSlots : kFewSlots; slots >= kFewSlots; slots >>= 1)
        for (uint32_t stages = kMaxStages; stages >= 3u; --stages)
            for (uint32_t buffers = 2; buffers >= 1u; --buffers) {
                const Layout layout(resident, rows, units_cta, stages, split, paired, slots);
                const uint32_t columns = buffers * layout.n + stages * (resident ? 16u : 32u) + (resident ? 16u : 0u);
                if (layout.bytes <= kSharedLimit && columns <= kTmemColumns) {
                    *out = {split, stages, layout.bytes, columns <= 128u ? 128u : columns <= 256u ? 256u : 512u, buffers, slots};
                    return true;
                }
            }
    return false;
}

inline bool plan_rows(uint32_t rows, uint32_t k, Plan* out) { return plan(true, rows, k, split_of(units_of(k)), false, out); }

inline bool takes(uint32_t k, uint32_t n) {
    Plan p;
    return n != 0 && n % 16u == 0 && k != 0 && k % 128u == 0 && plan_rows(1, k, &p);
}

// The tensor map of the code plane of the weight tensors the calling thread used last, with whether the weights are plain device
// memory: tensor maps address device memory only, so anything else (host-mapped, managed) is kept off this path, as the
// reference keeps such weights off its TMA kernels (core/.../gpu/ExecutionGpu.java:398-402). A map holds only the address and the
// shape, so a stale entry for a reused address is still the right map. Null: the encoder failed.
inline const CUtensorMap* codes_map(const void* w, uint32_t n, uint32_t k, bool* device_memory) {
    struct alignas(64) Cached {
        CUtensorMap map;
        const void* weights;
        uint32_t n, k;
        int device;
        bool plain;
    };
    constexpr uint32_t kCached = 512;
    thread_local std::vector<Cached> cache(kCached);
    int device = 0;
    (void)cudaGetDevice(&device);
    Cached& slot = cache[(uint32_t)(((uintptr_t)w >> 8) * 0x9E3779B1u >> 16) % kCached];
    if (slot.weights != w || slot.n != n || slot.k != k || slot.device != device) {
        cudaPointerAttributes attributes;
        const bool plain = cudaPointerGetAttributes(&attributes, w) == cudaSuccess && attributes.type == cudaMemoryTypeDevice;
        (void)cudaGetLastError();
        slot.weights = nullptr;
        if (plain) {
            const eb::EncodeTiled encode = eb::encoder();
            const cuuint64_t dims[2] = {k / 2u, n}, strides[1] = {k / 2u};
            const cuuint32_t box[2] = {128u, kTile / 2u}, ones[2] = {1u, 1u};
            if (encode == nullptr
                    || encode(&slot.map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(w), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                            != CUDA_SUCCESS)
                return nullptr;
        }
        slot.weights = w;
        slot.n = n;
        slot.k = k;
        slot.device = device;
        slot.plain = plain;
    }
    *device_memory = slot.plain;
    return &slot.map;
}

struct Item {
    const void* x;
    const void* w;
    void* y;
    uint32_t n;
};

// cudaErrorNotSupported: a tensor's weights are not plain device memory.
inline cudaError_t fill_tensor(Tensor* t, const Item& item, uint32_t k, bool table) {
    bool device_memory = false;
    const CUtensorMap* map = codes_map(item.w, item.n, k, &device_memory);
    if (map == nullptr) return cudaErrorInvalidValue;
    if (!device_memory) return cudaErrorNotSupported;
    const uint8_t* w = static_cast<const uint8_t*>(item.w);
    const uint64_t plane = nvfp4n::align256((uint64_t)item.n * (k / 2u)), after = nvfp4n::align256(plane + (uint64_t)item.n * (k / (table ? 32u : 16u)));
    t->codes = *map;
    t->x = static_cast<const uint16_t*>(item.x);
    t->weights = w;
    t->scales = w + plane;
    t->table = table ? w + after : nullptr;
    t->global = reinterpret_cast<const float*>(w + after + (table ? 16u : 0u));
    t->y = static_cast<uint16_t*>(item.y);
    t->n = item.n;
    return cudaSuccess;
}

// Clusters that the current device holds at once, at most the SMs' number of CTAs. 0: none, or there is no device.
inline uint32_t most_clusters(bool resident, bool table, const Plan& p, int sms) {
    const uint32_t most = (uint32_t)sms / p.split;
    return p.split == 1u ? most : std::min(most, eb::resident_clusters(reinterpret_cast<const void*>(kernel_of(resident, table)), kThreads, p.shared, p.split));
}

inline cudaError_t launch(bool resident, bool table, Group* group, const Plan& p, int sms, cudaStream_t stream, bool pdl, uint32_t* error) {
    group->stages = p.stages;
    group->split = p.split;
    group->tmem_columns = p.tmem;
    group->buffers = p.buffers;
    group->slots = p.slots;
    group->scale_row_bytes = group->k / (table ? 32u : 16u);
    const Kernel kernel = kernel_of(resident, table);
    const uint32_t most = most_clusters(resident, table, p, sms);
    if (most == 0u) return cudaErrorInvalidConfiguration;
    const uint32_t clusters = std::min(most, group->tiles);
    return eb::launch_on(stream, pdl, p.split, kernel, dim3(clusters * p.split), dim3(kThreads), p.shared, *group, error);
}

// `count` (at most kMaxGroup) tensors that share K: BF16 rows in groups of at most kMaxRows, fewer when their digits do not fit beside
// the ring. Every row is independent of the others.
inline cudaError_t decode(const Item* items, uint32_t count, uint32_t rows, uint32_t k, bool table, int sms, cudaStream_t stream, bool pdl, uint32_t* error) {
    Group group = {};
    group.k = k;
    group.count = count;
    group.row_groups = 1;
    for (uint32_t i = 0; i < count; ++i) {
        const cudaError_t e = fill_tensor(&group.tensor[i], items[i], k, table);
        if (e != cudaSuccess) return e;
        group.tiles += (items[i].n + kTile - 1u) / kTile;
        group.tensor[i].tile_end = group.tiles;
    }
    // equal shares of the rows, so that no launch of a call is left with a single row
    uint32_t launches = (rows + kMaxRows - 1u) / kMaxRows;
    Plan p;
    while (!plan_rows((rows + launches - 1u) / launches, k, &p)) {
        if (launches >= rows) return cudaErrorInvalidConfiguration;
        ++launches;
    }
    for (uint32_t l = 0; l < launches; ++l) {
        const uint32_t first = l * rows / launches, now = (l + 1u) * rows / launches - first;
        for (uint32_t i = 0; i < count; ++i) {
            group.tensor[i].x = static_cast<const uint16_t*>(items[i].x) + (uint64_t)first * k;
            group.tensor[i].y = static_cast<uint16_t*>(items[i].y) + (uint64_t)first * items[i].n;
        }
        group.rows = now;
        if (!plan_rows(now, k, &p)) return cudaErrorInvalidConfiguration;
        const cudaError_t e = launch(true, table, &group, p, sms, stream, pdl, error);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Columns of an item for quantized rows.
inline uint32_t columns_of(uint32_t rows) { return Layout(false, rows, 1u, 1u, 1u, false, kFewSlots).columns; }

// Whether this kernel takes a native call of `rows` quantized rows rather than the large GEMM (nvfp4_native.cuh), by what each keeps
// an SM busy with: per unit of K the GEMM spends about 1080 cycles on an output tile of 128 rows x 256 columns and leaves the SMs
// without a tile of the last wave idle; this kernel spends about 900 on 128 columns x 128 rows (shared-memory bandwidth) but
// spreads a call evenly. Up to one group of rows it always wins.
inline bool better_for(uint32_t rows, uint32_t k, uint32_t out_features, bool paired, uint32_t sms) {
    Plan p;
    if (!plan(false, rows, k, 8u, paired, &p)) return false;
    if (rows <= kMaxColumns) return true;
    const uint32_t gemm_tiles = (rows + 127u) / 128u * (paired ? out_features / 256u : (out_features + 255u) / 256u);
    const uint64_t gemm = (uint64_t)((gemm_tiles + sms - 1u) / sms) * sms * 1080u;
    const uint64_t here = (uint64_t)(out_features + 127u) / 128u * ((rows + kMaxColumns - 1u) / kMaxColumns) * 1000u;
    return here < gemm;
}

// One linear (or paired region) over the rows quantized into the scratch; map_a: the code planes with a box of 128 bytes x the
// item's columns.
inline cudaError_t quantized(const void* weights, void* output, const CUtensorMap& activations, const uint8_t* atoms, const float* row_globals, uint32_t rows,
        uint32_t k, uint32_t out_features, bool paired, bool table, int sms, cudaStream_t stream, bool pdl, uint32_t* error) {
    Group group = {};
    group.k = k;
    group.count = 1;
    group.rows = rows;
    const Item item = {nullptr, weights, output, out_features};
    const cudaError_t e = fill_tensor(&group.tensor[0], item, k, table);
    if (e != cudaSuccess) return e;
    group.activations = activations;
    group.atoms = atoms;
    group.row_globals = row_globals;
    group.row_groups = (rows + kMaxColumns - 1u) / kMaxColumns;
    group.pair_rows = paired ? out_features / 2u : 0u;
    group.tiles = (paired ? out_features / 128u : (out_features + kTile - 1u) / kTile) * group.row_groups;
    group.tensor[0].tile_end = group.tiles;
    Plan p;
    // Clusters only where the items alone leave SMs idle.
    uint32_t split = 1u;
    while (split < 8u && group.tiles * split * 2u <= (uint32_t)sms * 7u / 8u && split * 2u <= units_of(k)) split *= 2u;
    if (!plan(false, rows, k, split, paired, &p)) return cudaErrorInvalidConfiguration;
    return launch(false, table, &group, p, sms, stream, pdl, error);
}

}  // namespace nvfp4d

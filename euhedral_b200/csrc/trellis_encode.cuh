// Trellis tile encoder on sm_100a: quantizes 256-weight tiles to the tail-biting ring of 16-bit states that
// trellis.cuh decodes (the converter's side of the trellis-tile16-v1 format; the reference's encoder is
// quantization/src/main/resources/cuda/trellis.cu:34-399, from exllamav3's Viterbi kernels).
//
// The search is fixed by the format's golden tiles, so its arithmetic is the contract: position i brings
// d(i) = ka + [i odd][half-step rate] new bits; a node is the top 16 - d bits of a state; the cost of reaching node v at
// a position is the least, over the 2^d states that end in v, of fp16 fma(e, e, cost of the state's predecessor node)
// with e = fp16(value(state) - w) (first position: fp16(e * e)), the lowest predecessor on equal costs. Two passes: from
// an open start at position 128 all round, the best end node (ties by a bit-reversed rank of the node) traced back to
// the node that enters position 0; then from position 0 pinned to that node, traced back in full.
//
// How it runs here (2 to 4 bits, register_kernel): one CTA per SM. Its 512 searching threads hold the codebook value of every one of
// the 65,536 states in REGISTERS for good: thread t has the 128 states whose bits 3 to 11 are t, as 64 FP16 pairs of neighbouring
// nodes. At every rate from 2 to 4 bits a position's nodes then need nothing but their predecessors' costs, which the threads
// exchange through two rows in shared memory, one barrier a position. A step keeps the least cost only (one packed minimum a
// predecessor); which predecessor won is not kept but found again on the way back, from the costs of every second position, which
// go to a slab in global memory: a warp of its own walks back two positions at a time, all 2^(d + d') paths side by side, while
// the searching warps do a pass of another tile. So two tiles are in flight in a CTA, pass by pass in turn.
// Bound: packed FP16 arithmetic, which one of the two FMA pipes does at two cycles an instruction: a subtraction and a fused
// multiply-add per pair of states, 1024 cycles a position and tile. The kernel for more bits (viterbi_kernel) reads the values from
// shared memory for each position and selects winners with logic instructions, seven instructions per pair; 2 to 4 bits ran on it
// before. 4096 tiles at 2 / 2.5 / 3 / 3.5 / 4 bits 22.1 / 23.7 / 15.6 / 16.1 / 16.8 -> 9.9 / 10.2 / 10.1 / 10.1 / 10.2 ms (2 and 2.5 bits in half the
// scratch 19.4 and 20.3); 1024 x 1024 weights at 3 bits (4096 tiles and 1800 of the scale's search): 25.4 -> 17.1 ms.
//
// 5 and 6 bits (viterbi_kernel; a thread's states there would not share predecessors in registers): one CTA per SM, 1024 threads,
// persistent over the tile list. The CTA first writes the codebook value of every state to shared memory (128 KB of FP16) - a
// state's neighbours sit side by side there. The threads then work as two groups of 512 that encode tiles independently of each
// other (a named barrier per group): a group keeps its two cost rows in shared memory as FP16; a thread takes runs of 2 or 4
// neighbouring nodes, which share their predecessors, reads their values with one load per predecessor and updates their costs
// with packed FP16 arithmetic and bit selects. The history - one byte per position and node: which of the 2^d states won - goes
// to a slab of the group in global memory and one thread of the group walks it back; while it does, the other group has the SM's
// issue slots. No waits on other CTAs.
#pragma once

#include "common.cuh"
#include "trellis_codebook.cuh"

namespace trellis_encode {

constexpr int kThreads = 1024;
constexpr uint32_t kInfinity = 0x7C00u;
constexpr uint32_t kTableBytes = 65536u * 2u;

// The bits a position brings.
__host__ __device__ constexpr int position_bits(int position, int ka, bool half_step) { return ka + ((half_step && (position & 1)) ? 1 : 0); }

// Bytes of a tile's slab: 256 positions x the most nodes of a position a byte each (which state won), or FP16 costs of every second one.
__host__ __device__ constexpr uint64_t history_bytes(int ka) { return 256ull * (65536ull >> ka); }

constexpr int kGroups = 2;   // tiles of a CTA in flight

// ---- 2 to 4 bits ---------------------------------------------------------------------------------------------------------

constexpr int kSearchers = 512, kRegisterThreads = kSearchers + 32;
constexpr int kHigh = 4, kLow = 3;   // a thread's states: all values of the state's four highest and three lowest bits

__host__ __device__ constexpr uint32_t register_shared_bytes(int ka) { return 4u * (65536u >> ka); }   // two cost rows

__device__ __forceinline__ void searchers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kSearchers) : "memory"); }
// The searching warps and the one that walks back hand a pass over on barriers 2 and 3 (by the pass's parity) and its end on 4 and 5.
__device__ __forceinline__ void meet(uint32_t barrier) { asm volatile("bar.sync %0, %1;" ::"r"(barrier), "n"(kRegisterThreads) : "memory"); }
__device__ __forceinline__ void announce(uint32_t barrier) { asm volatile("bar.arrive %0, %1;" ::"r"(barrier), "n"(kRegisterThreads) : "memory"); }

__device__ __forceinline__ __half2 as_half2(uint32_t bits) { return *reinterpret_cast<const __half2*>(&bits); }
__device__ __forceinline__ uint32_t as_bits(__half2 pair) { return *reinterpret_cast<const uint32_t*>(&pair); }

// Thread t's part of a step: the costs of its nodes after a position that brings KIN bits, the next one KOUT.
//   values[hi][j]: of the states hi << 12 | t << 3 | 2 j, + 1. A node is a state's lower 16 - KOUT bits, so the top 4 - KOUT bits
//   of its twelfth and higher are fixed here with `high` and the predecessor s takes the rest of hi; eight nodes are neighbours.
template <int KIN, int KOUT, bool kFirst>
__device__ __forceinline__ void register_step(const uint32_t (&values)[1 << kHigh][4], const __half* __restrict__ before, __half* __restrict__ after,
        __half* __restrict__ kept, __half w, int pinned, int t) {
    static_assert(KIN >= 2 && KIN <= 4 && KOUT >= 2 && KOUT <= 4, "");
    const __half2 w2 = __half2half2(w);
#pragma unroll
    for (int high = 0; high < 1 << (kHigh - KOUT); ++high) {
        uint32_t best[4];
#pragma unroll
        for (int s = 0; s < 1 << KOUT; ++s) {
            const int hi = s << (kHigh - KOUT) | high;
            const int from = KIN == 2 ? hi << 10 | t << 1 : hi << (12 - KIN) | t >> (KIN - 3);   // KIN 2: of the first four nodes, + 1 of the others
            __half2 previous[2];
            if (!kFirst) {
                if (KIN == 2) {
                    const __half2 both = *reinterpret_cast<const __half2*>(before + from);
                    previous[0] = __low2half2(both), previous[1] = __high2half2(both);
                } else {
                    previous[0] = previous[1] = __half2half2(before[from]);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __half2 e = __hsub2(as_half2(values[hi][j]), w2);
                uint32_t cost;
                if (kFirst) cost = pinned >= 0 && from + (KIN == 2 ? j >> 1 : 0) != pinned ? kInfinity | kInfinity << 16 : as_bits(__hmul2(e, e));
                else cost = as_bits(__hfma2(e, e, previous[j >> 1]));
                best[j] = s == 0 ? cost : as_bits(__hmin2(as_half2(cost), as_half2(best[j])));
            }
        }
        const int node = high << 12 | t << 3;
        const uint4 eight = make_uint4(best[0], best[1], best[2], best[3]);
        *reinterpret_cast<uint4*>(after + node) = eight;
        if (kept != nullptr) __stcg(reinterpret_cast<uint4*>(kept + node), eight);
    }
}

// Walks back over two positions from `node` after the odd position `position` (taken by a whole warp). kept: the costs before the even
// position in front of it, or null where that is the pass's first, entered at `pinned`. Returns the two states, the even position's in
// the upper half. On equal costs the lowest predecessor wins, of the odd position before the even one's, as the search is defined. A NaN
// cost is less than none: behind a NaN weight all costs of a position are NaN or infinite, and the lowest predecessors win. They do here,
// where all are one or the other; only at a pass's first position does one path with the weight's NaN stand beside infinite ones.
template <int KA, int KB>
__device__ __forceinline__ uint32_t two_back(const __half* __restrict__ kept, const __half* weights, int position, uint32_t node, int pinned, int lane) {
    constexpr int kLanes = 32 >> KA, kEach = (1 << KB) > kLanes ? (1 << KB) / kLanes : 1;   // lanes of an odd predecessor; paths of a lane
    const uint32_t odd = (uint32_t)lane / kLanes, odd_state = odd << (16 - KA) | node, between = odd_state >> KB;
    const __half w_even = weights[position - 1], w_odd = weights[position];
    __half before[kEach];
#pragma unroll
    for (int m = 0; m < kEach; ++m) {
        const uint32_t even = (uint32_t)(lane % kLanes + m * kLanes), state = (even << (16 - KB) | between) & 0xFFFFu;
        before[m] = kept != nullptr ? __ldcg(kept + (state >> KA)) : __ushort_as_half(0);
    }
    uint32_t least = 0xFFFFFFFFu;   // cost << 16 | predecessor
#pragma unroll
    for (int m = 0; m < kEach; ++m) {
        const uint32_t even = (uint32_t)(lane % kLanes + m * kLanes), state = (even << (16 - KB) | between) & 0xFFFFu;
        const __half e = __hsub(__ushort_as_half(trellis::value_bits(state)), w_even);
        uint32_t cost;
        if (kept != nullptr) cost = __half_as_ushort(__hfma(e, e, before[m]));
        else cost = pinned >= 0 && (int)(state >> KA) != pinned ? kInfinity : min((uint32_t)__half_as_ushort(__hmul(e, e)), kInfinity);   // NaN: no less
        if (even < 1u << KB) least = min(least, cost << 16 | even);
    }
#pragma unroll
    for (int d = 1; d < kLanes; d <<= 1) least = min(least, __shfl_xor_sync(0xFFFFFFFFu, least, d));
    const __half e = __hsub(__ushort_as_half(trellis::value_bits(odd_state)), w_odd);
    const uint32_t cost = __half_as_ushort(__hfma(e, e, __ushort_as_half((unsigned short)(least >> 16))));
    const uint32_t won = __reduce_min_sync(0xFFFFFFFFu, cost << 16 | odd << 8 | (least & 0xFFu));
    const uint32_t last = ((won >> 8) & 0xFFu) << (16 - KA) | node;
    return ((won & 0xFFu) << (16 - KB) | last >> KB) << 16 | last;
}

__device__ __forceinline__ uint32_t reverse5(uint32_t v) { return __brev(v) >> 27; }

// tiles f32 [count][256] -> states u16 [count][256] (and, when asked for, their codebook values as f32). slabs: history_bytes(KA) bytes
// per tile in flight, at most count of them, on a 16-byte boundary; the last row of the last one (2 (65536 >> KA) bytes) is not touched.
//   grid: at most count CTAs (CTA b takes tiles b, b + gridDim.x, ...; two at a time), block kRegisterThreads, dynamic shared
//   register_shared_bytes(KA).
template <int KA, bool kHalfStep>
__global__ void __launch_bounds__(kRegisterThreads, 1) register_kernel(const float* __restrict__ tiles, uint32_t count, uint16_t* __restrict__ states,
        float* __restrict__ decoded, uint8_t* __restrict__ slabs) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int kMost = 65536 >> KA, KB = kHalfStep ? KA + 1 : KA;   // an even position brings KA bits, an odd one KB
    __shared__ __align__(4) __half weights[kGroups][256];
    __shared__ uint32_t warp_best[kGroups][kSearchers / 32];
    __shared__ int entered[kGroups];   // the node that a tile's second pass enters position 0 from
    const int t = threadIdx.x, lane = t & 31;
    // Pass n: of the CTA's tiles 2 (n / 4) and 2 (n / 4) + 1 in turn; n / 2 odd: the second pass. A CTA's last tile may be without a
    // partner, whose passes are then empty.
    const uint32_t mine = (count - blockIdx.x + gridDim.x - 1u) / gridDim.x, passes = (mine + 1u) / 2u * 4u;
    auto tile_of = [&](uint32_t n) { return blockIdx.x + (uint64_t)((n >> 2) * 2u + (n & 1u)) * gridDim.x; };
    auto slab_of = [&](uint32_t n) { return reinterpret_cast<__half*>(slabs + (blockIdx.x + (uint64_t)(n & 1u) * gridDim.x) * history_bytes(KA)); };

    if (t < kSearchers) {
        uint32_t values[1 << kHigh][4];
#pragma unroll
        for (int hi = 0; hi < 1 << kHigh; ++hi)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t state = (uint32_t)(hi << 12 | t << 3 | 2 * j);
                values[hi][j] = trellis::value_pair(state, state + 1u);
            }
        __half *row_even = reinterpret_cast<__half*>(smem), *row_odd = row_even + kMost;   // costs after an even and an odd position
#pragma unroll 1
        for (uint32_t n = 0; n < passes; ++n) {
            const uint32_t slot = n & 1u, second = (n >> 1) & 1u;
            if (n >= 2u) meet(4u + slot);   // the way back of pass n - 2 has been walked: its slab, weights and result
            if (tile_of(n) < count) {
                if (second == 0u && t < 256) weights[slot][t] = __float2half_rn(tiles[tile_of(n) * 256u + (uint32_t)t]);
                searchers_sync();
                const int pinned = second != 0u ? entered[slot] : -1, roll = second != 0u ? 0 : 128;
                __half* slab = slab_of(n);
#pragma unroll 1
                for (int i = 0; i < 256; i += 2) {
                    const __half2 w = *reinterpret_cast<const __half2*>(&weights[slot][(i + roll) & 255]);
                    if (i == 0) register_step<KA, KB, true>(values, row_odd, row_even, nullptr, __low2half(w), pinned, t);
                    else register_step<KA, KB, false>(values, row_odd, row_even, nullptr, __low2half(w), pinned, t);
                    searchers_sync();
                    const bool keeps = i < 254 && (second != 0u || i >= 126);   // what the way back reads: never a slab's last row
                    register_step<KB, KA, false>(values, row_even, row_odd, keeps ? slab + (size_t)(i >> 1) * kMost : nullptr, __high2half(w), pinned, t);
                    searchers_sync();
                }
                if (second == 0u) {
                    // the best node after position 127 (the open pass's last), ties by the rank of the node
                    uint32_t best = (kInfinity << 16) | 0xFFFFu;
                    for (int e = t; e < kMost; e += kSearchers) {
                        const uint32_t v = (uint32_t)e & 1023u;
                        const uint32_t rank = (reverse5(v >> 5) << 10) | (reverse5(v & 31u) << 5) | ((uint32_t)e >> 10);
                        best = min(best, ((uint32_t)__half_as_ushort(row_odd[e]) << 16) | rank);
                    }
                    best = __reduce_min_sync(0xFFFFFFFFu, best);
                    if (lane == 0) warp_best[slot][t >> 5] = best;
                }
            }
            announce(2u + slot);
        }
        // the ways back of the last two passes end on barriers that every thread must have come to
        for (uint32_t n = passes; n < passes + 2u; ++n) meet(4u + (n & 1u));
    } else {
#pragma unroll 1
        for (uint32_t n = 0; n < passes; ++n) {
            const uint32_t slot = n & 1u, second = (n >> 1) & 1u;
            meet(2u + slot);
            const uint64_t tile = tile_of(n);
            if (tile < count) {
                const __half* slab = slab_of(n);
                if (second == 0u) {
                    const uint32_t best = __reduce_min_sync(0xFFFFFFFFu, lane < kSearchers / 32 ? warp_best[slot][lane] : 0xFFFFFFFFu);
                    uint32_t node = 0;
                    if (best < (kInfinity << 16)) {
                        const uint32_t rank = best & 65535u;
                        node = ((rank & 31u) << 10) | (reverse5(rank >> 10) << 5) | reverse5((rank >> 5) & 31u);
                    }
                    // back through positions 127 .. 0 (steps 255 .. 128 of the pass) to the node that enters position 0
#pragma unroll 1
                    for (int position = 127; position > 0; position -= 2)
                        node = two_back<KA, KB>(slab + (size_t)((position + 126) >> 1) * kMost, weights[slot], position, node, -1, lane) >> (16 + KA);
                    if (lane == 0) entered[slot] = (int)node;
                } else {
                    const int pinned = entered[slot];
                    uint32_t node = (uint32_t)pinned;
#pragma unroll 1
                    for (int position = 255; position > 0; position -= 2) {
                        const uint32_t both = two_back<KA, KB>(position > 1 ? slab + (size_t)((position - 2) >> 1) * kMost : nullptr, weights[slot], position,
                                node, pinned, lane);
                        if (lane < 2) {
                            const uint32_t state = lane == 0 ? both >> 16 : both & 0xFFFFu;
                            const uint64_t at = tile * 256u + (uint32_t)(position - 1 + lane);
                            states[at] = (uint16_t)state;
                            if (decoded != nullptr) decoded[at] = __half2float(__ushort_as_half(trellis::value_bits(state)));
                        }
                        node = both >> (16 + KA);
                    }
                }
            }
            __syncwarp();
            announce(4u + slot);
        }
    }
}

// ---- 5 and 6 bits --------------------------------------------------------------------------------------------------------

// Dynamic shared memory of a CTA: the value table, then per group two cost rows and the tile's 256 weights.
__host__ __device__ constexpr uint32_t shared_bytes(int ka) { return kTableBytes + (uint32_t)kGroups * (4u * (65536u >> ka) + 512u); }

template <int GROUP_THREADS>
__device__ __forceinline__ void group_sync(int group) {
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(GROUP_THREADS) : "memory");
}

// Nodes a thread takes at a time: they must share their predecessors (2^KIN neighbours do) and there should be at least
// as many runs as threads.
template <int KA, int GROUP_THREADS>
struct Run {
    static constexpr int kNodes = 65536 >> KA;
    static constexpr int value = kNodes / GROUP_THREADS >= 4 ? 4 : 2;   // 2^KA neighbours share theirs: more than that
};

// One step of a pass: costs of the nodes after a position from the costs before it. `table`: FP16 value of every state.
template <int KA, int GROUP_THREADS, bool kFirst>
__device__ __forceinline__ void step(const __half* __restrict__ table, const __half* __restrict__ before, __half* __restrict__ after,
        uint8_t* __restrict__ history_row, __half w, int pinned, bool write, int tid) {
    constexpr int kShift = 16 - KA, kNodes = 65536 >> KA, kStates = 1 << KA;
    constexpr int G = Run<KA, GROUP_THREADS>::value, H = G / 2;
    const __half2 w2 = __half2half2(w);
    const uint32_t infinity = kInfinity | kInfinity << 16;
    for (int run = tid; run < kNodes / G; run += GROUP_THREADS) {
        const int node = run * G, from_low = node >> KA;   // the G nodes of the run have the same predecessors
        uint32_t best[H], winner[H];
#pragma unroll
        for (int s = 0; s < kStates; ++s) {
            const uint32_t state = ((uint32_t)s << kShift) | (uint32_t)node;
            const int from = (s << (kShift - KA)) | from_low;
            uint32_t values[H];
            if constexpr (G == 4) {
                const uint2 v = *reinterpret_cast<const uint2*>(table + state);
                values[0] = v.x, values[1] = v.y;
            } else {
                values[0] = *reinterpret_cast<const uint32_t*>(table + state);
            }
            __half2 previous;
            if (!kFirst) previous = __half2half2(before[from]);
#pragma unroll
            for (int j = 0; j < H; ++j) {
                const __half2 e = __hsub2(*reinterpret_cast<const __half2*>(&values[j]), w2);
                uint32_t cost;
                if (kFirst) {
                    const __half2 square = __hmul2(e, e);
                    cost = pinned >= 0 && from != pinned ? infinity : *reinterpret_cast<const uint32_t*>(&square);
                } else {
                    const __half2 sum = __hfma2(e, e, previous);
                    cost = *reinterpret_cast<const uint32_t*>(&sum);
                }
                if (s == 0) {
                    best[j] = cost;
                    winner[j] = 0;
                } else {
                    // strictly less, half by half: the lowest state keeps a tie
                    const uint32_t less = __hlt2_mask(*reinterpret_cast<const __half2*>(&cost), *reinterpret_cast<const __half2*>(&best[j]));
                    best[j] = (cost & less) | (best[j] & ~less);
                    winner[j] = (((uint32_t)s * 0x00010001u) & less) | (winner[j] & ~less);
                }
            }
        }
        if constexpr (G == 4) {
            *reinterpret_cast<uint2*>(after + node) = make_uint2(best[0], best[1]);
            if (write) *reinterpret_cast<uint32_t*>(history_row + node) = __byte_perm(winner[0], winner[1], 0x6420);
        } else {
            *reinterpret_cast<uint32_t*>(after + node) = best[0];
            if (write) *reinterpret_cast<uint16_t*>(history_row + node) = (uint16_t)__byte_perm(winner[0], 0, 0x4420);
        }
    }
}

// As register_kernel. history: history_bytes(KA) bytes per group that has a tile.
//   grid: at most count CTAs (group g of CTA b takes tiles b + g gridDim.x, + gridDim.x kGroups, ...), block kThreads, dynamic shared
//   shared_bytes(KA).
template <int KA>
__global__ void __launch_bounds__(kThreads, 1) viterbi_kernel(const float* __restrict__ tiles, uint32_t count, uint16_t* __restrict__ states,
        float* __restrict__ decoded, uint8_t* __restrict__ history) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int kMost = 65536 >> KA;   // nodes of a position that brings KA bits
    constexpr int T = kThreads / kGroups;
    __shared__ uint32_t warp_best[kGroups][T / 32];
    __shared__ int node_shared[kGroups];
    const int group = threadIdx.x / T, tid = threadIdx.x - group * T;
    __half* table = reinterpret_cast<__half*>(smem);
    __half* row_a = reinterpret_cast<__half*>(smem + kTableBytes + (uint32_t)group * (4u * kMost + 512u));
    __half* row_b = row_a + kMost;
    __half* weights = row_b + kMost;
    uint8_t* slab = history + (blockIdx.x + (uint64_t)group * gridDim.x) * history_bytes(KA);

    for (uint32_t state = threadIdx.x; state < 65536u; state += kThreads) table[state] = __ushort_as_half(trellis::value_bits(state));
    __syncthreads();

    for (uint32_t tile = blockIdx.x + group * gridDim.x; tile < count; tile += gridDim.x * kGroups) {
        group_sync<T>(group);   // the tile before is done with the group's rows
        if (tid < 256) weights[tid] = __float2half_rn(tiles[(uint64_t)tile * 256u + (uint32_t)tid]);
        group_sync<T>(group);
        __half *before = row_a, *after = row_b;
        int pinned = -1;
        for (int pass = 0; pass < 2; ++pass) {
            const int roll = pass == 0 ? 128 : 0;
            for (int i = 0; i < 256; ++i) {
                const int ri = (i + roll) & 255;
                __half* swap = before;
                before = after;
                after = swap;
                const bool write = pass == 1 || ri < 128;
                uint8_t* row = slab + (uint64_t)ri * kMost;
                const __half w = weights[ri];
                if (i == 0) step<KA, T, true>(table, before, after, row, w, pinned, write, tid);
                else step<KA, T, false>(table, before, after, row, w, pinned, write, tid);
                group_sync<T>(group);
            }
            if (pass == 0) {
                // the best node after position 127 (the open pass's last), ties by the rank of the node
                uint32_t best = (kInfinity << 16) | 0xFFFFu;
                for (int e = tid; e < kMost; e += T) {
                    const uint32_t v = (uint32_t)e & 1023u;
                    const uint32_t rank = (reverse5(v >> 5) << 10) | (reverse5(v & 31u) << 5) | ((uint32_t)e >> 10);
                    best = min(best, ((uint32_t)__half_as_ushort(after[e]) << 16) | rank);
                }
                best = __reduce_min_sync(0xFFFFFFFFu, best);
                if ((tid & 31) == 0) warp_best[group][tid >> 5] = best;
                group_sync<T>(group);
                if (tid == 0) {
                    for (int i = 1; i < T / 32; ++i) best = min(best, warp_best[group][i]);
                    int node = 0;
                    if (best < (kInfinity << 16)) {
                        const uint32_t rank = best & 65535u;
                        node = (int)(((rank & 31u) << 10) | (reverse5(rank >> 10) << 5) | reverse5((rank >> 5) & 31u));
                    }
                    // back through positions 127 .. 0 to the node that enters position 0
                    for (int ri = 127; ri >= 0; --ri) {
                        const int s = slab[(uint64_t)ri * kMost + (uint32_t)node];
                        node = (s << (16 - 2 * KA)) | (node >> KA);
                    }
                    node_shared[group] = node;
                }
                group_sync<T>(group);
                pinned = node_shared[group];
            } else if (tid == 0) {
                int node = pinned;
                for (int ri = 255; ri >= 0; --ri) {
                    const int s = slab[(uint64_t)ri * kMost + (uint32_t)node];
                    const int from = (s << (16 - 2 * KA)) | (node >> KA);
                    const uint32_t state = (((uint32_t)from << KA) | (uint32_t)node) & 0xFFFFu;
                    states[(uint64_t)tile * 256u + (uint32_t)ri] = (uint16_t)state;
                    if (decoded != nullptr) decoded[(uint64_t)tile * 256u + (uint32_t)ri] = __half2float(table[state]);
                    node = from;
                }
            }
        }
    }
}

// states u16 [count][256] -> payload words [count][w] (16-bit words; w = 16 ka + 8 at a half-step rate): the low d(i) bits of
// state i, most significant bit first, in 32-bit little-endian words - the ring trellis.cuh reads. A thread per 32-bit word.
__global__ void __launch_bounds__(256) pack_kernel(const uint16_t* __restrict__ states, uint32_t count, int ka, int half_step,
        uint32_t* __restrict__ words) {
    const uint32_t per_tile = (uint32_t)(8 * ka + (half_step ? 4 : 0));   // 32-bit words of a tile
    const uint64_t index = (uint64_t)blockIdx.x * 256u + threadIdx.x;
    if (index >= (uint64_t)count * per_tile) return;
    const uint32_t tile = (uint32_t)(index / per_tile), word = (uint32_t)(index % per_tile);
    const int first_bit = (int)word * 32;
    // position i starts at bit i ka + i / 2 (half-step: one more bit before every odd position's successor)
    uint32_t value = 0;
    for (int i = 0; i < 256; ++i) {
        const int start = i * ka + (half_step ? i / 2 : 0), bits = position_bits(i, ka, half_step != 0);
        if (start + bits <= first_bit) continue;
        if (start >= first_bit + 32) break;
        const uint32_t field = (uint32_t)states[(uint64_t)tile * 256u + (uint32_t)i] & ((1u << bits) - 1u);
        // the field occupies stream bits [start, start + bits); stream bit b of this word is word bit 31 - (b - first_bit)
        const int shift = first_bit + 32 - (start + bits);
        value |= shift >= 0 ? field << shift : field >> -shift;
    }
    words[index] = value;
}

}  // namespace trellis_encode

// BLAKE3 on the device where one hash's chain of compressions is what takes the
// time (transcripts): four lanes per compression.
//
// Lane i of a quad holds column i of the state.  The diagonal steps keep b in
// place and move a, c and d one, one and two lanes over: those three are final
// before b is, so their shuffles run behind the rest of the column step.  A
// compression is then a chain of 7 x 24 dependent operations: 970 cycles measured,
// against 1,570 for one thread per compression, whose warp issues four times the
// instructions.  Message words come from shared memory, each lane's own.  With
// more than two such warps per scheduler the shuffles and message loads fill the
// load/store pipe, and one thread per compression is faster again.
#pragma once

#include "dm_blake3.cuh"

namespace dm {

// Byte offsets of the words lane i takes in round r: column pair, then the pair of
// the diagonal it works on with b in place (diagonal i - 1), one byte each.
struct QuadSchedule {
    uint32_t w[7][4];
    constexpr QuadSchedule() : w{} {
        constexpr int perm[16] = {2, 6, 3, 10, 7, 0, 4, 13, 1, 11, 12, 5, 9, 14, 15, 8};
        int p[16] = {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15};
        for (int r = 0; r < 7; ++r) {
            for (int i = 0; i < 4; ++i) {
                const int j = (i + 3) & 3;
                w[r][i] = (uint32_t)(4 * p[2 * i] | 4 * p[2 * i + 1] << 8 | 4 * p[8 + 2 * j] << 16) |
                          (uint32_t)(4 * p[9 + 2 * j]) << 24;
            }
            int n[16] = {};
            for (int k = 0; k < 16; ++k) n[k] = p[perm[k]];
            for (int k = 0; k < 16; ++k) p[k] = n[k];
        }
    }
};
static __constant__ QuadSchedule c_quad_schedule{};

DM_D uint32_t b3_iv(uint32_t i) {
    const uint32_t lo = i & 2u ? (i & 1u ? DM_B3_IV3 : DM_B3_IV2) : (i & 1u ? DM_B3_IV1 : DM_B3_IV0);
    const uint32_t hi = i & 2u ? (i & 1u ? DM_B3_IV7 : DM_B3_IV6) : (i & 1u ? DM_B3_IV5 : DM_B3_IV4);
    return i & 4u ? hi : lo;
}

// What a lane keeps across compressions.
struct Quad {
    uint32_t i;             // lane in the quad
    uint32_t words[7];      // its column of the schedule
    uint32_t iv_lo, iv_hi;  // IV words i and 4 + i
    DM_D Quad() : i(threadIdx.x & 3u), iv_lo(b3_iv(i)), iv_hi(b3_iv(4 + i)) {
#pragma unroll
        for (int r = 0; r < 7; ++r) words[r] = c_quad_schedule.w[r][i];
    }
    // Lane i's part of (counter lo, counter hi, block length, flags).
    DM_D uint32_t tail(uint64_t counter, uint32_t len, uint32_t flags) const {
        return i & 2u ? (i & 1u ? flags : len) : (i & 1u ? (uint32_t)(counter >> 32) : (uint32_t)counter);
    }
    // (lo, hi): words i and 4 + i of the chaining value, in and out.  msg: the block's
    // sixteen words in shared memory.  Every lane of the warp takes part.
    DM_D void compress(uint32_t& lo, uint32_t& hi, const uint32_t* msg, uint32_t tail) const {
        const char* base = reinterpret_cast<const char*>(msg);
        uint32_t a = lo, b = hi, c = iv_lo, d = tail;
        auto word = [&](uint32_t offset) { return *reinterpret_cast<const uint32_t*>(base + offset); };
        auto mix = [&](uint32_t mx, uint32_t my) {
            a = b + (a + mx);  // the message joins a before b arrives
            d = b3_rotr(d ^ a, 16);
            c = c + d;
            b = b3_rotr(b ^ c, 12);
            a = b + (a + my);
            d = b3_rotr(d ^ a, 8);
            c = c + d;
            b = b3_rotr(b ^ c, 7);
        };
        auto from = [&](uint32_t v, uint32_t lane) { return __shfl_sync(0xFFFFFFFFu, v, (int)lane, 4); };
        // the next round's words are on their way while a round runs
        uint32_t m[4], n[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) n[k] = word((words[0] >> (8 * k)) & 0xFFu);
#pragma unroll
        for (int r = 0; r < 7; ++r) {
#pragma unroll
            for (int k = 0; k < 4; ++k) m[k] = n[k];
            if (r < 6) {
#pragma unroll
                for (int k = 0; k < 4; ++k) n[k] = word((words[r + 1] >> (8 * k)) & 0xFFu);
            }
            mix(m[0], m[1]);
            a = from(a, i + 3u);
            d = from(d, i + 2u);
            c = from(c, i + 1u);
            mix(m[2], m[3]);
            a = from(a, i + 1u);
            d = from(d, i + 2u);
            c = from(c, i + 3u);
        }
        lo = a ^ c;
        hi = b ^ d;
    }
};

// Chaining values of chunks and nodes sit in shared memory as 8 words each, two
// neighbours together as their parent's message, the messages 20 words apart
// (which brings the lanes' words to 1.8 bank cycles instead of 4).
DM_HD constexpr uint32_t node_at(uint32_t n) { return 20 * (n / 2) + 8 * (n & 1u); }
DM_HD constexpr uint32_t node_words(uint32_t n) { return 10 * (n + (n & 1u)); }
// Merges n nodes level by level between the buffers, a lone last node carried up:
// BLAKE3's left-complete tree.  Every thread of the block calls it, the nodes
// written before and a barrier passed; returns the buffer whose first eight words
// are the last node, also past a barrier.  `root`: the last merge is the root of
// the whole hash.
template <uint32_t THREADS>
DM_D uint32_t* merge_nodes(const Quad& q, uint32_t* nodes, uint32_t* other, uint32_t n, bool root) {
    while (n > 1) {
        const uint32_t pairs = n / 2;
        for (uint32_t p0 = (threadIdx.x & ~31u) / 4; p0 < pairs; p0 += THREADS / 4) {  // uniform per warp
            const uint32_t p = p0 + (threadIdx.x & 31u) / 4;
            uint32_t lo = q.iv_lo, hi = q.iv_hi;
            q.compress(lo, hi, nodes + 20 * (p < pairs ? p : 0u),
                       q.tail(0, 64, kB3Parent | (root && n == 2 ? kB3Root : 0u)));
            if (p < pairs) {
                other[node_at(p) + q.i] = lo;
                other[node_at(p) + 4 + q.i] = hi;
            }
        }
        if ((n & 1u) && threadIdx.x < 8) other[node_at(pairs) + threadIdx.x] = nodes[node_at(n - 1) + threadIdx.x];
        __syncthreads();
        n = pairs + (n & 1u);
        uint32_t* t = nodes;
        nodes = other;
        other = t;
    }
    return nodes;
}

}  // namespace dm

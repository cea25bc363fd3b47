// The absorbed stream of a Fiat-Shamir challenge (src/protocol/transcript.rs:22-90)
// hashed by one block, and the encoded commitments it reads: shared by the kernels
// that compute challenges on the device.
#pragma once

#include "dm_blake3_dev.cuh"
#include "dm_jobs.cuh"

namespace dm {

// The absorbed bytes: epoch seed, u64 label length, label, u64 32, file id, u64 0,
// u64 round (99 bytes for "vec", 100 for "poly"), the commitments' images, u32 counter 0.
DM_HD constexpr uint64_t message_bytes(bool poly, uint64_t image_words) { return (poly ? 100u : 99u) + 4 * image_words + 4; }

// The absorbed stream behind one challenge: the header's words in shared memory,
// whose word kHeadWords is C's image's first, then L's and R's.  PAST_L1: another SM
// may have written the images during the same launch.
template <bool PAST_L1>
struct Stream {
    const uint32_t* head;
    const uint32_t* c;
    const uint32_t* lr;
    uint32_t c_words, lr_words;
    bool poly;
    DM_D uint64_t bytes() const { return message_bytes(poly, (uint64_t)c_words + lr_words); }
    DM_D uint32_t chunks() const { return (uint32_t)((bytes() + kB3ChunkLen - 1) / kB3ChunkLen); }
    DM_D static uint32_t load(const uint32_t* p) { return PAST_L1 ? __ldcg(p) : *p; }
    // Word i of the stream, i >= kHeadWords; zeros past the end, the counter's bytes.
    DM_D uint32_t image(uint32_t i) const {
        i -= kHeadWords;
        const uint32_t* p = i < c_words ? c + i : lr + (i - c_words);
        return i < c_words + lr_words ? load(p) : 0u;
    }
    // Word w < kHeadWords of the message.  "vec" images start one byte before a word, so
    // its message is the stream from the second byte on.
    DM_D uint32_t header(uint32_t w) const {
        return poly ? head[w] : __funnelshift_r(head[w], w + 1 < kHeadWords ? head[w + 1] : image(w + 1), 8);
    }
};

// The hash of a run of chunks has two parts, each called by the whole block and a
// barrier due after each.  First the chunks' words go to shared memory, zeros behind
// the message's end, a chunk every kChunkStride words (which staggers the quads of a
// warp over the banks): with the loads one block ahead of the compressions instead, a
// block took 1,880 cycles, most of it their latency, and takes 1,080 now.  A proof of
// 52 KB went from 402 to 353 us, of 1 MiB from 952 to 902, the verification of a
// 4 MiB file's from 694 to 600.
constexpr uint32_t kChunkStride = 256 + 20;
template <uint32_t THREADS, class S>
DM_D void stage_chunks(const S& s, uint32_t first, uint32_t count, uint32_t* words) {
    const uint32_t all = (uint32_t)((s.bytes() + 63) / 64) * 16u - first * 256u;
    const uint32_t n = all < count * 256u ? all : count * 256u;
    // eight words a thread in flight; the header's, which memory does not hold, apart
    constexpr uint32_t kAtOnce = 8;
    for (uint32_t i0 = threadIdx.x; i0 < n; i0 += kAtOnce * THREADS) {
        uint32_t lo[kAtOnce], hi[kAtOnce];
#pragma unroll
        for (uint32_t b = 0; b < kAtOnce; ++b) {
            const uint32_t i = i0 + b * THREADS, w = first * 256u + i;
            if (i >= n) break;
            lo[b] = s.image(w);
            hi[b] = s.poly ? 0u : s.image(w + 1);
        }
#pragma unroll
        for (uint32_t b = 0; b < kAtOnce; ++b) {
            const uint32_t i = i0 + b * THREADS;
            if (i >= n) break;
            if (first * 256u + i >= kHeadWords)
                words[(i >> 8) * kChunkStride + (i & 255u)] = s.poly ? lo[b] : __funnelshift_r(lo[b], hi[b], 8);
        }
    }
    if (first == 0 && threadIdx.x < kHeadWords) words[threadIdx.x] = s.header(threadIdx.x);
}
// Then four lanes per chunk: chaining values of chunks first .. first + count - 1 into
// nodes, count <= THREADS / 4.
template <class S>
DM_D void hash_chunks(const Quad& q, const S& s, uint32_t first, uint32_t count, uint32_t nchunks,
                      const uint32_t* words, uint32_t* nodes) {
    if ((threadIdx.x & ~31u) / 4 >= count) return;  // uniform per warp
    const uint64_t len = s.bytes();
    const uint32_t k = threadIdx.x / 4, c = first + k;
    const uint64_t off = (uint64_t)c * kB3ChunkLen;
    const uint32_t clen = k >= count ? 0u : (uint32_t)(len - off < kB3ChunkLen ? len - off : kB3ChunkLen);
    const uint32_t nblocks = (clen + 63u) / 64u;
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, nblocks);
    const uint32_t* m = words + (k < count ? k : 0u) * kChunkStride;
    uint32_t lo = q.iv_lo, hi = q.iv_hi;
#pragma unroll 1
    for (uint32_t b = 0; b < most; ++b) {
        const bool last = b + 1 == nblocks;
        const uint32_t flags =
            (b == 0 ? kB3ChunkStart : 0u) | (last ? kB3ChunkEnd : 0u) | (last && nchunks == 1 ? kB3Root : 0u);
        uint32_t l = lo, h = hi;
        q.compress(l, h, m + 16 * b, q.tail(nchunks == 1 ? 0u : c, last ? clen - b * 64u : 64u, flags));
        if (b < nblocks) lo = l, hi = h;
    }
    if (k < count) {
        nodes[node_at(k) + q.i] = lo;
        nodes[node_at(k) + 4 + q.i] = hi;
    }
}
DM_D fq challenge_of(const uint32_t* digest) {
    uint32_t h[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = digest[i];
    return fq_reduce8(h);
}

DM_D void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
DM_D uint32_t cluster_blocks() {
    uint32_t n;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
    return n;
}
// Element e = coordinate * n + j of an encoded module (n = 2^L): its first word.
DM_D uint64_t element_at(uint32_t L, uint32_t e) { return 2 + (uint64_t)(e >> L) * (2 + (4ull << L)) + 2 + 4ull * (e & ((1u << L) - 1u)); }
DM_D fq load_element(const uint32_t* image, uint32_t L, uint32_t e) {
    const uint2* p = reinterpret_cast<const uint2*>(image + element_at(L, e));
    const uint2 lo = __ldcg(p), hi = __ldcg(p + 1);
    return fq{{lo.x, lo.y, hi.x, hi.y}};
}
DM_D void store_element(uint32_t* image, uint32_t L, uint32_t e, const fq& v) {
    uint2* p = reinterpret_cast<uint2*>(image + element_at(L, e));
    __stcg(p, make_uint2(v.w[0], v.w[1]));
    __stcg(p + 1, make_uint2(v.w[2], v.w[3]));
    if ((e & ((1u << L) - 1u)) == 0) {
        __stcg(p - 1, make_uint2(1u << L, 0u));
        if (e == 0) __stcg(p - 2, make_uint2(kRank, 0u));
    }
}
DM_HD constexpr uint32_t module_words(uint32_t L) { return 2 + kRank * (2 + (4u << L)); }

}  // namespace dm

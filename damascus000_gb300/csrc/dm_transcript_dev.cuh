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
    DM_D uint32_t word(uint32_t i) const {  // zeros past the end: the counter's bytes
        if (i < kHeadWords) return head[i];
        i -= kHeadWords;
        if (i < c_words) return load(c + i);
        i -= c_words;
        return i < lr_words ? load(lr + i) : 0u;
    }
    // Words w0 .. w0 + 3 of the message: "vec" images start one byte before a word,
    // so its message is the stream from the second byte on.
    DM_D uint4 message(uint32_t w0) const {
        const uint32_t i = w0 - kHeadWords;  // wraps below the header's end
        const uint32_t* p = nullptr;
        if (w0 >= kHeadWords && i + 5 <= c_words) p = c + i;
        else if (w0 >= kHeadWords + c_words && i - c_words + 5 <= lr_words) p = lr + (i - c_words);
        uint32_t v[5];
        if (p) {
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] = load(p + k);
        } else {
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] = word(w0 + k);
        }
        const uint32_t sh = poly ? 0u : 8u;
        return make_uint4(__funnelshift_r(v[0], v[1], sh), __funnelshift_r(v[1], v[2], sh),
                          __funnelshift_r(v[2], v[3], sh), __funnelshift_r(v[3], v[4], sh));
    }
};

// Chaining values of chunks first .. first + count - 1 into nodes (count of them; the
// whole block calls it, a barrier is due after).  Four lanes per chunk, THREADS / 4
// at a time, the words one block ahead; msg holds message_room<THREADS>() words.
constexpr uint32_t kStride = 20;  // a block's 16 words, staggered over the banks
template <uint32_t THREADS>
DM_HD constexpr uint32_t message_room() { return 2 * (THREADS / 4) * kStride; }
template <uint32_t THREADS, class S>
DM_D void hash_chunks(const Quad& q, const S& s, uint32_t first, uint32_t count, uint32_t nchunks, uint32_t* msg,
                      uint32_t* nodes) {
    const uint64_t len = s.bytes();
    for (uint32_t k0 = (threadIdx.x & ~31u) / 4; k0 < count; k0 += THREADS / 4) {  // uniform per warp
        const uint32_t k = k0 + (threadIdx.x & 31u) / 4, c = first + k;
        const uint64_t off = (uint64_t)c * kB3ChunkLen;
        const uint32_t clen = k >= count ? 0u : (uint32_t)(len - off < kB3ChunkLen ? len - off : kB3ChunkLen);
        const uint32_t nblocks = (clen + 63u) / 64u;
        const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, nblocks);
        uint32_t lo = q.iv_lo, hi = q.iv_hi;
        uint4 next = nblocks ? s.message(c * 256u + 4 * q.i) : make_uint4(0, 0, 0, 0);
#pragma unroll 1
        for (uint32_t b = 0; b < most; ++b) {
            uint32_t* m = msg + ((b & 1u) * (THREADS / 4) + threadIdx.x / 4) * kStride;  // last read two blocks ago
            reinterpret_cast<uint4*>(m)[q.i] = next;
            if (b + 1 < nblocks) next = s.message(c * 256u + (b + 1) * 16u + 4 * q.i);
            __syncwarp();
            const bool last = b + 1 == nblocks;
            const uint32_t flags =
                (b == 0 ? kB3ChunkStart : 0u) | (last ? kB3ChunkEnd : 0u) | (last && nchunks == 1 ? kB3Root : 0u);
            uint32_t l = lo, h = hi;
            q.compress(l, h, m, q.tail(nchunks == 1 ? 0u : c, last ? clen - b * 64u : 64u, flags));
            if (b < nblocks) lo = l, hi = h;
        }
        if (k < count) {
            nodes[node_at(k) + q.i] = lo;
            nodes[node_at(k) + 4 + q.i] = hi;
        }
        __syncwarp();  // the next pass writes the message words this one read
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

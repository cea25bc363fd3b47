// Fiat-Shamir challenges on the device (src/protocol/transcript.rs:22-90): the
// BLAKE3 hash of the absorbed bytes, its reduction mod q and the inverse, so that
// a proof's stages follow one another without a host round trip.
#include <cuda_runtime.h>

#include "dm_blake3_dev.cuh"
#include "dm_jobkit.cuh"

namespace dm {

namespace {

using namespace jobkit;

// The absorbed bytes: epoch seed, u64 label length, label, u64 32, file id, u64 0,
// u64 round (99 bytes for "vec", 100 for "poly"), the commitments' images, u32 counter 0.
DM_HD uint64_t message_bytes(bool poly, uint64_t image_words) { return (poly ? 100u : 99u) + 4 * image_words + 4; }

// A block hashes 32 chunks, four lanes each, and merges them; the block that
// finishes last merges the groups, reduces the digest and inverts it.  Bound by the
// chain of a chunk's 16 compressions (970 cycles each), the levels above and the
// inversion (13,600 cycles).  The chunks' words come one block ahead.
constexpr uint32_t kThreads = 128;
constexpr uint32_t kGroup = kThreads / 4;
constexpr uint32_t kMaxGroups = 128;  // 4,096 chunks: three commitments at rings of 2^13 take 3,073

__global__ void __launch_bounds__(kThreads) challenge_kernel(ChallengeJob jb) {
    constexpr uint32_t kStride = 20;
    __shared__ __align__(16) uint32_t msg[2][kGroup * kStride];
    __shared__ __align__(16) uint32_t nodes[node_words(kMaxGroups)], other[node_words(kMaxGroups / 2)];
    __shared__ uint32_t head[kHeadWords];
    __shared__ uint32_t order;
    const Quad q;
    const uint32_t quad = threadIdx.x / 4;
    if (threadIdx.x < kHeadWords) {
        const uint32_t f = threadIdx.x - 13;  // the file id: words 13..20 (challenge_head)
        head[threadIdx.x] = f < 8u ? jb.file_id[f] : jb.head[threadIdx.x];
    }
    __syncthreads();
    const uint64_t len = message_bytes(jb.poly, (uint64_t)jb.c_words + jb.lr_words);
    const uint32_t nchunks = (uint32_t)((len + kB3ChunkLen - 1) / kB3ChunkLen);
    const uint32_t c = blockIdx.x * kGroup + quad;
    const uint32_t in_group = nchunks - blockIdx.x * kGroup < kGroup ? nchunks - blockIdx.x * kGroup : kGroup;
    const bool lone = nchunks <= kGroup;
    // Word i of the images' stream, whose word kHeadWords is C's first: header, C, L
    // and R, and zeros (the counter's bytes).
    auto word = [&](uint32_t i) -> uint32_t {
        if (i < kHeadWords) return head[i];
        i -= kHeadWords;
        if (i < jb.c_words) return jb.c[i];
        i -= jb.c_words;
        return i < jb.lr_words ? jb.lr[i] : 0u;
    };
    auto load5 = [&](uint32_t w0, uint32_t v[5]) {
        const uint32_t i = w0 - kHeadWords;  // wraps below the header's end
        const uint32_t* p = nullptr;
        if (w0 >= kHeadWords && i + 5 <= jb.c_words) p = jb.c + i;
        else if (w0 >= kHeadWords + jb.c_words && i - jb.c_words + 5 <= jb.lr_words) p = jb.lr + (i - jb.c_words);
        if (p) {
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] = p[k];
        } else {
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] = word(w0 + k);
        }
    };
    const uint64_t off = (uint64_t)c * kB3ChunkLen;
    const uint32_t clen = c >= nchunks ? 0u : (uint32_t)(len - off < kB3ChunkLen ? len - off : kB3ChunkLen);
    const uint32_t nblocks = (clen + 63u) / 64u;
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, nblocks);
    uint32_t lo = q.iv_lo, hi = q.iv_hi, next[5] = {0, 0, 0, 0, 0};
    if (nblocks) load5(c * 256u + 4 * q.i, next);
#pragma unroll 1
    for (uint32_t b = 0; b < most; ++b) {
        uint32_t* m = msg[b & 1u] + quad * kStride;
        // "vec" images start one byte before a word: the message is the stream from its
        // second byte on
        const uint32_t sh = jb.poly ? 0u : 8u;
        reinterpret_cast<uint4*>(m)[q.i] =
            make_uint4(__funnelshift_r(next[0], next[1], sh), __funnelshift_r(next[1], next[2], sh),
                       __funnelshift_r(next[2], next[3], sh), __funnelshift_r(next[3], next[4], sh));
        if (b + 1 < nblocks) load5(c * 256u + (b + 1) * 16u + 4 * q.i, next);
        __syncwarp();
        const bool last = b + 1 == nblocks;
        const uint32_t flags =
            (b == 0 ? kB3ChunkStart : 0u) | (last ? kB3ChunkEnd : 0u) | (last && nchunks == 1 ? kB3Root : 0u);
        uint32_t l = lo, h = hi;
        q.compress(l, h, m, q.tail(nchunks == 1 ? 0u : c, last ? clen - b * 64u : 64u, flags));
        if (b < nblocks) lo = l, hi = h;
    }
    if (c < nchunks) {
        nodes[node_at(quad) + q.i] = lo;
        nodes[node_at(quad) + 4 + q.i] = hi;
    }
    __syncthreads();
    const uint32_t* node = merge_nodes<kThreads>(q, nodes, other, in_group, lone);
    if (!lone) {
        if (threadIdx.x < 8) {
            jb.cvs[8 * blockIdx.x + threadIdx.x] = node[threadIdx.x];
            __threadfence();
        }
        __syncthreads();
        if (threadIdx.x == 0) order = atomicInc(jb.ticket, gridDim.x - 1);  // zero again after the last block
        __syncthreads();
        if (order != gridDim.x - 1) return;
        __threadfence();
        for (uint32_t i = threadIdx.x; i < 8 * gridDim.x; i += kThreads)
            nodes[node_at(i / 8) + (i & 7u)] = __ldcg(jb.cvs + i);
        __syncthreads();
        node = merge_nodes<kThreads>(q, nodes, other, gridDim.x, true);
    }
    if (threadIdx.x == 0) {
        uint32_t h[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] = node[i];
        const fq x = fq_reduce8(h);
        stq(jb.out, 0, x);
        stq(jb.out, 1, fq_inv_gcd(x));
        if (fq_is_zero(x)) *jb.zero = 1u;
    }
}

uint32_t challenge_groups(bool poly, uint64_t image_words) {
    const uint64_t chunks = (message_bytes(poly, image_words) + kB3ChunkLen - 1) / kB3ChunkLen;
    return (uint32_t)((chunks + kGroup - 1) / kGroup);
}

}  // namespace

// As words of the message, or for "vec" of the message one byte later (a zero byte
// first): the file id then fills words 13..20 and the images start at word 25 in both.
void challenge_head(const uint8_t epoch[32], uint64_t round, bool poly, uint32_t head[kHeadWords]) {
    uint8_t b[4 * kHeadWords] = {0};
    uint8_t* p = b + (poly ? 0 : 1);
    for (int i = 0; i < 32; ++i) p[i] = epoch[i];
    const char* label = poly ? "poly" : "vec";
    const int ll = poly ? 4 : 3;
    p[32] = (uint8_t)ll;
    for (int i = 0; i < ll; ++i) p[40 + i] = (uint8_t)label[i];
    p[40 + ll] = 32;
    for (int i = 0; i < 8; ++i) p[88 + ll + i] = (uint8_t)(round >> (8 * i));
    for (uint32_t w = 0; w < kHeadWords; ++w) head[w] = b3_load_le32(b + 4 * w);
}

size_t challenge_scratch_words(uint32_t c_words, uint32_t lr_words) {
    return 8 * (size_t)challenge_groups(true, (uint64_t)c_words + lr_words);
}

cudaError_t launch_challenge(const ChallengeJob& job, cudaStream_t st) {
    const uint32_t groups = challenge_groups(job.poly, (uint64_t)job.c_words + job.lr_words);
    if (groups > kMaxGroups) return cudaErrorInvalidValue;
    challenge_kernel<<<groups, kThreads, 0, st>>>(job);
    return cudaGetLastError();
}

}  // namespace dm

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

// One challenge of a prover.  A block hashes 32 chunks and merges them; the block
// that finishes last merges the groups, reduces the digest and inverts it.  Bound
// by the chain of a chunk's 16 compressions (970 cycles each), the levels above and
// the inversion (12,200 cycles).
constexpr uint32_t kThreads = 128;
constexpr uint32_t kGroup = kThreads / 4;
constexpr uint32_t kMaxGroups = 128;  // 4,096 chunks: three commitments at rings of 2^13 take 3,073

__global__ void __launch_bounds__(kThreads) challenge_kernel(ChallengeJob jb) {
    stage_begin();
    __shared__ __align__(16) uint32_t msg[message_room<kThreads>()];
    __shared__ __align__(16) uint32_t nodes[node_words(kMaxGroups)], other[node_words(kMaxGroups / 2)];
    __shared__ uint32_t head[kHeadWords];
    __shared__ uint32_t order;
    const Quad q;
    if (threadIdx.x < kHeadWords) {
        const uint32_t f = threadIdx.x - 13;  // the file id: words 13..20 (challenge_head)
        head[threadIdx.x] = f < 8u ? jb.file_id[f] : jb.head[threadIdx.x];
    }
    __syncthreads();
    const Stream<false> s{head, jb.c, jb.lr, jb.c_words, jb.lr_words, jb.poly != 0u};
    const uint32_t nchunks = s.chunks(), first = blockIdx.x * kGroup;
    const uint32_t in_group = nchunks - first < kGroup ? nchunks - first : kGroup;
    const bool lone = nchunks <= kGroup;
    hash_chunks<kThreads>(q, s, first, in_group, nchunks, msg, nodes);
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
        const fq x = challenge_of(node);
        stq(jb.out, 0, x);
        stq(jb.out, 1, fq_inv_gcd(x));
        if (fq_is_zero(x)) *jb.zero = 1u;
    }
}

// ================================================================ verifier
// A verifier's transcript is one chain: each challenge hashes the commitment that
// the one before folded.  A cluster of up to eight blocks runs it in one launch:
// every block hashes a power of two of the chunks, leaves its node in memory, and
// after a cluster barrier each merges the nodes and inverts the challenge by itself
// (which saves a second barrier), folds its share of the commitment, and meets the
// others again.  Bound per stage as challenge_kernel, plus two barriers and two
// products a coefficient; a proof holds eight SMs at most, so a service's proofs
// run side by side.
constexpr uint32_t kReplayThreads = 512;
constexpr uint32_t kReplayNodes = 512;  // chunks per block: rings of 2^13 take 3,073 over eight

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
DM_HD uint32_t module_words(uint32_t L) { return 2 + kRank * (2 + (4u << L)); }

__global__ void __launch_bounds__(kReplayThreads) replay_kernel(ReplayJob jb) {
    __shared__ __align__(16) uint32_t msg[message_room<kReplayThreads>()], nodes[node_words(kReplayNodes)];
    uint32_t* other = msg;  // merged into once the chunks are hashed
    static_assert(message_room<kReplayThreads>() >= node_words(kReplayNodes / 2), "room for the merges");
    __shared__ uint32_t head[kHeadWords];
    __shared__ fq challenge[2];
    const Quad q;
    const uint32_t blocks = cluster_blocks(), me = blockIdx.x, d = jb.d;
    const uint32_t thread = me * kReplayThreads + threadIdx.x, threads = blocks * kReplayThreads;
    // deserialisation reduces every word (src/algebra/field.rs:121-129)
    auto canonical = [&](uint32_t* image, uint32_t L) {
        for (uint32_t e = thread; e < (uint32_t)kRank << L; e += threads) {
            const fq v = load_element(image, L, e);
            if (v.w[3] >= kQ3) {  // at or above q, or just below
                uint32_t r[8] = {v.w[0], v.w[1], v.w[2], v.w[3], 0, 0, 0, 0};
                const fq c = fq_reduce8(r);
                uint2* p = reinterpret_cast<uint2*>(image + element_at(L, e));
                __stcg(p, make_uint2(c.w[0], c.w[1]));
                __stcg(p + 1, make_uint2(c.w[2], c.w[3]));
            }
        }
    };
    uint32_t* com0 = jb.proof + 12;
    uint32_t* records = com0 + module_words(d) + 8 + 2;  // past the seed and the record count
    canonical(com0, d);
    {
        uint32_t* r = records;
        for (uint32_t L = d; L > 0; --L) {
            r += 2;
            for (int m = 0; m < 4; ++m) {
                canonical(r, m < 2 ? L : L - 1);
                r += module_words(m < 2 ? L : L - 1);
            }
        }
    }
    cluster_barrier();
    uint32_t* rec = records;
    for (uint32_t round = 0; round < d; ++round) {
        const uint32_t L = d - round;
        rec += 2;  // the round's number
        fq x_inv;
        for (int poly = 0; poly < 2; ++poly) {
            const uint32_t Ls = L - poly;  // ring of L and R, and of the folded commitment
            const uint32_t* c = poly ? jb.ct : (round == 0 ? com0 : jb.c);
            const uint32_t* l = rec + (poly ? 2 * module_words(L) : 0u);
            const uint32_t* r = l + module_words(Ls);
            __syncthreads();  // the last stage's use of the shared words
            if (threadIdx.x < kHeadWords) {
                // the round: words 23 and 24 of the message, one byte later for "vec"
                uint32_t w = jb.head[poly][threadIdx.x];
                if (threadIdx.x == 23) w |= round;
                if (threadIdx.x - 13u < 8u) w = jb.proof[threadIdx.x - 13];  // the file id
                head[threadIdx.x] = w;
            }
            __syncthreads();
            const Stream<true> s{head, c, l, module_words(L), 2 * module_words(Ls), poly != 0};
            const uint32_t nchunks = s.chunks();
            uint32_t span = 1;  // chunks per block, a power of two
            while (span * blocks < nchunks) span *= 2;
            const uint32_t first = me * span;
            const uint32_t count = first >= nchunks ? 0u : (nchunks - first < span ? nchunks - first : span);
            const bool lone = nchunks <= span;
            hash_chunks<kReplayThreads>(q, s, first, count, nchunks, msg, nodes);
            __syncthreads();
            const uint32_t* node = merge_nodes<kReplayThreads>(q, nodes, other, count, lone);
            if (threadIdx.x < 8 && count) __stcg(jb.cvs + 8 * me + threadIdx.x, node[threadIdx.x]);
            cluster_barrier();
            const uint32_t groups = (nchunks + span - 1) / span;
            if (threadIdx.x < 8 * groups)
                nodes[node_at(threadIdx.x / 8) + (threadIdx.x & 7u)] = __ldcg(jb.cvs + threadIdx.x);
            __syncthreads();
            node = merge_nodes<kReplayThreads>(q, nodes, other, groups, true);
            if (threadIdx.x == 0) {
                const fq x = challenge_of(node), xi = fq_inv_gcd(x);
                challenge[0] = x;
                challenge[1] = xi;
                if (me == 0) {
                    uint4* out = jb.rounds + kRoundWords * round;
                    if (fq_is_zero(x)) *jb.zero = 1u;
                    if (!poly) {
                        stq(out, 0, xi);
                    } else {
                        const fq xy = fq_mul(x_inv, xi);
                        stq(out, 1, xi);
                        stq(out, 2, xy);
                        stq(out, 3, fq_neg(xi));
                        stq(out, 4, fq_neg(xy));
                    }
                }
                x_inv = xi;
            }
            __syncthreads();
            const fq x = challenge[0], xi = challenge[1];
            uint32_t* out = poly ? jb.c : jb.ct;
            for (uint32_t e = thread; e < (uint32_t)kRank << Ls; e += threads) {
                // the even coefficients of the commitment in the second stage
                const fq base = load_element(c, L, e << poly);
                store_element(out, Ls, e, fq_fma(fq_fma(base, xi, load_element(l, Ls, e)), x, load_element(r, Ls, e)));
            }
            cluster_barrier();
        }
        rec += 2 * module_words(L) + 2 * module_words(L - 1);
    }
}

__global__ void opening_kernel(const uint4* g, const uint32_t* c, const uint32_t* opening, uint32_t* bad) {
    stage_begin();
    const uint32_t k = threadIdx.x;
    if (k >= (uint32_t)kRank) return;
    uint32_t r[8] = {opening[0], opening[1], opening[2], opening[3], 0, 0, 0, 0};
    const fq v = fq_mul(ldq(g, k), fq_reduce8(r));
    if (!fq_eq(v, load_element(c, 0, k))) *bad = 1u;
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

cudaError_t launch_replay(const ReplayJob& job, cudaStream_t st) {
    // a block per 64 chunks of the first, largest stage
    const uint64_t chunks = (message_bytes(true, 3ull * module_words(job.d)) + kB3ChunkLen - 1) / kB3ChunkLen;
    uint32_t blocks = 1;
    while (blocks < kReplayBlocks && blocks * 64 < chunks) blocks *= 2;
    if (chunks > (uint64_t)blocks * kReplayNodes) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kReplayThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = blocks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, replay_kernel, job);
}

cudaError_t launch_opening(const uint4* d_g, const uint32_t* d_c, const uint32_t* d_opening, uint32_t* d_bad,
                           cudaStream_t st) {
    return launch_overlapped(opening_kernel, 1, 32, 0, st, d_g, d_c, d_opening, d_bad);
}

cudaError_t launch_challenge(const ChallengeJob& job, cudaStream_t st) {
    const uint32_t groups = challenge_groups(job.poly, (uint64_t)job.c_words + job.lr_words);
    if (groups > kMaxGroups) return cudaErrorInvalidValue;
    return launch_overlapped(challenge_kernel, groups, kThreads, 0, st, job);
}

}  // namespace dm

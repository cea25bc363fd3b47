// Fiat-Shamir challenges on the device (src/protocol/transcript.rs:22-90): the
// BLAKE3 hash of the absorbed bytes, its reduction mod q and the inverse, so that
// a proof's stages follow one another without a host round trip.
#include <cuda_runtime.h>

#include "dm_jobkit.cuh"
#include "dm_transcript_dev.cuh"

namespace dm {

namespace {

using namespace jobkit;

// One challenge of a prover.  A block hashes 32 chunks and merges them; the block
// that finishes last merges the groups, reduces the digest and inverts it.  Bound
// by the chain of a chunk's 16 compressions (1,080 cycles each), the levels above and
// the inversion (7,440 cycles).
constexpr uint32_t kThreads = 512;  // a group's chunks take 128; the others are for its loads
constexpr uint32_t kGroup = 32;
constexpr uint32_t kMaxGroups = 128;  // 4,096 chunks: three commitments at rings of 2^13 take 3,073

__global__ void __launch_bounds__(kThreads) challenge_kernel(ChallengeJob jb) {
    stage_begin();
    __shared__ uint32_t words[kGroup * kChunkStride];
    __shared__ uint32_t nodes[node_words(kMaxGroups)], other[node_words(kMaxGroups / 2)];
    __shared__ uint32_t head[kHeadWords], inv_table[kInvTable];
    __shared__ uint32_t order;
    const Quad q;
    if (threadIdx.x < kInvTable) inv_table[threadIdx.x] = inv_table_word(threadIdx.x);
    if (threadIdx.x < kHeadWords) {
        const uint32_t f = threadIdx.x - 13;  // the file id: words 13..20 (challenge_head)
        head[threadIdx.x] = f < 8u ? jb.file_id[f] : jb.head[threadIdx.x];
    }
    __syncthreads();
    const Stream<false> s{head, jb.c, jb.lr, jb.c_words, jb.lr_words, jb.poly != 0u};
    const uint32_t nchunks = s.chunks(), first = blockIdx.x * kGroup;
    const uint32_t in_group = nchunks - first < kGroup ? nchunks - first : kGroup;
    const bool lone = nchunks <= kGroup;
    stage_chunks<kThreads>(s, first, in_group, words);
    __syncthreads();
    hash_chunks(q, s, first, in_group, nchunks, words, nodes);
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
        stq(jb.out, 1, fq_inv_steps(x, inv_table));
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
constexpr uint32_t kReplayPass = kReplayThreads / 4;
constexpr uint32_t kReplayWhole = 16;  // 382 -> 372 us at depth 8, 445 -> 440 at 9; 64 chunks 378, 447
constexpr size_t kReplayBytes = kReplayPass * kChunkStride * sizeof(uint32_t);

__global__ void __launch_bounds__(kReplayThreads) replay_kernel(ReplayJob jb) {
    extern __shared__ uint32_t words[];  // kReplayPass chunks
    __shared__ uint32_t nodes[node_words(kReplayNodes)];
    uint32_t* other = words;  // merged into once the chunks are hashed
    static_assert(kReplayPass * kChunkStride >= node_words(kReplayNodes / 2), "room for the merges");
    __shared__ uint32_t head[kHeadWords], inv_table[kInvTable];
    __shared__ fq challenge[2];
    const Beside beside = stage_open(false);  // a verifier's generators are expanded beside it
    const Quad q;
    if (threadIdx.x < kInvTable) inv_table[threadIdx.x] = inv_table_word(threadIdx.x);
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
            // Short messages every block hashes whole, which needs no other's node; of longer
            // ones a block's share takes longer than the barrier that this saves.
            const bool whole = nchunks <= kReplayWhole;
            uint32_t span = 1;  // chunks per block, a power of two
            while (span < nchunks && (whole || span * blocks < nchunks)) span *= 2;
            const uint32_t first = whole ? 0u : me * span;
            const uint32_t count = first >= nchunks ? 0u : (nchunks - first < span ? nchunks - first : span);
            const bool lone = nchunks <= span;
            for (uint32_t done = 0; done < count; done += kReplayPass) {
                const uint32_t now = count - done < kReplayPass ? count - done : kReplayPass;
                stage_chunks<kReplayThreads>(s, first + done, now, words);
                __syncthreads();
                hash_chunks(q, s, first + done, now, nchunks, words, nodes + node_at(done));
                __syncthreads();
            }
            const uint32_t* node = merge_nodes<kReplayThreads>(q, nodes, other, count, lone);
            if (!whole) {
                if (threadIdx.x < 8 && count) __stcg(jb.cvs + 8 * me + threadIdx.x, node[threadIdx.x]);
                cluster_barrier();
                const uint32_t groups = (nchunks + span - 1) / span;
                if (threadIdx.x < 8 * groups)
                    nodes[node_at(threadIdx.x / 8) + (threadIdx.x & 7u)] = __ldcg(jb.cvs + threadIdx.x);
                __syncthreads();
                node = merge_nodes<kReplayThreads>(q, nodes, other, groups, true);
            }
            if (threadIdx.x == 0) {
                const fq x = challenge_of(node), xi = fq_inv_steps(x, inv_table);
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

cudaError_t replay_opt_in() {
    return cudaFuncSetAttribute(replay_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kReplayBytes);
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
    cfg.dynamicSmemBytes = kReplayBytes;
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

// The last rounds of a proof in one launch (src/protocol/prover.rs:149-313): from
// rings of 2^6 down, every challenge, fold, commitment, check and cross term.
//
// A stage of such a ring is five kernels of 3 to 10 us, mostly launch, first loads
// and drain, and a challenge behind them.  Here a cluster of eight blocks keeps the
// rounds on chip: block k holds coordinate k of the generators and the whole
// witness, so its products, inverse transforms and checks are its own, and only the
// transcript needs the others: one cluster barrier a stage, after which every block
// hashes the whole message by itself (25 chunks at most).
//
// A stage is then the chain of a chunk's 16 compressions and the tree's levels, the
// challenge's inverse, and the stage's arithmetic.  The last two run side by side:
// warp 0 inverts while the others fold.  For that the generators are folded times the
// challenge (x g_l + g_r instead of g_l + x^-1 g_r), so their commitments carry the
// product of the challenges so far, and its inverse is multiplied in at the end.
// From 2^4 down the inverse (8,200 cycles) covers the arithmetic (5,000); the stages of
// 2^6 take 43,000 and 22,000 of it.  Against five kernels a stage and a challenge on
// the host or in a sixth a proof of 52 KB went from 522 to 402 us, of 1 MiB from 1,089
// to 952, of 16 MiB from 3,918 to 3,788; with the message staged in shared memory, the
// shorter inverse and what needs no inverse folded beside it 333, 817 and 3,582 (other
// kernels' gains among the last two).  In the engine a launch takes up to eight proofs
// whose commitments reach 2^6 in the same wave: 24 files of 50 KB to 16 MiB went from
// 11.0 to 10.5 ms, 32 of 50 KB to 4 MiB under one seed from 5.2 to 4.5.  More warps
// (640, 768 threads) take 2 to 3 % longer.
#include <cuda_runtime.h>

#include "dm_jobkit.cuh"
#include "dm_kernels.cuh"
#include "dm_ntt.cuh"
#include "dm_tables.h"
#include "dm_transcript_dev.cuh"

namespace dm {

namespace {

using namespace jobkit;

constexpr uint32_t kThreads = 512, kWorkers = kThreads - 32;
constexpr uint32_t kRing = 1u << kTailLog, kHalf = kRing / 2;
constexpr uint32_t kChunks = 32;  // of a message: three commitments at 2^6 take 25
static_assert(message_bytes(true, 3ull * module_words(kTailLog)) <= kChunks * kB3ChunkLen, "chunks of the first message");

// Final scales of the inverse transforms of rings 2^0 .. 2^(kTailLog - 1), with the
// CRT's (P / p_i)^-1.
struct TailScales {
    Tw f[kTailLog][kPrimes];
};

// Residue rows stand one word apart more than their length, so that a warp's threads
// can hold a row each.
struct Shared {
    uint4 vec[2][kHalf * kRing];                            // witness, generators after a vector fold
    uint32_t rows[4 * kHalf * kPrimes * (kHalf + 1)];       // transforms; the last part holds poly()
    uint32_t sums[3 * kPrimes * (kHalf + 1)];               // the products; during the hash its header
    uint4 c[kRing], l[kRing], r[kRing];                     // this coordinate's C, L and R
    Tw fwd[kPrimes][kRing], inv[kPrimes][kHalf + 1];
    uint32_t inv_table[kInvTable];
    uint32_t status;
    fq x, x_inv, inverse;                                   // the challenge; the inverse of the generators' factor
};
static_assert(sizeof(Shared) <= 227 * 1024, "shared memory of a block");
// Witness and generators after a polynomial fold: behind the rows of every stage but
// the first, which reads them from device memory instead.
constexpr uint32_t kPolyWords = 2 * kHalf * kHalf * 4;
static_assert(sizeof(Shared::rows) / 4 - kPolyWords >= 2 * kHalf * kPrimes * (kHalf + 1) &&
                  (sizeof(Shared::rows) / 4 - kPolyWords) % 4 == 0,
              "the rows of a polynomial stage leave room");
DM_D uint4* poly_of(Shared& sh) { return reinterpret_cast<uint4*>(sh.rows + sizeof(Shared::rows) / 4 - kPolyWords); }
// What a message is hashed in, and the products' coefficients: where the rows were.
static_assert((kChunks * kChunkStride + node_words(kChunks) + node_words(kChunks / 2)) <=
                  sizeof(Shared::rows) / 4 - kPolyWords,
              "room for the hash");

DM_D fq lds(const uint4* p, uint32_t i) { return ldq(p, i); }
DM_D void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kWorkers) : "memory"); }

// A thread per row: polynomials 0 .. 2^log_polys - 1, nine rows each, forward
// transforms in place.  A warp's rows are mostly one prime's.
template <int l>
DM_D void forward_rows(Shared& sh, uint32_t log_polys, uint32_t w, const PrimeConsts& pc) {
    constexpr uint32_t h = 1u << l;
    for (uint32_t i = w; i < (uint32_t)kPrimes << log_polys; i += kWorkers) {
        const uint32_t prime = i >> log_polys, poly = i & ((1u << log_polys) - 1u);
        const uint32_t p = pc.p[prime], one_s = pc.one_s[prime];
        uint32_t* row = sh.rows + (poly * kPrimes + prime) * (h + 1);
        uint32_t a[h];
#pragma unroll
        for (uint32_t j = 0; j < h; ++j) a[j] = row[j];
        ntt_fwd_small<l>(a, sh.fwd[prime], p);
#pragma unroll
        for (uint32_t j = 0; j < h; ++j) row[j] = ntt_fwd_final(a[j], one_s, p);
    }
}
// Row (warp, lane) = (sum, prime) of sh.sums: inverse transform and final scale.
template <int l>
DM_D void inverse_rows(Shared& sh, uint32_t nsums, uint32_t w, const PrimeConsts& pc, const TailScales& ts) {
    constexpr uint32_t h = 1u << l;
    const uint32_t sum = w / 32, prime = w % 32;
    if (sum >= nsums || prime >= (uint32_t)kPrimes) return;
    const uint32_t p = pc.p[prime];
    uint32_t* row = sh.sums + (sum * kPrimes + prime) * (h + 1);
    uint32_t a[h];
#pragma unroll
    for (uint32_t j = 0; j < h; ++j) a[j] = row[j];
    ntt_inv_small<l>(a, sh.inv[prime], p);
    const Tw f = ts.f[l][prime];
#pragma unroll
    for (uint32_t j = 0; j < h; ++j) row[j] = red_below(shoup_mul(a[j], f, p), p);
}

// Residues of one folded coefficient into its rows.
DM_D void put_residues(Shared& sh, uint32_t poly, uint32_t l, uint32_t j, const fq& v, const PrimeConsts& pc) {
    uint32_t* row = sh.rows + poly * kPrimes * ((1u << l) + 1) + j;
#pragma unroll
    for (int i = 0; i < kPrimes; ++i) row[i * ((1u << l) + 1)] = residue_fwd(v, pc, i);
}

struct TailJobs {
    TailJob j[kTailJobs];
    bool beside;
};

__global__ void __launch_bounds__(kThreads)
    tail_kernel(TailJobs J, PrimeConsts pc, CrtConsts cc, TailScales ts, const Tw* fwd, const Tw* inv) {
    extern __shared__ __align__(16) uint8_t raw[];
    Shared& sh = *reinterpret_cast<Shared*>(raw);
    const TailJob& jb = J.j[blockIdx.x / kRank];
    const uint32_t k = blockIdx.x % kRank, tid = threadIdx.x;
    const Quad q;
    // the tables need nothing of the kernels before
    for (uint32_t i = tid; i < kPrimes * kRing; i += kThreads) {
        const uint32_t prime = i / kRing, e = i % kRing;
        sh.fwd[prime][e] = fwd[prime * kMaxRing + e];
        if (e < kHalf) sh.inv[prime][e] = inv[prime * kMaxRing + e];
    }
    if (tid < kInvTable) sh.inv_table[tid] = inv_table_word(tid);
    const Beside beside = stage_open(J.beside);
    if (tid < 1u << jb.L) {
        const uint32_t e = (k << jb.L) + tid;
        sh.c[tid] = jb.c[e];
        sh.l[tid] = jb.l[e];
        sh.r[tid] = jb.r[e];
    }
    if (tid == 0) {
        sh.inverse = fq_from_u32(1);
        sh.status = 0;
    }
    uint4* poly = poly_of(sh);
    uint32_t* head = sh.sums;
    uint32_t* rec = jb.record;
    const uint32_t* image = jb.image;  // of the commitment the next challenge absorbs
    uint32_t round = jb.round;
    for (uint32_t L = jb.L; L > 0; --L, ++round) {
        const uint32_t s = 1u << L, l = L - 1, h = 1u << l;  // every transform is of ring 2^l
        for (uint32_t stage = 0; stage < 2; ++stage) {
            // ---- the challenge
            const uint32_t Ls = L - stage;  // ring of the L and R it absorbs
            const uint32_t* lr = rec + (stage ? 2 * module_words(L) : 0u);
            __syncthreads();
            if (tid < kHeadWords) {
                uint32_t v = jb.head[stage][tid];
                if (tid == 23) v |= round;  // the header of round 0 otherwise
                if (jb.file_id && tid - 13u < 8u) v = jb.file_id[tid - 13];
                head[tid] = v;
            }
            __syncthreads();
            const Stream<true> st{head, image, lr, module_words(L), 2 * module_words(Ls), stage != 0};
            const uint32_t nchunks = st.chunks();
            uint32_t* words = sh.rows;
            uint32_t* nodes = words + kChunks * kChunkStride;
            stage_chunks<kThreads>(st, 0, nchunks, words);
            __syncthreads();
            hash_chunks(q, st, 0, nchunks, nchunks, words, nodes);
            __syncthreads();
            const uint32_t* node = merge_nodes<kThreads>(q, nodes, nodes + node_words(kChunks), nchunks, true);
            if (tid == 0) {
                const fq x = challenge_of(node);
                if (fq_is_zero(x)) atomicOr(&sh.status, kTailZero);
                sh.x = x;
            }
            __syncthreads();
            const fq x = sh.x;
            const bool cross = !stage || h > 1;  // the last commitment has no cross terms
            const uint32_t folded = stage ? h : s;  // ring of the folded commitment
            uint4* out = reinterpret_cast<uint4*>(sh.rows);  // 3 x h coefficients, once the rows are read
            if (tid < 32) {
                if (tid == 0) {
                    const fq xi = fq_inv_steps(x, sh.inv_table);
                    sh.x_inv = xi;
                    sh.inverse = fq_mul(sh.inverse, xi);
                }
            } else {
                const uint32_t w = tid - 32;
                // ---- fold, residues
                if (!stage) {
                    // columns i and i + h; even and odd coefficients are transformed by themselves
                    const bool first = L == jb.L;
                    for (uint32_t i = w; i < 2 * h * s; i += kWorkers) {
                        const uint32_t gen = i >> (L + l), e = i & (h * s - 1), col = e >> L, t = e & (s - 1);
                        fq a, b;
                        if (first) {
                            const PastL1<uint4> src = gen ? jb.g + (((uint64_t)(col * kRank + k) << L) + t) : jb.m + e;
                            a = ldq(src, 0), b = ldq(src, (uint64_t)(gen ? kRank : 1) << (L + l));
                        } else {
                            const uint4* src = poly + gen * kHalf * kHalf + e;
                            a = lds(src, 0), b = lds(src, h * s);
                        }
                        const fq v = gen ? fq_fma(b, x, a) : fq_fma(a, x, b);
                        stq(sh.vec[gen], e, v);
                        put_residues(sh, (gen * h + col) * 2 + (t & 1u), l, t >> 1, v, pc);
                    }
                } else {
                    // even + y odd, and y even + X odd, whose top coefficient wraps around with a sign
                    for (uint32_t i = w; i < 2 * h * h; i += kWorkers) {
                        const uint32_t gen = i >> (2 * l), e = i & (h * h - 1), col = e >> l, j = e & (h - 1);
                        const uint4* src = sh.vec[gen] + col * s;
                        const fq a = lds(src, 2 * j);
                        fq v;
                        if (gen) {
                            const fq b = lds(src, j ? 2 * j - 1 : s - 1);
                            v = fq_fma(j ? b : fq_neg(b), x, a);
                        } else {
                            v = fq_fma(a, x, lds(src, 2 * j + 1));
                        }
                        stq(poly + gen * kHalf * kHalf, e, v);
                        put_residues(sh, gen * h + col, l, j, v, pc);
                    }
                }
                workers_sync();
                const uint32_t log_polys = stage ? L : L + 1;
                switch (l) {
                    case 0: forward_rows<0>(sh, log_polys, w, pc); break;
                    case 1: forward_rows<1>(sh, log_polys, w, pc); break;
                    case 2: forward_rows<2>(sh, log_polys, w, pc); break;
                    case 3: forward_rows<3>(sh, log_polys, w, pc); break;
                    case 4: forward_rows<4>(sh, log_polys, w, pc); break;
                    default: forward_rows<5>(sh, log_polys, w, pc); break;
                }
                workers_sync();
                // ---- products: at most 32 of 2^56 a sum
                if (w < kPrimes * h) {
                    const uint32_t prime = w >> l, slot = w & (h - 1), rowlen = h + 1, p = pc.p[prime];
                    const uint32_t* at = sh.rows + prime * rowlen + slot;
                    const uint32_t colstep = kPrimes * rowlen;
                    uint64_t s0 = 0, s1 = 0, s2 = 0, s3 = 0;
                    uint32_t full;
                    if (!stage) {
                        const uint32_t* gat = at + 2 * h * colstep;
#pragma unroll 4
                        for (uint32_t col = 0; col < h; ++col) {
                            const uint32_t me = at[2 * col * colstep], mo = at[(2 * col + 1) * colstep];
                            const uint32_t ge = gat[2 * col * colstep], go = gat[(2 * col + 1) * colstep];
                            s0 += (uint64_t)ge * me;
                            s3 += (uint64_t)go * mo;
                            s1 += (uint64_t)go * me;
                            s2 += (uint64_t)ge * mo;
                        }
                        // the even part of the full product: even even + Y odd odd, Y the slot's
                        // evaluation point, the square of the next stage's twiddle
                        const Tw y = sh.fwd[prime][h + slot];
                        full = red64_lazy(s0, pc, prime) +
                               shoup_mul(shoup_mul(red64_lazy(s3, pc, prime), y, p), y, p);
                    } else {
                        const uint32_t hh = h / 2;
                        const uint32_t* gat = at + h * colstep;
                        if (h == 1) s0 = (uint64_t)at[0] * gat[0];
#pragma unroll 4
                        for (uint32_t col = 0; col < hh; ++col) {
                            const uint32_t ml = at[col * colstep], mr = at[(col + hh) * colstep];
                            const uint32_t gl = gat[col * colstep], gr = gat[(col + hh) * colstep];
                            s0 += (uint64_t)gl * ml + (uint64_t)gr * mr;
                            s1 += (uint64_t)gr * ml;
                            s2 += (uint64_t)gl * mr;
                        }
                        full = red64_lazy(s0, pc, prime);
                    }
                    uint32_t* sum = sh.sums + prime * rowlen + slot;
                    sum[0] = shoup_one(full, pc.one_s[prime], p);
                    sum[colstep] = red_below(red64_lazy(s1, pc, prime), 2 * p);
                    sum[2 * colstep] = red_below(red64_lazy(s2, pc, prime), 2 * p);
                }
                workers_sync();
                const uint32_t nsums = cross ? 3 : 1;
                switch (l) {
                    case 0: inverse_rows<0>(sh, nsums, w, pc, ts); break;
                    case 1: inverse_rows<1>(sh, nsums, w, pc, ts); break;
                    case 2: inverse_rows<2>(sh, nsums, w, pc, ts); break;
                    case 3: inverse_rows<3>(sh, nsums, w, pc, ts); break;
                    case 4: inverse_rows<4>(sh, nsums, w, pc, ts); break;
                    default: inverse_rows<5>(sh, nsums, w, pc, ts); break;
                }
                workers_sync();
                if (w < nsums * h) {
                    const uint32_t sum = w >> l, j = w & (h - 1);
                    uint32_t y[kPrimes];
#pragma unroll
                    for (int i = 0; i < kPrimes; ++i) y[i] = sh.sums[(sum * kPrimes + i) * (h + 1) + j];
                    stq(out, w, crt_from_scaled(y, cc));
                } else if (w - 3 * kHalf < folded) {  // other warps
                    // what needs no inverse of the folded commitment C + x^-1 L + x R (C's even
                    // part in the second stage)
                    const uint32_t e = w - 3 * kHalf;
                    stq(sh.r, e, fq_fma(lds(sh.c, e << stage), x, lds(sh.r, e)));
                }
            }
            __syncthreads();
            // ---- this coordinate's commitments: the products over the generators'
            // factor, and the folded commitment
            const uint32_t nsums = cross ? 3 : 1, sum = tid >> l, e = tid - 3 * h;  // e wraps below
            const bool product = tid < nsums * h, fold = e < folded;
            fq v = fq_zero();
            if (product || fold)
                v = fq_fma(product ? fq_zero() : lds(sh.r, e), product ? sh.inverse : sh.x_inv,
                           product ? lds(out, tid) : lds(sh.l, e));
            __syncthreads();
            // where the cross terms go in the proof: this round's record, or the next one's
            uint32_t* terms = rec + 2 * module_words(L) + (stage ? 2 * module_words(l) + 2 : 0u);
            if (product) stq(out, tid, v);
            if (fold || (product && sum)) {
                uint32_t j = fold ? e : tid & (h - 1);
                if (!stage && !fold && sum == 1) {
                    // odd times even coefficients, times X to be L
                    if (j == h - 1) v = fq_neg(v);
                    j = (j + 1) & (h - 1);
                }
                const uint32_t ring = fold && !stage ? L : l;
                uint32_t* to = fold ? (stage ? jb.c_image : jb.ct_image) : terms + (sum - 1) * module_words(l);
                stq(fold ? sh.c : sum == 1 ? sh.l : sh.r, j, v);
                store_element(to, ring, (k << ring) + j, v);
            }
            __syncthreads();
            if (tid < folded) {
                // the commitment of what was folded, against the folded commitment
                fq got = lds(out, stage ? tid : tid >> 1);
                if (!stage && (tid & 1u)) got = fq_add(lds(out, h + (tid >> 1)), lds(out, 2 * h + (tid >> 1)));
                if (!fq_eq(got, lds(sh.c, tid))) atomicOr(&sh.status, 1u << (2 * (round - jb.round) + stage));
            }
            image = stage ? jb.c_image : jb.ct_image;
            if (stage) rec = terms;
            if (!stage || l > 0) cluster_barrier();
        }
    }
    __syncthreads();
    if (tid == 0) jb.status[k] = sh.status;
    if (k == 0 && tid == 0) {
        const uint4 v = poly[0];
        jb.opening[0] = make_uint2(v.x, v.y);
        jb.opening[1] = make_uint2(v.z, v.w);
    }
}

}  // namespace

cudaError_t tail_opt_in() {
    return cudaFuncSetAttribute(tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Shared));
}

cudaError_t launch_tail_jobs(const DeviceTables& T, const TailJob* jobs, int n, cudaStream_t st, bool beside) {
    if (n <= 0) return cudaSuccess;
    if (n > kTailJobs) return cudaErrorInvalidValue;
    TailJobs J;
    J.beside = beside;
    for (int i = 0; i < n; ++i) {
        if (jobs[i].L < 1 || jobs[i].L > kTailLog) return cudaErrorInvalidValue;
        J.j[i] = jobs[i];
    }
    const HostTables& H = host_tables();
    TailScales ts;
    for (uint32_t l = 0; l < kTailLog; ++l)
        for (int i = 0; i < kPrimes; ++i) ts.f[l][i] = Tw{H.fin[i][l], H.fins[i][l]};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kRank * (uint32_t)n);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = sizeof(Shared);
    cfg.stream = st;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kRank;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, tail_kernel, J, T.pc, T.cc, ts, T.fwd, T.inv);
}

}  // namespace dm

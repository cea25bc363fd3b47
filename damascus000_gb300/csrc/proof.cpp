#include "proof.h"

#include <chrono>

#include <cstring>

#include "dm_nvtx.h"
#include "host_blake3.h"

namespace dm {

namespace {

// Commitment slots in comm_ (each 8 * S elements).  L' has at most half of them and
// lies in its slot's second half: the first half, and so comm_, begins with the small
// words of a chain (ChainLayout).
enum Slot { kLp = 0, kC = 1, kL = 2, kR = 3, kCt = 4, kV = 5, kRp = 6, kChk = 7, kSlots = 8 };
constexpr uint32_t kMaxParts = kMaxMacParts;
// Pinned tail after the three commitment slots: [0,32) file id, [32,40) check
// flags, [48,64) m*.  The file id and the flags are written there by the kernels
// (mapped pinned memory), like the commitments of small rings that the finishes
// mirror into the slots, so such a stage needs no device-to-host copy; m* is
// copied once per proof.
constexpr size_t kTail = 128;

constexpr uint32_t kRows = kRank * kPrimes;  // MAC rows per job: (coordinate, prime)

void unpack_module(const uint8_t* src, uint32_t n, Module& m) {
    m.n = n;
    m.c.resize((size_t)kRank * n);
    const uint4* p = reinterpret_cast<const uint4*>(src);
    for (size_t i = 0; i < m.c.size(); ++i) m.c[i] = fq{{p[i].x, p[i].y, p[i].z, p[i].w}};
}

// The last rounds from a ring of 2^L: the family and the witness read; butterflies of
// every round's transforms, of half and of a quarter of its coefficients.
double tail_bytes(uint32_t L) { return (kRank + 1) * 16.0 * (double)(1u << 2 * L); }
double tail_ops(uint32_t L) {
    double ops = 0;
    for (; L > 0; --L) ops += 0.75 * (kRank + 1) * kPrimes * (double)(1u << 2 * L) / 2 * (L - 1);
    return ops;
}

template <class J, class F>
int launch_chunks(std::vector<J>& v, F fn, cudaStream_t st, int per_launch, int* launches) {
    for (size_t i = 0; i < v.size(); i += kMaxJobs) {
        const int n = (int)std::min<size_t>(kMaxJobs, v.size() - i);
        cudaError_t e = fn(v.data() + i, n, st);
        if (e != cudaSuccess) return (int)e;
        *launches += per_launch;
    }
    return 0;
}

}  // namespace

// ============================================================== Plan

void Plan::clear() {
    hash.clear();
    unpack.clear();
    mac.clear();
    split.clear();
    triple.clear();
    gen.clear();
    fold.clear();
    for (int L = 0; L <= kLogMaxProverRing; ++L) {
        ntt[L].clear();
        finish[L].clear();
    }
    tail.clear();
    d2h.clear();
    wait_events.clear();
    record_events.clear();
    fills.clear();
}

bool Plan::empty() const {
    if (!hash.empty() || !unpack.empty() || !gen.empty() || !fold.empty() || !mac.empty() || !split.empty() ||
        !triple.empty() || !tail.empty())
        return false;
    for (int L = 0; L <= kLogMaxProverRing; ++L)
        if (!ntt[L].empty() || !finish[L].empty())
            return false;
    return d2h.empty();
}

int Plan::launch(Context* ctx, cudaStream_t st, std::string* err) {
    const int n = launch_all(ctx, st, err);
    for (auto& f : fills) {
        if (n < 0) ctx->prover_cache()->poison(f);
        else ctx->prover_cache()->publish(f);
    }
    return n;
}

int Plan::launch_all(Context* ctx, cudaStream_t st, std::string* err) {
    const DeviceTables& T = ctx->tables();
    int launches = 0;
    for (cudaEvent_t e : wait_events) {
        const cudaError_t we = cudaStreamWaitEvent(st, e, 0);
        if (we != cudaSuccess) {
            *err = std::string("wait for a cached generator family: ") + cudaGetErrorString(we);
            return kECuda;
        }
    }
    const bool prof = ctx->profiling();
    auto timed = [&](const char* name, double bytes, double ops, auto&& body) -> int {
        cudaEvent_t a = nullptr;
        if (prof) {
            a = ctx->take_event();
            cudaEventRecord(a, st);
        }
        const int before = launches;
        NvtxRange range(name);
        const int rc = body();
        if (rc != 0) {
            *err = std::string(name) + ": " + cudaGetErrorString((cudaError_t)rc);
            return kECuda;
        }
        if (a) {
            cudaEvent_t b = ctx->take_event();
            cudaEventRecord(b, st);
            ctx->record(name, a, b, bytes, ops, launches - before, st);
        }
        return 0;
    };
    int rc;
    // unpacking and generators need nothing of the hash, which they run beside
    auto beside_hash = [&](auto fn) {
        return [&, fn](auto* jobs, int n, cudaStream_t s) { return fn(jobs, n, s, !hash.empty()); };
    };
    if (!hash.empty()) {
        double bytes = 0, ops = 0;
        for (auto& j : hash) {
            bytes += (double)j.len;
            ops += (double)((j.len + 63) / 64 + (j.len + 1023) / 1024);
        }
        if ((rc = timed("file_hash", bytes, ops, [&] {
                 for (size_t i = 0; i < hash.size(); i += kMaxJobs) {
                     const int n = (int)std::min<size_t>(kMaxJobs, hash.size() - i);
                     int k = 1;
                     cudaError_t e = launch_hash_jobs(hash.data() + i, n, st, &k);
                     if (e != cudaSuccess) return (int)e;
                     launches += k;
                 }
                 return 0;
             })))
            return rc;
    }
    if (!unpack.empty()) {
        double bytes = 0;
        for (auto& j : unpack) bytes += (double)j.len + (double)j.total * 16;
        if ((rc = timed("unpack_witness", bytes, 0,
                        [&] { return launch_chunks(unpack, beside_hash(launch_unpack_jobs), st, 1, &launches); })))
            return rc;
    }
    if (!gen.empty()) {
        double bytes = 0, ops = 0;
        for (auto& j : gen) {
            bytes += (double)j.total * 16;
            ops += (double)j.total;
        }
        if ((rc = timed("gen_generators", bytes, ops, [&] { return launch_chunks(gen, beside_hash(launch_gen_jobs), st, 1, &launches); })))
            return rc;
    }
    if (!fold.empty()) {
        double bytes = 0;
        for (auto& j : fold) bytes += (double)j.n * (j.mode == kCombine || j.mode == kCombineEven ? 64 : 48);
        if ((rc = timed("fold", bytes, 0, [&] { return launch_chunks(fold, launch_fold_jobs, st, 1, &launches); })))
            return rc;
    }
    for (int L = 0; L <= kLogMaxProverRing; ++L) {
        if (ntt[L].empty()) continue;
        double polys = 0;
        for (auto& j : ntt[L]) polys += j.npolys;
        const double bytes = polys * (double)(1u << L) * (16 + 4 * kPrimes);  // 16 B read + 9 residues written
        const double ops = polys * (double)kPrimes * (double)(1u << L) / 2 * L;  // butterflies
        if ((rc = timed("ntt_fwd", bytes, ops, [&] {
                 for (size_t i = 0; i < ntt[L].size(); i += kMaxJobs) {
                     const int n = (int)std::min<size_t>(kMaxJobs, ntt[L].size() - i);
                     cudaError_t e = launch_ntt_jobs(T, ntt[L].data() + i, n, (uint32_t)L, st,
                                                     ctx->tuning(kTuneNttGroup, (uint32_t)L),
                                                     ctx->tuning(kTuneNttRadix, (uint32_t)L));
                     if (e != cudaSuccess) return (int)e;
                     ++launches;
                 }
                 return 0;
             })))
            return rc;
    }
    for (int pass = 0; pass < 3; ++pass) {
        auto& v = pass == 0 ? mac : (pass == 1 ? split : triple);
        if (v.empty()) continue;
        // columns read: count (plain, split) or 2 * count (triple pairs)
        const double cols_per_count = pass == 2 ? 2.0 : 1.0;
        const double macs_per_col = pass == 0 ? 1.0 : 2.0;
        double macs = 0, bytes = 0;
        for (auto& j : v) {
            const double cols = (double)j.count * cols_per_count;
            macs += cols * (double)kRows * (double)(1u << j.L) * macs_per_col;
            // G residues (4 B per column, coordinate, prime, slot) + M residues (shared by 8 coordinates)
            bytes += cols * (double)(1u << j.L) * (kRows * 4.0 + kPrimes * 4.0);
        }
        const char* name = pass == 0 ? "mac" : (pass == 1 ? "mac_split" : "mac");
        if ((rc = timed(name, bytes, macs, [&] {
                 for (size_t i = 0; i < v.size(); i += kMaxJobs) {
                     const int n = (int)std::min<size_t>(kMaxJobs, v.size() - i);
                     int k = 1;
                     cudaError_t e = pass == 2 ? launch_mac_triple_jobs(T, v.data() + i, n, st, &k)
                                               : launch_mac_jobs(T, v.data() + i, n, pass == 1, st, &k);
                     if (e != cudaSuccess) return (int)e;
                     launches += k;
                 }
                 return 0;
             })))
            return rc;
    }
    bool finishing = false;  // a finish is launched: the others run beside it
    for (int L = kLogMaxProverRing; L >= 0; --L) {
        if (finish[L].empty()) continue;
        double bytes = 0;
        for (auto& j : finish[L]) bytes += ((double)j.parts + 2.0) * j.rows * (1u << L) * 4 + (j.rows / kPrimes) * (1u << L) * 16.0;
        if ((rc = timed("finish", bytes, 0, [&] {
                 for (size_t i = 0; i < finish[L].size(); i += kMaxJobs) {
                     const int n = (int)std::min<size_t>(kMaxJobs, finish[L].size() - i);
                     cudaError_t e = launch_finish_jobs(T, finish[L].data() + i, n, (uint32_t)L, st, finishing);
                     finishing = true;
                     if (e != cudaSuccess) return (int)e;
                     launches += L <= 10 ? 1 : 2;  // the fused finish, or inverse transform + CRT
                 }
                 return 0;
             })))
            return rc;
    }
    if (!tail.empty()) {
        double bytes = 0, ops = 0;
        for (auto& j : tail) bytes += tail_bytes(j.L), ops += tail_ops(j.L);
        if ((rc = timed("last_rounds", bytes, ops, [&] {
                 for (size_t i = 0; i < tail.size(); i += kTailJobs) {
                     const int n = (int)std::min<size_t>(kTailJobs, tail.size() - i);
                     const cudaError_t e = launch_tail_jobs(T, tail.data() + i, n, st, i > 0);
                     if (e != cudaSuccess) return (int)e;
                     ++launches;
                 }
                 return 0;
             })))
            return rc;
    }
    for (cudaEvent_t e : record_events) {
        const cudaError_t re = cudaEventRecord(e, st);
        if (re != cudaSuccess) {
            *err = std::string("record a cached generator family: ") + cudaGetErrorString(re);
            return kECuda;
        }
    }
    for (auto& c : d2h) {
        cudaError_t e = cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) {
            *err = std::string("device-to-host copy: ") + cudaGetErrorString(e);
            return kECuda;
        }
    }
    return launches;
}

// ============================================================== ProofState

uint64_t ProofState::footprint(uint64_t len) {
    uint32_t d;
    uint64_t S;
    if (!square_layout_for_byte_len(len, &d, &S)) return ~0ull;
    const uint64_t S2 = S * S;
    auto r = [](uint64_t b) { return (b + 255) & ~255ull; };
    return r(len + 16) + r(file_hash_scratch_words(len) * 4) + r(S2 * 16) + r(S2 / 2 * 16) + r(8 * S2 * 16) +
           r(4 * S2 * 16) + r(S2 * kPrimes * 4) + r(8 * S2 * kPrimes * 4) + r(3ull * kMaxParts * kRows * S * 4) +
           r((uint64_t)kSlots * kRank * S * 16);
}

const uint4* ProofState::g_round0() const { return cached_.g ? cached_.g : g_a_.as<uint4>(); }

void ProofState::release() {
    if (cached_.entry) {
        // a request ends only after its last stage's copies landed: nothing of it
        // still reads the entry
        ctx_->prover_cache()->release(cached_);
        cached_ = ProverGenCache::Ref{};
    }
    mem_.reset();
    if (pinned_) ctx_->put_pinned(pinned_, pinned_bytes_);
    pinned_ = nullptr;
}

ProofState::~ProofState() { release(); }

int ProofState::fail(int code, const std::string& msg) {
    stage_ = Stage::Failed;
    err_ = msg;
    err_code_ = code;
    return code;
}

uint32_t ProofState::stage_L() const {
    if (stage_ == Stage::Init) return d_;
    if (stage_ == Stage::Vec) return d_ - (uint32_t)round_;
    if (stage_ == Stage::Poly) return d_ - (uint32_t)round_ - 1;
    return 0;
}

bool ProofState::opening(fq* out) const {
    if (!have_opening_) return false;
    *out = opening_;
    return true;
}

int ProofState::setup(const uint8_t* file, uint64_t len, bool on_device, const uint8_t seed[32],
                      const uint8_t epoch[32], uint64_t max_preprocess_bytes, cudaStream_t stream) {
    uint32_t d;
    uint64_t S;
    if (!square_layout_for_byte_len(len, &d, &S)) return fail(kEInval, "square witness dimension overflow");
    const uint64_t est = S * S * 16 * 2;  // io.rs:42-49
    if (est > max_preprocess_bytes)
        return fail(kEInval, "full witness expansion requires " + std::to_string(est) +
                                 " bytes, above max_preprocess_bytes=" + std::to_string(max_preprocess_bytes) +
                                 "; split the file into smaller statements");
    if (d > (uint32_t)kMaxDepth)
        return fail(kEUnsupported,
                    "fold depth " + std::to_string(d) + " exceeds the supported maximum " + std::to_string(kMaxDepth));
    if (len > 0 && file == nullptr) return fail(kEInval, "null file buffer");
    d_ = d;
    S_ = N_ = n_ = (uint32_t)S;
    len_ = len;
    mcols_ = (uint32_t)((coeff_count_for_byte_len(len) + S - 1) / S);
    alloc_stream_ = stream;
    std::memcpy(seed_, seed, 32);
    const uint64_t S2 = S * S;
    int rc = kOk;
    for (int attempt = 0; attempt < 2; ++attempt) {
        Layout l;
        const size_t file_at = on_device ? 0 : l.put(len + 16);
        const size_t at[] = {l.put(file_hash_scratch_words(len) * 4),
                             l.put(S2 * 16),
                             l.put(S2 / 2 * 16),
                             l.put(8 * S2 * 16),
                             l.put(4 * S2 * 16),
                             l.put(S2 * kPrimes * 4),
                             l.put(8 * S2 * kPrimes * 4),
                             l.put((uint64_t)kSlots * kRank * S * 16),
                             l.put(3ull * kMaxParts * kRows * S * 4)};
        rc = mem_.alloc(ctx_, l.total(), stream);
        if (rc == kOk) {
            if (!on_device) file_ = Span(mem_, file_at);
            Span* spans[] = {&hash_scratch_, &m_a_, &m_b_, &g_a_, &g_b_, &mhat_, &ghat_, &comm_, &partials_};
            for (int i = 0; i < 9; ++i) *spans[i] = Span(mem_, at[i]);
            if (chained_) chain_ = Span(mem_, at[7] - chain_layout().id);  // up to comm_ and into it
        }
        if (rc == kOk || !ctx_->prover_cache()) break;
        // the budget is held by cached generator families: drop unreferenced ones, once
        release();
        if (!ctx_->prover_cache()->trim(footprint(len))) break;
    }
    if (rc != kOk) return fail(rc, "HBM budget exhausted allocating prover state (" + std::to_string(footprint(len)) + " bytes)");
    pinned_bytes_ = chained_ ? chain_layout().copied() : 3ull * kRank * S * 16 + kTail + tail_layout().out_bytes;
    pinned_ = static_cast<uint8_t*>(ctx_->get_pinned(pinned_bytes_));
    if (!pinned_) return fail(kECuda, "cudaMallocHost failed");
    if (chained_) {
        const ChainLayout l = chain_layout();
        if (l.id > 4 * S2 * kPrimes * 4) return fail(kEInvariant, "no room for the chain");
        cudaError_t e = cudaMemsetAsync(chain_.as<uint8_t>() + l.flags, 0, l.end - l.flags, stream);
        if (e != cudaSuccess) return fail(kECuda, std::string("clear check flags: ") + cudaGetErrorString(e));
    } else {
        // the check flags start clear (kernels only ever set them); no kernel of this
        // request has been launched yet, and the buffer's previous owner has finished
        std::memset(pinned_ + 3ull * kRank * S * 16, 0, kTail);
    }
    d_file_ = on_device ? file : file_.as<uint8_t>();
    if (!on_device && len) {
        cudaError_t e = cudaMemcpyAsync(file_.as<uint8_t>(), file, len, cudaMemcpyHostToDevice, stream);
        if (e != cudaSuccess) return fail(kECuda, std::string("H2D file: ") + cudaGetErrorString(e));
    }
    blake3_keyed_hash(seed, "g0", 2, st_.g_0_seed);  // sis.rs:70, 208-210
    st_.original_len_bytes = len;
    st_.d = d;
    std::memcpy(epoch_copy_, epoch, 32);  // the transcript is keyed after the Init stage yields the file id
    stage_ = Stage::Init;
    return kOk;
}

// Transforms and the multiply-accumulate of a commitment stage over `cols`
// columns of ring 2^L of which the first `c` can be nonzero: the full sum into
// `part`, and for cols >= 2 the cross terms L (pairs (i, i + cols/2)) and R.
// With c <= cols/2 the witness half from cols/2 on is zero: only c witness
// columns and the generator columns [0, c) and [cols/2, cols/2 + c) are
// transformed and read, and R is zero.  Returns whether the cross terms exist.
bool ProofState::plan_commit(Plan& P, uint32_t L, uint32_t cols, uint32_t c, const uint4* m_src, const uint4* g_src,
                             uint32_t* part, uint32_t* ghat, bool g_transformed) {
    const uint64_t s = 1ull << L;
    uint32_t* mh = mhat_.as<uint32_t>();
    uint32_t* gh = ghat ? ghat : ghat_.as<uint32_t>();
    const uint64_t gcol_in = 8 * s, gcol_out = 8 * (uint64_t)kPrimes * s;  // one generator column
    auto ntt = [&](const uint4* src, uint32_t* dst, uint64_t polys) {
        // generator columns that are already in `ghat` (a cached family) are not transformed again
        if (polys && !(g_transformed && dst != mh)) P.ntt[L].push_back(NttJob{src, dst, polys, 0});
    };
    if (cols < 2) {
        ntt(m_src, mh, c);
        ntt(g_src, gh, 8ull * c);
        parts_ = ctx_->mac_parts(kTuneMacPlain, L, (uint32_t)s, c);
        P.mac.push_back(MacJobX{gh, mh, part, nullptr, nullptr, 0, 0, c, parts_, 0, 0, L});
        return false;
    }
    const uint32_t half = cols / 2;
    const uint32_t kc = (uint32_t)ctx_->tuning(kTuneTripleCoords, L);
    const int bps = ctx_->tuning(kTuneMacTriple, L);
    if (c <= half) {
        ntt(m_src, mh, c);
        ntt(g_src, gh, 8ull * c);
        ntt(g_src + half * gcol_in, gh + half * gcol_out, 8ull * c);
        parts_ = ctx_->mac_parts_for(bps, (uint32_t)(s / 2), c, kRows / kc);
        const size_t ps = (size_t)parts_ * kRows * s;
        P.triple.push_back(MacJobX{gh, mh, part, part + ps, part + 2 * ps, 0, 0, c, parts_, 0, half, L, kc});
    } else {
        ntt(m_src, mh, cols);
        ntt(g_src, gh, 8ull * cols);
        parts_ = ctx_->mac_parts_for(bps, (uint32_t)(s / 2), half, kRows / kc);
        const size_t ps = (size_t)parts_ * kRows * s;
        P.triple.push_back(MacJobX{gh, mh, part, part + ps, part + 2 * ps, 0, 0, half, parts_, 0, 0, L, kc});
    }
    return true;
}

size_t ProofState::record_at(uint64_t round) const {
    size_t at = statement_encoded_size(S_) + 8;
    for (uint64_t j = 0; j < round; ++j) at += record_encoded_size(S_ >> j, S_ >> (j + 1));
    return at;
}

// Check flags: two per round, then the flag of a zero challenge and the ticket of
// the challenge kernel's last block, and the last rounds' status.
ProofState::ChainLayout ProofState::chain_layout() const {
    auto r = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t module = module_encoded_size(S_);
    ChainLayout l{};
    l.cvs = 0;
    l.challenges = r(challenge_scratch_words((uint32_t)(module / 4), (uint32_t)(2 * module / 4)) * 4);
    l.c = l.challenges + r(2ull * d_ * 32);
    l.ct = l.c + r(module);
    l.proof = l.ct + r(module);
    l.id = l.proof + r(proof_encoded_size(d_));
    l.flags = l.id + 32;
    l.end = l.flags + (2ull * d_ + 2 + kRank) * 4;
    return l;
}
// Up to `id` 1,152 S bytes (a proof is 896 S, an encoded commitment 128 S) and less than
// 8 KiB of lengths, challenges and rounding, in the 144 S^2 of half of ghat_; from there
// on 176 bytes at most in half a slot.
static_assert(1152u * (1u << kMinDepth) + 8192u <= (4u * kPrimes * 4 << 2 * kMinDepth), "room in half of ghat_");
static_assert(32 + (2 * kMaxDepth + 2 + kRank) * 4 <= (kRank * 16 << kMinDepth) / 2, "room in half a slot");

void ProofState::plan_stage(Plan& P) {
    const uint32_t S = S_;
    const size_t slot = (size_t)kRank * S;
    uint4* C = comm_.as<uint4>();
    auto cs = [&](int i) { return C + (size_t)i * slot + (i == kLp ? slot / 2 : 0); };
    uint32_t* part = partials_.as<uint32_t>();
    uint8_t* tail = pinned_ + 3 * slot * 16;
    uint32_t* flags = reinterpret_cast<uint32_t*>(tail + 32);
    // The three commitment slots the host reads after a stage.  Up to rings of
    // 2^(kCopyFromL - 1) the finishes mirror them into pinned host memory (no copy
    // to issue, which is what the small, latency-bound stages pay for); from
    // 2^kCopyFromL on (64 KiB slots and more; few, long stages) one copy per slot,
    // which keeps the finishes' stores on the device.
    constexpr uint32_t kCopyFromL = 9;
    const uint32_t Lout = stage_ == Stage::Init ? d_ : (stage_ == Stage::Vec ? d_ - (uint32_t)round_
                                                                                : d_ - (uint32_t)round_ - 1);
    const bool mapped = !chained_ && Lout < kCopyFromL;
    uint4* hm0 = mapped ? reinterpret_cast<uint4*>(pinned_) : nullptr;
    uint4* hm1 = mapped ? reinterpret_cast<uint4*>(pinned_ + slot * 16) : nullptr;
    uint4* hm2 = mapped ? reinterpret_cast<uint4*>(pinned_ + 2 * slot * 16) : nullptr;
    auto copy3 = [&](const uint4* s0, const uint4* s1, const uint4* s2, size_t n0, size_t n12) {
        if (mapped || chained_) return;
        P.d2h.push_back(Copy{pinned_, s0, n0 * 16});
        if (s1) P.d2h.push_back(Copy{pinned_ + slot * 16, s1, n12 * 16});
        if (s2) P.d2h.push_back(Copy{pinned_ + 2 * slot * 16, s2, n12 * 16});
    };
    // chained: the encodings' places, the challenges and flags in device memory
    const ChainLayout cl = chained_ ? chain_layout() : ChainLayout{};
    uint8_t* chain = chain_.as<uint8_t>();
    // or, where the last rounds start without a chain, the images they read
    const uint32_t Lnext = stage_ == Stage::Init ? d_ : (stage_ == Stage::Poly ? d_ - (uint32_t)round_ - 1 : 0);
    tail_planned_ = allow_tail_ && !chained_ && Lnext == kTailLog;
    const TailLayout tl = tail_layout();
    uint8_t* area = ghat_.as<uint8_t>();
    auto img = [&](size_t at) { return chained_ ? reinterpret_cast<uint2*>(chain + at) : nullptr; };
    auto img_c = [&](size_t at) { return tail_planned_ ? reinterpret_cast<uint2*>(area + tl.image) : img(at); };
    auto img_lr = [&](size_t at, size_t skip) {
        return tail_planned_ ? reinterpret_cast<uint2*>(area + tl.out + 8 + skip) : img(at + skip);
    };
    auto plan_tail = [&](uint64_t round) {
        // the file id: behind the commitments, where the Init stage's hash leaves it, or known
        TailJob j = tail_job(area + tl.out + 8, area + tl.c, area + tl.ct, area + tl.opening, area + tl.status,
                             round == 0 ? reinterpret_cast<uint8_t*>(cs(kCt)) : nullptr, area + tl.image, round);
        if (round)
            for (auto& head : j.head) std::memcpy(head + 13, st_.file_id, 32);
        P.tail.push_back(j);
        P.d2h.push_back(Copy{pinned_ + 3 * slot * 16 + kTail, area + tl.out, tl.out_bytes});
    };
    auto challenge = [&](uint64_t stage, int inverse) -> const uint4* {
        return chained_ ? reinterpret_cast<const uint4*>(chain + cl.challenges) + 2 * stage + inverse : nullptr;
    };
    if (chained_) flags = reinterpret_cast<uint32_t*>(chain + cl.flags) + 2 * round_;
    auto fin = [](uint32_t* partials, uint4* out, const uint4* expect, uint32_t* flag, uint32_t parts, uint32_t mode,
                  uint4* host_out, uint2* image) {
        return FinishJobX{partials, out, expect, flag, parts, mode, kRows, 0, nullptr, host_out, image};
    };
    if (stage_ == Stage::Init) {
        const uint32_t L = d_;
        const uint64_t S2 = (uint64_t)S * S;
        P.hash.push_back(HashJob{d_file_, len_, hash_scratch_.as<uint32_t>(),
                                 chained_        ? reinterpret_cast<uint32_t*>(chain + cl.id)
                                 : tail_planned_ ? reinterpret_cast<uint32_t*>(cs(kCt))
                                                 : reinterpret_cast<uint32_t*>(tail),
                                 0});
        P.unpack.push_back(UnpackJob{d_file_, len_, m_a_.as<uint4>(), S2, 0});
        GenJob g{};
        for (int i = 0; i < 8; ++i)
            g.key[i] = (uint32_t)st_.g_0_seed[4 * i] | ((uint32_t)st_.g_0_seed[4 * i + 1] << 8) |
                       ((uint32_t)st_.g_0_seed[4 * i + 2] << 16) | ((uint32_t)st_.g_0_seed[4 * i + 3] << 24);
        g.dst = g_a_.as<uint4>();
        g.total = 8 * S2;
        g.log_n = L;
        ProverGenCache* cache = ctx_->prover_cache();
        cached_ = ProverGenCache::Ref{};
        if (cache && cache->acquire(st_.g_0_seed, L, &P, &cached_) == kOk) {
            if (cached_.fill) {
                // expand into the entry and transform every column (later holders
                // may have more nonzero witness columns than this file)
                g.dst = cached_.g;
                P.gen.push_back(g);
                P.ntt[L].push_back(NttJob{cached_.g, cached_.ghat, 8ull * S, 0});
                P.record_events.push_back(cached_.ready);
                P.fills.push_back(cached_);
            } else if (cached_.ready) {
                P.wait_events.push_back(cached_.ready);
            }
        } else {
            cached_ = ProverGenCache::Ref{};
            P.gen.push_back(g);
        }
        const bool nj = plan_commit(P, L, S, mcols_ < S ? mcols_ : S, m_a_.as<uint4>(), g_round0(), part,
                                    cached_.ghat, cached_.ghat != nullptr);
        if (nj) {
            const size_t pstride = (size_t)parts_ * kRows * S, rec = cl.proof + record_at(0) + 8;
            P.finish[L].push_back(fin(part + pstride, cs(kL), nullptr, nullptr, parts_, kFinishPlain, hm1, img_lr(rec, 0)));
            P.finish[L].push_back(fin(part + 2 * pstride, cs(kR), nullptr, nullptr, parts_, kFinishPlain, hm2,
                                      img_lr(rec, module_encoded_size(S))));
        }
        P.finish[L].push_back(fin(part, cs(kC), nullptr, nullptr, parts_, kFinishPlain, hm0, img_c(cl.proof + 48)));
        copy3(cs(kC), nj ? cs(kL) : nullptr, nj ? cs(kR) : nullptr, slot, slot);
        if (tail_planned_) {
            P.d2h.push_back(Copy{tail, cs(kCt), 32});
            plan_tail(0);
        }
        return;
    }
    const uint32_t L = d_ - (uint32_t)round_, s = 1u << L, h = s / 2;
    const uint64_t s2 = (uint64_t)s * s;
    if (stage_ == Stage::Vec) {
        P.fold.push_back(FoldJob{m_b_.as<uint4>(), m_a_.as<uint4>(), m_a_.as<uint4>() + (uint64_t)h * s, nullptr, x_,
                                 fq_zero(), (uint64_t)h * s, kFoldVec, 0, 0, challenge(2 * round_, 0)});
        const uint4* gsrc = round_ == 0 ? g_round0() : g_a_.as<uint4>();
        P.fold.push_back(FoldJob{g_b_.as<uint4>(), gsrc, gsrc + 4 * s2, nullptr, xi_, fq_zero(), 4 * s2, kFoldVec, 0, 0,
                                 challenge(2 * round_, 1)});
        P.fold.push_back(FoldJob{cs(kCt), cs(kC), cs(kL), cs(kR), xi_, x_, (uint64_t)kRank * s, kCombine, 0, 0,
                                 challenge(2 * round_, 1), challenge(2 * round_, 0)});
        // the folded witness has h columns, of which the first c can be nonzero:
        // the check and both cross terms only need those columns
        const uint32_t c = mcols_ < h ? mcols_ : h;
        if (c) {
            P.ntt[L].push_back(NttJob{m_b_.as<uint4>(), mhat_.as<uint32_t>(), c, 0});
            P.ntt[L].push_back(NttJob{g_b_.as<uint4>(), ghat_.as<uint32_t>(), 8ull * c, 0});
        }
        const uint32_t kc = (uint32_t)ctx_->tuning(kTuneSplitCoords, L);
        parts_ = ctx_->mac_parts_for(ctx_->tuning(kTuneMacSplit, L), h, c, kRows / kc);
        uint32_t* pchk = part;
        uint32_t* plp = part + (size_t)parts_ * kRows * s;
        uint32_t* prp = plp + (size_t)parts_ * kRows * h;
        P.split.push_back(
            MacJobX{ghat_.as<uint32_t>(), mhat_.as<uint32_t>(), pchk, plp, prp, 0, 0, c, parts_, 0, 0, L, kc});
        // The recomputed commitment V is checked against the folded one (Ct); the
        // host reads V's mirror as Ct, which it equals unless the check flag is set
        // (and then the stage fails before anything is absorbed).
        const size_t rec = cl.proof + record_at(round_) + 8 + 2 * module_encoded_size(s);
        P.finish[L].push_back(fin(pchk, cs(kV), cs(kCt), flags, parts_, kFinishPlain, hm0, img(cl.ct)));
        P.finish[L - 1].push_back(fin(plp, cs(kLp), nullptr, nullptr, parts_, kFinishSplitL, hm1, img(rec)));
        P.finish[L - 1].push_back(
            fin(prp, cs(kRp), nullptr, nullptr, parts_, kFinishSplitR, hm2, img(rec + module_encoded_size(h))));
        copy3(cs(kCt), cs(kLp), cs(kRp), (size_t)kRank * s, (size_t)kRank * h);
        return;
    }
    if (stage_ == Stage::Poly) {
        const uint32_t Ln = L - 1;
        const uint64_t h2 = (uint64_t)h * h;
        P.fold.push_back(FoldJob{m_a_.as<uint4>(), m_b_.as<uint4>(), nullptr, nullptr, y_, fq_zero(), h2, kFoldPoly, Ln, 0,
                                 challenge(2 * round_ + 1, 0)});
        P.fold.push_back(FoldJob{g_a_.as<uint4>(), g_b_.as<uint4>(), nullptr, nullptr, yi_, fq_zero(), 8 * h2, kFoldPolyX,
                                 Ln, 0, challenge(2 * round_ + 1, 1)});
        P.fold.push_back(FoldJob{cs(kC), cs(kCt), cs(kLp), cs(kRp), yi_, y_, (uint64_t)kRank * h, kCombineEven, Ln, 0,
                                 challenge(2 * round_ + 1, 1), challenge(2 * round_ + 1, 0)});
        const bool nj = plan_commit(P, Ln, h, mcols_ < h ? mcols_ : h, m_a_.as<uint4>(), g_a_.as<uint4>(), part);
        if (nj) {
            const size_t pstride = (size_t)parts_ * kRows * h, rec = cl.proof + record_at(round_ + 1) + 8;
            P.finish[Ln].push_back(fin(part + pstride, cs(kL), nullptr, nullptr, parts_, kFinishPlain, hm1, img_lr(rec, 0)));
            P.finish[Ln].push_back(fin(part + 2 * pstride, cs(kR), nullptr, nullptr, parts_, kFinishPlain, hm2,
                                       img_lr(rec, module_encoded_size(h))));
        }
        // as in the vector stage: the recomputed Chk's mirror is the folded C
        P.finish[Ln].push_back(fin(part, cs(kChk), cs(kC), flags + 1, parts_, kFinishPlain, hm0, img_c(cl.c)));
        if (tail_planned_) plan_tail(round_ + 1);
        copy3(cs(kC), nj ? cs(kL) : nullptr, nj ? cs(kR) : nullptr, (size_t)kRank * h, (size_t)kRank * h);
        if (round_ + 1 == d_) P.d2h.push_back(Copy{tail + 48, m_a_.as<uint4>(), 16});
    }
}

int ProofState::chain_next(cudaStream_t stream) {
    const ChainLayout l = chain_layout();
    uint8_t* chain = chain_.as<uint8_t>();
    if (stage_ == Stage::Poly) {
        N_ = n_ = n_ / 2;
        round_ += 1;
    }
    if (stage_ != Stage::Vec && d_ - round_ <= kTailLog) return chain_tail(stream);
    const bool poly = stage_ == Stage::Vec;  // the challenge that ends this stage
    const uint32_t n = S_ >> round_;
    const size_t c = module_encoded_size(n), lr = module_encoded_size(poly ? n / 2 : n);
    ChallengeJob j{};
    j.c = reinterpret_cast<const uint32_t*>(chain + (poly ? l.ct : (round_ == 0 ? l.proof + 48 : l.c)));
    j.lr = reinterpret_cast<const uint32_t*>(chain + l.proof + record_at(round_) + 8 + (poly ? 2 * c : 0));
    j.c_words = (uint32_t)(c / 4);
    j.lr_words = (uint32_t)(2 * lr / 4);
    j.file_id = reinterpret_cast<const uint32_t*>(chain + l.id);
    challenge_head(epoch_copy_, round_, poly, j.head);
    j.poly = poly;
    j.cvs = reinterpret_cast<uint32_t*>(chain + l.cvs);
    uint32_t* flags = reinterpret_cast<uint32_t*>(chain + l.flags);
    j.zero = flags + 2 * d_;
    j.ticket = flags + 2 * d_ + 1;
    j.out = reinterpret_cast<uint4*>(chain + l.challenges) + 2 * (2 * round_ + (poly ? 1 : 0));
    const double bytes = 4.0 * (j.c_words + j.lr_words);
    const cudaError_t e =
        ctx_->timed("challenge", bytes, bytes / 64, stream, [&] { return launch_challenge(j, stream); });
    if (e != cudaSuccess) return fail(kECuda, std::string("challenge: ") + cudaGetErrorString(e));
    stage_ = poly ? Stage::Poly : Stage::Vec;
    return kOk;
}

TailJob ProofState::tail_job(uint8_t* records, uint8_t* c_image, uint8_t* ct_image, uint8_t* opening, uint8_t* status,
                             const uint8_t* file_id, const uint8_t* image, uint64_t round) const {
    const size_t slot = (size_t)kRank * S_;
    TailJob j{};
    j.L = d_ - (uint32_t)round;
    j.round = (uint32_t)round;
    j.m = m_a_.as<uint4>();
    j.g = round == 0 ? g_round0() : g_a_.as<uint4>();
    j.c = comm_.as<uint4>() + kC * slot;
    j.l = comm_.as<uint4>() + kL * slot;
    j.r = comm_.as<uint4>() + kR * slot;
    challenge_head(epoch_copy_, 0, false, j.head[0]);
    challenge_head(epoch_copy_, 0, true, j.head[1]);
    j.file_id = reinterpret_cast<const uint32_t*>(file_id);
    j.image = reinterpret_cast<const uint32_t*>(image);
    j.record = reinterpret_cast<uint32_t*>(records);
    j.c_image = reinterpret_cast<uint32_t*>(c_image);
    j.ct_image = reinterpret_cast<uint32_t*>(ct_image);
    j.opening = reinterpret_cast<uint2*>(opening);
    j.status = reinterpret_cast<uint32_t*>(status);
    return j;
}

int ProofState::tail_failure(const uint32_t status[kRank], uint32_t rounds) {
    uint32_t all = 0;
    for (int k = 0; k < kRank; ++k) all |= status[k];
    for (uint32_t i = 0; i < rounds; ++i) {
        if (all >> (2 * i) & 1u) return 1;
        if (all >> (2 * i + 1) & 1u) return 2;
    }
    return 0;
}

// The remaining rounds in one launch, and the proof to the host.
int ProofState::chain_tail(cudaStream_t stream) {
    const ChainLayout l = chain_layout();
    uint8_t* chain = chain_.as<uint8_t>();
    uint8_t* proof = chain + l.proof;
    const TailJob j = tail_job(proof + record_at(round_) + 8, chain + l.c, chain + l.ct,
                               proof + proof_encoded_size(d_) - 16, chain + l.flags + 4 * (2 * d_ + 2), chain + l.id,
                               round_ == 0 ? proof + 48 : chain + l.c, round_);
    cudaError_t e = ctx_->timed("last_rounds", tail_bytes(j.L), tail_ops(j.L), stream,
                                [&] { return launch_tail_jobs(ctx_->tables(), &j, 1, stream); });
    // the proof, and the file id and the flags behind it
    if (e == cudaSuccess) e = cudaMemcpyAsync(pinned_, proof, l.copied(), cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess) return fail(kECuda, std::string("last rounds: ") + cudaGetErrorString(e));
    N_ = n_ = 1;
    round_ = d_;
    have_opening_ = true;
    stage_ = Stage::Done;
    return kOk;
}

ProofState::TailLayout ProofState::tail_layout() {
    auto r = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t module = r(module_encoded_size(1u << kTailLog));
    TailLayout l{};
    l.image = 0;
    l.c = module;
    l.ct = 2 * module;
    l.out = 3 * module;
    l.opening = l.out;
    for (uint32_t L = kTailLog; L > 0; --L) l.opening += record_encoded_size(1u << L, 1u << (L - 1));
    l.status = l.opening + 16;
    l.out_bytes = l.status + 4 * kRank - l.out;
    return l;
}

// The rounds that ran on the device from their records' encodings; *done is false if a
// challenge candidate was zero, and the host goes on with this round.
int ProofState::complete_tail(bool* done) {
    const TailLayout l = tail_layout();
    const uint8_t* out = pinned_ + 3ull * kRank * S_ * 16 + kTail;
    uint32_t status[kRank];
    std::memcpy(status, out + (l.status - l.out), sizeof(status));
    *done = false;
    bool zero = ctx_->pretend_zero();
    for (uint32_t w : status) zero = zero || (w & kTailZero);
    if (zero) return kOk;
    const int failed = tail_failure(status, d_ - (uint32_t)round_);
    if (failed) return fail(kEInvariant, failed == 1 ? "vector folding invariant failed" : "round folding invariant failed");
    const uint8_t *p = out, *end = out + (l.opening - l.out);
    for (uint64_t j = round_; j < d_; ++j) {
        RoundRecord rec;
        if (!decode_record(p, end, rec)) return fail(kEInvariant, "record of a round on the device");
        rec.round = j;
        records_.push_back(std::move(rec));
    }
    uint32_t w[4];
    std::memcpy(w, end, 16);
    opening_ = fq{{w[0], w[1], w[2], w[3]}};
    N_ = n_ = 1;
    round_ = d_;
    have_opening_ = true;
    stage_ = Stage::Done;
    *done = true;
    return kOk;
}

int ProofState::complete_chain() {
    const ChainLayout l = chain_layout();
    const uint32_t* flags = reinterpret_cast<const uint32_t*>(pinned_ + (l.flags - l.proof));
    const uint32_t tail = kTailLog;
    static_assert(kMinDepth >= (int)kTailLog, "every proof ends with the last rounds");
    const uint32_t* status = flags + 2 * d_ + 2;
    if (flags[2 * d_] || ctx_->pretend_zero()) return kChainRepeat;
    for (int k = 0; k < kRank; ++k)
        if (status[k] & kTailZero) return kChainRepeat;
    for (uint32_t j = 0; j < d_ - tail; ++j) {
        if (flags[2 * j]) return fail(kEInvariant, "vector folding invariant failed");     // prover.rs:204-207
        if (flags[2 * j + 1]) return fail(kEInvariant, "round folding invariant failed");  // prover.rs:288-291
    }
    const int failed = tail_failure(status, tail);
    if (failed) return fail(kEInvariant, failed == 1 ? "vector folding invariant failed" : "round folding invariant failed");
    // what the device did not write there: the statement's file id, length, depth and
    // seed, the record count and the rounds (the limbs are little-endian words as encoded)
    auto put = [&](size_t at, uint64_t v) {
        for (int i = 0; i < 8; ++i) pinned_[at + i] = (uint8_t)(v >> (8 * i));
    };
    std::memcpy(pinned_, pinned_ + (l.id - l.proof), 32);
    put(32, st_.original_len_bytes);
    put(40, st_.d);
    std::memcpy(pinned_ + 48 + module_encoded_size(S_), st_.g_0_seed, 32);
    put(statement_encoded_size(S_), d_);
    for (uint32_t j = 0; j < d_; ++j) put(record_at(j), j);
    return kOk;
}

int ProofState::complete_stage() {
    const size_t slot = (size_t)kRank * S_;
    const uint8_t* tail = pinned_ + 3 * slot * 16;
    uint32_t fl[2];
    std::memcpy(fl, tail + 32, 8);
    if (stage_ == Stage::Init) {
        std::memcpy(st_.file_id, tail, 32);
        tr_ = Transcript(epoch_copy_, st_.file_id);
        unpack_module(pinned_, S_, st_.com_0);
        current_ = st_.com_0;
        if (S_ >= 2) {
            unpack_module(pinned_ + slot * 16, S_, pend_l_);
            unpack_module(pinned_ + 2 * slot * 16, S_, pend_r_);
        }
        if (tail_planned_) {
            bool done;
            const int rc = complete_tail(&done);
            if (rc != kOk || done) return rc;
        }
        x_ = tr_.challenge_vec(0, current_, pend_l_, pend_r_);  // prover.rs:177-180
        xi_ = fq_inv(x_);
        stage_ = Stage::Vec;
        return kOk;
    }
    const uint32_t L = d_ - (uint32_t)round_, s = 1u << L, h = s / 2;
    if (stage_ == Stage::Vec) {
        if (round_ == 0 && cached_.entry) {
            // round 0's vector stage was the last reader of the cached family
            ctx_->prover_cache()->release(cached_);
            cached_ = ProverGenCache::Ref{};
        }
        if (fl[0]) return fail(kEInvariant, "vector folding invariant failed");  // prover.rs:204-207
        unpack_module(pinned_, s, ct_);
        unpack_module(pinned_ + slot * 16, h, lp_);
        unpack_module(pinned_ + 2 * slot * 16, h, rp_);
        y_ = tr_.challenge_poly(round_, ct_, lp_, rp_);  // prover.rs:253-259
        yi_ = fq_inv(y_);
        stage_ = Stage::Poly;
        return kOk;
    }
    if (stage_ == Stage::Poly) {
        if (fl[1]) return fail(kEInvariant, "round folding invariant failed");  // prover.rs:288-291
        RoundRecord rec;
        rec.round = round_;
        rec.l_vec = std::move(pend_l_);
        rec.r_vec = std::move(pend_r_);
        rec.l_poly = std::move(lp_);
        rec.r_poly = std::move(rp_);
        records_.push_back(std::move(rec));
        unpack_module(pinned_, h, current_);
        if (h >= 2) {
            unpack_module(pinned_ + slot * 16, h, pend_l_);
            unpack_module(pinned_ + 2 * slot * 16, h, pend_r_);
        } else {
            pend_l_ = Module::zero(h);
            pend_r_ = Module::zero(h);
        }
        N_ = n_ = h;
        round_ += 1;
        if (round_ == d_) {
            const uint4* m = reinterpret_cast<const uint4*>(tail + 48);
            opening_ = fq{{m->x, m->y, m->z, m->w}};
            have_opening_ = true;
            stage_ = Stage::Done;
            return kOk;
        }
        if (tail_planned_) {
            bool done;
            const int rc = complete_tail(&done);
            if (rc != kOk || done) return rc;
        }
        x_ = tr_.challenge_vec(round_, current_, pend_l_, pend_r_);
        xi_ = fq_inv(x_);
        stage_ = Stage::Vec;
        return kOk;
    }
    return fail(kEState, "no stage to complete");
}

void ProofState::encode_proof(std::vector<uint8_t>* out) const {
    out->clear();
    out->reserve(proof_encoded_size(d_));
    encode_statement(*out, st_);
    put_u64(*out, records_.size());
    for (const auto& r : records_) encode_record(*out, r);
    const size_t base = out->size();
    out->resize(base + 16);
    fq_to_bytes(opening_, out->data() + base);
}

// ============================================================== GpuProver

GpuProver::~GpuProver() {
    if (s_) cudaStreamSynchronize(s_);
    ps_.release();  // stream-ordered frees on s_, before the stream goes away
    if (s_) {
        cudaStreamSynchronize(s_);
        cudaStreamDestroy(s_);
    }
    if (ev_start_) cudaEventDestroy(ev_start_);
    if (ev_end_) cudaEventDestroy(ev_end_);
}

int GpuProver::fail(int code, const std::string& msg) {
    failed_ = true;
    ctx_->set_error(msg);
    return code;
}

int GpuProver::init(const uint8_t* file, uint64_t len, bool on_device, const uint8_t seed[32], const uint8_t epoch[32],
                    uint64_t max_preprocess_bytes) {
    cudaError_t e = cudaSetDevice(ctx_->device());
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s_, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&ev_start_);
    if (e == cudaSuccess) e = cudaEventCreate(&ev_end_);
    if (e != cudaSuccess) return fail(kECuda, std::string("stream/event setup: ") + cudaGetErrorString(e));
    cudaEventRecord(ev_start_, s_);
    if (ask_chain_) ps_.ask_chain();
    int rc = ps_.setup(file, len, on_device, seed, epoch, max_preprocess_bytes, s_);
    if (rc != kOk) return fail(rc, ps_.error());
    if (ask_chain_) return kOk;  // run_chain() does every stage
    return run_stage();  // Init: commitment and round 0's vector cross terms
}

int GpuProver::run_stage() {
    NvtxRange range(stage_name((int)ps_.stage()));
    Plan plan;
    ps_.plan_stage(plan);
    std::string err;
    const int n = plan.launch(ctx_, s_, &err);
    if (n < 0) return fail(kECuda, err);
    const bool last = ps_.stage() == Stage::Poly && ps_.round() + 1 == ps_.depth();
    if (last) cudaEventRecord(ev_end_, s_);
    cudaError_t e = cudaStreamSynchronize(s_);
    if (e != cudaSuccess) return fail(kECuda, std::string("stage: ") + cudaGetErrorString(e));
    int rc;
    {
        NvtxRange fs("fiat-shamir");
        rc = ps_.complete_stage();
    }
    if (rc != kOk) return fail(rc, ps_.error());
    return kOk;
}

int GpuProver::fold_round(uint64_t j, RoundRecord* out, double times_ms[3]) {
    if (failed_) return fail(kEState, "prover is in a failed state");
    if (j != ps_.round()) return fail(kEState, "round index mismatch");
    if (ps_.stage() != Stage::Vec) return fail(kEState, "all rounds have finished");
    using Clk = std::chrono::steady_clock;
    const Clk::time_point t0 = Clk::now();
    int rc = run_stage();  // vector stage
    if (rc != kOk) return rc;
    const Clk::time_point t1 = Clk::now();
    rc = run_stage();  // poly stage
    if (rc != kOk) return rc;
    const Clk::time_point t2 = Clk::now();
    if (out) *out = ps_.records().back();
    if (times_ms) {
        times_ms[0] = std::chrono::duration<double, std::milli>(t1 - t0).count();
        times_ms[1] = std::chrono::duration<double, std::milli>(t2 - t1).count();
        times_ms[2] = std::chrono::duration<double, std::milli>(t2 - t0).count();
    }
    return kOk;
}

double GpuProver::device_ms() const {
    float ms = 0.f;
    if (!ev_start_ || !ev_end_ || cudaEventElapsedTime(&ms, ev_start_, ev_end_) != cudaSuccess) return -1.0;
    return ms;
}

int GpuProver::run_chain() {
    NvtxRange range("chain");
    std::string err;
    while (ps_.stage() != Stage::Done) {
        Plan plan;
        ps_.plan_stage(plan);
        if (plan.launch(ctx_, s_, &err) < 0) return fail(kECuda, err);
        const int rc = ps_.chain_next(s_);
        if (rc != kOk) return fail(rc, ps_.error());
    }
    cudaEventRecord(ev_end_, s_);
    const cudaError_t e = cudaStreamSynchronize(s_);
    if (e != cudaSuccess) return fail(kECuda, std::string("proof: ") + cudaGetErrorString(e));
    const int rc = ps_.complete_chain();
    if (rc == ProofState::kChainRepeat) return rc;
    return rc == kOk ? kOk : fail(rc, ps_.error());
}

// The proof into `out` when it holds `cap` bytes or fewer; *need is its size.
static int deliver(Context* ctx, const uint8_t* proof, size_t size, uint8_t* out, size_t cap, size_t* need) {
    if (need) *need = size;
    if (!out || cap < size) {
        ctx->set_error("proof buffer too small");
        return kESize;
    }
    std::memcpy(out, proof, size);
    return kOk;
}

int prove_all(Context* ctx, const uint8_t* file, uint64_t len, bool on_device, const uint8_t seed[32],
              const uint8_t epoch[32], uint8_t* out, size_t cap, size_t* need, double* device_ms) {
    {
        GpuProver p(ctx);
        p.ask_chain();
        int rc = p.init(file, len, on_device, seed, epoch, ctx->max_preprocess());
        if (rc == kOk) rc = p.run_chain();
        if (rc == kOk) {
            if (device_ms) *device_ms = p.device_ms();
            return deliver(ctx, p.chain_proof(), proof_encoded_size(p.rounds_total()), out, cap, need);
        }
        if (rc != ProofState::kChainRepeat) return rc;
    }
    // a challenge candidate was zero: stage by stage with challenges on the host
    GpuProver p(ctx);
    int rc = p.init(file, len, on_device, seed, epoch, ctx->max_preprocess());
    if (rc != kOk) return rc;
    for (uint32_t r = 0; r < p.rounds_total(); ++r) {
        rc = p.fold_round(r, nullptr);
        if (rc != kOk) return rc;
    }
    fq o;
    if (!p.final_opening(&o)) {
        ctx->set_error("final opening unavailable");
        return kEState;
    }
    std::vector<uint8_t> proof;
    p.encode_proof(&proof);
    if (device_ms) *device_ms = p.device_ms();
    return deliver(ctx, proof.data(), proof.size(), out, cap, need);
}

}  // namespace dm

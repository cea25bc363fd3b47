// One proof as a sequence of GPU stages separated by host Fiat-Shamir steps.
//
//   Init : file id, witness unpack, generator expansion, transforms of m and g,
//          commitment com_0 and round 0's vector cross terms
//   Vec  : fold m, g with x; transforms; recompute check + even/odd cross terms
//   Poly : fold m, g with y; transforms; recompute check + next vector cross terms
//
// Each stage emits jobs into a Plan; a Plan launches every job kind once (per
// ring size), so a single request and a batch of same-stage requests run through
// the same kernels.  After a stage's device->host copies land, complete_stage()
// runs the host part (checks, transcript, records) and arms the next stage.
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "dm_jobs.cuh"
#include "engine.h"

namespace dm {

struct Copy {
    void* dst;
    const void* src;
    size_t bytes;
};

class Plan {
   public:
    std::vector<HashJob> hash;
    std::vector<UnpackJob> unpack;
    std::vector<GenJob> gen;
    std::vector<FoldJob> fold;
    std::vector<NttJob> ntt[kLogMaxProverRing + 1];
    // multiply-accumulates of every ring size (each job carries its own)
    std::vector<MacJobX> mac, split, triple;
    std::vector<FinishJobX> finish[kLogMaxProverRing + 1];
    std::vector<TailJob> tail;  // last rounds of proofs whose products finish in this plan
    std::vector<Copy> d2h;
    // Cached generator families: events the stream waits on before the first
    // launch (entries other stages filled) and events recorded after the last
    // (entries this plan fills), with the fills' references for poisoning when
    // the plan fails to launch.
    std::vector<cudaEvent_t> wait_events, record_events;
    std::vector<ProverGenCache::Ref> fills;
    // Launches every non-empty job kind in dependency order on `st`, then the copies.
    // Returns the number of kernel launches, or a negative status.
    int launch(Context* ctx, cudaStream_t st, std::string* err);
    void clear();

   private:
    int launch_all(Context* ctx, cudaStream_t st, std::string* err);

   public:
    bool empty() const;
};

enum class Stage { Init, Vec, Poly, Done, Failed };

class ProofState {
   public:
    explicit ProofState(Context* ctx) : ctx_(ctx) {}
    ~ProofState();
    ProofState(const ProofState&) = delete;
    ProofState& operator=(const ProofState&) = delete;

    // Validates the input, allocates device state on `stream` and stages the file.
    int setup(const uint8_t* file, uint64_t len, bool on_device, const uint8_t seed[32], const uint8_t epoch[32],
              uint64_t max_preprocess_bytes, cudaStream_t stream);
    // With it, the stage whose commitments are of ring 2^kTailLog also plans the rounds
    // from there (k_tail.cu), and its complete_stage() ends the proof.
    void allow_tail(bool on) { allow_tail_ = on; }
    void plan_stage(Plan& plan);  // jobs + copies of the current stage
    int complete_stage();         // host part once the stage's copies landed

    // The whole proof as one chain of launches: challenges are computed on the
    // device (k_transcript.cu), folds read them there, and the finishes write the
    // commitments into the proof's encoding, which is copied to the host once at the
    // end.  Asked for before setup().
    void ask_chain() { chained_ = true; }
    // After a stage's plan is launched: the stage's challenge, then the next stage.
    int chain_next(cudaStream_t stream);
    // After the stream has passed everything: the checks in stage order.  kChainRepeat:
    // a challenge candidate was zero, which the host path's counter resolves.
    static constexpr int kChainRepeat = 1;
    int complete_chain();
    // The proof's bytes (chained: valid until release()).
    const uint8_t* chain_proof() const { return pinned_; }

    Stage stage() const { return stage_; }
    uint32_t stage_L() const;  // ring size exponent of the stage's transforms (batching key)
    uint32_t depth() const { return d_; }
    uint64_t round() const { return round_; }
    uint32_t vector_len() const { return N_; }
    uint32_t ring_len() const { return n_; }
    uint64_t file_len() const { return len_; }
    const Statement& statement() const { return st_; }
    const Module& current_commitment() const { return current_; }
    std::vector<RoundRecord>& records() { return records_; }
    bool opening(fq* out) const;
    const std::string& error() const { return err_; }
    int error_code() const { return err_code_; }
    static uint64_t footprint(uint64_t len);
    void encode_proof(std::vector<uint8_t>* out) const;  // bincode((Statement, Vec<RoundRecord>, Fp))
    // Frees the device state (stream-ordered on the setup stream) and the pinned buffer.
    void release();

   private:
    int fail(int code, const std::string& msg);
    int chain_tail(cudaStream_t stream);
    // The launch of the rounds from the current one on: where their records, the two
    // folded commitments' images, the opening and the status go, and the file id's place.
    TailJob tail_job(uint8_t* records, uint8_t* c_image, uint8_t* ct_image, uint8_t* opening, uint8_t* status,
                     const uint8_t* file_id, const uint8_t* image, uint64_t round) const;
    int complete_tail(bool* done);
    static int tail_failure(const uint32_t status[kRank], uint32_t rounds);  // 0, 1 (vector) or 2 (round check)
    bool plan_commit(Plan& P, uint32_t L, uint32_t cols, uint32_t c, const uint4* m_src, const uint4* g_src,
                     uint32_t* part, uint32_t* ghat = nullptr, bool g_transformed = false);
    const uint4* g_round0() const;  // the family round 0's vector fold reads
    Context* ctx_;
    cudaStream_t alloc_stream_ = nullptr;
    Stage stage_ = Stage::Init;
    uint32_t d_ = 0, S_ = 0, N_ = 0, n_ = 0;
    uint64_t round_ = 0, len_ = 0;
    Statement st_{};
    Transcript tr_;
    Module current_, pend_l_, pend_r_, ct_, lp_, rp_;
    fq x_{}, xi_{}, y_{}, yi_{};
    fq opening_{};
    bool have_opening_ = false;
    std::vector<RoundRecord> records_;
    std::string err_;
    int err_code_ = 0;
    const uint8_t* d_file_ = nullptr;
    DevMem mem_;
    Span file_, hash_scratch_, m_a_, m_b_, g_a_, g_b_, mhat_, ghat_, partials_, comm_;  // in mem_
    uint8_t* pinned_ = nullptr;
    size_t pinned_bytes_ = 0;
    // The chain's device state, which takes no memory of its own, so a caller that fits
    // beside a prover's footprint still does: hash scratch, challenges, the encodings of
    // the two folded commitments and the proof's end where ghat_ does, whose second half
    // is free once the first stage's products are there; the file id, check flags and
    // status, which are written or cleared before, follow in comm_'s first half slot.
    // Proof and flags are neighbours and go to the host in one copy.
    bool chained_ = false;
    Span chain_;  // in mem_
    struct ChainLayout {
        size_t cvs, challenges, c, ct, proof, id, flags, end;
        size_t copied() const { return end - proof; }
    };
    ChainLayout chain_layout() const;
    size_t record_at(uint64_t round) const;  // offset of a round's record in the proof
    bool allow_tail_ = false, tail_planned_ = false;
    struct TailLayout {  // in ghat_, free once the products are there; the outputs together
        size_t image, c, ct, out, opening, status, out_bytes;
    };
    static TailLayout tail_layout();
    uint32_t parts_ = 1;
    // Witness columns that can be nonzero: the file fills the coefficients in
    // order and the square layout pads with zeros, and folds keep zero columns
    // zero, so a stage's columns from min(mcols_, columns) on are zero.  Their
    // transforms and the generator columns that only meet them are skipped.
    uint32_t mcols_ = 0;
    uint8_t seed_[32];
    uint8_t epoch_copy_[32];
    // g_0 and its transform from the context's cache, held from the Init stage
    // until round 0's vector stage (the last reader) has completed
    ProverGenCache::Ref cached_{};
};

// Round-by-round prover (src/protocol/prover.rs:56-313): one ProofState driven
// stage by stage on its own stream.
class GpuProver {
   public:
    explicit GpuProver(Context* ctx) : ctx_(ctx), ps_(ctx) {}
    ~GpuProver();
    // file is a host pointer, or a device pointer when on_device.
    int init(const uint8_t* file, uint64_t len, bool on_device, const uint8_t seed_generators[32],
             const uint8_t epoch_seed[32], uint64_t max_preprocess_bytes);
    // times_ms (optional): wall time of the vector stage, the polynomial stage
    // and the whole round, as RoundOutput's vector_fold_time / poly_fold_time /
    // total_round_time (src/protocol/prover.rs:26-31)
    int fold_round(uint64_t round_idx, RoundRecord* out, double times_ms[3] = nullptr);
    bool final_opening(fq* out) const { return ps_.opening(out); }
    const Statement& statement() const { return ps_.statement(); }
    uint32_t rounds_total() const { return ps_.depth(); }
    uint64_t current_round() const { return ps_.round(); }
    const Module& current_commitment() const { return ps_.current_commitment(); }
    uint32_t vector_len() const { return ps_.vector_len(); }
    uint32_t ring_len() const { return ps_.ring_len(); }
    static uint64_t footprint(uint64_t len) { return ProofState::footprint(len); }
    double device_ms() const;  // first to last operation of the proof (CUDA events)
    void encode_proof(std::vector<uint8_t>* out) const { ps_.encode_proof(out); }
    // The whole proof without a host round trip (ProofState::ask_chain): init() then
    // only sets up.
    void ask_chain() { ask_chain_ = true; }
    int run_chain();
    const uint8_t* chain_proof() const { return ps_.chain_proof(); }

   private:
    bool ask_chain_ = false;
    int run_stage();
    int fail(int code, const std::string& msg);
    Context* ctx_;
    ProofState ps_;
    cudaStream_t s_ = nullptr;
    cudaEvent_t ev_start_ = nullptr, ev_end_ = nullptr;
    bool failed_ = false;
};

}  // namespace dm

// A ring product as the kernels run it from 2^5 on, on the CPU: forward transforms with
// the padded exchanges between their passes, rows stored in the order a warp writes them,
// slotwise products, the inverse transform with its exchanges in reverse and the CRT.
// A factor with few terms, so that the schoolbook product is cheap up to 2^13.
// Exit status 0 = all checks pass.
#include <cstdio>
#include <random>
#include <vector>

#include "dm_ntt.cuh"
#include "dm_tables.h"

using namespace dm;

namespace {

std::mt19937_64 rng(20261205);
int fails = 0;

fq random_fq() {
    fq x;
    for (int i = 0; i < 4; ++i) x.w[i] = (uint32_t)rng();
    x.w[3] &= 0xFFFFu;
    return fq_canon(x);
}

// A block's row: its threads' registers, and shared memory it exchanges them through.
struct Row {
    int L;
    uint32_t base;  // the third row of a block
    std::vector<uint32_t> a, sm;
    explicit Row(int l) : L(l), base(2u << l), a(1u << l), sm(ntt_pad_words(4u << l), 0xFFFFFFFFu) {}
    uint32_t threads() const { return 1u << (L - 4); }
    uint32_t* regs(uint32_t t) { return a.data() + 16 * t; }
    void exchange(int e, int from, int to) {
        for (uint32_t t = 0; t < threads(); ++t)
            for (int r = 0; r < kNttE; ++r) {
                const uint32_t w = ntt_pad_base(base, L, e, from, t) + ntt_pad_reg(L, e, from, r);
                if (w < sm.size()) sm[w] = regs(t)[r];
                else ++fails;
            }
        for (uint32_t t = 0; t < threads(); ++t)
            for (int r = 0; r < kNttE; ++r) {
                const uint32_t w = ntt_pad_base(base, L, e, to, t) + ntt_pad_reg(L, e, to, r);
                regs(t)[r] = w < sm.size() ? sm[w] : 0u;
            }
    }
};

const Tw* last_table(const std::vector<Tw>& t, int pi, int L) {
    return t.data() + (size_t)pi * kLastSpan + (1u << L) - 16u;
}

std::vector<uint32_t> forward(const std::vector<fq>& x, int L, int pi) {
    const HostTables& T = host_tables();
    const uint32_t p = T.pc.p[pi];
    Row row(L);
    for (uint32_t t = 0; t < row.threads(); ++t)
        for (int r = 0; r < kNttE; ++r) row.regs(t)[r] = residue_fwd(x[ntt_place(L, 0, t, r)], T.pc, pi);
    for (int pass = 0; pass < ntt_pass_count(L); ++pass) {
        for (uint32_t t = 0; t < row.threads(); ++t)
            ntt_fwd_pass(row.regs(t), L, pass, t, T.fwd.data() + (size_t)pi * kMaxRing, last_table(T.fwd_last, pi, L), p);
        if (pass + 1 < ntt_pass_count(L)) row.exchange(pass, pass, pass + 1);
    }
    std::vector<uint32_t> out(1u << L);
    for (uint32_t slot = 0; slot < out.size(); ++slot) {
        const uint32_t v = shoup_one(row.a[slot], T.pc.one_s[pi], p);  // thread t holds slots 16 t ..
        if (v >= 2 * p) ++fails;
        out[ntt_slot_pos(L, slot)] = v;
    }
    return out;
}

std::vector<uint32_t> inverse(const std::vector<uint32_t>& y, int L, int pi) {
    const HostTables& T = host_tables();
    const uint32_t p = T.pc.p[pi];
    Row row(L);
    for (uint32_t slot = 0; slot < y.size(); ++slot)
        row.a[slot] = shoup_one(y[ntt_slot_pos(L, slot)], T.pc.one_s[pi], p);
    for (int pass = ntt_pass_count(L) - 1; pass >= 0; --pass) {
        for (uint32_t t = 0; t < row.threads(); ++t)
            ntt_inv_pass(row.regs(t), L, pass, t, T.inv.data() + (size_t)pi * kMaxRing, last_table(T.inv_last, pi, L), p);
        if (pass > 0) row.exchange(pass - 1, pass, pass - 1);
    }
    std::vector<uint32_t> out(y.size());
    for (uint32_t t = 0; t < row.threads(); ++t)
        for (int r = 0; r < kNttE; ++r)
            out[ntt_place(L, 0, t, r)] = red_below(shoup_mul(row.regs(t)[r], T.fin[pi][L], T.fins[pi][L], p), p);
    return out;
}

}  // namespace

int main() {
    const HostTables& T = host_tables();
    for (int L = 5; L <= 13; ++L) {
        const uint32_t s = 1u << L;
        std::vector<fq> a(s), b(s, fq_zero()), want(s, fq_zero());
        for (fq& v : a) v = random_fq();
        for (int k = 0; k < 5; ++k) b[k == 0 ? 0 : k == 1 ? s - 1 : rng() % s] = random_fq();
        for (uint32_t j = 0; j < s; ++j) {
            if (fq_is_zero(b[j])) continue;
            for (uint32_t i = 0; i < s; ++i) {
                const fq t = fq_mul(a[i], b[j]);
                fq& w = want[(i + j) % s];
                w = i + j < s ? fq_add(w, t) : fq_sub(w, t);
            }
        }
        std::vector<std::vector<uint32_t>> y(kPrimes);
        for (int pi = 0; pi < kPrimes; ++pi) {
            const std::vector<uint32_t> fa = forward(a, L, pi), fb = forward(b, L, pi);
            std::vector<uint32_t> prod(s);
            for (uint32_t i = 0; i < s; ++i) prod[i] = red64_lazy((uint64_t)fa[i] * fb[i], T.pc, pi);
            y[pi] = inverse(prod, L, pi);
        }
        for (uint32_t j = 0; j < s; ++j) {
            uint32_t z[kPrimes];
            for (int pi = 0; pi < kPrimes; ++pi) z[pi] = y[pi][j];
            if (!fq_eq(crt_from_scaled(z, T.cc), want[j]) && fails++ < 10) std::printf("FAIL L=%d j=%u\n", L, j);
        }
    }
    std::printf("%s\n", fails ? "FAILED" : "ok");
    return fails ? 1 : 0;
}

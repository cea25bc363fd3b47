// The transforms' padded exchanges and stored slot order (dm_ntt.cuh compiled for
// the CPU) at every ring size and block shape.  Exit status 0 = all checks pass.
#include <cstdio>
#include <vector>

#include "dm_ntt.cuh"

using namespace dm;

int main() {
    int fails = 0;
    auto check = [&](bool ok, const char* what, int L) {
        if (!ok && fails++ < 10) std::printf("FAIL %s (L=%d)\n", what, L);
    };
    for (int L = 5; L <= 13; ++L)
        for (uint32_t group : {32u, 64u, 288u, 576u}) {
            const uint32_t T = 1u << (L - 4), rows = T >= group ? 1 : group / T, n = rows << L;
            for (int e = 0; e + 1 < ntt_pass_count(L); ++e)
                for (int pass = e; pass <= e + 1; ++pass) {
                    std::vector<int> used(ntt_pad_words(n), 0);
                    for (uint32_t th = 0; th < rows * T; ++th)
                        for (int r = 0; r < kNttE; ++r) {
                            const uint32_t base = (th / T) << L, t = th % T;
                            const uint32_t w = ntt_pad_base(base, L, e, pass, t) + ntt_pad_reg(L, e, pass, r);
                            check(w == ntt_pad(ntt_last_exchange(L, e), base + ntt_place(L, pass, t, r)), "word", L);
                            check(w >= ntt_pad(false, base) && w < ntt_pad(false, base + (1u << L)), "row range", L);
                            check(w < used.size() && !used[w]++, "distinct words", L);
                        }
                    for (uint32_t w0 = 0; w0 + 32 <= rows * T; w0 += 32)
                        for (int r = 0; r < kNttE; ++r) {
                            uint32_t banks = 0;
                            for (uint32_t th = w0; th < w0 + 32; ++th)
                                banks |= 1u << ((ntt_pad_base((th / T) << L, L, e, pass, th % T) +
                                                 ntt_pad_reg(L, e, pass, r)) % 32);
                            check(banks == 0xFFFFFFFFu, "bank conflict", L);
                        }
                }
        }
    for (int L = 0; L <= 13; ++L) {
        const uint32_t s = 1u << L;
        std::vector<int> used(s, 0);
        for (uint32_t i = 0; i < s; ++i) {
            const uint32_t pos = ntt_slot_pos(L, i);
            check(pos < s && !used[pos]++, "slot order", L);
            if (L >= 1 && !(i & 1)) {
                check(pos % 2 == 0 && ntt_slot_pos(L, i + 1) == pos + 1, "slot pair", L);
                check(ntt_pair_at(L, pos / 2) == i / 2, "pair at", L);
            }
            if (L >= 4) {  // word q of thread t at q T + t
                const uint32_t T = s / 16, t = i / 16, r = i % 16;
                check(pos == 4 * ((r / 4) * T + t) + r % 4, "thread order", L);
            }
        }
    }
    std::printf("%s\n", fails ? "FAILED" : "ok");
    return fails ? 1 : 0;
}

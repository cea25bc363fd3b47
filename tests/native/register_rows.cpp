// Whole-row transforms (ntt_fwd_small, ntt_inv_small) of rings 2^0 .. 2^5 under every
// prime, at the ends of the inputs' range and in between, against the evaluations
// themselves: slot i of ring 2h's pair (2i, 2i + 1) is taken at +w and -w, w the
// twiddle h + i, and of ring h at w^2.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "dm_ntt.cuh"
#include "dm_tables.h"

using namespace dm;
using u64 = unsigned long long;

template <int L>
static bool check(const HostTables& H, int i, const std::vector<uint32_t>& in) {
    constexpr int n = 1 << L;
    const uint32_t p = H.pc.p[i];
    const Tw* fwd = &H.fwd[(size_t)i * kMaxRing];
    uint32_t a[n];
    for (int j = 0; j < n; ++j) a[j] = in[j];
    ntt_fwd_small<L>(a, fwd, p);
    for (int s = 0; s < n; ++s) {
        const u64 w = fwd[n + s].w, at = w * w % p;
        u64 want = 0;
        for (int j = n - 1; j >= 0; --j) want = (want * at + in[j]) % p;
        const uint32_t got = ntt_fwd_final(a[s], H.pc.one_s[i], p);
        if (got != want) return std::printf("prime %d ring 2^%d slot %d\n", i, L, s), false;
        a[s] = got;
    }
    ntt_inv_small<L>(a, &H.inv[(size_t)i * kMaxRing], p);
    for (int j = 0; j < n; ++j)
        if (red_below(shoup_mul(a[j], H.ninv[i][L], H.ninvs[i][L], p), p) != in[j] % p)
            return std::printf("prime %d ring 2^%d coefficient %d\n", i, L, j), false;
    return true;
}

int main() {
    const HostTables& H = host_tables();
    std::srand(3);
    for (int i = 0; i < kPrimes; ++i) {
        const uint32_t top = 8 * H.pc.p[i] - 1;
        for (int trial = 0; trial < 40; ++trial) {
            std::vector<uint32_t> in(32);
            for (auto& x : in)
                x = trial == 0 ? top : trial == 1 ? 0u : (trial & 1) ? top - (uint32_t)(std::rand() & 1) * top
                                                                     : (uint32_t)(((u64)std::rand() << 16 ^ std::rand()) % ((u64)top + 1));
            if (!check<0>(H, i, in) || !check<1>(H, i, in) || !check<2>(H, i, in) || !check<3>(H, i, in) ||
                !check<4>(H, i, in) || !check<5>(H, i, in))
                return 1;
        }
    }
    return 0;
}

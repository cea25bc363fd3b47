// Reads elements (hex), writes fq_inv_gcd and whether it equals Fermat's inverse.
#include <cstdio>
#include <cstring>

#include "dm_field.cuh"

using namespace dm;

int main() {
    char line[64];
    while (std::scanf("%60s", line) == 1) {
        fq a = fq_zero();
        for (int i = 0; line[i]; ++i) {
            for (int w = 3; w > 0; --w) a.w[w] = a.w[w] << 4 | a.w[w - 1] >> 28;
            a.w[0] = a.w[0] << 4 | (uint32_t)(line[i] <= '9' ? line[i] - '0' : line[i] - 'a' + 10);
        }
        const fq g = fq_inv_gcd(a), f = fq_inv(a);
        std::printf("%08x%08x%08x%08x %d\n", g.w[3], g.w[2], g.w[1], g.w[0], (int)fq_eq(g, f));
    }
}

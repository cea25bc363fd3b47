// Reads lines of nine residues, writes the element of Z_q that the kernels' CRT
// recombines from them (dm_field.cuh compiled for the CPU); "primes" first.
#include <cstdio>

#include "dm_tables.h"

using namespace dm;

int main() {
    const HostTables& T = host_tables();
    for (int i = 0; i < kPrimes; ++i) std::printf("%u%c", T.primes[i], i + 1 < kPrimes ? ' ' : '\n');
    uint32_t r[kPrimes];
    for (;;) {
        for (int i = 0; i < kPrimes; ++i)
            if (std::scanf("%u", &r[i]) != 1) return 0;
        const fq x = crt_to_fq(r, T.pc, T.cc);
        std::printf("%08x%08x%08x%08x\n", x.w[3], x.w[2], x.w[1], x.w[0]);
    }
}

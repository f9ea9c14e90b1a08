// Host-side sweep of the quotient by a matrix's norm (gefen_b200/csrc/quant_core.h), compiled by g++ for the CPU test-suite:
// for every pair of bf16 values with |v| up to a little above the norm, both signs, subnormals, infinities and NaN included,
// it must be the IEEE quotient bit for bit (NaN as NaN).
//
//   norm_divider_sweep -> prints "mismatches checked reciprocal"
#include <cstdio>
#include <cstring>
#include "../../gefen_b200/csrc/quant_core.h"

using namespace gefen;

static float from_bf16(uint32_t h) {
    const uint32_t u = h << 16;
    float f;
    memcpy(&f, &u, 4);
    return f;
}

int main() {
    unsigned long long bad = 0, checked = 0, reciprocal = 0;
#pragma omp parallel for reduction(+ : bad, checked, reciprocal) schedule(dynamic, 64)
    for (int n = 0; n <= 0x7F80; ++n) {
        const float norm = from_bf16(n);
        const NormDivider quotient(norm);
        const int most = n + 2 <= 0x7F80 ? n + 2 : 0x7F80;
        for (int v = 0; v <= most + 1; ++v) {
            const int h = v <= most ? v : 0x7FC0;   // (and a NaN)
            const float a = from_bf16(h);
            const float got[2] = {quotient(a), quotient(-a)}, want[2] = {a / norm, -a / norm};
            for (int s = 0; s < 2; ++s) {
                uint32_t g, w;
                memcpy(&g, &got[s], 4);
                memcpy(&w, &want[s], 4);
                if (g != w && !(got[s] != got[s] && want[s] != want[s])) ++bad;
            }
            checked += 2;
            if (fabsf(a) > quotient.least) reciprocal += 2;
        }
    }
    printf("%llu %llu %llu\n", bad, checked, reciprocal);
    return 0;
}

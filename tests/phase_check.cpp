// Host check of sde_geom::tiny_phase against the DOUBLE arithmetic it stands in for:
// SNGL(TWOPI*(S*W - W)) with S = 1 + k 2^-53, |k| <= 10, over W of all magnitudes, powers of
// two and their neighbours, and W whose product with k ends on a tie.  Prints "cases decided
// mismatches".
#include <stdio.h>
#include <stdlib.h>

#include "geom.cuh"

int main(int argc, char **argv) {
    const long long n = argc > 1 ? atoll(argv[1]) : 1000000;
    const double twopi = (double)(8.0f * atanf(1.0f));
    unsigned long long z = 88172645463325252ull;
    long long decided = 0, bad = 0;
    for (long long i = 0; i < n; i++) {
        z ^= z << 13;
        z ^= z >> 7;
        z ^= z << 17;
        int k = (int)(z % 21) - 10;
        if (k > 0) k &= ~1;  // above 1 the spacing is 2^-52
        const double s = 1.0 + k * 0x1p-53;
        unsigned m = (unsigned)(z >> 20) & 0x7FFFFFu;
        switch ((z >> 50) & 3) {
            case 0: m = 0; break;
            case 1: m = (z >> 52) & 1 ? 1 : 0x7FFFFF; break;
            case 2: m &= 0x700000u; break;  // products that end on a tie
        }
        float w = ldexpf((float)(0x800000u | m), (int)((z >> 43) % 100) - 90);
        if ((z >> 63) & 1) w = -w;
        if ((i & 1023) == 0) w = 0.0f;
        float got;
        if (!sde_geom::tiny_phase(s, w, got)) continue;
        decided++;
        const volatile double wl = s * (double)w;
        const volatile double d = wl - (double)w;
        const float want = (float)(twopi * d);
        if (memcmp(&got, &want, 4) != 0 && bad++ < 10) fprintf(stderr, "k %d w %a: %a, not %a\n", k, w, got, want);
    }
    printf("%lld %lld %lld\n", n, decided, bad);
    return bad != 0;
}

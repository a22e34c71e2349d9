// Host check of sde_geom::tiny_phase at the limits of its arguments: where it decides, the phase
// is SNGL(TWOPI*(S*W - W)) in DOUBLE, NaN for an infinite W or a NaN.  Prints "decided mismatches".
#include <math.h>
#include <stdio.h>

#include "geom.cuh"

int main() {
    const double twopi = (double)(8.0f * atanf(1.0f));
    const float big = 3.4028235e38f, tiny = 1e-45f, ws[] = {0.0f, -0.0f, 1.0f, -3.5f, tiny, -tiny, big, -big,
                                                              INFINITY, -INFINITY, NAN};
    const double ss[] = {1.0, 1.0 + 0x1p-52, 1.0 - 0x1p-53, 1.0 + 0x1p-40, 0.5, -1.0, INFINITY, NAN};
    int decided = 0, bad = 0;
    for (double s : ss)
        for (float w : ws) {
            float got;
            if (!sde_geom::tiny_phase(s, w, got)) continue;
            decided++;
            const volatile double wl = s * (double)w;
            const volatile double d = wl - (double)w;
            const float want = (float)(twopi * d);
            if (!(got == want) && bad++ < 20) fprintf(stderr, "s %a w %a: %a, not %a\n", s, w, got, want);
        }
    printf("%d %d\n", decided, bad);
    return bad != 0;
}

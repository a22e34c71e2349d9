// Host check of sde_geom::geom_vis for coordinates far off the grid: whatever they are, a point that
// the degridding geometry calls valid has a cell whose window lies in the grid and offsets in the
// tap table, and one that the gridding geometry calls sane has a cell of fewer than 2^31.  Prints
// "points bad".
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <initializer_list>

#include "geom.cuh"

using namespace sde_geom;

int main() {
    const float vals[] = {0.0f, 1.0f, -40.0f, 1e5f, -1e8f, 1.07e9f, 2.1474836e9f, -2.1474836e9f, 2.1474830e9f, 2.2e9f, -4.3e9f,
                          8.6e9f, 1e20f, -1e30f, 3.4e38f, -3.4e38f, INFINITY, -INFINITY};
    const double diag[] = {1.0, 1.0 - 0x1p-53, 1.0 - 0x1p-30};
    long points = 0, bad = 0;
    for (double d : diag)
        for (double off : {0.0, 1e-4})
            for (float scale : {1.0f, -1.0f, 0.001f, 700.0f})
                for (float u : vals)
                    for (float v : vals)
                        for (float w : {0.0f, -1e6f}) {
                            GParams p;
                            memset(&p, 0, sizeof p);
                            p.uscale = scale;
                            p.vscale = fabsf(scale);
                            p.uorigin = 1;
                            p.vorigin = 128;
                            p.nu = 129;
                            p.nv = 256;
                            p.supp = 3;
                            p.osamp = 128;
                            for (int k = 0; k < 9; k++) p.s[k] = k % 4 == 0 ? d : off;
                            p.identity = d == 1.0 && off == 0.0;
                            p.diagonal = off == 0.0;
                            p.doshift = !p.identity;
                            p.fast = p.identity;
                            p.near_id = p.diagonal && fabs(d - 1.0) <= 0x1p-50;
                            p.ntu = 1;
                            p.twopi = (double)(8.0f * atanf(1.0f));
                            const GGeo g = geom_vis(p, u, v, w, 1.0f, 0.0f);
                            points++;
                            const long lim = 1l << 31, nu = g.dg.nud, nv = g.dg.nvd;
                            bool ok = !g.dg.valid || (nu + 3 <= p.nu && nv + 3 <= p.nv && nv - 3 >= 1 && nu > -lim / 2 &&
                                                      g.dg.dui >= -64 && g.dg.dui <= 64 && g.dg.dvi >= -64 && g.dg.dvi <= 64);
                            if (g.sane) ok = ok && labs((long)g.nuc) < lim - 8 && labs((long)g.nvc) < lim - 8;
                            if (!ok && bad++ < 10)
                                fprintf(stderr, "u %g v %g scale %g: valid cell %ld %ld offsets %d %d\n", u, v, scale, nu, nv,
                                        g.dg.dui, g.dg.dvi);
                        }
    printf("%ld %ld\n", points, bad);
    return bad != 0;
}

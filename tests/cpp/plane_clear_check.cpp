// Host check of the clearance that plane_gap gives a triangle pair (zdx_math.cuh): stdin holds pairs of triangles, 18
// doubles as hex bit patterns each, then 6 more numbers in [-1, 1] per corner pair's motion.  Every corner moves by
// less than the clearance allows; one line out: pairs, pairs with a clearance, and those with a segment after the
// move (0 expected).
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "zdx_math.cuh"

using namespace zdx;

int main() {
    long n = 0, held = 0, wrong = 0;
    for (;;) {
        double v[24];
        for (int i = 0; i < 24; ++i) {
            uint64_t u;
            if (std::scanf("%" SCNx64, &u) != 1) {
                std::printf("%ld %ld %ld\n", n, held, wrong);
                return 0;
            }
            std::memcpy(v + i, &u, 8);
        }
        ++n;
        V3 T[2][3], nn[2];
        std::memcpy(&T[0][0].x, v, 18 * 8);
        double d[2], scale = 0.0;
        for (int i = 0; i < 18; ++i) scale = smax(scale, fabs(v[i]));
        bool ok = true;
        for (int k = 0; k < 2; ++k) ok = plane_from_tri(T[k][0], T[k][1], T[k][2], nn[k], d[k]) && ok;
        if (!ok) continue;
        const double infl = smax(tri_inflation(T[0][0], T[0][1], T[0][2]), tri_inflation(T[1][0], T[1][1], T[1][2]));
        const double g0 = plane_gap(nn[1], d[1], T[0][0], T[0][1], T[0][2]), g1 = plane_gap(nn[0], d[0], T[1][0], T[1][1], T[1][2]);
        const double pad = 1e-9 * 3.0 * scale, clear = (g0 > g1 ? g0 : g1) - infl - 8.0 * pad;
        if (!(clear > 8.0 * pad)) continue;
        ++held;
        // rigid moves: each triangle by half of what is left, towards the other one and then as the numbers say
        const double half = 0.5 * (clear - 8.0 * pad) * (1.0 - 1e-8);
        for (int kind = 0; kind < 2; ++kind) {
            V3 M[2][3], mn[2];
            double md[2];
            V3 c = (T[1][0] + T[1][1] + T[1][2] - T[0][0] - T[0][1] - T[0][2]) * (1.0 / 3.0);
            if (kind == 1) c = g0 > g1 ? nn[1] * (dot(nn[1], T[0][0]) + d[1] > 0 ? -1.0 : 1.0) : nn[0] * (dot(nn[0], T[1][0]) + d[0] > 0 ? 1.0 : -1.0);
            c = c * (1.0 / norm(c));
            for (int k = 0; k < 2; ++k) {
                V3 s = c * (k == 0 ? half : -half);
                if (kind == 0) {
                    const V3 r{v[18 + 3 * k], v[19 + 3 * k], v[20 + 3 * k]};
                    s = (s * 0.5) + r * (0.5 * half / 1.7320508075688774);
                }
                for (int i = 0; i < 3; ++i) M[k][i] = T[k][i] + s;
                ok = plane_from_tri(M[k][0], M[k][1], M[k][2], mn[k], md[k]) && ok;
            }
            V3 o0, o1;
            if (ok && tri_tri(M[0], mn[0], md[0], M[1], mn[1], md[1], o0, o1)) ++wrong;
        }
    }
}

// Host check of the parts the triangle stage takes tri_tri apart into (zdx_math.cuh, zdx_npmath.cuh): stdin holds
// pairs of triangles, 18 doubles as hex bit patterns each; one line out: pairs, segments, pairs the planes rule
// out, and the pairs on which the parts and the whole differ or a plane rules out a segment (0 0 0 expected).
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "zdx_math.cuh"
#include "zdx_npmath.cuh"

using namespace zdx;

int main() {
    long n = 0, seg = 0, out = 0, differ = 0, differ_np = 0, wrong = 0;
    for (;;) {
        V3 T[2][3];
        double* v = &T[0][0].x;
        for (int i = 0; i < 18; ++i) {
            uint64_t u;
            if (std::scanf("%" SCNx64, &u) != 1) {
                std::printf("%ld %ld %ld %ld %ld %ld\n", n, seg, out, differ, differ_np, wrong);
                return 0;
            }
            std::memcpy(v + i, &u, 8);
        }
        ++n;
        V3 nn[2];
        double d[2];
        bool ok = true;
        for (int k = 0; k < 2; ++k) ok = plane_from_tri(T[k][0], T[k][1], T[k][2], nn[k], d[k]) && ok;
        if (!ok) continue;
        V3 a0{}, a1{}, b0{}, b1{};
        int ca[2] = {-1, -1}, cb[2] = {-1, -1};
        const bool whole = tri_tri_src(T[0], nn[0], d[0], T[1], nn[1], d[1], a0, a1, &ca[0], &ca[1]);
        V3 cut[6];
        unsigned valid = 0, valid_np = 0;
        double cut_np[6][3];
        for (int c = 0; c < 6; ++c) {
            const V3* E = T[c / 3];
            const V3* U = T[1 - c / 3];
            const V3 m = nn[1 - c / 3];
            if (tri_cut(E[c % 3], E[(c + 1) % 3], U[0], U[1], U[2], m, d[1 - c / 3], cut[c])) valid |= 1u << c;
            if (np::tri_cut(&E[c % 3].x, &E[(c + 1) % 3].x, &U[0].x, &m.x, d[1 - c / 3], cut_np[c])) valid_np |= 1u << c;
        }
        const bool parts = tri_join(nn[0], nn[1], valid, [&](int c) { return cut[c]; }, b0, b1, cb[0], cb[1]);
        if (whole != parts || (whole && (std::memcmp(&a0, &b0, 24) || std::memcmp(&a1, &b1, 24) || ca[0] != cb[0] || ca[1] != cb[1])))
            ++differ;
        double p[6], q[6];
        const bool whole_np = np::tri_tri(&T[0][0].x, &nn[0].x, d[0], &T[1][0].x, &nn[1].x, d[1], p, p + 3);
        const bool parts_np = np::tri_join(&nn[0].x, &nn[1].x, valid_np,
                                           [&](int c, double* o) { std::memcpy(o, cut_np[c], 24); }, q, q + 3);
        if (whole_np != parts_np || (whole_np && std::memcmp(p, q, 48))) ++differ_np;
        // the triangle stage's margin: inflation plus 8 pads of 1e-9 of the coordinate scale
        double scale = 0.0;
        for (int i = 0; i < 18; ++i) scale = smax(scale, fabs(v[i]));
        const double more = 8e-9 * scale;
        const bool ruled = beyond_plane(nn[1], d[1], T[0][0], T[0][1], T[0][2], tri_inflation(T[0][0], T[0][1], T[0][2]) + more) ||
                           beyond_plane(nn[0], d[0], T[1][0], T[1][1], T[1][2], tri_inflation(T[1][0], T[1][1], T[1][2]) + more);
        seg += whole;
        out += ruled;
        if (ruled && (whole || whole_np)) ++wrong;
    }
}

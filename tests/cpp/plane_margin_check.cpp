// Host check of the triangle stage's plane test (tri_inflation's reach, plane_off, reaches_hold, beyond_plane of zdx_math.cuh,
// put together as k_segments does): stdin holds pairs of triangles in the mesh frame, 18 doubles as hex bit patterns each,
// then a pose (position and quaternion, 7 more) that both are placed by.  One line out: pairs, pairs with a segment,
// pairs ruled out, and pairs ruled out that have one (0 expected).
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "zdx_math.cuh"
#include "zdx_npmath.cuh"

using namespace zdx;

int main() {
    long n = 0, seg = 0, out = 0, wrong = 0;
    for (;;) {
        double v[25];
        for (int i = 0; i < 25; ++i) {
            uint64_t u;
            if (std::scanf("%" SCNx64, &u) != 1) {
                std::printf("%ld %ld %ld %ld\n", n, seg, out, wrong);
                return 0;
            }
            std::memcpy(v + i, &u, 8);
        }
        ++n;
        V3 T[2][3], nn[2];
        std::memcpy(&T[0][0].x, v, 18 * 8);
        const V3 x{v[18], v[19], v[20]};
        const Q4 q = qnormalize(Q4{v[21], v[22], v[23], v[24]});
        double r[2], d[2], R[2] = {0.0, 0.0};
        bool ok = true;
        for (int k = 0; k < 2; ++k) {
            tri_inflation(T[k][0], T[k][1], T[k][2], &r[k]);
            r[k] = std::nextafterf((float)r[k], INFINITY);
            for (int i = 0; i < 3; ++i) {
                R[k] = smax(R[k], norm(T[k][i]));
                T[k][i] = qrotate_n(q, T[k][i]) + x;
            }
            ok = plane_from_tri(T[k][0], T[k][1], T[k][2], nn[k], d[k]) && ok;
        }
        if (!ok) continue;
        V3 o0, o1;
        double p[6];
        const bool hit = tri_tri(T[0], nn[0], d[0], T[1], nn[1], d[1], o0, o1) ||
                         np::tri_tri(&T[0][0].x, &nn[0].x, d[0], &T[1][0].x, &nn[1].x, d[1], p, p + 3);
        const double pad = 1e-9 * (2.0 * smax3(fabs(x.x), fabs(x.y), fabs(x.z)) + R[0] + R[1]);  // k_segments's
        const double more = plane_off(r[0], R[0]) + plane_off(r[1], R[1]) + 8.0 * pad;
        const bool ruled = (beyond_plane(nn[1], d[1], T[0][0], T[0][1], T[0][2], r[0] + more) ||
                            beyond_plane(nn[0], d[0], T[1][0], T[1][1], T[1][2], r[1] + more)) &&
                           reaches_hold(r[0], r[1], pad);
        seg += hit;
        out += ruled;
        wrong += ruled && hit;
    }
}

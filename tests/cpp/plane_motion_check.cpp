// Host check of the clearance that planes give a triangle pair (planes_clearance of zdx_math.cuh) under what the
// clearance cache lets bodies do: stdin holds rows of 40 doubles as hex bit patterns, the two triangles in their
// bodies' frames (18), two poses (position, quaternion: 14), then 4 for each body's motion (rotation axis, and the
// share of the motion that is rotation).  The bodies turn about their origins and shift so that |dx| + 2 R |dq|, summed
// over both, stays below the clearance as k_cache_skip measures it.  One line out: rows, those with a clearance, and
// motions after which tri_tri finds a segment (0 expected).
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "zdx_math.cuh"

using namespace zdx;

static double qdist(Q4 q, Q4 p) {
    const double a = std::sqrt((q.w - p.w) * (q.w - p.w) + (q.x - p.x) * (q.x - p.x) + (q.y - p.y) * (q.y - p.y) + (q.z - p.z) * (q.z - p.z));
    const double b = std::sqrt((q.w + p.w) * (q.w + p.w) + (q.x + p.x) * (q.x + p.x) + (q.y + p.y) * (q.y + p.y) + (q.z + p.z) * (q.z + p.z));
    return a < b ? a : b;
}

int main() {
    long n = 0, held = 0, wrong = 0;
    for (;;) {
        double v[40];
        for (int i = 0; i < 40; ++i) {
            uint64_t u;
            if (std::scanf("%" SCNx64, &u) != 1) {
                std::printf("%ld %ld %ld\n", n, held, wrong);
                return 0;
            }
            std::memcpy(v + i, &u, 8);
        }
        ++n;
        V3 L[2][3], T[2][3], x[2], nn[2];
        std::memcpy(&L[0][0].x, v, 18 * 8);
        Q4 q[2];
        double R[2] = {0.0, 0.0}, r[2], d[2];
        bool ok = true;
        for (int k = 0; k < 2; ++k) {
            const double* ps = v + 18 + 7 * k;
            x[k] = V3{ps[0], ps[1], ps[2]};
            q[k] = qnormalize(Q4{ps[3], ps[4], ps[5], ps[6]});
            for (int i = 0; i < 3; ++i) {
                R[k] = smax(R[k], norm(L[k][i]) * (1.0 + 1e-12));
                T[k][i] = qrotate_n(q[k], L[k][i]) + x[k];
            }
            tri_inflation(L[k][0], L[k][1], L[k][2], &r[k]);
            r[k] = std::nextafterf((float)r[k], INFINITY);
            ok = plane_from_tri(T[k][0], T[k][1], T[k][2], nn[k], d[k]) && ok;
        }
        if (!ok) continue;
        auto inf = [](V3 p) { return smax3(fabs(p.x), fabs(p.y), fabs(p.z)); };
        const double pad = 1e-9 * (inf(x[0]) + inf(x[1]) + R[0] + R[1]);
        const double gA = plane_gap(nn[1], d[1], T[0][0], T[0][1], T[0][2]), gB = plane_gap(nn[0], d[0], T[1][0], T[1][1], T[1][2]);
        const double clear = planes_clearance(gA, gB, r[0], r[1], R[0], R[1], pad);
        if (!(clear > 17.0 * pad)) continue;
        ++held;
        // towards each other across the wider gap: A by +, B by -
        const V3 w = gA > gB ? nn[1] * (dot(nn[1], T[0][0]) + d[1] > 0 ? -1.0 : 1.0) : nn[0] * (dot(nn[0], T[1][0]) + d[0] > 0 ? 1.0 : -1.0);
        const double all = (clear - 8.5 * pad) * (1.0 - 1e-8);
        for (int kind = 0; kind < 4; ++kind) {
            V3 M[2][3], mn[2], y[2];
            double md[2], moved = 0.0;
            bool use = true;
            for (int k = 0; k < 2; ++k) {
                // all of the motion A's, B's, or half each; one kind turned about a free axis, the others about the
                // one that takes the corner nearest to the other triangle towards it fastest
                const double mine = all * (kind == 0 ? (k == 0 ? 1.0 : 0.0) : kind == 1 ? (k == 1 ? 1.0 : 0.0) : 0.5);
                const double* m = v + 32 + 4 * k;
                const V3 to = w * (k == 0 ? 1.0 : -1.0);
                int best = 0;
                for (int i = 1; i < 3; ++i)
                    if (dot(T[k][i], to) > dot(T[k][best], to)) best = i;
                V3 ax = kind == 3 ? V3{m[0], m[1], m[2]} : cross(T[k][best] - x[k], to);
                if (!(norm(ax) > 0.0)) ax = V3{1.0, 0.0, 0.0};
                ax = ax * (1.0 / norm(ax));
                // 2 R |dq| = 4 R sin(angle / 4)
                double s = R[k] > 0.0 ? mine * fabs(m[3]) / (4.0 * R[k]) : 0.0;
                s = s < 0.5 ? s : 0.5;
                const double h = 2.0 * asin(s);  // half the angle
                const Q4 t = qmul(Q4{cos(h), ax.x * sin(h), ax.y * sin(h), ax.z * sin(h)}, q[k]);
                const Q4 qn = qnormalize(t);
                y[k] = x[k] + to * (mine - 4.0 * R[k] * s);
                moved += norm(y[k] - x[k]) + 2.0 * R[k] * qdist(qn, q[k]);
                for (int i = 0; i < 3; ++i) M[k][i] = qrotate_n(qn, L[k][i]) + y[k];
                use = plane_from_tri(M[k][0], M[k][1], M[k][2], mn[k], md[k]) && use;
            }
            // k_cache_skip's own condition
            const double pad2 = 1e-9 * (inf(y[0]) + inf(y[1]) + R[0] + R[1]);
            V3 o0, o1;
            if (use && moved * (1.0 + 1e-9) + 8.0 * pad2 < clear && tri_tri(M[0], mn[0], md[0], M[1], mn[1], md[1], o0, o1)) ++wrong;
        }
    }
}

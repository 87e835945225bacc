// Checks of parts of the per-ray walk (ytgb_ray.cuh) against their plain
// forms, compiled for the CPU -- TEST INFRASTRUCTURE.
#include <cmath>
#include <cstring>
#include <random>
#include "ytgb.h"
#include "ytgb_ray.cuh"
using namespace ytgb;

static void make_brick(const double le[3], const double re[3], const int dims[3], ytgb_brick &b, double *bounds) {
    std::memset(&b, 0, sizeof(b));
    int o = 0;
    for (int i = 0; i < 3; i++) {
        b.left_edge[i] = le[i];
        b.right_edge[i] = re[i];
        b.dims[i] = dims[i];
        b.dds[i] = (re[i] - le[i]) / dims[i];
        b.idds[i] = 1.0 / b.dds[i];
        b.snap[i] = 1e-10 * b.dds[i];
        b.lef[i] = (float)le[i];
        b.ref[i] = (float)re[i];
        b.iddsf[i] = (float)b.idds[i];
        for (int k = 0; k <= dims[i]; k++) bounds[o++] = k * b.dds[i] + le[i];
    }
}

static void finish_ray(Ray &r) {
    for (int i = 0; i < 3; i++) {
        r.step[i] = r.dir[i] < 0 ? -1 : (r.dir[i] == 0.0 ? 0 : 1);
        r.iv[i] = r.step[i] != 0 ? 1.0 / r.dir[i] : 0.0;
        r.fpos[i] = (float)r.pos[i];
        r.fdir[i] = (float)r.dir[i];
        r.ifd[i] = 1.0f / r.fdir[i];
        r.td_dds[i] = -1.0;
        r.td[i] = 0.0;
    }
}

// Random rays at random bricks: aim 0 through the brick's interior, 1 through
// its edges and corners (within 1e-12 .. 1e-3), 2 along the axes (zero
// components, starts on face planes), 3 from inside the brick.  out: walks
// that the face form decided, that it left to the general form, and the
// mismatches between the two.
extern "C" void check_setup(long long n, int aim, unsigned long long seed, long long out[3]) {
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    out[0] = out[1] = out[2] = 0;
    for (long long k = 0; k < n; k++) {
        double le[3], re[3], bounds[256];
        int dims[3];
        for (int i = 0; i < 3; i++) {
            dims[i] = 1 + (int)(g() % 33);
            const double dx = g() % 3 ? std::ldexp(1.0, -(int)(4 + g() % 6)) : 0.01 + 0.05 * u(g);
            le[i] = g() % 2 ? std::ldexp((double)(g() % 64), -6) : u(g);
            re[i] = le[i] + dims[i] * dx;
        }
        ytgb_brick b;
        make_brick(le, re, dims, b, bounds);
        Ray r;
        double q[3];
        for (int i = 0; i < 3; i++) {
            q[i] = le[i] + u(g) * (re[i] - le[i]);
            r.pos[i] = 0.5 + 2.0 * (u(g) - 0.5) * 2.0;
            if (aim == 1 && g() % 2) {
                const double e = std::pow(10.0, -3.0 - 9.0 * u(g)) * (g() % 2 ? 1.0 : -1.0);
                q[i] = (g() % 2 ? le[i] : re[i]) + (g() % 4 ? e : 0.0);
            }
            if (aim == 3) r.pos[i] = le[i] + u(g) * (re[i] - le[i]);
        }
        const double s = 0.5 + u(g);
        for (int i = 0; i < 3; i++) r.dir[i] = (q[i] - r.pos[i]) / s;
        if (aim == 2)
            for (int i = 0; i < 3; i++)
                if (g() % 2) {
                    r.dir[i] = 0.0;
                    r.pos[i] = g() % 3 ? q[i] : (g() % 2 ? le[i] : re[i]);
                }
        finish_ray(r);
        BrickF bf;
        load_brick_f(&b, bf);
        const double max_t = g() % 4 ? 1.0 : u(g);
        const long long kmax = dkey(max_t);
        Walk wf, wg;
        const int f = walk_setup_face(bf, &b, bounds, r, r.ifd, kmax, wf);
        const bool w = walk_setup_general(bf, &b, bounds, r, r.ifd, max_t, kmax, wg);
        if (f < 0) {
            out[1]++;
            continue;
        }
        out[0]++;
        bool same = (f > 0) == w;
        if (same && w) {
            same = dbits(wf.enter_t) == dbits(wg.enter_t);
            for (int i = 0; i < 3; i++)
                same = same && dbits(wf.tmax[i]) == dbits(wg.tmax[i]) && wf.cur[i] == wg.cur[i] && wf.P[i] == wg.P[i];
        }
        if (!same) out[2]++;
    }
}

// Runs of integer steps (run_axis) against float64 adds: from each start a
// walk of steps on one axis, taken as the cell loop takes them -- adds of the
// run's increment below its limit, the float64 add and a new run at it.
// ties: tdelta with few significant bits (exact halves); left: the brick's
// remaining steps.  Returns the mismatches; looks: the steps taken in full.
extern "C" long long check_runs(long long n, int steps, int ties, unsigned long long seed, long long *looks) {
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    const long long kmax = dkey(1.0);
    long long bad = 0;
    *looks = 0;
    for (long long k = 0; k < n; k++) {
        double x = std::pow(2.0, -14.0 * u(g)) * 0.999, d = std::pow(2.0, -2.0 - 14.0 * u(g));
        if (ties) {
            long long b = dbits(d);
            b &= ~((1LL << (40 + g() % 12)) - 1);
            d = dfrom(b);
            b = dbits(x) & ~((1LL << (g() % 52)) - 1);
            x = dfrom(b | (long long)(g() % 2));
        }
        const float v = (float)(1.0 / d);
        int left = 1 + (int)(g() % (2 * steps));
        long long t = dbits(x), at = kmax, inc = 0;
        double ref = x;
        if (t < kmax) inc = run_axis(t, dbits(d), v, left, at);
        for (int j = 0; j < steps && left > 0 && t < kmax; j++, left--) {
            if (t < at) {
                if (left == 1) { bad++; break; }  // the leaving step must be looked at
                t += inc;
            } else {
                ++*looks;
                t = dbits(dfrom(t) + d);
                at = kmax;
                inc = 0;
                if (left > 1 && t < kmax) inc = run_axis(t, dbits(d), v, left - 1, at);
            }
            ref = ref + d;
            if (t != dbits(ref)) { bad++; break; }
        }
    }
    return bad;
}

#include "ytgb_octree.cuh"

static double rand_t(std::mt19937_64 &g) {  // t of either sign over many binades, some with short mantissas
    std::uniform_real_distribution<double> u(0.0, 1.0);
    double x = std::ldexp(1.0 + u(g), (int)(g() % 40) - 30);
    if (g() % 3 == 0) x = dfrom(dbits(x) & ~((1LL << (g() % 52)) - 1));
    if (g() % 50 == 0) x = 0.0;
    return x;
}

// The octree path's integer forms against float64: midpoints (positive t and
// any t), the pair of float32 and the float32 difference; returns mismatches.
extern "C" long long check_octree_values(long long n, unsigned long long seed) {
    std::mt19937_64 g(seed);
    long long bad = 0;
    for (long long k = 0; k < n; k++) {
        const double a = rand_t(g), b = g() % 2 ? a * (1.0 + 1e-3 * (double)(g() % 1000)) : rand_t(g);
        const double mid = (a + b) * 0.5;
        if (dbits(midpoint<T_BITS>(a, b)) != dbits(mid) || dbits(midpoint<T_KEYS>(a, b)) != dbits(mid)) bad++;
        const double c = g() % 2 ? -b : b, m2 = (a + c) * 0.5;
        const double got = midpoint<T_KEYS>(a, c);
        if (!(got == m2)) bad++;
        float hi, lo;
        split_pair(c, hi, lo);
        const float fh = (float)c;
        const bool tie = std::fabs(c - (double)fh) == std::fabs((double)std::nextafter(fh, c > (double)fh ? INFINITY : -INFINITY) - c);
        if (!tie && (hi != fh || lo != (float)(c - (double)fh))) bad++;
        if (tie && (double)hi + (double)lo != c) bad++;
        if (diff_nearest(b, a) != (float)(b - a)) bad++;
    }
    return bad;
}

// Checks of the per-ray conversions (ytgb_ray.cuh) against the language's own,
// compiled for the CPU -- TEST INFRASTRUCTURE.
#include <cmath>
#include <cstring>
#include <random>
#include "ytgb.h"
#include "ytgb_ray.cuh"
using namespace ytgb;

static bool same(float a, float b) { return (a != a && b != b) || std::memcmp(&a, &b, sizeof(a)) == 0; }

// Mismatches of narrow with the conversion: every exponent and sign with
// mantissas at, next to and between the float32 values and their midpoints
// (carries into the next binade among them), and n random bit patterns.
extern "C" long long check_narrow(long long n, unsigned long long seed) {
    std::mt19937_64 g(seed);
    long long bad = 0;
    const long long half = 1LL << 28, ulp = 1LL << 29, top = (1LL << 52) - 1;
    const long long mant[] = {0, 1, half - 1, half, half + 1, ulp - 1, ulp, ulp + half - 1, ulp + half, ulp + half + 1,
                              top - ulp - half, top - ulp, top - half - 1, top - half, top - half + 1, top};
    for (long long e = 0; e <= 0x7ff; e++)
        for (long long s = 0; s < 2; s++)
            for (long long m : mant) {
                const double x = dfrom((s << 63) | (e << 52) | m);
                if (!same(narrow(x), (float)x)) bad++;
            }
    for (long long k = 0; k < n; k++) {
        const double x = dfrom((long long)g()), y = std::ldexp(1.0 + (double)(g() >> 12) * 0x1p-52, (int)(g() % 300) - 160);
        if (!same(narrow(x), (float)x)) bad++;
        if (!same(narrow(-y), (float)-y)) bad++;
    }
    return bad;
}

// A ray's float32 position, direction and reciprocals as make_ray forms them for
// both lenses against plain casts and divisions; returns the mismatches.
extern "C" long long check_rays(long long n, unsigned long long seed) {
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    long long bad = 0;
    for (long long k = 0; k < n; k++) {
        ytgb_view v;
        std::memset(&v, 0, sizeof(v));
        v.nx = 1 + (int)(g() % 9);
        v.ny = 1 + (int)(g() % 9);
        v.lens = g() % 2 ? YTGB_LENS_PLANE_PARALLEL : YTGB_LENS_PERSPECTIVE;
        const double scale = std::ldexp(1.0, (int)(g() % 60) - 30);
        for (double &x : v.vp_pos) x = u(g) * scale;
        for (double &x : v.vp_dir) x = g() % 8 ? u(g) * scale : 0.0;
        for (double &x : v.width) x = 0.1 + std::fabs(u(g));
        v.ray_scale = 1.0 + std::fabs(u(g));
        view_derive(v);
        Ray r;
        make_ray(v, (int)(g() % v.nx), (int)(g() % v.ny), r);
        for (int i = 0; i < 3; i++) {
            if (!same(r.fpos[i], (float)r.pos[i]) || !same(r.fdir[i], (float)r.dir[i])) bad++;
            const double iv = r.dir[i] != 0.0 ? 1.0 / r.dir[i] : 0.0;
            if (r.dir[i] == r.dir[i] && dbits(r.iv[i]) != dbits(iv)) bad++;
            if (!same(r.ifd[i], 1.0f / r.fdir[i])) bad++;
        }
    }
    return bad;
}

// Every form of the per-ray walk (ytgb_ray.cuh) over exactly sized arrays --
// TEST INFRASTRUCTURE.  Built with the address and undefined-behaviour
// sanitizers, a read of one element outside a brick's fields, mask, boundary
// table, low parts or transfer-function tables ends the program; built without,
// it prints the same sums over the images and counters, so that the builds (the
// two cell loops, and local variables that start as zero or as a pattern) can be
// compared.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <random>
#include <vector>
#include "ytgb.h"
#include "ytgb_ray.cuh"
#if defined(__SANITIZE_ADDRESS__)
#include <sanitizer/asan_interface.h>
#define POISON(p, n) __asan_poison_memory_region(p, n)
#define UNPOISON(p, n) __asan_unpoison_memory_region(p, n)
#else
#define POISON(p, n)
#define UNPOISON(p, n)
#endif
using namespace ytgb;

static std::mt19937_64 rng;
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }

// An array whose items lie between poisoned gaps.
template <typename T> struct Gapped {
    static constexpr size_t GAP = 32;
    std::vector<T> mem;
    std::vector<size_t> at;
    size_t add(size_t n) {
        at.push_back(mem.size() + GAP);
        mem.resize(mem.size() + GAP + ((n + 7) & ~(size_t)7) + GAP);
        lens.push_back(n);
        return at.back();
    }
    std::vector<size_t> lens;
    void guard() {
        if (mem.empty()) return;
        POISON(mem.data(), mem.size() * sizeof(T));
        for (size_t k = 0; k < at.size(); k++) UNPOISON(mem.data() + at[k], lens[k] * sizeof(T));
    }
    ~Gapped() { if (!mem.empty()) UNPOISON(mem.data(), mem.size() * sizeof(T)); }
};

struct Scene {
    std::vector<ytgb_brick> bricks;
    Gapped<float> data, lo;
    Gapped<uint8_t> masks;
    Gapped<double> bounds;
    std::vector<int32_t> order;
};

// Bricks side by side along x, of these cells each; verts: vertex fields.
static void make_scene(Scene &s, const int dims[3], int nf, bool verts, bool masked, double cell) {
    const double start[3] = {uni(0.0, 0.2), uni(0.0, 0.2), uni(0.0, 0.2)};
    double x = start[0];
    for (int k = 0; k < 3; k++) {
        ytgb_brick b;
        std::memset(&b, 0, sizeof(b));
        const double h = k < 2 ? cell : 0.5 * cell;  // (the last of another level)
        int64_t n = 1;
        size_t nb = 0;
        for (int i = 0; i < 3; i++) {
            const double l = i == 0 ? x : start[i], r = l + dims[i] * h;
            b.left_edge[i] = l;
            b.right_edge[i] = r;
            b.dds[i] = (r - l) / dims[i];
            b.idds[i] = 1.0 / b.dds[i];
            b.snap[i] = 1e-10 * b.dds[i];
            b.dims[i] = dims[i];
            b.lef[i] = (float)l;
            b.ref[i] = (float)r;
            b.iddsf[i] = (float)b.idds[i];
            n *= dims[i] + (verts ? 1 : 0);
            nb += dims[i] + 1;
        }
        x = b.right_edge[0];
        b.n_fields = nf;
        b.field_stride = n;
        b.data_offset = (int64_t)s.data.add(n * nf);
        const size_t o = s.lo.add(n * nf);
        (void)o;  // (the same offsets)
        b.bounds_offset = (int64_t)s.bounds.add(nb);
        b.mask_offset = -1;
        const size_t cells = (size_t)dims[0] * dims[1] * dims[2];
        if (masked && k != 1) {
            b.mask_offset = (int64_t)s.masks.add(cells);
            for (size_t c = 0; c < cells; c++) s.masks.mem[b.mask_offset + c] = rng() % 4 != 0;
        }
        size_t q = (size_t)b.bounds_offset;
        for (int i = 0; i < 3; i++)
            for (int c = 0; c <= dims[i]; c++) s.bounds.mem[q++] = c * b.dds[i] + b.left_edge[i];
        for (int64_t c = 0; c < n * nf; c++) {
            // values in, at and beyond the tables' bounds [0, 1], zeros, infinities and NaN
            const unsigned pick = rng() % 64;
            double v = pick == 0 ? 0.0 : pick == 1 ? 1.0 : pick == 2 ? INFINITY : pick == 3 ? NAN : pick == 4 ? 3e38 : uni(-0.1, 1.1);
            s.data.mem[b.data_offset + c] = (float)v;
            const double rest = v - (double)(float)v;
            s.lo.mem[b.data_offset + c] = rest == rest && rest - rest == 0.0 ? (float)rest : 0.0f;
        }
        s.bricks.push_back(b);
    }
    for (int k : {2, 0, 1}) s.order.push_back(k);
    s.data.guard();
    s.lo.guard();
    s.masks.guard();
    s.bounds.guard();
}

// nt tables over [0, 1] of differing bins (nt 0: a ColorTransferFunction's four)
static void make_tf(ytgb_tf &t, std::unique_ptr<float4[]> &tab, size_t &n, int nt, int nf, int bins, int grey) {
    std::memset(&t, 0, sizeof(t));
    const bool ctf = nt == 0;
    t.n_fits = ctf ? 4 : nt;
    t.grey_opacity = grey;
    t.nbins_max = bins;
    t.ctf_fast = ctf;
    for (int c = 0; c < 6; c++) t.field_table_ids[c] = c < t.n_fits ? c : 0;
    n = (size_t)t.n_fits * bins;
    tab.reset(new float4[n]);
    for (int q = 0; q < t.n_fits; q++) {
        const int nb = ctf || q == 0 ? bins : std::max(2, bins - q);
        t.field_id[q] = ctf ? 0 : q % nf;
        t.weight_field_id[q] = !ctf && q == 2 && nf > 1 ? 1 : -1;
        t.weight_table_id[q] = ctf ? (q < 3 ? 3 : -1) : (q == 1 && nt > 2 ? 2 : -1);
        t.nbins[q] = nb;
        t.lo_excl[q] = 0.0f;
        t.hi_excl[q] = 1.0f;
        t.b0[q] = 0.0f;
        t.idbin[q] = (float)(nb - 1);
        t.bound64[q][0] = 0.0;
        t.bound64[q][1] = 1.0;
        for (int b = 0; b < bins; b++)
            tab[(size_t)q * bins + b] = make_float4((float)uni(0, 1), (float)uni(-1, 1), (float)b / (nb - 1), 0.0f);
    }
}

constexpr int RAYS = 48;

static void make_rays(const Scene &s, std::vector<double> &pos, std::vector<double> &dir) {
    const ytgb_brick &a = s.bricks[0], &z = s.bricks[2];
    for (int k = 0; k < RAYS; k++) {
        double p[3], q[3], d[3];
        const ytgb_brick &b = s.bricks[rng() % 3];
        for (int i = 0; i < 3; i++) {
            const double l = a.left_edge[i], r = i == 0 ? z.right_edge[i] : a.right_edge[i];
            q[i] = uni(b.left_edge[i], b.right_edge[i]);
            p[i] = l + (r - l) * uni(-1.5, 2.5);
            if (k % 6 == 1) q[i] = rng() % 2 ? b.left_edge[i] : b.right_edge[i];          // a corner
            if (k % 6 == 2) q[i] = (rng() % 2 ? b.left_edge[i] : b.right_edge[i]) + uni(-1e-9, 1e-9);
            if (k % 6 == 3) p[i] = uni(b.left_edge[i], b.right_edge[i]);                  // from inside
        }
        const double f = uni(0.3, 2.0);
        for (int i = 0; i < 3; i++) d[i] = (q[i] - p[i]) * f;
        if (k % 6 == 4)  // along one or two axes, often on the cells' planes
            for (int i = 0; i < 3; i++)
                if (rng() % 2) {
                    d[i] = 0.0;
                    p[i] = rng() % 2 ? q[i] : b.left_edge[i] + b.dds[i] * (double)(rng() % (b.dims[i] + 1));
                }
        if (k % 6 == 5) {  // along a diagonal through the cells' corners (ties)
            const double h = b.dds[0];
            for (int i = 0; i < 3; i++) {
                p[i] = b.left_edge[i] - 4.0 * h;
                d[i] = (8.0 + b.dims[0]) * h;
            }
        }
        for (int i = 0; i < 3; i++) {
            pos.push_back(p[i]);
            dir.push_back(d[i]);
        }
    }
}

template <int MODE, int VAR, bool TG>
static void walk_all(const ytgb_render_args &a, const float4 *tab, unsigned long long *cnt) {
    for (int vi = 0; vi < a.view.nx; vi++) {
        std::unique_ptr<Ray> r(new Ray);
        make_ray(a.view, vi, 0, *r);
        double *img = a.image + (size_t)vi * 4;
        RayState st;
        ray_state_init(st, img, a.zbuffer ? a.zbuffer[vi] : 1.0, a.zbuffer != nullptr, a.flags);
        for (int k = 0; k < a.n_order; k++) walk_brick<MODE, VAR, TG>(a, tab, *r, a.order[k], st);
        for (int c = 0; c < 4; c++)
            if (st.touched & (1u << c)) img[c] = image_value(st, c);
        cnt[0] += st.visits;
        cnt[1] += st.walks;
        cnt[2] += st.guarded;
    }
}

template <int MODE, int VAR> static void both(const ytgb_render_args &a, const float4 *packed, unsigned long long *cnt, bool tg) {
    if (tg || !(MODE == MODE_VR || MODE == MODE_LIGHT)) {
        walk_all<MODE, VAR, true>(a, packed, cnt);
        return;
    }
    const int nb = a.tf.nbins_max;
    if (VAR & V_CTF) {  // the shared-memory layout
        std::unique_ptr<float4[]> t(new float4[3 * (size_t)nb]);
        for (int b = 0; b < nb; b++) {
            const float4 t0 = packed[b], t1 = packed[nb + b], t2 = packed[2 * nb + b], t3 = packed[3 * nb + b];
            t[3 * b] = make_float4(t0.x, t1.x, t2.x, t3.x);
            t[3 * b + 1] = make_float4(t0.y, t1.y, t2.y, t3.y);
            t[3 * b + 2] = make_float4(t3.z, t3.w, 0.f, 0.f);
        }
        walk_all<MODE, VAR, false>(a, t.get(), cnt);
    } else {
        walk_all<MODE, VAR, false>(a, packed, cnt);
    }
}

static unsigned long long sum(const void *p, size_t n) {
    unsigned long long h = 0xcbf29ce484222325ull;
    for (size_t i = 0; i < n; i++) h = (h ^ ((const unsigned char *)p)[i]) * 0x100000001b3ull;
    return h;
}

int main() {
    const int shapes[][3] = {{1, 1, 1}, {1, 7, 2}, {5, 1, 33}, {16, 16, 16}, {1100, 1, 2}, {2, 1500, 1}};
    struct Form { int kind, nf, nt; };  // nt: tables, 0 a ColorTransferFunction
    const Form forms[] = {{MODE_VR, 1, 0}, {MODE_VR, 1, 1}, {MODE_VR, 2, 3}, {MODE_VR, 6, 6}, {MODE_IPROJ, 1, 0}, {MODE_IPROJ, 2, 0},
                          {MODE_IPROJ, 5, 0}, {MODE_PROJ, 1, 0}, {MODE_PROJ, 6, 0}, {MODE_MIP, 1, 0}, {MODE_MIP, 3, 0},
                          {MODE_LIGHT, 1, 0}, {MODE_LIGHT, 1, 1}, {MODE_LIGHT, 3, 4}};
    unsigned long long total = 0;
    int id = 0;
    for (const Form &f : forms)
        for (const auto &dims : shapes)
            for (int opt = 0; opt < 12; opt++) {
                rng.seed(1000 + id++);
                const bool verts = f.kind != MODE_PROJ && f.kind != MODE_MIP, tables = f.kind == MODE_VR || f.kind == MODE_LIGHT;
                const int ns = opt % 4 == 0 ? 1 : (opt % 4 == 1 ? 2 : (opt % 4 == 2 ? 7 : 1));
                const bool masked = opt % 3 == 1, ref = tables && opt % 2 == 1, tg = opt % 4 >= 2, grey = opt % 5 >= 2;
                Scene s;
                make_scene(s, dims, f.nf, verts, masked, std::ldexp(opt % 2 ? 1.0 : uni(0.7, 1.4), opt % 3 ? -6 : -4));
                std::vector<double> pos, dir, img((size_t)RAYS * 4, 0.0), zb;
                make_rays(s, pos, dir);
                ytgb_render_args a;
                std::memset(&a, 0, sizeof(a));
                a.kind = f.kind;
                a.n_samples = ns;
                a.n_order = (int)s.order.size();
                a.flags = opt % 6 == 5 ? YTGB_FLAG_NO_COMPENSATION : 0;
                a.view.nx = RAYS;
                a.view.ny = 1;
                a.view.lens = YTGB_LENS_PER_PIXEL;
                a.view.px_pos = pos.data();
                a.view.px_dir = dir.data();
                a.bricks = s.bricks.data();
                a.order = s.order.data();
                a.data = s.data.mem.data();
                a.masks = s.masks.mem.empty() ? nullptr : s.masks.mem.data();
                a.bounds = s.bounds.mem.data();
                a.image = img.data();
                if (opt % 5 == 4) {
                    for (int k = 0; k < RAYS; k++) zb.push_back(uni(-0.1, 1.2));
                    a.zbuffer = zb.data();
                }
                std::unique_ptr<float4[]> tab;
                size_t n_tab = 0;
                if (tables) {
                    make_tf(a.tf, tab, n_tab, f.nt, f.nf, opt % 3 == 0 ? 2 : 67, grey);
                    a.tf_tables = &tab[0].x;
                }
                if (ref || (f.kind == MODE_LIGHT && opt % 3 == 2)) a.data_lo = s.lo.mem.data();
                a.range_eps = ref ? 1.5f * 0x1p-24f : 0.0f;
                a.light_dir[0] = 0.6f;
                a.light_dir[2] = -0.8f;
                for (float &c : a.light_rgba) c = 0.7f;
                view_derive(a.view);
                unsigned long long cnt[3] = {0, 0, 0};
                const int var = render_variant(a);
                switch (f.kind) {
                case MODE_VR:
                    switch (var) {
                    case V_CTF: both<MODE_VR, V_CTF>(a, tab.get(), cnt, tg); break;
                    case V_REF: both<MODE_VR, V_REF>(a, tab.get(), cnt, tg); break;
                    case V_CTF | V_REF: both<MODE_VR, V_CTF | V_REF>(a, tab.get(), cnt, tg); break;
                    default: both<MODE_VR, 0>(a, tab.get(), cnt, tg);
                    }
                    break;
                case MODE_PROJ: both<MODE_PROJ, 0>(a, nullptr, cnt, tg); break;
                case MODE_IPROJ: both<MODE_IPROJ, 0>(a, nullptr, cnt, tg); break;
                case MODE_MIP: both<MODE_MIP, 0>(a, nullptr, cnt, tg); break;
                default:
                    if (var & V_REF) both<MODE_LIGHT, V_REF>(a, tab.get(), cnt, tg);
                    else both<MODE_LIGHT, 0>(a, tab.get(), cnt, tg);
                }
                for (double &v : img)
                    if (v != v) v = NAN;  // (one NaN)
                std::printf("%d/%d/%d %dx%dx%d %d: %llu visits %llu walks %016llx\n", f.kind, f.nf, f.nt, dims[0], dims[1], dims[2], opt,
                            cnt[0], cnt[1], sum(img.data(), img.size() * sizeof(double)) ^ cnt[2]);
                total += cnt[0];
            }
    std::printf("cells %llu\n", total);
    return total > 100000 ? 0 : 2;
}

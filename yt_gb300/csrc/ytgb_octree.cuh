// ytgb_octree.cuh -- the octree ray caster of yt's octree volume source,
// per ray, host/device (the test harness runs it on the CPU).
//
// ImageSampler.cast_through_octree (image_samplers.pyx:202-288) casts each
// pixel's ray through an octree of cells (Octree<int>::cast_ray,
// _octree_raytracing.hpp:199-230: the parametric traversal of Revelles,
// Urena and Lastra, proc_subtree :276-337) and hands every terminal cell it
// meets, in traversal order, to the sampler as a 1x1x1 vertex-centred brick
// with the cell's own edges.  The traversal's float64 values (the direction
// normalisation, the t of the six slab planes, the midpoints) are formed
// from the same operands in the same order as the reference, unfused, so
// the cells and their enter/exit t are bit-identical; the recursion becomes
// an explicit stack of at most depth + 1 frames.
#pragma once

#include "ytgb_ray.cuh"

namespace ytgb {

// Device form of one octree node: children (-1: none), key, flags.
struct ONode {
    int32_t child[8];
    int32_t key;
    int32_t flags;  // bit 0: terminal, bit 1: has a children array
};

struct OctreeView {
    const ONode *nodes;
    int32_t n_nodes;
    const float *verts;    // 8 per cell, (i,j,k) C order
    const double *edges;   // 9 per cell: left edge, right edge, 1/(right - left)
    const float4 *edges_f; // 3 per cell (or null): left edge hi, lo, (float)(1/(right - left))
    int32_t n_cells;
    int32_t depth;
    double dle[3], dre[3], size[3];
};

constexpr int OCT_MAX_DEPTH = 30;

// The traversal's comparisons, by what is known of the ray's six slab t.
// T_BITS: all are +0 or positive and below 2^1023, so every midpoint
// (a + b) * 0.5 is too, no NaN arises, and the float64 bits order like the
// values (a ray that starts outside the domain).  T_KEYS: all are below 2^1023
// in magnitude: order-preserving int64 keys.  Both run on the integer pipe
// (GB300's float64 pipe is 1/64 of its float32 rate).  T_FLOAT: any other ray
// (a direction component of 0 makes inf and, at a midpoint, NaN) takes the
// float64 comparisons.
constexpr int T_FLOAT = 0, T_KEYS = 1, T_BITS = 2;
template <int K> YTGB_HD bool lt(double a, double b) {
    return K == T_BITS ? dbits(a) < dbits(b) : K == T_KEYS ? dkey(a) < dkey(b) : a < b;
}
template <int K> YTGB_HD bool ge(double a, double b) { return K ? !lt<K>(a, b) : a >= b; }

// std::max / std::min as the reference calls them
template <int K> YTGB_HD double smax(double a, double b) { return lt<K>(a, b) ? b : a; }
template <int K> YTGB_HD double smin(double a, double b) { return lt<K>(b, a) ? b : a; }

// (a + b) * 0.5.  T_BITS: inside one binade the mean of the bits, an odd sum
// going to the even neighbour as the float64 sum's rounding does (its quantum
// is two ulps of a and b); most nodes' slabs lie in one binade, so the float64
// add is rare.  Else the halving takes one off the exponent (exact while the
// sum's exponent field is above 1).
template <int K> YTGB_HD double midpoint(double a, double b) {
    if (K == T_BITS && ((dbits(a) ^ dbits(b)) >> 52) == 0 && dbits(a) >= (2LL << 52)) {
        const unsigned long long s = (unsigned long long)dbits(a) + (unsigned long long)dbits(b), q = s >> 1;
        return dfrom((long long)(q + (s & q & 1)));
    }
    const double s = dadd(a, b);
    if (K && ((dbits(s) >> 52) & 0x7ff) > 1) return dfrom(dbits(s) - (1LL << 52));
    return dmul(s, 0.5);
}

template <int K>
YTGB_HD int first_node(const double t0[3], const double tm[3]) {
    int index = 0;
    if (ge<K>(t0[0], smax<K>(t0[1], t0[2]))) {
        if (lt<K>(tm[1], t0[0])) index |= 2;
        if (lt<K>(tm[2], t0[0])) index |= 1;
    } else if (ge<K>(t0[1], smax<K>(t0[0], t0[2]))) {
        if (lt<K>(tm[0], t0[1])) index |= 4;
        if (lt<K>(tm[2], t0[1])) index |= 1;
    } else {
        if (lt<K>(tm[0], t0[2])) index |= 4;
        if (lt<K>(tm[1], t0[2])) index |= 2;
    }
    return index;
}

// The successor of child q, which the ray leaves through the nearest of its
// exit planes t1 (next_node's exit-plane table, :225-253): the sibling across
// that plane, or 8 where the plane is the parent's own.
template <int K>
YTGB_HD int next_node(int q, const double t1[3]) {
    if (lt<K>(t1[0], smin<K>(t1[1], t1[2]))) return q & 4 ? 8 : q | 4;
    if (lt<K>(t1[1], smin<K>(t1[0], t1[2]))) return q & 2 ? 8 : q | 2;
    return q & 1 ? 8 : q | 1;
}

// s + e == a + b exactly (TwoSum, Knuth TAOCP vol. 2, 4.2.2)
YTGB_HD void two_sum(float a, float b, float &s, float &e) {
    s = fadd(a, b);
    const float bp = fsub(s, a);
    e = fadd(fsub(a, fsub(s, bp)), fsub(b, bp));
}

// What a node's frame needs beside its child's slab to be restored: the child
// q has t0 = (upper half ? tm : t0) and t1 = (upper half ? t1 : tm) on each
// axis, so only the plane it lost.
struct OFrame {
    double lost[3];
    int32_t node;
    int32_t next;  // the node's next child, the child q taken << 4
};

// Calls cell(key, t_in, t_out) for every terminal cell of the ray's path,
// in proc_subtree's order.  Returns false if the stack or step budget ran
// out (a malformed tree).
template <int K, typename F>
YTGB_HD bool octree_walk(const OctreeView &o, const double t0[3], const double t1[3], int a, F &cell);

// dd: the direction's length, sqrt(x^2 + y^2 + z^2) summed in that order.
template <typename F>
YTGB_HD bool octree_cast(const OctreeView &o, const double o_in[3], const double d_in[3], double dd, F cell) {
    double p[3], d[3], t0[3], t1[3];
    int a = 0, bmask = 4;
    YTGB_UNROLL
    for (int i = 0; i < 3; i++) {
        p[i] = o_in[i];
        d[i] = ddiv(d_in[i], dd);
    }
    YTGB_UNROLL
    for (int i = 0; i < 3; i++) {
        if (d[i] < 0.0) {
            p[i] = dsub(o.size[i], p[i]);
            d[i] = -d[i];
            a |= bmask;
        }
        bmask >>= 1;
    }
    YTGB_UNROLL
    for (int i = 0; i < 3; i++) {
        t0[i] = ddiv(dsub(o.dle[i], p[i]), d[i]);
        t1[i] = ddiv(dsub(o.dre[i], p[i]), d[i]);
    }
    double mx = t0[0], mn = t1[0];  // std::max_element / std::min_element
    if (mx < t0[1]) mx = t0[1];
    if (mx < t0[2]) mx = t0[2];
    if (t1[1] < mn) mn = t1[1];
    if (t1[2] < mn) mn = t1[2];
    if (!(mx < mn)) return true;
    bool bounded = true, positive = true;  // exponent field below 0x7fe: |t| < 2^1023
    YTGB_UNROLL
    for (int i = 0; i < 3; i++) {
        bounded = bounded && (dbits(t0[i]) & 0x7ff0000000000000ll) < 0x7fe0000000000000ll &&
                  (dbits(t1[i]) & 0x7ff0000000000000ll) < 0x7fe0000000000000ll;
        positive = positive && dbits(t0[i]) >= 0 && dbits(t1[i]) >= 0;
    }
    return bounded ? (positive ? octree_walk<T_BITS>(o, t0, t1, a, cell) : octree_walk<T_KEYS>(o, t0, t1, a, cell))
                   : octree_walk<T_FLOAT>(o, t0, t1, a, cell);
}

// proc_subtree (_octree_raytracing.hpp:276-337) from the root over the slab
// [t0, t1].  The current node's slab is held in registers; the stack keeps 32
// bytes per level (80 with whole frames, which spilled out of L1 and L2).  The
// lanes of a warp each look for their next terminal cell, then sample
// together.
template <int K, typename F>
YTGB_HD bool octree_walk(const OctreeView &o, const double t0_in[3], const double t1_in[3], int a, F &cell) {
    OFrame st[OCT_MAX_DEPTH + 2];
    const int max_depth = o.depth < OCT_MAX_DEPTH ? o.depth : OCT_MAX_DEPTH;
    double t0[3], t1[3], tm[3];
    int node = 0, q = 8, sp = 0;  // q: the current node's next child
    bool ok = true, found = false;
    int key = 0;
    double t_in = 0.0, t_out = 0.0;
    if (lt<K>(t1_in[0], 0.0) || lt<K>(t1_in[1], 0.0) || lt<K>(t1_in[2], 0.0) || o.n_nodes < 1) return o.n_nodes >= 1;
    {
        const int flags = ldg(&o.nodes[0].flags);
        if (flags & 1) {
            cell(ldg(&o.nodes[0].key), smax<K>(smax<K>(t0_in[0], t0_in[1]), t0_in[2]),
                 smin<K>(smin<K>(t1_in[0], t1_in[1]), t1_in[2]));
            return true;
        }
        if (!(flags & 2)) return true;
    }
    YTGB_UNROLL
    for (int i = 0; i < 3; i++) {
        t0[i] = t0_in[i];
        t1[i] = t1_in[i];
        tm[i] = midpoint<K>(t0[i], t1[i]);
    }
    q = first_node<K>(t0, tm);
    const unsigned lanes = walking_lanes();
    int budget = 1 << 26;
    bool done = false;
    while (true) {
        // ---- the next terminal cell
        found = false;
        while (!done && !found) {
            // leave the nodes that are through: restore their parents' slabs
            while (q >= 8 && sp > 0) {
                const OFrame &f = st[--sp];
                const int took = f.next >> 4;
                node = f.node;
                q = f.next & 15;
                YTGB_UNROLL
                for (int i = 0; i < 3; i++) {
                    const bool up = (took >> (2 - i)) & 1;
                    const double lost = f.lost[i];
                    tm[i] = up ? t0[i] : t1[i];
                    t0[i] = up ? lost : t0[i];
                    t1[i] = up ? t1[i] : lost;
                }
            }
            if (--budget <= 0 || q >= 8) {
                ok = ok && budget > 0;
                done = true;
            } else {
                // child q's slab: lower or upper half on each axis (bit 2: x, 1: y, 0: z)
                double c0[3], c1[3];
                YTGB_UNROLL
                for (int i = 0; i < 3; i++) {
                    const bool up = (q >> (2 - i)) & 1;
                    c0[i] = up ? tm[i] : t0[i];
                    c1[i] = up ? t1[i] : tm[i];
                }
                const int child = ldg(&o.nodes[node].child[q ^ a]);
                const int took = q;
                q = next_node<K>(q, c1);
                const bool behind = K != T_BITS && (lt<K>(c1[0], 0.0) || lt<K>(c1[1], 0.0) || lt<K>(c1[2], 0.0));
                if (!behind && child >= 0) {
                    const int flags = child < o.n_nodes ? ldg(&o.nodes[child].flags) : 0;
                    if (child >= o.n_nodes) {
                        ok = false;
                        done = true;
                    } else if (flags & 1) {
                        key = ldg(&o.nodes[child].key);
                        t_in = smax<K>(smax<K>(c0[0], c0[1]), c0[2]);
                        t_out = smin<K>(smin<K>(c1[0], c1[1]), c1[2]);
                        found = true;
                    } else if (flags & 2) {
                        if (sp >= max_depth) {
                            ok = false;
                            done = true;
                        } else {
                            OFrame &f = st[sp++];
                            f.node = node;
                            f.next = q | (took << 4);
                            node = child;
                            YTGB_UNROLL
                            for (int i = 0; i < 3; i++) {
                                f.lost[i] = (took >> (2 - i)) & 1 ? t0[i] : t1[i];
                                t0[i] = c0[i];
                                t1[i] = c1[i];
                                tm[i] = midpoint<K>(c0[i], c1[i]);
                            }
                            q = first_node<K>(t0, tm);
                        }
                    }
                }
            }
        }
        meet(lanes);
        if (any_lane(lanes, found) == false) break;
        if (found) cell(key, t_in, t_out);
        meet(lanes);
    }
    return ok;
}

// x as two float32, hi its nearest (ties away from zero) and lo the rest
// rounded, from the bits of x (the conversions run on the float64 pipe), while
// both are normal; else by the conversions.
YTGB_HD void split_pair(double x, float &hi, float &lo) {
    const long long b = dbits(x);
    const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
    if (e - 949u <= 200u) {
        const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
        const unsigned long long m = (unsigned long long)b & 0x7fffffffffffffffull;
        hi = ffrom(sign | ((unsigned)((m + (1ull << 28)) >> 29) - (896u << 23)));
        const int rest = (int)((unsigned)b & 0x1fffffffu) - (int)(((unsigned)b & 0x10000000u) << 1);
        lo = fmul((float)rest, ffrom(sign | ((e - 948u) << 23)));
    } else {
        hi = (float)x;
        lo = (float)dsub(x, (double)hi);
    }
}

// (float)(x - y), the nearest float32 to the exact difference: for y <= x in
// one binade (inside the scaled conversion's range) as 24 + 24 bits of it,
// each exact as a float32, in one fma; else by float64.
YTGB_HD float diff_nearest(double x, double y) {
    const long long xb = dbits(x), yb = dbits(y), F = xb - yb;
    const unsigned ex = (unsigned)(xb >> 52);
    if (((xb ^ yb) >> 52) == 0 && F >= 0 && F < (1LL << 48) && ex - 949u <= 199u) {
        const float f = ffma((float)(int)(F >> 24), 16777216.0f, (float)(int)((unsigned)F & 0xffffffu));
        return fmul(f, ffrom((ex - 948u) << 23));
    }
    return (float)dsub(x, y);
}

// One pixel of cast_through_octree: the ray cast through the octree and
// each terminal cell handed to sample_cell as a 1x1x1 brick (dims 1, vertex
// strides 4 and 2, no mask, one field), with enter/exit t divided by the
// direction's length (image_samplers.pyx:245-283).  In MODE_TRACE it hashes
// (key, enter bits, exit bits) into th instead.  Returns false when the
// traversal gave up (malformed tree).
template <int MODE, int CTF>
YTGB_HD bool octree_ray(const ytgb_render_args &a, const OctreeView &o, const float4 *s_tab, const Ray &r,
                        RayState &st, unsigned long long &th, long long &tcount) {
    const double len = dsqrt(dadd(dadd(dmul(r.dir[0], r.dir[0]), dmul(r.dir[1], r.dir[1])), dmul(r.dir[2], r.dir[2])));
    // The sampler uses enter/exit t only through float32 quantities (dt and
    // the in-cell position), so a product with 1/len (within an ulp of the
    // quotient) serves it; the trace keeps the reference's exact quotients.
    const double ilen = ddiv(1.0, len);
    // the ray as float32 pairs (hi + lo = the float64 value to ~2^-48)
    float ph[3], pl[3], dh[3], dl[3];
    YTGB_UNROLL
    for (int i = 0; i < 3; i++) {
        split_pair(r.pos[i], ph[i], pl[i]);
        split_pair(r.dir[i], dh[i], dl[i]);
    }
    // the previous cell's exit t and what was formed from it: the next cell's
    // entry, where the ray goes from cell to cell.  Before the first cell: of
    // t = 0 (every t is a possible entry, so what stands here must be its own)
    double t_last = 0.0, x_last = dmul(0.0, ilen);
    float xh_last, xl_last;
    split_pair(x_last, xh_last, xl_last);
    return octree_cast(o, r.pos, r.dir, len, [&](int key, double t_in, double t_out) {
        if (key < 0 || key >= o.n_cells) {
            st.guarded++;
            return;
        }
        double e, x;
        float eh, el;
        if (MODE == MODE_TRACE) {
            e = ddiv(t_in, len);
            x = ddiv(t_out, len);
        } else {
            e = x_last;
            eh = xh_last;
            el = xl_last;
            if (dbits(t_in) != dbits(t_last)) {
                e = dmul(t_in, ilen);
                split_pair(e, eh, el);
            }
            x = dmul(t_out, ilen);
            split_pair(x, xh_last, xl_last);
            x_last = x;
            t_last = t_out;
        }
        if (MODE == MODE_TRACE) {
            th = fnv_mix(th, (unsigned long long)(unsigned)key);
            // a NaN (rays with zero direction components meet NaN slab
            // midpoints) enters the hash as one pattern: its sign and payload
            // differ between the GPU and CPUs
            th = fnv_mix(th, e != e ? 0x7ff8000000000000ull : (unsigned long long)dbits(e));
            th = fnv_mix(th, x != x ? 0x7ff8000000000000ull : (unsigned long long)dbits(x));
            tcount++;
            st.visits++;
            return;
        }
        CellCtx c;
        c.base = o.verts + 8ll * key;
        c.fstride = 0;
        c.moff = -1;
        c.nf = 1;
        c.sx = 4;
        c.sy = 2;
        c.tol = -1.0f;  // octree cells: float32 range decisions
        c.ray = nullptr;
        c.bp = nullptr;
        float P[3];
        if (o.edges_f) {
            // (enter * v_dir + v_pos - left_edge) * idds (image_samplers.pyx:
            // 475-478) in float32 pairs: the products exact by FMA, the sums
            // by TwoSum, so the difference keeps ~2^-48 of the operands' scale
            // (the cell is ~2^-9 of it), then one float32 rounding and the
            // float32 idds: within a float32 ulp or two of the float64 form,
            // on the float32 pipes rather than six float64 operations
            const float4 A = ldg(o.edges_f + 3ll * key), B = ldg(o.edges_f + 3ll * key + 1);
            const float4 D = ldg(o.edges_f + 3ll * key + 2);
            const float leh[3] = {A.x, A.y, A.z}, lel[3] = {A.w, B.x, B.y}, idf[3] = {B.z, B.w, D.x};
            YTGB_UNROLL
            for (int i = 0; i < 3; i++) {
                c.dims[i] = 1;
                c.vel[i] = fmul(r.fdir[i], idf[i]);
                const float mh = fmul(eh, dh[i]);
                float ml = ffma(eh, dh[i], -mh);
                ml = ffma(eh, dl[i], ml);
                ml = ffma(el, dh[i], ml);
                float sh, se, uh, ue;
                two_sum(mh, ph[i], sh, se);
                const float sl = fadd(fadd(se, ml), pl[i]);
                two_sum(sh, -leh[i], uh, ue);
                const float ul = fsub(fadd(ue, sl), lel[i]);
                P[i] = fmul(fadd(uh, ul), idf[i]);
            }
        } else {
            const double *ed = o.edges + 9ll * key;
            YTGB_UNROLL
            for (int i = 0; i < 3; i++) {
                c.dims[i] = 1;
                const double idds = ldg(ed + 6 + i);
                c.vel[i] = fmul(r.fdir[i], (float)idds);
                // (enter * v_dir + v_pos - left_edge) * idds (image_samplers.pyx:475-478)
                P[i] = (float)dmul(dsub(dadd(dmul(e, r.dir[i]), r.pos[i]), ldg(ed + i)), idds);
            }
        }
        const int cur[3] = {0, 0, 0};
        st.walks++;
        sample_cell<MODE, CTF, false>(a, s_tab, key, c, cur, P, diff_nearest(x, e), dbits(e), dbits(x), st);
    });
}

}  // namespace ytgb

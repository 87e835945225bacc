// ytgb_rects.cuh -- the bricks' pixel rectangles on the device, beside the
// render that reads them (included by ytgb_render.cu alone).
#pragma once

namespace {

// The pixel rectangle of each brick of an order (ytgb_brick_rects on the
// device: the same float64 and single-precision operations in the same order,
// not contracted, so the same integers): eight lanes per brick, one corner
// each.  1145 bricks take 4 us and no transfer back, against 0.4 ms on eight
// host threads between two launches.
constexpr int RECT_BLOCK = 128;
constexpr unsigned RECT_FRONT = 0x25469899u;

// calculate_extent_plane_parallel (lenses.pyx:22-55), one corner
__device__ __forceinline__ void corner_plane(const ytgb_view &im, const double v[3], double &tx, double &ty) {
    tx = ytgb::dadd(ytgb::dadd(ytgb::dmul(v[0], im.x_vec[0]), ytgb::dmul(v[1], im.x_vec[1])), ytgb::dmul(v[2], im.x_vec[2]));
    ty = ytgb::dadd(ytgb::dadd(ytgb::dmul(v[0], im.y_vec[0]), ytgb::dmul(v[1], im.y_vec[1])), ytgb::dmul(v[2], im.y_vec[2]));
}

__device__ __forceinline__ double dot3(const double a[3], const double *b) {
    return ytgb::dadd(ytgb::dadd(ytgb::dmul(a[0], b[0]), ytgb::dmul(a[1], b[1])), ytgb::dmul(a[2], b[2]));
}

// calculate_extent_perspective (lenses.pyx:60-161), one corner
__device__ __forceinline__ void corner_perspective(const ytgb_view &im, const double vertex[3], int &px, int &py) {
    const double *pos = im.camera_data, *east = im.camera_data + 6, *north = im.camera_data + 9,
                 *normal = im.camera_data + 12;
    const double w0 = im.camera_data[3], w2 = im.camera_data[5];
    const double w1 = ytgb::ddiv(ytgb::dmul(w0, (double)im.ny), (double)im.nx);
    double sight[3], q[3];
    for (int i = 0; i < 3; i++) sight[i] = ytgb::dsub(vertex[i], pos[i]);
    const float norm =
        (float)ytgb::dsqrt(ytgb::dadd(ytgb::dadd(ytgb::dmul(sight[0], sight[0]), ytgb::dmul(sight[1], sight[1])), ytgb::dmul(sight[2], sight[2])));
    if (norm != 0)
        for (int i = 0; i < 3; i++) sight[i] = ytgb::ddiv(sight[i], (double)norm);
    float c = (float)dot3(sight, normal);
    c = c > -1.0f ? c : -1.0f;
    c = c < 1.0f ? c : 1.0f;
    float length;
    // acos(c) < pi / 2 in float64: from this float on (below it acos rounds to pi / 2)
    if (c >= __uint_as_float(RECT_FRONT)) {
        length = (float)ytgb::ddiv(w2, (double)c);
    } else {
        length = (float)ytgb::dsqrt(ytgb::dadd(ytgb::dmul(w0, w0), ytgb::dmul(w1, w1)));
        length = (float)ytgb::ddiv((double)length, ytgb::dsqrt(ytgb::dsub(1.0, (double)ytgb::fmul(c, c))));
    }
    for (int i = 0; i < 3; i++) {
        const double centre = ytgb::dadd(ytgb::dmul(w2, normal[i]), pos[i]);
        q[i] = ytgb::dsub(ytgb::dadd(ytgb::dmul((double)length, sight[i]), pos[i]), centre);
    }
    const float dx = (float)dot3(q, east), dy = (float)dot3(q, north);
    px = (int)ytgb::dadd(ytgb::dmul((double)im.nx, 0.5), ytgb::dmul(ytgb::ddiv((double)im.nx, w0), (double)dx));
    py = (int)ytgb::dadd(ytgb::dmul((double)im.ny, 0.5), ytgb::dmul(ytgb::ddiv((double)im.ny, w1), (double)dy));
}

__device__ __forceinline__ int clip_pixel(long long v, int n) { return (int)(v < 0 ? 0 : (v > n ? n : v)); }

__global__ void __launch_bounds__(RECT_BLOCK)
brick_rects_kernel(const ytgb_view im, const ytgb_brick *bricks, int32_t n_bricks, const int32_t *order,
                   int32_t n_order, int4 *rects) {
    const int t = blockIdx.x * RECT_BLOCK + threadIdx.x, lane8 = t & 7;
    const int k = min(t >> 3, n_order - 1);  // (the last brick's lanes again past the end: shuffles are whole)
    const int b = order[k];
    const bool known = b >= 0 && b < n_bricks;
    const ytgb_brick &bk = bricks[known ? b : 0];
    // corner order of lenses.pyx does not matter: only extremes are kept
    const double v[3] = {lane8 & 1 ? bk.right_edge[0] : bk.left_edge[0], lane8 & 2 ? bk.right_edge[1] : bk.left_edge[1],
                         lane8 & 4 ? bk.right_edge[2] : bk.left_edge[2]};
    long long r0 = 0, r1 = im.nx, r2 = 0, r3 = im.ny;
    if (im.extent == YTGB_EXTENT_PLANE_PARALLEL) {
        double x0, y0;
        corner_plane(im, v, x0, y0);
        double x1 = x0, y1 = y0;
        for (int d = 1; d < 8; d <<= 1) {
            const double a = __shfl_xor_sync(0xffffffffu, x0, d), c = __shfl_xor_sync(0xffffffffu, x1, d);
            const double e = __shfl_xor_sync(0xffffffffu, y0, d), f = __shfl_xor_sync(0xffffffffu, y1, d);
            x0 = a < x0 ? a : x0;
            x1 = c > x1 ? c : x1;
            y0 = e < y0 ? e : y0;
            y1 = f > y1 ? f : y1;
        }
        double cx = 0.0, cy = 0.0;
        for (int i = 0; i < 3; i++) {
            cx = ytgb::dadd(cx, ytgb::dmul(im.center[i], im.x_vec[i]));
            cy = ytgb::dadd(cy, ytgb::dmul(im.center[i], im.y_vec[i]));
        }
        r0 = __double2ll_rn(ytgb::ddiv(ytgb::dsub(ytgb::dsub(x0, cx), im.bounds[0]), im.pdx));
        r1 = r0 + __double2ll_rn(ytgb::ddiv(ytgb::dsub(x1, x0), im.pdx));
        r2 = __double2ll_rn(ytgb::ddiv(ytgb::dsub(ytgb::dsub(y0, cy), im.bounds[2]), im.pdy));
        r3 = r2 + __double2ll_rn(ytgb::ddiv(ytgb::dsub(y1, y0), im.pdy));
    } else if (im.extent == YTGB_EXTENT_PERSPECTIVE) {
        int x0, y0;
        corner_perspective(im, v, x0, y0);
        int x1 = x0, y1 = y0;
        for (int d = 1; d < 8; d <<= 1) {
            x0 = min(x0, __shfl_xor_sync(0xffffffffu, x0, d));
            x1 = max(x1, __shfl_xor_sync(0xffffffffu, x1, d));
            y0 = min(y0, __shfl_xor_sync(0xffffffffu, y0, d));
            y1 = max(y1, __shfl_xor_sync(0xffffffffu, y1, d));
        }
        // the reference starts from +-SHRT_MAX
        r0 = max(min(x0, 32767), 0);
        r1 = min(max(x1, -32767), im.nx);
        r2 = max(min(y0, 32767), 0);
        r3 = min(max(y1, -32767), im.ny);
    }
    if (lane8 == 0 && (t >> 3) < n_order)
        rects[k] = known ? make_int4(clip_pixel(r0 - 1, im.nx), clip_pixel(r1 + 1, im.nx), clip_pixel(r2 - 1, im.ny),
                                     clip_pixel(r3 + 1, im.ny))
                         : make_int4(0, 0, 0, 0);
}

}  // namespace

extern "C" int ytgb_brick_rects_device(const ytgb_view *view, const ytgb_brick *d_bricks, int32_t n_bricks,
                                       const int32_t *d_order, int32_t n_order, int32_t *d_rects, void *stream) {
    if (!view || n_order < 0 || n_bricks < 0 || (n_order > 0 && (!d_bricks || !d_order || !d_rects || n_bricks == 0)) ||
        ((uintptr_t)d_bricks & 7) || ((uintptr_t)d_order & 3) || ((uintptr_t)d_rects & 15)) {
        ytgb_set_error("ytgb_brick_rects_device: null or misaligned argument, or bad sizes");
        return YTGB_ERR_INVALID;
    }
    if (view->nx <= 0 || view->ny <= 0) {
        ytgb_set_error("ytgb_brick_rects_device: empty image");
        return YTGB_ERR_INVALID;
    }
    if (n_order == 0) return YTGB_OK;
    const long long blocks = ((long long)n_order * 8 + RECT_BLOCK - 1) / RECT_BLOCK;
    if (n_order > (1 << 27)) {
        ytgb_set_error("ytgb_brick_rects_device: too many bricks");
        return YTGB_ERR_INVALID;
    }
    brick_rects_kernel<<<(unsigned)blocks, RECT_BLOCK, 0, (cudaStream_t)stream>>>(*view, d_bricks, n_bricks, d_order,
                                                                                 n_order, (int4 *)d_rects);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        ytgb_set_error(std::string("ytgb_brick_rects_device: ") + cudaGetErrorString(e));
        return YTGB_ERR_CUDA;
    }
    return YTGB_OK;
}

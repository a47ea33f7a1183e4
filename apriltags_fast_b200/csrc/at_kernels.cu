// The sm_100a kernels of the AprilTag detection path.
//
// Every kernel takes a batch of frames (FrameDesc array) and works on all
// of them at once: blockIdx.y is the frame, blockIdx.x strides over the
// frame's rows, pixels or items. Compiled with --fmad=false, -prec-div and
// -prec-sqrt: each floating point operation is rounded on its own, as the
// reference (built with -ffp-contract=off) rounds it, so the results are
// bit-identical. Each kernel names the reference lines it follows.
#include <cuda_runtime.h>
#include <stdint.h>

#include "at_gpu.h"
#include "at_device.cuh"
#include "at_kernels.h"
#include "at_launch.h"

// ---------------------------------------------------------------------------
// Small helpers.

// C's (int) of a double on x86-64: truncation, INT_MIN out of range or NaN
// (fast/decode.c:8-11).
__device__ __forceinline__ int64_t c_int(double x) {
    if (x > -2147483649.0 && x < 2147483648.0) return (int64_t)x;
    return -2147483648LL;
}

#define FRAME_LOOP_BEGIN(n_items)                                                               \
    const FrameDesc fd = frames[blockIdx.y];                                                   \
    for (int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; it < (n_items);          \
         it += (int64_t)gridDim.x * blockDim.x) {
#define FRAME_LOOP_END }

// ---------------------------------------------------------------------------
// 1. Decimation (fast/image.c:6-88). A block per output row, a thread per
// output pixel.

__global__ void k_decimate(const FrameDesc *frames, const uint8_t *img, uint8_t *qim, float factor) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const uint8_t *src = f.img;
    const int64_t stride = f.stride;
    const int qw = (int)f.qw, qh = (int)f.qh;
    for (int y = blockIdx.x; y < qh; y += gridDim.x) {
        uint8_t *out = qim + f.q_off + (int64_t)y * qw;
        if (factor == 1.5f) {
            // 3x3 weights over 9; output pixel (2k+dx, 2m+dy) from input
            // block (3k.., 3m..) (fast/image.c:50-62)
            const int m = y >> 1;
            const uint8_t *r0 = src + (int64_t)(3 * m) * stride, *r1 = r0 + stride, *r2 = r1 + stride;
            for (int x = threadIdx.x; x < qw; x += blockDim.x) {
                const int k3 = 3 * (x >> 1);
                const int e = r1[k3 + 1];
                int v;
                if ((y & 1) == 0)
                    v = (x & 1) == 0 ? 4 * r0[k3] + 2 * r0[k3 + 1] + 2 * r1[k3] + e
                                     : 4 * r0[k3 + 2] + 2 * r0[k3 + 1] + 2 * r1[k3 + 2] + e;
                else
                    v = (x & 1) == 0 ? 4 * r2[k3] + 2 * r1[k3] + 2 * r2[k3 + 1] + e
                                     : 4 * r2[k3 + 2] + 2 * r1[k3 + 2] + 2 * r2[k3 + 1] + e;
                out[x] = (uint8_t)(v / 9);
            }
        } else if (factor > 1.0f) {
            const int k = (int)factor;
            if (k == 2) {
                // 2x2 box; the part of the row below the largest multiple of
                // 32 rounds twice (the C library's AVX2 path), the rest once
                // (fast/image.c:26-46)
                const uint8_t *r0 = src + (int64_t)(2 * y) * stride, *r1 = r0 + stride;
                const int xv = qw - qw % 32;
                auto box = [&](int x, int a, int b, int c, int d) {
                    out[x] = x < xv ? (uint8_t)((((a + c + 1) >> 1) + ((b + d + 1) >> 1) + 1) >> 1)
                                    : (uint8_t)((a + b + c + d + 2) >> 2);
                };
                if ((((uintptr_t)r0 | (uintptr_t)r1) & 7) == 0) {
                    // four outputs a thread from 8-byte loads of both rows
                    for (int x4 = 4 * threadIdx.x; x4 < qw; x4 += 4 * blockDim.x) {
                        if (x4 + 3 < qw) {
                            const uint2 p = *reinterpret_cast<const uint2 *>(r0 + 2 * x4);
                            const uint2 q = *reinterpret_cast<const uint2 *>(r1 + 2 * x4);
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                const uint32_t pw = u < 2 ? p.x : p.y, qv = u < 2 ? q.x : q.y;
                                const int sh = 16 * (u & 1);
                                box(x4 + u, (pw >> sh) & 255, (pw >> (sh + 8)) & 255, (qv >> sh) & 255,
                                    (qv >> (sh + 8)) & 255);
                            }
                        } else {
                            for (int x = x4; x < qw; x++) box(x, r0[2 * x], r0[2 * x + 1], r1[2 * x], r1[2 * x + 1]);
                        }
                    }
                } else {
                    for (int x = threadIdx.x; x < qw; x += blockDim.x)
                        box(x, r0[2 * x], r0[2 * x + 1], r1[2 * x], r1[2 * x + 1]);
                }
            } else {
                const uint8_t *r0 = src + (int64_t)y * k * stride;
                for (int x = threadIdx.x; x < qw; x += blockDim.x) out[x] = r0[(int64_t)x * k];
            }
        } else {
            const uint8_t *r0 = src + (int64_t)y * stride;
            for (int x = threadIdx.x; x < qw; x += blockDim.x) out[x] = r0[x];
        }
    }
}

// ---------------------------------------------------------------------------
// 2. Blur / sharpen of the quad image (fast/image.c:93-173). The taps are
// integers made on the host. A separable pass: `dir` 0 filters rows, 1
// columns. The line's first nk/2 outputs and its tail copy the input; the
// wide variant (images of 65536 pixels or more) filters one more output.

__global__ void k_blur_pass(const FrameDesc *frames, const uint8_t *in, uint8_t *out, BlurTaps taps, int dir) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const int qw = (int)f.qw, qh = (int)f.qh;
    const bool wide = (int64_t)qw * qh >= 65536;
    const int nk = taps.n, r = nk / 2;
    const int len = dir == 0 ? qw : qh;
    const int m = wide ? len - nk + 1 : len - nk;
    const int64_t step = dir == 0 ? 1 : qw;
    for (int y = blockIdx.x; y < qh; y += gridDim.x) {
        for (int x = threadIdx.x; x < qw; x += blockDim.x) {
            const int pos = dir == 0 ? x : y;
            const uint8_t *line = in + f.q_off + (dir == 0 ? (int64_t)y * qw : (int64_t)x);
            uint8_t v;
            if (pos >= r && pos - r < m) {
                uint32_t acc = 0;
                for (int j = 0; j < nk; j++) acc += (uint32_t)taps.k[j] * line[(int64_t)(pos - r + j) * step];
                v = (uint8_t)(acc >> 8);
            } else {
                v = line[(int64_t)pos * step];
            }
            out[f.q_off + (int64_t)y * qw + x] = v;
        }
    }
}

// sharpen: im = clamp(2 * orig - blurred) (fast/image.c:484-489); else copy
__global__ void k_blur_finish(const FrameDesc *frames, const uint8_t *blurred, uint8_t *qim, int sharpen) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const int64_t n = (int64_t)f.qw * f.qh;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint8_t b = blurred[f.q_off + i];
        if (sharpen) {
            int v = 2 * (int)qim[f.q_off + i] - b;
            qim[f.q_off + i] = (uint8_t)(v < 0 ? 0 : v > 255 ? 255 : v);
        } else {
            qim[f.q_off + i] = b;
        }
    }
}

// ---------------------------------------------------------------------------
// 3. Adaptive threshold (fast/threshold.c:15-161). First each 4x4 tile's
// max and min, then per pixel the max and min of its tile's 3x3 tile
// neighbourhood (cells outside the grid left out).

__global__ void k_tile_minmax(const FrameDesc *frames, const uint8_t *qim, uint8_t *tmax, uint8_t *tmin) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const int64_t tw = f.qw / 4, th = f.qh / 4, n = tw * th;
    // 4-byte loads when every tile row is 4-byte aligned, else byte loads
    const bool al = (((uintptr_t)(qim + f.q_off)) & 3) == 0 && (f.qw & 3) == 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t ty = i / tw, tx = i - ty * tw;
        const uint8_t *p = qim + f.q_off + 4 * ty * f.qw + 4 * tx;
        uint32_t hi = 0, lo = 255;
        if (al) {
            uint32_t mx = 0, mn = 0xffffffffu;
#pragma unroll
            for (int dy = 0; dy < 4; dy++) {
                const uint32_t v = *reinterpret_cast<const uint32_t *>(p + dy * f.qw);
                mx = __vmaxu4(mx, v);
                mn = __vminu4(mn, v);
            }
            hi = max(max(mx & 255u, mx >> 8 & 255u), max(mx >> 16 & 255u, mx >> 24));
            lo = min(min(mn & 255u, mn >> 8 & 255u), min(mn >> 16 & 255u, mn >> 24));
        } else {
#pragma unroll
            for (int dy = 0; dy < 4; dy++) {
                const uint8_t *r = p + dy * f.qw;
                hi = max(hi, (uint32_t)max(max(r[0], r[1]), max(r[2], r[3])));
                lo = min(lo, (uint32_t)min(min(r[0], r[1]), min(r[2], r[3])));
            }
        }
        tmax[f.tile_off + i] = (uint8_t)hi;
        tmin[f.tile_off + i] = (uint8_t)lo;
    }
}

// The streaming stages fused for decimate 2 without blur (fast/image.c:26-46
// and fast/threshold.c:15-161 in one pass): a block takes a region of
// DT_ROWS x DT_COLS 4x4 cells of one frame. It reads the input rows of the
// region's tiles and of a one-tile halo around them (16-byte loads), makes
// each tile's 16 quad pixels in registers, keeps the region's own quad
// pixels and every tile's max/min in shared memory, then per cell the 3x3
// tile neighbourhood's max/min and per pixel the threshold, and writes the
// quad image and the threshold image once (16-byte stores). Cells right of
// the last whole tile column or below the last whole tile row (no tile of
// their own) use the nearest tile's neighbourhood and are never flat.
#define DT_ROWS 16
#define DT_COLS 64
#define DT_THREADS 256

// 2x2 box of the reference's decimate2_row: columns below the largest
// multiple of 32 round twice (its AVX2 path), the rest once.
__device__ __forceinline__ uint32_t box2(int x, int xv, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return x < xv ? ((((a + c + 1) >> 1) + ((b + d + 1) >> 1) + 1) >> 1) : ((a + b + c + d + 2) >> 2);
}

__global__ void __launch_bounds__(DT_THREADS) k_decimate_threshold(const FrameDesc *frames, uint8_t *qim, uint8_t *thr,
                                                                   int32_t diff) {
    kernel_begin();
    __shared__ __align__(16) uint8_t s_q[4 * DT_ROWS][4 * DT_COLS];
    __shared__ uint8_t s_tmax[DT_ROWS + 2][DT_COLS + 4], s_tmin[DT_ROWS + 2][DT_COLS + 4];
    __shared__ uint16_t s_cell[DT_ROWS][DT_COLS];  // threshold | flat << 8
    const FrameDesc f = frames[blockIdx.y];
    const int qw = f.qw, qh = f.qh, tw = qw / 4, th = qh / 4;
    const int cw = (qw + 3) / 4, ch = (qh + 3) / 4;
    const int ncb = (cw + DT_COLS - 1) / DT_COLS;
    const int rb = blockIdx.x / ncb, cb = blockIdx.x - rb * ncb;
    const int cy0 = rb * DT_ROWS, cx0 = cb * DT_COLS;
    if (cy0 >= ch) return;
    const int cy1 = min(cy0 + DT_ROWS, ch), cx1 = min(cx0 + DT_COLS, cw);  // own cells
    // tiles needed: the own cells' tiles (clamped to the grid) and one around
    const int ty0 = max(min(cy0, th - 1) - 1, 0), ty1 = min(min(cy1 - 1, th - 1) + 1, th - 1);
    const int tx0 = max(min(cx0, tw - 1) - 1, 0), tx1 = min(min(cx1 - 1, tw - 1) + 1, tw - 1);
    const int px0 = tx0 & ~1;  // tiles go in pairs (16 input bytes) from an even tile
    const int npair = (tx1 - px0) / 2 + 1, ntr = ty1 - ty0 + 1;
    const int xv = qw - qw % 32;
    const uint8_t *img = f.img;
    const int64_t st = f.stride;
    const bool al16 = ((((uintptr_t)img) | (uintptr_t)st) & 15) == 0;
    // 1. tiles: max/min of each, and the own tiles' quad pixels
    for (int i = threadIdx.x; i < npair * ntr; i += DT_THREADS) {
        const int r = i / npair, tp = px0 + 2 * (i - r * npair);
        const int ty = ty0 + r;
        uint32_t qw4[2][4];  // [tile][row]: the tile row's 4 quad pixels as bytes of a word
        if (al16 && tp + 1 < tw && 4 * tp + 8 <= xv) {
            // 16 input bytes of two rows give 8 quad pixels: the byte average
            // of the rows, then of even and odd columns (the reference's two
            // rounded averages of its AVX2 path)
#pragma unroll
            for (int dy = 0; dy < 4; dy++) {
                const uint8_t *r0 = img + (int64_t)(8 * ty + 2 * dy) * st + 8 * tp;
                const uint4 u = *reinterpret_cast<const uint4 *>(r0), v = *reinterpret_cast<const uint4 *>(r0 + st);
                const uint32_t a0 = __vavgu4(u.x, v.x), a1 = __vavgu4(u.y, v.y), a2 = __vavgu4(u.z, v.z),
                               a3 = __vavgu4(u.w, v.w);
                qw4[0][dy] = __vavgu4(__byte_perm(a0, a1, 0x6420), __byte_perm(a0, a1, 0x7531));
                qw4[1][dy] = __vavgu4(__byte_perm(a2, a3, 0x6420), __byte_perm(a2, a3, 0x7531));
            }
        } else {
#pragma unroll
            for (int dy = 0; dy < 4; dy++) {
                const uint8_t *r0 = img + (int64_t)(8 * ty + 2 * dy) * st + 8 * tp, *r1 = r0 + st;
                uint32_t a[4], b[4];  // 16 input bytes of each row, as words
                if (al16 && tp + 1 < tw) {
                    const uint4 u = *reinterpret_cast<const uint4 *>(r0), v = *reinterpret_cast<const uint4 *>(r1);
                    a[0] = u.x, a[1] = u.y, a[2] = u.z, a[3] = u.w;
                    b[0] = v.x, b[1] = v.y, b[2] = v.z, b[3] = v.w;
                } else {
                    const int nb = tp + 1 < tw ? 16 : 8;
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        a[w] = b[w] = 0;
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            if (4 * w + k < nb) {
                                a[w] |= (uint32_t)r0[4 * w + k] << (8 * k);
                                b[w] |= (uint32_t)r1[4 * w + k] << (8 * k);
                            }
                    }
                }
                qw4[0][dy] = qw4[1][dy] = 0;
#pragma unroll
                for (int o = 0; o < 8; o++) {  // quad pixel 4 tp + o of row 4 ty + dy
                    const uint32_t w0 = a[o >> 1], w1 = b[o >> 1];
                    const int sh = 16 * (o & 1);
                    qw4[o >> 2][dy] |= box2(4 * tp + o, xv, (w0 >> sh) & 255, (w0 >> (sh + 8)) & 255, (w1 >> sh) & 255,
                                            (w1 >> (sh + 8)) & 255)
                                       << (8 * (o & 3));
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int tx = tp + k;
            if (tx < tx0 || tx > tx1) continue;
            uint32_t mx = qw4[k][0], mn = qw4[k][0];
#pragma unroll
            for (int dy = 1; dy < 4; dy++) {
                mx = __vmaxu4(mx, qw4[k][dy]);
                mn = __vminu4(mn, qw4[k][dy]);
            }
            s_tmax[ty - ty0][tx - tx0] = (uint8_t)max(max(mx & 255u, mx >> 8 & 255u), max(mx >> 16 & 255u, mx >> 24));
            s_tmin[ty - ty0][tx - tx0] = (uint8_t)min(min(mn & 255u, mn >> 8 & 255u), min(mn >> 16 & 255u, mn >> 24));
            if (ty >= cy0 && ty < cy1 && tx >= cx0 && tx < cx1) {
#pragma unroll
                for (int dy = 0; dy < 4; dy++)
                    *reinterpret_cast<uint32_t *>(&s_q[4 * (ty - cy0) + dy][4 * (tx - cx0)]) = qw4[k][dy];
            }
        }
    }
    __syncthreads();
    // 2. per own cell: its tile's 3x3 neighbourhood (clipped to the grid)
    for (int i = threadIdx.x; i < (cy1 - cy0) * (cx1 - cx0); i += DT_THREADS) {
        const int cy = cy0 + i / (cx1 - cx0), cx = cx0 + i % (cx1 - cx0);
        const int ty = min(cy, th - 1), tx = min(cx, tw - 1);
        const bool may_flat = cy < th && cx < tw;
        uint32_t hi = 0, lo = 255;
        for (int yy = max(ty - 1, 0); yy <= min(ty + 1, th - 1); yy++)
            for (int xx = max(tx - 1, 0); xx <= min(tx + 1, tw - 1); xx++) {
                hi = max(hi, (uint32_t)s_tmax[yy - ty0][xx - tx0]);
                lo = min(lo, (uint32_t)s_tmin[yy - ty0][xx - tx0]);
            }
        const uint32_t t = lo + (hi - lo) / 2;
        const bool flat = may_flat && (int32_t)(hi - lo) < diff;
        s_cell[cy - cy0][cx - cx0] = (uint16_t)(t | (flat ? 256u : 0u));
    }
    __syncthreads();
    // 3. the own pixels, 16 a thread: quad image and threshold image
    const int y0 = 4 * cy0, y1 = min(4 * cy1, qh), x0 = 4 * cx0, x1 = min(4 * cx1, qw);
    const int nseg = (x1 - x0 + 15) / 16;
    const bool st16 = ((((uintptr_t)(qim + f.q_off)) | ((uintptr_t)(thr + f.q_off)) | (uintptr_t)qw) & 15) == 0;
    for (int i = threadIdx.x; i < (y1 - y0) * nseg; i += DT_THREADS) {
        const int y = y0 + i / nseg, xs = x0 + 16 * (i % nseg);
        const int n = min(16, x1 - xs);
        const bool whole_tiles = y < 4 * th;
        if (st16 && n == 16 && whole_tiles && xs + 16 <= 4 * tw) {
            // 16 pixels of 4 cells, 4 at a time: above the cell's threshold
            // 255, else 0; a flat cell 127
            const uint4 q = *reinterpret_cast<const uint4 *>(&s_q[y - y0][xs - x0]);
            const uint32_t qa[4] = {q.x, q.y, q.z, q.w};
            uint32_t t4[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t c = s_cell[(y >> 2) - cy0][(xs >> 2) - cx0 + k];
                t4[k] = (c & 256u) ? 0x7f7f7f7fu : __vcmpgtu4(qa[k], (c & 255u) * 0x01010101u);
            }
            const int64_t o = f.q_off + (int64_t)y * qw + xs;
            *reinterpret_cast<uint4 *>(qim + o) = q;
            *reinterpret_cast<uint4 *>(thr + o) = make_uint4(t4[0], t4[1], t4[2], t4[3]);
            continue;
        }
        uint32_t qv[4] = {0, 0, 0, 0}, tv[4] = {0, 0, 0, 0};
#pragma unroll
        for (int o = 0; o < 16; o++) {
            if (o >= n) break;
            const int x = xs + o;
            uint32_t v;
            if (whole_tiles && x < 4 * tw) {
                v = s_q[y - y0][x - x0];
            } else {  // a pixel of no tile: decimated here
                const uint8_t *r0 = img + (int64_t)(2 * y) * st + 2 * x, *r1 = r0 + st;
                v = box2(x, xv, r0[0], r0[1], r1[0], r1[1]);
            }
            const uint32_t c = s_cell[(y >> 2) - cy0][(x >> 2) - cx0];
            const uint32_t tb = (c & 256u) ? 127u : (v > (c & 255u) ? 255u : 0u);
            qv[o >> 2] |= v << (8 * (o & 3));
            tv[o >> 2] |= tb << (8 * (o & 3));
        }
        const int64_t o = f.q_off + (int64_t)y * qw + xs;
        if (st16 && n == 16) {
            *reinterpret_cast<uint4 *>(qim + o) = make_uint4(qv[0], qv[1], qv[2], qv[3]);
            *reinterpret_cast<uint4 *>(thr + o) = make_uint4(tv[0], tv[1], tv[2], tv[3]);
        } else {
            for (int k = 0; k < n; k++) {
                qim[o + k] = (uint8_t)(qv[k >> 2] >> (8 * (k & 3)));
                thr[o + k] = (uint8_t)(tv[k >> 2] >> (8 * (k & 3)));
            }
        }
    }
}

// A thread per 4x4 tile: the max and min of its 3x3 tile neighbourhood
// (cells outside the grid left out) once, then its 16 pixels. Pixels right
// of the last whole tile column use that column and are never 127; rows
// below the last whole tile row use that row and are never 127
// (fast/threshold.c:85-91, 144-148): the partial tiles there clamp.
__global__ void k_threshold(const FrameDesc *frames, const uint8_t *qim, const uint8_t *tmax, const uint8_t *tmin,
                            uint8_t *thr, int32_t diff) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const int qw = (int)f.qw, qh = (int)f.qh;
    const int tw = qw / 4, th = qh / 4, cw = (qw + 3) / 4, ch = (qh + 3) / 4;
    const int n = cw * ch;
    const uint8_t *tx_max = tmax + f.tile_off, *tx_min = tmin + f.tile_off;
    const bool al = ((((uintptr_t)(qim + f.q_off)) | ((uintptr_t)(thr + f.q_off))) & 3) == 0 && (qw & 3) == 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int cy = i / cw, cx = i - cy * cw;
        int ty = cy, tx = cx;
        bool may_flat = true;
        if (ty >= th) {
            ty = th - 1;
            may_flat = false;
        }
        if (tx >= tw) {
            tx = tw - 1;
            may_flat = false;
        }
        uint32_t hi = 0, lo = 255;
        const int y0t = ty - 1 > 0 ? ty - 1 : 0, y1t = ty + 1 < th - 1 ? ty + 1 : th - 1;
        const int x0t = tx - 1 > 0 ? tx - 1 : 0, x1t = tx + 1 < tw - 1 ? tx + 1 : tw - 1;
        for (int yy = y0t; yy <= y1t; yy++)
            for (int xx = x0t; xx <= x1t; xx++) {
                hi = max(hi, (uint32_t)tx_max[yy * tw + xx]);
                lo = min(lo, (uint32_t)tx_min[yy * tw + xx]);
            }
        const uint32_t t = lo + (hi - lo) / 2;
        const bool flat = may_flat && (int32_t)(hi - lo) < diff;
        const int x0 = 4 * cx, y0 = 4 * cy;
        const int xe = x0 + 4 < qw ? x0 + 4 : qw, ye = y0 + 4 < qh ? y0 + 4 : qh;
        if (al && xe == x0 + 4) {
            // a whole tile row at a time: per byte 255 above t, else 0
            const uint32_t t4 = t * 0x01010101u;
            for (int y = y0; y < ye; y++) {
                const int64_t o = f.q_off + (int64_t)y * qw + x0;
                const uint32_t v = *reinterpret_cast<const uint32_t *>(qim + o);
                *reinterpret_cast<uint32_t *>(thr + o) = flat ? 0x7f7f7f7fu : __vcmpgtu4(v, t4);
            }
        } else {
            for (int y = y0; y < ye; y++) {
                const int64_t o = f.q_off + (int64_t)y * qw;
                for (int x = x0; x < xe; x++) thr[o + x] = flat ? 127 : (qim[o + x] > t ? 255 : 0);
            }
        }
    }
}

// Deglitch (fast/threshold.c:173-193): 3x3 dilate into tmp (its border
// zero), then 3x3 erode back; the image border keeps its values.
__global__ void k_morph(const FrameDesc *frames, const uint8_t *in, uint8_t *out, int dilate) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const int qw = (int)f.qw, qh = (int)f.qh;
    for (int y = blockIdx.x; y < qh; y += gridDim.x) {
        const int64_t row = f.q_off + (int64_t)y * qw;
        for (int x = threadIdx.x; x < qw; x += blockDim.x) {
            const bool border = x == 0 || y == 0 || x == qw - 1 || y == qh - 1;
            if (border) {
                if (dilate) out[row + x] = 0;
                continue;
            }
            uint32_t m = dilate ? 0 : 255;
            for (int dy = -1; dy <= 1; dy++)
                for (int dx = -1; dx <= 1; dx++) {
                    const uint32_t v = in[row + (int64_t)dy * qw + x + dx];
                    m = dilate ? max(m, v) : min(m, v);
                }
            out[row + x] = (uint8_t)m;
        }
    }
}

// ---------------------------------------------------------------------------
// 6. Boundary points (fast/clusters.c:144-252). Pixel (x, y), y in
// 1..qh-2, against (1,0), (0,1), (-1,1), (1,1): a point where one pixel is
// 0 and the other 255 and both labels are not AT_NOK. The (-1,1) point is
// left out when the pixel to the left gave its (1,1) point, except at x=1;
// x = 0 gives only (1,0) (point_mask). Points are emitted in (y, x,
// neighbour) order.

// Block-per-row forms of the point passes (a block scan per 256 columns),
// for batches too small to fill the GPU with a warp per row.
__global__ void k_point_count_block(const FrameDesc *frames, const uint8_t *thr, const uint32_t *lab, uint64_t *row_npts) {
    kernel_begin();
    __shared__ uint32_t sh[32];
    const FrameDesc f = frames[blockIdx.y];
    for (int64_t y = blockIdx.x; y < f.qh; y += gridDim.x) {
        uint32_t cnt = 0;
        if (y >= 1 && y + 1 < f.qh) {
            const uint8_t *a = thr + f.q_off + y * f.qw, *b = a + f.qw;
            const uint32_t *la = lab + f.q_off + y * f.qw, *lb = la + f.qw;
            for (int64_t x = threadIdx.x; x < f.qw; x += blockDim.x) cnt += __popc(point_mask(a, b, la, lb, x, f.qw));
        }
        uint32_t total;
        block_excl_scan(cnt, &total, sh);
        if (threadIdx.x == 0) row_npts[f.row0 + y] = total;
    }
}

__global__ void k_point_emit_block(const FrameDesc *frames, const uint8_t *thr, const uint32_t *lab,
                             const uint64_t *row_pt_off, uint64_t *pt_key, uint64_t *pt_val, int nb) {
    kernel_begin();
    __shared__ uint32_t sh[32];
    const FrameDesc f = frames[blockIdx.y];
    for (int64_t y = 1 + blockIdx.x; y + 1 < f.qh; y += gridDim.x) {
        const uint8_t *a = thr + f.q_off + y * f.qw, *b = a + f.qw;
        const uint32_t *la = lab + f.q_off + y * f.qw, *lb = la + f.qw;
        uint64_t out = row_pt_off[f.row0 + y];
        for (int64_t x0 = 0; x0 < f.qw; x0 += blockDim.x) {
            int64_t x = x0 + threadIdx.x;
            uint32_t m = x < f.qw ? point_mask(a, b, la, lb, x, f.qw) : 0u;
            uint32_t total;
            uint32_t off = block_excl_scan(__popc(m), &total, sh);
            uint64_t o = out + off;
            int g = a[x < f.qw ? x : 0] == 0 ? 255 : -255;
            for (int j = 0; j < 4; j++) {
                if (!(m >> j & 1u)) continue;
                int dx = j == 0 || j == 3 ? 1 : j == 2 ? -1 : 0;
                int dy = j == 0 ? 0 : 1;
                uint32_t l0 = la[x], l1 = dy ? lb[x + dx] : la[x + dx];
                uint64_t hi = l0 > l1 ? l0 : l1, lo = l0 > l1 ? l1 : l0;
                uint64_t px = (uint64_t)(2 * x + dx), py = (uint64_t)(2 * y + dy);
                uint64_t gx = (uint16_t)(int16_t)(dx * g), gy = (uint16_t)(int16_t)(dy * g);
                pt_key[o] = hi << nb | lo;
                pt_val[o] = px | py << 16 | gx << 32 | gy << 48;
                o++;
            }
            out += total;
        }
    }
}

// A warp per row for both passes: the row's points counted, then emitted
// in (x, neighbour) order at the row's offset (warp scans, no block
// barriers).

__global__ void __launch_bounds__(256) k_point_count(const FrameDesc *frames, const uint8_t *thr,
                                                     const uint32_t *lab, uint64_t *row_npts) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const int lane = threadIdx.x & 31;
    const int64_t wpb = blockDim.x >> 5;
    for (int64_t y = blockIdx.x * wpb + (threadIdx.x >> 5); y < f.qh; y += gridDim.x * wpb) {
        uint32_t cnt = 0;
        if (y >= 1 && y + 1 < f.qh) {
            const uint8_t *a = thr + f.q_off + y * f.qw, *b = a + f.qw;
            const uint32_t *la = lab + f.q_off + y * f.qw, *lb = la + f.qw;
            for (int64_t x = lane; x < f.qw; x += 32) cnt += __popc(point_mask(a, b, la, lb, x, f.qw));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0) row_npts[f.row0 + y] = cnt;
    }
}

// The cluster key of a point: (larger label, smaller label) packed as
// larger << nb | smaller, nb = bits of the largest node id.
__global__ void __launch_bounds__(256) k_point_emit(const FrameDesc *frames, const uint8_t *thr,
                                                    const uint32_t *lab, const uint64_t *row_pt_off,
                                                    uint64_t *pt_key, uint64_t *pt_val, int nb) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const int lane = threadIdx.x & 31;
    const int64_t wpb = blockDim.x >> 5;
    for (int64_t y = 1 + blockIdx.x * wpb + (threadIdx.x >> 5); y + 1 < f.qh; y += gridDim.x * wpb) {
        const uint8_t *a = thr + f.q_off + y * f.qw, *b = a + f.qw;
        const uint32_t *la = lab + f.q_off + y * f.qw, *lb = la + f.qw;
        uint64_t out = row_pt_off[f.row0 + y];
        for (int64_t x0 = 0; x0 < f.qw; x0 += 32) {
            const int64_t x = x0 + lane;
            const uint32_t m = x < f.qw ? point_mask(a, b, la, lb, x, f.qw) : 0u;
            uint32_t total;
            const uint32_t off = warp_excl_scan(__popc(m), &total);
            uint64_t o = out + off;
            const int g = a[x < f.qw ? x : 0] == 0 ? 255 : -255;
            for (int j = 0; j < 4; j++) {
                if (!(m >> j & 1u)) continue;
                const int dx = j == 0 || j == 3 ? 1 : j == 2 ? -1 : 0;
                const int dy = j == 0 ? 0 : 1;
                const uint32_t l0 = la[x], l1 = dy ? lb[x + dx] : la[x + dx];
                const uint64_t hi = l0 > l1 ? l0 : l1, lo = l0 > l1 ? l1 : l0;
                const uint64_t px = (uint64_t)(2 * x + dx), py = (uint64_t)(2 * y + dy);
                const uint64_t gx = (uint16_t)(int16_t)(dx * g), gy = (uint16_t)(int16_t)(dy * g);
                pt_key[o] = hi << nb | lo;
                pt_val[o] = px | py << 16 | gx << 32 | gy << 48;
                o++;
            }
            out += total;
        }
    }
}

// ---------------------------------------------------------------------------
// 7. Clusters (fast/clusters.c:16-66, 318-382). The pair table and the
// placing of the points are in at_cluster.cu; here the distinct pairs of
// the table, and the fallback when the table overflows.

// The occupied slots, in no particular order: (pair, slot).
__global__ void k_cluster_collect(const uint64_t *tkeys, uint32_t size, uint64_t *okeys, uint32_t *oslots,
                                  uint32_t *count) {
    kernel_begin();
    const int lane = threadIdx.x & 31;
    for (uint32_t s0 = blockIdx.x * blockDim.x; s0 < size; s0 += gridDim.x * blockDim.x) {
        const uint32_t s = s0 + threadIdx.x;
        const uint64_t k = s < size ? tkeys[s] : CH_EMPTY;
        const bool occ = k != CH_EMPTY;
        const uint32_t bal = __ballot_sync(0xffffffffu, occ);
        if (!bal) continue;
        uint32_t at = 0;
        if (lane == __ffs(bal) - 1) at = atomicAdd(count, (uint32_t)__popc(bal));
        at = __shfl_sync(0xffffffffu, at, __ffs(bal) - 1) + __popc(bal & ((1u << lane) - 1u));
        if (occ) {
            okeys[at] = k;
            oslots[at] = s;
        }
    }
}

// ---------------------------------------------------------------------------
// 7b. Clusters by the full sort (the fallback): after the stable sort by
// key, each run of equal keys is a cluster (points in emission order).

__global__ void k_cluster_heads(const uint64_t *key, int64_t n, uint32_t *head) {
    kernel_begin();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        head[i] = i == 0 || key[i] != key[i - 1];
}

__global__ void k_cluster_starts(const uint64_t *key, const uint32_t *head, const uint32_t *head_scan, int64_t n,
                                 int nb, const FrameDesc *frames, int nframes, uint32_t *cstart, int32_t *cframe,
                                 uint64_t *ckey) {
    kernel_begin();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (!head[i]) continue;
        uint32_t c = head_scan[i];
        cstart[c] = (uint32_t)i;
        ckey[c] = key[i];
        int64_t node = (int64_t)(key[i] >> nb);
        int lo = 0, hi = nframes - 1;  // the frame whose node range holds node
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (frames[mid].node_off <= node)
                lo = mid;
            else
                hi = mid - 1;
        }
        cframe[c] = lo;
    }
}

// ---------------------------------------------------------------------------
// 8. Quad fitting, one block per cluster (fast/quads.c:429-1160).

__device__ __forceinline__ uint32_t f32_bits(float f) { return __float_as_uint(f); }

// The angle key (fast/quads.c:429-453): quadrant + slope in f32, as
// order-preserving bits, above the complemented point index.
__device__ __forceinline__ uint64_t angle_key(float dx, float dy, uint32_t idx) {
    float quadrant = dy > 0.0f ? (dx > 0.0f ? 65536.0f : 131072.0f) : (dx > 0.0f ? 0.0f : -65536.0f);
    float fx = dx, fy = dy;
    if (dy < 0.0f) {
        fx = __uint_as_float(f32_bits(dx) ^ 0x80000000u);
        fy = __uint_as_float(f32_bits(dy) ^ 0x80000000u);
    }
    float ndx = fx, ndy = fy;
    if (fx < 0.0f) {
        ndx = fy;
        ndy = -fx;
    }
    float slope = __fadd_rn(quadrant, __fdiv_rn(ndy, ndx));
    uint32_t b = f32_bits(slope);
    uint32_t s = (uint32_t)((int32_t)b >> 31);
    return (uint64_t)(b ^ (s | 0x80000000u)) << 32 | (uint32_t)~idx;
}

// The leaf [lo, lo + len) of the reference's angle sort that holds position p
// of n (fast/quads.c:181-237): cut in four while half the range has more than
// 5 keys, then in two down to 5 or fewer.
__device__ __forceinline__ void leaf_of(int n, int p, int &lo, int &len) {
    int l = 0, sz = n;
    while (sz / 2 > 5) {
        const int half = sz / 2, q1 = half / 2, q3 = half + (sz - half) / 2;
        const int r = p - l;
        if (r < q1) {
            sz = q1;
        } else if (r < half) {
            l += q1;
            sz = half - q1;
        } else if (r < q3) {
            l += half;
            sz = q3 - half;
        } else {
            l += q3;
            sz = sz - q3;
        }
    }
    while (sz > 5) {
        const int half = sz / 2;
        if (p - l >= half) {
            l += half;
            sz -= half;
        } else {
            sz = half;
        }
    }
    lo = l;
    len = sz;
}

// The leaf networks of the reference (fast/quads.c:56-85): compare-exchange
// on the upper 32 bits only.
__device__ __forceinline__ void leaf_network(uint64_t *k, int n) {
#define CX(a, b)                                      \
    if ((k[a] >> 32) > (k[b] >> 32)) {                \
        uint64_t t_ = k[a];                           \
        k[a] = k[b];                                  \
        k[b] = t_;                                    \
    }
    if (n == 2) {
        CX(0, 1)
    } else if (n == 3) {
        CX(0, 1) CX(1, 2) CX(0, 1)
    } else if (n == 4) {
        CX(0, 1) CX(2, 3) CX(0, 2) CX(1, 3) CX(1, 2)
    } else if (n == 5) {
        CX(0, 1) CX(3, 4) CX(1, 2) CX(0, 1) CX(0, 3) CX(2, 4) CX(1, 2) CX(2, 3) CX(1, 2)
    }
#undef CX
}


// The six moment terms of a point (fast/quads.c:968-1035): w =
// sqrt(gx^2 + gy^2) + 1 on the quad image (1 at its border), fx = x / 2 +
// 1 / 2, the reference's products. g2: the squared gradient at pt.
__device__ __forceinline__ int32_t point_grad2(const uint8_t *im, int qw, int qh, uint64_t pt) {
    const int32_t px = (int32_t)(pt & 0xffff), py = (int32_t)(pt >> 16 & 0xffff);
    const int32_t ix = (px >> 1) + (px & 1), iy = (py >> 1) + (py & 1);
    if (ix <= 0 || ix + 1 >= qw || iy <= 0 || iy + 1 >= qh) return 0;
    const int64_t cc = (int64_t)iy * qw + ix;
    const int32_t gx = (int32_t)im[cc + 1] - im[cc - 1];
    const int32_t gy = (int32_t)im[cc + qw] - im[cc - qw];
    return gx * gx + gy * gy;
}
__device__ __forceinline__ void moment_terms(uint64_t pt, int32_t g2, double m[6]) {
    const int32_t px = (int32_t)(pt & 0xffff), py = (int32_t)(pt >> 16 & 0xffff);
    const double w = __dadd_rn(__dsqrt_rn((double)g2), 1.0);
    const double fx = __dadd_rn(__dmul_rn((double)px, 0.5), 0.5);
    const double fy = __dadd_rn(__dmul_rn((double)py, 0.5), 0.5);
    const double wx = __dmul_rn(w, fx), wy = __dmul_rn(w, fy);
    m[0] = wx;
    m[1] = wy;
    m[2] = __dmul_rn(wx, fx);
    m[3] = __dmul_rn(wx, fy);
    m[4] = __dmul_rn(wy, fy);
    m[5] = w;
}

// The prefix sums of src[0, n) in place (16-byte aligned), after `run`, one
// lane: a chain of dependent additions, 8.4 cycles each. The next 8 terms are
// loaded, and the sums stored, two at a time between the additions: 9.4
// cycles a term, where eight loads, eight additions and eight stores in turn
// took 12.5 (the chain stood still while the loads and stores issued).
__device__ __forceinline__ void prefix_chain(double *src, int n, double &run) {
    int t = 0;
    if (n >= 8) {
        double2 *p = reinterpret_cast<double2 *>(src), v[4], r;
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = p[u];
        for (; t + 16 <= n; t += 8, p += 4) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                r.x = __dadd_rn(run, v[u].x);
                r.y = __dadd_rn(r.x, v[u].y);
                v[u] = p[4 + u];
                run = r.y;
                p[u] = r;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            r.x = __dadd_rn(run, v[u].x);
            r.y = __dadd_rn(r.x, v[u].y);
            run = r.y;
            p[u] = r;
        }
        t += 8;
    }
    for (; t < n; t++) {
        run = __dadd_rn(run, src[t]);
        src[t] = run;
    }
}

struct MSum {
    double x, y, xx, xy, yy, w;
};

struct Moments {
    const double *mx, *my, *mxx, *mxy, *myy, *mw;
};

__device__ __forceinline__ MSum moments_at(const Moments &a, int64_t i) {
    return {a.mx[i], a.my[i], a.mxx[i], a.mxy[i], a.myy[i], a.mw[i]};
}

// Moments of sorted points i0..i1, wrapping past the end, summed in the
// reference's forms (fast/quads.c:539-569, 658-700, 885-921); `all`: the
// moments of all points. One path for all cases, as code size is time here.
__device__ __forceinline__ MSum seg_moments(const Moments &a, const MSum &all, int64_t i0, int64_t i1) {
    const MSum q = moments_at(a, i1);
    MSum p = moments_at(a, i0 > 0 ? i0 - 1 : 0);
    if (i0 <= 0) p = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // q - 0 is q
    if (i0 <= i1) return {q.x - p.x, q.y - p.y, q.xx - p.xx, q.xy - p.xy, q.yy - p.yy, q.w - p.w};
    return {(all.x - p.x) + q.x,    (all.y - p.y) + q.y,    (all.xx - p.xx) + q.xx,
            (all.xy - p.xy) + q.xy, (all.yy - p.yy) + q.yy, (all.w - p.w) + q.w};
}

// The moments of the window of 2 ksz + 1 points centred on i, wrapping
// around the ends (fast/quads.c:797-808).
template <typename I>
__device__ __forceinline__ MSum window_moments(const Moments &a, const MSum &all, I sz, I ksz, I i) {
    const I i0 = i - ksz, i1 = i + ksz;
    return seg_moments(a, all, i0 < 0 ? i0 + sz : i0, i1 >= sz ? i1 - sz : i1);
}

// The smoothed error at i (fast/quads.c:809-826): the 7-tap filter over
// errs, wrapping around the ends; the sum in tap order.
template <typename I>
__device__ __forceinline__ double smooth_at(const double *e, I n, I i, const double *q) {
    double acc;
    if (i >= 3 && i < n - 3) {
        acc = e[i - 3] * q[0];
        for (int t = 1; t < 7; t++) acc = acc + e[i - 3 + t] * q[t];
    } else {
        acc = 0.0;
        for (int t = 0; t < 7; t++) {
            I j = i - 3 + t;
            if (j < 0) j += n;
            if (j >= n) j -= n;
            acc = acc + e[j] * q[t];
        }
    }
    return acc;
}

// Centroid and covariance of the moments (fast/quads.c:570-600, 604-653).
struct MCov {
    double ex, ey, xx, xy, yy;
};
__device__ __forceinline__ MCov moments_cov(const MSum &s) {
    const double r = __drcp_rn(s.w);
    const double ex = div_by(s.x, s.w, r), ey = div_by(s.y, s.w, r);
    return {ex, ey, div_by(s.xx, s.w, r) - ex * ex, div_by(s.xy, s.w, r) - ex * ey, div_by(s.yy, s.w, r) - ey * ey};
}

// The error of a window of nn points (fast/quads.c:604-653).
__device__ __forceinline__ double window_error(const MSum &s, double nn) {
    const MCov c = moments_cov(s);
    const double d = c.xx - c.yy;
    const double root = (double)__fsqrt_rn((float)(d * d + 4.0 * (c.xy * c.xy)));
    return nn * (0.5 * (c.xx + c.yy - root));
}

// The line of the moments: centroid, unit normal, smaller eigenvalue
// (fast/quads.c:570-600, 756-783).
__device__ __forceinline__ void line_of(const MSum &s, double lp[4], double *mse) {
    const MCov c = moments_cov(s);
    const double ex = c.ex, ey = c.ey, cxx = c.xx, cxy = c.xy, cyy = c.yy;
    double root = (double)__fsqrt_rn((float)((cxx - cyy) * (cxx - cyy) + 4.0 * cxy * cxy));
    double eig_small = 0.5 * (cxx + cyy - root);
    double eig = 0.5 * (cxx + cyy + root);
    double nx1 = cxx - eig, ny1 = cxy, m1 = nx1 * nx1 + ny1 * ny1;
    double nx2 = cxy, ny2 = cyy - eig, m2 = nx2 * nx2 + ny2 * ny2;
    double nx = nx2, ny = ny2, m = m2;
    if (m1 > m2) {
        nx = nx1;
        ny = ny1;
        m = m1;
    }
    double len = (double)__fsqrt_rn((float)m);
    lp[0] = ex;
    lp[1] = ey;
    lp[2] = 0.0;
    lp[3] = 0.0;
    if (!(fabs(len) < 1e-12)) {
        lp[2] = nx / len;
        lp[3] = ny / len;
    }
    *mse = eig_small;
}

// A double's place among doubles (no NaN; both zeros are one).
__device__ __forceinline__ uint64_t double_order(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x + 0.0);
    return b >> 63 ? ~b : b | 1ull << 63;
}

// A v such that what is above the (r + 1)-th largest of e[0, n) (r < n) has
// a place >= v and the rest has not. By the whole block: the places from the
// least to the largest are halved, one barrier a step (as many pivots at a
// time as there are warps took 3000 cycles longer with 8 of them).
template <int NT>
__device__ uint64_t block_above(const double *e, int n, int r, uint64_t *part) {
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t lo = ~0ull, hi = 0;
    for (int i = threadIdx.x; i < n; i += NT) {
        const uint64_t k = double_order(e[i]);
        lo = k < lo ? k : lo;
        hi = k > hi ? k : hi;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t l = __shfl_xor_sync(0xffffffffu, lo, o), h = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = l < lo ? l : lo;
        hi = h > hi ? h : hi;
    }
    if (lane == 0) {
        part[w] = lo;
        part[NW + w] = hi;
    }
    __syncthreads();
    for (int v = 0; v < NW; v++) {
        lo = part[v] < lo ? part[v] : lo;
        hi = part[NW + v] > hi ? part[NW + v] : hi;
    }
    hi++;  // more than r have a place >= lo, at most r one >= hi
    for (int step = 0; hi - lo > 1; step++) {
        const uint64_t mid = lo + (hi - lo) / 2;
        int c = 0;
        for (int i = threadIdx.x; i < n; i += NT) c += double_order(e[i]) >= mid;
        c = __reduce_add_sync(0xffffffffu, c);
        // two halves in turn: nobody still reads the one before the last
        int *cnt = reinterpret_cast<int *>(part + 2 * NW) + (step & 1) * NW;
        if (lane == 0) cnt[w] = c;
        __syncthreads();
        c = 0;
        for (int v = 0; v < NW; v++) c += cnt[v];
        if (c > r)
            lo = mid;
        else
            hi = mid;
        if (c == r) break;
    }
    return hi;
}

// Three size classes of clusters, one kernel template: 128 threads for
// clusters of at most FIT_SMALL points, FIT_LARGE_NT threads, two blocks an
// SM, up to FIT_LARGE_SORT, FIT_HUGE_NT threads, one block an SM, above. The
// last sorts in shared memory up to FIT_HUGE_SORT points and in global
// scratch beyond (the same radix sort). Clusters above 6144 points come only
// from quad images above about 1080p (a cluster has at most 4 (qw + qh)
// points); a merge sort in global memory, with the blocks of the class
// below, took 1.4M cycles for 9000 points and 3.9M for 21000.
#define FIT_SMALL 1024
#define FIT_LARGE_SORT 6144
#define FIT_HUGE_SORT 13312
#define FIT_HUGE_NT 512
#define FIT_CHUNK_SMALL 256
// Clusters of 257-512 points: a warp each when there are more than this many
// of them, a block of 128 when not. A block is done in half the time (49000
// instead of 87000 cycles), but keeps four warps for it: 643 of them (eight
// 1280 x 720 frames) take the fit stage 131 us in blocks and 151 in warps, 25
// (640 x 480) 79 and 89; 3592 (4032 x 3024) 941 and 849, 4338 (32 frames of
// 1920 x 1080) 606 and 525. The line is two waves of the blocks (4 an SM).
#define FIT_FEW (2 * 4 * 148)
#define FIT_CHUNK_LARGE 512
#define FIT_LARGE_NT 256  // threads of the largest class's blocks (two blocks an SM)

// dynamic shared memory of one block of the fit kernel
// Shared memory of the block fit kernel for clusters of up to sort_cap
// points: region X (the angle keys; then the radix sort's second buffers;
// then the staged moment terms of a chunk of points), the sort keys (4 B)
// and point indices (2 B), and the radix histograms (256 per warp). The
// moment terms take two chunks of six rows of chunk + 2 doubles (the pad
// puts the six rows that one warp walks in step on distinct banks).
__host__ __device__ constexpr size_t fit_x_bytes(int sort_cap, int chunk) {
    return (size_t)sort_cap * 8 > (size_t)(chunk + 2) * 96 ? (size_t)sort_cap * 8 : (size_t)(chunk + 2) * 96;
}
__host__ __device__ constexpr size_t fit_smem_bytes(int sort_cap, int chunk, int nwarps) {
    return fit_x_bytes(sort_cap, chunk) + (size_t)sort_cap * 6 + (size_t)256 * nwarps * 4;
}

// The bucket, of NB, of a slope's order bits (angle_key): the slopes of one
// quadrant are the tangents t in [0, inf) above a multiple of 65536, spread
// by 1 - 1 / (1 + t) with the reciprocal drawn straight between powers of
// two. Never falls as the bits rise: a rounded sum, then integers.
template <int NB>
__device__ __forceinline__ int slope_bucket(uint32_t bits) {
    const float s = __uint_as_float(bits >> 31 ? bits ^ 0x80000000u : ~bits);
    const float q = floorf(__fmul_rn(s, 1.0f / 65536.0f));
    if (q < -1.0f) return 0;
    if (q > 2.0f) return NB - 1;
    const uint32_t x = __float_as_uint(__fadd_rn(1.0f, __fsub_rn(s, __fmul_rn(q, 65536.0f))));  // 1 + t < 2^17
    const uint32_t v = (0x1000000u - (x & 0x7fffffu)) >> ((x >> 23) - 127u);                    // 2^24 / (1 + t)
    const uint32_t b = (0x1000000u - v) / (0x4000000u / NB);
    return ((int)q + 1) * (NB / 4) + (int)b;
}

// A cluster is sorted by buckets while its points share theirs with at most
// this many on average (themselves included); a comb of nearly equal angles
// takes the sort it had before.
#define FIT_SHARE 16

// The block's sort of n (32-bit slope bits, 16-bit value) pairs in a stable
// order: counted into 8 NT buckets, listed by bucket (list: slope bits, place
// before, value), and each pair's place in its bucket found by comparing it
// with the bucket's others. The values end up in va. False (and the pairs as
// they were) if the buckets are too uneven. hist: 8 NT counters.
// Against the radix sort's four passes: 9900 instead of 27400 cycles for 700
// points and 128 threads, 21000 instead of 47600 for 3200 and 256.
template <int NT>
__device__ __forceinline__ bool block_bucket_sort(const uint32_t *ka, uint16_t *va, uint64_t *list, int n,
                                                  uint32_t *hist) {
    constexpr int NB = 8 * NT;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    __shared__ uint32_t s_sum[NT / 32];
    __shared__ uint64_t s_share[NT / 32];
    uint4 *h4 = reinterpret_cast<uint4 *>(hist) + 2 * tid;
    h4[0] = h4[1] = make_uint4(0, 0, 0, 0);
    __syncthreads();
#pragma unroll 4
    for (int i = tid; i < n; i += NT) atomicAdd(hist + slope_bucket<NB>(ka[i]), 1u);
    __syncthreads();
    const uint4 a = h4[0], b = h4[1];
    const uint32_t c[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t o[8], sum = 0;
    uint64_t share = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        o[k] = sum;
        sum += c[k];
        share += (uint64_t)c[k] * c[k];
    }
    for (int d = 16; d > 0; d >>= 1) share += __shfl_xor_sync(0xffffffffu, share, d);
    uint32_t incl = sum;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) {
        s_sum[w] = incl;
        s_share[w] = share;
    }
    __syncthreads();
    for (int v = 1; v < NT / 32; v++) share += s_share[(w + v) % (NT / 32)];
    if (share > (uint64_t)FIT_SHARE * n) return false;
    uint32_t before = incl - sum;
    for (int v = 0; v < w; v++) before += s_sum[v];
    h4[0] = make_uint4(before + o[0], before + o[1], before + o[2], before + o[3]);
    h4[1] = make_uint4(before + o[4], before + o[5], before + o[6], before + o[7]);
    __syncthreads();
    // from here on a bucket's counter runs to its end
    for (int i = tid; i < n; i += 2 * NT) {
        const int i2 = i + NT;
        const uint32_t k = ka[i], k2 = i2 < n ? ka[i2] : 0u;
        const uint64_t e = (uint64_t)k << 32 | (uint32_t)i << 16 | va[i],
                       e2 = i2 < n ? (uint64_t)k2 << 32 | (uint32_t)i2 << 16 | va[i2] : 0ull;
        const int b1 = slope_bucket<NB>(k), b2 = slope_bucket<NB>(k2);
        const uint32_t j = atomicAdd(hist + b1, 1u), j2 = i2 < n ? atomicAdd(hist + b2, 1u) : 0u;
        list[j] = e;
        if (i2 < n) list[j2] = e2;
    }
    __syncthreads();
    for (int j = tid; j < n; j += NT) {
        const uint64_t e = list[j];
        const int bk = slope_bucket<NB>((uint32_t)(e >> 32)), s0 = bk ? (int)hist[bk - 1] : 0, s1 = (int)hist[bk];
        int at = s0;
        for (int q = s0; q < s1; q++) at += list[q] < e;
        va[at] = (uint16_t)e;
    }
    __syncthreads();
    return true;
}

// The exclusive prefix sums of a warp's NB counts, in place. False if the
// buckets of n are too uneven (the counts as they were).
template <int NB>
__device__ bool warp_bucket_scan(uint32_t *hist, int n, int lane) {
    constexpr int PER = NB / 32;
    uint32_t o[PER], sum = 0, share = 0;
#pragma unroll
    for (int k = 0; k < PER; k += 4) {
        const uint4 c = reinterpret_cast<const uint4 *>(hist)[lane * (PER / 4) + k / 4];
        const uint32_t v[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            o[k + j] = sum;
            sum += v[j];
            share += v[j] * v[j];
        }
    }
    uint32_t incl = sum;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
    }
    if (__reduce_add_sync(0xffffffffu, share) > (uint32_t)(FIT_SHARE * n)) return false;
    const uint32_t before = incl - sum;
#pragma unroll
    for (int k = 0; k < PER; k += 4)
        reinterpret_cast<uint4 *>(hist)[lane * (PER / 4) + k / 4] =
            make_uint4(before + o[k], before + o[k + 1], before + o[k + 2], before + o[k + 3]);
    __syncwarp();
    return true;
}

// Stable sort of n (32-bit key, 16-bit value) pairs by key: four passes of
// 8 bits. Each pass counts digits per warp over the warp's contiguous range,
// scans the counts in (digit, warp) order, and scatters each warp's range in
// order, 32 at a time, ranking equal digits by lane (match_any). ka/va hold
// the input and get the result; kb/vb are the second buffers; hist holds
// 256 counters per warp.
__device__ void block_radix_sort32(uint32_t *ka, uint16_t *va, uint32_t *kb, uint16_t *vb, int n, uint32_t *hist) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
    const int per = ((n + nw - 1) / nw + 31) & ~31;
    const int w0 = w * per < n ? w * per : n, w1 = w0 + per < n ? w0 + per : n;
    const int nh = 256 * nw;
    __shared__ uint32_t s_part[32];
    for (int shift = 0; shift < 32; shift += 8) {
        for (int i = tid; i < nh; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        for (int i = w0 + lane; i < w1; i += 32) atomicAdd(hist + (int)(ka[i] >> shift & 255u) * nw + w, 1u);
        __syncthreads();
        // exclusive scan of hist: thread t owns entries [t * e, t * e + e)
        const int e = (nh + blockDim.x - 1) / blockDim.x;
        const int h0 = tid * e < nh ? tid * e : nh, h1 = h0 + e < nh ? h0 + e : nh;
        uint32_t sum = 0;
        for (int i = h0; i < h1; i++) sum += hist[i];
        uint32_t incl = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_part[w] = incl;
        __syncthreads();
        if (w == 0) {
            uint32_t v = lane < nw ? s_part[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += t;
            }
            if (lane < nw) s_part[lane] = v;
        }
        __syncthreads();
        uint32_t run = (w > 0 ? s_part[w - 1] : 0) + incl - sum;
        for (int i = h0; i < h1; i++) {
            const uint32_t c = hist[i];
            hist[i] = run;
            run += c;
        }
        __syncthreads();
        for (int i0 = w0; i0 < w1; i0 += 32) {
            const int i = i0 + lane;
            const bool valid = i < w1;
            const uint32_t k = valid ? ka[i] : 0;
            const int d = valid ? (int)(k >> shift & 255u) : 256 + lane;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            const uint32_t base = valid ? hist[d * nw + w] : 0;
            if (valid) {
                const uint32_t at = base + __popc(peers & ((1u << lane) - 1u));
                kb[at] = k;
                vb[at] = va[i];
            }
            __syncwarp();
            if (valid && lane == __ffs(peers) - 1) hist[d * nw + w] = base + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        uint32_t *tk = ka;
        ka = kb;
        kb = tk;
        uint16_t *tv = va;
        va = vb;
        vb = tv;
    }
}

// ---------------------------------------------------------------------------
// The fit's size classes: clusters of at most 128, 256, 512 points (a warp
// each; few of the last: see FIT_FEW), at most 1024 (a block of 128), at most 6144 (a block of 256), and
// larger (a block of 512). A class's clusters are listed by size in a few
// buckets, and its blocks take those of the largest bucket first, so that a
// long cluster does not start last (unsorted, the 513-1024 class took 175
// instead of 159 us; sorting the lists took a kernel of 27 us before each
// block class). Clusters outside [min_cluster_pixels, max_px] of their frame
// get no list (fast/quads.c:1180-1190), and none does when the row tables were
// too small (AT_ERR_SEGCAP: the points are not placed, the host runs the batch
// again). Every cluster's quad flag starts at 0.
__device__ __forceinline__ int fit_bucket(int64_t sz) {
    if (sz <= 512) return sz <= 128 ? 0 : sz <= 256 ? 1 : 2;
    if (sz <= FIT_SMALL) return sz <= 640 ? 3 : sz <= 768 ? 4 : sz <= 896 ? 5 : 6;
    if (sz <= FIT_LARGE_SORT) return sz <= 1536 ? 7 : sz <= 2048 ? 8 : sz <= 3072 ? 9 : sz <= 4096 ? 10 : 11;
    return sz <= 9216 ? 12 : sz <= FIT_HUGE_SORT ? 13 : sz <= 20480 ? 14 : 15;
}

// The next cluster of buckets top .. bottom (0xffffffff: none left): counts
// holds each bucket's length, then per bucket (used at `top`) the clusters
// taken.
__device__ __forceinline__ uint32_t fit_next(const FitScratch &scr, int64_t nclusters, int top, int bottom) {
    uint32_t i = atomicAdd(scr.counts + FIT_NBUCKET + top, 1u);
    for (int q = top; q >= bottom; q--) {
        const uint32_t n = scr.counts[q];
        if (i < n) return scr.lists[(int64_t)q * nclusters + i];
        i -= n;
    }
    return 0xffffffffu;
}

__global__ void k_fit_classify(const FrameDesc *frames, const uint32_t *cstart, const int32_t *cframe,
                               int64_t nclusters, int64_t npoints, int32_t min_px, uint32_t *quad_ok,
                               uint32_t *lists, uint32_t *counts, const uint32_t *err) {
    kernel_begin();
    const bool placed = !(*err & AT_ERR_SEGCAP);
    __shared__ uint32_t s_n[FIT_NBUCKET], s_at[FIT_NBUCKET];
    for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x; c0 < nclusters; c0 += (int64_t)gridDim.x * blockDim.x) {
        __syncthreads();
        if (threadIdx.x < FIT_NBUCKET) s_n[threadIdx.x] = 0;
        __syncthreads();
        const int64_t c = c0 + threadIdx.x;
        int k = -1;
        uint32_t at = 0;
        if (c < nclusters) {
            quad_ok[c] = 0;
            const int64_t sz = (c + 1 < nclusters ? (int64_t)cstart[c + 1] : npoints) - cstart[c];
            if (placed && sz >= min_px && sz <= frames[cframe[c]].max_px) k = fit_bucket(sz);
            if (k >= 0) at = atomicAdd(s_n + k, 1u);
        }
        __syncthreads();
        // (all buckets' places at once: one after the other took 9 us for 132 clusters)
        if (threadIdx.x < FIT_NBUCKET && s_n[threadIdx.x])
            s_at[threadIdx.x] = atomicAdd(counts + threadIdx.x, s_n[threadIdx.x]);
        __syncthreads();
        if (k >= 0) lists[(int64_t)k * nclusters + s_at[k] + at] = (uint32_t)c;
    }
}

// The 4-subsets {m0 < m1 < m2 < m3} of {0..15} in colex order (by m3, then
// m2, m1, m0), one per entry as nibbles m0 | m1 << 4 | m2 << 8 | m3 << 12:
// the first C(n, 4) entries are the 4-subsets of {0..n-1}.
struct Quad4Table {
    uint16_t v[1820];
};
constexpr Quad4Table make_quad4() {
    Quad4Table t{};
    int k = 0;
    for (int d = 3; d < 16; d++)
        for (int c = 2; c < d; c++)
            for (int b = 1; b < c; b++)
                for (int a = 0; a < b; a++) t.v[k++] = (uint16_t)(a | b << 4 | c << 8 | d << 12);
    return t;
}
__device__ const Quad4Table g_quad4 = make_quad4();
static_assert(AT_MAX_NMAXIMA <= 16, "the 4-subset table covers 16 maxima");

__host__ __device__ constexpr int binom4(int n) { return n < 4 ? 0 : n * (n - 1) * (n - 2) * (n - 3) / 24; }

// The quad of four lines (x, y, nx, ny; line i and its fit's error in lane i
// of the warp, i < 4): its corners (corner i in lane i), and whether it passes
// the fit, area and convexity gates (fast/quads.c:1079-1125). A lane a corner:
// one thread for all four took 5000 cycles.
__device__ __forceinline__ bool quad_of(int lane, const double ln[4], double lmse, const GpuParams &prm, int tag_width,
                                        float p[2]) {
    const unsigned FULL = 0xffffffffu;
    const int nx = (lane + 1) & 3;
    double lj[4];
#pragma unroll
    for (int k = 0; k < 4; k++) lj[k] = __shfl_sync(FULL, ln[k], nx);
    const double a00 = ln[3], a01 = -lj[3], a10 = -ln[2], a11 = lj[2];
    const double b0 = -ln[0] + lj[0], b1 = -ln[1] + lj[1];
    const double det = a00 * a11 - a10 * a01;
    if (__any_sync(FULL, lane < 4 && (lmse > prm.max_mse || fabs(det) < 0.001))) return false;
    const double w00 = a11 / det, w01 = -a01 / det;
    const double l0 = w00 * b0 + w01 * b1;
    p[0] = (float)(ln[0] + l0 * a00);
    p[1] = (float)(ln[1] + l0 * a10);
    float q[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        q[i][0] = __shfl_sync(FULL, p[0], (lane + i) & 3);
        q[i][1] = __shfl_sync(FULL, p[1], (lane + i) & 3);
    }
    // the triangles (0, 1, 2) and (2, 3, 0) by Heron: lane t the one that
    // starts at corner t (lanes 0 and 2 count)
    double len[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int ib = i == 2 ? 0 : i + 1;
        const double ddx = (double)__fsub_rn(q[ib][0], q[i][0]), ddy = (double)__fsub_rn(q[ib][1], q[i][1]);
        len[i] = sqrt(ddx * ddx + ddy * ddy);
    }
    const double pp = (len[0] + len[1] + len[2]) / 2.0;
    const double tri = sqrt(pp * (pp - len[0]) * (pp - len[1]) * (pp - len[2]));
    const double area = __shfl_sync(FULL, tri, 0) + __shfl_sync(FULL, tri, 2);
    // convexity at corner lane + 1
    const double dx1 = (double)__fsub_rn(q[1][0], q[0][0]), dy1 = (double)__fsub_rn(q[1][1], q[0][1]);
    const double dx2 = (double)__fsub_rn(q[2][0], q[1][0]), dy2 = (double)__fsub_rn(q[2][1], q[1][1]);
    const double den = sqrt((dx1 * dx1 + dy1 * dy1) * (dx2 * dx2 + dy2 * dy2));
    const double cs = (dx1 * dx2 + dy1 * dy2) / den;
    const bool bad = den == 0.0 || (cs > prm.max_dot || cs < -prm.max_dot) || dx1 * dy2 < dy1 * dx2;
    return !__any_sync(FULL, lane < 4 && bad) && !(area < 0.95 * (double)tag_width * (double)tag_width);
}

template <int NT>
__global__ void __launch_bounds__(NT, (NT <= 128 ? 4 : NT <= 256 ? 2 : 1)) k_fit_quads(const FrameDesc *frames, GpuParams prm, const uint8_t *qim,
                                                   const uint64_t *pts, const uint32_t *cstart,
                                                   const int32_t *cframe, int64_t nclusters, int64_t npoints,
                                                   FitScratch scr, GpuQuad *quads, uint32_t *quad_ok, uint32_t *err,
                                                   int top, int bottom, int sort_cap, int chunk) {
    kernel_begin();
    extern __shared__ __align__(16) unsigned char fit_smem[];
    const size_t xb = fit_x_bytes(sort_cap, chunk);
    uint64_t *s_key = reinterpret_cast<uint64_t *>(fit_smem);  // X: angle keys
    uint32_t *s_kb = reinterpret_cast<uint32_t *>(fit_smem);   // X: the sort's second buffers
    uint16_t *s_vb = reinterpret_cast<uint16_t *>(fit_smem + (size_t)sort_cap * 4);
    double *s_w = reinterpret_cast<double *>(fit_smem);        // X: six terms per staged point
    uint32_t *s_ka = reinterpret_cast<uint32_t *>(fit_smem + xb);
    uint16_t *s_val = reinterpret_cast<uint16_t *>(fit_smem + xb + (size_t)sort_cap * 4);
    uint32_t *s_hist = reinterpret_cast<uint32_t *>(fit_smem + xb + (size_t)sort_cap * 6);
    __shared__ float s_lane[8];
    __shared__ int s_rev, s_ok;
    __shared__ uint32_t s_bb[4][NT / 32];
    __shared__ uint32_t s_scan[32];
    __shared__ double s_perr[AT_MAX_NMAXIMA * AT_MAX_NMAXIMA], s_pmse[AT_MAX_NMAXIMA * AT_MAX_NMAXIMA],
        s_pnx[AT_MAX_NMAXIMA * AT_MAX_NMAXIMA], s_pny[AT_MAX_NMAXIMA * AT_MAX_NMAXIMA];
    __shared__ double s_be[NT / 32], s_lines[4][4], s_lmse[4];
    __shared__ int s_bo[NT / 32];
    __shared__ uint32_t s_next;
    __shared__ uint64_t s_part[3 * NT / 32];
    __shared__ int s_kept[AT_MAX_NMAXIMA], s_nkept;
    const int tid = threadIdx.x;
    const int low = NT == 128 && scr.counts[2] <= FIT_FEW ? bottom - 1 : bottom;

    // the class's clusters, its largest sizes first, each to the next free block
    for (;;) {
        __syncthreads();
        if (tid == 0) s_next = fit_next(scr, nclusters, top, low);
        __syncthreads();
        if (s_next == 0xffffffffu) break;
        const int64_t c = s_next;
        const int64_t s0 = cstart[c];
        const int64_t sz = (c + 1 < nclusters ? (int64_t)cstart[c + 1] : npoints) - s0;
        const FrameDesc f = frames[cframe[c]];
        if (sz > 65535) {
            if (tid == 0) atomicOr(err, AT_ERR_CLUSTER_TOO_BIG);
            continue;
        }
        const uint64_t *P = pts + s0;
        // bounding box (fast/quads.c:515-528)
        uint32_t xmin = 0xffff, xmax = 0, ymin = 0xffff, ymax = 0;
        for (int64_t i = tid; i < sz; i += NT) {
            uint32_t x = (uint32_t)(P[i] & 0xffff), y = (uint32_t)(P[i] >> 16 & 0xffff);
            xmin = min(xmin, x);
            xmax = max(xmax, x);
            ymin = min(ymin, y);
            ymax = max(ymax, y);
        }
        for (int o = 16; o > 0; o >>= 1) {
            xmin = min(xmin, __shfl_xor_sync(0xffffffffu, xmin, o));
            xmax = max(xmax, __shfl_xor_sync(0xffffffffu, xmax, o));
            ymin = min(ymin, __shfl_xor_sync(0xffffffffu, ymin, o));
            ymax = max(ymax, __shfl_xor_sync(0xffffffffu, ymax, o));
        }
        __syncthreads();
        if ((tid & 31) == 0) {
            s_bb[0][tid >> 5] = xmin;
            s_bb[1][tid >> 5] = xmax;
            s_bb[2][tid >> 5] = ymin;
            s_bb[3][tid >> 5] = ymax;
        }
        __syncthreads();
        for (int w = 0; w < NT / 32; w++) {
            xmin = min(xmin, s_bb[0][w]);
            xmax = max(xmax, s_bb[1][w]);
            ymin = min(ymin, s_bb[2][w]);
            ymax = max(ymax, s_bb[3][w]);
        }
        if ((int64_t)(xmax - xmin) * (int64_t)(ymax - ymin) < f.tag_width) continue;
        const float cx = (float)((double)(xmin + xmax) * 0.5 + 0.05118);
        const float cy = (float)((double)(ymin + ymax) * 0.5 + -0.028581);

        // angle keys, and the dot product of offsets and gradients: 8 lanes
        // over the whole groups of 8, then the rest (fast/quads.c:467-512)
        // clusters that fit keep their keys in shared memory, where the
        // leaf step turns them into sort keys in place
        const bool in_smem = sz <= sort_cap;
        uint64_t *keys = in_smem ? s_key : scr.keys + s0;
        for (int64_t i = tid; i < sz; i += NT) {
            float dx = __fsub_rn((float)(P[i] & 0xffff), cx), dy = __fsub_rn((float)(P[i] >> 16 & 0xffff), cy);
            keys[i] = angle_key(dx, dy, (uint32_t)i);
        }
        const int64_t nv = sz - sz % 8;
        {
            // the terms dx*gx + dy*gy by all threads into shared memory (the
            // moment staging area, free here), then lane l < 8 sums terms
            // l, l+8, ... in order
            float *s_term = reinterpret_cast<float *>(s_ka);
            const int64_t tcap = sort_cap;  // a multiple of 8
            float acc = 0.0f;
            for (int64_t c0 = 0; c0 < nv; c0 += tcap) {
                const int64_t cn = dmin(tcap, nv - c0);
                for (int64_t i = tid; i < cn; i += NT) {
                    uint64_t pt = P[c0 + i];
                    float dx = __fsub_rn((float)(pt & 0xffff), cx), dy = __fsub_rn((float)(pt >> 16 & 0xffff), cy);
                    float gx = (float)(int16_t)(pt >> 32 & 0xffff), gy = (float)(int16_t)(pt >> 48);
                    s_term[i] = __fadd_rn(__fmul_rn(dx, gx), __fmul_rn(dy, gy));
                }
                __syncthreads();
                if (tid < 8) {
                    int64_t i = tid;
                    for (; i + 56 < cn; i += 64) {
                        float v[8];
#pragma unroll
                        for (int u = 0; u < 8; u++) v[u] = s_term[i + 8 * u];
#pragma unroll
                        for (int u = 0; u < 8; u++) acc = __fadd_rn(acc, v[u]);
                    }
                    for (; i < cn; i += 8) acc = __fadd_rn(acc, s_term[i]);
                }
                __syncthreads();
            }
            if (tid < 8) s_lane[tid] = acc;
        }
        __syncthreads();
        if (tid == 0) {
            float dot = __fadd_rn(__fadd_rn(__fadd_rn(s_lane[0], s_lane[4]), __fadd_rn(s_lane[2], s_lane[6])),
                                  __fadd_rn(__fadd_rn(s_lane[1], s_lane[5]), __fadd_rn(s_lane[3], s_lane[7])));
            for (int64_t i = nv; i < sz; i++) {
                float dx = __fsub_rn((float)(P[i] & 0xffff), cx), dy = __fsub_rn((float)(P[i] >> 16 & 0xffff), cy);
                float gx = (float)(int16_t)(P[i] >> 32 & 0xffff), gy = (float)(int16_t)(P[i] >> 48);
                dot = __fadd_rn(dot, __fadd_rn(__fmul_rn(dx, gx), __fmul_rn(dy, gy)));
            }
            int rev = dot < 0.0f;
            int ok = 1;
            if (!f.reversed_border && rev) ok = 0;
            if (!f.normal_border && !rev) ok = 0;
            s_ok = ok;
            s_rev = rev;
        }
        __syncthreads();
        if (!s_ok) continue;
        const int rev = s_rev;

        // The angle sort. The reference's merge sort keeps each leaf's
        // "blocks" (a key larger than all before it in the leaf's network
        // order, and the smaller keys after it) together and orders them by
        // their first key. So: per leaf, the network order, each key's
        // block head and its place in the leaf; then one sort by (head,
        // place), packed into 64 bits as head's slope bits, 0xffff - head's
        // index, and the place.
        // the sort's two pairs of buffers, in shared memory or global scratch
        uint32_t *ka = in_smem ? s_ka : reinterpret_cast<uint32_t *>(scr.skey + s0), *kb = in_smem ? s_kb : ka + sz;
        uint16_t *va = in_smem ? s_val : reinterpret_cast<uint16_t *>(scr.sval + s0), *vb = in_smem ? s_vb : va + sz;
        // Lay the points out in (head index descending, place) order:
        // leaves in reverse order, and in each leaf its blocks by head
        // index descending, each block in network order. A stable sort
        // by the head's slope bits then gives the (head, place) order.
        // Each warp finds the leaves that start in its 32 points at a
        // time, queues them in its slice of the (still unused) radix
        // histograms, and arranges them 32 leaves at a time.
        auto arrange = [&](uint32_t lf) {
            const int lo = (int)(lf >> 8), len = (int)(lf & 255);
            // everything indexed by constants: registers only
            uint64_t k5[5];
#pragma unroll
            for (int t = 0; t < 5; t++) k5[t] = t < len ? keys[lo + t] : ~0ull;
            leaf_network(k5, len);
            uint32_t hid[5], hkey[5];
            int bs[5];
            uint64_t head = k5[0];
            int start = 0;
#pragma unroll
            for (int t = 0; t < 5; t++) {
                if (t > 0 && k5[t] > head) {
                    head = k5[t];
                    start = t;
                }
                hid[t] = ~(uint32_t)head;
                hkey[t] = (uint32_t)(head >> 32);
                bs[t] = start;
            }
            const int base = (int)sz - lo - len;
#pragma unroll
            for (int t = 0; t < 5; t++) {
                if (t >= len) continue;
                int before = 0;  // points of blocks with a larger head index
#pragma unroll
                for (int t2 = 0; t2 < 5; t2++) before += t2 < len && hid[t2] > hid[t];
                const int pos = base + before + (t - bs[t]);
                ka[pos] = hkey[t];
                va[pos] = (uint16_t)~(uint32_t)k5[t];
            }
        };
        {
            const int lane = tid & 31;
            uint32_t *lq = s_hist + (tid >> 5) * 256;
            int qn = 0;
            for (int64_t p0 = (int64_t)(tid >> 5) * 32; p0 < sz; p0 += NT) {
                const int64_t p = p0 + lane;
                int llo = -1, llen = 0;
                if (p < sz) leaf_of((int)sz, (int)p, llo, llen);
                const bool lead = llo == (int)p;
                const uint32_t lf = (uint32_t)llo << 8 | (uint32_t)llen;
                const uint32_t bal = __ballot_sync(0xffffffffu, lead);
                if (lead) lq[qn + __popc(bal & ((1u << lane) - 1u))] = lf;
                qn += __popc(bal);
                __syncwarp();
                if (qn >= 32) {
                    qn -= 32;
                    arrange(lq[qn + lane]);
                    __syncwarp();
                }
            }
            if (lane < qn) arrange(lq[lane]);
        }
        __syncthreads();
        if (!block_bucket_sort<NT>(ka, va, keys, (int)sz, s_hist))
            block_radix_sort32(ka, va, kb, vb, (int)sz, s_hist);

        // cumulative weighted moments in angle order (fast/quads.c:968-1035):
        // Chunks of points get their six terms (moment_terms) staged in
        // shared memory, two buffers deep: while lane q < 6 of warp 0 runs
        // prefix sum q over chunk c in point order, the other warps stage
        // chunk c + 1.
        const uint8_t *im = qim + f.q_off;
        double *M[6] = {scr.mx + s0, scr.my + s0, scr.mxx + s0, scr.mxy + s0, scr.myy + s0, scr.mw + s0};
        double run = 0.0;
        const int cs = chunk + 2;  // row stride of the staged terms
        // (two points a thread at a time, so that their gathers overlap)
        auto stage = [&](int64_t k0, double *buf, int first, int stride) {
            const int kn = (int)dmin((int64_t)chunk, sz - k0);
            for (int t = first; t < kn; t += 2 * stride) {
                const int t2 = t + stride < kn ? t + stride : t;
                const uint64_t p1 = P[va[k0 + t]], p2 = P[va[k0 + t2]];
                const int32_t g1 = point_grad2(im, f.qw, f.qh, p1), g2 = point_grad2(im, f.qw, f.qh, p2);
                double m1[6], m2[6];
                moment_terms(p1, g1, m1);
                moment_terms(p2, g2, m2);
#pragma unroll
                for (int q = 0; q < 6; q++) {
                    buf[q * cs + t] = m1[q];
                    buf[q * cs + t2] = m2[q];
                }
            }
        };
        // the prefix sums are taken in place in shared memory; the other
        // warps copy a finished chunk out before staging into its buffer
        auto copy_out = [&](int64_t k0, const double *buf, int first, int stride) {
            const int kn = (int)dmin((int64_t)chunk, sz - k0);
            for (int i = first; i < kn; i += stride) {
#pragma unroll
                for (int q = 0; q < 6; q++) M[q][k0 + i] = buf[q * cs + i];
            }
        };
        stage(0, s_w, tid, NT);
        __syncthreads();
        int64_t ch = 0;
        for (int64_t k0 = 0; k0 < sz; k0 += chunk, ch++) {
            double *cur = s_w + (ch & 1) * 6 * cs, *oth = s_w + ((ch + 1) & 1) * 6 * cs;
            if (tid < 32) {
                if (tid < 6) prefix_chain(cur + tid * cs, (int)dmin((int64_t)chunk, sz - k0), run);
            } else {
                if (ch > 0) copy_out(k0 - chunk, oth, tid - 32, NT - 32);
                asm volatile("bar.sync 1, %0;" ::"r"(NT - 32));
                if (k0 + chunk < sz) stage(k0 + chunk, oth, tid - 32, NT - 32);
            }
            __syncthreads();
        }
        if (ch > 0) copy_out((ch - 1) * chunk, s_w + ((ch - 1) & 1) * 6 * cs, tid, NT);
        __syncthreads();
        const Moments mo = {M[0], M[1], M[2], M[3], M[4], M[5]};
        const MSum all = moments_at(mo, sz - 1);

        // corner search (fast/quads.c:788-959)
        const int64_t ksz = dmin(20, sz / 12);
        if (ksz < 2) continue;
        const double nn = (double)(2 * ksz + 1);
        // errors, filtered errors and maxima in shared memory where they fit:
        // the errors where the angle keys were, the filtered errors over the
        // sort's first buffers and histograms, then the maxima (at most one
        // in two points) over the errors. From global memory the maxima took
        // 11500 cycles for 700 points and 32000 for 3200, now 10000 and 16000.
        double *errs = in_smem ? reinterpret_cast<double *>(s_key) : scr.errs + s0;
        double *filt = 8 * sz <= 6 * (int64_t)sort_cap + 32 * NT ? reinterpret_cast<double *>(s_ka) : scr.filt + s0;
        // two points a thread at a time: both windows' loads before either
        // store (a store could alias the next loads)
        for (int64_t i = tid; i < sz; i += 2 * NT) {
            const int64_t i2 = i + NT < sz ? i + NT : i;
            const MSum sa = window_moments(mo, all, sz, ksz, i), sb = window_moments(mo, all, sz, ksz, i2);
            const double ea = window_error(sa, nn), eb = window_error(sb, nn);
            errs[i] = ea;
            errs[i2] = eb;
        }
        __syncthreads();
        for (int64_t i = tid; i < sz; i += 2 * NT) {
            const int64_t i2 = i + NT < sz ? i + NT : i;
            const double fa = smooth_at(errs, sz, i, prm.qsm), fb = smooth_at(errs, sz, i2, prm.qsm);
            filt[i] = fa;
            filt[i2] = fb;
        }
        __syncthreads();
        // local maxima with wrap-around, compacted in index order: each
        // warp counts those of its own stretch, then writes them after the
        // warps' before it (two reads of filt, but only two barriers)
        double *mxe = in_smem ? reinterpret_cast<double *>(s_key) : scr.mxe + s0;
        int32_t *mxi = in_smem ? reinterpret_cast<int32_t *>(fit_smem + (size_t)4 * sort_cap) : scr.mxi + s0;
        int nm;
        if (tid == 0) s_nkept = 0;
        {
            const int n = (int)sz, lane = tid & 31, w = tid >> 5;
            const int per = ((n + NT / 32 - 1) / (NT / 32) + 31) & ~31, i0 = w * per, i1 = min(i0 + per, n);
            auto is_max = [&](int i, double &e) {
                e = filt[i];
                return e > filt[i == 0 ? n - 1 : i - 1] && e > filt[i + 1 == n ? 0 : i + 1];
            };
            int cnt = 0;
            double e;
            for (int i = i0 + lane; i < i1; i += 32) cnt += is_max(i, e);
            cnt = __reduce_add_sync(0xffffffffu, cnt);
            if (lane == 0) s_scan[w] = (uint32_t)cnt;
            __syncthreads();
            int at = 0;
            nm = 0;
            for (int v = 0; v < NT / 32; v++) {
                if (v == w) at = nm;
                nm += (int)s_scan[v];
            }
            for (int j0 = i0; j0 < i1; j0 += 32) {
                const int i = j0 + lane;
                const bool mx = i < i1 && is_max(i, e);
                const uint32_t bal = __ballot_sync(0xffffffffu, mx);
                if (mx) {
                    const int o = at + __popc(bal & ((1u << lane) - 1u));
                    mxi[o] = i;
                    mxe[o] = e;
                }
                at += __popc(bal);
            }
            __syncthreads();
        }
        if (nm < 4) continue;
        if (nm > prm.max_nmaxima) {
            // The reference keeps the maxima whose error is above the
            // (max_nmaxima+1)-th largest (its quickselect, quads.c:827-862).
            const uint64_t v = block_above<NT>(mxe, nm, prm.max_nmaxima, s_part);
            for (int i = tid; i < nm; i += NT)
                if (double_order(mxe[i]) >= v) s_kept[atomicAdd(&s_nkept, 1)] = mxi[i];
            __syncthreads();
            nm = s_nkept;
            if (tid < nm) {
                int before = 0;
                for (int j = 0; j < nm; j++) before += s_kept[j] < s_kept[tid];
                mxi[before] = s_kept[tid];
            }
            __syncthreads();
        }
        // line fits of pairs of maxima: (a, b), a < b, and the closing pair
        // (b, a) wrapping around for b >= a + 3
        for (int t = tid; t < nm * nm; t += NT) {
            const int p = t / nm, q = t - p * nm;
            bool used = p < q || p >= q + 3;
            if (!used) continue;
            int64_t i0 = mxi[p], i1 = mxi[q];
            MSum s = seg_moments(mo, all, i0, i1);
            double n = (double)(i0 <= i1 ? i1 - i0 + 1 : sz - i0 + i1 + 1);
            double lp[4], mse;
            line_of(s, lp, &mse);
            s_perr[t] = n * mse;
            s_pmse[t] = mse;
            s_pnx[t] = lp[2];
            s_pny[t] = lp[3];
        }
        __syncthreads();
        // the 4 maxima with the smallest total error (quads.c:931-958): the
        // reference keeps the first strictly smaller error in (m0, m1, m2, m3)
        // order, i.e. the smallest error and, among equal ones, the first in
        // that order. Each thread scans some of the 4-subsets (g_quad4); then
        // a block-wide minimum of (error, order), which every thread then has.
        const double inf = __longlong_as_double(0x7ff0000000000000ll);
        double be = inf;
        {
            int bo = 0x10000;
            const int n = nm, nsub = binom4(n);
            for (int t = tid; t < nsub; t += NT) {
                const int v = g_quad4.v[t];
                const int m0 = v & 15, m1 = v >> 4 & 15, m2 = v >> 8 & 15, m3 = v >> 12;
                const int p01 = m0 * n + m1, p12 = m1 * n + m2;
                if (s_pmse[p01] > prm.max_mse || s_pmse[p12] > prm.max_mse) continue;
                const double dot = s_pnx[p01] * s_pnx[p12] + s_pny[p01] * s_pny[p12];
                if (fabs(dot) > prm.max_dot) continue;
                const int p23 = m2 * n + m3, p30 = m3 * n + m0;
                const double e012 = s_perr[p01] + s_perr[p12];
                const double e23 = s_pmse[p23] > prm.max_mse ? inf : s_perr[p23];
                const double e30 = s_pmse[p30] > prm.max_mse ? inf : s_perr[p30];
                const double e = e012 + e23 + e30;
                const int ord = m0 << 12 | m1 << 8 | m2 << 4 | m3;
                if (e < be || (e == be && ord < bo)) {
                    be = e;
                    bo = ord;
                }
            }
            // block minimum of (be, bo)
            for (int o = 16; o > 0; o >>= 1) {
                double e2 = __shfl_xor_sync(0xffffffffu, be, o);
                const int o2 = __shfl_xor_sync(0xffffffffu, bo, o);
                if (e2 < be || (e2 == be && o2 < bo)) {
                    be = e2;
                    bo = o2;
                }
            }
            if ((tid & 31) == 0) {
                s_be[tid >> 5] = be;
                s_bo[tid >> 5] = bo;
            }
            __syncthreads();
            if (tid == 0) {
                for (int w = 1; w < NT / 32; w++)
                    if (s_be[w] < be || (s_be[w] == be && s_bo[w] < bo)) {
                        be = s_be[w];
                        bo = s_bo[w];
                    }
                s_be[0] = be;
                s_bo[0] = bo;
            }
            __syncthreads();
            be = s_be[0];
            bo = s_bo[0];
            // the 4 line fits (quads.c:1069-1075), one per thread
            if (be != inf && tid < 4) {
                double mse;
                const int ma = bo >> (12 - 4 * tid) & 15, mb = bo >> (12 - 4 * ((tid + 1) & 3)) & 15;
                line_of(seg_moments(mo, all, mxi[ma], mxi[mb]), s_lines[tid], &mse);
                s_lmse[tid] = mse;
            }
            __syncthreads();
        }
        if (tid < 32) {
            if (be != inf && be / (double)sz < prm.max_mse) {
                const double *l = s_lines[tid & 3];
                const double ln[4] = {l[0], l[1], l[2], l[3]};
                float p[2];
                if (quad_of(tid, ln, s_lmse[tid & 3], prm, f.tag_width, p) && tid < 4) {
                    quads[c].p[tid][0] = p[0];
                    quads[c].p[tid][1] = p[1];
                    if (tid == 0) {
                        quads[c].reversed_border = rev;
                        quads[c].frame = cframe[c];
                        quad_ok[c] = 1;
                    }
                }
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Clusters of at most 32 * R points: one warp each, FIT_WPB per block, no
// block barriers. The same steps as k_fit_quads; up to 256 points the prefix
// moments stay in shared memory.
#define FIT_WPB 2

// per warp: six prefix arrays, then region x0 (angle keys; errors; the
// maxima) and region x1 (dot terms; filtered errors; the pair fits)
__host__ __device__ constexpr size_t fit_warp_x1(int cap, int mm) {
    return (size_t)8 * cap > (size_t)32 * mm * mm ? (size_t)8 * cap : (size_t)32 * mm * mm;
}
// gp: the prefix arrays in global scratch (the largest warp class, where
// 48 B per point of shared memory would leave few warps per SM)
__host__ __device__ constexpr size_t fit_warp_smem(int cap, int mm, bool gp = false) {
    return (size_t)8 * cap + (gp ? 0 : 48 * (cap + 2)) + fit_warp_x1(cap, mm);
}



// Bitonic sort, ascending, of a warp's keys k[0, np) in shared memory (np
// a power of two): log2(np) (log2(np) + 1) / 2 steps of np / 2 exchanges.
__device__ void warp_bitonic(uint64_t *k, int np, int lane) {
    for (int kk = 2; kk <= np; kk <<= 1) {
        for (int j = kk >> 1; j > 0; j >>= 1) {
            for (int q = lane; q < np / 2; q += 32) {
                const int i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), l = i + j;
                const uint64_t a = k[i], b = k[l];
                if (((i & kk) == 0) == (a > b)) {
                    k[i] = b;
                    k[l] = a;
                }
            }
            __syncwarp();
        }
    }
}

// Stable sort of a warp's n (32-bit key, 16-bit value) pairs by key: four
// passes of 8 bits; equal digits keep their order (ranked by lane among 32
// consecutive pairs, match_any). ka/va hold the input and get the result,
// kb/vb are the second buffers, hist 256 counters.
__device__ void warp_radix_sort32(uint32_t *ka, uint16_t *va, uint32_t *kb, uint16_t *vb, int n, uint32_t *hist,
                                  int lane) {
    for (int shift = 0; shift < 32; shift += 8) {
#pragma unroll
        for (int j = 0; j < 8; j++) hist[lane * 8 + j] = 0;
        __syncwarp();
        for (int i = lane; i < n; i += 32) atomicAdd(hist + (ka[i] >> shift & 255u), 1u);
        __syncwarp();
        uint32_t c[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            c[j] = hist[lane * 8 + j];
            sum += c[j];
        }
        uint32_t incl = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        uint32_t run = incl - sum;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            hist[lane * 8 + j] = run;
            run += c[j];
        }
        __syncwarp();
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const bool valid = i < n;
            const uint32_t k = valid ? ka[i] : 0;
            const int d = valid ? (int)(k >> shift & 255u) : 256 + lane;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            const uint32_t base = valid ? hist[d] : 0;
            if (valid) {
                const uint32_t at = base + __popc(peers & ((1u << lane) - 1u));
                kb[at] = k;
                vb[at] = va[i];
            }
            __syncwarp();
            if (valid && lane == __ffs(peers) - 1) hist[d] = base + __popc(peers);
            __syncwarp();
        }
        uint32_t *tk = ka;
        ka = kb;
        kb = tk;
        uint16_t *tv = va;
        va = vb;
        vb = tv;
    }
}

template <int R>
__global__ void __launch_bounds__(FIT_WPB * 32, 12) k_fit_warp(const FrameDesc *frames, GpuParams prm, const uint8_t *qim,
                                                          const uint64_t *pts, const uint32_t *cstart,
                                                          const int32_t *cframe, int64_t nclusters, int64_t npoints,
                                                          int top, GpuQuad *quads, uint32_t *quad_ok, int mm,
                                                          FitScratch scr) {
    kernel_begin();
    constexpr int CAP = 32 * R;
    constexpr bool GP = R >= 16;  // prefix arrays in global scratch
    constexpr int RS = CAP + 2;   // row stride of the prefix arrays (six rows on distinct banks, 16-byte aligned)
    extern __shared__ __align__(16) unsigned char fw_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned FULL = 0xffffffffu;
    unsigned char *base = fw_smem + fit_warp_smem(CAP, mm, GP) * wid;
    double *pm = reinterpret_cast<double *>(base);  // prefix array q at pm + q * RS (not GP)
    unsigned char *x0 = base + (GP ? 0 : 48 * RS), *x1 = x0 + 8 * CAP;
    uint64_t *s_akey = reinterpret_cast<uint64_t *>(x0);
    double *s_err = reinterpret_cast<double *>(x0);
    double *s_mxe = reinterpret_cast<double *>(x0);
    int32_t *s_mxi = reinterpret_cast<int32_t *>(x0 + 4 * CAP);
    float *s_term = reinterpret_cast<float *>(x1);
    double *s_filt = reinterpret_cast<double *>(x1);
    double *s_perr = reinterpret_cast<double *>(x1), *s_pmse = s_perr + mm * mm, *s_pnx = s_pmse + mm * mm,
           *s_pny = s_pnx + mm * mm;
    const double inf = __longlong_as_double(0x7ff0000000000000ll);

    if (R == 16 && scr.counts[2] <= FIT_FEW) return;  // a block of 128 each
    // one resident wave of warps, each taking the class's next cluster
    // from a shared counter as it finishes one (no static share to wait on)
    for (;;) {
        uint32_t li = 0;
        if (lane == 0) li = fit_next(scr, nclusters, top, top);
        li = __shfl_sync(FULL, li, 0);
        if (li == 0xffffffffu) break;
        const int64_t c = li;
        const int64_t s0 = cstart[c];
        const int64_t sz = (c + 1 < nclusters ? (int64_t)cstart[c + 1] : npoints) - s0;
        const FrameDesc f = frames[cframe[c]];
        const int n = (int)sz;
        const uint64_t *P = pts + s0;
        // bounding box (fast/quads.c:515-528)
        uint32_t xmin = 0xffff, xmax = 0, ymin = 0xffff, ymax = 0;
        for (int i = lane; i < n; i += 32) {
            const uint64_t pt = P[i];
            const uint32_t x = (uint32_t)(pt & 0xffff), y = (uint32_t)(pt >> 16 & 0xffff);
            xmin = min(xmin, x);
            xmax = max(xmax, x);
            ymin = min(ymin, y);
            ymax = max(ymax, y);
        }
        for (int o = 16; o > 0; o >>= 1) {
            xmin = min(xmin, __shfl_xor_sync(FULL, xmin, o));
            xmax = max(xmax, __shfl_xor_sync(FULL, xmax, o));
            ymin = min(ymin, __shfl_xor_sync(FULL, ymin, o));
            ymax = max(ymax, __shfl_xor_sync(FULL, ymax, o));
        }
        if ((int64_t)(xmax - xmin) * (int64_t)(ymax - ymin) < f.tag_width) continue;
        const float cx = (float)((double)(xmin + xmax) * 0.5 + 0.05118);
        const float cy = (float)((double)(ymin + ymax) * 0.5 + -0.028581);

        // angle keys (fast/quads.c:429-453) and the dot product of offsets
        // and gradients (fast/quads.c:467-512): lane l < 8 sums terms l,
        // l+8, ... of the whole groups of 8; then the rest in order
        const int nv = n - n % 8;
        for (int i = lane; i < n; i += 32) {
            const uint64_t pt = P[i];
            const float dx = __fsub_rn((float)(pt & 0xffff), cx), dy = __fsub_rn((float)(pt >> 16 & 0xffff), cy);
            s_akey[i] = angle_key(dx, dy, (uint32_t)i);
            const float gx = (float)(int16_t)(pt >> 32 & 0xffff), gy = (float)(int16_t)(pt >> 48);
            s_term[i] = __fadd_rn(__fmul_rn(dx, gx), __fmul_rn(dy, gy));
        }
        __syncwarp();
        float acc = 0.0f;
        if (lane < 8) {
            int i = lane;
            for (; i + 56 < nv; i += 64) {
                float v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = s_term[i + 8 * u];
#pragma unroll
                for (int u = 0; u < 8; u++) acc = __fadd_rn(acc, v[u]);
            }
            for (; i < nv; i += 8) acc = __fadd_rn(acc, s_term[i]);
        }
        float l8[8];
#pragma unroll
        for (int k = 0; k < 8; k++) l8[k] = __shfl_sync(FULL, acc, k);
        int okrev = 0;
        if (lane == 0) {
            float dot = __fadd_rn(__fadd_rn(__fadd_rn(l8[0], l8[4]), __fadd_rn(l8[2], l8[6])),
                                  __fadd_rn(__fadd_rn(l8[1], l8[5]), __fadd_rn(l8[3], l8[7])));
            for (int i = nv; i < n; i++) dot = __fadd_rn(dot, s_term[i]);
            const int rev = dot < 0.0f;
            int ok = 1;
            if (!f.reversed_border && rev) ok = 0;
            if (!f.normal_border && !rev) ok = 0;
            okrev = ok | rev << 1;
        }
        okrev = __shfl_sync(FULL, okrev, 0);
        if (!(okrev & 1)) continue;
        const int rev = okrev >> 1;

        // The angle sort (see k_fit_quads). Up to 256 points: packed keys by
        // buckets (177 points: 4900 cycles, a bitonic sort 19900); above: the
        // points laid out in (head index, place) order, then by buckets
        // (360 points: 22000 cycles, four radix passes 33000).
        const uint16_t *s_order = nullptr;  // GP: point index of each sorted position
        if constexpr (!GP) {
            // The angle sort (see k_fit_quads): position i of leaf (lo, len)
            // takes place t = i - lo of the leaf's network order; its sort key
            // packs the slope bits of its block head, 0xffff - the head's index,
            // t, and (below the order, since the rest is distinct) the index of
            // its point. The keys live in the last prefix array until the moments.
            uint64_t *s_skey = reinterpret_cast<uint64_t *>(pm + 5 * RS);
            // buckets, as block_bucket_sort: the counts in x1, each key's
            // bucket and arrival in prefix array 0, the keys by bucket in 1
            // and the buckets beside them in 2
            constexpr int NB = CAP;
            uint32_t *s_hist = reinterpret_cast<uint32_t *>(x1), *s_at = reinterpret_cast<uint32_t *>(pm);
            uint64_t *s_list = reinterpret_cast<uint64_t *>(pm + RS);
            uint16_t *s_bk = reinterpret_cast<uint16_t *>(pm + 2 * RS);
            for (int i = lane; i < NB; i += 32) s_hist[i] = 0;
            __syncwarp();
            int np = 32;
            while (np < n) np <<= 1;
            for (int i = lane; i < np; i += 32) {
                uint64_t key = ~0ull;
                if (i < n) {
                    int lo, len;
                    leaf_of(n, i, lo, len);
                    uint64_t a[5];
    #pragma unroll
                    for (int t = 0; t < 5; t++) a[t] = t < len ? s_akey[lo + t] : ~0ull;
                    leaf_network(a, len);
                    const int tp = i - lo;
                    uint64_t head = a[0], e = a[0];
    #pragma unroll
                    for (int t = 1; t < 5; t++) {
                        if (t <= tp) {
                            if (a[t] > head) head = a[t];
                            e = a[t];
                        }
                    }
                    const uint32_t hidx = ~(uint32_t)head;
                    key = (head & 0xffffffff00000000ull) | (uint64_t)(0xffffu - hidx) << 16 | (uint64_t)tp << 13 |
                          (uint64_t)(~(uint32_t)e & 0x1fffu);
                    const int b = slope_bucket<NB>((uint32_t)(key >> 32));
                    s_at[i] = (uint32_t)b << 16 | atomicAdd(s_hist + b, 1u);
                }
                s_skey[i] = key;
            }
            __syncwarp();
            if (warp_bucket_scan<NB>(s_hist, n, lane)) {
                for (int i = lane; i < n; i += 32) {
                    const uint32_t b = s_at[i] >> 16, j = s_hist[b] + (s_at[i] & 0xffffu);
                    s_list[j] = s_skey[i];
                    s_bk[j] = (uint16_t)b;
                }
                __syncwarp();
                for (int j = lane; j < n; j += 32) {
                    const uint64_t k = s_list[j];
                    const int b = s_bk[j], q0 = (int)s_hist[b], q1 = b + 1 < NB ? (int)s_hist[b + 1] : n;
                    int at = q0;
                    for (int q = q0; q < q1; q++) at += s_list[q] < k;
                    s_skey[at] = k;
                }
                __syncwarp();
            } else {
                warp_bitonic(s_skey, np, lane);
            }
        } else {
            // The angle sort (see k_fit_quads): the points laid out in (head
            // index descending, place) order, a lane per leaf, then a stable
            // sort by the head's slope bits. The sort keys and indices live in
            // region x1.
            uint32_t *s_ka = reinterpret_cast<uint32_t *>(x1);
            uint16_t *s_va = reinterpret_cast<uint16_t *>(x1 + 4 * CAP);
            // second buffers: in x0 once the angle keys are read (x0 holds 8 B
            // per point of capacity, 4 + 2 for the buffers and 1 KB for the
            // histogram)
            uint32_t *s_kb = reinterpret_cast<uint32_t *>(x0);
            uint16_t *s_vb = reinterpret_cast<uint16_t *>(x0 + 4 * CAP);
            uint32_t *s_hist = reinterpret_cast<uint32_t *>(x0 + 6 * CAP);
            // (the leaves found 32 points at a time, queued behind s_va, and
            // laid out 32 leaves at a time)
            uint32_t *lq = reinterpret_cast<uint32_t *>(x1 + 6 * CAP);
            auto arrange = [&](uint32_t lf) {
                const int lo = (int)(lf >> 8), len = (int)(lf & 255);
                uint64_t a[5];
    #pragma unroll
                for (int t = 0; t < 5; t++) a[t] = t < len ? s_akey[lo + t] : ~0ull;
                leaf_network(a, len);
                uint32_t hid[5], hkey[5];
                int bs[5];
                uint64_t head = a[0];
                int start = 0;
    #pragma unroll
                for (int t = 0; t < 5; t++) {
                    if (t > 0 && a[t] > head) {
                        head = a[t];
                        start = t;
                    }
                    hid[t] = ~(uint32_t)head;
                    hkey[t] = (uint32_t)(head >> 32);
                    bs[t] = start;
                }
                const int base = n - lo - len;
    #pragma unroll
                for (int t = 0; t < 5; t++) {
                    if (t >= len) continue;
                    int before = 0;
    #pragma unroll
                    for (int t2 = 0; t2 < 5; t2++) before += t2 < len && hid[t2] > hid[t];
                    const int pos = base + before + (t - bs[t]);
                    s_ka[pos] = hkey[t];
                    s_va[pos] = (uint16_t)~(uint32_t)a[t];
                }
            };
            int qn = 0;
            for (int p0 = 0; p0 < n; p0 += 32) {
                const int p = p0 + lane;
                int lo = -1, len = 0;
                if (p < n) leaf_of(n, p, lo, len);
                const uint32_t bal = __ballot_sync(FULL, lo == p);
                if (lo == p) lq[qn + __popc(bal & ((1u << lane) - 1u))] = (uint32_t)lo << 8 | (uint32_t)len;
                qn += __popc(bal);
                __syncwarp();
                if (qn >= 32) {
                    qn -= 32;
                    arrange(lq[qn + lane]);
                    __syncwarp();
                }
            }
            if (lane < qn) arrange(lq[lane]);
            __syncwarp();
            // buckets, as block_bucket_sort: the counts behind s_va, the list in x0
            constexpr int NB = 256;
            static_assert(4 * NB <= 2 * CAP, "the counts fit x1");
            uint32_t *s_cnt = reinterpret_cast<uint32_t *>(x1 + 6 * CAP);
            uint64_t *s_list = reinterpret_cast<uint64_t *>(x0);
            for (int i = lane; i < NB; i += 32) s_cnt[i] = 0;
            __syncwarp();
#pragma unroll 4
            for (int i = lane; i < n; i += 32) atomicAdd(s_cnt + slope_bucket<NB>(s_ka[i]), 1u);
            __syncwarp();
            s_order = s_va;
            if (warp_bucket_scan<NB>(s_cnt, n, lane)) {
                for (int i = lane; i < n; i += 32) {
                    const uint32_t k = s_ka[i];
                    s_list[atomicAdd(s_cnt + slope_bucket<NB>(k), 1u)] = (uint64_t)k << 32 | (uint32_t)i << 16 | s_va[i];
                }
                __syncwarp();
                for (int j = lane; j < n; j += 32) {
                    const uint64_t e = s_list[j];
                    const int b = slope_bucket<NB>((uint32_t)(e >> 32)), q0 = b ? (int)s_cnt[b - 1] : 0, q1 = (int)s_cnt[b];
                    int at = q0;
                    for (int q = q0; q < q1; q++) at += s_list[q] < e;
                    s_va[at] = (uint16_t)e;
                }
            } else {
                warp_radix_sort32(s_ka, s_va, s_kb, s_vb, n, s_hist, lane);
            }
            __syncwarp();
        }

        // cumulative weighted moments in angle order (fast/quads.c:968-1035):
        // the six terms of each position (moment_terms), then lane q < 6
        // turns row q into its prefix sums
        double *M0 = GP ? scr.mx + s0 : pm, *M1 = GP ? scr.my + s0 : pm + RS, *M2 = GP ? scr.mxx + s0 : pm + 2 * RS,
               *M3 = GP ? scr.mxy + s0 : pm + 3 * RS, *M4 = GP ? scr.myy + s0 : pm + 4 * RS,
               *M5 = GP ? scr.mw + s0 : pm + 5 * RS;
        const uint8_t *im = qim + f.q_off;
        if constexpr (GP) {
            // the prefix arrays are in global memory: chunks of 64 points in
            // shared memory (x0), two a lane; a chunk's gathers are under way
            // while the chain of the one before runs (point values two chunks
            // ahead, pixels one). With the terms and the chain in global
            // memory the moments took 77k cycles for 360 points.
            double *buf = reinterpret_cast<double *>(x0);
            constexpr int BS = 66;  // row stride: the six rows on distinct banks
            static_assert(6 * BS <= CAP, "the chunk's terms fit x0");
            auto point = [&](int k) { return k < n ? P[s_order[k]] : 0ull; };
            uint64_t pa = point(lane), pb = point(32 + lane), na = point(64 + lane), nb2 = point(96 + lane);
            int32_t ga = point_grad2(im, f.qw, f.qh, pa), gb = point_grad2(im, f.qw, f.qh, pb);
            double run = 0.0;
            for (int k0 = 0; k0 < n; k0 += 64) {
                double m[6];
                moment_terms(pa, ga, m);
#pragma unroll
                for (int q = 0; q < 6; q++) buf[q * BS + lane] = m[q];
                moment_terms(pb, gb, m);
#pragma unroll
                for (int q = 0; q < 6; q++) buf[q * BS + 32 + lane] = m[q];
                pa = na;
                pb = nb2;
                na = point(k0 + 128 + lane);
                nb2 = point(k0 + 160 + lane);
                ga = point_grad2(im, f.qw, f.qh, pa);
                gb = point_grad2(im, f.qw, f.qh, pb);
                __syncwarp();
                if (lane < 6) prefix_chain(buf + lane * BS, min(64, n - k0), run);
                __syncwarp();
                double *out[6] = {M0, M1, M2, M3, M4, M5};
#pragma unroll
                for (int h = 0; h < 64; h += 32)
                    if (k0 + h + lane < n) {
#pragma unroll
                        for (int q = 0; q < 6; q++) out[q][k0 + h + lane] = buf[q * BS + h + lane];
                    }
                __syncwarp();
            }
        } else {
            for (int k = lane; k < n; k += 64) {
                const int k2 = k + 32 < n ? k + 32 : k;
                const uint64_t *key = reinterpret_cast<const uint64_t *>(M5);
                const uint64_t p1 = P[key[k] & 0x1fffu], p2 = P[key[k2] & 0x1fffu];
                const int32_t g1 = point_grad2(im, f.qw, f.qh, p1), g2 = point_grad2(im, f.qw, f.qh, p2);
                double m1[6], m2[6];
                moment_terms(p1, g1, m1);
                moment_terms(p2, g2, m2);
#pragma unroll
                for (int q = 0; q < 6; q++) {
                    pm[q * RS + k] = m1[q];
                    pm[q * RS + k2] = m2[q];
                }
            }
            __syncwarp();
            if (lane < 6) {
                double run = 0.0;
                prefix_chain(pm + lane * RS, n, run);
            }
        }
        __syncwarp();
        const Moments mo = {M0, M1, M2, M3, M4, M5};
        const MSum all = moments_at(mo, n - 1);

        // corner search (fast/quads.c:788-959)
        const int ksz = min(20, n / 12);
        if (ksz < 2) continue;
        const double nn = (double)(2 * ksz + 1);
        for (int i = lane; i < n; i += 64) {
            const int i2 = i + 32 < n ? i + 32 : i;
            const MSum sa = window_moments(mo, all, n, ksz, i), sb = window_moments(mo, all, n, ksz, i2);
            const double ea = window_error(sa, nn), eb = window_error(sb, nn);
            s_err[i] = ea;
            s_err[i2] = eb;
        }
        __syncwarp();
        for (int i = lane; i < n; i += 64) {
            const int i2 = i + 32 < n ? i + 32 : i;
            const double fa = smooth_at(s_err, n, i, prm.qsm), fb = smooth_at(s_err, n, i2, prm.qsm);
            s_filt[i] = fa;
            s_filt[i2] = fb;
        }
        __syncwarp();
        int nm = 0;
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            bool is_max = false;
            double e = 0.0;
            if (i < n) {
                e = s_filt[i];
                const double lft = s_filt[i == 0 ? n - 1 : i - 1], rgt = s_filt[i + 1 == n ? 0 : i + 1];
                is_max = e > lft && e > rgt;
            }
            const uint32_t bal = __ballot_sync(FULL, is_max);
            if (is_max) {
                const int at = nm + __popc(bal & ((1u << lane) - 1u));
                s_mxi[at] = i;
                s_mxe[at] = e;
            }
            nm += __popc(bal);
        }
        __syncwarp();
        if (nm < 4) continue;
        if (nm > prm.max_nmaxima) {
            // keep e_i when at most max_nmaxima errors are >= e_i (quads.c:827-862)
            const int k = prm.max_nmaxima;
            int kept = 0;
            for (int i0 = 0; i0 < nm; i0 += 32) {
                const int i = i0 + lane;
                bool keep = false;
                int32_t mi = 0;
                if (i < nm) {
                    const double ei = s_mxe[i];
                    int ge = 0;
                    for (int j = 0; j < nm && ge <= k; j++) ge += s_mxe[j] >= ei;
                    keep = ge <= k;
                    mi = s_mxi[i];
                }
                const uint32_t bal = __ballot_sync(FULL, keep);
                __syncwarp();
                if (keep) s_mxi[kept + __popc(bal & ((1u << lane) - 1u))] = mi;
                kept += __popc(bal);
            }
            __syncwarp();
            nm = kept;
        }
        // line fits of pairs of maxima
        for (int t = lane; t < nm * nm; t += 32) {
            const int p = t / nm, q = t - p * nm;
            if (!(p < q || p >= q + 3)) continue;
            const int i0 = s_mxi[p], i1 = s_mxi[q];
            const MSum s = seg_moments(mo, all, i0, i1);
            const double cnt = (double)(i0 <= i1 ? i1 - i0 + 1 : n - i0 + i1 + 1);
            double lp[4], mse;
            line_of(s, lp, &mse);
            s_perr[t] = cnt * mse;
            s_pmse[t] = mse;
            s_pnx[t] = lp[2];
            s_pny[t] = lp[3];
        }
        __syncwarp();
        // the first smallest total error in (m0, m1, m2, m3) order: the
        // smallest (error, m0 m1 m2 m3) over the 4-subsets of the maxima
        double be = inf;
        int bo = 0xffff;
        const int nsub = binom4(nm);
        for (int t = lane; t < nsub; t += 32) {
            const int v = g_quad4.v[t];
            const int m0 = v & 15, m1 = v >> 4 & 15, m2 = v >> 8 & 15, m3 = v >> 12;
            const int p01 = m0 * nm + m1, p12 = m1 * nm + m2;
            if (s_pmse[p01] > prm.max_mse || s_pmse[p12] > prm.max_mse) continue;
            const double dot = s_pnx[p01] * s_pnx[p12] + s_pny[p01] * s_pny[p12];
            if (fabs(dot) > prm.max_dot) continue;
            const int p23 = m2 * nm + m3, p30 = m3 * nm + m0;
            const double e012 = s_perr[p01] + s_perr[p12];
            const double e23 = s_pmse[p23] > prm.max_mse ? inf : s_perr[p23];
            const double e30 = s_pmse[p30] > prm.max_mse ? inf : s_perr[p30];
            const double e = e012 + e23 + e30;
            const int ord = m0 << 12 | m1 << 8 | m2 << 4 | m3;
            if (e < be || (e == be && ord < bo)) {
                be = e;
                bo = ord;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double e2 = __shfl_xor_sync(FULL, be, o);
            const int o2 = __shfl_xor_sync(FULL, bo, o);
            if (e2 < be || (e2 == be && o2 < bo)) {
                be = e2;
                bo = o2;
            }
        }
        if (!(be != inf && be / (double)sz < prm.max_mse)) continue;
        // the 4 line fits, lanes 0-3 (quads.c:1069-1075)
        double ln[4] = {0.0, 0.0, 0.0, 0.0}, lmse = 0.0;
        if (lane < 4) {
            const int ma = bo >> (12 - 4 * lane) & 15, mb = bo >> (12 - 4 * ((lane + 1) & 3)) & 15;
            line_of(seg_moments(mo, all, s_mxi[ma], s_mxi[mb]), ln, &lmse);
        }
        float p[2];
        if (quad_of(lane, ln, lmse, prm, f.tag_width, p) && lane < 4) {
            quads[c].p[lane][0] = p[0];
            quads[c].p[lane][1] = p[1];
            if (lane == 0) {
                quads[c].reversed_border = rev;
                quads[c].frame = cframe[c];
                quad_ok[c] = 1;
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// 9. Decoding, one block per quad (fast/decode.c, fast/detector.c:83-139).

struct DView {
    const uint8_t *im;
    int64_t s, w, h;
};

__device__ __forceinline__ double bil_seq(double a, double b, const uint8_t *p, int64_t s) {
    return (1.0 - a) * (1.0 - b) * p[0] + a * (1.0 - b) * p[1] + (1.0 - a) * b * p[s] + a * b * p[s + 1];
}

__device__ __forceinline__ double bil_vals(double a, double b, int p00, int p01, int p10, int p11) {
    double na = 1.0 - a, nb = 1.0 - b;
    return ((na * nb) * p00 + (a * nb) * p01) + ((na * b) * p10 + (a * b) * p11);
}

// One sample point of edge refinement (fast/decode.c:549-735) gives the
// weighted mean of its steps along the normal. The reference sums the first
// vsteps steps (a multiple of 4) into 4 interleaved partial sums: lane u's
// share, the steps k = u, u + 4, ..., in that order into (ln, lc).
__device__ __forceinline__ void refine_part(const DView &v, double x0, double y0, double nx, double ny, int64_t range,
                                            int64_t vsteps, int u, double *ln, double *lc) {
    const double wl = (double)(v.w - 1), hl = (double)(v.h - 1);
    const bool tiny = v.w < 2 || v.h < 2;
    double sn = 0.0, sc = 0.0;
#pragma unroll 3
    for (int64_t k = u; k < vsteps; k += 4) {
        const double n = (double)-range + 0.25 * (double)k;
        const double x1 = x0 + (n + 1.0) * nx - 0.5, y1 = y0 + (n + 1.0) * ny - 0.5;
        const double x2 = x0 + (n - 1.0) * nx - 0.5, y2 = y0 + (n - 1.0) * ny - 0.5;
        const bool in = x1 > -1.0 && x1 < wl && y1 > -1.0 && y1 < hl && x2 > -1.0 && x2 < wl && y2 > -1.0 && y2 < hl;
        const double tx1 = trunc(x1), ty1 = trunc(y1), tx2 = trunc(x2), ty2 = trunc(y2);
        double wgt = 0.0;
        if (in || !tiny) {
            const uint8_t *p1 = v.im + (in ? (int64_t)ty1 * v.s + (int64_t)tx1 : 0);
            const uint8_t *p2 = v.im + (in ? (int64_t)ty2 * v.s + (int64_t)tx2 : 0);
            const int a0 = p1[0], a1 = p1[1], a2 = p1[v.s], a3 = p1[v.s + 1];
            const int b0 = p2[0], b1 = p2[1], b2 = p2[v.s], b3 = p2[v.s + 1];
            if (in) {
                const double g1 = bil_vals(x1 - tx1, y1 - ty1, a0, a1, a2, a3);
                const double g2 = bil_vals(x2 - tx2, y2 - ty2, b0, b1, b2, b3);
                const double d = g2 - g1;
                wgt = !(g1 < g2) ? d * d : 0.0;
            }
        }
        sn = sn + wgt * n;
        sc = sc + wgt;
    }
    *ln = sn;
    *lc = sc;
}

// The steps after the first vsteps of one sample, in order, added to the
// sums (mn, mc).
__device__ __forceinline__ void refine_tail(const DView &v, double x0, double y0, double nx, double ny, int64_t range,
                                            int64_t vsteps, int64_t nsteps, double *mn, double *mc) {
    for (int64_t k = vsteps; k < nsteps; k++) {
        double n = (double)-range + 0.25 * (double)k;
        double x1 = x0 + (n + 1.0) * nx - 0.5, y1 = y0 + (n + 1.0) * ny - 0.5;
        int64_t x1i = c_int(x1), y1i = c_int(y1);
        if (x1i < 0 || x1i + 1 >= v.w || y1i < 0 || y1i + 1 >= v.h) continue;
        double x2 = x0 + (n - 1.0) * nx - 0.5, y2 = y0 + (n - 1.0) * ny - 0.5;
        int64_t x2i = c_int(x2), y2i = c_int(y2);
        if (x2i < 0 || x2i + 1 >= v.w || y2i < 0 || y2i + 1 >= v.h) continue;
        double g1 = bil_seq(x1 - (double)x1i, y1 - (double)y1i, v.im + y1i * v.s + x1i, v.s);
        double g2 = bil_seq(x2 - (double)x2i, y2 - (double)y2i, v.im + y2i * v.s + x2i, v.s);
        if (g1 < g2) continue;
        double wgt = (g2 - g1) * (g2 - g1);
        *mn = *mn + wgt * n;
        *mc = *mc + wgt;
    }
}

// Correctly rounded f32 trig as the golden vectors need: the double
// function, then one rounding (fast/decode.c:740-744).
__device__ __forceinline__ float cr_atan2f(float y, float x) { return (float)atan2((double)y, (double)x); }
__device__ __forceinline__ float cr_cosf(float x) { return (float)cos((double)x); }
__device__ __forceinline__ float cr_sinf(float x) { return (float)sin((double)x); }

// Homography of 4 correspondences by one warp: the 8x9 Gaussian elimination
// with partial pivoting of fast/decode.c:114-165. Lane l holds row l / 4,
// columns l % 4 and l % 4 + 4 (and column 8 when l % 4 == 0). Each cell
// takes the same operations as in the sequential elimination, so the result
// is the same; the pivot is the first largest |a[r][col]|, r >= col, as the
// scan for a strictly larger value finds it. The back substitution runs on
// lane 0 from shared memory (m: 72 doubles). Returns false on a failed pivot
// check, on every lane. The loops stay rolled: this runs once per quad, so
// its code size is its cost.
__device__ __noinline__ bool homography_warp(const float (*p)[2], double *m, double H[9], int lane) {
    const unsigned FULL = 0xffffffffu;
    const int r = lane >> 2, g = lane & 3;
    double cell[3];
    {
        const int i = r >> 1;
        const double x = i == 0 || i == 3 ? -1.0 : 1.0, y = i == 0 || i == 1 ? -1.0 : 1.0;
        const double X = (double)p[i][0], Y = (double)p[i][1];
#pragma unroll
        for (int sl = 0; sl < 3; sl++) {
            const int col = sl == 2 ? 8 : g + 4 * sl;
            double v = 0.0;
            if ((r & 1) == 0) {
                v = col == 0 ? x : col == 1 ? y : col == 2 ? 1.0 : col == 6 ? -x * X : col == 7 ? -y * X : col == 8 ? X : 0.0;
            } else {
                v = col == 3 ? x : col == 4 ? y : col == 5 ? 1.0 : col == 6 ? -x * Y : col == 7 ? -y * Y : col == 8 ? Y : 0.0;
            }
            cell[sl] = v;
        }
    }
    bool ok = true;
#pragma unroll 1
    for (int col = 0; col < 8; col++) {
        const int cg = col & 3, cs = col >> 2;
        // pivot: the largest |a[r][col]| over r >= col, first r on ties
        double v = -1.0;
        if (g == cg && r >= col) {
            const double a = fabs(cs ? cell[1] : cell[0]);
            if (a == a) v = a;
        }
        int pr = r;
        for (int o = 16; o > 0; o >>= 1) {
            const double v2 = __shfl_xor_sync(FULL, v, o);
            const int r2 = __shfl_xor_sync(FULL, pr, o);
            if (v2 > v || (v2 == v && r2 < pr)) {
                v = v2;
                pr = r2;
            }
        }
        if (!(v > 0.0) || v < 1e-10) ok = false;
        const int piv = v > 0.0 ? pr : col;
        // swap rows col and piv (their columns left of col are zero in both)
        const int src = r == col ? 4 * piv + g : r == piv ? 4 * col + g : lane;
#pragma unroll
        for (int sl = 0; sl < 3; sl++) cell[sl] = __shfl_sync(FULL, cell[sl], src);
        // eliminate below the pivot
        const double pv = __shfl_sync(FULL, cs ? cell[1] : cell[0], 4 * col + cg);
        const double mine = cs ? cell[1] : cell[0];
        const double fct = __shfl_sync(FULL, mine / pv, 4 * r + cg);
        double prow[3];
#pragma unroll
        for (int sl = 0; sl < 3; sl++) prow[sl] = __shfl_sync(FULL, cell[sl], 4 * col + g);
        if (r > col) {
#pragma unroll
            for (int sl = 0; sl < 3; sl++) {
                const int cc = sl == 2 ? 8 : g + 4 * sl;
                if (sl == 2 && g != 0) continue;
                if (cc == col)
                    cell[sl] = 0.0;
                else if (cc > col)
                    cell[sl] = cell[sl] - fct * prow[sl];
            }
        }
    }
    m[r * 9 + g] = cell[0];
    m[r * 9 + g + 4] = cell[1];
    if (g == 0) m[r * 9 + 8] = cell[2];
    __syncwarp();
    if (ok && lane == 0) {
#pragma unroll 1
        for (int col = 7; col >= 0; col--) {
            double s = 0.0;
#pragma unroll 1
            for (int i = col + 1; i < 8; i++) s = s + m[col * 9 + i] * m[i * 9 + 8];
            m[col * 9 + 8] = (m[col * 9 + 8] - s) / m[col * 9 + col];
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; i++) H[i] = m[i * 9 + 8];
    H[8] = 1.0;
    return ok;
}

// Invertibility as the C library's PLU decomposition decides it
// (fast/decode.c:168-196).
__device__ bool invertible3(const double m[9]) {
    double lu[9];
    for (int i = 0; i < 9; i++) lu[i] = m[i];
    for (int j = 0; j < 3; j++) {
        for (int i = 0; i < 3; i++) {
            int kmax = i < j ? i : j;
            double acc = 0.0;
            for (int k = 0; k < kmax; k++) acc = acc + lu[i * 3 + k] * lu[k * 3 + j];
            lu[i * 3 + j] = lu[i * 3 + j] - acc;
        }
        int p = j;
        for (int i = j + 1; i < 3; i++)
            if (fabs(lu[i * 3 + j]) > fabs(lu[p * 3 + j])) p = i;
        if (p != j)
            for (int k = 0; k < 3; k++) {
                double t = lu[p * 3 + k];
                lu[p * 3 + k] = lu[j * 3 + k];
                lu[j * 3 + k] = t;
            }
        double d = lu[j * 3 + j];
        if (fabs(d) < 1e-8) return false;
        if (d != 0.0) {
            double inv = 1.0 / d;
            for (int i = j + 1; i < 3; i++) lu[i * 3 + j] = lu[i * 3 + j] * inv;
        }
    }
    return true;
}

__device__ __forceinline__ void project(const double H[9], double x, double y, double *ox, double *oy) {
    double xx = H[0] * x + H[1] * y + H[2];
    double yy = H[3] * x + H[4] * y + H[5];
    double zz = H[6] * x + H[7] * y + H[8];
    *ox = xx / zz;
    *oy = yy / zz;
}

struct GrayModel {
    double a[9], b[3], c[3];
};

// mat33_sym_solve as the C library does it (fast/decode.c:241-265).
__device__ __forceinline__ void gm_solve(GrayModel *g) {
    const double *a = g->a;
    double L0 = sqrt(a[0]);
    double L3 = a[1] / L0;
    double L6 = a[2] / L0;
    double L4 = sqrt(a[4] - L3 * L3);
    double L7 = (a[5] - L3 * L6) / L4;
    double L8 = sqrt(a[8] - L6 * L6 - L7 * L7);
    double M0 = 1.0 / L0;
    double M3 = -L3 * M0 / L4;
    double M4 = 1.0 / L4;
    double M6 = (-L6 * M0 - L7 * M3) / L8;
    double M7 = -L7 * M4 / L8;
    double M8 = 1.0 / L8;
    const double *b = g->b;
    double t0 = M0 * b[0];
    double t1 = M3 * b[0] + M4 * b[1];
    double t2 = M6 * b[0] + M7 * b[1] + M8 * b[2];
    g->c[0] = M0 * t0 + M3 * t1 + M6 * t2;
    g->c[1] = M4 * t1 + M7 * t2;
    g->c[2] = M8 * t2;
}

__device__ __forceinline__ double bilinear_at(const DView &v, double px, double py) {
    int64_t x1 = c_int(floor(px - 0.5)), x2 = c_int(ceil(px - 0.5));
    double x = px - 0.5 - (double)x1;
    int64_t y1 = c_int(floor(py - 0.5)), y2 = c_int(ceil(py - 0.5));
    double y = py - 0.5 - (double)y1;
    if (x1 < 0 || x2 >= v.w || y1 < 0 || y2 >= v.h) return -1.0;
    const uint8_t *r1 = v.im + y1 * v.s, *r2 = v.im + y2 * v.s;
    return r1[x1] * (1.0 - x) * (1.0 - y) + r1[x2] * x * (1.0 - y) + r2[x1] * (1.0 - x) * y + r2[x2] * x * y;
}

__device__ __forceinline__ uint64_t rot90(uint64_t w0, int64_t nbits) {
    int64_t p = nbits, l = 0;
    if (nbits % 4 == 1) {
        p = nbits - 1;
        l = 1;
    }
    uint64_t w = ((w0 >> l) << (p / 4 + l)) | (w0 >> (3 * p / 4 + l) << l) | (w0 & (uint64_t)l);
    return w & ((nbits >= 64) ? ~0ull : (((uint64_t)1 << nbits) - 1));
}

// The first code within maxham bits, by rotation, then chunk, then code
// index (fast/decode.c:87-107). Returns id | hamming << 16 | rot << 24.
__device__ uint32_t qd_lookup(const GpuFamily &F, uint64_t rcode, int lane) {
    // lane 4 r + j (r rotations, chunk j) scans its bucket; the first lane
    // with a match holds the first match in the sequential order
    const uint64_t mask = (uint64_t)F.cap - 1;
    uint32_t res = 0xffffffffu;
    if (lane < 16) {
        const int r = lane >> 2, j = lane & 3;
        uint64_t rc = rcode;
        for (int t = 0; t < r; t++) rc = rot90(rc, F.nbits);
        const int64_t val = (int64_t)((rc >> (j * F.chunk)) & mask);
        const int64_t ob = j * (F.cap + 1) + val, base = j * F.ncodes;
        for (int64_t e = base + F.off[ob]; e < base + F.off[ob + 1]; e++) {
            const int hd = __popcll(F.codes[e] ^ rc);
            if (hd <= F.maxham) {
                res = (uint32_t)F.idx[e] | (uint32_t)hd << 16 | (uint32_t)r << 24;
                break;
            }
        }
    }
    const uint32_t found = __ballot_sync(0xffffffffu, res != 0xffffffffu);
    if (!found) return 65535u | 255u << 16;
    return __shfl_sync(0xffffffffu, res, __ffs(found) - 1);
}

#define REF_CHUNK 128

__global__ void __launch_bounds__(AT_DEC_THREADS) k_refine(const FrameDesc *frames, GpuParams prm,
                                                              const uint8_t *img, const uint8_t *qim,
                                                              const GpuQuad *quads, const uint32_t *nq, float *corners,
                                                              uint32_t *det_ok) {
    kernel_begin();
    const int64_t nquads = *nq;
    __shared__ float s_p[4][2];
    __shared__ double s_lines[4][4];
    __shared__ double s_bx[REF_CHUNK], s_by[REF_CHUNK];
    __shared__ int s_bok[REF_CHUNK];
    __shared__ double s_enx[4], s_eny[4];
    __shared__ int64_t s_ens[4];
    const int tid = threadIdx.x;
    for (int64_t qi = blockIdx.x; qi < nquads; qi += gridDim.x) {
        const GpuQuad q = quads[qi];
        const FrameDesc f = frames[q.frame];
        DView v;
        if (prm.decode_blurred)
            v = DView{qim + f.q_off, (int64_t)f.qw, (int64_t)f.qw, (int64_t)f.qh};
        else
            v = DView{f.img, f.stride, (int64_t)f.w, (int64_t)f.h};
        if (tid < 8) {
            float val = q.p[tid >> 1][tid & 1];
            if (prm.quad_decimate > 1.0f) val = __fmul_rn(val, prm.quad_decimate);
            s_p[tid >> 1][tid & 1] = val;
        }
        for (int fi = tid; fi < prm.nfam; fi += blockDim.x) det_ok[qi * prm.nfam + fi] = 0;
        __syncthreads();
        if (prm.refine_edges) {
            // fast/decode.c:657-761. The 4 edges are independent until the
            // corners are moved: their sample points, one per thread, are
            // refined together, and thread e < 4 sums edge e's in order.
            const int64_t range = (int64_t)__fadd_rn(prm.quad_decimate, 1.0f);
            const int64_t nsteps = 2 * 4 * range + 1;
            const int64_t vsteps = nsteps - nsteps % 4;
            if (tid < 4) {
                int a = tid, b = (tid + 1) & 3;
                double nx = (double)__fsub_rn(s_p[b][1], s_p[a][1]);
                double ny = (double)__fadd_rn(-s_p[b][0], s_p[a][0]);
                double mag = sqrt(nx * nx + ny * ny);
                nx = nx / mag;
                ny = ny / mag;
                if (q.reversed_border) {
                    nx = -nx;
                    ny = -ny;
                }
                s_enx[tid] = nx;
                s_eny[tid] = ny;
                s_ens[tid] = dmax(16, c_int(mag / 8.0));
            }
            __syncthreads();
            // the 4 edges' samples in one packed range, edge after edge
            const int64_t o1 = s_ens[0], o2 = o1 + s_ens[1], o3 = o2 + s_ens[2], total = o3 + s_ens[3];
            double mx = 0.0, my = 0.0, mxx = 0.0, mxy = 0.0, myy = 0.0, cnt = 0.0;
            for (int64_t c0 = 0; c0 < total; c0 += REF_CHUNK) {
                // four lanes per sample, lane u summing partial sum u
                const int u = tid & 3;
                for (int w0 = 0; w0 < REF_CHUNK; w0 += (int)(blockDim.x >> 2)) {
                    const int w = w0 + (tid >> 2);
                    const int64_t gi = c0 + w;
                    const bool valid = w < REF_CHUNK && gi < total;
                    double ln = 0.0, lc = 0.0, x0 = 0.0, y0 = 0.0, nx = 0.0, ny = 0.0;
                    if (valid) {
                        const int e = gi < o1 ? 0 : gi < o2 ? 1 : gi < o3 ? 2 : 3;
                        const int64_t si = gi - (e == 0 ? 0 : e == 1 ? o1 : e == 2 ? o2 : o3), ns = s_ens[e];
                        const int a = e, b = (e + 1) & 3;
                        nx = s_enx[e];
                        ny = s_eny[e];
                        double alpha = (1.0 + (double)si) / (double)(ns + 1);
                        x0 = alpha * (double)s_p[a][0] + (1.0 - alpha) * (double)s_p[b][0];
                        y0 = alpha * (double)s_p[a][1] + (1.0 - alpha) * (double)s_p[b][1];
                        refine_part(v, x0, y0, nx, ny, range, vsteps, u, &ln, &lc);
                    }
                    const double ln0 = __shfl_sync(0xffffffffu, ln, 0, 4), ln1 = __shfl_sync(0xffffffffu, ln, 1, 4),
                                 ln2 = __shfl_sync(0xffffffffu, ln, 2, 4), ln3 = __shfl_sync(0xffffffffu, ln, 3, 4);
                    const double lc0 = __shfl_sync(0xffffffffu, lc, 0, 4), lc1 = __shfl_sync(0xffffffffu, lc, 1, 4),
                                 lc2 = __shfl_sync(0xffffffffu, lc, 2, 4), lc3 = __shfl_sync(0xffffffffu, lc, 3, 4);
                    if (valid && u == 0) {
                        double mn = 0.0 + ((ln0 + ln2) + (ln1 + ln3));
                        double mc = 0.0 + ((lc0 + lc2) + (lc1 + lc3));
                        refine_tail(v, x0, y0, nx, ny, range, vsteps, nsteps, &mn, &mc);
                        const bool ok = mc != 0.0;
                        s_bok[w] = ok;
                        if (ok) {
                            const double n0 = mn / mc;
                            s_bx[w] = x0 + n0 * nx;
                            s_by[w] = y0 + n0 * ny;
                        }
                    }
                }
                __syncthreads();
                if (tid < 4) {
                    const int64_t eo = tid == 0 ? 0 : tid == 1 ? o1 : tid == 2 ? o2 : o3, ee = eo + s_ens[tid];
                    const int64_t lo = dmax(eo, c0), hi = dmin(ee, c0 + REF_CHUNK);
                    for (int64_t gi = lo; gi < hi; gi++) {
                        const int64_t t = gi - c0;
                        if (!s_bok[t]) continue;
                        double bx = s_bx[t], by = s_by[t];
                        mx = mx + bx;
                        my = my + by;
                        mxx = mxx + bx * bx;
                        mxy = mxy + bx * by;
                        myy = myy + by * by;
                        cnt = cnt + 1.0;
                    }
                }
                __syncthreads();
            }
            if (tid < 4) {
                double ex = mx / cnt, ey = my / cnt;
                double cxx = mxx / cnt - ex * ex, cxy = mxy / cnt - ex * ey, cyy = myy / cnt - ey * ey;
                double theta = 0.5 * (double)cr_atan2f((float)(-2.0 * cxy), (float)(cyy - cxx));
                s_lines[tid][0] = ex;
                s_lines[tid][1] = ey;
                s_lines[tid][2] = (double)cr_cosf((float)theta);
                s_lines[tid][3] = (double)cr_sinf((float)theta);
            }
            __syncthreads();
            if (tid == 0) {
                for (int i = 0; i < 4; i++) {
                    int j = (i + 1) & 3;
                    double a00 = s_lines[i][3], a01 = -s_lines[j][3], a10 = -s_lines[i][2], a11 = s_lines[j][2];
                    double b0 = -s_lines[i][0] + s_lines[j][0], b1 = -s_lines[i][1] + s_lines[j][1];
                    double det = a00 * a11 - a10 * a01;
                    if (fabs(det) > 0.001) {
                        double w00 = a11 / det, w01 = -a01 / det;
                        double l0 = w00 * b0 + w01 * b1;
                        s_p[j][0] = (float)(s_lines[i][0] + l0 * a00);
                        s_p[j][1] = (float)(s_lines[i][1] + l0 * a10);
                    }
                }
            }
            __syncthreads();
        }
        if (tid < 8) corners[qi * 8 + tid] = s_p[tid >> 1][tid & 1];
        __syncthreads();
    }
}

// The homography of each quad's corners (fast/decode.c:114-196), a warp
// per quad: H, and whether it was found and is invertible.
#define QH_WARPS 4
__global__ void __launch_bounds__(QH_WARPS * 32) k_quad_homography(const float *corners, const uint32_t *nq, double *hs,
                                                                     uint32_t *hok) {
    kernel_begin();
    const int64_t nquads = *nq;
    __shared__ float s_p[QH_WARPS][4][2];
    __shared__ double s_hm[QH_WARPS][72];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int64_t qi = (int64_t)blockIdx.x * QH_WARPS + w; qi < nquads; qi += (int64_t)gridDim.x * QH_WARPS) {
        if (lane < 8) s_p[w][lane >> 1][lane & 1] = corners[qi * 8 + lane];
        __syncwarp();
        double H[9];
        const bool ok = homography_warp(s_p[w], s_hm[w], H, lane);
        if (lane == 0) {
            hok[qi] = ok && invertible3(H);
#pragma unroll
            for (int i = 0; i < 9; i++) hs[qi * 9 + i] = H[i];
        }
        __syncwarp();
    }
}

// A block per quad. Most of its time goes to one warp (gray models, bit sums,
// lookup), so it has only one more for the 64 border samples and the bits: 42
// us for 32 frames of 1920 x 1080, with blocks of 128 threads 55.
#define DECODE_THREADS 64
__global__ void __launch_bounds__(DECODE_THREADS, 12) k_decode(const FrameDesc *frames, GpuParams prm,
                                                              const GpuFamily *fams, const uint8_t *img,
                                                              const uint8_t *qim, const GpuQuad *quads,
                                                              const uint32_t *nq, const double *hs, const uint32_t *hok,
                                                              GpuDetection *dets, uint32_t *det_ok) {
    kernel_begin();
    const int64_t nquads = *nq;
    __shared__ double s_H[9];
    __shared__ double s_gx[8 * AT_MAX_TW], s_gy[8 * AT_MAX_TW], s_gv[8 * AT_MAX_TW];
    __shared__ int s_gk[8 * AT_MAX_TW];
    __shared__ double s_wc[3], s_bc[3];
    __shared__ int s_pol;
    __shared__ double s_vals[AT_MAX_TW * AT_MAX_TW], s_sharp[AT_MAX_TW * AT_MAX_TW];
    const int tid = threadIdx.x;
    for (int64_t qi = blockIdx.x; qi < nquads; qi += gridDim.x) {
        if (!hok[qi]) continue;
        const GpuQuad q = quads[qi];
        const FrameDesc f = frames[q.frame];
        DView v;
        if (prm.decode_blurred)
            v = DView{qim + f.q_off, (int64_t)f.qw, (int64_t)f.qw, (int64_t)f.qh};
        else
            v = DView{f.img, f.stride, (int64_t)f.w, (int64_t)f.h};
        __syncthreads();
        if (tid < 9) s_H[tid] = hs[qi * 9 + tid];
        __syncthreads();
        for (int fi = 0; fi < prm.nfam; fi++) {
            const GpuFamily &F = fams[fi];
            if (F.reversed_border != q.reversed_border) continue;
            if (!(f.fam_mask >> fi & 1u)) continue;
            // border gray models (fast/decode.c:291-337): 8 patterns x wab
            const int32_t wab = F.wab;
            const float wf = (float)wab;
            for (int t = tid; t < 8 * wab; t += blockDim.x) {
                int pi = t / wab, i = t - pi * wab;
                float pat[5];
                switch (pi) {
                case 0: pat[0] = -0.5f, pat[1] = 0.5f, pat[2] = 0.0f, pat[3] = 1.0f; break;
                case 1: pat[0] = 0.5f, pat[1] = 0.5f, pat[2] = 0.0f, pat[3] = 1.0f; break;
                case 2: pat[0] = (float)(wab + 0.5), pat[1] = 0.5f, pat[2] = 0.0f, pat[3] = 1.0f; break;
                case 3: pat[0] = (float)(wab - 0.5), pat[1] = 0.5f, pat[2] = 0.0f, pat[3] = 1.0f; break;
                case 4: pat[0] = 0.5f, pat[1] = -0.5f, pat[2] = 1.0f, pat[3] = 0.0f; break;
                case 5: pat[0] = 0.5f, pat[1] = 0.5f, pat[2] = 1.0f, pat[3] = 0.0f; break;
                case 6: pat[0] = 0.5f, pat[1] = (float)(wab + 0.5), pat[2] = 1.0f, pat[3] = 0.0f; break;
                default: pat[0] = 0.5f, pat[1] = (float)(wab - 0.5), pat[2] = 1.0f, pat[3] = 0.0f; break;
                }
                double tx01 = (double)__fdiv_rn(__fadd_rn(pat[0], __fmul_rn((float)i, pat[2])), wf);
                double ty01 = (double)__fdiv_rn(__fadd_rn(pat[1], __fmul_rn((float)i, pat[3])), wf);
                double tx = 2.0 * (tx01 - 0.5), ty = 2.0 * (ty01 - 0.5);
                double zz = s_H[6] * tx + s_H[7] * ty + s_H[8];
                double px = (s_H[0] * tx + s_H[1] * ty + s_H[2]) / zz;
                double py = (s_H[3] * tx + s_H[4] * ty + s_H[5]) / zz;
                int64_t ix = c_int(px), iy = c_int(py);
                int keep = !(ix < 0 || iy < 0 || ix >= v.w || iy >= v.h);
                s_gk[t] = keep;
                s_gx[t] = tx;
                s_gy[t] = ty;
                s_gv[t] = keep ? (double)v.im[iy * v.s + ix] : 0.0;
            }
            __syncthreads();
            if (tid < 32) {
                // the white model (even patterns) in even lanes, the black
                // one (odd patterns) in odd ones, one of the nine sums a lane,
                // in pattern order; then lanes 0 and 1 get theirs and solve.
                // (All nine in one lane took each sample 15 FP64 instructions
                // with two lanes busy.)
                const int acc = tid >> 1;
                const bool ux = acc < 3 || acc == 6, uy = acc == 3 || acc == 4 || acc == 7;
                const bool vx = acc == 0, vy = acc == 1 || acc == 3, vv = acc == 6 || acc == 7;
                const double *pu = ux ? s_gx : uy ? s_gy : s_gv, *pv = vx ? s_gx : vy ? s_gy : s_gv;
                double sum = 0.0;
                if (tid < 18)
                    for (int pi = tid & 1; pi < 8; pi += 2)
                        for (int t = pi * wab; t < (pi + 1) * wab; t++) {
                            const double u = acc == 5 ? 1.0 : pu[t], v = vx || vy || vv ? pv[t] : 1.0;
                            const double next = sum + u * v;
                            sum = s_gk[t] ? next : sum;
                        }
                GrayModel gm;
                gm.a[3] = gm.a[6] = gm.a[7] = 0.0;
                {
                    const int m = tid & 1;
                    gm.a[0] = __shfl_sync(0xffffffffu, sum, m);
                    gm.a[1] = __shfl_sync(0xffffffffu, sum, m + 2);
                    gm.a[2] = __shfl_sync(0xffffffffu, sum, m + 4);
                    gm.a[4] = __shfl_sync(0xffffffffu, sum, m + 6);
                    gm.a[5] = __shfl_sync(0xffffffffu, sum, m + 8);
                    gm.a[8] = __shfl_sync(0xffffffffu, sum, m + 10);
                    gm.b[0] = __shfl_sync(0xffffffffu, sum, m + 12);
                    gm.b[1] = __shfl_sync(0xffffffffu, sum, m + 14);
                    gm.b[2] = __shfl_sync(0xffffffffu, sum, m + 16);
                }
                if (tid == 0 || (tid == 1 && wab > 1)) {
                    gm_solve(&gm);
                } else {
                    gm.c[0] = 0.0;
                    gm.c[1] = 0.0;
                    gm.c[2] = gm.b[2] / 4.0;
                }
                const double ci = gm.c[0] * 0.0 + gm.c[1] * 0.0 + gm.c[2];
                const double bi = __shfl_sync(0xffffffffu, ci, 1);
                if (tid == 0) s_pol = (ci - bi < 0.0) == (F.reversed_border != 0);
                if (tid < 2)
                    for (int i = 0; i < 3; i++) (tid == 0 ? s_wc : s_bc)[i] = gm.c[i];
            }
            __syncthreads();
            if (!s_pol) continue;
            // bit values less the local threshold, sharpened (decode.c:340-377)
            const int64_t tw = F.tw;
            const int64_t minc = (wab - tw) / 2;
            for (int64_t t = tid; t < tw * tw; t += blockDim.x) s_vals[t] = 0.0;
            __syncthreads();
            for (int64_t i = tid; i < F.nbits; i += blockDim.x) {
                int64_t bx = F.bit_x[i], by = F.bit_y[i];
                double tx = 2.0 * (((double)bx + 0.5) / wab - 0.5), ty = 2.0 * (((double)by + 0.5) / wab - 0.5);
                double zz = s_H[6] * tx + s_H[7] * ty + s_H[8];
                double px = (s_H[0] * tx + s_H[1] * ty + s_H[2]) / zz;
                double py = (s_H[3] * tx + s_H[4] * ty + s_H[5]) / zz;
                double val = bilinear_at(v, px, py);
                if (val == -1.0) continue;
                double thr = ((s_bc[0] * tx + s_bc[1] * ty + s_bc[2]) + (s_wc[0] * tx + s_wc[1] * ty + s_wc[2])) / 2.0;
                s_vals[tw * (by - minc) + (bx - minc)] = val - thr;
            }
            __syncthreads();
            for (int64_t t = tid; t < tw * tw; t += blockDim.x) {
                int64_t y = t / tw, x = t - y * tw;
                double acc = 0.0;
                if (y > 0) acc = acc + -s_vals[(y - 1) * tw + x];
                if (x > 0) acc = acc + -s_vals[y * tw + x - 1];
                acc = acc + s_vals[y * tw + x] * 4.0;
                if (x + 1 < tw) acc = acc + -s_vals[y * tw + x + 1];
                if (y + 1 < tw) acc = acc + -s_vals[(y + 1) * tw + x];
                s_sharp[t] = acc;
            }
            __syncthreads();
            if (tid < 32) {
                // the bits a lane each; then lane 0 sums the white ones in
                // order and lane 1 the black ones (one lane for all of it
                // took 3 us a quad of 36 bits)
                uint64_t white = 0;
                for (int i0 = 0; i0 < F.nbits; i0 += 32) {
                    const int i = i0 + tid;
                    double vv = 0.0;
                    if (i < F.nbits) {
                        const int64_t cell = (F.bit_y[i] - minc) * tw + (F.bit_x[i] - minc);
                        vv = s_vals[cell] + prm.decode_sharpening * s_sharp[cell];
                        s_gx[i] = vv;
                    }
                    white |= (uint64_t)__ballot_sync(0xffffffffu, vv > 0.0) << i0;
                }
                __syncwarp();
                const uint64_t all = F.nbits > 0 ? ~0ull >> (64 - F.nbits) : 0ull;
                const uint64_t rcode = F.nbits > 0 ? __brevll(white) >> (64 - F.nbits) : 0ull;
                float sum = 0.0f;
                if (tid < 2) {
                    uint64_t m = tid == 0 ? white : ~white & all;
                    double next = m ? s_gx[__ffsll(m) - 1] : 0.0;
                    while (m) {
                        const double vv = next;
                        m &= m - 1;
                        if (m) next = s_gx[__ffsll(m) - 1];
                        sum = (float)(tid == 0 ? (double)sum + vv : (double)sum - vv);
                    }
                }
                const float ws = sum, bs = __shfl_sync(0xffffffffu, sum, 1);
                const float wc = (float)(1 + __popcll(white)), bc = (float)(1 + F.nbits - __popcll(white));
                const uint32_t lk = qd_lookup(F, rcode, tid);
                double x = (double)__fdiv_rn(ws, wc), y = (double)__fdiv_rn(bs, bc);
                double m = x != x ? y : y != y ? x : x < y ? x : y;  // fmin
                float margin = (float)m;
                int64_t id = lk & 0xffff, ham = (lk >> 16) & 0xff, rot = lk >> 24;
                if (tid == 0 && margin >= 0.0f && ham < 255) {
                    // H = qH * R(rot * pi/2) (fast/detector.c:83-107)
                    double c = prm.rot_cs[rot][0], s = prm.rot_cs[rot][1];
                    const double r[9] = {c, -s, 0.0, s, c, 0.0, 0.0, 0.0, 1.0};
                    GpuDetection d;
                    for (int i = 0; i < 3; i++)
                        for (int j = 0; j < 3; j++) {
                            double acc = 0.0;
                            for (int k = 0; k < 3; k++) acc = acc + s_H[i * 3 + k] * r[k * 3 + j];
                            d.H[i * 3 + j] = acc;
                        }
                    d.family = fi;
                    d.id = (int32_t)id;
                    d.hamming = (int32_t)ham;
                    d.decision_margin = margin;
                    project(d.H, 0.0, 0.0, &d.c[0], &d.c[1]);
                    for (int i = 0; i < 4; i++) {
                        double tx = i == 1 || i == 2 ? 1.0 : -1.0;
                        double ty = i < 2 ? 1.0 : -1.0;
                        project(d.H, tx, ty, &d.p[i][0], &d.p[i][1]);
                    }
                    dets[qi * prm.nfam + fi] = d;
                    det_ok[qi * prm.nfam + fi] = 1;
                }
            }
            __syncthreads();
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// 10. Per frame: gather the detections in (quad, family) order, remove
// overlapping detections of one tag (fast/decode.c:766-891), stable sort by
// id (fast/detector.c:164-179). A block per frame.

struct GLine {
    double p[2], u[2];
};

__device__ GLine gline_of(const double *p0, const double *p1) {
    double u0 = p1[0] - p0[0], u1 = p1[1] - p0[1];
    double mag = (double)__fsqrt_rn((float)(u0 * u0 + u1 * u1));
    GLine l;
    l.p[0] = p0[0];
    l.p[1] = p0[1];
    l.u[0] = u0 / mag;
    l.u[1] = u1 / mag;
    return l;
}
__device__ __forceinline__ double gline_coord(const GLine &l, const double *q) {
    return (q[0] - l.p[0]) * l.u[0] + (q[1] - l.p[1]) * l.u[1];
}
__device__ bool segments_cross(const double *a0, const double *a1, const double *b0, const double *b1) {
    GLine la = gline_of(a0, a1), lb = gline_of(b0, b1);
    double m00 = la.u[0], m01 = -lb.u[0], m10 = la.u[1], m11 = -lb.u[1];
    double det = m00 * m11 - m01 * m10;
    if (fabs(det) < 0.00000001) return false;
    double i00 = m11 / det, i01 = -m01 / det;
    double b00 = lb.p[0] - la.p[0], b10 = lb.p[1] - la.p[1];
    double x00 = i00 * b00 + i01 * b10;
    double t[2] = {la.u[0] * x00 + la.p[0], la.u[1] * x00 + la.p[1]};
    double a = gline_coord(la, la.p), b = gline_coord(la, a1), c = gline_coord(la, t);
    if ((c < a && c < b) || (c > a && c > b)) return false;
    a = gline_coord(lb, lb.p);
    b = gline_coord(lb, b1);
    c = gline_coord(lb, t);
    if ((c < a && c < b) || (c > a && c > b)) return false;
    return true;
}
__device__ bool poly_contains(const double (*poly)[2], const double *q) {
    int last = 0, acc = 0;
    for (int i = 0; i < 5; i++) {
        const double *p = poly[i % 4];
        int quad = p[0] < q[0] ? (p[1] < q[1] ? 2 : 1) : (p[1] < q[1] ? 3 : 0);
        if (i > 0) {
            int dq = quad - last;
            if (dq == -3 || dq == 1)
                acc++;
            else if (dq == -1 || dq == 3)
                acc--;
            else if (dq == -2 || dq == 2) {
                const double *p0 = poly[i - 1];
                double nx = p[1] - q[1], ny = -p[0] + q[0];
                double dot = nx * (p0[0] - q[0]) + ny * (p0[1] - q[1]);
                acc += dot < 0.0 ? -2 : 2;
            }
        }
        last = quad;
    }
    return acc >= 2 || acc <= -2;
}
// Whether two quads overlap, by a warp: an edge pair or a containment a lane.
__device__ bool quads_overlap(const double (*pa)[2], const double (*pb)[2]) {
    const int l = threadIdx.x & 31;
    bool x = false;
    if (l < 16) {
        x = segments_cross(pa[l >> 2], pa[((l >> 2) + 1) & 3], pb[l & 3], pb[((l & 3) + 1) & 3]);
    } else if (l < 18) {
        const double(*in)[2] = l == 16 ? pb : pa, (*poly)[2] = l == 16 ? pa : pb;
        const double q[2] = {(in[0][0] + in[1][0] + in[2][0]) / 3.0, (in[0][1] + in[1][1] + in[2][1]) / 3.0};
        x = poly_contains(poly, q);
    }
    return __any_sync(0xffffffffu, x);
}
__device__ __forceinline__ int prefer(int pref, double a, double b) {
    return pref ? pref : a < b ? -1 : b < a ? 1 : 0;
}

// The bucket count of the reference's cluster table for a quad image of
// w x h at one thread (fast/clusters.c:97-103, fast/detector.c:223).
__device__ __forceinline__ uint64_t ref_buckets(int64_t w, int64_t h) {
    const int64_t chunk = 1 + (h - 1) / 6;
    int64_t n = 1024;
    while (n < chunk * w / 64 && n < 65536) n <<= 1;
    return (uint64_t)n;
}

// One block per frame. Overlap removal only ever drops a detection in favour
// of another with the same (family, id), and its outcome for one such
// group depends only on that group's detections in quad order; so the
// groups are resolved independently (a warp each, the rare groups of
// two or more), and the survivors are placed by their stable rank by id.
__global__ void k_finalize(int nframes, const int64_t *frame_qstart, int nfam, const GpuDetection *dets,
                           const uint32_t *det_ok, uint32_t *idx, uint8_t *removed, GpuDetection *out,
                           const int64_t *out_off, int64_t *out_n, const FrameDesc *frames, RefOrder ref,
                           const uint32_t *qcl, const uint64_t *ckey, int nb, uint64_t *okey, uint32_t *idx2,
                           uint32_t *err) {
    kernel_begin();
    __shared__ uint32_t sh[32];
    const int f = blockIdx.x;
    if (f >= nframes) return;
    const int64_t a = frame_qstart[f] * nfam, b = frame_qstart[f + 1] * nfam;
    uint32_t *ix = idx + a;
    uint8_t *rm = removed + a;
    // the detections of the frame in (quad, family) order
    int64_t n = 0;
    for (int64_t s0 = a; s0 < b; s0 += blockDim.x) {
        int64_t s = s0 + threadIdx.x;
        uint32_t ok = s < b ? det_ok[s] : 0u;
        uint32_t total;
        uint32_t off = block_excl_scan(ok, &total, sh);
        if (ok) ix[n + off] = (uint32_t)s;
        n += total;
    }
    __syncthreads();
    if (ref.need[f]) {
        // detections that share an id take the reference's quad order:
        // (bucket, key) of their clusters' reference roots
        // (fast/clusters.c:44, 338-356), then family; the others keep
        // theirs (only detections of one id are ever compared)
        const FrameDesc fd = frames[f];
        const uint64_t nbuck = ref_buckets(fd.qw, fd.qh);
        const uint32_t nt = ref.nt[f];
        const uint32_t *tl = ref.tlabel + (int64_t)f * AT_REF_MAXT, *tr = ref.troot + (int64_t)f * AT_REF_MAXT;
        const uint64_t lmask = ((uint64_t)1 << nb) - 1;
        uint64_t *k0 = okey + 2 * a, *k1 = k0 + (b - a);
        for (int64_t p = threadIdx.x; p < n; p += blockDim.x) {
            const uint32_t s = ix[p];
            const uint64_t key = ckey[qcl[s / nfam]];
            const uint32_t lh = (uint32_t)(key >> nb), ll = (uint32_t)(key & lmask);
            uint32_t th = 0xffffffffu, tlo = 0xffffffffu;
            for (uint32_t t = 0; t < nt; t++) {
                if (tl[t] == lh) th = t;
                if (tl[t] == ll) tlo = t;
            }
            if (th != 0xffffffffu && tlo != 0xffffffffu) {
                const uint64_t rh = tr[th], rl = tr[tlo];
                if (rh == 0xffffffffu || rl == 0xffffffffu) atomicOr(err, AT_ERR_ORDER);
                const uint64_t hi = rh > rl ? rh : rl, lo = rh > rl ? rl : rh;
                const uint64_t cid = hi << 32 | lo;
                const uint64_t bucket = ((cid * 2654435761ull) >> 32) & (nbuck - 1);
                k0[p] = bucket << 32 | hi;
                k1[p] = lo << 8 | (uint64_t)(s % nfam);
            } else {
                k0[p] = ~0ull;
                k1[p] = (uint64_t)p;
            }
        }
        __syncthreads();
        for (int64_t p = threadIdx.x; p < n; p += blockDim.x) {
            int64_t r = 0;
            for (int64_t q = 0; q < n; q++) r += k0[q] < k0[p] || (k0[q] == k0[p] && k1[q] < k1[p]);
            idx2[a + r] = ix[p];
        }
        __syncthreads();
        for (int64_t p = threadIdx.x; p < n; p += blockDim.x) ix[p] = idx2[a + p];
        __syncthreads();
    }
    // each place's (family, id), and the group each first place of two or more begins
    uint32_t *key = idx2 + a;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        rm[i] = 0;
        key[i] = (uint32_t)dets[ix[i]].family << 16 | (uint32_t)dets[ix[i]].id;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int64_t w0 = (threadIdx.x >> 5) * 32; w0 < n; w0 += blockDim.x) {
        const int64_t i = w0 + lane;
        bool first = i < n, more = false;
        for (int64_t j = 0; first && j < n; j++)
            if (j != i && key[j] == key[i]) {
                if (j < i) first = false;
                else more = true;
            }
        for (uint32_t bal = __ballot_sync(0xffffffffu, first && more); bal; bal &= bal - 1) {
            // the reference's loop (fast/decode.c:860-891) over this group only
            const int64_t g = w0 + __ffs(bal) - 1;
            const uint32_t k = key[g];
            // the group's next place from p on that is still there
            auto next = [&](int64_t p) {
                for (int64_t q0 = p; q0 < n; q0 += 32) {
                    const int64_t q = q0 + lane;
                    const bool in = q < n && key[q] == k && !*(volatile uint8_t *)(rm + q);
                    const uint32_t m = __ballot_sync(0xffffffffu, in);
                    if (m) return q0 + __ffs(m) - 1;
                }
                return n;
            };
            for (int64_t i0 = g; i0 < n; i0 = next(i0 + 1))
                for (int64_t i1 = next(i0 + 1); i1 < n; i1 = next(i1 + 1)) {
                    const GpuDetection &d0 = dets[ix[i0]], &d1 = dets[ix[i1]];
                    if (!quads_overlap(d0.p, d1.p)) continue;
                    int pref = prefer(0, d0.hamming, d1.hamming);
                    pref = prefer(pref, -(double)d0.decision_margin, -(double)d1.decision_margin);
                    for (int c = 0; c < 4; c++) {
                        pref = prefer(pref, d0.p[c][0], d1.p[c][0]);
                        pref = prefer(pref, d0.p[c][1], d1.p[c][1]);
                    }
                    if (lane == 0) rm[pref < 0 ? i1 : i0] = 1;
                    __syncwarp();
                    if (pref >= 0) break;
                }
        }
    }
    __syncthreads();
    // stable sort by id (fast/detector.c:164-179): rank among survivors
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) key[i] = rm[i] ? 0xffffffffu : key[i] & 0xffffu;
    __syncthreads();
    GpuDetection *o = out + out_off[f];
    uint32_t kept = 0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t id = key[i];
        if (id == 0xffffffffu) continue;
        kept++;
        int64_t r = 0;
        for (int64_t j = 0; j < n; j++) r += key[j] < id || (key[j] == id && j < i);
        o[r] = dets[ix[i]];
    }
    uint32_t total;
    block_excl_scan(kept, &total, sh);
    if (threadIdx.x == 0) out_n[f] = total;
}

// The quads in cluster order (so grouped by frame), and their count.
__global__ void k_gather_quads(const GpuQuad *quads, const uint32_t *ok, const uint32_t *scan, int64_t n,
                               GpuQuad *out, uint32_t *nq, uint32_t *qcl) {
    kernel_begin();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (ok[i]) {
            out[scan[i]] = quads[i];
            qcl[scan[i]] = (uint32_t)i;
        }
        if (i == n - 1) *nq = scan[i] + ok[i];
    }
}

// Per frame: its first quad and its first detection slot (nfam per quad).
__global__ void k_frame_bounds(const GpuQuad *quads, const uint32_t *nq, int nframes, int nfam, int64_t *qstart,
                               int64_t *out_off) {
    kernel_begin();
    const int64_t n = *nq;
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f <= nframes; f += gridDim.x * blockDim.x) {
        int64_t lo = 0, hi = n;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (quads[mid].frame < f)
                lo = mid + 1;
            else
                hi = mid;
        }
        qstart[f] = lo;
        out_off[f] = lo * nfam;
    }
}

// The four kernels' work (prefix sums of ok, the quads gathered, their count,
// the frames' bounds) for at most GATHER_SMALL clusters, in one block: five
// launches of 3-5 us each take 18 us for the 132 clusters of a 640 x 480
// frame, this 6 (decode and fit stages of eight 1280 x 720 frames, 3539
// clusters: 180 us, so 169).
#define GATHER_SMALL 4096
__global__ void __launch_bounds__(1024) k_gather_small(const GpuQuad *quads, const uint32_t *ok, int n, int nframes,
                                                       int nfam, GpuQuad *out, uint32_t *nq, uint32_t *qcl,
                                                       int64_t *qstart, int64_t *out_off) {
    kernel_begin();
    __shared__ uint32_t sh[32];
    __shared__ int s_frame[GATHER_SMALL];
    const int c0 = 4 * threadIdx.x;
    uint32_t f[4], sum = 0, total;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        f[k] = c0 + k < n ? ok[c0 + k] : 0u;
        sum += f[k];
    }
    uint32_t at = block_excl_scan(sum, &total, sh);
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (f[k]) {
            const GpuQuad q = quads[c0 + k];
            out[at] = q;
            s_frame[at] = q.frame;
            qcl[at++] = (uint32_t)(c0 + k);
        }
    if (threadIdx.x == 0) *nq = total;
    __syncthreads();
    for (int fr = threadIdx.x; fr <= nframes; fr += 1024) {
        int lo = 0, hi = (int)total;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (s_frame[mid] < fr)
                lo = mid + 1;
            else
                hi = mid;
        }
        qstart[fr] = lo;
        out_off[fr] = (int64_t)lo * nfam;
    }
}

// Each frame's detections, packed frame after frame into host memory
// (mapped pinned). k_output_meta (one block): meta[3 f ..] = (first, count,
// quads) per frame, meta[3 n], meta[3 n + 1] = the totals of detections and
// quads, and the offsets again on the device (first, with the total last).
// k_output_copy: a warp per detection, its 21 words in one coalesced write.
__global__ void __launch_bounds__(256) k_output_meta(int nframes, const int64_t *qstart, const int64_t *out_n,
                                                     int64_t *first, int64_t *meta) {
    kernel_begin();
    __shared__ uint32_t sh[32];
    int64_t base = 0;
    for (int f0 = 0; f0 < nframes; f0 += blockDim.x) {
        const int f = f0 + threadIdx.x;
        const uint32_t cnt = f < nframes ? (uint32_t)out_n[f] : 0u;
        uint32_t total;
        const uint32_t off = block_excl_scan(cnt, &total, sh);
        if (f < nframes) {
            first[f] = base + off;
            meta[3 * f] = base + off;
            meta[3 * f + 1] = cnt;
            meta[3 * f + 2] = qstart[f + 1] - qstart[f];
        }
        base += total;
    }
    if (threadIdx.x == 0) {
        first[nframes] = base;
        meta[3 * nframes] = base;
        meta[3 * nframes + 1] = qstart[nframes];
    }
}

__global__ void k_output_copy(int nframes, const GpuDetection *out, const int64_t *out_off, const int64_t *first,
                              GpuDetection *host) {
    kernel_begin();
    constexpr int W = (int)(sizeof(GpuDetection) / 8);
    const int lane = threadIdx.x & 31;
    const int64_t total = first[nframes];
    for (int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < total;
         j += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        int lo = 0, hi = nframes - 1;  // the frame holding detection j
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first[mid] <= j)
                lo = mid;
            else
                hi = mid - 1;
        }
        const uint64_t *src = reinterpret_cast<const uint64_t *>(out + out_off[lo] + (j - first[lo]));
        uint64_t *dst = reinterpret_cast<uint64_t *>(host + j);
        if (lane < W) dst[lane] = src[lane];
    }
}

// ---------------------------------------------------------------------------
// Launchers.

static inline dim3 frame_grid(const Launch &L) { return dim3((unsigned)L.blocks_per_frame, (unsigned)L.nframes); }
// a warp per row when the batch has rows enough to fill the GPU with warps
// (16 per SM), else a block per row (lower latency for a few frames)
static inline bool warp_rows(const Launch &L) { return (int64_t)L.nframes * L.max_qh >= 148 * 16; }
// a warp per row, 8 rows a block
static inline dim3 row_warp_grid(const Launch &L) {
    const int64_t b = (L.max_qh + 7) / 8;
    return dim3((unsigned)(b < 1 ? 1 : b < 148 * 8 ? b : 148 * 8), (unsigned)L.nframes);
}
static inline unsigned flat_blocks(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148 * 32) b = 148 * 32;
    return (unsigned)b;
}

void launch_decimate(const Launch &L, const FrameDesc *frames, const uint8_t *img, uint8_t *qim, float factor) {
    launch(k_decimate, frame_grid(L), 256, 0, L.stream, frames, img, qim, factor);
}

void launch_blur(const Launch &L, const FrameDesc *frames, uint8_t *qim, uint8_t *tmp_a, uint8_t *tmp_b,
                 const BlurTaps &taps, bool sharpen) {
    launch(k_blur_pass, frame_grid(L), 256, 0, L.stream, frames, qim, tmp_a, taps, 0);
    launch(k_blur_pass, frame_grid(L), 256, 0, L.stream, frames, tmp_a, tmp_b, taps, 1);
    launch(k_blur_finish, frame_grid(L), 256, 0, L.stream, frames, tmp_b, qim, sharpen ? 1 : 0);
}

void launch_threshold(const Launch &L, const FrameDesc *frames, const uint8_t *qim, uint8_t *tmax, uint8_t *tmin,
                      uint8_t *thr, int32_t diff) {
    launch(k_tile_minmax, frame_grid(L), 256, 0, L.stream, frames, qim, tmax, tmin);
    launch(k_threshold, frame_grid(L), 256, 0, L.stream, frames, qim, tmax, tmin, thr, diff);
}

void launch_decimate_threshold(const Launch &L, const FrameDesc *frames, int64_t max_cells, uint8_t *qim, uint8_t *thr,
                               int32_t diff) {
    // blocks per frame: enough regions for the frame with the most cells
    // (each block finds its region from its frame's width; extra ones exit)
    launch(k_decimate_threshold, dim3((unsigned)max_cells, (unsigned)L.nframes), DT_THREADS, 0, L.stream, frames, qim, thr,
                                                                                                     diff);
}

int64_t decimate_threshold_blocks(int64_t qw, int64_t qh) {
    const int64_t cw = (qw + 3) / 4, ch = (qh + 3) / 4;
    return ((cw + DT_COLS - 1) / DT_COLS) * ((ch + DT_ROWS - 1) / DT_ROWS);
}

void launch_deglitch(const Launch &L, const FrameDesc *frames, uint8_t *thr, uint8_t *tmp) {
    launch(k_morph, frame_grid(L), 256, 0, L.stream, frames, thr, tmp, 1);
    launch(k_morph, frame_grid(L), 256, 0, L.stream, frames, tmp, thr, 0);
}

void launch_point_count(const Launch &L, const FrameDesc *frames, const uint8_t *thr, const uint32_t *lab,
                        uint64_t *row_npts) {
    if (warp_rows(L))
        launch(k_point_count, row_warp_grid(L), 256, 0, L.stream, frames, thr, lab, row_npts);
    else
        launch(k_point_count_block, frame_grid(L), 256, 0, L.stream, frames, thr, lab, row_npts);
}

void launch_point_emit(const Launch &L, const FrameDesc *frames, const uint8_t *thr, const uint32_t *lab,
                       const uint64_t *row_pt_off, uint64_t *pt_key, uint64_t *pt_val, int nb) {
    if (warp_rows(L))
        launch(k_point_emit, row_warp_grid(L), 256, 0, L.stream, frames, thr, lab, row_pt_off, pt_key, pt_val, nb);
    else
        launch(k_point_emit_block, frame_grid(L), 256, 0, L.stream, frames, thr, lab, row_pt_off, pt_key, pt_val, nb);
}

void launch_cluster_collect(cudaStream_t s, const uint64_t *tkeys, uint32_t size, uint64_t *okeys, uint32_t *oslots,
                            uint32_t *count) {
    launch(k_cluster_collect, flat_blocks(size, 256), 256, 0, s, tkeys, size, okeys, oslots, count);
}

void launch_cluster_heads(cudaStream_t s, const uint64_t *key, int64_t n, uint32_t *head) {
    launch(k_cluster_heads, flat_blocks(n, 256), 256, 0, s, key, n, head);
}

void launch_cluster_starts(cudaStream_t s, const uint64_t *key, const uint32_t *head, const uint32_t *head_scan,
                           int64_t n, int nb, const FrameDesc *frames, int nframes, uint32_t *cstart, int32_t *cframe,
                           uint64_t *ckey) {
    launch(k_cluster_starts, flat_blocks(n, 256), 256, 0, s, key, head, head_scan, n, nb, frames, nframes, cstart, cframe,
                                                         ckey);
}

// One size class of the warp fit kernel on stream s: enough blocks to fill
// every SM as far as shared memory allows.
template <int R>
static void launch_fit_warp(cudaStream_t s, const FrameDesc *frames, const GpuParams &prm, const uint8_t *qim,
                            const uint64_t *pts, const uint32_t *cstart, const int32_t *cframe, int64_t nclusters,
                            int64_t npoints, const FitScratch &scr, int q, GpuQuad *quads, uint32_t *quad_ok, int mm) {
    const size_t wsm = fit_warp_smem(32 * R, mm, R >= 16) * FIT_WPB;
    cudaFuncSetAttribute(k_fit_warp<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wsm);
    // as many blocks as fit on the SMs at once (registers and shared memory)
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fit_warp<R>, FIT_WPB * 32, wsm) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    const int64_t full = 148 * (int64_t)per_sm;
    const int64_t wb = (nclusters + FIT_WPB - 1) / FIT_WPB;
    launch(k_fit_warp<R>, (unsigned)(wb < full ? wb : full), FIT_WPB * 32, wsm, s, frames, prm, qim, pts, cstart,
           cframe, nclusters, npoints, q, quads, quad_ok, mm, scr);
}

int launch_fit_quads(cudaStream_t s, const FitStreams &S, const FrameDesc *frames, const GpuParams &prm,
                      const uint8_t *qim, const uint64_t *pts, const uint32_t *cstart, const int32_t *cframe,
                      int64_t nclusters, int64_t npoints, int64_t max_px, const FitScratch &scr, GpuQuad *quads,
                      uint32_t *quad_ok, uint32_t *err) {
    if (nclusters <= 0) return 0;
    const size_t small = fit_smem_bytes(FIT_SMALL, FIT_CHUNK_SMALL, 128 / 32),
                 large = fit_smem_bytes(FIT_LARGE_SORT, FIT_CHUNK_LARGE, FIT_LARGE_NT / 32);
    cudaFuncSetAttribute(k_fit_quads<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small);
    cudaFuncSetAttribute(k_fit_quads<FIT_LARGE_NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)large);
    const int mm = prm.max_nmaxima > 4 ? prm.max_nmaxima : 4;
    cudaMemsetAsync(scr.counts, 0, 2 * FIT_NBUCKET * sizeof(uint32_t), s);
    launch(k_fit_classify, flat_blocks(nclusters, 256), 256, 0, s, frames, cstart, cframe, nclusters, npoints,
                                                                prm.min_cluster_pixels, quad_ok, scr.lists,
                                                                scr.counts, err);
    // five streams, one per group of classes: above 6144 points (a block of
    // FIT_HUGE_NT each; only when a frame allows such clusters at all); the
    // other large clusters (a block of FIT_LARGE_NT each, two an SM: one
    // cluster's serial steps overlap the other's); 513-1024 points (a block of
    // 128, few of 257-512 too); 257-512 (a warp each); up to 256 (a warp
    // each). No stream has a priority: with higher ones for the larger
    // clusters, so that their few long blocks start first, eight 1280 x 720
    // frames take 587 instead of 603 us, but 32 of 1920 x 1080 1772 instead of
    // 1749, and other streams of the process would wait behind them.
    const bool huge = max_px > FIT_LARGE_SORT;
    cudaEventRecord(S.fork, s);
    for (int k = 0; k < (huge ? 4 : 3); k++) cudaStreamWaitEvent(S.side[k], S.fork, 0);
    if (huge) {
        const size_t hsm = fit_smem_bytes(FIT_HUGE_SORT, FIT_CHUNK_LARGE, FIT_HUGE_NT / 32);
        cudaFuncSetAttribute(k_fit_quads<FIT_HUGE_NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hsm);
        launch(k_fit_quads<FIT_HUGE_NT>, (unsigned)(nclusters < 148 ? nclusters : 148), FIT_HUGE_NT, hsm, S.side[3],
               frames, prm, qim, pts, cstart, cframe, nclusters, npoints, scr, quads, quad_ok, err, 15, 12,
               FIT_HUGE_SORT, FIT_CHUNK_LARGE);
        cudaEventRecord(S.join[3], S.side[3]);
    }
    launch(k_fit_quads<FIT_LARGE_NT>, (unsigned)(nclusters < 2 * 148 ? nclusters : 2 * 148), FIT_LARGE_NT, large,
           S.side[0], frames, prm, qim, pts, cstart, cframe, nclusters, npoints, scr, quads, quad_ok, err, 11, 7,
           FIT_LARGE_SORT, FIT_CHUNK_LARGE);
    cudaEventRecord(S.join[0], S.side[0]);
    launch(k_fit_quads<128>, (unsigned)(nclusters < 148 * 4 ? nclusters : 148 * 4), 128, small, S.side[1], frames, prm,
           qim, pts, cstart, cframe, nclusters, npoints, scr, quads, quad_ok, err, 6, 3, FIT_SMALL, FIT_CHUNK_SMALL);
    cudaEventRecord(S.join[1], S.side[1]);
    launch_fit_warp<16>(S.side[2], frames, prm, qim, pts, cstart, cframe, nclusters, npoints, scr, 2, quads, quad_ok,
                        mm);
    cudaEventRecord(S.join[2], S.side[2]);
    launch_fit_warp<4>(s, frames, prm, qim, pts, cstart, cframe, nclusters, npoints, scr, 0, quads, quad_ok, mm);
    launch_fit_warp<8>(s, frames, prm, qim, pts, cstart, cframe, nclusters, npoints, scr, 1, quads, quad_ok, mm);
    for (int k = 0; k < (huge ? 4 : 3); k++) cudaStreamWaitEvent(s, S.join[k], 0);
    return huge ? 7 : 6;
}

int launch_gather_quads(cudaStream_t s, const GpuQuad *quads, const uint32_t *ok, int64_t n, uint32_t *scan,
                        uint32_t *scratch, int nframes, int nfam, GpuQuad *out, uint32_t *nq, uint32_t *qcl,
                        int64_t *qstart, int64_t *out_off) {
    if (n <= 0) return 0;
    if (n <= GATHER_SMALL) {
        launch(k_gather_small, 1, 1024, 0, s, quads, ok, (int)n, nframes, nfam, out, nq, qcl, qstart, out_off);
        return 1;
    }
    launch_scan_u32(s, ok, n, scan, scratch);
    launch(k_gather_quads, flat_blocks(n, 256), 256, 0, s, quads, ok, scan, n, out, nq, qcl);
    launch(k_frame_bounds, flat_blocks(nframes + 1, 256), 256, 0, s, out, nq, nframes, nfam, qstart, out_off);
    return 5;
}

void launch_output(cudaStream_t s, int nframes, const int64_t *qstart, const GpuDetection *out,
                   const int64_t *out_off, const int64_t *out_n, int64_t *first, GpuDetection *host,
                   int64_t *meta, int64_t max_dets) {
    launch(k_output_meta, 1, 256, 0, s, nframes, qstart, out_n, first, meta);
    const int64_t blocks = (max_dets + 7) / 8;
    launch(k_output_copy, (unsigned)(blocks < 1 ? 1 : blocks < 148 * 4 ? blocks : 148 * 4), 256, 0, s, nframes, out, out_off,
                                                                                                first, host);
}

void launch_decode(cudaStream_t s, const FrameDesc *frames, const GpuParams &prm, const GpuFamily *fams,
                   const uint8_t *img, const uint8_t *qim, const GpuQuad *quads, int64_t max_quads,
                   const DecodeScratch &scr, GpuDetection *dets, uint32_t *det_ok) {
    // grids for at most max_quads quads; the kernels read the count (scr.nq)
    if (max_quads <= 0) return;
    const unsigned blocks = (unsigned)(max_quads < 148 * 64 ? max_quads : 148 * 64);
    launch(k_refine, blocks, AT_DEC_THREADS, 0, s, frames, prm, img, qim, quads, scr.nq, scr.corners, det_ok);
    const int64_t hb = (max_quads + QH_WARPS - 1) / QH_WARPS;
    launch(k_quad_homography, (unsigned)(hb < 148 * 16 ? hb : 148 * 16), QH_WARPS * 32, 0, s, scr.corners, scr.nq,
                                                                                        scr.h, scr.hok);
    launch(k_decode, blocks, DECODE_THREADS, 0, s, frames, prm, fams, img, qim, quads, scr.nq, scr.h, scr.hok, dets,
                                               det_ok);
}

void launch_finalize(cudaStream_t s, int nframes, const int64_t *frame_qstart, int nfam, const GpuDetection *dets,
                     const uint32_t *det_ok, uint32_t *idx, uint8_t *removed, GpuDetection *out,
                     const int64_t *out_off, int64_t *out_n, const FrameDesc *frames, const RefOrder &ref,
                     const uint32_t *qcl, const uint64_t *ckey, int nb, uint64_t *okey, uint32_t *idx2,
                     uint32_t *err) {
    launch(k_finalize, nframes, 256, 0, s, nframes, frame_qstart, nfam, dets, det_ok, idx, removed, out, out_off, out_n,
                                       frames, ref, qcl, ckey, nb, okey, idx2, err);
}

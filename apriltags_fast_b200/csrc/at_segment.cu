// Runs and connected components over runs (fast/threshold.c:196-283,
// fast/unionfind.c:89-196, 284-298), from bit masks of the threshold image.
//
// A row is cut in words of 32 columns (RowWord: the white and the black
// pixels, the columns where a run starts, the runs before the word), so the
// run that covers a column is one popcount away. Two runs of adjacent rows
// touch where their masks meet: with C and A the white (or black) pixels of
// a row and of the row above, each maximal stretch of C & A at columns >= 1
// is one touching pair, and white pixels also touch over a corner (C at x,
// A at x - 1 or x + 1, without meeting beside it). So a thread takes a word
// and has exactly the pairs that begin in it, a few each: no search, and no
// lane waits for a long run of its neighbour. Searching the runs above per
// run took 333 us per 32 frames of 1920 x 1080 (quad images 960 x 540) with
// the runs made by a kernel of its own (76 us); bands of more than 3072 runs
// went through global memory (1.07 ms for 16 frames up to 3840 x 2160,
// 1.65 ms for 4032 x 3024 at full resolution).
//
//   k_band_union   a block per band of rows: masks, runs, the unions inside
//                  the band in shared memory; every run then points at its
//                  band root, which holds the band component's pixels.
//   k_band_join    the unions across band edges and of the last column, in
//                  global memory.
//   k_root_sums    each band root adds its pixels to its component's root
//                  and points at it (so a run is two steps from its root).
#include <cuda_runtime.h>
#include <stdint.h>

#include "at_device.cuh"
#include "at_gpu.h"
#include "at_kernels.h"

__device__ __forceinline__ uint32_t uf_find(uint32_t *par, uint32_t x) {
    volatile uint32_t *p = par;
    uint32_t px = p[x];
    while (px != x) {
        uint32_t ppx = p[px];
        if (ppx == px) return px;
        p[x] = ppx;  // path halving: only ever an ancestor
        x = ppx;
        px = p[x];
    }
    return x;
}

// Roots are linked in the order of a bijective hash of their ids: one fixed
// total order, so concurrent links can never form a cycle, and a random one,
// so trees stay shallow (linking by id would chain the pieces of a row).
// The label of a component, its smallest node id, is tracked apart.
__device__ __forceinline__ uint32_t uf_rank(uint32_t x) {
    uint32_t h = x * 0x9e3779b1u;
    return h ^ (h >> 16);
}

__device__ __forceinline__ void uf_unite(uint32_t *par, uint32_t a, uint32_t b) {
    for (;;) {
        a = uf_find(par, a);
        b = uf_find(par, b);
        if (a == b) return;
        if (uf_rank(a) < uf_rank(b)) {
            uint32_t t = a;
            a = b;
            b = t;
        }
        if (atomicCAS(par + a, a, b) == a) return;
    }
}

// Bands: rows per band for a quad image qw wide, so that the band's local
// ids (row << band_shift | run) stay within 16384 (and their two 16-bit
// arrays within 64 KB). Images over 16384 wide get bands of one row, whose
// runs are their own band roots.
#define BAND_IDS 16384
__host__ __device__ inline int band_shift(int qw) {
    int s = 5;
    while ((1 << s) < qw) s++;
    return s;
}
__host__ __device__ inline int band_rows(int qw) {
    const int s = band_shift(qw), r = BAND_IDS >> s;
    return r < 1 ? 1 : r < 8 ? r : 8;
}
__host__ __device__ inline size_t band_smem(int qw) {
    const int s = band_shift(qw), r = band_rows(qw);
    return (size_t)r * ((qw + 31) / 32) * 16 + ((1 << s) > BAND_IDS ? 0 : (size_t)r * 4 << s);
}

// The 4 bits 0, 8, 16, 24 of x as bits 0 to 3.
__device__ __forceinline__ uint32_t gather4(uint32_t x) { return ((x & 0x01010101u) * 0x01020408u) >> 24 & 15u; }

// The masks of 32 columns of a threshold row from column x0: 255 has bit 7,
// 0 is the only value without bit 0. Unaligned rows go by aligned words
// (the word of the last byte may reach 3 bytes past the row).
__device__ __forceinline__ void row_masks(const uint8_t *row, int x0, int qw, uint32_t &W, uint32_t &K) {
    const uint8_t *p = row + x0;
    const int n = min(32, qw - x0);
    uint32_t v[8];
    if (n == 32 && ((uintptr_t)p & 15) == 0) {
        const uint4 a = reinterpret_cast<const uint4 *>(p)[0], b = reinterpret_cast<const uint4 *>(p)[1];
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
        v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
        const int o = (int)((uintptr_t)p & 3), last = (o + n - 1) >> 2;
        const uint32_t *q = reinterpret_cast<const uint32_t *>(p - o);
        uint32_t w[9];
#pragma unroll
        for (int k = 0; k < 9; k++) w[k] = k <= last ? q[k] : 0u;
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = __funnelshift_r(w[k], w[k + 1], 8 * o);
    }
    W = K = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        W |= gather4(v[k] >> 7) << (4 * k);
        K |= gather4(~v[k]) << (4 * k);
    }
    if (n < 32) {
        const uint32_t m = (1u << n) - 1u;
        W &= m;
        K &= m;
    }
}

// The touching pairs of runs of a row and the row above that begin in word
// i (fast/unionfind.c:112-146: columns 0 do not count, the row's pixel of a
// corner is at a column >= 1): columns where runs meet, where the row's
// run meets one to its upper left, and to its upper right.
struct PairMasks {
    uint32_t meet, left, right;
};
__device__ __forceinline__ PairMasks pair_masks(const RowWord *cur, const RowWord *abv, int i, int nw, int qw) {
    const RowWord c = cur[i], a = abv[i];
    const uint32_t vm = run_columns(i, qw), c1 = i == 0 ? ~1u : ~0u;
    const uint32_t Wc = c.white & vm, Kc = c.black & vm, Wa = a.white & vm, Ka = a.black & vm;
    uint32_t pWc = 0, pWa = 0, pKK = 0, nWc = 0, nWa = 0;  // the columns beside the word
    if (i > 0) {
        pWc = cur[i - 1].white >> 31;
        pWa = abv[i - 1].white >> 31;
        pKK = (cur[i - 1].black & abv[i - 1].black) >> 31;
    }
    if (i + 1 < nw) {
        const uint32_t nm = run_columns(i + 1, qw) & 1u;
        nWc = cur[i + 1].white & nm;
        nWa = abv[i + 1].white & nm;
    }
    const uint32_t MW = Wc & Wa & c1, MK = Kc & Ka & c1;
    uint32_t lc = Wc << 1 | pWc;
    if (i == 0) lc &= ~2u;  // meeting at column 0 does not count
    // a corner's runs that also meet at a column beside it are taken there
    return {(MW & ~(MW << 1 | (pWc & pWa))) | (MK & ~(MK << 1 | pKK)), Wc & (Wa << 1 | pWa) & ~Wa & ~lc & c1,
            Wc & (Wa >> 1 | nWa << 31) & ~Wa & ~(Wc >> 1 | nWc << 31) & c1};
}
// Calls fn(run of the row, run of the row above) for each of them.
template <class F>
__device__ __forceinline__ void for_pairs(const RowWord *cur, const RowWord *abv, int i, PairMasks p, F fn) {
    const RowWord c = cur[i], a = abv[i];
    for (uint32_t m = p.meet; m; m &= m - 1) {
        const int b = __ffs(m) - 1;
        fn(run_at(c, b), run_at(a, b));
    }
    for (uint32_t m = p.left; m; m &= m - 1) {
        const int b = __ffs(m) - 1;
        fn(run_at(c, b), b > 0 ? run_at(a, b - 1) : run_at(abv[i - 1], 31));
    }
    for (uint32_t m = p.right; m; m &= m - 1) {
        const int b = __ffs(m) - 1;
        fn(run_at(c, b), b < 31 ? run_at(a, b + 1) : run_at(abv[i + 1], 0));
    }
}

// Places of the block's pairs in a list: n of this thread; *count (shared)
// grows by the warp's sum. Every lane of the warp calls it.
__device__ __forceinline__ uint32_t list_places(uint32_t n, uint32_t *count) {
    uint32_t total, base = 0;
    const uint32_t off = warp_excl_scan(n, &total);
    if ((threadIdx.x & 31) == 0 && total) base = atomicAdd(count, total);
    return __shfl_sync(0xffffffffu, base, 0) + off;
}
__device__ __forceinline__ uint32_t pair_count(const PairMasks &p) {
    return __popc(p.meet) + __popc(p.left) + __popc(p.right);
}

// Pairs listed at once (more are united where they are found). A union per
// thread from the list: unions straight from the words' loops kept their
// warps waiting for their slowest lane (the band joins of one 640 x 480
// frame took 200 us that way).
#define BAND_LIST 4096

// Unions over band-local ids in shared memory, lock-free, the larger id
// hooked under the smaller, so a root is its set's smallest node.
__device__ __forceinline__ uint32_t lu_find(volatile uint16_t *par, uint32_t x) {
    uint32_t p = par[x];
    while (p != x) {
        const uint32_t pp = par[p];
        if (pp != p) par[x] = (uint16_t)pp;  // path halving: only ever an ancestor
        x = p;
        p = par[x];
    }
    return x;
}
__device__ __forceinline__ void lu_unite(uint16_t *par, uint32_t a, uint32_t b) {
    for (;;) {
        a = lu_find(par, a);
        b = lu_find(par, b);
        if (a == b) return;
        if (a < b) {
            const uint32_t t = a;
            a = b;
            b = t;
        }
        if (atomicCAS(par + a, (unsigned short)a, (unsigned short)b) == a) return;
    }
}

__global__ void __launch_bounds__(256) k_band_union(const FrameDesc *frames, const uint8_t *thr, RunArrays runs,
                                                    uint32_t *row_nruns, RowWord *words) {
    extern __shared__ __align__(16) uint8_t s_band[];
    const FrameDesc f = frames[blockIdx.y];
    const int tid = threadIdx.x, lane = tid & 31;
    const int qw = f.qw, nw = (qw + 31) / 32, sh = band_shift(qw), R = band_rows(qw);
    const bool solo = (1 << sh) > BAND_IDS;
    RowWord *s_word = reinterpret_cast<RowWord *>(s_band);
    uint16_t *s_par = reinterpret_cast<uint16_t *>(s_word + R * nw);
    uint16_t *s_px = s_par + (R << sh);  // pixels per band root: at most 16384
    __shared__ uint32_t s_list[BAND_LIST], s_n;
    if (tid == 0) s_n = 0;
    const int nband = (f.qh + R - 1) / R;
    for (int b = blockIdx.x; b < nband; b += gridDim.x) {
        const int y0 = b * R, nr = min(R, f.qh - y0);
        const uint8_t *img = thr + f.q_off + (int64_t)y0 * qw;
        const int64_t node0 = f.node_off + (int64_t)y0 * qw;
        RowWord *out = words + f.word_off + (int64_t)y0 * nw;
        __syncthreads();
        for (int it = tid; it < nr * nw; it += blockDim.x) {
            const int r = it / nw, i = it - r * nw;
            RowWord w;
            row_masks(img + (int64_t)r * qw, 32 * i, qw, w.white, w.black);
            w.starts = w.before = 0;
            s_word[it] = w;
        }
        __syncthreads();
        // run starts and the runs before each word, a warp per row
        for (int r = tid >> 5; r < nr; r += blockDim.x >> 5) {
            uint32_t base = 0;
            for (int i0 = 0; i0 < nw; i0 += 32) {
                const int i = i0 + lane;
                RowWord *w = s_word + r * nw + i;
                uint32_t S = 0;
                if (i < nw) {
                    const uint32_t vm = run_columns(i, qw), W = w->white & vm, K = w->black & vm;
                    const uint32_t pW = i > 0 ? w[-1].white >> 31 : 0u, pK = i > 0 ? w[-1].black >> 31 : 0u;
                    S = (W & ~(W << 1 | pW)) | (K & ~(K << 1 | pK));
                }
                uint32_t total;
                const uint32_t off = warp_excl_scan(__popc(S), &total);
                if (i < nw) {
                    w->starts = S;
                    w->before = base + off;
                }
                base += total;
            }
            if (lane == 0) {
                row_nruns[f.row0 + y0 + r] = base;
                const int64_t vn = f.node_off + (int64_t)qw * f.qh + y0 + r;
                runs.parent[vn] = (uint32_t)vn;
                runs.px[vn] = 1;
                runs.minid[vn] = (uint32_t)vn;
            }
        }
        __syncthreads();
        // the runs (start, end, value), each its own set
        for (int it = tid; it < nr * nw; it += blockDim.x) {
            const int r = it / nw, i = it - r * nw;
            const RowWord w = s_word[it];
            out[it] = w;
            const uint32_t vm = run_columns(i, qw), W = w.white & vm, K = w.black & vm;
            const int64_t base = node0 + (int64_t)r * qw;
            uint32_t k = w.before;
            for (uint32_t m = w.starts; m; m &= m - 1, k++) {
                const int c = __ffs(m) - 1;
                runs.start[base + k] = (uint16_t)(32 * i + c);
                runs.v[base + k] = W >> c & 1u ? 255 : 0;
                if (!solo) {
                    s_par[(r << sh) + k] = (uint16_t)((r << sh) + k);
                    s_px[(r << sh) + k] = 0;
                } else {
                    runs.parent[base + k] = runs.minid[base + k] = (uint32_t)(base + k);
                    runs.px[base + k] = 0;
                }
            }
            uint32_t nW = 0, nK = 0;
            if (i + 1 < nw) {
                const uint32_t nm = run_columns(i + 1, qw) & 1u;
                nW = s_word[it + 1].white & nm;
                nK = s_word[it + 1].black & nm;
            }
            for (uint32_t m = (W & ~(W >> 1 | nW << 31)) | (K & ~(K >> 1 | nK << 31)); m; m &= m - 1) {
                const int c = __ffs(m) - 1;
                runs.end[base + run_at(w, c)] = (uint16_t)(32 * i + c);
            }
        }
        __syncthreads();
        for (int it0 = nw; it0 < nr * nw; it0 += blockDim.x) {
            const int it = it0 + tid, r = it / nw, i = it - r * nw;
            const RowWord *cur = s_word + r * nw, *abv = cur - nw;
            PairMasks pm = {0, 0, 0};
            if (it < nr * nw) pm = pair_masks(cur, abv, i, nw, qw);
            uint32_t at = list_places(pair_count(pm), &s_n);
            if (it < nr * nw)
                for_pairs(cur, abv, i, pm, [&](uint32_t c, uint32_t a) {
                    c += (uint32_t)r << sh;
                    a += (uint32_t)(r - 1) << sh;
                    if (at < BAND_LIST)
                        s_list[at] = c | a << 16;
                    else
                        lu_unite(s_par, c, a);
                    at++;
                });
        }
        __syncthreads();
        const uint32_t np = min(s_n, (uint32_t)BAND_LIST);
        for (uint32_t p = tid; p < np; p += blockDim.x) lu_unite(s_par, s_list[p] & 0xffffu, s_list[p] >> 16);
        __syncthreads();
        if (tid == 0) s_n = 0;
        // each run's band root; the pixels of the word's pieces of runs
        for (int it = tid; it < nr * nw; it += blockDim.x) {
            const int r = it / nw, i = it - r * nw;
            const RowWord w = s_word[it];
            uint32_t m = (w.white | w.black) & run_columns(i, qw);
            const uint32_t stop = w.starts | ~m;
            while (m) {
                const int c = __ffs(m) - 1;
                const uint32_t past = c < 31 ? stop & (~0u << (c + 1)) : 0u;
                const int e = past ? __ffs(past) - 1 : 32;
                m = e < 32 ? m & (~0u << e) : 0u;
                const uint32_t k = run_at(w, c);
                if (solo) {
                    atomicAdd(runs.px + node0 + (int64_t)r * qw + k, (uint32_t)(e - c));
                    continue;
                }
                const uint32_t l = (uint32_t)(r << sh) + k;
                uint32_t x = l;
                const volatile uint16_t *par = s_par;
                for (uint32_t p = par[x]; p != x; p = par[x]) x = p;
                s_par[l] = (uint16_t)x;
                // two 16-bit counts a word, neither of which can overflow
                atomicAdd(reinterpret_cast<uint32_t *>(s_px) + (x >> 1), (uint32_t)(e - c) << (16 * (x & 1)));
            }
        }
        __syncthreads();
        if (solo) continue;
        for (int r = 0; r < nr; r++) {
            const RowWord &lw = s_word[r * nw + nw - 1];
            const uint32_t n = lw.before + __popc(lw.starts);
            const int64_t base = node0 + (int64_t)r * qw;
            for (uint32_t k = tid; k < n; k += blockDim.x) {
                const uint32_t l = (uint32_t)(r << sh) + k, x = s_par[l];
                runs.parent[base + k] = (uint32_t)(node0 + (int64_t)(x >> sh) * qw + (x & ((1u << sh) - 1u)));
                runs.px[base + k] = x == l ? s_px[l] : 0u;  // not 0: a band root
                if (x == l) runs.minid[base + k] = (uint32_t)(base + k);
            }
        }
    }
}

// The unions across band edges, a block per edge, and the last-column links
// of every row (fast/unionfind.c:89-97).
__global__ void __launch_bounds__(256) k_band_join(const FrameDesc *frames, const uint8_t *thr, RunArrays runs,
                                                   const uint32_t *row_nruns, const RowWord *words) {
    __shared__ uint32_t s_list[BAND_LIST], s_n;
    const FrameDesc f = frames[blockIdx.y];
    const int tid = threadIdx.x, qw = f.qw, nw = (qw + 31) / 32, R = band_rows(qw > 0 ? qw : 1);
    const int nband = (f.qh + R - 1) / R;
    for (int b = 1 + blockIdx.x; b < nband; b += gridDim.x) {
        const int64_t y = (int64_t)b * R;
        const RowWord *cur = words + f.word_off + y * nw, *abv = cur - nw;
        const uint32_t base = (uint32_t)(f.node_off + y * qw), above = base - (uint32_t)qw;
        __syncthreads();
        if (tid == 0) s_n = 0;
        __syncthreads();
        for (int i0 = 0; i0 < nw; i0 += blockDim.x) {
            const int i = i0 + tid;
            PairMasks pm = {0, 0, 0};
            if (i < nw) pm = pair_masks(cur, abv, i, nw, qw);
            uint32_t at = list_places(pair_count(pm), &s_n);
            if (i < nw)
                for_pairs(cur, abv, i, pm, [&](uint32_t c, uint32_t a) {
                    if (at < BAND_LIST)
                        s_list[at] = c | a << 16;
                    else
                        uf_unite(runs.parent, base + c, above + a);
                    at++;
                });
        }
        __syncthreads();
        const uint32_t np = min(s_n, (uint32_t)BAND_LIST);
        for (uint32_t p = tid; p < np; p += blockDim.x)
            uf_unite(runs.parent, base + (s_list[p] & 0xffffu), above + (s_list[p] >> 16));
    }
    for (int64_t y = 1 + (int64_t)blockIdx.x * blockDim.x + tid; y < f.qh; y += (int64_t)gridDim.x * blockDim.x) {
        const int64_t ncur = row_nruns[f.row0 + y];
        if (ncur == 0) continue;
        const int64_t last = f.node_off + y * f.qw + ncur - 1;
        const uint8_t *above = thr + f.q_off + (y - 1) * f.qw;
        if (runs.end[last] == f.qw - 2 && runs.v[last] == 255 && above[f.qw - 1] == 255 && above[f.qw - 2] != 255)
            uf_unite(runs.parent, (uint32_t)last, (uint32_t)(f.node_off + (int64_t)f.qw * f.qh + y - 1));
    }
}

// The root of x without writes (after the unions: a path-halving write that
// read its value before another thread stored a root would undo it).
__device__ __forceinline__ uint32_t uf_root(const uint32_t *par, uint32_t x) {
    const volatile uint32_t *p = par;
    uint32_t px = p[x];
    while (px != x) {
        x = px;
        px = p[x];
    }
    return x;
}

// Each band root (and last-column node) adds its pixels and offers its id,
// the smallest of its band component, to its component's root (one atomic
// per distinct root of a warp), and from here on points at it.
__global__ void __launch_bounds__(256) k_root_sums(const FrameDesc *frames, RunArrays runs, const uint32_t *row_nruns) {
    const FrameDesc f = frames[blockIdx.y];
    const int lane = threadIdx.x & 31;
    for (int64_t y = blockIdx.x; y < f.qh; y += gridDim.x) {
        const int64_t base = f.node_off + y * f.qw;
        const int64_t n = row_nruns[f.row0 + y];
        for (int64_t i0 = 0; i0 <= n; i0 += blockDim.x) {
            const int64_t i = i0 + threadIdx.x;
            const int64_t node = i < n ? base + i : f.node_off + (int64_t)f.qw * f.qh + y;
            // a component's root is a band root too, and its count may grow
            // meanwhile, but it adds to no other
            const uint32_t px = i <= n ? runs.px[node] : 0u;
            uint32_t r = 0;
            bool add = false;
            if (px) {
                r = uf_root(runs.parent, (uint32_t)node);
                add = r != (uint32_t)node;
            }
            const uint32_t live = __ballot_sync(0xffffffffu, add);
            if (!add) continue;
            // no unions run any more: pointing straight at the root is safe
            // for the walks of other threads
            runs.parent[node] = r;
            const uint32_t peers = __match_any_sync(live, r);
            const uint32_t sum = __reduce_add_sync(peers, px), mn = __reduce_min_sync(peers, (uint32_t)node);
            if (lane == __ffs(peers) - 1) {
                atomicAdd(runs.px + r, sum);
                atomicMin(runs.minid + r, mn);
            }
        }
    }
}

#define ROW_STAGE 4096
// Per pixel: its component's label if the component has at least
// min_cluster_pixels pixels, else AT_NOK (no run: 127, or too small). A
// block per row: each run's label once (root_of), spread over the run's pixels by a max-scan of the run starts;
// the last column is the row's extra node.
#define LAB_THREADS 256
__global__ void __launch_bounds__(LAB_THREADS) k_labels(const FrameDesc *frames, const RunArrays runs,
                                                        const uint32_t *row_nruns, uint32_t *lab, int32_t min_px) {
    __shared__ uint32_t s_run[ROW_STAGE];
    __shared__ uint32_t s_rlab[ROW_STAGE];
    __shared__ uint16_t s_end[ROW_STAGE];
    __shared__ uint32_t s_wmax[LAB_THREADS / 32];
    const FrameDesc f = frames[blockIdx.y];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int qw = (int)f.qw, W = qw - 1;
    for (int y = blockIdx.x; y < (int)f.qh; y += gridDim.x) {
        const int64_t base = f.node_off + (int64_t)y * qw;
        const int nr = (int)row_nruns[f.row0 + y];
        uint32_t *out = lab + f.q_off + (int64_t)y * qw;
        if (tid == 0) {
            const uint32_t r = root_of(runs, f.node_off + (int64_t)qw * f.qh + y);
            out[W] = (int64_t)runs.px[r] >= min_px ? runs.minid[r] : AT_NOK;
        }
        if (W > ROW_STAGE) {
            // rows too wide to stage: a binary search per pixel
            for (int x = tid; x < W; x += LAB_THREADS) {
                int lo = 0, hi = nr;
                while (lo < hi) {  // the first run with start > x
                    const int mid = (lo + hi) >> 1;
                    if ((int)runs.start[base + mid] <= x)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                uint32_t l = AT_NOK;
                if (lo > 0 && (int)runs.end[base + lo - 1] >= x) {
                    const uint32_t r = root_of(runs, base + lo - 1);
                    if ((int64_t)runs.px[r] >= min_px) l = runs.minid[r];
                }
                out[x] = l;
            }
            continue;
        }
        __syncthreads();
        for (int x = tid; x < W; x += LAB_THREADS) s_run[x] = 0;
        __syncthreads();
        for (int i = tid; i < nr; i += LAB_THREADS) {
            s_run[runs.start[base + i]] = (uint32_t)i + 1;
            s_end[i] = runs.end[base + i];
            const uint32_t r = root_of(runs, base + i);
            s_rlab[i] = (int64_t)runs.px[r] >= min_px ? runs.minid[r] : AT_NOK;
        }
        __syncthreads();
        // thread t owns pixels [t * seg, t * seg + seg): the largest run
        // number started at or before each of them
        const int seg = (W + LAB_THREADS - 1) / LAB_THREADS;
        const int x0 = tid * seg, x1 = x0 + seg < W ? x0 + seg : W;
        uint32_t m = 0;
        for (int x = x0; x < x1; x++) m = max(m, s_run[x]);
        uint32_t incl = m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl = max(incl, t);
        }
        if (lane == 31) s_wmax[wid] = incl;
        uint32_t run = __shfl_up_sync(0xffffffffu, incl, 1);
        if (lane == 0) run = 0;
        __syncthreads();
        for (int w = 0; w < wid; w++) run = max(run, s_wmax[w]);
        for (int x = x0; x < x1; x++) {
            run = max(run, s_run[x]);
            s_run[x] = run && x <= (int)s_end[run - 1] ? s_rlab[run - 1] : AT_NOK;
        }
        __syncthreads();
        for (int x = tid; x < W; x += LAB_THREADS) out[x] = s_run[x];
    }
}

// The same labels with a warp per row (8 rows a block, for batches large
// enough to fill the GPU that way): the run starting at each column staged
// in the warp's slice of shared memory, then 128 columns at a time, 4 a
// lane: a max-scan gives each column its run (carried across chunks), the
// label is read through the run's root (the L1 cache holds the few roots of
// a row; a lane's 4 pixels usually share one run), and a pixel that no
// stored run covers is a 127 of the threshold image. Rows wider than
// LW_CAP columns search the runs per pixel instead.
#define LW_CAP 2048
__global__ void __launch_bounds__(256) k_labels_w(const FrameDesc *frames, const uint8_t *thr, const RunArrays runs,
                                                  const uint32_t *row_nruns, uint32_t *lab, int32_t min_px) {
    __shared__ __align__(16) uint16_t s_run[8][LW_CAP + 8];
    const FrameDesc f = frames[blockIdx.y];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int qw = (int)f.qw, W = qw - 1;
    uint16_t *sr = s_run[w];
    for (int y = (int)blockIdx.x * 8 + w; y < (int)f.qh; y += (int)gridDim.x * 8) {
        const int64_t base = f.node_off + (int64_t)y * qw;
        const int nr = (int)row_nruns[f.row0 + y];
        uint32_t *out = lab + f.q_off + (int64_t)y * qw;
        const uint8_t *row = thr + f.q_off + (int64_t)y * qw;
        auto label_of = [&](int i) -> uint32_t {
            const uint32_t r = root_of(runs, base + i);
            return (int64_t)runs.px[r] >= min_px ? runs.minid[r] : AT_NOK;
        };
        if (lane == 0) {
            const uint32_t r = root_of(runs, f.node_off + (int64_t)qw * f.qh + y);
            out[W] = (int64_t)runs.px[r] >= min_px ? runs.minid[r] : AT_NOK;
        }
        if (W > LW_CAP) {
            for (int x = lane; x < W; x += 32) {
                int lo = 0, hi = nr;
                while (lo < hi) {  // the first run with start > x
                    const int mid = (lo + hi) >> 1;
                    if ((int)runs.start[base + mid] <= x)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                out[x] = lo > 0 && (int)runs.end[base + lo - 1] >= x ? label_of(lo - 1) : AT_NOK;
            }
            continue;
        }
        const int Wp = (W + 3) & ~3;
        for (int x = lane; x < Wp; x += 32) sr[x] = 0;
        __syncwarp();
        for (int i = lane; i < nr; i += 32) sr[runs.start[base + i]] = (uint16_t)(i + 1);
        __syncwarp();
        // 16-byte stores when the row and the label array allow
        const bool v4 = ((((uintptr_t)out) | ((uintptr_t)row)) & 15) == 0;
        uint32_t carry = 0;
        for (int x0 = 0; x0 < W; x0 += 128) {
            const int x = x0 + 4 * lane;
            const uint2 pr = x < Wp ? *reinterpret_cast<const uint2 *>(sr + x) : make_uint2(0, 0);
            uint32_t m[4] = {pr.x & 0xffffu, pr.x >> 16, pr.y & 0xffffu, pr.y >> 16};
            m[1] = max(m[1], m[0]);
            m[2] = max(m[2], m[1]);
            m[3] = max(m[3], m[2]);
            uint32_t incl = m[3];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl = max(incl, t);
            }
            uint32_t excl = __shfl_up_sync(0xffffffffu, incl, 1);
            if (lane == 0) excl = 0;
            excl = max(excl, carry);
            carry = max(carry, __shfl_sync(0xffffffffu, incl, 31));
            uint32_t l4[4];
            uint32_t prev_run = 0, prev_lab = AT_NOK;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t v = max(m[k], excl);
                uint32_t l = AT_NOK;
                if (x + k < W && v) {
                    if (v != prev_run) {
                        prev_run = v;
                        prev_lab = label_of((int)v - 1);
                    }
                    l = row[x + k] != 127 ? prev_lab : AT_NOK;
                }
                l4[k] = l;
            }
            if (v4 && x + 4 <= W) {
                *reinterpret_cast<uint4 *>(out + x) = make_uint4(l4[0], l4[1], l4[2], l4[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (x + k < W) out[x + k] = l4[k];
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Launchers.

// a warp per row when the batch has rows enough to fill the GPU with warps
// (16 per SM), else a block per row (lower latency for a few frames)
static inline bool warp_rows(const Launch &L) { return (int64_t)L.nframes * L.max_qh >= 148 * 16; }

bool segment_set_smem() {
    // the most a band takes: 8 rows of 2048 columns (the last 16384 wide
    // with arrays of its own), or one row of 65536
    return cudaFuncSetAttribute(k_band_union, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024) == cudaSuccess;
}

int launch_segment(const Launch &L, const FrameDesc *frames, int64_t max_bands, size_t smem, const uint8_t *thr,
                   RunArrays runs, uint32_t *row_nruns, RowWord *words, uint32_t *lab, int32_t min_px) {
    const unsigned n = (unsigned)L.nframes;
    const dim3 rg((unsigned)(L.max_qh < 148 * 16 ? L.max_qh : 148 * 16), n);
    const unsigned nb = (unsigned)(max_bands < 148 * 8 ? max_bands : 148 * 8);
    k_band_union<<<dim3(nb, n), 256, smem, L.stream>>>(frames, thr, runs, row_nruns, words);
    k_band_join<<<dim3(nb, n), 256, 0, L.stream>>>(frames, thr, runs, row_nruns, words);
    k_root_sums<<<rg, 256, 0, L.stream>>>(frames, runs, row_nruns);
    if (warp_rows(L)) {
        const int64_t b = (L.max_qh + 7) / 8;
        k_labels_w<<<dim3((unsigned)(b < 1 ? 1 : b < 148 * 8 ? b : 148 * 8), n), 256, 0, L.stream>>>(
            frames, thr, runs, row_nruns, lab, min_px);
    } else
        k_labels<<<rg, LAB_THREADS, 0, L.stream>>>(frames, runs, row_nruns, lab, min_px);
    return 4;
}

void segment_plan(int qw, int qh, int64_t *max_bands, size_t *smem) {
    if (qw <= 0) return;
    const int64_t b = (qh + band_rows(qw) - 1) / band_rows(qw);
    if (b > *max_bands) *max_bands = b;
    if (band_smem(qw) > *smem) *smem = band_smem(qw);
}

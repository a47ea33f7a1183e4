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
//   k_band_union   a block per band of rows: masks, run numbers, the unions
//                  inside the band in shared memory; every run then points
//                  at its band root (its set's smallest run), which holds
//                  the band component's pixels.
//   k_band_join    the unions across band edges and of the last column, in
//                  global memory.
//   k_root_sums    each band root adds its pixels to its component's root
//                  and points at it (so a run is two steps from its root).
//   k_run_labels   each run's label; the masks of pixels without one cleared.
//   k_labels       the labels per pixel, for the sorting fallback of the
//                  clusters and the diagnostics only.
#include <cuda_runtime.h>
#include <stdint.h>

#include "at_device.cuh"
#include "at_gpu.h"
#include "at_kernels.h"
#include "at_launch.h"

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
// ids (row << band_shift | run) stay within 16384 (and their 16-bit array
// within 32 KB). Images over 16384 wide get bands of one row, whose runs are
// their own band roots.
#define BAND_IDS 16384
#define BAND_SEEN 512
#define BAND_LIST 4096  // touching pairs listed at once (more are united where they are found)
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
    const size_t ids = (1 << s) > BAND_IDS ? 0 : (size_t)r << s;
    return (size_t)r * ((qw + 31) / 32) * 16 + 2 * ids + (2 * ids > 4 * BAND_LIST ? 2 * ids : 4 * BAND_LIST);
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

// Calls add(x, val) for the active lanes (every lane calls it): once with
// the sum for the lanes that share the first active lane's x, then for the
// others each. Components are few and large or many and small; finding all
// groups (match_any, a reduction per group) took 10 times as long.
template <class F>
__device__ __forceinline__ void by_root(uint32_t x, uint32_t val, bool act, F add) {
    const uint32_t am = __ballot_sync(0xffffffffu, act);
    if (!am) return;
    const uint32_t x0 = __shfl_sync(0xffffffffu, x, __ffs(am) - 1);
    const bool same = act && x == x0;
    const uint32_t sum = __reduce_add_sync(0xffffffffu, same ? val : 0u);
    if ((int)(threadIdx.x & 31) == __ffs(am) - 1) add(x0, sum);
    if (act && !same) add(x, val);
}

// Unions over band-local ids in shared memory, lock-free, the larger id
// hooked under the smaller, so a root is its set's smallest node and the
// large sets' roots stay where they are (in the order of a hash the root of
// the largest set moves and every union that meets it waits for the others:
// 42k cycles a band instead of 32k).
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
                                                    uint32_t *row_nruns, uint32_t *band_roots, RowWord *words) {
    kernel_begin();
    extern __shared__ __align__(16) uint8_t s_band[];
    __shared__ uint32_t s_n, s_m;
    const FrameDesc f = frames[blockIdx.y];
    const int tid = threadIdx.x, lane = tid & 31;
    const int qw = f.qw, nw = (qw + 31) / 32, sh = band_shift(qw), R = band_rows(qw);
    const bool solo = (1 << sh) > BAND_IDS;
    RowWord *s_word = reinterpret_cast<RowWord *>(s_band);
    uint16_t *s_par = reinterpret_cast<uint16_t *>(s_word + R * nw);
    uint32_t *s_list = reinterpret_cast<uint32_t *>(s_par + (solo ? 0 : R << sh));
    const uint32_t list_cap = max((uint32_t)BAND_LIST, solo ? 0u : (uint32_t)(R << sh) / 2);
    uint32_t *s_px = s_list;  // after the unions: two 16-bit counts a word (a band has at most 16384 pixels)
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
        if (tid == 0) s_n = s_m = 0;
        __syncthreads();
        // run starts and the runs before each word, a warp per row; each run
        // its own set (the rows' nodes are written in order)
        for (int r = tid >> 5; r < nr; r += blockDim.x >> 5) {
            uint32_t n = 0;
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
                    w->before = n + off;
                }
                n += total;
            }
            const int64_t base = node0 + (int64_t)r * qw;
            for (uint32_t k = lane; k < n; k += 32) {
                if (!solo)
                    s_par[(r << sh) + k] = (uint16_t)((r << sh) + k);
                else
                    runs.px[base + k] = 0;
            }
            if (lane == 0) {
                row_nruns[f.row0 + y0 + r] = n;
                const int64_t vn = f.node_off + (int64_t)qw * f.qh + y0 + r;
                runs.parent[vn] = (uint32_t)vn;
                runs.px[vn] = 1;
                runs.minid[vn] = (uint32_t)vn;
            }
        }
        // every run to its root so far (a thread walks on from what others
        // found); at last the pixel counts, in the list's place, cleared
        auto flatten = [&](bool last) {
            if (solo) return;
            for (int r = tid >> 5; r < nr; r += blockDim.x >> 5) {
                const RowWord &lw = s_word[r * nw + nw - 1];
                const uint32_t n = lw.before + __popc(lw.starts);
                for (uint32_t k = lane; k < n; k += 32) {
                    const uint32_t l = (uint32_t)(r << sh) + k;
                    const volatile uint16_t *par = s_par;
                    uint32_t x = l;
                    for (uint32_t p = par[x]; p != x; p = par[x]) x = p;
                    s_par[l] = (uint16_t)x;
                    if (last) reinterpret_cast<uint16_t *>(s_px)[l] = 0;
                }
            }
        };
        __syncthreads();
        for (int it = tid; it < nr * nw; it += blockDim.x) out[it] = s_word[it];
        // the touching pairs; any run above that a run touches is its first
        // parent (one plain store wins: the trees go up row by row, so no
        // cycle), which leaves few unions to make
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
                    s_par[c] = (uint16_t)a;
                    if (at < list_cap) s_list[at] = c | a << 16;
                    at++;
                });
        }
        __syncthreads();
        flatten(false);  // most pairs are then one step from one root
        __syncthreads();
        // the pairs of different roots, as root pairs, to the list's front;
        // then a union per thread
        const uint32_t np = min(s_n, list_cap);
        for (uint32_t p0 = 0; p0 < np; p0 += blockDim.x) {
            uint32_t c = 0, a = 0;
            if (p0 + tid < np) {
                const uint32_t e = s_list[p0 + tid];
                c = s_par[e & 0xffffu];
                a = s_par[e >> 16];
            }
            __syncthreads();
            const uint32_t at = list_places(c != a ? 1u : 0u, &s_m);
            if (c != a) s_list[at] = c | a << 16;  // at or before the places read
            __syncthreads();
        }
        const uint32_t nu = s_m;
        for (uint32_t p = tid; p < nu; p += blockDim.x) lu_unite(s_par, s_list[p] & 0xffffu, s_list[p] >> 16);
        if (s_n > list_cap) {  // the pairs that the list did not hold: all of them again
            for (int it = nw + tid; it < nr * nw; it += blockDim.x) {
                const int r = it / nw, i = it - r * nw;
                const RowWord *cur = s_word + r * nw, *abv = cur - nw;
                for_pairs(cur, abv, i, pair_masks(cur, abv, i, nw, qw), [&](uint32_t c, uint32_t a) {
                    lu_unite(s_par, c + ((uint32_t)r << sh), a + ((uint32_t)(r - 1) << sh));
                });
            }
        }
        __syncthreads();
        flatten(true);
        if (tid == 0) s_n = 0;
        __syncthreads();
        // the pixels of the words' pieces of runs to their band roots
        for (int it0 = 0; it0 < nr * nw; it0 += blockDim.x) {
            const int it = it0 + tid, r = it / nw, i = it - r * nw;
            RowWord w = {0, 0, 0, 0};
            uint32_t m = 0;
            if (it < nr * nw) {
                w = s_word[it];
                m = (w.white | w.black) & run_columns(i, qw);
            }
            const uint32_t stop = w.starts | ~m;
            while (__any_sync(0xffffffffu, m != 0)) {
                const bool act = m != 0;
                uint32_t x = 0, z = 0;
                if (act) {
                    const int c = __ffs(m) - 1;
                    const uint32_t past = c < 31 ? stop & (~0u << (c + 1)) : 0u;
                    const int e = past ? __ffs(past) - 1 : 32;
                    m = e < 32 ? m & (~0u << e) : 0u;
                    x = (uint32_t)(r << sh) + run_at(w, c);
                    z = (uint32_t)(e - c);
                    if (!solo) x = s_par[x];
                }
                by_root(x, z, act, [&](uint32_t to, uint32_t sum) {
                    if (solo)
                        atomicAdd(runs.px + node0 + to, sum);
                    else
                        atomicAdd(s_px + (to >> 1), sum << (16 * (to & 1)));
                });
            }
        }
        __syncthreads();
        for (int r = tid >> 5; r < nr; r += blockDim.x >> 5) {
            const RowWord &lw = s_word[r * nw + nw - 1];
            const uint32_t n = lw.before + __popc(lw.starts);
            const int64_t base = node0 + (int64_t)r * qw;
            for (uint32_t k = lane; k < n; k += 32) {
                const uint32_t l = (uint32_t)(r << sh) + k, x = solo ? l : s_par[l];
                runs.parent[base + k] = (uint32_t)(node0 + (int64_t)(x >> sh) * qw + (x & ((1u << sh) - 1u)));
                if (!solo) runs.px[base + k] = x == l ? reinterpret_cast<uint16_t *>(s_px)[l] : 0u;  // not 0: a band root
                if (x == l) {
                    runs.minid[base + k] = (uint32_t)(base + k);
                    runs.lab[node0 + atomicAdd(&s_n, 1u)] = (uint32_t)(base + k);  // the band's roots, listed
                }
            }
        }
        __syncthreads();
        if (tid == 0) band_roots[f.row0 + y0] = s_n;
    }
}

// The unions across band edges, a block per edge, and the last-column links
// of every row (fast/unionfind.c:89-97).
__global__ void __launch_bounds__(256) k_band_join(const FrameDesc *frames, RunArrays runs, const uint32_t *row_nruns,
                                                   const RowWord *words) {
    kernel_begin();
    // a union per thread from the list: unions straight from the words' loops
    // kept their warps waiting for their slowest lane (200 us for one
    // 640 x 480 frame)
    __shared__ uint32_t s_list[BAND_LIST], s_n;
    __shared__ unsigned long long s_seen[BAND_SEEN];
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
        // most pairs repeat another's two band roots: a lossy table of the
        // last pair met per place lets most of them through once only
        for (int t = tid; t < BAND_SEEN; t += blockDim.x) s_seen[t] = 0;
        __syncthreads();
        const uint32_t np = min(s_n, (uint32_t)BAND_LIST);
        for (uint32_t p = tid; p < np; p += blockDim.x) {
            const uint32_t c = runs.parent[base + (s_list[p] & 0xffffu)], a = runs.parent[above + (s_list[p] >> 16)];
            const unsigned long long k = (unsigned long long)c << 32 | a;  // never 0: c is below the frame's first row
            if (atomicExch(s_seen + ((c * 0x9e3779b1u ^ a * 0x85ebca6bu) >> 23), k) == k) continue;
            uf_unite(runs.parent, c, a);
        }
    }
    // the last run of row y reaches column qw - 2, white; above it only the
    // last column is white
    for (int64_t y = 1 + (int64_t)blockIdx.x * blockDim.x + tid; y < f.qh; y += (int64_t)gridDim.x * blockDim.x) {
        const RowWord *cur = words + f.word_off + y * nw, *abv = cur - nw;
        auto white = [&](const RowWord *row, int x) { return row[x >> 5].white >> (x & 31) & 1u; };
        if (white(cur, qw - 2) && white(abv, qw - 1) && !white(abv, qw - 2))
            uf_unite(runs.parent, (uint32_t)(f.node_off + y * qw + row_nruns[f.row0 + y] - 1),
                     (uint32_t)(f.node_off + (int64_t)qw * f.qh + y - 1));
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

// Each band root (and last-column node) adds its pixels and offers its id
// to its component's root, and from here on points at it. A block gathers
// its sums by root in shared memory first: the pieces of a frame's background
// all lie under one node, whose atomics followed one another (4032 x 3024:
// 160 us with the sums of a warp's lanes gathered, 60 us so).
#define SUM_ROOTS 256
#define SUM_PROBES 8
__global__ void __launch_bounds__(128) k_root_sums(const FrameDesc *frames, RunArrays runs, const uint32_t *band_roots) {
    kernel_begin();
    __shared__ uint32_t s_root[SUM_ROOTS], s_px[SUM_ROOTS], s_min[SUM_ROOTS];
    const FrameDesc f = frames[blockIdx.y];
    const int R = band_rows(f.qw > 0 ? f.qw : 1), nband = (f.qh + R - 1) / R;
    if ((int)blockIdx.x >= nband) return;
    for (int t = threadIdx.x; t < SUM_ROOTS; t += blockDim.x) {
        s_root[t] = s_min[t] = 0xffffffffu;
        s_px[t] = 0;
    }
    __syncthreads();
    for (int b = blockIdx.x; b < nband; b += gridDim.x) {
        const int y0 = b * R, nr = min(R, f.qh - y0);
        const uint32_t n = band_roots[f.row0 + y0];
        const uint32_t *list = runs.lab + f.node_off + (int64_t)y0 * f.qw;
        for (uint32_t i0 = 0; i0 < n + nr; i0 += blockDim.x) {
            const uint32_t i = i0 + threadIdx.x;
            uint32_t node = 0, px = 0, r = 0;
            bool add = false;
            if (i < n + nr) {
                node = i < n ? list[i] : (uint32_t)(f.node_off + (int64_t)f.qw * f.qh + y0 + (i - n));
                // a component's root is a band root too, and its count may
                // grow meanwhile, but it adds to no other
                px = runs.px[node];
                r = uf_root(runs.parent, node);
                add = r != node;
            }
            // no unions run any more: pointing straight at the root is safe
            // for the walks of other threads
            if (add) runs.parent[node] = r;
            // the lanes of the first one's root together, the others alone
            const uint32_t am = __ballot_sync(0xffffffffu, add);
            if (!am) continue;
            const int lead = __ffs(am) - 1;
            const uint32_t r0 = __shfl_sync(0xffffffffu, r, lead);
            const bool same = add && r == r0;
            const uint32_t sum = __reduce_add_sync(0xffffffffu, same ? px : 0u);
            const uint32_t low = __reduce_min_sync(0xffffffffu, same ? node : 0xffffffffu);
            if ((int)(threadIdx.x & 31) == lead) {
                px = sum;
                node = low;
            } else if (same || !add) {
                continue;
            }
            uint32_t h = (r * 0x9e3779b1u) >> 24;
            int p = 0;
            for (; p < SUM_PROBES; p++, h = (h + 1) & (SUM_ROOTS - 1)) {
                uint32_t cur = *(volatile uint32_t *)(s_root + h);
                if (cur == 0xffffffffu) cur = atomicCAS(s_root + h, 0xffffffffu, r);
                if (cur == 0xffffffffu || cur == r) break;
            }
            if (p < SUM_PROBES) {
                atomicAdd(s_px + h, px);
                atomicMin(s_min + h, node);
            } else {
                atomicAdd(runs.px + r, px);
                atomicMin(runs.minid + r, node);
            }
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < SUM_ROOTS; t += blockDim.x) {
        const uint32_t r = s_root[t];
        if (r == 0xffffffffu) continue;
        atomicAdd(runs.px + r, s_px[t]);
        if (s_min[t] < *(volatile uint32_t *)(runs.minid + r)) atomicMin(runs.minid + r, s_min[t]);
    }
}

// Each run's label (its component's smallest node id, or AT_NOK when the
// component has fewer than min_px pixels), and the last-column nodes'; the
// row masks keep only the pixels of labelled runs (and of the last column),
// so that the points need no labels to be found. A warp per row: the runs in
// order, then a word a lane.
__global__ void __launch_bounds__(256) k_run_labels(const FrameDesc *frames, RunArrays runs, const uint32_t *row_nruns,
                                                    RowWord *words, int32_t min_px) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const int qw = f.qw, nw = (qw + 31) / 32;
    auto label_of = [&](int64_t node) -> uint32_t {
        const uint32_t r = root_of(runs, node);
        return (int64_t)runs.px[r] >= min_px ? runs.minid[r] : AT_NOK;
    };
    for (int y = (int)blockIdx.x * wpb + (threadIdx.x >> 5); y < f.qh; y += (int)gridDim.x * wpb) {
        const int64_t base = f.node_off + (int64_t)y * qw, vn = f.node_off + (int64_t)qw * f.qh + y;
        const uint32_t n = row_nruns[f.row0 + y];
        for (uint32_t k = lane; k < n; k += 64) {
            const uint32_t k2 = k + 32 < n ? k + 32 : k;
            const uint32_t a = label_of(base + k), b = label_of(base + k2);
            runs.lab[base + k] = a;
            runs.lab[base + k2] = b;
        }
        const uint32_t lv = label_of(vn);
        if (lane == 0) runs.lab[vn] = lv;
        __syncwarp();
        for (int i = lane; i < nw; i += 32) {
            RowWord *w = words + f.word_off + (int64_t)y * nw + i;
            const RowWord o = *w;
            uint32_t m = (o.white | o.black) & run_columns(i, qw), keep = 0;
            const uint32_t stop = o.starts | ~m;
            while (m) {
                const int c = __ffs(m) - 1;
                const uint32_t past = c < 31 ? stop & (~0u << (c + 1)) : 0u;
                const uint32_t below = past ? (past & (0u - past)) - 1u : ~0u;  // columns before the piece's end
                if (runs.lab[base + run_at(o, c)] != AT_NOK) keep |= m & below;
                m &= ~below;
            }
            if (i == (qw - 1) >> 5 && lv != AT_NOK) keep |= 1u << ((qw - 1) & 31);
            w->white = o.white & keep;
            w->black = o.black & keep;
        }
        __syncwarp();
    }
}

// The labels per pixel, a block per row (the last column: the row's extra
// node), from k_run_labels.
__global__ void __launch_bounds__(256) k_labels(const FrameDesc *frames, RunArrays runs, const RowWord *words,
                                                uint32_t *lab) {
    kernel_begin();
    const FrameDesc f = frames[blockIdx.y];
    const int qw = f.qw, nw = (qw + 31) / 32;
    for (int y = blockIdx.x; y < f.qh; y += gridDim.x)
        for (int x = threadIdx.x; x < qw; x += blockDim.x) {
            const RowWord w = words[f.word_off + (int64_t)y * nw + (x >> 5)];
            uint32_t l = AT_NOK;
            if (x == qw - 1)
                l = runs.lab[f.node_off + (int64_t)qw * f.qh + y];
            else if ((w.white | w.black) >> (x & 31) & 1u)
                l = runs.lab[f.node_off + (int64_t)y * qw + run_at(w, x & 31)];
            lab[f.q_off + (int64_t)y * qw + x] = l;
        }
}

// ---------------------------------------------------------------------------
// Launchers.

bool segment_set_smem() {
    // 80 KB hold 8 rows of 2048 columns or one of 16384; the words alone of a
    // wider row take 16 bytes per 32 columns
    return cudaFuncSetAttribute(k_band_union, cudaFuncAttributeMaxDynamicSharedMemorySize, SEGMENT_SMEM) == cudaSuccess;
}

int launch_segment(const Launch &L, const FrameDesc *frames, int64_t max_bands, size_t smem, const uint8_t *thr,
                   RunArrays runs, uint32_t *row_nruns, uint32_t *band_roots, RowWord *words, int32_t min_px) {
    const unsigned n = (unsigned)L.nframes;
    const unsigned nb = (unsigned)(max_bands < 148 * 8 ? max_bands : 148 * 8);
    launch(k_band_union, dim3(nb, n), 256, smem, L.stream, frames, thr, runs, row_nruns, band_roots, words);
    launch(k_band_join, dim3(nb, n), 256, 0, L.stream, frames, runs, row_nruns, words);
    launch(k_root_sums, dim3(nb, n), 128, 0, L.stream, frames, runs, band_roots);
    const int64_t b = (L.max_qh + 7) / 8;
    launch(k_run_labels, dim3((unsigned)(b < 1 ? 1 : b < 148 * 8 ? b : 148 * 8), n), 256, 0, L.stream, 
        frames, runs, row_nruns, words, min_px);
    return 4;
}

void launch_labels(const Launch &L, const FrameDesc *frames, RunArrays runs, const RowWord *words, uint32_t *lab) {
    const unsigned rows = (unsigned)(L.max_qh < 148 * 16 ? L.max_qh : 148 * 16);
    launch(k_labels, dim3(rows < 1 ? 1 : rows, (unsigned)L.nframes), 256, 0, L.stream, frames, runs, words, lab);
}

void segment_plan(int qw, int qh, int64_t *max_bands, size_t *smem) {
    if (qw <= 0) return;
    const int64_t b = (qh + band_rows(qw) - 1) / band_rows(qw);
    if (b > *max_bands) *max_bands = b;
    if (band_smem(qw) > *smem) *smem = band_smem(qw);
}

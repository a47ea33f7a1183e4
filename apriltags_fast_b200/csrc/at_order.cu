// The reference's order of the quads whose detections share an id.
//
// Why it matters. The reference hands its detections to a stable sort by
// id in quad order (fast/detector.c:143-179), and its reconcile of
// overlapping detections of one tag walks them in that order
// (fast/decode.c:860-891). So the quad order decides the output exactly
// when two detections of a frame have the same id. Quad order is cluster
// order, and the reference orders clusters by (hash bucket, id) of the key
// (larger root << 32) + smaller root of the two components a cluster lies
// between (fast/clusters.c:44, 97-103, 338-356), where a component's root
// is the node that the reference's sequential union by size over the runs
// in raster order leaves at the top (fast/unionfind.c:15-45, 152-196,
// 284-298), numbered as the reference packs its nodes (the runs row after
// row, then one node per row for the last column).
//
// The GPU's union-find is parallel and labels a component by its smallest
// node, which fixes the partition but not the reference's root. These
// kernels find that root for the few components that matter and give the
// final stage the reference's order keys:
//
//   k_ref_targets   per frame: the ids that two or more detections share;
//                   the components of their quads are the targets (their
//                   GPU labels and pixel counts); the packed run numbering.
//   k_ref_mark      the runs of the target components, row by row, compacted
//                   (start, end, index in row, value, target).
//   k_ref_link      all unions of the targets' runs, in any order, each with
//                   its time, into a forest that holds every set at every
//                   time (see below).
//   k_ref_sums      the pixels below each node of the forest; per target
//                   and row, the pixels its first set gains there.
//   k_ref_root      a block per target: the root, from the last union back.
//   k_finalize      (at_kernels.cu) orders those detections by the keys.
//
// The time of a union is the node id of the row's run that makes it: the
// reference's calls of run i (its touching runs above, in order) all have
// time i, and a row's last-column link the id after the row's last possible
// run. A node u of the forest has a parent p and a time w: from time w on, u
// is in p's set. Parents have smaller ids, so the top of a set is its oldest
// run, and the set of u at time T is found by climbing while w <= T. A union
// of a and b at time w climbs both to their tops at w and hangs the younger
// under the older; if that node had a (later) parent already, the old edge
// is inserted again, from its new parent. The result does not depend on the
// order of insertion, so all unions of a frame run in parallel (lock-free,
// one 64-bit word per node). Last, each parent is moved up to its set's top
// at the edge's time (k_ref_sums), so that times grow strictly towards the
// top and the pixels below u are its whole set when it joins p.
//
// The root. In a union the set with more pixels keeps its root. So the root
// of a set of Z pixels is the root of the first set inside it to hold more
// than Z / 2: no later union inside can take the root from that one. From
// the whole component back: with x the top of the current set, its size
// after each row is len(x) plus a prefix sum of what it gains per row; the
// first row that leaves more than Z / 2 takes over as the current set, with
// its own Z. When that is the current row itself, the row's events on x are
// summed in order up to the one that crosses Z / 2, the reference's calls
// of that one event are replayed on the sets' sizes, and the winner's set
// just before it is the current set, until a set is a single run. Z halves
// each time, so a set of 8 million pixels takes some tens of steps; the
// unions that cannot decide (nearly all) are never replayed. A row-by-row
// replay of every union of the target runs in bands, with a pass over the
// bands' edges, took 36 ms for a 4032 x 3024 frame whose background is a
// target, and 10.7 ms for 16 frames of 640 x 480 to 3840 x 2160.
#include <cuda_runtime.h>
#include <stdint.h>

#include "at_device.cuh"
#include "at_gpu.h"
#include "at_kernels.h"
#include "at_launch.h"

#define REF_HASH 1024          // open-addressing table of target labels (k_ref_targets, k_ref_mark)
#define REF_NONE 0xffu         // no target
static_assert(AT_REF_MAXT < REF_NONE, "target indices fit a byte");
static_assert(2 * AT_REF_MAXT <= REF_HASH, "the label table stays half empty");

__device__ __forceinline__ uint32_t ref_hash(uint32_t x) {
    x *= 0x9e3779b1u;
    return x ^ (x >> 15);
}

// A label's target index in a table of (label + 1, index) pairs; REF_NONE
// when absent.
__device__ __forceinline__ uint32_t ref_lookup(const uint32_t *keys, const uint8_t *idx, uint32_t label) {
    uint32_t h = ref_hash(label) & (REF_HASH - 1);
    for (int p = 0; p < REF_HASH; p++) {
        const uint32_t k = keys[h];
        if (k == 0) return REF_NONE;
        if (k == label + 1) return idx[h];
        h = (h + 1) & (REF_HASH - 1);
    }
    return REF_NONE;
}

// ---------------------------------------------------------------------------
// Targets: a block per frame. The ids seen twice are found with two bit
// sets over all ids (an id is below 65536): one pass over the detections.
// (Comparing every pair of slots took 4.1 ms for 2602 quads x 2 families.)

__global__ void __launch_bounds__(256) k_ref_targets(const FrameDesc *frames, int nfam, const int64_t *qstart,
                                                     const GpuDetection *dets, const uint32_t *det_ok,
                                                     const uint32_t *qcl, const uint64_t *ckey, int nb,
                                                     RunArrays runs, const uint32_t *row_nruns, RefOrder ref,
                                                     uint32_t *err) {
    kernel_begin();
    __shared__ uint32_t s_once[2048], s_twice[2048];
    __shared__ uint32_t s_key[REF_HASH];
    __shared__ uint32_t s_n, s_need, s_over;
    __shared__ uint32_t s_scan[32];
    const int f = blockIdx.x;
    const FrameDesc fd = frames[f];
    for (int i = threadIdx.x; i < 2048; i += blockDim.x) s_once[i] = s_twice[i] = 0;
    for (int i = threadIdx.x; i < REF_HASH; i += blockDim.x) s_key[i] = 0;
    if (threadIdx.x == 0) s_n = s_need = s_over = 0;
    __syncthreads();
    const int64_t a = qstart[f] * nfam, b = qstart[f + 1] * nfam;
    const uint64_t lmask = ((uint64_t)1 << nb) - 1;
    for (int64_t s = a + threadIdx.x; s < b; s += blockDim.x) {
        if (!det_ok[s]) continue;
        const uint32_t id = (uint32_t)dets[s].id & 0xffffu, bit = 1u << (id & 31);
        if (atomicOr(&s_once[id >> 5], bit) & bit) {
            atomicOr(&s_twice[id >> 5], bit);
            s_need = 1;
        }
    }
    __syncthreads();
    if (s_need)
        for (int64_t s = a + threadIdx.x; s < b; s += blockDim.x) {
            if (!det_ok[s]) continue;
            const uint32_t id = (uint32_t)dets[s].id & 0xffffu;
            if (!(s_twice[id >> 5] >> (id & 31) & 1u)) continue;
            const uint64_t key = ckey[qcl[s / nfam]];
            const uint32_t lab[2] = {(uint32_t)(key >> nb), (uint32_t)(key & lmask)};
            for (int k = 0; k < 2; k++) {
                uint32_t h = ref_hash(lab[k]) & (REF_HASH - 1);
                int p = 0;
                for (; p < REF_HASH; p++) {
                    const uint32_t old = atomicCAS(&s_key[h], 0u, lab[k] + 1);
                    if (old == 0u || old == lab[k] + 1) break;
                    h = (h + 1) & (REF_HASH - 1);
                }
                if (p == REF_HASH) s_over = 1;
            }
        }
    __syncthreads();
    uint32_t *tl = ref.tlabel + (int64_t)f * AT_REF_MAXT;
    uint32_t *tp = ref.tpx + (int64_t)f * AT_REF_MAXT;
    for (int i = threadIdx.x; i < REF_HASH; i += blockDim.x) {
        if (!s_key[i]) continue;
        const uint32_t t = atomicAdd(&s_n, 1u);
        if (t >= AT_REF_MAXT) {
            s_over = 1;
            continue;
        }
        const uint32_t label = s_key[i] - 1;
        tl[t] = label;
        tp[t] = runs.px[root_of(runs, label)];
    }
    __syncthreads();
    const bool need = s_need && !s_over;
    if (threadIdx.x == 0) {
        ref.need[f] = need ? 1u : 0u;
        ref.nt[f] = need ? s_n : 0u;
        if (s_over) atomicOr(err, AT_ERR_CAPACITY);
    }
    if (!need) return;
    // the reference's packed numbering: runs of the rows above row y
    uint32_t *pre = ref.rpre + fd.row0 + f;
    uint32_t base = 0;
    for (int64_t y0 = 0; y0 < fd.qh; y0 += blockDim.x) {
        const int64_t y = y0 + threadIdx.x;
        const uint32_t c = y < fd.qh ? row_nruns[fd.row0 + y] : 0u;
        uint32_t total;
        const uint32_t off = block_excl_scan(c, &total, s_scan);
        if (y < fd.qh) pre[y] = base + off;
        base += total;
    }
    if (threadIdx.x == 0) pre[fd.qh] = base;
}

// ---------------------------------------------------------------------------
// The target runs of each row, compacted, a warp per row:
//   tlist[node_off + y qw + j] = start | end << 16 | index << 32 | v << 48 | target << 56
//   trow[row0 + y] = count | (the last-column link joins a target run) << 31
// and each of them (and each link's last-column node) a root of the forest.

// A row's targets are looked up a run a lane first (its labels lie side by
// side), and their entries gathered before they are written (4032 x 3024: 155
// us when a lane looked up and wrote its word's runs one by one, 107 with the
// look-up alone, 75 so; 16 frames of mixed sizes 57 and 44).
#define REF_ROW_RUNS ((REF_PCAP + 32) & ~31)  // runs of a row, at most
#define REF_STAGE 128                         // entries gathered before they are written

#define REF_INF 0xffffffffu  // the time of a root: never joined

__device__ __forceinline__ uint32_t ref_col(uint64_t e) { return (uint32_t)(e >> 32) & 0xffffu; }  // run index in the row
__device__ __forceinline__ uint32_t ref_len(uint64_t e) { return (uint32_t)(e >> 16 & 0xffff) - (uint32_t)(e & 0xffff) + 1; }

__device__ __forceinline__ void ref_node_init(const RefOrder &ref, uint32_t node, uint32_t px) {
    ref.par[node] = (uint64_t)REF_INF << 32 | node;
    ref.sum[node] = px;
    ref.stamp[node] = 0;
}

__global__ void __launch_bounds__(256) k_ref_mark(const FrameDesc *frames, const RowWord *words, RunArrays runs,
                                                  const uint32_t *row_nruns, RefOrder ref) {
    kernel_begin();
    __shared__ uint32_t s_key[REF_HASH];
    __shared__ uint8_t s_idx[REF_HASH];
    const int f = blockIdx.y;
    if (!ref.need[f]) return;
    const FrameDesc fd = frames[f];
    for (int i = threadIdx.x; i < REF_HASH; i += blockDim.x) s_key[i] = 0;
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < ref.nt[f]; t += blockDim.x) {
        const uint32_t label = ref.tlabel[(int64_t)f * AT_REF_MAXT + t];
        uint32_t h = ref_hash(label) & (REF_HASH - 1);
        while (atomicCAS(s_key + h, 0u, label + 1)) h = (h + 1) & (REF_HASH - 1);  // (the table is half empty)
        s_idx[h] = (uint8_t)t;
    }
    __syncthreads();
    extern __shared__ __align__(16) uint8_t s_target[];  // by run of the warp's row
    uint8_t *mine = s_target + (threadIdx.x >> 5) * (REF_ROW_RUNS + 8 * REF_STAGE);
    uint64_t *stage = reinterpret_cast<uint64_t *>(mine + REF_ROW_RUNS);
    const int lane = threadIdx.x & 31;
    const int64_t wpb = blockDim.x >> 5;
    const int qw = fd.qw, nw = (qw + 31) / 32;
    for (int64_t y = blockIdx.x * wpb + (threadIdx.x >> 5); y < fd.qh; y += gridDim.x * wpb) {
        const int64_t base = fd.node_off + y * qw;
        const RowWord *row = words + fd.word_off + y * nw;
        uint32_t cnt = 0;
        // the row's runs, 32 at a time: their targets (a run of no label
        // looks up what no table holds)
        const uint32_t nr = row_nruns[fd.row0 + y];
        __syncwarp();
        for (uint32_t k = lane; k < nr; k += 32) mine[k] = (uint8_t)ref_lookup(s_key, s_idx, runs.lab[base + k]);
        __syncwarp();
        for (int i0 = 0; i0 < nw; i0 += 32) {
            // a word a lane: its target runs, then (after the lanes before) their entries
            const int i = i0 + lane;
            RowWord w = {0, 0, 0, 0};
            uint32_t tm = 0;
            if (i < nw) {
                w = row[i];
                uint32_t k = w.before;
                for (uint32_t m = w.starts; m; m &= m - 1, k++)
                    if (((w.white | w.black) & m & (0u - m)) && mine[k] != REF_NONE) tm |= m & (0u - m);
            }
            uint32_t total;
            const uint32_t off = warp_excl_scan(__popc(tm), &total), last = off + __popc(tm);
            // the entries of as many words as there is room for (a word has
            // 32 at most), then written a run a lane
            for (uint32_t from = 0, to; from < total; from = to) {
                const bool fits = last <= from + REF_STAGE;
                to = __reduce_max_sync(0xffffffffu, fits ? last : 0u);
                if (fits && off >= from) {
                    uint64_t *out = stage + (off - from);
                    for (uint32_t m = tm; m; m &= m - 1) {
                        const int c = __ffs(m) - 1;
                        const uint32_t k = run_at(w, c), t = mine[k];
                        const bool white = w.white >> c & 1u;
                        // the run's end: the first later column of another value or the last run column
                        int e = 32 * i + c + 1;
                        for (int j = i; j < nw; j++) {
                            const uint32_t colour = (white ? row[j].white : row[j].black) & run_columns(j, qw);
                            const uint32_t stop = ~colour & (j == i ? ~0u << c : ~0u);
                            e = 32 * j + (stop ? __ffs(stop) - 1 : 32);
                            if (stop) break;
                        }
                        *out++ = (uint64_t)(uint32_t)(32 * i + c) | (uint64_t)(uint32_t)(e - 1) << 16 | (uint64_t)k << 32 |
                                 (uint64_t)(white ? 255 : 0) << 48 | (uint64_t)t << 56;
                    }
                }
                __syncwarp();
                for (uint32_t j = from + lane; j < to; j += 32) {
                    const uint64_t e = stage[j - from];
                    const int64_t node = base + ref_col(e);
                    ref.tlist[base + cnt + j] = e;
                    ref_node_init(ref, (uint32_t)node, ref_len(e));
                    ref.len[node] = (uint16_t)ref_len(e);
                }
                __syncwarp();
            }
            cnt += total;
        }
        if (lane == 0) {
            // the last-column link (the masks hold labelled pixels only; a
            // target's are, and so is what it touches)
            bool link = false;
            if (y >= 1) {
                auto white = [&](const RowWord *r, int x) { return r[x >> 5].white >> (x & 31) & 1u; };
                link = white(row, qw - 2) && white(row - nw, qw - 1) && !white(row - nw, qw - 2) &&
                       mine[nr - 1] != REF_NONE;
            }
            if (link) ref_node_init(ref, (uint32_t)(fd.node_off + (int64_t)qw * fd.qh + y - 1), 1u);
            ref.trow[fd.row0 + y] = cnt | (link ? 0x80000000u : 0u);
        }
    }
}

// ---------------------------------------------------------------------------
// The forest: par[node] = time << 32 | parent (a root: REF_INF << 32 | node).

__device__ __forceinline__ uint64_t ref_par(const RefOrder &ref, uint32_t u) {
    return *(const volatile uint64_t *)(ref.par + u);
}

// The top of u's set at time T.
__device__ __forceinline__ uint32_t ref_climb(const RefOrder &ref, uint32_t u, uint32_t T) {
    uint64_t p = ref_par(ref, u);
    while ((uint32_t)(p >> 32) <= T) {
        u = (uint32_t)p;
        p = ref_par(ref, u);
    }
    return u;
}

// u and v are in one set from time w on (w < REF_INF). A failed CAS means
// another thread changed u's edge: climb again. Ids fall along every path,
// so there is no cycle, and each CAS that succeeds replaces an edge by an
// earlier one.
__device__ __forceinline__ void ref_insert(const RefOrder &ref, uint32_t u, uint32_t v, uint32_t w) {
    for (;;) {
        u = ref_climb(ref, u, w);
        v = ref_climb(ref, v, w);
        if (u == v) return;
        if (u < v) {
            const uint32_t t = u;
            u = v;
            v = t;
        }
        const uint64_t old = ref_par(ref, u);
        if ((uint32_t)(old >> 32) <= w) continue;
        if (atomicCAS(reinterpret_cast<unsigned long long *>(ref.par + u), old, (uint64_t)w << 32 | v) != old) continue;
        if ((uint32_t)(old >> 32) == REF_INF) return;
        u = v;  // the edge that was there, from the new parent
        v = (uint32_t)old;
        w = (uint32_t)(old >> 32);
    }
}


// A block per row: each target run's touching runs in the row above (they
// are target runs too), kept for k_ref_root in tch[rbase + j] (first | last
// << 16 of the row above's list, 0xffffffff: none; the runs of its value
// between them touch it as well), and the unions with them, listed first
// and then one per thread (a union climbs to two tops through L2; from the
// runs' own loops the warps waited for their slowest lane). A block per row:
// the rows of one frame alone have too few runs for a warp per row.
#define REF_ROW_THREADS 128
#define REF_LIST 2048  // unions listed at once (more are made where they are found)
__global__ void __launch_bounds__(REF_ROW_THREADS) k_ref_link(const FrameDesc *frames, RefOrder ref) {
    kernel_begin();
    __shared__ uint32_t s_list[REF_LIST], s_n;
    const int f = blockIdx.y;
    if (!ref.need[f]) return;
    const FrameDesc fd = frames[f];
    for (int64_t y = 1 + blockIdx.x; y < fd.qh; y += gridDim.x) {
        const uint32_t tr = ref.trow[fd.row0 + y];
        const uint32_t n = tr & 0x7fffffffu, na = ref.trow[fd.row0 + y - 1] & 0x7fffffffu;
        const int64_t rb = fd.node_off + y * fd.qw, ra = rb - fd.qw;
        __syncthreads();
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
            const uint64_t e = ref.tlist[rb + j];
            const int64_t a0 = e & 0xffff, a1 = e >> 16 & 0xffff;
            const uint8_t v = (uint8_t)(e >> 48);
            uint32_t lo = 0, hi = na;
            while (lo < hi) {  // the first run above whose end reaches a0 - 1
                const uint32_t mid = (lo + hi) >> 1;
                if ((int64_t)(ref.tlist[ra + mid] >> 16 & 0xffff) + 1 < a0)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            uint32_t first = 0xffffu, last = 0;
            for (uint32_t k = lo; k < na; k++) {
                const uint64_t b = ref.tlist[ra + k];
                if ((int64_t)(b & 0xffff) > a1 + 1) break;
                if ((uint8_t)(b >> 48) != v || !runs_touch(a0, a1, b & 0xffff, b >> 16 & 0xffff, v)) continue;
                if (first == 0xffffu) first = k;
                last = k;
                const uint32_t at = atomicAdd(&s_n, 1u);
                if (at < REF_LIST)
                    s_list[at] = ref_col(e) | ref_col(b) << 16;
                else
                    ref_insert(ref, (uint32_t)rb + ref_col(e), (uint32_t)ra + ref_col(b), (uint32_t)rb + ref_col(e));
            }
            ref.tch[rb + j] = first == 0xffffu ? 0xffffffffu : first | last << 16;
        }
        __syncthreads();
        const uint32_t np = min(s_n, (uint32_t)REF_LIST);
        for (uint32_t p = threadIdx.x; p < np; p += blockDim.x) {
            const uint32_t i = (uint32_t)rb + (s_list[p] & 0xffffu);
            ref_insert(ref, i, (uint32_t)ra + (s_list[p] >> 16), i);
        }
        if (threadIdx.x == 0 && (tr >> 31))
            ref_insert(ref, (uint32_t)rb + ref_col(ref.tlist[rb + n - 1]),
                       (uint32_t)(fd.node_off + (int64_t)fd.qw * fd.qh + y - 1), (uint32_t)(rb + fd.qw - 1));
    }
}

// The parent of u as the top of its set at the edge's time (every union
// done; parents only move up, so other threads may do the same meanwhile).
__device__ __forceinline__ uint64_t ref_true_parent(const RefOrder &ref, uint32_t u) {
    const uint64_t p = ref_par(ref, u);
    const uint32_t w = (uint32_t)(p >> 32);
    if (w == REF_INF) return p;
    return (uint64_t)w << 32 | ref_climb(ref, (uint32_t)p, w);
}

// A block per row: each run's true parent, its pixels added to every node
// above it but the top (whose sum is the target's pixel count), and to the
// target's gain in the row where its branch joins the top (hist). Lanes of
// a warp that add to one place add once.
__global__ void __launch_bounds__(REF_ROW_THREADS) k_ref_sums(const FrameDesc *frames, RefOrder ref) {
    kernel_begin();
    const int f = blockIdx.y;
    if (!ref.need[f]) return;
    const FrameDesc fd = frames[f];
    const uint32_t off = (uint32_t)fd.node_off, qw = (uint32_t)fd.qw;
    const int lane = threadIdx.x & 31;
    uint32_t *hist = ref.hist + fd.row0 * AT_REF_MAXT;
    for (int64_t y = blockIdx.x; y < fd.qh; y += gridDim.x) {
        const uint32_t tr = ref.trow[fd.row0 + y];
        const uint32_t n = tr & 0x7fffffffu, ne = n + (tr >> 31);  // the link's node is the row's last element
        const int64_t rb = fd.node_off + y * fd.qw;
        for (uint32_t j0 = 0; j0 < ne; j0 += blockDim.x) {
            const uint32_t j = j0 + threadIdx.x;
            const uint64_t e = j < ne ? ref.tlist[rb + (j < n ? j : n - 1)] : 0;
            const uint32_t t = (uint32_t)(e >> 56);
            uint32_t u = 0, px = 0;
            bool act = j < ne;
            uint64_t p = 0;
            if (act) {
                u = j < n ? (uint32_t)rb + ref_col(e) : (uint32_t)(fd.node_off + (int64_t)fd.qw * fd.qh + y - 1);
                px = j < n ? ref_len(e) : 1u;
                p = ref_true_parent(ref, u);
                *(volatile uint64_t *)(ref.par + u) = p;
                act = (uint32_t)(p >> 32) != REF_INF;
            }
            while (__any_sync(0xffffffffu, act)) {
                uint64_t q = 0;
                uint32_t *at = nullptr;
                if (act) {
                    q = ref_true_parent(ref, (uint32_t)p);
                    at = (uint32_t)(q >> 32) == REF_INF ? hist + (int64_t)t * fd.qh + ((uint32_t)(p >> 32) - off) / qw
                                                        : ref.sum + (uint32_t)p;
                }
                const uint32_t peers = __match_any_sync(0xffffffffu, (unsigned long long)(uintptr_t)at);
                const uint32_t add = __reduce_add_sync(peers, px);
                if (act) {
                    if (lane == __ffs(peers) - 1) atomicAdd(at, add);
                    act = (uint32_t)(q >> 32) != REF_INF;
                    p = q;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// The root of each target, a block per target: from the whole component
// back to the run that the reference's unions leave as its root (see the top
// of the file). (48 blocks a frame take them in turn.) x: the top of the current set; Z its pixels; ymax the last
// row that it holds whole; with `part`, also the events before node `lim` of
// the row after. gain[y]: the pixels x's set gained up to row y (x alone
// before its own row).
// Nearly all its time goes into the gains of a new top (two or three per
// target, each over the target runs of all rows of its set): 1024 threads,
// four loads each in flight (with 128 threads and one: 271 us for 32 frames
// of 1920 x 1080, 1380 us for 4032 x 3024 at full resolution).
#define REF_ROOT_THREADS 1024

__global__ void __launch_bounds__(REF_ROOT_THREADS) k_ref_root(const FrameDesc *frames, RefOrder ref, uint32_t *err) {
    kernel_begin();
    __shared__ uint32_t s_scan[32];
    __shared__ uint32_t s_ev, s_before, s_evj;
    __shared__ uint32_t s_win, s_winz;
    const int f = blockIdx.y;
    if (!ref.need[f]) return;
    const FrameDesc fd = frames[f];
    const int tid = threadIdx.x, lane = tid & 31;
    for (uint32_t t = blockIdx.x; t < ref.nt[f]; t += gridDim.x) {
        __syncthreads();
        const uint32_t off = (uint32_t)fd.node_off, qw = (uint32_t)fd.qw;
        const uint32_t vbase = off + (uint32_t)((int64_t)fd.qw * fd.qh);
        uint32_t *gain = ref.hist + fd.row0 * AT_REF_MAXT + (int64_t)t * fd.qh;
        uint32_t x = ref.tlabel[(int64_t)f * AT_REF_MAXT + t], root = 0xffffffffu;
        uint32_t Z = ref.tpx[(int64_t)f * AT_REF_MAXT + t];
        // the prefix sums of gain over rows [y0, y1]
        auto scan_gain = [&](int y0, int y1) {
            uint32_t base = 0;
            for (int r0 = y0; r0 <= y1; r0 += REF_ROOT_THREADS) {
                const int r = r0 + tid;
                const uint32_t v = r <= y1 ? gain[r] : 0u;
                uint32_t total;
                const uint32_t o = block_excl_scan(v, &total, s_scan);
                if (r <= y1) gain[r] = base + o + v;
                base += total;
            }
            __syncthreads();
        };
        if (x >= vbase) {  // a last-column pixel alone
            root = x;
        } else {
            int ymax = fd.qh - 1, y0 = (int)((x - off) / qw);
            bool part = false;
            uint32_t lim = REF_INF, gen = 0;
            uint32_t lx = ref.len[x];
            scan_gain(y0, ymax);
            for (int guard = 0; guard < (1 << 16); guard++) {
                // the first row (y0 - 1: x alone) that leaves more than Z / 2:
                // each warp narrows [lo, hi) by 32 probes at a time
                int lo = y0 - 1, hi = ymax + 1;
                while (lo < hi) {
                    const int step = (hi - lo + 31) / 32;
                    const int r = lo + lane * step;
                    const bool over = r >= hi || 2ull * (lx + (r < y0 ? 0u : gain[r])) > Z;
                    const uint32_t bal = __ballot_sync(0xffffffffu, over);
                    const int k = bal ? __ffs(bal) - 1 : 32;
                    const int nhi = k == 32 ? hi : min(hi, lo + k * step);
                    lo = k == 0 ? lo : lo + (k - 1) * step + 1;
                    hi = nhi;
                }
                if (lo == y0 - 1) {
                    root = x;
                    break;
                }
                if (lo <= ymax && (lo < ymax || part)) {
                    Z = lx + gain[lo];
                    ymax = lo;
                    part = false;
                    continue;
                }
                // row r, event by event: those before lim that end in x's set
                const int r = part ? ymax + 1 : ymax;
                const uint32_t L = part ? lim : REF_INF;
                const uint32_t rb = off + (uint32_t)r * qw, ra = rb - qw;
                const uint32_t tr = ref.trow[fd.row0 + r], n = tr & 0x7fffffffu;
                uint32_t base = lx + (r - 1 < y0 ? 0u : gain[r - 1]);
                __syncthreads();
                if (tid == 0) s_ev = s_evj = REF_INF;
                __syncthreads();
                gen++;
                for (uint32_t j0 = 0; j0 < n; j0 += REF_ROOT_THREADS) {
                    const uint32_t j = j0 + tid;
                    uint32_t d = 0, i = 0;
                    if (j < n) {
                        const uint64_t e = ref.tlist[rb + j];
                        i = rb + ref_col(e);
                        if (i < L && (uint32_t)(e >> 56) == t && ref.par[i] == ((uint64_t)i << 32 | x)) {
                            d = ref_len(e);
                            const uint32_t tc = ref.tch[rb + j];
                            if (tc != 0xffffffffu)
                                for (uint32_t k = tc & 0xffffu; k <= tc >> 16; k++) {
                                    const uint64_t b = ref.tlist[ra + k];
                                    if ((b ^ e) >> 48 & 0xff) continue;
                                    const uint32_t c = ref_climb(ref, ra + ref_col(b), i - 1);
                                    // each set once (only this thread meets it)
                                    if (c == x || ref.stamp[c] == gen) continue;
                                    ref.stamp[c] = gen;
                                    d += ref.sum[c];
                                }
                        }
                    }
                    uint32_t total;
                    const uint32_t o = block_excl_scan(d, &total, s_scan);
                    if (d && 2ull * (base + o) <= Z && 2ull * (base + o + d) > Z) {  // one thread at most
                        s_ev = i;
                        s_evj = j;
                        s_before = base + o;
                    }
                    __syncthreads();
                    if (s_ev != REF_INF) break;
                    base += total;
                }
                if (s_ev == REF_INF) {
                    // the row's last-column link: one pixel, which takes the
                    // root only from a set of one pixel
                    const uint32_t wl = rb + qw - 1, vn = vbase + (uint32_t)r - 1;
                    if (!(tr >> 31) || wl >= L || ref.par[vn] != ((uint64_t)wl << 32 | x) || 2ull * (base + 1) <= Z) break;
                    if (base <= 1) {
                        root = vn;
                        break;
                    }
                    Z = base;
                    ymax = r - 1;
                    part = true;
                    lim = wl;
                    continue;
                }
                // the calls of that event, by warp 0: run i's set against each
                // set it meets, in order; the larger keeps its root, run i's
                // side only with strictly more
                const uint32_t i = s_ev, before = s_before;
                gen++;
                if (tid < 32) {
                    const uint64_t e = ref.tlist[rb + s_evj];
                    const uint32_t tc = ref.tch[rb + s_evj];
                    uint32_t win = i, winz = ref_len(e), z = winz;
                    if (tc != 0xffffffffu)
                        for (uint32_t k0 = tc & 0xffffu; k0 <= tc >> 16; k0 += 32) {
                            const uint32_t k = k0 + lane;
                            uint32_t c = REF_INF, zc = 0;
                            if (k <= tc >> 16) {
                                const uint64_t b = ref.tlist[ra + k];
                                if (!((b ^ e) >> 48 & 0xff)) {
                                    c = ref_climb(ref, ra + ref_col(b), i - 1);
                                    zc = c == x ? before : ref.sum[c];
                                    if (*(volatile uint32_t *)(ref.stamp + c) == gen) c = REF_INF;  // met already
                                }
                            }
                            const uint32_t peers = __match_any_sync(0xffffffffu, c);
                            const bool first = c != REF_INF && lane == __ffs(peers) - 1;
                            if (first) *(volatile uint32_t *)(ref.stamp + c) = gen;
                            uint32_t bal = __ballot_sync(0xffffffffu, first);
                            __syncwarp();
                            while (bal) {
                                const int l = __ffs(bal) - 1;
                                bal &= bal - 1;
                                const uint32_t cl = __shfl_sync(0xffffffffu, c, l), zl = __shfl_sync(0xffffffffu, zc, l);
                                if (z <= zl) {
                                    win = cl;
                                    winz = zl;
                                }
                                z += zl;
                            }
                        }
                    if (lane == 0) {
                        s_win = win;
                        s_winz = winz;
                    }
                }
                __syncthreads();
                const uint32_t win = s_win;
                if (win == i) {
                    root = i;
                    break;
                }
                Z = s_winz;
                ymax = r - 1;
                part = true;
                lim = i;
                if (win == x) continue;
                // another set's root wins: what its top gained per row (its
                // branches start in its own row at the earliest, and join by row r)
                x = win;
                y0 = (int)((x - off) / qw);
                lx = ref.len[x];
                for (int y = y0 + tid; y <= r; y += REF_ROOT_THREADS) gain[y] = 0;
                __syncthreads();
                for (int y = y0 + (tid >> 5); y <= r; y += REF_ROOT_THREADS / 32) {
                    const uint32_t try_ = ref.trow[fd.row0 + y], ny = try_ & 0x7fffffffu;
                    const uint32_t rby = off + (uint32_t)y * qw;
                    for (uint32_t j0 = lane; j0 < ny; j0 += 128) {
                        uint32_t u[4];
                        uint64_t p[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const uint32_t j = j0 + 32 * q;
                            const uint64_t e = j < ny ? ref.tlist[rby + j] : ~0ull;
                            u[q] = (uint32_t)(e >> 56) == t ? rby + ref_col(e) : x;
                        }
#pragma unroll
                        for (int q = 0; q < 4; q++) p[q] = u[q] != x ? ref.par[u[q]] : 0ull;
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (u[q] != x && (uint32_t)p[q] == x)
                                atomicAdd(gain + ((uint32_t)(p[q] >> 32) - off) / qw, ref.sum[u[q]]);
                    }
                    if (lane == 0 && (try_ >> 31)) {  // the link's last-column node
                        const uint64_t p = ref.par[vbase + (uint32_t)y - 1];
                        if ((uint32_t)p == x) atomicAdd(gain + ((uint32_t)(p >> 32) - off) / qw, 1u);
                    }
                }
                __syncthreads();
                scan_gain(y0, r);
            }
        }
        // GPU node ids -> the reference's packed node numbers
        if (tid == 0) {
            if (root == 0xffffffffu) {
                atomicOr(err, AT_ERR_ORDER);
            } else {
                const uint32_t *pre = ref.rpre + fd.row0 + f;
                root = root < vbase ? pre[(root - off) / qw] + (root - off) % qw : pre[fd.qh] + (root - vbase);
            }
            ref.troot[(int64_t)f * AT_REF_MAXT + t] = root;
        }
    }
}

// ---------------------------------------------------------------------------
// Launchers.

int launch_ref_order(const Launch &L, const FrameDesc *frames, const RowWord *words, RunArrays runs,
                     const uint32_t *row_nruns, int nfam, const int64_t *qstart, const GpuDetection *dets,
                     const uint32_t *det_ok, const uint32_t *qcl, const uint64_t *ckey, int nb, const RefOrder &ref,
                     uint32_t *err) {
    launch(k_ref_targets, L.nframes, 256, 0, L.stream, frames, nfam, qstart, dets, det_ok, qcl, ckey, nb, runs, row_nruns,
                                                   ref, err);
    const int64_t b = (L.max_qh + 7) / 8;
    const dim3 grid((unsigned)(b < 1 ? 1 : b < 148 * 4 ? b : 148 * 4), (unsigned)L.nframes);
    launch(k_ref_mark, grid, 256, 8 * (REF_ROW_RUNS + 8 * REF_STAGE), L.stream, frames, words, runs, row_nruns, ref);
    const dim3 rows((unsigned)(L.max_qh < 148 * 16 ? L.max_qh : 148 * 16), (unsigned)L.nframes);
    launch(k_ref_link, rows, REF_ROW_THREADS, 0, L.stream, frames, ref);
    launch(k_ref_sums, rows, REF_ROW_THREADS, 0, L.stream, frames, ref);
    launch(k_ref_root, dim3(48, (unsigned)L.nframes), REF_ROOT_THREADS, 0, L.stream, frames, ref, err);
    return 5;
}

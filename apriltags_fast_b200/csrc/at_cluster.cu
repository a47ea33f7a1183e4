// Clusters of boundary points without sorting the points
// (fast/clusters.c:16-66, 123-252, 318-382).
//
// The reference groups the boundary points by the pair of components they
// lie between, each cluster's points in emission order (y, x, neighbour),
// and orders the clusters. Here each point is made once, from the row
// masks and the run labels, as a 4-byte record in its row's region; the
// records are then placed, each at its place in its cluster:
//
//   k_point_scan     a warp per row: its points, found as bits of 32 columns
//                    a lane, then looked up a point a lane; their label pairs
//                    gathered in the warp's table (shared memory), the
//                    records in emission order; at the
//                    row's end each pair of the row into the frame's pair
//                    table (point count, first and last row) and the row's
//                    pair list.
//   k_cluster_collect (at_kernels.cu): the distinct pairs.
//   -- the host reads the pair and point counts (its only wait here) --
//   k_pair_frame, k_pair_offsets, k_pair_scatter, k_pair_rank: the distinct
//                    pairs in order. A frame's pairs sort before the next
//                    frame's (the larger label is a node of the frame).
//   k_cluster_span   per cluster: count, frame, first row, rows spanned.
//   scans            each cluster's first point; its row table's offset.
//   (all from k_pair_frame to here in k_pair_small when there are few pairs)
//   k_seg_fill       a warp per row: its pairs' point counts into the
//                    clusters' row tables.
//   k_seg_scan       a warp per cluster: the counts of its rows become the
//                    places of each row's first point of the cluster.
//   k_point_place    a warp per row: every record to its place; records of
//                    a row are in emission order, so a cluster's points
//                    keep the reference's order.
#include <cuda_runtime.h>
#include <stdint.h>

#include "at_device.cuh"
#include "at_gpu.h"
#include "at_kernels.h"
#include "at_launch.h"

// Rows 1 .. qh-2 of each frame, a warp per row.
#define ROW_WARPS_BEGIN                                                                              \
    const FrameDesc f = frames[blockIdx.y];                                                          \
    const int lane = threadIdx.x & 31;                                                               \
    const int64_t wpb = blockDim.x >> 5;                                                             \
    for (int64_t y = 1 + blockIdx.x * wpb + (threadIdx.x >> 5); y + 1 < f.qh; y += gridDim.x * wpb) {
#define ROW_WARPS_END }

// What a warp of the scan keeps: its row's pairs, open addressing over 2
// nd_cap slots (larger label << 32 | smaller, points); (starts, before) of
// the 32 words it is at in this row and the next, with those beside; up to
// SCAN_BUF of their points in emission order (column | neighbour << 10 |
// black << 12); the pairs' count; behind it their slots.
#define SCAN_BUF 1024
struct ScanPart {
    uint2 at[2][34];
    uint16_t pts[SCAN_BUF];
    uint32_t npair, pad[3];
};
__host__ __device__ inline size_t row_pairs_bytes(int nd_cap) { return (size_t)26 * nd_cap + sizeof(ScanPart); }

// Point records: the pair's slot in the row's table | neighbour j << 12 |
// (pixel is 0) << 14 | x << 15.
#define PREC_ID 0xfffu

// The run of column c of a word with (starts, before) s.
__device__ __forceinline__ uint32_t run_in(uint2 s, int c) { return s.y + __popc(s.x & ((2u << (c & 31)) - 1u)) - 1u; }

// Every boundary point, once. The points of 32 columns are bit operations
// on the masks of the row and the row below (the masks hold labelled pixels
// only; fast/clusters.c:144-252, as point_mask per pixel), a word a lane.
// Each lane lists its word's points in emission order (x, then neighbour);
// then a lane takes a point: the labels by run number, the pair looked up in
// the row's table by the first of a run of equal ones, the record written. At
// the row's end each pair goes into the frame's pair table (count, first and
// last row) and, with its points in the row, into the row's pair list. Any
// capacity exceeded (pairs of a row, records of a row, probes of the pair
// table) sets *full and the batch takes the sorting path instead.
//
// Bound by instruction issue. For 32 frames of 1920 x 1080 (9.4 million
// points): a lane per pixel with labels per pixel 313 us; a lane looking up
// all its word's points, where the fullest of 32 words sets the pace, 180 us
// (10 of 32 lanes busy, 13 instructions a warp and point); 8 columns a lane
// from a queue 208 us; this 105 us (228 to 140 for 16 of mixed sizes,
// 346 to 194 for one 4032 x 3024).
__global__ void __launch_bounds__(256) k_point_scan(const FrameDesc *frames, const RowWord *words, const uint32_t *lab,
                                                    int nb, PairTable T, PointRows P, uint32_t *full,
                                                    unsigned long long *npoints) {
    kernel_begin();
    extern __shared__ __align__(16) uint8_t s_mem[];
    const int nd_cap = P.nd_cap, rt = 2 * nd_cap;
    uint64_t *tkey = reinterpret_cast<uint64_t *>(s_mem + (threadIdx.x >> 5) * row_pairs_bytes(nd_cap));
    uint32_t *tcnt = reinterpret_cast<uint32_t *>(tkey + rt);
    ScanPart &W = *reinterpret_cast<ScanPart *>(tcnt + rt);
    uint16_t *used = reinterpret_cast<uint16_t *>(&W + 1);
    for (int i = threadIdx.x & 31; i < rt; i += 32) {
        tkey[i] = CH_EMPTY;
        tcnt[i] = 0;
    }
    if ((threadIdx.x & 31) == 0) W.npair = 0;
    __syncwarp();
    const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u;
    uint64_t pts = 0;
    ROW_WARPS_BEGIN
    const int qw = f.qw, nw = (qw + 31) / 32;
    const RowWord *wa = words + f.word_off + y * nw, *wb = wa + nw;
    const uint32_t *la_of = lab + f.node_off + y * qw, *lb_of = la_of + qw;
    const uint32_t *lcol = lab + f.node_off + (int64_t)qw * f.qh + y;  // last column: this row, the next
    uint32_t *rec = P.rec + 2 * (f.q_off + y * qw);
    const uint32_t rcap = (uint32_t)(2 * qw);
    uint32_t nrec = 0;
    for (int i0 = 0; i0 < nw; i0 += 32) {
        const int i = i0 + lane;
        // the lane's word of both rows and the words beside it
        RowWord a = {0, 0, 0, 0}, b = a, an = a, bn = a, bp = a;
        uint32_t pWa = 0, pKa = 0;
        if (i < nw) {
            a = wa[i];
            b = wb[i];
            if (i + 1 < nw) {
                an = wa[i + 1];
                bn = wb[i + 1];
            }
            if (i > 0) {
                bp = wb[i - 1];
                pWa = wa[i - 1].white >> 31;
                pKa = wa[i - 1].black >> 31;
            }
        }
        const uint32_t Wa1 = a.white >> 1 | an.white << 31, Ka1 = a.black >> 1 | an.black << 31;
        const uint32_t Wb1 = b.white >> 1 | bn.white << 31, Kb1 = b.black >> 1 | bn.black << 31;
        const uint32_t Wbm = b.white << 1 | bp.white >> 31, Kbm = b.black << 1 | bp.black >> 31;
        const uint32_t Wam = a.white << 1 | pWa, Kam = a.black << 1 | pKa;
        const uint32_t xm = i < nw ? run_columns(i, qw) : 0u, x1 = i == 0 ? xm & ~1u : xm;  // column 0: only (1, 0)
        const uint32_t left11 = ((Wam & b.black) | (Kam & b.white)) & (i == 0 ? ~3u : ~0u);
        const uint32_t c10 = ((a.white & Ka1) | (a.black & Wa1)) & xm;
        const uint32_t c01 = ((a.white & b.black) | (a.black & b.white)) & x1;
        const uint32_t cm1 = ((a.white & Kbm) | (a.black & Wbm)) & x1 & ~left11;
        const uint32_t c11 = ((a.white & Kb1) | (a.black & Wb1)) & x1;
        uint32_t total;
        const uint32_t own = __popc(c10) + __popc(c01) + __popc(cm1) + __popc(c11);
        const uint32_t off = warp_excl_scan(own, &total), end = off + own;
        if (total == 0) continue;
        if (nrec + total > rcap) {
            if (lane == 0) atomicOr(full, 1u);
            return;
        }
        W.at[0][lane + 1] = make_uint2(a.starts, a.before);
        W.at[1][lane + 1] = make_uint2(b.starts, b.before);
        if (lane == 0) W.at[1][0] = make_uint2(bp.starts, bp.before);
        if (lane == 31) {
            W.at[0][33] = make_uint2(an.starts, an.before);
            W.at[1][33] = make_uint2(bn.starts, bn.before);
        }
        for (uint32_t base = 0, lim; base < total; base = lim) {
            // the words whose points there is room for (a word has 128 at most)
            const bool fits = end <= base + SCAN_BUF;
            lim = __reduce_max_sync(0xffffffffu, fits ? end : 0u);
            const uint32_t n = lim - base;
            if (fits && off >= base) {
                uint16_t *to = W.pts + (off - base);
                for (uint32_t any = c10 | c01 | cm1 | c11; any; any &= any - 1) {
                    const int c = __ffs(any) - 1;
                    const uint32_t px = (uint32_t)(32 * lane + c) | (a.black >> c & 1u) << 12;
                    if (c10 >> c & 1u) *to++ = (uint16_t)px;
                    if (c01 >> c & 1u) *to++ = (uint16_t)(px | 1u << 10);
                    if (cm1 >> c & 1u) *to++ = (uint16_t)(px | 2u << 10);
                    if (c11 >> c & 1u) *to++ = (uint16_t)(px | 3u << 10);
                }
            }
            __syncwarp();
            for (uint32_t t0 = 0; t0 < n; t0 += 32) {
                const bool on = t0 + lane < n;
                uint32_t pt = 0, la = 0, lb = 0;
                if (on) {
                    pt = W.pts[t0 + lane];
                    const int xl = pt & 1023u, j = pt >> 10 & 3u;
                    la = la_of[run_in(W.at[0][(xl >> 5) + 1], xl)];
                    // the neighbour's label: this row or the next, a column on, none, or back
                    const int d = j == 0 || j == 3 ? 1 : j == 2 ? -1 : 0, row = j == 0 ? 0 : 1, cl = xl + d;
                    const uint32_t *lp = (row ? lb_of : la_of) + run_in(W.at[row][(cl >> 5) + 1], cl);
                    if (d > 0 && 32 * i0 + cl == qw - 1) lp = lcol + row;
                    lb = *lp;
                }
                // the first of each run of points of one pair finds it
                const uint32_t ua = __shfl_up_sync(0xffffffffu, la, 1), ub = __shfl_up_sync(0xffffffffu, lb, 1);
                const bool head = on && (lane == 0 || ua != la || ub != lb);
                const uint32_t heads = __ballot_sync(0xffffffffu, head), ons = __ballot_sync(0xffffffffu, on);
                uint32_t id = 0;
                if (head) {
                    const uint32_t later = heads & ~lt & ~(1u << lane);
                    const uint32_t hi = la > lb ? la : lb, lo = la > lb ? lb : la;
                    const uint64_t k = (uint64_t)hi << 32 | lo;
                    id = hi * 0x9e3779b1u + lo * 0x85ebca6bu;
                    id = (id ^ id >> 16) & (uint32_t)(rt - 1);
                    for (int p = 0; p < rt; p++) {  // a table without room has set *full below
                        uint64_t cur = *(volatile uint64_t *)(tkey + id);
                        if (cur == CH_EMPTY) {
                            cur = atomicCAS(reinterpret_cast<unsigned long long *>(tkey + id), CH_EMPTY, k);
                            if (cur == CH_EMPTY) {
                                const uint32_t at = atomicAdd(&W.npair, 1u);
                                if (at >= (uint32_t)nd_cap)
                                    atomicOr(full, 1u);
                                else
                                    used[at] = (uint16_t)id;
                                break;
                            }
                        }
                        if (cur == k) break;
                        id = (id + 1) & (uint32_t)(rt - 1);
                    }
                    atomicAdd(tcnt + id, (uint32_t)((later ? __ffs(later) - 1 : __popc(ons)) - lane));
                }
                const uint32_t mine = heads & (lt | 1u << lane);
                id = __shfl_sync(0xffffffffu, id, mine ? 31 - __clz(mine) : 0);
                if (on) rec[nrec + base + t0 + lane] = id | (pt & 0x1c00u) << 2 | ((uint32_t)(32 * i0) + (pt & 1023u)) << 15;
            }
            __syncwarp();
        }
        if (*(volatile uint32_t *)&W.npair > (uint32_t)nd_cap) return;  // *full is set
        __syncwarp();
        nrec += total;
    }
    // the row's pairs into the frame's pair table; the table cleared
    uint32_t *ps = P.pslot + (f.row0 + y) * nd_cap, *pc = P.pcnt + (f.row0 + y) * nd_cap;
    uint16_t *pi = P.pid + (f.row0 + y) * nd_cap;
    const uint32_t nd = W.npair;
    for (uint32_t at = lane; at < nd; at += 32) {
        const uint32_t id = used[at], n = tcnt[id];
        const uint64_t kk = tkey[id], k = (kk >> 32) << nb | (kk & 0xffffffffu);
        uint32_t slot = ch_hash(k) & T.mask;
        int p = 0;
        for (; p < CH_PROBES; p++) {
            uint64_t cur = *(volatile uint64_t *)(T.keys + slot);
            if (cur == CH_EMPTY) {
                const unsigned long long old =
                    atomicCAS(reinterpret_cast<unsigned long long *>(T.keys + slot), CH_EMPTY, k);
                cur = old == CH_EMPTY ? k : old;
            }
            if (cur == k) break;
            slot = (slot + 1) & T.mask;
        }
        if (p == CH_PROBES) {
            atomicOr(full, 1u);
        } else {
            atomicAdd(T.count + slot, n);
            atomicMin(T.ymin + slot, (uint32_t)y);
            atomicMax(T.ymax + slot, (uint32_t)y);
        }
        ps[at] = slot;
        pc[at] = n;
        pi[at] = (uint16_t)id;
        tkey[id] = CH_EMPTY;
        tcnt[id] = 0;
    }
    __syncwarp();
    if (lane == 0) {
        P.info[f.row0 + y] = make_uint2(nrec, nd);
        W.npair = 0;
    }
    pts += nrec;
    __syncwarp();
    ROW_WARPS_END
    if ((threadIdx.x & 31) == 0 && pts) atomicAdd(npoints, (unsigned long long)pts);
}

__device__ __forceinline__ int frame_of_node(const FrameDesc *frames, int nframes, int64_t node) {
    int lo = 0, hi = nframes - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (frames[mid].node_off <= node)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// The pairs in order: first in buckets, PAIR_BUCKETS per frame by where the
// larger label lies among the frame's nodes (a monotone function of the
// pair), then ranked among their bucket's. (Ranked among all pairs of the
// frame: 210 us for the 24396 pairs of a 4032 x 3024 frame.)
#define PAIR_BUCKETS 256
__global__ void k_pair_frame(const uint64_t *okeys, int64_t ncl, int nb, const FrameDesc *frames, int nframes,
                             uint32_t *kbucket, uint32_t *bcount) {
    kernel_begin();
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < ncl; r += (int64_t)gridDim.x * blockDim.x) {
        const int64_t hi = (int64_t)(okeys[r] >> nb);
        const int fr = frame_of_node(frames, nframes, hi);
        const FrameDesc &f = frames[fr];
        const uint64_t nodes = (uint64_t)f.qw * f.qh + f.qh;
        const uint32_t b = (uint32_t)fr * PAIR_BUCKETS + (uint32_t)((uint64_t)(hi - f.node_off) * PAIR_BUCKETS / nodes);
        kbucket[r] = b;
        atomicAdd(bcount + b, 1u);
    }
}

// One block: each bucket's first pair (boff, nbuckets + 1 entries).
__global__ void __launch_bounds__(1024) k_pair_offsets(const uint32_t *bcount, int nbuckets, uint32_t *boff,
                                                       uint32_t *bcur) {
    kernel_begin();
    __shared__ uint32_t sh[32];
    uint32_t base = 0;
    for (int b0 = 0; b0 < nbuckets; b0 += 4 * blockDim.x) {
        const int b = b0 + 4 * threadIdx.x;  // nbuckets is a multiple of 4
        const uint4 c = b < nbuckets ? *reinterpret_cast<const uint4 *>(bcount + b) : make_uint4(0, 0, 0, 0);
        uint32_t total;
        const uint32_t o = base + block_excl_scan(c.x + c.y + c.z + c.w, &total, sh);
        if (b < nbuckets) {
            *reinterpret_cast<uint4 *>(boff + b) = make_uint4(o, o + c.x, o + c.x + c.y, o + c.x + c.y + c.z);
            *reinterpret_cast<uint4 *>(bcur + b) = make_uint4(0, 0, 0, 0);
        }
        base += total;
    }
    if (threadIdx.x == 0) boff[nbuckets] = base;
}

__global__ void k_pair_scatter(const uint64_t *okeys, const uint32_t *oslots, int64_t ncl, const uint32_t *kbucket,
                               const uint32_t *boff, uint32_t *bcur, uint64_t *gkeys, uint32_t *gslots,
                               uint32_t *gbucket) {
    kernel_begin();
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < ncl; r += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t b = kbucket[r];
        const uint32_t p = boff[b] + atomicAdd(bcur + b, 1u);
        gkeys[p] = okeys[r];
        gslots[p] = oslots[r];
        gbucket[p] = b;
    }
}

// A warp per pair: its place = its bucket's first place + the number of
// smaller pairs of the bucket (the pairs are distinct).
__global__ void __launch_bounds__(256) k_pair_rank(const uint64_t *gkeys, const uint32_t *gslots,
                                                   const uint32_t *gbucket, int64_t ncl, const uint32_t *boff,
                                                   uint64_t *skeys, uint32_t *sslots) {
    kernel_begin();
    const int lane = threadIdx.x & 31;
    for (int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < ncl;
         p += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const uint32_t b = gbucket[p], q0 = boff[b], q1 = boff[b + 1];
        const uint64_t k = gkeys[p];
        uint32_t below = 0;
        for (uint32_t q = q0 + lane; q < q1; q += 32) below += gkeys[q] < k;
        below = __reduce_add_sync(0xffffffffu, below);
        if (lane == 0) {
            skeys[q0 + below] = k;
            sslots[q0 + below] = gslots[p];
        }
    }
}

// Cluster c (in pair order): its slot's rank; its point count, frame,
// first row and rows spanned.
__global__ void k_cluster_span(const uint64_t *skeys, const uint32_t *sslots, int64_t ncl, PairTable T, int nb,
                               const FrameDesc *frames, int nframes, uint32_t *rank_of_slot, uint32_t *ccount,
                               uint32_t *cspan, uint32_t *cy0, int32_t *cframe) {
    kernel_begin();
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncl; c += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t s = sslots[c];
        rank_of_slot[s] = (uint32_t)c;
        ccount[c] = T.count[s];
        cy0[c] = T.ymin[s];
        cspan[c] = T.ymax[s] - T.ymin[s] + 1;
        cframe[c] = frame_of_node(frames, nframes, (int64_t)(skeys[c] >> nb));
    }
}

// All of the above and below up to the row tables for at most PAIR_SMALL
// pairs, in one block: the pairs sorted in shared memory (bitonic, the
// distances up to 32 within a warp), then the clusters' fields, both prefix
// sums and the zeroed row tables. Bound by its barriers. Nine kernels of 3-5
// us each, one after the other, take the 132 pairs of a 640 x 480 frame to a
// clusters stage of 99 us, this one (11 us) to 76; 820 pairs (1920 x 1080) 118
// and 108 (18 us); with a limit of 4096, the 3500 pairs of eight 1280 x 720
// frames 125 and 158.
#define PAIR_SMALL 1024
__global__ void __launch_bounds__(1024) k_pair_small(const uint64_t *okeys, const uint32_t *oslots, int ncl, PairTable T,
                                                     int nb, const FrameDesc *frames, int nframes, uint64_t *skeys,
                                                     uint32_t *rank_of_slot, uint32_t *cspan, uint32_t *cy0,
                                                     int32_t *cframe, uint32_t *cstart, uint32_t *spanoff, uint32_t *seg,
                                                     int64_t cap, uint32_t *err) {
    kernel_begin();
    __shared__ uint64_t s_key[PAIR_SMALL];
    __shared__ uint16_t s_idx[PAIR_SMALL];
    __shared__ uint32_t sh[32];
    const int tid = threadIdx.x;
    int np = 64;
    while (np < ncl) np <<= 1;
    if (tid < np) {
        s_key[tid] = tid < ncl ? okeys[tid] : ~0ull;
        s_idx[tid] = (uint16_t)tid;
    }
    __syncthreads();
    for (int kk = 2; kk <= np; kk <<= 1)
        for (int j = kk >> 1; j > 0; j >>= 1) {
            if (tid < np / 2) {
                const int i = ((tid & ~(j - 1)) << 1) | (tid & (j - 1)), l = i + j;
                const uint64_t a = s_key[i], b = s_key[l];
                if ((a > b) == ((i & kk) == 0)) {
                    const uint16_t t = s_idx[i];
                    s_key[i] = b;
                    s_key[l] = a;
                    s_idx[i] = s_idx[l];
                    s_idx[l] = t;
                }
            }
            // distances up to 32 stay within the 64 keys of a warp
            if (j > 32 || (j == 1 && kk >= 64))
                __syncthreads();
            else
                __syncwarp();
        }
    uint32_t n = 0, span = 0;
    if (tid < ncl) {
        const uint64_t key = s_key[tid];
        const uint32_t s = oslots[s_idx[tid]], y0 = T.ymin[s];
        n = T.count[s];
        span = T.ymax[s] - y0 + 1;
        skeys[tid] = key;
        rank_of_slot[s] = (uint32_t)tid;
        cspan[tid] = span;
        cy0[tid] = y0;
        cframe[tid] = frame_of_node(frames, nframes, (int64_t)(key >> nb));
    }
    uint32_t points, rows;
    const uint32_t oa = block_excl_scan(n, &points, sh), ob = block_excl_scan(span, &rows, sh);
    if (tid < ncl) {
        cstart[tid] = oa;
        spanoff[tid] = ob;
    }
    if (tid == 0) {
        cstart[ncl] = points;
        spanoff[ncl] = rows;
    }
    if (rows > cap) {
        if (tid == 0) atomicOr(err, AT_ERR_SEGCAP);
        return;
    }
    for (uint32_t i = tid; i < rows; i += 1024) seg[i] = 0;
}

// Exclusive scans of two arrays of n values at once (a pass per block of
// SCAN_ITEMS, one block over the block sums, a pass that adds them):
// out_a, out_b get n + 1 entries (the totals last).
#define SCAN_THREADS 256
#define SCAN_ITEMS (4 * SCAN_THREADS)

__global__ void __launch_bounds__(SCAN_THREADS) k_scan2_sums(const uint32_t *a, const uint32_t *b, int64_t n,
                                                             uint32_t *sa, uint32_t *sb) {
    kernel_begin();
    __shared__ uint32_t sh[32];
    const int64_t i0 = (int64_t)blockIdx.x * SCAN_ITEMS + 4 * threadIdx.x;
    uint32_t va = 0, vb = 0;
    for (int k = 0; k < 4; k++)
        if (i0 + k < n) {
            va += a[i0 + k];
            vb += b[i0 + k];
        }
    uint32_t ta, tb;
    block_excl_scan(va, &ta, sh);
    block_excl_scan(vb, &tb, sh);
    if (threadIdx.x == 0) {
        sa[blockIdx.x] = ta;
        sb[blockIdx.x] = tb;
    }
}

__global__ void __launch_bounds__(1024) k_scan2_top(uint32_t *sa, uint32_t *sb, int64_t nblocks) {
    kernel_begin();
    __shared__ uint32_t sh[32];
    uint32_t ba = 0, bb = 0;
    for (int64_t i0 = 0; i0 < nblocks; i0 += blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        const uint32_t va = i < nblocks ? sa[i] : 0u, vb = i < nblocks ? sb[i] : 0u;
        uint32_t ta, tb;
        const uint32_t oa = block_excl_scan(va, &ta, sh), ob = block_excl_scan(vb, &tb, sh);
        if (i < nblocks) {
            sa[i] = ba + oa;
            sb[i] = bb + ob;
        }
        ba += ta;
        bb += tb;
    }
    if (threadIdx.x == 0) {
        sa[nblocks] = ba;
        sb[nblocks] = bb;
    }
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan2_apply(const uint32_t *a, const uint32_t *b, int64_t n,
                                                              const uint32_t *sa, const uint32_t *sb,
                                                              int64_t nblocks, uint32_t *out_a, uint32_t *out_b) {
    kernel_begin();
    __shared__ uint32_t sh[32];
    const int64_t i0 = (int64_t)blockIdx.x * SCAN_ITEMS + 4 * threadIdx.x;
    uint32_t xa[4], xb[4], va = 0, vb = 0;
    for (int k = 0; k < 4; k++) {
        xa[k] = i0 + k < n ? a[i0 + k] : 0u;
        xb[k] = i0 + k < n ? b[i0 + k] : 0u;
        va += xa[k];
        vb += xb[k];
    }
    uint32_t ta, tb;
    uint32_t oa = block_excl_scan(va, &ta, sh) + sa[blockIdx.x], ob = block_excl_scan(vb, &tb, sh) + sb[blockIdx.x];
    for (int k = 0; k < 4; k++)
        if (i0 + k < n) {
            out_a[i0 + k] = oa;
            out_b[i0 + k] = ob;
            oa += xa[k];
            ob += xb[k];
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        out_a[n] = sa[nblocks];
        out_b[n] = sb[nblocks];
    }
}

// The row tables: zeroed up to their total (checked against the capacity:
// a shortfall sets AT_ERR_SEGCAP and the host runs the batch again with
// room enough; the point kernels then skip their work).
__global__ void k_seg_zero(const uint32_t *spanoff, int64_t ncl, uint32_t *seg, int64_t cap, uint32_t *err) {
    kernel_begin();
    const int64_t total = spanoff[ncl];
    if (total > cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, AT_ERR_SEGCAP);
        return;
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
        seg[i] = 0;
}

// A warp per cluster: seg[spanoff[c] + r] = the place of the cluster's
// first point in row cy0[c] + r.
__global__ void __launch_bounds__(256) k_seg_scan(const uint32_t *cstart, const uint32_t *spanoff,
                                                  const uint32_t *cspan, int64_t ncl, uint32_t *seg, int64_t cap) {
    kernel_begin();
    if (spanoff[ncl] > cap) return;
    const int lane = threadIdx.x & 31;
    for (int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < ncl;
         c += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        uint32_t *row = seg + spanoff[c];
        const uint32_t n = cspan[c];
        uint32_t carry = cstart[c];
        for (uint32_t i0 = 0; i0 < n; i0 += 32) {
            const uint32_t i = i0 + lane;
            const uint32_t v = i < n ? row[i] : 0u;
            uint32_t total;
            const uint32_t o = warp_excl_scan(v, &total);
            if (i < n) row[i] = carry + o;
            carry += total;
        }
    }
}

// Each row's pairs: their point counts into the row tables
// (seg[spanoff[c] + y - cy0[c]] for the pair's cluster c).
__global__ void __launch_bounds__(256) k_seg_fill(const FrameDesc *frames, PointRows P, const uint32_t *rank_of_slot,
                                                  const uint32_t *spanoff, const uint32_t *cy0, int64_t ncl,
                                                  uint32_t *seg, int64_t cap) {
    kernel_begin();
    if (spanoff[ncl] > cap) return;
    ROW_WARPS_BEGIN
    const uint32_t nd = P.info[f.row0 + y].y;
    const uint32_t *ps = P.pslot + (f.row0 + y) * P.nd_cap, *pc = P.pcnt + (f.row0 + y) * P.nd_cap;
    for (uint32_t i = lane; i < nd; i += 32) {
        const uint32_t c = rank_of_slot[ps[i]];
        seg[spanoff[c] + ((uint32_t)y - cy0[c])] = pc[i];
    }
    ROW_WARPS_END
}

// A warp per row: each record to its place, the row's first place of each
// pair's cluster (seg, after the scan) plus the pair's points before it in
// the row; the records are in emission order, so a cluster's points keep
// the reference's order.
//
// Bound by memory latency: the records of the next two steps are on their way
// during one (32 frames of 1920 x 1080: 72 -> 51 us).
__global__ void __launch_bounds__(256) k_point_place(const FrameDesc *frames, PointRows P,
                                                     const uint32_t *rank_of_slot, const uint32_t *spanoff,
                                                     const uint32_t *cy0, int64_t ncl, const uint32_t *seg, int64_t cap,
                                                     uint64_t *out, int64_t npts, uint32_t *err) {
    kernel_begin();
    extern __shared__ __align__(16) uint32_t s_base[];
    if (spanoff[ncl] > cap) return;
    uint32_t *base = s_base + (threadIdx.x >> 5) * 2 * P.nd_cap;  // by the pair's slot in the row's table
    const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u;
    ROW_WARPS_BEGIN
    const uint2 inf = P.info[f.row0 + y];
    const uint32_t *ps = P.pslot + (f.row0 + y) * P.nd_cap;
    const uint16_t *pi = P.pid + (f.row0 + y) * P.nd_cap;
    for (uint32_t i = lane; i < inf.y; i += 32) {
        const uint32_t c = rank_of_slot[ps[i]];
        base[pi[i]] = seg[spanoff[c] + ((uint32_t)y - cy0[c])];
    }
    __syncwarp();
    const uint32_t *rec = P.rec + 2 * (f.q_off + y * f.qw);
    uint32_t rc0 = lane < inf.x ? rec[lane] : 0u, rc1 = lane + 32 < inf.x ? rec[lane + 32] : 0u;
    for (uint32_t r0 = 0; r0 < inf.x; r0 += 32) {
        const uint32_t r = r0 + lane;
        const bool valid = r < inf.x;
        const uint32_t rc = rc0;
        rc0 = rc1;
        if (r + 64 < inf.x) rc1 = rec[r + 64];
        const uint32_t id = valid ? rc & PREC_ID : 0xffffffffu;
        const uint32_t peers = __match_any_sync(0xffffffffu, id);
        const uint32_t at = valid ? base[id] + __popc(peers & lt) : 0u;
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) base[id] += __popc(peers);
        if (valid) {
            const uint32_t j = (rc >> 12) & 3u, x = rc >> 15;
            const int dx = j == 0 || j == 3 ? 1 : j == 2 ? -1 : 0, dy = j == 0 ? 0 : 1;
            const int g = (rc >> 14 & 1u) ? 255 : -255;
            const uint64_t px = (uint64_t)(2 * (int64_t)x + dx), py = (uint64_t)(2 * y + dy);
            const uint64_t gx = (uint16_t)(int16_t)(dx * g), gy = (uint16_t)(int16_t)(dy * g);
            if (at < npts)  // always, unless the counts disagree: then an error, not a stray write
                out[at] = px | py << 16 | gx << 32 | gy << 48;
            else
                atomicOr(err, AT_ERR_CAPACITY);
        }
        __syncwarp();
    }
    ROW_WARPS_END
}

// ---------------------------------------------------------------------------
// Launchers.

static inline unsigned flat_grid(int64_t n, int threads) {
    const int64_t b = (n + threads - 1) / threads;
    return (unsigned)(b < 1 ? 1 : b < 148 * 16 ? b : 148 * 16);
}

static inline dim3 row_warps(const Launch &L) {
    const int64_t b = (L.max_qh + 7) / 8;
    return dim3((unsigned)(b < 1 ? 1 : b < 148 * 8 ? b : 148 * 8), (unsigned)L.nframes);
}

// Warps per block of the point scan: their row tables within 96 KB.
static inline int scan_warps(int nd_cap) {
    const int w = (int)((96 * 1024) / row_pairs_bytes(nd_cap));
    return w < 1 ? 1 : w > 8 ? 8 : w;
}

bool point_scan_set_smem() {
    return cudaFuncSetAttribute(k_point_scan, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024) == cudaSuccess &&
           cudaFuncSetAttribute(k_point_place, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024) == cudaSuccess;
}

void launch_point_scan(const Launch &L, const FrameDesc *frames, const RowWord *words, const uint32_t *lab, int nb,
                       const PairTable &T, const PointRows &P, uint32_t *full, unsigned long long *npoints) {
    const int w = scan_warps(P.nd_cap);
    const int64_t b = (L.max_qh + w - 1) / w;
    const dim3 grid((unsigned)(b < 1 ? 1 : b < 148 * 8 ? b : 148 * 8), (unsigned)L.nframes);
    launch(k_point_scan, grid, 32 * w, w * row_pairs_bytes(P.nd_cap), L.stream, frames, words, lab, nb, T, P, full, npoints);
}

int launch_pair_order(cudaStream_t s, const uint64_t *okeys, const uint32_t *oslots, int64_t ncl, int nb,
                      const FrameDesc *frames, int nframes, const PairTable &T, const PairScratch &P,
                      uint64_t *skeys, uint32_t *sslots, uint32_t *rank_of_slot, uint32_t *ccount, uint32_t *cspan,
                      uint32_t *cy0, int32_t *cframe, uint32_t *cstart, uint32_t *spanoff, uint32_t *seg, int64_t cap,
                      uint32_t *err) {
    if (ncl <= 0) return 0;
    if (ncl <= PAIR_SMALL) {
        launch(k_pair_small, 1, 1024, 0, s, okeys, oslots, (int)ncl, T, nb, frames, nframes, skeys, rank_of_slot, cspan, cy0,
               cframe, cstart, spanoff, seg, cap, err);
        return 1;
    }
    const int nbuckets = nframes * PAIR_BUCKETS;
    cudaMemsetAsync(P.bcount, 0, (size_t)nbuckets * 4, s);
    launch(k_pair_frame, flat_grid(ncl, 256), 256, 0, s, okeys, ncl, nb, frames, nframes, P.kbucket, P.bcount);
    launch(k_pair_offsets, 1, 1024, 0, s, P.bcount, nbuckets, P.boff, P.bcur);
    launch(k_pair_scatter, flat_grid(ncl, 256), 256, 0, s, okeys, oslots, ncl, P.kbucket, P.boff, P.bcur, P.gkeys,
           P.gslots, P.gbucket);
    launch(k_pair_rank, flat_grid(ncl * 32, 256), 256, 0, s, P.gkeys, P.gslots, P.gbucket, ncl, P.boff, skeys, sslots);
    launch(k_cluster_span, flat_grid(ncl, 256), 256, 0, s, skeys, sslots, ncl, T, nb, frames, nframes, rank_of_slot,
                                                       ccount, cspan, cy0, cframe);
    const int64_t nblk = (ncl + SCAN_ITEMS - 1) / SCAN_ITEMS;
    launch(k_scan2_sums, (unsigned)nblk, SCAN_THREADS, 0, s, ccount, cspan, ncl, P.bsum_a, P.bsum_b);
    launch(k_scan2_top, 1, 1024, 0, s, P.bsum_a, P.bsum_b, nblk);
    launch(k_scan2_apply, (unsigned)nblk, SCAN_THREADS, 0, s, ccount, cspan, ncl, P.bsum_a, P.bsum_b, nblk, cstart,
                                                          spanoff);
    launch(k_seg_zero, flat_grid(cap, 256), 256, 0, s, spanoff, ncl, seg, cap, err);
    return 9;
}

int64_t pair_buckets(int nframes) { return (int64_t)nframes * PAIR_BUCKETS; }
int64_t pair_scan_blocks(int64_t ncl) { return (ncl + SCAN_ITEMS - 1) / SCAN_ITEMS + 1; }

// An exclusive scan of n u32 values into out (n + 1 entries, the total
// last) with the two-array kernels above, the second array the first
// again; scratch: scan_u32_scratch(n) values.
int64_t scan_u32_scratch(int64_t n) { return 2 * ((n + SCAN_ITEMS - 1) / SCAN_ITEMS + 1) + n + 1; }

void launch_scan_u32(cudaStream_t s, const uint32_t *a, int64_t n, uint32_t *out, uint32_t *scratch) {
    if (n <= 0) return;
    const int64_t nblk = (n + SCAN_ITEMS - 1) / SCAN_ITEMS;
    uint32_t *sa = scratch, *sb = scratch + nblk + 1, *ob = scratch + 2 * (nblk + 1);
    launch(k_scan2_sums, (unsigned)nblk, SCAN_THREADS, 0, s, a, a, n, sa, sb);
    launch(k_scan2_top, 1, 1024, 0, s, sa, sb, nblk);
    launch(k_scan2_apply, (unsigned)nblk, SCAN_THREADS, 0, s, a, a, n, sa, sb, nblk, out, ob);
}

void launch_point_place(const Launch &L, const FrameDesc *frames, const PointRows &P, const uint32_t *rank_of_slot,
                        const uint32_t *cstart, const uint32_t *spanoff, const uint32_t *cspan, const uint32_t *cy0,
                        int64_t ncl, uint32_t *seg, int64_t cap, uint64_t *out, int64_t npts, uint32_t *err) {
    if (ncl <= 0) return;
    launch(k_seg_fill, row_warps(L), 256, 0, L.stream, frames, P, rank_of_slot, spanoff, cy0, ncl, seg, cap);
    launch(k_seg_scan, flat_grid(ncl * 32, 256), 256, 0, L.stream, cstart, spanoff, cspan, ncl, seg, cap);
    launch(k_point_place, row_warps(L), 256, 16 * P.nd_cap * 4, L.stream, frames, P, rank_of_slot, spanoff, cy0, ncl, seg,
                                                                    cap, out, npts, err);
}

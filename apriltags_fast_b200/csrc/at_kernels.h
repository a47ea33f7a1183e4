// Launchers of the detection kernels (defined in at_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "at_gpu.h"

// Union-find nodes, indexed by node id.
struct RunArrays {
    uint32_t *parent;  // union-find parent (in the end: a run's band root, a band root's component root)
    uint32_t *px;      // at a root: its component's pixel count
    uint32_t *minid;   // at a root: its component's smallest node id (the label)
    uint32_t *lab;     // each node's label, or AT_NOK
};

#define FIT_NBUCKET 16
// Per-point scratch of the quad fit, indexed by point position.
struct FitScratch {
    uint64_t *keys, *skey;
    uint32_t *sval;
    double *mx, *my, *mxx, *mxy, *myy, *mw;
    double *errs, *filt, *mxe;
    int32_t *mxi;
    uint32_t *lists;   // one list of cluster ids per size bucket, nclusters apart
    uint32_t *counts;  // per bucket: list length, then the clusters taken
};

struct BlurTaps {
    int n;
    uint8_t k[64];
};

// The grid of the per-frame kernels: x blocks per frame, one row of frames.
struct Launch {
    cudaStream_t stream;
    int nframes;
    int blocks_per_frame;
    int64_t max_qh;  // the tallest quad image of the batch
};

void launch_decimate(const Launch &L, const FrameDesc *frames, const uint8_t *img, uint8_t *qim, float factor);
void launch_blur(const Launch &L, const FrameDesc *frames, uint8_t *qim, uint8_t *tmp_a, uint8_t *tmp_b,
                 const BlurTaps &taps, bool sharpen);
void launch_threshold(const Launch &L, const FrameDesc *frames, const uint8_t *qim, uint8_t *tmax, uint8_t *tmin,
                      uint8_t *thr, int32_t diff);
// Decimate 2 + tile max/min + threshold in one pass (no blur): max_blocks
// from decimate_threshold_blocks of the batch's largest frame.
void launch_decimate_threshold(const Launch &L, const FrameDesc *frames, int64_t max_blocks, uint8_t *qim,
                               uint8_t *thr, int32_t diff);
int64_t decimate_threshold_blocks(int64_t qw, int64_t qh);
void launch_deglitch(const Launch &L, const FrameDesc *frames, uint8_t *thr, uint8_t *tmp);
// Runs, components and labels (at_segment.cu). segment_plan: the most bands
// of a frame and the shared memory of a band, over the batch's frames.
#define SEGMENT_SMEM (224 * 1024)  // a band's, at most: quad images up to 425984 columns
bool segment_set_smem();
void segment_plan(int qw, int qh, int64_t *max_bands, size_t *smem);
int launch_segment(const Launch &L, const FrameDesc *frames, int64_t max_bands, size_t smem, const uint8_t *thr,
                   RunArrays runs, uint32_t *row_nruns, uint32_t *band_roots, RowWord *words, int32_t min_px);
// the labels per pixel (the sorting fallback of the clusters, diagnostics)
void launch_labels(const Launch &L, const FrameDesc *frames, RunArrays runs, const RowWord *words, uint32_t *lab);
void launch_point_count(const Launch &L, const FrameDesc *frames, const uint8_t *thr, const uint32_t *lab,
                        uint64_t *row_npts);
void launch_point_emit(const Launch &L, const FrameDesc *frames, const uint8_t *thr, const uint32_t *lab,
                       const uint64_t *row_pt_off, uint64_t *pt_key, uint64_t *pt_val, int nb);
void launch_cluster_heads(cudaStream_t s, const uint64_t *key, int64_t n, uint32_t *head);
void launch_cluster_collect(cudaStream_t s, const uint64_t *tkeys, uint32_t size, uint64_t *okeys, uint32_t *oslots,
                            uint32_t *count);
// Clusters without sorting the points (at_cluster.cu). The pair table:
// key (label pair), point count, first and last row with points, per slot.
struct PairTable {
    uint64_t *keys;
    uint32_t *count, *ymin, *ymax;
    uint32_t mask;
};
// Scratch of the pair ordering: per pair its bucket, per bucket (pair_buckets)
// its pair count, first pair (one more entry) and a cursor, the pairs grouped
// by bucket with their buckets, and the block sums of the scans
// (pair_scan_blocks each). The bucket arrays are 16-byte aligned.
struct PairScratch {
    uint32_t *kbucket, *bcount, *boff, *bcur;
    uint64_t *gkeys;
    uint32_t *gslots, *gbucket, *bsum_a, *bsum_b;
};
int64_t pair_buckets(int nframes);
// The points of each row (rows 1 .. qh-2): records in emission order at
// rec + 2 (q_off + y qw), at most 2 qw a row (the pair's place in the row's
// table | neighbour << 12 | pixel is 0 << 14 | x << 15); the row's distinct
// pairs (slot in the pair table, points, place in the row's table) at (row0 +
// y) nd_cap; info[row0 + y] = (records, pairs).
struct PointRows {
    uint32_t *rec;
    uint32_t *pslot, *pcnt;
    uint16_t *pid;
    uint2 *info;
    int32_t nd_cap;
};
bool point_scan_set_smem();
void launch_point_scan(const Launch &L, const FrameDesc *frames, const RowWord *words, const uint32_t *lab, int nb,
                       const PairTable &T, const PointRows &P, uint32_t *full, unsigned long long *npoints);
int launch_pair_order(cudaStream_t s, const uint64_t *okeys, const uint32_t *oslots, int64_t ncl, int nb,
                      const FrameDesc *frames, int nframes, const PairTable &T, const PairScratch &P,
                      uint64_t *skeys, uint32_t *sslots, uint32_t *rank_of_slot, uint32_t *ccount, uint32_t *cspan,
                      uint32_t *cy0, int32_t *cframe, uint32_t *cstart, uint32_t *spanoff, uint32_t *seg, int64_t cap,
                      uint32_t *err);
int64_t pair_scan_blocks(int64_t ncl);
int64_t scan_u32_scratch(int64_t n);
void launch_scan_u32(cudaStream_t s, const uint32_t *a, int64_t n, uint32_t *out, uint32_t *scratch);
void launch_point_place(const Launch &L, const FrameDesc *frames, const PointRows &P, const uint32_t *rank_of_slot,
                        const uint32_t *cstart, const uint32_t *spanoff, const uint32_t *cspan, const uint32_t *cy0,
                        int64_t ncl, uint32_t *seg, int64_t cap, uint64_t *out, int64_t npts, uint32_t *err);
void launch_cluster_starts(cudaStream_t s, const uint64_t *key, const uint32_t *head, const uint32_t *head_scan,
                           int64_t n, int nb, const FrameDesc *frames, int nframes, uint32_t *cstart, int32_t *cframe,
                           uint64_t *ckey);
// The streams of the fit's size classes, their start and ends (events
// without timing). max_px: the largest FrameDesc.max_px of the batch.
// Returns the kernels launched.
struct FitStreams {
    cudaStream_t side[4];
    cudaEvent_t fork, join[4];
};
int launch_fit_quads(cudaStream_t s, const FitStreams &S, const FrameDesc *frames, const GpuParams &prm,
                     const uint8_t *qim, const uint64_t *pts, const uint32_t *cstart, const int32_t *cframe,
                     int64_t nclusters, int64_t npoints, int64_t max_px, const FitScratch &scr, GpuQuad *quads,
                     uint32_t *quad_ok, uint32_t *err);
// The quads in cluster order (grouped by frame), their clusters (qcl) and
// count; each frame's first quad and first detection slot (nfam a quad).
// scan: n + 1 values; scratch: scan_u32_scratch(n). Returns the launches.
int launch_gather_quads(cudaStream_t s, const GpuQuad *quads, const uint32_t *ok, int64_t n, uint32_t *scan,
                        uint32_t *scratch, int nframes, int nfam, GpuQuad *out, uint32_t *nq, uint32_t *qcl,
                        int64_t *qstart, int64_t *out_off);
void launch_output(cudaStream_t s, int nframes, const int64_t *qstart, const GpuDetection *out,
                   const int64_t *out_off, const int64_t *out_n, int64_t *first, GpuDetection *host,
                   int64_t *meta, int64_t max_dets);
// per quad: refined corners (8 floats), homography (9 doubles), and whether
// the homography was found and is invertible
struct DecodeScratch {
    float *corners;
    double *h;
    uint32_t *hok;
    const uint32_t *nq;  // the number of quads, on the device
};
void launch_decode(cudaStream_t s, const FrameDesc *frames, const GpuParams &prm, const GpuFamily *fams,
                   const uint8_t *img, const uint8_t *qim, const GpuQuad *quads, int64_t max_quads,
                   const DecodeScratch &scr, GpuDetection *dets, uint32_t *det_ok);
// The reference's order of the quads whose detections share an id
// (at_order.cu). Per frame: whether it has such detections (need), the
// target components (GPU labels, pixel counts, and at last their roots in
// the reference's packed node numbering); per node, the frame's target runs
// compacted by row (tlist); per row, their count (trow); per row plus one
// per frame, the runs above the row (rpre).
#define AT_REF_MAXT 192
#define REF_PCAP 4160       // runs of a row, at most (quad images up to 4161 px wide)
struct RefOrder {
    uint32_t *need, *nt;
    uint32_t *tlabel, *tpx, *troot;
    uint64_t *tlist;
    uint32_t *trow;
    uint32_t *rpre;
    // per node: its edge in the forest of unions (time << 32 | parent), the
    // pixels below it, a mark; per target run (in tlist's order): the first
    // and last run of the row above that it touches
    uint64_t *par;
    uint32_t *sum, *stamp, *tch;
    uint16_t *len;            // per target run: its pixels
    // per target (AT_REF_MAXT a frame) and row: pixels gained (zeroed by the caller)
    uint32_t *hist;
};
// returns the kernels launched
int launch_ref_order(const Launch &L, const FrameDesc *frames, const RowWord *words, RunArrays runs,
                     const uint32_t *row_nruns, int nfam, const int64_t *qstart, const GpuDetection *dets,
                     const uint32_t *det_ok, const uint32_t *qcl, const uint64_t *ckey, int nb, const RefOrder &ref,
                     uint32_t *err);
// okey: 2 u64 + 1 u32 per detection slot (the order keys, a second index)
void launch_finalize(cudaStream_t s, int nframes, const int64_t *frame_qstart, int nfam, const GpuDetection *dets,
                     const uint32_t *det_ok, uint32_t *idx, uint8_t *removed, GpuDetection *out,
                     const int64_t *out_off, int64_t *out_n, const FrameDesc *frames, const RefOrder &ref,
                     const uint32_t *qcl, const uint64_t *ckey, int nb, uint64_t *okey, uint32_t *idx2,
                     uint32_t *err);

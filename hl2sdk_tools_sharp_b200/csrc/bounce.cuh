// bounce.cuh -- the radiosity bounce resident on one device.
//
// Layout in HBM (P patches in the reference's index order, R receivers,
// F faces, Q candidate pairs, T transfers):
//   origin[P]    float4 (origin xyz, area)
//   normal[P]    float4 (shading normal xyz, plane dist)
//   mins[P]      float4 (winding bounds min xyz, face bits)
//   maxs[P]      float4 (winding bounds max xyz, cluster bits)
//   tree[P]      int4   (parent, child1, child2, sky)
//   refl[P]      float4 (reflectivity xyz, -)
//   wind[P]      int2   (first point, count) into points[] float4
//   face_range[F] int4  (root patch, first descendant, end of descendants, -)
//   face_samples[F] int2 (first sample, count)
//   face_plane[F] float4 (plane normal xyz, dist)
//   recv[R]      int32  receiver order (VisMatrix.ReceiverOrder): cluster by
//                       cluster, each cluster's leaf patches in index order
//   start[R]     int32  the opaque BVH node where the receiver's transfer
//                       rays start their walk (traverse.cuh:start_node)
//   row_off / row_faces  per cluster, the faces its PVS row reaches, in
//                       VisMatrix.FacesInRow order
//   cand_off[R+1] int64, cand_src[Q] int32, cand_w[Q] float: each receiver's
//                       candidate sources in enumeration order and the
//                       transfer each earns (0 when blocked or none)
//   tr_off[R+1] int64, tr[T] int2 (source, weight bits): the transfer lists
//                       (TransferSet), by receiver
//   direct[P], total[P], emit[2][P], shoot[2][P] float4: PatchLighting and Radiosity state
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "direct.cuh"
#include "host_parallel.h"
#include "scene.cuh"
#include "vrad_internal.cuh"

struct vrad_mlp;

namespace vrad {

struct FinalView;

constexpr int64_t kMaxTransfersPerReceiver = 4 * 65536;  // VisMatrix.MaxPatches
constexpr int kSums = 9;  // doubles in a part of BounceBuffers::sums
constexpr int kSumParts = 64;
constexpr int kCountBits = 20;  // of a SELL key: a receiver has at most 2^18 transfers
constexpr uint32_t kCountMask = (1u << kCountBits) - 1;
// Segments to a receiver's row in the candidate walk: as many as make 32 k
// warps (seven rounds of the chip's 4736 resident ones, so that the last
// round weighs little), up to 16 (k_candidates; about ten faces each then).
inline int32_t row_segments(int32_t receivers) {
    return (int32_t)std::min<int64_t>(16, std::max<int64_t>(1, 32 * 32768ll / std::max(receivers, 1)));
}
// Receivers to a window of the slices' sort, for `receivers` in all: 1024
// (k_gather), or so many that the windows' numbers fit the key's other 12 bits.
inline int32_t sell_window(int32_t receivers) {
    const int64_t least = ((int64_t)receivers + 4095) / 4096;
    return (int32_t)std::max<int64_t>(1024, (least + 31) / 32 * 32);
}
constexpr int kGroup = 16;  // receivers of a transfer group (k_transfer_groups)
constexpr int32_t kGroupedReceivers = 65536;
constexpr int kFeatures = 32;                            // the warm start network's inputs

struct BounceView {
    int32_t npatches, nfaces, nreceivers;
    const float4 *origin;
    const float4 *normal;
    const float4 *mins;
    const float4 *maxs;
    const int4 *tree;
    const float4 *refl;
    const int2 *wind;
    const float4 *points;
    const int4 *face_range;
    const int2 *face_samples;
    const float4 *face_plane;
    const int32_t *recv;
    const int32_t *row_off;
    const int32_t *row_faces;
    const float *sample_area;
    const float4 *sample_pos;  // the world's (xyz, face bits)
};

struct BounceBuffers {
    // Geometry and tables, built once by vrad_bounce_upload.
    float4 *origin = nullptr, *normal = nullptr, *mins = nullptr, *maxs = nullptr, *refl = nullptr;
    int4 *tree = nullptr;
    int2 *wind = nullptr;
    float4 *points = nullptr;
    int4 *face_range = nullptr;
    int2 *face_samples = nullptr;
    float4 *face_plane = nullptr;
    int32_t *recv = nullptr, *start = nullptr, *row_off = nullptr, *row_faces = nullptr;
    float *sample_area = nullptr;
    // Transfer build.
    int64_t *cand_off = nullptr;   // R + 1
    int64_t *seg_off = nullptr;    // R * segments + 1: the same by segment of the receiver's row
    int32_t segments = 1;
    // The transfer rays' warps, by group of kGroup receivers
    // (k_transfer_groups): group g's are group_off[g] .. group_off[g + 1].
    int64_t *group_off = nullptr;
    int32_t *warp_group = nullptr;  // per such warp, its group
    int64_t transfer_warps = 0;
    bool grouped() const { return nreceivers >= kGroupedReceivers; }
    int32_t ngroups() const { return (nreceivers + kGroup - 1) / kGroup; }
    int32_t *cand_src = nullptr;   // Q
    float *cand_w = nullptr;       // Q
    int64_t *tr_off = nullptr;     // R + 1
    int2 *tr = nullptr;            // T
    void *scan_tmp = nullptr;
    size_t scan_tmp_bytes = 0;
    // The transfers again, in slices for the gather (SELL-32): each window of
    // sell_window consecutive receivers sorted by transfer count, descending
    // (stable), 32 receivers to a slice; entry j of lane l of slice s at
    // sell[sell_off[s] + 32 j + l], so a warp's loads of step j are one
    // contiguous 256 B row.  Keys: window << kCountBits | kCountMask - count.
    uint32_t *sell_key = nullptr, *sell_sorted = nullptr;  // R: before and after the sort
    int32_t *sell_idx = nullptr, *sell_order = nullptr;    // R: the receivers alike
    int32_t sell_window = 0;  // a multiple of 32; all receivers where memory is short
    int64_t sell_cap = 0;     // entries sell has room for
    int64_t *sell_off = nullptr;   // slices + 1
    int2 *sell = nullptr;          // at most T + 32 * (each window's largest count) entries
    void *sort_tmp = nullptr;
    size_t sort_tmp_bytes = 0;
    int64_t ncand = 0, ntransfers = 0;
    // Light state.
    float4 *direct = nullptr, *total = nullptr;
    float4 *emit[2] = {nullptr, nullptr}, *shoot[2] = {nullptr, nullptr};
    // fp64 totals of a bounce in kSumParts parts of kSums: 3 sums, 3 absolute
    // sums, 3 absolute sums weighted by the terms left in CollectLight's order.
    double *sums = nullptr;
    float *exact = nullptr;        // the sequential float total, when needed
    double *exact_sums = nullptr;  // per channel and chunk of exact_per leaves (k_exact_sums)
    void *exact_steps = nullptr;   // alike (k_exact_steps)
    int32_t exact_per = 0, exact_chunks = 0;
    int32_t *leaf_desc = nullptr;  // the sky-free leaves, descending index (CollectLight's total order)
    int32_t *leaf_rank = nullptr;  // per patch: its position in leaf_desc, -1 off it
    // Each face's parents level by level, bottom up (a level: the depth of
    // the subtree below): face f's level k are the entries level_off[face_level[f]
    // + k] .. level_off[face_level[f] + k + 1] of parent (patch, its children,
    // sky) and share (the children's shares of its area).
    int32_t *face_level = nullptr, *level_off = nullptr, *parent_list = nullptr;
    int4 *parent = nullptr;
    float2 *share = nullptr;
    int32_t nparents = 0;
    // Per face, what the candidate walk reads of its root: (normal, the
    // largest float up to plane dist + 0.01), (origin, area), (patch, child1,
    // child2, face).
    float4 *root_plane = nullptr, *root_origin = nullptr;
    int4 *root_tree = nullptr;
    int4 *patch_box = nullptr;     // per patch: its cells in reach (k_patch_boxes)
    // Learned warm start.
    float4 *first = nullptr;       // the first bounce's light per patch (bounce 0's total)
    float4 *guess = nullptr;       // the network's guess per patch
    uint16_t *feat = nullptr;      // R x 32 BF16 inputs
    float *pred = nullptr;         // R x 3 outputs
    const vrad_mlp *model = nullptr;
    // [0] the slices' padding, at the upload; [1] blocked transfer rays, [2]
    // asin ties left open, of a transfer build.
    unsigned long long *counters = nullptr;
    double *h_parts = nullptr;     // pinned host copy of the parts
    double h_sums[9] = {};         // their sums (add_parts)
    float *h_exact = nullptr;
    // Final pass: each face's leaf patches whose radial box reaches it.
    int32_t *pr_off = nullptr;     // F + 1
    int32_t *pr_patch = nullptr;
    int4 *pr_box = nullptr;        // sMin, tMin, sMax, tMax
    float4 *pr_coord = nullptr;    // coordS, coordT, distS, distT
    float4 *prad_light = nullptr;  // per cell
    float *prad_weight = nullptr;

    BounceView view{};
    uvector<int32_t> h_recv;         // host copy of the receiver order
    int32_t npatches = 0, nfaces = 0, nreceivers = 0, nleaves = 0;
    int32_t max_bounces = 0;
    float threshold = 1.0f;
    int32_t last_buffer = 0;         // which emit/shoot half the last bounce wrote
    // One bounce of each parity captured as a graph (gather with the totals,
    // CollectLight's parents, the totals' copy to h_parts), made on first use.
    cudaGraphExec_t bounce_graph[2] = {nullptr, nullptr};
    bool ready = false;
    // The transfer lists came from vrad_transfer_install: every light pass
    // bounces with them instead of building, until the next upload.
    bool installed = false;
    // tr_off / tr hold a set (a light pass bounced, or one was installed).
    bool lists_ready = false;
    // Statistics of the last pass.
    int32_t bounces_run = 0, exact_totals = 0;
    double added[3] = {0, 0, 0};
    float patch_light_ms = 0, transfer_ms = 0, bounce_ms = 0, final_ms = 0;
    unsigned long long rays = 0, blocked = 0, open_ties = 0;

    // The last bounce's totals from the copied parts.
    void add_parts() {
        for (int k = 0; k < kSums; k++) {
            h_sums[k] = 0.0;
            for (int p = 0; p < kSumParts; p++) h_sums[k] += h_parts[kSums * p + k];
        }
    }

    void release();      // the device tables; the pinned sums stay
    void free_pinned();  // the pinned sums
};

// The tables the bounce's kernels read that follow from the uploaded patches
// (the leaves' cells, the parents and their shares), once per upload;
// face_fit: F float4 of scratch.
cudaError_t launch_bounce_tables(const BounceBuffers &b, const FinalView &fv, float4 *face_fit, cudaStream_t stream);
// The transfer warps' groups, once group_off is known and warp_group allocated.
cudaError_t launch_warp_groups(const BounceBuffers &b, cudaStream_t stream);
// How many entries the slices can need beyond the transfers, from the
// candidate counts (cand_off), added to *d_pad.
cudaError_t launch_sell_pad(const BounceBuffers &b, unsigned long long *d_pad, cudaStream_t stream);
// The slices' sort: the bytes of its scratch (tmp == nullptr) or the sort.
cudaError_t sell_sort(BounceBuffers &b, int32_t window, void *tmp, size_t &bytes, cudaStream_t stream);
// Device phases of one bounce pass, all on `stream`.
cudaError_t launch_patch_light(const BounceBuffers &b, const FinalView &fv, const float4 *sample_light, cudaStream_t stream);
cudaError_t launch_transfers(BounceBuffers &b, const DeviceScene &scene, uint32_t *overflow, cudaStream_t stream,
                             bool count_only);
// The gather's slices from the transfer lists (the transfer build's last
// step; also after the lists are installed from a cache), sorted within
// windows of `window` receivers, a multiple of 32.
cudaError_t launch_sell(BounceBuffers &b, int32_t window, cudaStream_t stream);
cudaError_t launch_gather(BounceBuffers &b, int bounce, cudaStream_t stream);
// The sequential total's buffers, for b.nleaves leaves.
cudaError_t alloc_exact(BounceBuffers &b);
cudaError_t launch_exact_total(BounceBuffers &b, int bounce, cudaStream_t stream);
// Bounce number `bounce` and the copy of its totals to h_parts as one graph
// launch on `stream`; the graph of its parity is captured on `capture` (a
// stream of the library's own) the first time.
cudaError_t launch_bounce_graph(BounceBuffers &b, int bounce, cudaStream_t capture, cudaStream_t stream);
cudaError_t launch_features(BounceBuffers &b, const DeviceWorld &w, cudaStream_t stream);
cudaError_t launch_warm_start(BounceBuffers &b, const DeviceWorld &w, const vrad_mlp &m, cudaStream_t stream);

}  // namespace vrad

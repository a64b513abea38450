// dtrt_gb300 — host-side scene object and the per-width render entry points.
#pragma once
#include <string>
#include <vector>

#include "../../include/dtrt_gb300.h"
#include "dt_buffers.h"
#include "dt_bvh.h"
#include "dt_kernels.cuh"
#include "dt_lanes.h"

namespace dt {

void set_last_error(const std::string &msg);

// The density replay keeps 684 B a path (144 B of state, 32 of inputs, 16 of queues, 12 of values,
// 480 of events), and a program that holds many scenes holds a workspace for each: 2^22 paths in
// all (2.9 GB). C3 density adjoint: one lane of 2^22 40.7 ms, 2 of 2^21 38.5, 4 of 2^20 37.2, 8 of
// 2^19 38.0 (8 of 2^21, 11.5 GB, 34.7).
constexpr int kReplayLanes = 4;
constexpr long long kReplayBatchPaths = 1ll << 20;

// Device buffers reused across renders of one scene, grown on demand.
struct Scratch : Lanes {
    double *acc1 = nullptr, *acc2 = nullptr;
    size_t acc1_n = 0, acc2_n = 0;
    float *out = nullptr;
    size_t out_n = 0;
    void *qe = nullptr, *ql = nullptr, *qli = nullptr;
    size_t qe_bytes = 0, ql_bytes = 0, qli_bytes = 0;
    unsigned long long *counts = nullptr;  // [0] edge recs, [1] lins recs, [2] li tasks, [8..] counters
    unsigned int *err = nullptr;
    // adjoint render: dL/dI staging, density gradient, FP64 image accumulator, image staging
    float *adj_dimg = nullptr, *adj_grad = nullptr, *adj_out = nullptr;
    double *adj_img = nullptr;
    size_t adj_dimg_n = 0, adj_grad_n = 0, adj_out_n = 0, adj_img_n = 0;
    // wavefront schedules: path states and vertex inputs, four path-index queues, per-level counts
    void *cam_state = nullptr, *cam_q = nullptr, *cam_cnt = nullptr;
    size_t cam_state_bytes = 0, cam_q_bytes = 0, cam_cnt_bytes = 0;
    // sort of the Li sub-path pairs: keys, values, their double buffers and digit counts
    void *li_sort = nullptr;
    size_t li_sort_bytes = 0;
    // density cells of a render (DevScene::cells), then the replay's gradient in that layout
    void *cells = nullptr;
    size_t cells_bytes = 0;
};

// A buffer of at least `need` bytes at *ptr; a full device gives up the density cells, which no kernel
// of the render reads yet: prepare_cells comes after every other buffer.
bool ensure_buffer(Scratch &sb, void **ptr, size_t *have, size_t need);
// The wavefront workspaces (cam_state, cam_q, cam_cnt) given back
void drop_wavefront(Scratch &sb);

// Buffers of the Li pair sort for queues of li_cap tasks (li_cap / 2 pairs): false (and
// the allocation error cleared) when the device has no room, the Li kernels then read the
// queue in order.
inline bool ensure_li_sort(Scratch &sb, uint64_t li_cap) {
    const long long cap = (long long)(li_cap / 2);
    if (ensure_buffer(sb, &sb.li_sort, &sb.li_sort_bytes, (size_t)cap * 16 + radix_hist_entries(cap) * 4)) return true;
    cudaGetLastError();
    return false;
}

// Fewer pairs or samples than this run in queue order: the sort's 13 launches take about 60 us,
// more than it saves them (2^12 / 2^17 / 2^18 here: preview of 3,300 pairs 0.66 / 0.64 / 0.67 ms,
// the last two the same code there; render_scene, some 2^17 samples a stage, 8.6 / 8.3 / 8.3; C0
// forward, 10^7, equal).
constexpr long long kSortMin = 1 << 17;

// The n queued Li tasks' pairs (slots 2m, 2m + 1) in key order (k_li_keys) on stream st;
// nullptr when n is odd or small (the queue is then read in order). Adds the
// kernels it launches to `launches`.
template <class Task>
const int *sort_li_pairs(const DevScene &sc, const Task *tasks, long long n, Scratch &sb, uint64_t li_cap,
                         cudaStream_t st, uint64_t &launches) {
    const long long np = n / 2, cap = (long long)(li_cap / 2);
    if ((n & 1) || np < kSortMin || np > cap) return nullptr;
    unsigned *keys = (unsigned *)sb.li_sort, *keys2 = keys + cap;
    int *vals = (int *)(keys2 + cap), *vals2 = vals + cap;
    unsigned *hist = (unsigned *)(vals2 + cap);
    k_li_keys<Task><<<(unsigned)((np + 255) / 256), 256, 0, st>>>(sc, tasks, np, keys, vals);
    launches += 1 + radix_sort_launches(kLiSortKeyBits);
    return radix_sort_bits(keys, vals, keys2, vals2, hist, (int)np, kLiSortKeyBits, st);
}

// The primary-edge samples [rp.prim_begin, + rp.prim_count) in key order (k_primary_keys),
// in the Li sort's buffers (a chunk holds at most li_cap / 2 samples); nullptr for few.
// Adds the kernels it launches to `launches`.
inline const int *sort_primary_samples(const RenderParams &rp, Scratch &sb, uint64_t li_cap, cudaStream_t st,
                                       uint64_t &launches) {
    const long long cap = (long long)(li_cap / 2);
    if (rp.prim_count < kSortMin || rp.prim_count > cap) return nullptr;
    unsigned *keys = (unsigned *)sb.li_sort, *keys2 = keys + cap;
    int *vals = (int *)(keys2 + cap), *vals2 = vals + cap;
    unsigned *hist = (unsigned *)(vals2 + cap);
    k_primary_keys<<<(unsigned)((rp.prim_count + 255) / 256), 256, 0, st>>>(rp, keys, vals);
    launches += 1 + radix_sort_launches(20);
    return radix_sort_bits(keys, vals, keys2, vals2, hist, (int)rp.prim_count, 20, st);
}


// Rays and hits of the scene carry no derivatives: nothing moves but materials and media (vertex
// and camera velocities all absent or exactly zero, and no shape has vertex normals: their
// derivative array is there with them, velocities or not, and the general kernels read it).
// Continuation rays then have none either: a scatter point lies on its ray, a new direction is
// sampled from values.
inline bool static_rays(const DevScene &sc) {
    if (sc.vert_der || sc.face_n_der || sc.normal_der || sc.moving_geometry) return false;
    for (int j = 0; j < sc.nder; ++j)
        for (int a = 0; a < 3; ++a) {
            if (sc.cam.d_cpos[j][a] != 0.f) return false;
            for (int k = 0; k < 3; ++k)
                if (sc.cam.d_cframe[j][a][k] != 0.f) return false;
        }
    return true;
}

// The queries that apply to the scene's Li, Lins and edge kernels
inline int media_kind(const DevScene &sc) {
    if (sc.num_media == 0 && !sc.has_null && sc.cam.med_id < 0) return kNoMedia;
    return sc.has_grid_media ? kAnyMedia : kNoGrids;
}

// Camera paths per batch of a scene of static_rays(): its batches hold no records, only path
// states, vertex inputs and queues (224 to 384 B a path from nder 1 to 8: 0.24 to 0.40 GB a
// batch), and up to kLanes of them run at once (1.9 to 3.2 GB)
constexpr long long kStaticBatchPaths = 1ll << 20;

// Buffers of the camera wavefront for `cap` paths: path states, vertex inputs, four
// path-index queues, level counts
struct CamWave {
    void *states, *vins;
    int *q;
    unsigned long long *cnt;
    long long cap;
    int levels;
};

// Connectivity kept from the last build, so that a rebuild from a description with the
// same triangles (an optimisation step that moves vertices) skips the edge search and
// refits the BVH instead of building it again.
struct SceneTopology {
    bool valid = false;
    std::vector<int> shape_nv, shape_nt;
    std::vector<int> indices;                // every shape's triangles, shape-local vertex ids
    std::vector<int4> adj;                   // per shape: (a, b, f0, f1 or -1), shape-local, sorted by (a, b)
    std::vector<int> adj_off;                // num_shapes + 1 offsets into adj
    std::vector<int> media_type, media_res;  // per medium: type; density resolution (3 ints)
    BvhBuildOut bvh;                         // the tree as last built or refit (host builds)
    double sah_build = 0.0;                  // its surface-area cost right after the last full build
};

// Process-wide choice of the BVH builder for scenes created or updated afterwards.
int bvh_builder_setting();

}  // namespace dt

struct dtrt_scene {
    int nder = 0;
    int device = 0;
    dt::DevScene dev{};
    std::vector<void *> allocs;       // scene-lifetime device allocations, one per upload (null: empty)
    std::vector<size_t> alloc_bytes;  // byte size of each entry of allocs
    dt::Scratch scratch;
    bool counters = false;
    uint64_t queue_cap = 0;  // 0: automatic
    int camera_schedule = 0;  // DTRT_CAMERA_AUTO / _MEGAKERNEL / _WAVEFRONT
    dtrt_render_stats last{};
    int num_shapes = 0;
    std::vector<float> shape_edge_len;  // per shape total edge length (for re-weighting)
    std::vector<int> shape_skip;        // null-BSDF shapes without emitter
    std::vector<dt::DevMedium> media_host;  // host copy of the device media array
    std::vector<void *> dgrid_bufs;         // per medium: per-voxel derivative directions (owned)
    long long density_voxels = 0;           // voxels of all heterogeneous media (adjoint gradient length)
    dt::SceneTopology topo;
    dtrt_bvh_info bvh_info{};               // how the current tree was made
};

namespace dt {
// Density cells of a render of `paths` camera paths (with_grad: and zeroed gradient cells) in
// sc, from the scene's grids as they are now, on stream st; nothing when the render is too
// small for them (`per_path` voxels for each path: 16, or 2 for a primal path, which makes few
// lookups) or the device has no room. Returns the kernels launched.
int prepare_cells(dtrt_scene *s, DevScene &sc, long long paths, int per_path, bool with_grad, cudaStream_t st);
// sc.grad_cells summed into the voxels of `grad` (zeroed before); returns the kernels launched
int gather_cells(const dtrt_scene *s, const DevScene &sc, float *grad, cudaStream_t st);
template <int N>
int render_n(dtrt_scene *s, const dtrt_render_options *o, float *out, int out_on_device, cudaStream_t stream);
int render_adjoint(dtrt_scene *s, const dtrt_render_options *o, const float *d_image, float *image, float *d_density,
                   int on_device, cudaStream_t stream);
cudaError_t launch_adjoint(const DevScene &sc, const RenderParams &rp, const float *dimg, float *grad, double *img_acc,
                           unsigned long long *ctr, long long stride, cudaStream_t st);
// Device workspace of the wavefront density replay: path states, vertex inputs, four path-index queues,
// pass-A values and event values for `cap` paths, level counts of both passes.
struct AdjWave {
    void *states = nullptr, *vins = nullptr;
    int *q = nullptr;
    float3 *tots = nullptr, *ev = nullptr;
    unsigned long long *cnt = nullptr;
    long long cap = 0;
    int levels = 0;
    static size_t bytes(long long cap, int levels);
    void carve(void *base, long long cap, int levels);  // lay the arrays out in one allocation
};
cudaError_t launch_adjoint_wave(const DevScene &sc, const RenderParams &range, const float *dimg, float *grad,
                                double *img_acc, unsigned long long *ctr, const AdjWave &w, int sms, cudaStream_t st,
                                uint64_t *launches);
int render_vertex_adjoint(dtrt_scene *s, const dtrt_render_options *o, const float *d_image, float *image,
                          float *d_vertices, int on_device, cudaStream_t stream);
template <int N>
int render_n_noalloc(dtrt_scene *s, const dtrt_render_options *o, float *out, int out_on_device, cudaStream_t stream,
                     unsigned char *scratch, size_t scratch_bytes);
}  // namespace dt

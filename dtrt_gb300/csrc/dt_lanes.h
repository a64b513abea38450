// dtrt_gb300 — side streams of a render: batches in flight at once, and work beside the main stream.
#pragma once
#include <algorithm>

#include <cuda_runtime_api.h>

namespace dt {

// Wavefront batches in flight at once, each on a stream and a workspace of its own: a batch's
// last levels hold few paths and take as long as their slowest vertex, and the other batches
// run in the meantime; small batches read neighbouring voxels. C3 forward (33.6 M paths) / C1
// forward (16.8 M): 2 lanes of 2^23 paths 64.8 / 12.2 ms, 4 of 2^21 61.4 / 11.2, 8 of 2^20 60.8 /
// 11.1, 8 of 2^21 61.2 / 11.2, 8 of 2^19 64.0 / 11.6; C1 primal: 2 lanes of 2^22 15.3, 4 of 2^21
// 14.9, 8 of 2^20 14.7, 8 of 2^19 14.0, 8 of 2^18 14.7. Eight streams are what the device queues.
constexpr int kLanes = 8;

// Streams of the lanes 1..., the fork and join events (made by the first render that needs them)
struct Lanes {
    cudaStream_t side[kLanes - 1] = {};
    cudaEvent_t fork_ev = nullptr, side_ev[kLanes - 1] = {};
};

// Lanes for n batches of batch_paths paths each: `most`, or fewer where so many workspaces would
// hold more than most_paths paths (a batch takes whole pixels, and one may have 2^24 samples).
inline int lanes_for(long long n, long long batch_paths, int most, long long most_paths) {
    return (int)std::max<long long>(1, std::min({(long long)most, n, most_paths / std::max<long long>(1, batch_paths)}));
}

// Streams and events of `lanes` lanes: false (and the error cleared) when they cannot be made.
inline bool ensure_lanes(Lanes &sb, int lanes) {
    bool ok = sb.fork_ev || cudaEventCreateWithFlags(&sb.fork_ev, cudaEventDisableTiming) == cudaSuccess;
    for (int k = 0; k < lanes - 1 && ok; ++k) {
        ok = sb.side[k] || cudaStreamCreateWithFlags(&sb.side[k], cudaStreamNonBlocking) == cudaSuccess;
        ok = ok && (sb.side_ev[k] || cudaEventCreateWithFlags(&sb.side_ev[k], cudaEventDisableTiming) == cudaSuccess);
    }
    if (!ok) cudaGetLastError();
    return ok;
}

inline void free_lanes(Lanes &sb) {
    for (cudaStream_t q : sb.side)
        if (q) cudaStreamDestroy(q);
    for (cudaEvent_t e : sb.side_ev)
        if (e) cudaEventDestroy(e);
    if (sb.fork_ev) cudaEventDestroy(sb.fork_ev);
    sb = Lanes();
}

// f(batch, lane, stream) for each of n batches, dealt in turn to st and lanes - 1 side streams
// that fork from st and join it again.
template <class F>
cudaError_t in_lanes(Lanes &sb, cudaStream_t st, int lanes, long long n, F f) {
    cudaError_t e = cudaSuccess;
    auto ck = [&](cudaError_t r) { e = e == cudaSuccess ? r : e; };
    if (lanes > 1) {
        ck(cudaEventRecord(sb.fork_ev, st));
        for (int k = 1; k < lanes; ++k) ck(cudaStreamWaitEvent(sb.side[k - 1], sb.fork_ev, 0));
    }
    for (long long k = 0; k < n && e == cudaSuccess; ++k) {
        const int lane = (int)(k % lanes);
        ck(f(k, lane, lane ? sb.side[lane - 1] : st));
    }
    for (int k = 1; k < lanes; ++k) {
        ck(cudaEventRecord(sb.side_ev[k - 1], sb.side[k - 1]));
        ck(cudaStreamWaitEvent(st, sb.side_ev[k - 1], 0));
    }
    return e;
}

// Work on the first side stream beside what st does after fork(), joined into st by join() or,
// when a render gives up in between, at the end of the scope: no kernel is left behind that
// the buffers' next user would meet.
class SideWork {
  public:
    SideWork(Lanes &sb, cudaStream_t st) : sb_(sb), st_(st) {}
    ~SideWork() { join(); }
    SideWork(const SideWork &) = delete;
    SideWork &operator=(const SideWork &) = delete;
    bool open() const { return open_; }
    cudaStream_t stream() const { return sb_.side[0]; }
    cudaError_t fork() {  // needs ensure_lanes(sb, 2)
        const cudaError_t e = cudaEventRecord(sb_.fork_ev, st_);
        if (e != cudaSuccess) return e;
        open_ = true;
        return cudaStreamWaitEvent(sb_.side[0], sb_.fork_ev, 0);
    }
    cudaError_t join() {
        if (!open_) return cudaSuccess;
        open_ = false;
        const cudaError_t e = cudaEventRecord(sb_.side_ev[0], sb_.side[0]), f = cudaStreamWaitEvent(st_, sb_.side_ev[0], 0);
        return e != cudaSuccess ? e : f;
    }

  private:
    Lanes &sb_;
    cudaStream_t st_;
    bool open_ = false;
};

}  // namespace dt

// skg_wave.h -- host side of the wavefront packet tracer (kernels in skg_tracer.cu).
//
// A phase runs as a sequence of waves on one stream.  Wave w: a launch pass (scatter the packets that
// the previous wave brought to their interaction point, launch new packets into the records that it freed, and write the
// next traversals as jobs), the walks of every job, their ends (escape, termination, detection) and the re-walks.
// The number of waves is not known in advance: begin() enqueues an estimate (as many as the last phase took),
// finish() reads, behind the last of them, how many packets still had work and enqueues more until none has and
// no record waits for a new packet -- or, if few have by then, the tail pass, which finishes every remaining
// packet in one launch.  (A phase that ends within the estimate never sees the tail pass.)  Phases of few packets are
// the tail pass alone.
#pragma once
#include "skg_scene.cuh"

#include <vector>

namespace skg {

class WaveRunner {
public:
    WaveRunner() = default;
    WaveRunner(const WaveRunner&) = delete;
    WaveRunner& operator=(const WaveRunner&) = delete;
    ~WaveRunner();

    // Sizes the pool and job buffers (allocates; call outside stream capture).  pool packets,
    // ngroups peel-off groups at most per packet; grid_type decides whether path walks keep
    // checkpoints (grids whose FP32 walk resumes); walk_bytes, what the FP32 walks read of the (largest)
    // grid, with the pool whether the jobs are walked in spatial order.
    cudaError_t reserve(size_t pool, int ngroups, int grid_type, size_t walk_bytes);
    // Enqueues the reset of the pool and the first waves of a phase on stream s.  P holds the
    // staged tables; fits: the phase has no more packets than the pool; absorbs: some simulation tallies absorption in this phase or has several dust
    // components (its path walks then carry luminosities); nslots the slots whose DevGrid the traversal pass keeps in shared memory;
    // tree_walk the FP32 tree walk (TreeWalk) of tree grids; one_grid (host copy), when given with
    // nslots = 1, the grid the FP32 traversal kernels take as a kernel parameter instead.
    cudaError_t begin(const RunParams& P, int grid_type, int tree_walk, int precision, int nslots,
                      size_t npool, bool fits, int trav_blocks, bool absorbs, cudaStream_t s,
                      const DevGrid* one_grid = nullptr);
    // Waits for the enqueued waves and enqueues more until no packet is left; then records
    // `end` (if given) on the phase's stream.  timeout_ms < 0 waits without limit.
    cudaError_t finish(int timeout_ms, cudaEvent_t end, bool* timed_out);
    // What the waves of a phase are launched with.
    struct Phase {
        RunParams P{};
        int grid_type = 0, tree_walk = TW_ROPE, precision = 0, nslots = 1, trav_blocks = 0, npool = 0;
        bool one = false;              // a single-slot launch with its grid in g0
        DevGrid g0{};
        bool path_tau = false;
        int tail_div = 16;
        bool ckpt_on = true;           // path-walk checkpoints (environment variable SKG_CKPT=0: off)
        bool order_on = false;         // its jobs are walked in spatial order
        bool big_records = false;      // the walks' records of one direction exceed half the L2
    };
    const Phase& phase() const { return ph_; }
    // A captured begin() (pool reset and n waves) of the phase `was` was launched as a graph on stream s: the
    // waves that finish() adds are launched as the captured ones, whatever ran in between.
    void replayed(cudaStream_t s, int n, const Phase& was) {
        ph_ = was; pending_ = true; timed_ = tail_ran_ = false; stream_ = s; waves_ = n; tail_only_ = n == 0;
    }
    bool pending() const { return pending_; }
    int waves() const { return waves_; }
    cudaStream_t stream() const { return stream_; }
    size_t pool_capacity() const { return cap_pool_; }
    // changes when reserve() has moved a buffer (a captured launch then holds freed memory)
    int generation() const { return generation_; }
    // With timing on, each wave's launch and traversal passes are bracketed by events (not inside graph capture).
    bool timing = false;
    // Device time of the finished phase's launch passes and traversal passes (ms).
    cudaError_t times(float* event_ms, float* trav_ms) const;

    int estimate = 24;                // waves the next phase enqueues up front
    // the tail pass takes over when finish() finds at most npool / tail_div packets with work in the last
    // enqueued wave (0: waves to the end; the environment variable SKG_TAIL_DIV overrides it per phase)
    int tail_div = 16;

private:
    cudaError_t start(const RunParams& P, int grid_type, int tree_walk, int precision, int nslots, size_t npool, bool fits,
                      int trav_blocks, bool absorbs, cudaStream_t s, const DevGrid* one_grid);
    cudaError_t over(cudaError_t e);
    cudaError_t enqueue(int n);
    cudaError_t enqueue_tail();
    cudaError_t record_copied();

    Packet* pk_ = nullptr;
    int* lists_[2] = {nullptr, nullptr};   // [pool] free records, [pool] records at their interaction
                                      // point: a wave's, and the next wave's (which it fills)
    int2* rlist_ = nullptr;           // [pool] paths to re-walk
    float4* ckpt_ = nullptr;          // [pool][checkpoints][2] path-walk checkpoints
    size_t cap_ckpt_ = 0;
    size_t cap_pool_ = 0;
    int2* jobs_ = nullptr;
    double* jtau_ = nullptr;
    double* jL_ = nullptr;
    size_t cap_jobs_ = 0;
    int generation_ = 0;
    unsigned* bins_ = nullptr;        // [2][JOB_BINS] counts, [2][JOB_BINS] first places (walk order)
    uint2* order_ = nullptr;          // peel-off jobs in walk order; at its end, the path jobs' packets
    size_t cap_order_ = 0;
    bool order_on_ = false, big_records_ = false;   // of the phase that reserve() was called for
    static constexpr int NCTR = 2 * J_N + 1;
    unsigned* ctr_ = nullptr;         // [J_N (w & 1) + JobCount]: counters of wave w; [2 J_N]: last busy wave
    unsigned* h_ctr_ = nullptr;       // pinned copy read by finish()
    cudaEvent_t copied_ = nullptr;

    bool pending_ = false;
    cudaStream_t stream_ = nullptr;
    Phase ph_;
    int waves_ = 0;
    std::vector<cudaEvent_t> ev_;      // 3 per wave: before the launch pass, before the walks, after the ends and re-walks
    bool timed_ = false;               // the running phase records ev_
    bool tail_only_ = false;           // the phase is the tail pass alone
    bool tail_ran_ = false;            // the phase ended with the tail pass
    cudaEvent_t tail_ev_[2] = {nullptr, nullptr};
};

}  // namespace skg

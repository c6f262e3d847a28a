// engine_host.h -- host side of the batched engine (engine.cu).
#pragma once

#include "engine.h"
#include "hosono_gpu.h"

#include <string>
#include <vector>

namespace hosono {

struct TraceRec {
    int slot, stage, pass, nInner, nDetect;
    std::vector<unsigned char> inner, detect;  // nxt*nyt, i fastest
};

// Where an engine takes instance memory from: cudaMalloc by default, or a
// caller's pool (the server's arena).
struct DeviceAllocator {
    virtual ~DeviceAllocator() = default;
    virtual void* alloc(size_t bytes) = 0;  // nullptr when it does not fit
    virtual void release(void* p) = 0;
};

// Most listed cells (pass 1's failing cells, then the cells detect lowered in
// it) an instance may have for one cluster to take its stage; above it the
// kernel chain, which has the whole GPU for a pass but nine launches.  ms per
// step with 200 / 400 / 800 / 2000 / all in the cluster / none: blast 256^2 R=3
// from t=0.01 2.30 / 1.70 / 1.59 / 1.58 / - / 2.3, blast 512^2 R=3 from 0.015
// 3.31 / 3.31 / 3.31 / 5.02 / 5.16 / 3.47, blast 1024^2 R=2 from 0.01 4.00 / 4.00
// / 4.00 / 4.02 / 6.61 / 4.17, Orszag-Tang 256^2 R=2 from 0.3 3.08 / 3.08 / 3.00;
// a batch of 16 blasts, whose instances then share a stage's launches, 132 / 101
// / 92 / 92 ms.
constexpr int kClusterCells = 800;

// Blocks of a cluster: 16 >> class, 16 (where the GPU can place a cluster of this
// non-portable size, else 8) down to 2 by the number of stepping instances: as
// many as the GPU holds at once (a block takes an SM), half as many again at four.
// A pass of few cells is latency, so a smaller cluster loses less time on it than
// a second wave of clusters does.  us per step with 8 / 4 / 2 / 1 blocks / none,
// blasts of 40^2 R=2: 18 of them 742 / 769 / 977 / 1432 / 1527, 36: 1177 / 966 / 1148 /
// 1617 / 1899, 74: 2199 / 1724 / 1475 / 1942 / 2428, 256: 6884 / 4973 / 4140 / 4094 /
// 4781; 128 of 128^2: 9423 / 8230 / 7876 / 7978 / 8914; with 4 / 2 blocks 40 of 128^2
// to 512^2 10.3 / 12.6 ms, 64 of them 16.0 / 16.8, 64 of 64^2 2.35 / 2.21.
constexpr int kClusterClasses = 4;
inline int cluster_room(int cls, int sms) { return cls == 2 ? 3 * sms / 8 : sms / (16 >> cls); }
inline int cluster_class(int stepping, int sms) {
    int c = 0;
    while (c < kClusterClasses - 1 && stepping > cluster_room(c, sms)) c++;
    return c;
}

// Clusters of a launch of the last class: a power of two (no more than slots).
inline int clusters_for(int stepping, int slots) {
    int n = 64;
    while (n < stepping) n *= 2;
    return n < slots ? n : slots;
}

struct StepGraphs {
    cudaGraphExec_t advance = nullptr, run = nullptr, prof = nullptr;
    cudaGraphExec_t advRest = nullptr;  // advance without the first stage's set-up and pass 1
};

class Engine {
  public:
    Engine() = default;
    ~Engine();
    Engine(const Engine&) = delete;
    Engine& operator=(const Engine&) = delete;

    // capacity: instance slots and 32x8 tiles over all instances
    int init(int max_inst, int max_tiles, int fp_mode);
    // commit_tables = false defers the tile-list upload to commit_tables(),
    // so that many admissions or retirements rebuild it once
    int add(const hosono_params& p, const double* pv, const double* qw, int* slot, bool commit_tables = true);
    int remove(int slot, bool commit_tables = true);
    int commit_tables() { return upload_tables(); }
    // staging for upload/download of instances up to `cells` cells
    int reserve_staging(size_t cells);
    void set_allocator(DeviceAllocator* a) { alloc_ = a; }
    int upload(int slot, const double* U, const double* V);
    // U host -> device (Fortran-order AoS with guards), nothing else
    int upload_u(int slot, const double* U);
    // hosono_gpu_advance_host: U up, one step of dt, U (and V) down.  With
    // upload bands, U goes up in row bands on a second stream while the first
    // stage's pass 1 computes the tiles of the bands already landed.
    int advance_host(int slot, double dt, double* U, double* V);
    int download(int slot, double* U, double* V, int* scheme);
    // the initial state built on the device (hosono_ic_describe's output)
    int ic(int slot, const hosono_ic_desc& d, const double* xtab, const double* ytab);
    // output_writeHdf5's fields of the interior (13 double planes + scheme,
    // ordr; any may be null) and mean / max |div B|; allocates device scratch
    int diagnostics(int slot, double* fields, int* scheme, int* ordr, double* divb_l1, double* divb_linf);
    int set_time(int slot, double t, double tmax, int nstep, int nstepmax);
    // per slot (maxInst entries): nonzero holds the instance out of the
    // following run() launches, its state untouched (serving priority)
    int set_holds(const int* holds);
    // MOOD passes a stage may take before the instance stops with
    // HOSONO_EMOODCAP (cap <= 0: the proven bound R*nx*ny + 1)
    int set_mood_cap(int slot, int cap);
    int state(int slot, InstState* out);
    // cfl_computedt of one instance (dt to the host)
    int cfl(int slot, double* dt);
    // timeStep_advanceSolution of one instance with a host dt
    int advance(int slot, double dt);
    // time loop of every live instance: up to max_steps steps (<=0: until done)
    int run(int max_steps);
    // one step of every live instance with the pass-1 kernel bracketed by events
    int run_profiled_step(double* pass1_ms, int* pass1_launches);

    int tiles_of(const hosono_params& p) const;
    // ---- per-module form (the reference's stage modules one at a time on
    // one instance; modules.cuh).  Host arrays in the reference's Fortran
    // order; NULL pointers are skipped.
    int mod_set(int slot, const int* scheme, const int* rec, const int* recF);
    int mod_get(int slot, double* faceVals, double* fluxRaw, double* flux, double* Unew, int* scheme, int* rec,
                int* recF);
    int mod_reconstruct(int slot);
    int mod_getfluxes(int slot);
    int mod_flicd(int slot);
    int mod_update(int slot, double dt);
    int mod_detect(int slot, int* exit_mood_loop);
    int mod_bc(int slot, int which);
    int mod_bc_mood(int slot);
    int riemann(int slot, int n, const double* uL, const double* uR, int dir, double* F);
    int eigenvecs(int slot, int n, const double* V, int dir, int cons, double* L, double* R);

    // launch geometry of the kernels for radius R over this engine's tile capacity, as it is tuned now
    void launch_info(int R, int* pass1_grid, int* tile_grid_max) const { K_->launch_info(batch(), R, pass1_grid, tile_grid_max); }
    int live_count() const;
    size_t instance_bytes(const hosono_params& p) const;
    const hosono_params& params(int slot) const { return slots_[slot].p; }
    const Geo& geo(int slot) const { return slots_[slot].dev.geo; }
    const InstDev& dev(int slot) const { return slots_[slot].dev; }
    cudaStream_t stream() const { return s_; }
    int max_inst() const { return maxInst_; }
    int max_tiles() const { return maxTiles_; }
    int used_tiles() const {  // of every live slot, committed to the tile list or not
        int n = 0;
        for (const auto& sl : slots_) n += sl.live ? sl.ntiles : 0;
        return n;
    }

    // run() fails when an instance stopped with an error; when false, the
    // instance just ends (done, with its error code) and the others go on
    bool instance_errors_fatal = true;
    // per-slot states as of the end of the last run() (pinned host copy)
    const InstState* host_states() const { return h_st_; }
    // launch choices (hosono_tuning); changing them rebuilds the step graphs
    int set_tuning(const hosono_tuning& t);
    // time the candidate tunings on the live instances, apply the fastest
    int autotune(int trials, bool force, hosono_tune_report* rep);
    const hosono_tuning& tuning() const { return tune_; }
    // GP radii among the held instances (one pass-1 launch each per stage)
    int radii_held() const { return __builtin_popcount((unsigned)radii_); }
    bool use_graphs = true;
    bool trace = false;
    std::vector<TraceRec> traces;
    std::vector<int> traceStageBase;
    long long launches = 0;  // kernels launched (eager) or executed (graph, counted per node)

    int err = HOSONO_OK;
    std::string msg;
    int fail(int code, const char* fmt, ...);

  private:
    struct Slot {
        bool live = false;
        hosono_params p{};
        InstDev dev{};
        std::vector<void*> allocs;
        int ntiles = 0;
        ModBuf mod{};         // per-module buffers, allocated on first use
        void* modAlloc = nullptr;
    };
    int mod_ensure(int slot);
    int encode_tmaps(InstDev& dev);
    void drop_graphs();
    // a new engine's launch choices: the fastest on the benchmarked workloads
    // (TMA staging, dynamic tile schedule, two blocks per SM with one box each)
    hosono_tuning tune_{HOSONO_STAGE_TMA, HOSONO_SCHED_DYNAMIC, 2, HOSONO_LATER_KERNELS, 1, 0, 0, HOSONO_STAGE_CP_ASYNC};
    class Rec;
    friend class Rec;

    Batch batch() const;
    int upload_tables();
    void fit_clusters(int stepping);
    int fit_one(int slot);
    int going() const;
    int write_state_field(int slot, size_t offset, const void* src, size_t n);
    int write_state(int slot, const InstState& st);
    template <typename T>
    int write_field(int slot, T InstState::*field, T value) {
        const InstState* z = nullptr;
        return write_state_field(slot, (size_t)((const char*)&(z->*field) - (const char*)z), &value, sizeof(T));
    }
    // head = false leaves out the stage's set-up and pass 1 (run before, by the banded upload)
    int record_stage(Rec& r, int uin, int uout, cudaEvent_t ev0, cudaEvent_t ev1, bool head = true);
    template <class Cascade>
    int record_chain(Rec& r, const Batch& B, int uin, int uout, Cascade& cascade_body);
    enum StepForm { STEP_HOST_DT, STEP_WHOLE, STEP_TURN };
    int record_begin(Rec& r);
    int record_step(Rec& r, StepForm form, cudaGraphConditionalHandle run_cond, bool profile, bool first_head = true);
    int build_graph(cudaGraphExec_t StepGraphs::*which);
    int launch(cudaGraphExec_t g);
    int sync();
    int fetch();
    int check_errors();
    int errors();
    int trace_before_pass();
    int trace_snapshot();
    int trace_after_pass();

    void* dalloc(size_t bytes);
    void dfree(void* p);

    DeviceAllocator* alloc_ = nullptr;
    const KernelSet* K_ = nullptr;
    cudaStream_t s_ = nullptr;
    int maxInst_ = 0, maxTiles_ = 0;
    int sms_ = 148;
    int mcClass_ = 0, mcCount_ = 0;  // the launches' cluster_class and number of clusters (fit_clusters)
    int mcMany_ = 0;                 // the last class's number
    int radii_ = 0;       // BatchFlags::radii of the committed tile list
    int graphRadii_ = 0;  // radii_ when the step graphs were recorded (their pass-1 launches)
    InstDev* d_dev_ = nullptr;
    InstState* d_st_ = nullptr;
    int4* d_tiles_ = nullptr;
    int2* d_instTiles_ = nullptr;
    int* d_mcSlots_ = nullptr;  // Batch::mcSlots
    int2* d_actRange_ = nullptr;
    int* d_actInfo_ = nullptr;
    int2* d_casRange_ = nullptr;
    int* d_casInfo_ = nullptr;
    int* d_hold_ = nullptr;
    unsigned* d_gbar_ = nullptr;
    std::vector<int2> instTiles_;
    std::vector<int> hold_;  // d_hold_
    int* d_ntiles_ = nullptr;
    BatchFlags* d_flags_ = nullptr;
    Lists lists_{};
    BatchFlags* h_flags_ = nullptr;  // pinned
    InstState* h_st_ = nullptr;      // pinned mirror of d_st_ at rest
    double* staging_ = nullptr;
    size_t stagingCells_ = 0;
    int* schemeInt_ = nullptr;
    std::vector<Slot> slots_;
    std::vector<int4> tiles_;
    StepGraphs graphs_[kClusterClasses];
    cudaStream_t sCopy_ = nullptr;        // the banded upload's copy stream
    cudaEvent_t bandEv_[HOSONO_UPLOAD_BANDS_MAX + 1] = {};
    cudaEvent_t profEv_[6] = {};
    std::vector<long long> tracePassesSeen_;
    std::vector<std::vector<unsigned char>> snapInner_, snapLow_;
};

}  // namespace hosono

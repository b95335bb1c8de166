// The launchers of one numerics variant of the kernels, as a table the
// host runtime picks from at dgswe_create.
#pragma once

#include <cuda_runtime.h>

#include "device.hpp"

namespace dgswe {

// A stream beside a pass's own, of a higher priority, and the events that
// order the two: for the passes of a step graph and of the adjoint's sweeps,
// whose launches the host does not wait for (a 4,000-quad drying channel's
// run at N = 2 108.8 → 96.9 ms, a 50,000-quad coastal box's at N = 3 83.5 →
// 79.9). A multirate pass, launched call by call, gains nothing by it (the
// four event calls cost the host what the device saves: 167.5 ms in one
// stream, 169.6 with the side stream, for 40 coarse steps of 120,000 quads).
struct StageSide {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, sources = nullptr, ready = nullptr, done = nullptr;
};

// A side stream with the highest priority, so that its few long blocks start
// before the pass beside it fills the multiprocessors, and its events
inline cudaError_t make_side(StageSide& side) {
    if (side.stream) return cudaSuccess;
    int least = 0, greatest = 0;
    cudaError_t e = cudaDeviceGetStreamPriorityRange(&least, &greatest);
    for (cudaEvent_t* ev : {&side.fork, &side.sources, &side.ready, &side.done})
        if (e == cudaSuccess && !*ev) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&side.stream, cudaStreamNonBlocking, greatest);
    return e;
}

inline void free_side(StageSide& side) {
    for (cudaEvent_t ev : {side.fork, side.sources, side.ready, side.done})
        if (ev) cudaEventDestroy(ev);
    if (side.stream) cudaStreamDestroy(side.stream);
    side = StageSide{};
}

struct KernelSet {
    void (*face)(int n1, const DevTables&, const Physics&, const DevBuf& in, double* fh,
                 double* fhu, double* fhv, const StepCtl* ctl, int slot, const int* active,
                 cudaStream_t);
    void (*stage)(int n1, const DevTables&, const Physics&, const StageExtra&, const DevBuf& in,
                  const DevBuf& base, const DevBuf& out, const DevBuf& acc, const double* fh,
                  const double* fhu, const double* fhv, StepCtl* ctl, int slot, int mode,
                  int check_finite, const int* active, cudaStream_t);
    void (*finish)(int n1, const DevTables&, const Physics&, const DevBuf& acc,
                   const DevBuf& state, StepCtl* ctl, cudaStream_t);
    void (*dt)(int n1, const DevTables&, const Physics&, const DevBuf& q, const DtParams&,
               double* dt_el, StepCtl* ctl, const int* active, cudaStream_t);
    void (*velocity)(const DevBuf&, int64_t n, double h_min, cudaStream_t);
    // the adjoint of one stage (adjoint_kernels.cuh): the wet elements'
    // pass (`subcells` 0) or the listed subcell elements' (1)
    void (*stage_adjoint)(int n1, const DevTables&, const Physics&, const StageExtra&,
                          const DevBuf& in, const DevBuf& keep, const AdjStage&,
                          const StepCtl* ctl, int slot, int subcells, cudaStream_t);
    void (*face_adjoint)(int n1, const DevTables&, const Physics&, const DevBuf& in,
                         const AdjStage&, const StepCtl* ctl, int slot, cudaStream_t);
    // out = λ of the stage input; with `base` (the first stage), + base,
    // which is cleared
    void (*adjoint_combine)(const DevBuf& in, const AdjStage&, double* out_h, double* out_hu,
                            double* out_hv, double* const* base, int64_t n, double h_min,
                            cudaStream_t);
    void (*station_eval)(const double* h, const double* bed, const int64_t* node0,
                         const double* w, int n_stations, int nn, double* eta, cudaStream_t);
    void (*station_seed)(const double* eta, const double* obs, const int64_t* node0,
                         const double* w, int n_stations, int nn, double* lh, double* lbed,
                         cudaStream_t);
    // the run's clock, one thread per StepCtl of ctl[0..n)
    void (*step_begin)(StepCtl*, int n, cudaStream_t);
    void (*step_dt)(StepCtl*, int n, cudaStream_t);
    void (*step_end)(StepCtl*, int n, cudaStream_t);
    // a multirate pass (LtsPass): the listed faces, the listed elements'
    // stage (mode kModePost, or kModeAccumulate for the last stage), the
    // end of the listed elements' substeps
    void (*face_listed)(int n1, const DevTables&, const Physics&, const DevBuf& in, double* fh,
                        double* fhu, double* fhv, StepCtl* ctl, const LtsPass&, cudaStream_t);
    void (*stage_listed)(int n1, const DevTables&, const Physics&, const StageExtra&,
                         const DevBuf& in, const DevBuf& base, const DevBuf& out,
                         const DevBuf& acc, const double* fh, const double* fhu,
                         const double* fhv, StepCtl* ctl, int mode, const LtsPass&, cudaStream_t);
    void (*finish_listed)(int n1, const DevTables&, const Physics&, const DevBuf& acc,
                          const DevBuf& state, StepCtl* ctl, const LtsPass&, cudaStream_t);
    // per element: every node deeper than d0, d1, d2 (bits 0, 1, 2)
    void (*depth_flags)(const double* h, int64_t K, int nn, double d0, double d1, double d2,
                        uint8_t* flags, cudaStream_t);
    // the subcell elements of a step's three stage inputs, one list each,
    // for the stage adjoint's subcell pass
    void (*subcell_list)(const DevTables&, const Physics&, const double* h0, const double* h1,
                         const double* h2, const AdjStage&, int nn, cudaStream_t);
    // the point-implicit damping of `stage` over dt, rates frozen at `from`
    // (n values), and the stage's node velocities
    void (*implicit_damping)(const DevTables&, const Physics&, const DevBuf& stage,
                             const DevBuf& from, double dt, int64_t n, cudaStream_t);
    // a global stage's face fluxes of the listed interior edges and boundary
    // faces, without the node sources (a stage taken in parts as its input
    // arrives); the node sources alone (weather, relaxation band)
    void (*face_ready)(int n1, const DevTables&, const Physics&, const DevBuf& in, double* fh,
                       double* fhu, double* fhv, const StepCtl* ctl, int slot, const int* active,
                       const int32_t* edges, int64_t n_edges, const int32_t* bfaces,
                       int64_t n_bfaces, cudaStream_t);
    void (*node_sources)(const DevTables&, const Physics&, const DevBuf& in, const StepCtl* ctl,
                         int slot, cudaStream_t);
    // the smallest step over the listed elements; as `dt` without dt_el, it starts
    // from the +∞ of StepCtl's dt_bits and dt_up
    void (*dt_listed)(int n1, const DevTables&, const Physics&, const DevBuf& q, const DtParams&,
                      StepCtl* ctl, const int* active, const int32_t* list, int64_t n,
                      cudaStream_t);
    // the fixed-point tables from pair_hm, gdb and lift_scale
    // (DevTables::fx_*), where the variant has them
    void (*fixed_tables)(int n1, const DevTables&, FxPair* hm, FxPair* gdb, FxLimb* lift,
                         FxExp* exps, cudaStream_t);
    bool has_fixed;
    // face and stage as above, for a pass over the whole mesh, one after the
    // other: the node sources and the list of the elements with subcells run
    // on the side stream beside the face pass, those elements' stage there
    // beside the others'. `keep` (null: not) takes the combination and the
    // damped momentum (the adjoint's recomputation)
    void (*face_beside)(int n1, const DevTables&, const Physics&, const DevBuf& in, double* fh,
                        double* fhu, double* fhv, const StepCtl* ctl, int slot, const int* active,
                        cudaStream_t, const StageSide&);
    void (*stage_beside)(int n1, const DevTables&, const Physics&, const StageExtra&,
                         const DevBuf& in, const DevBuf& base, const DevBuf& out,
                         const DevBuf& acc, const double* fh, const double* fhu,
                         const double* fhv, StepCtl* ctl, int slot, int mode, int check_finite,
                         const int* active, const DevBuf& keep, cudaStream_t, const StageSide&);
    // the subcell interfaces' metrics (DevTables::sub_metric)
    void (*sub_metrics)(int n1, const DevTables&, const Physics&, double* out, cudaStream_t);
};

// kernels_fast.cu: FMA contraction, division-free Manning rate
const KernelSet* kernels_fast();
// kernels_exact.cu: every operation separately rounded, the reference's cube root
const KernelSet* kernels_exact();

// stage modes of the stage kernel
enum { kModeRhsOnly = 0, kModePost = 1, kModeAccumulate = 2 };

}  // namespace dgswe

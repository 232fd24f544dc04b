// One Lloyd fit: workspace, iteration body and device-resident loop state.
#pragma once

#include <memory>
#include <utility>
#include <vector>

#include "km_kernels.cuh"
#include "km_panel.cuh"
#include "km_step.cuh"

namespace kmc {

template <typename T, typename I>
struct FitParams {
    const T *X = nullptr;         // (d, n) feature-major samples, or (n, d) if x_rowmajor
    const T *w = nullptr;         // (n,) sample weights
    T *centroids = nullptr;       // (d, k) current centroids; overwritten
    T *new_centroids = nullptr;   // (d, k) result buffer
    I *labels = nullptr;          // (n,)
    int64_t n = 0, d = 0, k = 0;
    double tol = 0.0;
    int64_t max_iter = 0;
    int verbose = 0;
    kmc_print_fn print_fn = nullptr;
    void *print_ctx = nullptr;
    cudaStream_t stream = nullptr;
    int x_rowmajor = 0;           // X given as (n, d) C-contiguous
};

struct FitBase {
    // Optional CUDA-event timing of the assignment + accumulation phase.
    bool profiling = false;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> phase_events;
    int64_t launches = 0;

    virtual ~FitBase() {
        for (auto &e : phase_events) {
            cudaEventDestroy(e.first);
            cudaEventDestroy(e.second);
        }
    }
    int phase_time(double *total_ms, int64_t *count) {
        double tot = 0.0;
        for (auto &e : phase_events) {
            KMC_CUDA_TRY(cudaEventSynchronize(e.second));
            float ms = 0.f;
            KMC_CUDA_TRY(cudaEventElapsedTime(&ms, e.first, e.second));
            tot += ms;
        }
        *total_ms = tot;
        *count = (int64_t)phase_events.size();
        return KMC_OK;
    }
    // Enqueue iterations until the loop stops (batches of at most max_batch
    // iterations between host checks; <= 0 means unbounded growth).
    virtual int run(int64_t max_batch) = 0;
    // Enqueue exactly one iteration (no host synchronisation).  An iteration
    // that leaves clusters empty pauses the loop (km_step.cuh) until
    // enqueue_relocation; with `relocate` that is enqueued too.
    virtual int enqueue_iteration(bool relocate) = 0;
    virtual int enqueue_relocation() = 0;
    virtual int read_state(LoopState &out) = 0;
    // Device copy of the loop state (read by every kernel of an iteration).
    virtual const LoopState *device_state() const = 0;
    virtual int finalize(int64_t *n_iter_out, double *inertia_out) = 0;
    // The final pass without host synchronisation: the loop state and the
    // inertia total land in *state_out and *inertia_out (pinned host memory)
    // once the fit's stream reaches this point.
    virtual int finalize_enqueue(LoopState *state_out, double *inertia_out) = 0;
    // Limit (SM clocks; <= 0: the default) of the device-side waits: of the
    // tensor-core kernels and of a relocation's grid barriers.  With `stall`,
    // the next tensor-core assignment pass first waits on a barrier that
    // nothing completes, so that wait runs out (test of the timeout path).
    virtual int set_wait_limit(long long clocks, int stall) = 0;
    // Centroid-tile variant of a plain fit whose iterations run in the tiles
    // (the autotuner's choice unless set here); other fits ignore it.
    virtual int set_tile_variant(int v) {
        (void)v;
        return KMC_OK;
    }
    // Samples re-evaluated in exact arithmetic (mixed form): last pass and
    // total; and whether a device-side wait ran out.
    virtual int counters(int64_t *last, int64_t *total, int *device_error) = 0;
};

// Pinned host memory for a fit's loop state (two reads in flight) and inertia,
// with the events that mark the reads.  Allocating pinned memory costs more
// than a small fit, so freed slots are kept: at most kKeptHostSlots, given back
// by trim_pools().  Any thread may take and return them; a slot belongs to the
// device that was current when it was made.
struct HostSlot {
    LoopState st[2];
    double inertia;
};
constexpr int kKeptHostSlots = 16;
struct HostSlotRef {
    HostSlot *p = nullptr;  // null: no pinned memory was to be had
    cudaEvent_t ev[2] = {nullptr, nullptr};
    int device = -1;
    HostSlotRef();
    ~HostSlotRef();
    HostSlotRef(const HostSlotRef &) = delete;
    HostSlotRef &operator=(const HostSlotRef &) = delete;
};
void release_host_slots();

template <typename T, typename I>
struct PlainFit : FitBase {
    FitParams<T, I> prm;
    int64_t P = 1;  // private copies used internally
    Scratch ws;
    LoopState *state = nullptr;
    StepCtl *ctl = nullptr;
    T *hn = nullptr, *prev = nullptr, *sums = nullptr, *sizes = nullptr, *shifts = nullptr, *sq_dist = nullptr;
    double *sums_cp = nullptr, *sizes_cp = nullptr;  // float64 accumulators, zero between steps
    int64_t *empty_list = nullptr, *reloc = nullptr;  // (k); relocation lists (3 k)
    double *partials = nullptr, *dsum = nullptr;
    int64_t issued = 0;
    int host_done = 0;
    // hn holds the half norms of the centroids as the enqueued work leaves
    // them (plain forms; not after a relocation, nor across run() calls, between
    // which the caller may change its centroids)
    bool hn_current = false;
    bool split64 = false;  // float64 samples: labels, then sums (sums64.cu)
    int tile_variant = 0;  // autotuned centroid-tile width (fits that run in the tiles)
    Scratch xt;  // feature-major copy of a row-major X (forms that need one)
    static constexpr long long kWaitClocks = 4000000000LL;  // about two seconds
    long long wait_limit = kWaitClocks;

    int set_wait_limit(long long clocks, int stall) override {
        (void)stall;
        wait_limit = clocks > 0 ? clocks : kWaitClocks;
        return KMC_OK;
    }
    int counters(int64_t *last, int64_t *total, int *device_error) override;
    int set_tile_variant(int v) override {
        KMC_CHECK_ARG(v >= 0 && v <= 2, "tile variant must be 0, 1 or 2");
        tile_variant = v;
        return KMC_OK;
    }

    int init(const FitParams<T, I> &p);
    int enqueue_iteration(bool relocate) override;
    int enqueue_relocation() override;
    int read_state(LoopState &out) override;
    int run(int64_t max_batch) override;
    int run_pipelined(HostSlotRef &slot);
    int finalize(int64_t *n_iter_out, double *inertia_out) override;
    int finalize_enqueue(LoopState *state_out, double *inertia_out) override;
    const LoopState *device_state() const override { return state; }
    // Assignment + accumulation of one iteration (the fused Lloyd step);
    // reports the number of kernels it launched.
    virtual int step_assign_and_accumulate(const T *cur, int64_t *n_launches);
    // Labels against the final centroids (kmeans_lloyd_driver.hpp:372-386).
    virtual int final_assignment();
    // Cluster sums -> next centroids, shifts, stop rule (km_step.cuh).
    virtual int finish_step(int64_t *n_launches);
    FinishArgs<T> finish_args() const {
        const FitParams<T, I> &p = prm;
        return FinishArgs<T>{p.centroids, p.new_centroids, prev, sums, sizes, shifts,
                             uses_private_copies() ? hn : nullptr, empty_list, p.d, p.k, 1, state, ctl};
    }
    // Half norms of the current centroids, where neither the form's own
    // preparation nor the end of the iteration before made them.
    virtual int begin_step(int64_t *n_launches) {
        *n_launches = hn_current ? 0 : 1;
        if (hn_current) return KMC_OK;
        return launch_half_norm<T>(prm.centroids, hn, prm.d, prm.k, prm.stream, state);
    }
    // Whether the step accumulates into the driver's float64 private copies
    // (the mixed forms keep their own sums).
    virtual bool uses_private_copies() const { return true; }
    // Whether the form reads a row-major X itself (else init makes a
    // feature-major copy).
    virtual bool reads_rowmajor() const { return false; }
    // The samples as the inertia and relocation kernels read them: element
    // (f, i) at x[f * fs + i * ss].
    virtual void x_view(const T **x, int64_t *fs, int64_t *ss) const {
        *x = prm.X;
        *fs = prm.n;
        *ss = 1;
    }
    // Row-major copy of the last assignment's centroids beside a row-major view,
    // or null.
    virtual const T *c_rows(int64_t *stride) const {
        *stride = 0;
        return nullptr;
    }
};

// Mixed tensor-core form (kernels_mixed.cu); float32 data only.
template <typename T, typename I>
int make_mixed_fit(const FitParams<T, I> &p, int form, std::unique_ptr<FitBase> *out);
// Whether the mixed form takes n_features = d and n_clusters = k.
bool mixed_fit_supported(int64_t d, int64_t k);
// Mixed-form variant (10 stages + packed rows in flight per lane of the sums, 0
// where there are none): forced for every fit created afterwards (-1: the
// autotuner's choice again), and a session's choice (-1: not a mixed fit).
int force_mixed_variant(int code);
// Fits created on this thread while on use cached variant choices or the
// default and never time variants (the request server).
void mixed_tuning_lookup_only(bool on);
// The packed fixed-point term of v at scale 2^shift (host copy of the
// device's packing, for tests).
int pack_fixed_term(float v, int shift);
int mixed_variant_of(FitBase *fit, int *code);

}  // namespace kmc

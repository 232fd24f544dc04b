// Lloyd driver: the host loop of driver_lloyd (src/kmeans_lloyd_driver.hpp:
// 21-431), re-designed so that the GPU decides when to stop.
//
// Reference loop, per iteration (kmeans_lloyd_driver.hpp:83-354):
//   half norms -> zero private copies -> fused step -> reduce copies (sums,
//   sizes, empty list) -> [verbose inertia print] -> host reads n_empty ->
//   [relocate empty clusters] -> divide -> shifts -> host reads shift sum ->
//   swap -> ++n_iter;   while (n_iter < max_iter && shift_sum > tol).
//
// Here every kernel of an iteration is guarded by a device-resident loop
// state: the end of an iteration (km_step.cuh) sets `done` once the
// reference's condition fails, after which the remaining enqueued kernels
// return immediately, and pauses the loop when a cluster is empty, until the
// host has launched the relocation.  The host therefore enqueues iterations in batches and reads the
// state once per batch instead of twice per iteration.  Centroid buffers do
// not ping-pong: new centroids overwrite the current buffer at the end of an
// iteration, so one iteration body works for every iteration (and can be
// captured once into a CUDA graph).  The convergence total and the final inertia are summed
// in float64.
#include <algorithm>
#include <cstdarg>
#include <memory>
#include <mutex>
#include <vector>

#include "km_kernels.cuh"
#include "km_fit.cuh"

namespace kmc {

namespace {
struct KeptSlot {
    HostSlot *p;
    cudaEvent_t ev[2];
    int device;
};
std::mutex g_slots_mutex;
std::vector<KeptSlot> g_slots;

void free_slot(const KeptSlot &k) {
    for (cudaEvent_t e : k.ev)
        if (e != nullptr) cudaEventDestroy(e);
    if (k.p != nullptr) cudaFreeHost(k.p);
}
}  // namespace

HostSlotRef::HostSlotRef() {
    if (cudaGetDevice(&device) != cudaSuccess) return;
    {
        std::lock_guard<std::mutex> lock(g_slots_mutex);
        for (size_t q = 0; q < g_slots.size(); ++q)
            if (g_slots[q].device == device) {
                p = g_slots[q].p;
                ev[0] = g_slots[q].ev[0];
                ev[1] = g_slots[q].ev[1];
                g_slots.erase(g_slots.begin() + (long)q);
                return;
            }
    }
    KeptSlot k{nullptr, {nullptr, nullptr}, device};
    void *mem = nullptr;
    if (cudaHostAlloc(&mem, sizeof(HostSlot), cudaHostAllocDefault) == cudaSuccess)
        k.p = static_cast<HostSlot *>(mem);
    bool ok = k.p != nullptr;
    for (cudaEvent_t &e : k.ev)
        ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        free_slot(k);
        cudaGetLastError();  // the caller goes on without
        return;
    }
    p = k.p;
    ev[0] = k.ev[0];
    ev[1] = k.ev[1];
}

HostSlotRef::~HostSlotRef() {
    if (p == nullptr) return;
    const KeptSlot k{p, {ev[0], ev[1]}, device};
    {
        std::lock_guard<std::mutex> lock(g_slots_mutex);
        if (g_slots.size() < (size_t)kKeptHostSlots) {
            g_slots.push_back(k);
            return;
        }
    }
    free_slot(k);
}

void release_host_slots() {
    std::vector<KeptSlot> drop;
    {
        std::lock_guard<std::mutex> lock(g_slots_mutex);
        drop.swap(g_slots);
    }
    for (const KeptSlot &k : drop) free_slot(k);
}

template <typename T, typename I>
int PlainFit<T, I>::init(const FitParams<T, I> &p) {
    prm = p;
    const int64_t n = p.n, d = p.d, k = p.k;
    KMC_CHECK_ARG(n >= 0 && d >= 0 && k >= 0, "negative array dimension");
    // Small sums get one float64 copy per CTA of the fused step, filled with
    // fire-and-forget global reductions; shared-memory float64 atomics would
    // be compare-and-swap loops on the critical path.  float64 samples are
    // summed in a fixed order (bit-reproducible centroids): by sums64.cu, or by
    // the fused tiles with a copy per CTA up to 256 MiB of copies.
    split64 = sizeof(T) == 8 && panel::fits(d) && sums64_fits(d, k);
    if (!uses_private_copies()) {
        P = 1;
    } else if (split64) {
        P = sums64_copies(n, d, k);
    } else if (sizeof(T) == 8) {
        const int64_t per_copy = 8 * (d + 1) * std::max<int64_t>(k, 1);
        P = std::max<int64_t>(1, std::min<int64_t>(2 * (int64_t)num_sms(),
                                                   (int64_t(256) << 20) / per_copy));
    } else if ((d + 1) * k <= 8192) {
        // With few clusters more copies, so that about 32 addresses per SM and
        // feature share the reductions (each warp adds into a copy of its own; 1M x
        // 8, k = 8: 152 copies 61 us, 608 41; 5M x 2, 4: 300, 1216 103).
        const int64_t m = panel::fits(d) ? std::max<int64_t>(1, std::min<int64_t>(8, 32 / std::max<int64_t>(k, 1))) : 2;
        P = (int64_t)num_sms() * m;
        if (panel::fits(d)) P = std::max<int64_t>(num_sms(), std::min<int64_t>(P, n / 512));
    } else {
        // Large sums: a few copies, which every iteration reads and clears
        // (1M x 32, k = 250: 1 copy 482 us, 4 363, 16 356, 152 356; 200,000 x
        // 64, 300: 240, 213, 208, 205; x 128, 400: 702, 692, 686, 688).
        P = (d + 1) * k <= 65536 ? 16 : (d + 1) * k <= 524288 ? 4 : 1;
        P = std::max<int64_t>(1, std::min<int64_t>(P, n / 4096));
    }
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t o = off;
        off += align256(bytes);
        return o;
    };
    const size_t o_state = take(sizeof(LoopState));
    const size_t o_ctl = take(sizeof(StepCtl));
    const size_t o_scp = take(sizeof(double) * P * d * k);
    const size_t o_zcp = take(sizeof(double) * P * k);
    const size_t o_hn = take(sizeof(T) * k);
    const size_t o_prev = take(sizeof(T) * d * k);
    const size_t o_sums = take(sizeof(T) * d * k);
    const size_t o_sizes = take(sizeof(T) * k);
    const size_t o_shifts = take(sizeof(T) * k);
    const size_t o_sq = take(sizeof(T) * n);
    const size_t o_list = take(sizeof(int64_t) * k);
    const size_t o_rel = take(sizeof(int64_t) * 3 * k);
    const size_t o_part = take(sizeof(double) * sum_partials_size());
    const size_t o_dsum = take(sizeof(double) * 2);
    KMC_TRY(ws.alloc(off, p.stream));
    // the tile kernels' width for this (d, k, dtype), where they are used
    if (uses_private_copies() && (!panel::fits(d) || (sizeof(T) == 8 && !split64)))
        KMC_TRY(tune_fit_variant<T>(d, k, p.stream, &tile_variant));
    if (p.x_rowmajor && !reads_rowmajor()) {
        KMC_TRY(xt.alloc(sizeof(T) * (size_t)n * (size_t)d, p.stream));
        if (sizeof(T) == 4)
            KMC_TRY(kmc_transpose_f32(reinterpret_cast<const float *>(p.X), xt.as<float>(), n, d,
                                      reinterpret_cast<kmc_stream_t>(p.stream)));
        else
            KMC_TRY(kmc_transpose_f64(reinterpret_cast<const double *>(p.X), xt.as<double>(), n,
                                      d, reinterpret_cast<kmc_stream_t>(p.stream)));
        prm.X = xt.as<T>();
        prm.x_rowmajor = 0;
    }
    char *b = ws.as<char>();
    state = reinterpret_cast<LoopState *>(b + o_state);
    ctl = reinterpret_cast<StepCtl *>(b + o_ctl);
    sums_cp = reinterpret_cast<double *>(b + o_scp);
    sizes_cp = reinterpret_cast<double *>(b + o_zcp);
    hn = reinterpret_cast<T *>(b + o_hn);
    prev = reinterpret_cast<T *>(b + o_prev);
    sums = reinterpret_cast<T *>(b + o_sums);
    sizes = reinterpret_cast<T *>(b + o_sizes);
    shifts = reinterpret_cast<T *>(b + o_shifts);
    sq_dist = reinterpret_cast<T *>(b + o_sq);
    empty_list = reinterpret_cast<int64_t *>(b + o_list);
    reloc = reinterpret_cast<int64_t *>(b + o_rel);
    partials = reinterpret_cast<double *>(b + o_part);
    dsum = reinterpret_cast<double *>(b + o_dsum);
    // the control block and the private copies start at zero; each iteration
    // leaves them so
    KMC_CUDA_TRY(cudaMemsetAsync(ctl, 0, uses_private_copies() ? o_hn - o_ctl : o_scp - o_ctl,
                                 p.stream));

    LoopState h{};
    h.done = 0;
    h.n_iter = 0;
    h.max_iter = p.max_iter;
    const T tol_t = (T)p.tol;
    h.tol = (double)tol_t;
    // while (n_iter < max_iter && shift_sum > tol) with shift_sum = +inf
    // initially (kmeans_lloyd_driver.hpp:78, 83).
    if (!(0 < p.max_iter && pos_inf<T>() > tol_t)) h.done = 1;
    host_done = h.done;
    KMC_CUDA_TRY(cudaMemcpyAsync(state, &h, sizeof(h), cudaMemcpyHostToDevice, p.stream));
    return KMC_OK;
}

template <typename T, typename I>
int PlainFit<T, I>::enqueue_iteration(bool relocate) {
    const FitParams<T, I> &p = prm;
    const int64_t n = p.n, d = p.d, k = p.k;
    cudaStream_t s = p.stream;
    // kmeans_lloyd_driver.hpp:86-111
    int64_t begin_launches = 0, step_launches = 0, finish_launches = 0;
    KMC_TRY(begin_step(&begin_launches));
    // kmeans_lloyd_driver.hpp:124-143
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (profiling) {
        KMC_CUDA_TRY(cudaEventCreate(&e0));
        KMC_CUDA_TRY(cudaEventCreate(&e1));
        KMC_CUDA_TRY(cudaEventRecord(e0, s));
    }
    KMC_TRY(step_assign_and_accumulate(p.centroids, &step_launches));
    if (profiling) {
        KMC_CUDA_TRY(cudaEventRecord(e1, s));
        phase_events.emplace_back(e0, e1);
    }
    // kmeans_lloyd_driver.hpp:155-170, 317-353
    KMC_TRY(finish_step(&finish_launches));
    launches += begin_launches + step_launches + finish_launches;
    if (p.verbose) {
        // kmeans_lloyd_driver.hpp:179-197: inertia of the *undivided* sums
        // (before a relocation moves any)
        const T *xv = nullptr;
        int64_t xfs = 0, xss = 0;
        x_view(&xv, &xfs, &xss);
        KMC_TRY(launch_inertia<T, I>(xv, p.w, sums, p.labels, sq_dist, n, d, k, s, xfs, xss));
        KMC_TRY(launch_sum_f64<T>(sq_dist, n, partials, dsum, s));
        launches += 3;
    }
    hn_current = true;
    if (relocate) KMC_TRY(enqueue_relocation());
    ++issued;
    return KMC_OK;
}

// kmeans_lloyd_driver.hpp:217-312, of an iteration that left clusters empty
template <typename T, typename I>
int PlainFit<T, I>::enqueue_relocation() {
    const FitParams<T, I> &p = prm;
    const T *xv = nullptr;
    int64_t xfs = 0, xss = 0, crs = 0;
    x_view(&xv, &xfs, &xss);
    const T *cr = c_rows(&crs);
    const RelocArgs<T, I> ra{p.centroids, p.new_centroids, prev, sums, sizes, shifts, empty_list,
                             reloc, reloc + p.k, reloc + 2 * p.k, xv, p.w, p.labels, sq_dist, p.n,
                             p.d, p.k, xfs, xss, cr, crs, wait_limit, state, ctl};
    KMC_TRY((launch_relocation<T, I>(ra, p.stream)));
    hn_current = false;
    ++launches;
    return KMC_OK;
}

template <typename T, typename I>
int PlainFit<T, I>::step_assign_and_accumulate(const T *cur, int64_t *n_launches) {
    const FitParams<T, I> &p = prm;
    *n_launches = 1;
    if constexpr (sizeof(T) == 8) {
        if (split64) {
            *n_launches = 2;
            KMC_TRY((launch_assignment<T, I>(p.X, cur, hn, p.labels, p.n, p.d, p.k, p.stream,
                                             state)));
            return launch_sums64<I>(p.X, p.w, p.labels, sums_cp, sizes_cp, p.n, p.d, p.k, P,
                                    p.stream, state);
        }
    }
    return launch_fused_step<T, I, double>(p.X, p.w, cur, hn, p.labels, sums_cp, sizes_cp, p.n,
                                           p.d, p.k, P, p.stream, state, tile_variant);
}

template <typename T, typename I>
int PlainFit<T, I>::read_state(LoopState &out) {
    KMC_CUDA_TRY(cudaMemcpyAsync(&out, state, sizeof(LoopState), cudaMemcpyDeviceToHost,
                                 prm.stream));
    KMC_CUDA_TRY(cudaStreamSynchronize(prm.stream));
    host_done = out.done;
    return check_device_error(out);
}

template <typename T, typename I>
int PlainFit<T, I>::counters(int64_t *last, int64_t *total, int *device_error) {
    LoopState h{};
    KMC_CUDA_TRY(cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, prm.stream));
    KMC_CUDA_TRY(cudaStreamSynchronize(prm.stream));
    if (last) *last = 0;
    if (total) *total = 0;
    if (device_error) *device_error = h.err != 0;
    return KMC_OK;
}

// Two batches of iterations are in flight: while one runs, the host waits for
// the loop state at the end of the one before, so the device never waits for
// the host (reading the state after each of batches of 1, 2, 4, ... iterations
// left it idle for 15 to 30 us each; 50,000 x 14, 20 iterations: 742 -> 706 us,
// 300,000 x 100 bf16, 6 iterations: 1357 -> 1311).  Batches stay small: what is enqueued
// behind the end of the loop, or behind a pause, still costs a few launches
// that return at once.
template <typename T, typename I>
int PlainFit<T, I>::run_pipelined(HostSlotRef &slot) {
    constexpr int64_t kMaxBatch = 4;
    const FitParams<T, I> &p = prm;
    LoopState h{};
    if (issued == 0) {
        h.done = host_done;  // nothing has run: as init left it
    } else {
        KMC_TRY(read_state(h));
    }
    // iterations of the batches in flight, oldest first
    int64_t in_flight[2] = {0, 0};
    int first = 0, flying = 0;
    auto send = [&](int64_t m) -> int {
        for (int64_t t = 0; t < m; ++t) KMC_TRY(enqueue_iteration(false));
        const int q = (first + flying) & 1;
        KMC_CUDA_TRY(cudaMemcpyAsync(&slot.p->st[q], state, sizeof(LoopState),
                                     cudaMemcpyDeviceToHost, p.stream));
        ++flying;  // a copy into the slot is under way, whatever follows
        in_flight[q] = m;
        KMC_CUDA_TRY(cudaEventRecord(slot.ev[q], p.stream));
        return KMC_OK;
    };
    auto receive = [&]() -> int {
        KMC_CUDA_TRY(cudaEventSynchronize(slot.ev[first]));
        h = slot.p->st[first];
        first ^= 1;
        --flying;
        return KMC_OK;
    };
    auto loop = [&]() -> int {
        int64_t batch = 1;
        if (h.done == kPaused) {
            KMC_TRY(enqueue_relocation());
            KMC_TRY(send(0));
            KMC_TRY(receive());
            KMC_TRY(check_device_error(h));
        }
        while (true) {
            while (flying < 2 && !h.done) {
                int64_t ahead = h.n_iter;
                for (int q = 0; q < flying; ++q) ahead += in_flight[(first + q) & 1];
                const int64_t m = std::min(batch, p.max_iter - ahead);
                if (m <= 0) break;
                KMC_TRY(send(m));
                batch = std::min(2 * batch, kMaxBatch);
            }
            if (flying == 0) return KMC_OK;
            KMC_TRY(receive());
            KMC_TRY(check_device_error(h));
            if (h.done == 0) continue;
            // nothing behind the end or the pause did anything
            while (flying > 0) KMC_TRY(receive());
            if (h.done != kPaused) return check_device_error(h);
            KMC_TRY(enqueue_relocation());  // ends the paused iteration
            ++h.n_iter;
            h.done = 0;
            batch = 1;
            if (h.n_iter >= p.max_iter) KMC_TRY(send(0));
        }
    };
    const int rc = loop();
    host_done = h.done;
    // no copy into the slot outlives this call
    if (flying > 0) cudaStreamSynchronize(p.stream);
    return rc;
}

template <typename T, typename I>
int PlainFit<T, I>::run(int64_t max_batch) {
    const FitParams<T, I> &p = prm;
    hn_current = false;
    if (!p.verbose && max_batch <= 0) {
        HostSlotRef slot;
        if (slot.p != nullptr) return run_pipelined(slot);
    }
    LoopState h{};
    KMC_TRY(read_state(h));
    int64_t batch = 1;
    while (h.done == kPaused || (!h.done && h.n_iter < p.max_iter)) {
        // an iteration that left clusters empty paused the loop; the rest of
        // its batch did nothing
        if (h.done == kPaused) {
            KMC_TRY(enqueue_relocation());
            batch = 1;
        }
        const int64_t left = p.max_iter - h.n_iter - (h.done == kPaused ? 1 : 0);
        int64_t m = p.verbose ? 1 : std::min<int64_t>(batch, left);
        if (p.verbose && h.done == kPaused) m = 0;
        if (max_batch > 0) m = std::min<int64_t>(m, max_batch);
        const bool fresh = h.done != kPaused;
        for (int64_t t = 0; t < m; ++t) KMC_TRY(enqueue_iteration(false));
        KMC_TRY(read_state(h));
        if (p.verbose && p.print_fn != nullptr && fresh) {
            double tot = 0.0;
            KMC_CUDA_TRY(cudaMemcpy(&tot, dsum, sizeof(double), cudaMemcpyDeviceToHost));
            char line[128];
            // kmeans_lloyd_driver.hpp:199-204
            snprintf(line, sizeof(line), "Iteration: %lld Inertia: %.9g",
                     (long long)(h.done == kPaused ? h.n_iter : h.n_iter - 1), (double)(T)tot);
            p.print_fn(line, p.print_ctx);
        }
        if (batch < 64) batch *= 2;
    }
    return KMC_OK;
}

template <typename T, typename I>
int PlainFit<T, I>::finalize_enqueue(LoopState *state_out, double *inertia_out) {
    const FitParams<T, I> &p = prm;
    const int64_t n = p.n, d = p.d, k = p.k;
    cudaStream_t s = p.stream;
    // kmeans_lloyd_driver.hpp:360-418: final assignment and inertia against
    // the final centroids.
    KMC_TRY(final_assignment());
    const T *xv = nullptr;
    int64_t xfs = 0, xss = 0, crs = 0;
    x_view(&xv, &xfs, &xss);
    const T *cr = c_rows(&crs);
    KMC_TRY(launch_inertia<T, I>(xv, p.w, p.centroids, p.labels, sq_dist, n, d, k, s, xfs, xss, cr,
                                 crs));
    KMC_TRY(launch_sum_f64<T>(sq_dist, n, partials, dsum, s));
    launches += 5;
    if (p.new_centroids != p.centroids && d * k > 0)
        KMC_CUDA_TRY(cudaMemcpyAsync(p.new_centroids, p.centroids, sizeof(T) * d * k,
                                     cudaMemcpyDeviceToDevice, s));
    KMC_CUDA_TRY(cudaMemcpyAsync(inertia_out, dsum, sizeof(double), cudaMemcpyDeviceToHost, s));
    KMC_CUDA_TRY(cudaMemcpyAsync(state_out, state, sizeof(LoopState), cudaMemcpyDeviceToHost, s));
    return KMC_OK;
}

template <typename T, typename I>
int PlainFit<T, I>::finalize(int64_t *n_iter_out, double *inertia_out) {
    LoopState h{};
    double tot = 0.0;
    {
        HostSlotRef slot;  // pinned, so that the second copy does not wait for the first
        LoopState *hs = slot.p != nullptr ? &slot.p->st[0] : &h;
        double *ts = slot.p != nullptr ? &slot.p->inertia : &tot;
        const int rc = finalize_enqueue(hs, ts);
        KMC_CUDA_TRY(cudaStreamSynchronize(prm.stream));
        KMC_TRY(rc);
        h = *hs;
        tot = *ts;
    }
    host_done = h.done;
    KMC_TRY(check_device_error(h));
    if (n_iter_out) *n_iter_out = h.n_iter;
    if (inertia_out) *inertia_out = tot;
    return KMC_OK;
}

template <typename T, typename I>
int PlainFit<T, I>::finish_step(int64_t *n_launches) {
    const FitParams<T, I> &p = prm;
    const PlainSums src{sums_cp, sizes_cp, p.d * p.k, p.k, P};
    return launch_reduce_and_finish<T>(src, P, finish_args(), n_launches, p.stream);
}

template <typename T, typename I>
int PlainFit<T, I>::final_assignment() {
    const FitParams<T, I> &p = prm;
    KMC_TRY(launch_half_norm<T>(p.centroids, hn, p.d, p.k, p.stream));
    return launch_assignment<T, I>(p.X, p.centroids, hn, p.labels, p.n, p.d, p.k, p.stream,
                                   nullptr, tile_variant);
}

template struct PlainFit<float, int32_t>;
template struct PlainFit<float, int64_t>;
template struct PlainFit<double, int32_t>;
template struct PlainFit<double, int64_t>;

}  // namespace kmc

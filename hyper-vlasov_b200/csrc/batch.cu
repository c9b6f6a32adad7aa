// Batched runs: many independent nuclei advanced together on one GPU.
//
// The reference runs one nucleus per process.  A batch holds several float
// contexts (each its own nucleus, test-particle count, grid and parameters,
// created with hv_ctx_create) and advances them step by step together: per
// step, every instance's particle step, smoothing and Skyrme potential run as
// parallel branches on per-instance streams, then the Coulomb solves run as a
// few cooperative launches ("waves") that each solve several instances at once
// (k_sor_fast in its batched form: every block looks up its instance, and
// barriers, residual sums and the boundary exchange stay within the
// instance), then every instance's forces.  Chunks of steps are captured into
// one CUDA graph and replayed.  The results of every instance are those of
// its own hv_run on the fused path, up to float rounding.
//
// How many blocks each instance's solve uses is a plan choice: fewer blocks
// pack more instances into a wave, more blocks make each solve faster.
// hv_batch_plan takes a cap; hv_batch_autotune times candidate caps on trial
// steps and keeps the fastest, then the particle step's block size.  The cap
// shapes the sweeps only: direct solves (k_poisson.cu), the float default,
// share the SMs by their work.
#include <algorithm>
#include <cstring>
#include <numeric>
#include <vector>

#include "hv_internal.h"

using namespace hv;

struct hv_batch {
    int device = 0;
    int sm_count = 0;
    cudaStream_t stream = nullptr;
    std::vector<hv_ctx *> ctx;
    std::vector<cudaStream_t> streams;
    std::vector<cudaEvent_t> ev_a, ev_c;  // per instance: end of its phase A / C
    cudaEvent_t ev_fork_a = nullptr, ev_fork_c = nullptr;
    std::vector<SorWave> waves;
    std::vector<int> blocks;              // blocks of each instance's solve
    std::vector<unsigned> gen;            // each context's plan_gen that the waves were built from
    int cap = -1;                         // SOR block cap of the current plan (0: own plans)
    cudaGraphExec_t graph = nullptr;
    cudaGraphExec_t tail_graph = nullptr; // a run's last, shorter chunk, once its length has come twice
    int tail_len = 0;
    int chunk = 8;
    cudaEvent_t ev_done[2] = {nullptr, nullptr};  // end of a chunk's copies, by the chunk's parity
    char *staging = nullptr;              // pinned: two chunks' rows, iteration rings and status words, and
                                          // the instances' seed words
};

namespace {

void drop_graph(hv_batch *b) {
    if (b->graph) cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
    if (b->tail_graph) cudaGraphExecDestroy(b->tail_graph);
    b->tail_graph = nullptr;
    b->tail_len = 0;
}

// One step of every instance, on the batch stream with per-instance branches.
hv_status enqueue_batch_step(hv_batch *b) {
    const int n = (int)b->ctx.size();
    HV_CUDA(cudaEventRecord(b->ev_fork_a, b->stream));
    for (int i = 0; i < n; i++) {
        HV_CUDA(cudaStreamWaitEvent(b->streams[i], b->ev_fork_a, 0));
        HV_TRY(fused_batch_phase_a(b->ctx[i], b->streams[i]));
        HV_CUDA(cudaEventRecord(b->ev_a[i], b->streams[i]));
        HV_CUDA(cudaStreamWaitEvent(b->stream, b->ev_a[i], 0));
    }
    for (const SorWave &w : b->waves) HV_TRY(sor_wave_launch(w, b->stream));
    HV_CUDA(cudaEventRecord(b->ev_fork_c, b->stream));
    for (int i = 0; i < n; i++) {
        HV_CUDA(cudaStreamWaitEvent(b->streams[i], b->ev_fork_c, 0));
        HV_TRY(fused_batch_phase_c(b->ctx[i], b->streams[i]));
        HV_CUDA(cudaEventRecord(b->ev_c[i], b->streams[i]));
        HV_CUDA(cudaStreamWaitEvent(b->stream, b->ev_c[i], 0));
    }
    return HV_OK;
}

hv_status enqueue_batch_steps(hv_batch *b, int k) {
    for (int s = 0; s < k; s++) HV_TRY(enqueue_batch_step(b));
    return HV_OK;
}

// k steps captured as a graph (null when that is not possible here).
cudaGraphExec_t capture_steps(hv_batch *b, int k) {
    cudaGraph_t gr = nullptr;
    cudaGraphExec_t ex = nullptr;
    if (cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        const hv_status es = enqueue_batch_steps(b, k);
        const cudaError_t ce = cudaStreamEndCapture(b->stream, &gr);
        if (es != HV_OK || ce != cudaSuccess || !gr || cudaGraphInstantiate(&ex, gr, 0) != cudaSuccess) ex = nullptr;
        if (gr) cudaGraphDestroy(gr);
        cudaGetLastError();
    }
    return ex;
}

void release_waves(hv_batch *b) {
    for (SorWave &w : b->waves) sor_wave_release(w);
    b->waves.clear();
}

}  // namespace

extern "C" {

hv_status hv_batch_create(int n, hv_ctx *const *ctxs, hv_batch **out) {
    if (!out || n < 1 || !ctxs) return HV_ERR_BAD_ARG;
    *out = nullptr;
    for (int i = 0; i < n; i++) {
        if (!ctxs[i]) return HV_ERR_BAD_ARG;
        if (ctxs[i]->prec != HV_F32 || ctxs[i]->device != ctxs[0]->device) return HV_ERR_UNSUPPORTED;
        for (int j = 0; j < i; j++)
            if (ctxs[j] == ctxs[i]) return HV_ERR_BAD_ARG;
    }
    hv_batch *b = new hv_batch();
    b->device = ctxs[0]->device;
    b->sm_count = ctxs[0]->sm_count;
    b->ctx.assign(ctxs, ctxs + n);
    auto fail = [&](hv_status s) {
        hv_batch_destroy(b);
        return s;
    };
    if (cudaSetDevice(b->device) != cudaSuccess) return fail(HV_ERR_CUDA);
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(HV_ERR_CUDA);
    for (cudaEvent_t *e : {&b->ev_fork_a, &b->ev_fork_c, &b->ev_done[0], &b->ev_done[1]})
        if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) return fail(HV_ERR_CUDA);
    b->streams.resize(n);
    b->ev_a.resize(n);
    b->ev_c.resize(n);
    for (int i = 0; i < n; i++) {
        if (cudaStreamCreateWithFlags(&b->streams[i], cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&b->ev_a[i], cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&b->ev_c[i], cudaEventDisableTiming) != cudaSuccess)
            return fail(HV_ERR_CUDA);
    }
    for (hv_ctx *c : b->ctx) {
        hv_status st = fused_batch_ready(c);
        if (st != HV_OK) return fail(st);
    }
    hv_status st = hv_batch_plan(b, 0);
    if (st != HV_OK) return fail(st);
    *out = b;
    return HV_OK;
}

hv_status hv_batch_destroy(hv_batch *b) {
    if (!b) return HV_OK;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    drop_graph(b);
    release_waves(b);
    if (b->staging) cudaFreeHost(b->staging);
    for (cudaStream_t s : b->streams)
        if (s) cudaStreamDestroy(s);
    for (cudaEvent_t e : b->ev_a)
        if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : b->ev_c)
        if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : {b->ev_fork_a, b->ev_fork_c, b->ev_done[0], b->ev_done[1]})
        if (e) cudaEventDestroy(e);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return HV_OK;
}

hv_status hv_batch_plan(hv_batch *b, int sor_max_blocks) {
    if (!b || sor_max_blocks < 0) return HV_ERR_BAD_ARG;
    HV_CUDA(cudaSetDevice(b->device));
    HV_CUDA(cudaStreamSynchronize(b->stream));
    drop_graph(b);
    release_waves(b);
    b->gen.clear();
    const int n = (int)b->ctx.size();
    for (hv_ctx *c : b->ctx) {
        HV_CUDA(cudaStreamSynchronize(c->stream));
        if (c->fused.graph) {  // a context's own graph holds the old SOR buffers
            cudaGraphExecDestroy(c->fused.graph);
            c->fused.graph = nullptr;
            c->fused.graph_len = 0;
        }
        // the cap, doubled for an instance whose grid needs more blocks' shared
        // memory (the batched solve is a tagged sweep: it needs the source and
        // the row tables in shared memory too)
        auto usable = [&] { return c->fused.sor.ok && c->fused.sor.tables; };
        int m = sor_max_blocks;
        HV_TRY(sor_fast_replan(c, m));
        while (!usable() && m > 0 && m < b->sm_count) {
            m = std::min(2 * m, b->sm_count);
            HV_TRY(sor_fast_replan(c, m));
        }
        if (!usable()) {
            set_last_error("batch: an instance's SOR does not fit on chip");
            return HV_ERR_UNSUPPORTED;
        }
    }
    // instances whose solves take the direct form share launches of all SMs;
    // the others' sweeps go, first fit by decreasing block count, into waves of
    // at most one block per SM
    std::vector<int> order(n);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(),
                     [&](int x, int y) { return b->ctx[x]->fused.sor.nblocks > b->ctx[y]->fused.sor.nblocks; });
    std::vector<std::vector<int>> groups;
    std::vector<int> used;
    std::vector<bool> direct;
    for (int i : order) {
        const bool d = poisson_direct_runs(b->ctx[i]);
        const int nb = d ? 1 : b->ctx[i]->fused.sor.nblocks;
        size_t g = 0;
        while (g < groups.size() && (direct[g] != d || used[g] + nb > b->sm_count)) g++;
        if (g == groups.size()) {
            groups.emplace_back();
            used.push_back(0);
            direct.push_back(d);
        }
        groups[g].push_back(i);
        used[g] += nb;
    }
    b->blocks.assign(n, 0);
    for (size_t q = 0; q < groups.size(); q++) {
        const std::vector<int> &grp = groups[q];
        std::vector<hv_ctx *> cs;
        std::vector<const float *> rho;
        std::vector<int *> ctl, its;
        int ring = 0;
        for (int i : grp) {
            const float *r;
            int *cl, *it;
            fused_batch_sor_inputs(b->ctx[i], &r, &cl, &it, &ring);
            cs.push_back(b->ctx[i]);
            rho.push_back(r);
            ctl.push_back(cl);
            its.push_back(it);
        }
        b->waves.emplace_back();
        std::vector<int> blocks;
        hv_status st = direct[q] ? poisson_wave_build(b->waves.back(), cs, rho, ctl, its, ring, blocks)
                                 : sor_wave_build(b->waves.back(), cs, rho, ctl, its, ring);
        if (st != HV_OK) {
            set_last_error("batch: a wave of solves cannot be launched together");
            return st;
        }
        for (size_t k = 0; k < grp.size(); k++)
            b->blocks[grp[k]] = direct[q] ? blocks[k] : b->ctx[grp[k]]->fused.sor.nblocks;
    }
    b->cap = sor_max_blocks;
    b->gen.clear();
    for (hv_ctx *c : b->ctx) b->gen.push_back(c->plan_gen);
    return HV_OK;
}

int hv_batch_waves(const hv_batch *b) { return b ? (int)b->waves.size() : -1; }

hv_status hv_batch_run(hv_batch *b, int n_steps, hv_observables *obs) {
    if (!b || n_steps < 0) return HV_ERR_BAD_ARG;
    if (n_steps == 0) return HV_OK;
    HV_CUDA(cudaSetDevice(b->device));
    const int n = (int)b->ctx.size();
    // an instance's particles, parameters or options may have changed since the
    // plan: its fields are solved, and the waves, which hold its buffers and
    // options, built anew
    bool stale = (int)b->gen.size() != n;
    for (int i = 0; i < n; i++) {
        HV_TRY(fused_batch_ready(b->ctx[i]));
        stale = stale || b->gen[i] != b->ctx[i]->plan_gen;
    }
    if (stale) HV_TRY(hv_batch_plan(b, std::max(b->cap, 0)));
    // pinned room for what two chunks read back, per instance: the rows, the
    // iteration ring, the status word and (used once) the solver's seed
    const int ring = fused_batch_ring();
    const size_t rows_bytes = sizeof(double) * 8 * (size_t)b->chunk, its_bytes = sizeof(int) * (size_t)ring;
    const size_t per = rows_bytes + its_bytes + 64;
    if (!b->staging) HV_CUDA(cudaMallocHost((void **)&b->staging, 2 * per * n));
    auto slot = [&](int q, int i) { return b->staging + per * ((size_t)(q & 1) * n + i); };
    auto rows = [&](int q, int i) { return reinterpret_cast<double *>(slot(q, i)); };
    auto its = [&](int q, int i) { return reinterpret_cast<int *>(slot(q, i) + rows_bytes); };
    auto words = [&](int q, int i) { return reinterpret_cast<int *>(slot(q, i) + rows_bytes + its_bytes); };
    std::vector<int> exc(n, -1), start(n);
    for (int i = 0; i < n; i++) {
        hv_ctx *c = b->ctx[i];
        start[i] = c->step_index;
        HV_TRY(fused_batch_begin(c, n_steps, &exc[i]));
        HV_CUDA(cudaEventRecord(b->ev_a[i], c->stream));
        HV_CUDA(cudaStreamWaitEvent(b->stream, b->ev_a[i], 0));
    }
    const int chunks = (n_steps + b->chunk - 1) / b->chunk;
    // Waits for chunk q and decodes its rows.  A solve that gave up ends the
    // run for every instance; the others' rows of that chunk, and all rows of
    // the chunks before it, are written.
    auto settle = [&](int q) -> hv_status {
        HV_CUDA(cudaEventSynchronize(b->ev_done[q & 1]));
        const int s0 = q * b->chunk, k = std::min(b->chunk, n_steps - s0);
        hv_status failed = HV_OK;
        for (int i = 0; i < n; i++) {
            const hv_status st = fused_batch_status(b->ctx[i], words(q, i)[0]);
            if (st != HV_OK) failed = st;
            else if (obs)
                fused_batch_decode(b->ctx[i], start[i] + s0, k, rows(q, i), its(q, i), obs + (size_t)i * n_steps + s0);
        }
        return failed;
    };
    // the host stays one chunk ahead of the device: it learns of a solve that
    // gave up before a second further chunk is enqueued, and the device never
    // waits for it
    for (int q = 0; q < chunks; q++) {
        const int s0 = q * b->chunk, k = std::min(b->chunk, n_steps - s0);
        cudaGraphExec_t graph = nullptr;
        if (k == b->chunk) {
            if (!b->graph) b->graph = capture_steps(b, k);
            graph = b->graph;
        } else if (b->tail_len == k) {
            if (!b->tail_graph) b->tail_graph = capture_steps(b, k);
            graph = b->tail_graph;
        } else {
            // launched directly the first time: a length that does not come
            // again is not worth a capture
            if (b->tail_graph) cudaGraphExecDestroy(b->tail_graph);
            b->tail_graph = nullptr;
            b->tail_len = k;
        }
        if (graph) HV_CUDA(cudaGraphLaunch(graph, b->stream));
        else HV_TRY(enqueue_batch_steps(b, k));
        // the instances' rows side by side; the next chunk starts after them
        HV_CUDA(cudaEventRecord(b->ev_fork_a, b->stream));
        for (int i = 0; i < n; i++) {
            const cudaStream_t st = b->streams[i];
            HV_CUDA(cudaStreamWaitEvent(st, b->ev_fork_a, 0));
            HV_TRY(fused_batch_rows(b->ctx[i], st, start[i] + s0, k, rows(q, i), its(q, i)));
            HV_CUDA(cudaMemcpyAsync(words(q, i), b->ctx[i]->fused.sor.status, sizeof(int), cudaMemcpyDeviceToHost, st));
            HV_CUDA(cudaEventRecord(b->ev_a[i], st));
            HV_CUDA(cudaStreamWaitEvent(b->stream, b->ev_a[i], 0));
        }
        HV_CUDA(cudaEventRecord(b->ev_done[q & 1], b->stream));
        hv_status st = q > 0 ? settle(q - 1) : HV_OK;
        if (st == HV_OK && q + 1 == chunks) st = settle(q);
        if (st != HV_OK) {
            // the chunk behind the failed one may have failed in others too
            HV_CUDA(cudaStreamSynchronize(b->stream));
            for (int i = 0; i < n; i++) fused_batch_status(b->ctx[i], words(q, i)[0]);
            return st;
        }
    }
    for (int i = 0; i < n; i++) HV_TRY(fused_batch_end(b->ctx[i], n_steps, exc[i], words(0, i) + 1));
    for (int i = 0; i < n; i++) {
        HV_CUDA(cudaStreamSynchronize(b->ctx[i]->stream));
        if (words(0, i)[1] > 0) b->ctx[i]->fused.m_hint = words(0, i)[1];
    }
    return HV_OK;
}

hv_status hv_batch_autotune(hv_batch *b, int trial_steps, int *chosen_cap) {
    if (!b || trial_steps < 1) return HV_ERR_BAD_ARG;
    HV_CUDA(cudaSetDevice(b->device));
    // the cap shapes sweeps only: with direct solves alone there is nothing to
    // choose, and the instances' own plans stay
    bool sweeps = false;
    for (hv_ctx *c : b->ctx) sweeps = sweeps || !poisson_direct_runs(c);
    std::vector<int> caps = {0, 64, 32, 16, 8, 4};
    if (!sweeps) {
        caps.clear();
        if (b->cap != 0) HV_TRY(hv_batch_plan(b, 0));
    }
    cudaEvent_t e0, e1;
    HV_CUDA(cudaEventCreate(&e0));
    HV_CUDA(cudaEventCreate(&e1));
    int best = sweeps ? -1 : 0;
    float best_ms = 0.0f;
    for (int cap : caps) {
        if (hv_batch_plan(b, cap) != HV_OK) continue;
        HV_TRY(hv_batch_run(b, 1, nullptr));  // first use: graphs, caches
        HV_CUDA(cudaEventRecord(e0, b->stream));
        HV_TRY(hv_batch_run(b, trial_steps, nullptr));
        HV_CUDA(cudaEventRecord(e1, b->stream));
        HV_CUDA(cudaEventSynchronize(e1));
        float ms = 0.0f;
        HV_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (best < 0 || ms < best_ms) {
            best = cap;
            best_ms = ms;
        }
    }
    if (best < 0) {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        return HV_ERR_UNSUPPORTED;
    }
    if (sweeps) HV_TRY(hv_batch_plan(b, best));
    // then the particle step's block size, the same for every instance
    int best_pb = 0;
    best_ms = 0.0f;
    for (int pb : {128, 256, 512}) {
        for (hv_ctx *c : b->ctx) c->fused.pblock = pb;
        drop_graph(b);
        HV_TRY(hv_batch_run(b, 1, nullptr));
        HV_CUDA(cudaEventRecord(e0, b->stream));
        HV_TRY(hv_batch_run(b, trial_steps, nullptr));
        HV_CUDA(cudaEventRecord(e1, b->stream));
        HV_CUDA(cudaEventSynchronize(e1));
        float ms = 0.0f;
        HV_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (best_pb == 0 || ms < best_ms) {
            best_pb = pb;
            best_ms = ms;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    for (hv_ctx *c : b->ctx) c->fused.pblock = best_pb;
    drop_graph(b);
    if (chosen_cap) *chosen_cap = best;
    return HV_OK;
}

hv_status hv_batch_tiles(const hv_batch *b, int *sor_planes, int *sor_rows, int *sor_blocks, int *particle_block,
                         int n) {
    if (!b || n < 0 || n > (int)b->ctx.size()) return HV_ERR_BAD_ARG;
    for (int i = 0; i < n; i++) {
        const hv_ctx *c = b->ctx[i];
        int planes = c->fused.sor.P, rows = c->fused.sor.R;
        if (poisson_direct_runs(c)) poisson_tile(c, b->blocks[i], &planes, &rows);
        if (sor_planes) sor_planes[i] = planes;
        if (sor_rows) sor_rows[i] = rows;
        if (sor_blocks) sor_blocks[i] = b->blocks[i];
        if (particle_block) particle_block[i] = c->fused.pblock;
    }
    return HV_OK;
}

}  // extern "C"

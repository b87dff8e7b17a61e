// solvers.cu -- device-resident Krylov loops of the B200 lmp platform.
//
// The reference's solvers (src/linear_solver/cg.cc, gmres.cc, mpir.cc) return
// every dot product to the host and synchronise the device before each of
// the ~11 launches of an iteration.  Here the recurrence scalars and the
// IterateControl test live in device memory (DevState): the last CTA of each
// reducing kernel updates them, every later kernel of the iteration checks the
// stop state first and does nothing once the test has fired, and iterations
// are replayed from a captured CUDA graph in batches, so the host reads the
// state only once per batch.  The iteration count and the stop decision are
// exactly those of IterateControl::Check (src/common/iterate_control.cc:84-110).
#include "b200la.h"
#include "b200la_internal.h"
#include "grid_gather.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

using namespace b200;

#define SK(call)                                                                         \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess) return ctx_fail(ctx, B200LA_ERR_CUDA, #call, e_);        \
    } while (0)

void graph_cache_clear(b200la_ctx *ctx)
{
    for (auto &g : ctx->graphs)
        if (g.exec) cudaGraphExecDestroy(g.exec);
    ctx->graphs.clear();
}

static int batch_size()
{
    if (const char *e = std::getenv("B200LA_BATCH")) return std::max(1, std::atoi(e));
    return 16;
}

// The parts of a graph's key that stand for the objects whose buffers it
// holds: their numbers, and for a Jacobi preconditioner (which may be a
// temporary) its one buffer.
static const void *graph_key(const b200la_csr *A) { return reinterpret_cast<const void *>((uintptr_t)A->uid); }
static const void *graph_key(const b200la_precond *P)
{
    if (!P || P->kind == B200LA_PRECOND_JACOBI) return P ? P->invd : nullptr;
    return reinterpret_cast<const void *>((uintptr_t)P->uid);
}

// Capture `body` (which enqueues kernels on ctx->stream) into a graph keyed by
// `key`, or reuse the cached one.  Returns the executable graph.
template <class Body>
static int get_graph(b200la_ctx *ctx, const std::vector<const void *> &key, Body body, cudaGraphExec_t *exec,
                     int *nodes)
{
    for (auto &g : ctx->graphs)
        if (g.key == key) {
            *exec = g.exec;
            *nodes = g.launches;
            return B200LA_OK;
        }
    if (ctx->graphs.size() >= 32) graph_cache_clear(ctx);
    cudaGraph_t graph;
    SK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    const long long before = ctx->launches;
    const int rc = body();
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &graph);
    if (rc) {
        if (e == cudaSuccess) cudaGraphDestroy(graph);
        return rc;
    }
    if (e != cudaSuccess) return ctx_fail(ctx, B200LA_ERR_CUDA, "graph capture", e);
    GraphEntry g;
    g.key = key;
    g.launches = (int)(ctx->launches - before);
    ctx->launches = before;
    e = cudaGraphInstantiate(&g.exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return ctx_fail(ctx, B200LA_ERR_CUDA, "graph instantiate", e);
    ctx->graphs.push_back(g);
    *exec = g.exec;
    *nodes = g.launches;
    return B200LA_OK;
}

// The same for a graph whose single node is a device-side while loop: its
// body is `body(h)` captured once (K iterations), and the loop runs again as
// long as the conditional handle h -- set by the update kernel after each
// Check -- says "iterate".  One launch runs the solve to its stop; the host
// waits once instead of once per batch, and no batch of gated iterations
// runs after the stop.
template <class Body>
static int get_while_graph(b200la_ctx *ctx, const std::vector<const void *> &key, Body body, cudaGraphExec_t *exec,
                           int *nodes)
{
    for (auto &g : ctx->graphs)
        if (g.key == key) {
            *exec = g.exec;
            *nodes = g.launches;
            return B200LA_OK;
        }
    if (ctx->graphs.size() >= 32) graph_cache_clear(ctx);
    cudaGraph_t graph = nullptr;
    SK(cudaGraphCreate(&graph, 0));
    struct GraphGuard {
        cudaGraph_t g;
        ~GraphGuard()
        {
            if (g) cudaGraphDestroy(g);
        }
    } guard{graph};
    cudaGraphConditionalHandle h;
    SK(cudaGraphConditionalHandleCreate(&h, graph, 1u, cudaGraphCondAssignDefault));
    cudaGraphNodeParams prm = {cudaGraphNodeTypeConditional};
    prm.conditional.handle = h;
    prm.conditional.type = cudaGraphCondTypeWhile;
    prm.conditional.size = 1;
    cudaGraphNode_t node;
    SK(cudaGraphAddNode(&node, graph, nullptr, 0, &prm));
    cudaGraph_t loop = prm.conditional.phGraph_out[0];
    SK(cudaStreamBeginCaptureToGraph(ctx->stream, loop, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    const long long before = ctx->launches;
    const int rc = body((unsigned long long)h);
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &loop);
    if (rc) return rc;
    if (e != cudaSuccess) return ctx_fail(ctx, B200LA_ERR_CUDA, "loop body capture", e);
    GraphEntry g;
    g.key = key;
    g.launches = (int)(ctx->launches - before);
    ctx->launches = before;
    e = cudaGraphInstantiate(&g.exec, graph, 0);
    if (e != cudaSuccess) return ctx_fail(ctx, B200LA_ERR_CUDA, "loop graph instantiate", e);
    ctx->graphs.push_back(g);
    *exec = g.exec;
    *nodes = g.launches;
    return B200LA_OK;
}

// Device-side loop control of the CG iterations (B200LA_GRAPH_LOOP=0: host
// reads the stop state after every batch instead).
static bool loop_policy()
{
    const char *e = std::getenv("B200LA_GRAPH_LOOP");
    return !e || std::atoi(e) != 0;
}

static void state_init(DevState &s, const b200la_control *ctl, double *hist, int hist_len)
{
    std::memset(&s, 0, sizeof s);
    s.maxits = ctl->maxits;
    s.abstol = ctl->abstol;
    s.reltol = ctl->reltol;
    s.divtol = ctl->divtol;
    s.status = kIterate;
    s.hist = hist;
    s.hist_len = hist_len;
}

// ------------------------------------------------------------------ CG

struct CgWork {
    void *r, *p, *Ap, *z;
};

static int cg_core(b200la_ctx *ctx, const b200la_csr *A, const b200la_precond *P, const void *b, void *x,
                   const b200la_control *ctl, b200la_result *res, double *hist_dev, int hist_len, CgWork w,
                   bool time_it)
{
    const int n = A->n, dt = A->dtype;
    const int pc = !P ? 0 : (P->kind == B200LA_PRECOND_JACOBI ? 1 : 2);
    const void *invd = (pc == 1) ? P->invd : nullptr;
    const int *gate = &ctx->st->status;
    const Scratch sc = ctx_scratch(ctx);
    const long long l0 = ctx->launches;

    bool fused = false;
    if (const int rows = pc < 2 ? cg_fused_rows(ctx, A) : 0) {
        if (time_it) SK(cudaEventRecord(ctx->ev0, ctx->stream));
        const cudaError_t e = cg_fused_run(ctx, A, invd, b, x, w.r, w.p, ctl, hist_dev, hist_len, rows);
        if (e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorMemoryAllocation) SK(e);
        fused = e == cudaSuccess;
        if (!fused) cudaGetLastError();   // a launch per step needs neither
    }
    if (fused) {
        DevState *fs = ctx->st_host;
        ctx->launches += 1;
        if (time_it) SK(cudaEventRecord(ctx->ev1, ctx->stream));
        SK(cudaStreamSynchronize(ctx->stream));
        float ms = 0.f;
        if (time_it) SK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
        if (fs->pad0 != 0.0)
            if (const int rc = ctx_check_device_error(ctx)) return rc;
        if (res) {
            res->iters = fs->iter;
            res->status = fs->status;
            res->res0 = fs->res0;
            res->res = fs->res;
            res->outer = 0;
            res->launches = (int)(ctx->launches - l0);
            res->solve_ms = ms;
        }
        return B200LA_OK;
    }
    DevState *hs = ctx->st_host;
    state_init(*hs, ctl, hist_dev, hist_len);
    SK(cudaMemcpyAsync(ctx->st, hs, sizeof(DevState), cudaMemcpyHostToDevice, ctx->stream));
    if (time_it) SK(cudaEventRecord(ctx->ev0, ctx->stream));

    // r = b - A x; res0 = ||r||; status = Check(0, res0)   (cg.cc:200-204)
    SpmvOp op;
    op.epi = EPI_RESID;
    op.fin = FIN_RES_INIT;
    op.x = x;
    op.y = w.r;
    op.b = b;
    op.st = ctx->st;
    int rc = spmv_run(ctx, A, A->all, op);
    if (rc) return rc;
    // z = M^-1 r; p = z; rho = r.z   (cg.cc:205-214)
    if (pc == 2) {
        rc = precond_apply_async(ctx, P, w.r, w.z, nullptr);
        if (rc) return rc;
    }
    SK(launch_cg_start(sc, dt, n, pc, w.r, invd, w.z, w.p, ctx->st, ctx->stream));
    ctx->launches += 1;
    unsigned long long cond = 0;   // loop condition of the device-side while node (when captured in one)

    auto iteration = [&]() -> int {
        // Ap = A p; alpha = rho / (Ap.p)                       (cg.cc:219-220)
        SpmvOp o;
        o.epi = EPI_DOT_X;
        o.fin = FIN_CG_ALPHA;
        o.x = w.p;
        o.y = w.Ap;
        o.st = ctx->st;
        o.gate = gate;
        int r2 = spmv_run(ctx, A, A->all, o);
        if (r2) return r2;
        // x += alpha p; r -= alpha Ap; res = ||r||; Check       (cg.cc:221-230)
        SK(launch_cg_update(sc, dt, n, pc, x, w.r, w.p, w.Ap, invd, ctx->st, ctx->stream, cond));
        ctx->launches += 1;
        if (pc == 2) {
            // z = M^-1 r; gamma = r.z; beta = gamma / rho     (cg.cc:236-240)
            r2 = precond_apply_async(ctx, P, w.r, w.z, gate);
            if (r2) return r2;
            SK(launch_cg_rz(sc, dt, n, w.r, w.z, ctx->st, ctx->stream));
            ctx->launches += 1;
        }
        // p = beta p + z                                        (cg.cc:241)
        SK(launch_cg_pupdate(dt, n, pc, w.p, w.r, invd, w.z, ctx->st, ctx->stream));
        ctx->launches += 1;
        return B200LA_OK;
    };

    const int K = batch_size();
    cudaGraphExec_t exec = nullptr;
    int nodes = 0;
    const bool no_graph = std::getenv("B200LA_NOGRAPH") != nullptr;
    if (no_graph) {
        // batches launched kernel by kernel on the stream (same work, no graph)
        SK(cudaMemcpyAsync(hs, ctx->st, sizeof(DevState), cudaMemcpyDeviceToHost, ctx->stream));
        SK(cudaStreamSynchronize(ctx->stream));
        const long long max_b = (long long)ctl->maxits / K + 2;
        for (long long bt = 0; hs->status == kIterate && bt < max_b; ++bt) {
            for (int k = 0; k < K; ++k) {
                rc = iteration();
                if (rc) return rc;
            }
            SK(cudaMemcpyAsync(hs, ctx->st, sizeof(DevState), cudaMemcpyDeviceToHost, ctx->stream));
            SK(cudaStreamSynchronize(ctx->stream));
        }
    }
    const bool loop = !no_graph && loop_policy();
    const std::vector<const void *> key = {graph_key(A), graph_key(P), b, x, w.r, w.p, w.Ap, w.z, (const void *)(intptr_t)K,
                                           (const void *)(intptr_t)pc, ctx->stream, (const void *)(intptr_t)loop};
    auto batch = [&]() -> int {
        for (int k = 0; k < K; ++k) {
            int r2 = iteration();
            if (r2) return r2;
        }
        return B200LA_OK;
    };
    if (loop)
        rc = get_while_graph(
            ctx, key,
            [&](unsigned long long h) -> int {
                cond = h;
                const int r2 = batch();
                cond = 0;
                return r2;
            },
            &exec, &nodes);
    else if (!no_graph)
        rc = get_graph(ctx, key, batch, &exec, &nodes);
    if (rc) return rc;
    SK(cudaMemcpyAsync(hs, ctx->st, sizeof(DevState), cudaMemcpyDeviceToHost, ctx->stream));
    SK(cudaStreamSynchronize(ctx->stream));
    long long graph_launches = 0;
    if (loop && hs->status == kIterate) {
        // one launch; the loop ends on the device at the stop of IterateControl
        const int it0 = hs->iter;
        SK(cudaGraphLaunch(exec, ctx->stream));
        SK(cudaMemcpyAsync(hs, ctx->st, sizeof(DevState), cudaMemcpyDeviceToHost, ctx->stream));
        SK(cudaStreamSynchronize(ctx->stream));
        graph_launches += (long long)nodes * std::max(1, (hs->iter - it0 + K - 1) / K);
    }
    const long long max_batches = (long long)ctl->maxits / K + 2;
    for (long long bt = 0; !no_graph && !loop && hs->status == kIterate && bt < max_batches; ++bt) {
        SK(cudaGraphLaunch(exec, ctx->stream));
        graph_launches += nodes;
        SK(cudaMemcpyAsync(hs, ctx->st, sizeof(DevState), cudaMemcpyDeviceToHost, ctx->stream));
        SK(cudaStreamSynchronize(ctx->stream));
    }
    float ms = 0.f;
    if (time_it) {
        SK(cudaEventRecord(ctx->ev1, ctx->stream));
        SK(cudaEventSynchronize(ctx->ev1));
        SK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    }
    rc = ctx_check_device_error(ctx);
    if (rc) return rc;
    if (res) {
        res->iters = hs->iter;
        res->status = hs->status;
        res->res0 = hs->res0;
        res->res = hs->res;
        res->outer = 0;
        res->launches = (int)(ctx->launches - l0 + graph_launches);
        res->solve_ms = ms;
    }
    ctx->launches += graph_launches;
    return B200LA_OK;
}

static int cg_entry(b200la_ctx *ctx, const b200la_csr *A, const b200la_precond *P, const void *b, void *x,
                    const b200la_control *ctl, b200la_result *res, double *hist, int hist_len)
{
    if (!ctx || !A || !b || !x || !ctl || A->n != A->m || ctl->maxits < 0)
        return ctx_fail(ctx, B200LA_ERR_ARG, "cg: invalid argument", cudaSuccess);
    if (P && (P->dtype != A->dtype || P->n != A->n))
        return ctx_fail(ctx, B200LA_ERR_ARG, "cg: preconditioner does not match the operator", cudaSuccess);
    const size_t es = A->dtype == B200LA_F64 ? 8 : 4;
    const size_t vb = ((es * std::max(A->n, 1) + 255) / 256) * 256;
    const int hl = hist ? hist_len : 0;
    void *wk;
    int rc = ctx_work(ctx, 4 * vb + sizeof(double) * (hl + 1), &wk);
    if (rc) return rc;
    char *base = static_cast<char *>(wk);
    CgWork w{base, base + vb, base + 2 * vb, base + 3 * vb};
    double *hd = hl ? reinterpret_cast<double *>(base + 4 * vb) : nullptr;
    rc = cg_core(ctx, A, P, b, x, ctl, res, hd, hl, w, true);
    if (rc) return rc;
    if (hl) {
        const int cnt = std::min(hl, (res ? res->iters : 0) + 1);
        SK(cudaMemcpy(hist, hd, sizeof(double) * cnt, cudaMemcpyDeviceToHost));
    }
    return B200LA_OK;
}

extern "C" int b200la_cg(b200la_ctx *ctx, const b200la_csr *A, const b200la_precond *P, const void *b, void *x,
                         const b200la_control *ctl, b200la_result *res)
{
    NvtxScope nvtx_range("b200la_cg");
    return cg_entry(ctx, A, P, b, x, ctl, res, nullptr, 0);
}

extern "C" int b200la_cg_hist(b200la_ctx *ctx, const b200la_csr *A, const b200la_precond *P, const void *b,
                              void *x, const b200la_control *ctl, b200la_result *res, double *hist, int hist_len)
{
    NvtxScope nvtx_range("b200la_cg_hist");
    return cg_entry(ctx, A, P, b, x, ctl, res, hist, hist_len);
}

// ------------------------------------------------------------------ MPIR

extern "C" int b200la_mpir(b200la_ctx *ctx, const b200la_csr *A64, const b200la_csr *A32in, const double *b,
                           double *x, const b200la_control *outer, const b200la_control *inner, int max_outer,
                           b200la_result *res)
{
    NvtxScope nvtx_range("b200la_mpir");
    if (!ctx || !A64 || !b || !x || !outer || !inner || A64->dtype != B200LA_F64 || A64->n != A64->m ||
        max_outer < 0 || (A32in && (A32in->dtype != B200LA_F32 || A32in->n != A64->n || A32in->nnz != A64->nnz)))
        return ctx_fail(ctx, B200LA_ERR_ARG, "mpir: invalid argument", cudaSuccess);
    const int n = A64->n;
    b200la_csr *A32 = const_cast<b200la_csr *>(A32in);
    bool own32 = false;
    if (!A32) {
        int rc = b200la_csr_cast(ctx, A64, B200LA_F32, &A32);
        if (rc) return rc;
        own32 = true;
    }
    struct Guard {
        b200la_csr *m;
        bool own;
        ~Guard()
        {
            if (own) b200la_csr_destroy(m);
        }
    } guard{A32, own32};
    const size_t v8 = ((8 * (size_t)std::max(n, 1) + 255) / 256) * 256, v4 = ((4 * (size_t)std::max(n, 1) + 255) / 256) * 256;
    void *wk;
    // r (f64), invd64 scratch (f64), rl, cl, and the inner CG's r, p, Ap (f32)
    int rc = ctx_work(ctx, 2 * v8 + 6 * v4, &wk);
    if (rc) return rc;
    char *base = static_cast<char *>(wk);
    double *r = reinterpret_cast<double *>(base);
    double *invd64 = reinterpret_cast<double *>(base + v8);
    float *invd32 = nullptr;   // the operator's cached FP32 Jacobi scaling (below)
    float *rl = reinterpret_cast<float *>(base + 2 * v8 + v4);
    float *cl = reinterpret_cast<float *>(base + 2 * v8 + 2 * v4);
    CgWork w{base + 2 * v8 + 3 * v4, base + 2 * v8 + 4 * v4, base + 2 * v8 + 5 * v4, nullptr};
    const long long l0 = ctx->launches;

    // FP32 Jacobi from the FP64 diagonal (1/a_ii rounded once), made at the
    // operator's first defect correction and kept with it until its values change
    if (!A64->invd32) {
        b200la_csr *Am = const_cast<b200la_csr *>(A64);
        SK(cudaMalloc(&Am->invd32, sizeof(float) * std::max(n, 1)));
        SK(launch_invdiag(B200LA_F64, n, A64->row, A64->col, A64->val, invd64, ctx->stream));
        SK(launch_cast(B200LA_F64, invd64, B200LA_F32, Am->invd32, n, ctx->stream));
        ctx->launches += 2;
    }
    invd32 = A64->invd32;
    SK(cudaEventRecord(ctx->ev0, ctx->stream));
    b200la_precond J;
    J.kind = B200LA_PRECOND_JACOBI;
    J.n = n;
    J.dtype = B200LA_F32;
    J.invd = invd32;

    auto residual = [&](double *out) -> int {
        // r = b - A x in FP64 and ||r||   (mpir.cc:125-128, 271-273)
        SpmvOp op;
        op.epi = EPI_RESID;
        op.fin = FIN_STORE;
        op.x = x;
        op.y = r;
        op.b = b;
        op.dot_out = ctx->dscal;
        int r2 = spmv_run(ctx, A64, A64->all, op);
        if (r2) return r2;
        SK(cudaMemcpyAsync(ctx->hscal, ctx->dscal, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        SK(cudaStreamSynchronize(ctx->stream));
        *out = std::sqrt(ctx->hscal[0]);
        return B200LA_OK;
    };
    double rnorm;
    rc = residual(&rnorm);
    if (rc) return rc;
    const double res0 = rnorm;
    int n_outer = 0, inner_total = 0;
    long long inner_launches = 0;
    // ContinueIteration (mpir.cc:308-326) with the relative test against the
    // initial residual
    while (rnorm > outer->abstol && rnorm > outer->reltol * res0 && rnorm < outer->divtol && n_outer < max_outer) {
        ++n_outer;
        // resl = (float) resh; corl = 0   (mpir.cc:169-170)
        SK(launch_cast_residual(n, r, rl, cl, ctx->stream));
        ctx->launches += 1;
        // low-precision error correction: Jacobi-CG on A32 (mpir.cc:193)
        b200la_result ir;
        std::memset(&ir, 0, sizeof ir);
        rc = cg_core(ctx, A32, &J, rl, cl, inner, &ir, nullptr, 0, w, false);
        if (rc) return rc;
        inner_total += ir.iters;
        inner_launches += ir.launches;
        // x += (double) corl   (mpir.cc:223, 253)
        SK(launch_add_correction(n, cl, x, ctx->stream));
        ctx->launches += 1;
        rc = residual(&rnorm);
        if (rc) return rc;
    }
    SK(cudaEventRecord(ctx->ev1, ctx->stream));
    SK(cudaEventSynchronize(ctx->ev1));
    float ms = 0.f;
    SK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    if (res) {
        res->iters = inner_total;
        res->outer = n_outer;
        res->res0 = res0;
        res->res = rnorm;
        res->status = rnorm < outer->abstol ? B200LA_SUCCESS_ABS
                      : rnorm < outer->reltol * res0 ? B200LA_SUCCESS_REL
                      : rnorm >= outer->divtol     ? B200LA_FAIL_DIV
                                                   : B200LA_FAIL_MAXITS;
        res->launches = (int)(ctx->launches - l0);
        res->solve_ms = ms;
    }
    (void)inner_launches;
    return ctx_check_device_error(ctx);
}

// ------------------------------------------------------------------ MPIR with a GMRES correction

extern "C" int b200la_mpir_gmres(b200la_ctx *ctx, const b200la_csr *A64, const b200la_csr *A32,
                                 const b200la_precond *P32, int m, const double *b, double *x,
                                 const b200la_control *outer, const b200la_control *inner, int max_outer,
                                 b200la_result *res)
{
    NvtxScope nvtx_range("b200la_mpir_gmres");
    if (!ctx || !A64 || !A32 || !b || !x || !outer || !inner || m < 1 || max_outer < 0 ||
        A64->dtype != B200LA_F64 || A32->dtype != B200LA_F32 || A64->n != A64->m || A32->n != A64->n ||
        (P32 && (P32->dtype != B200LA_F32 || P32->n != A64->n)))
        return ctx_fail(ctx, B200LA_ERR_ARG, "mpir_gmres: invalid argument", cudaSuccess);
    const int n = A64->n;
    const size_t v8 = ((8 * (size_t)std::max(n, 1) + 255) / 256) * 256, v4 = ((4 * (size_t)std::max(n, 1) + 255) / 256) * 256;
    void *wk;
    int rc = ctx_work_outer(ctx, v8 + 2 * v4, &wk);
    if (rc) return rc;
    char *base = static_cast<char *>(wk);
    double *r = reinterpret_cast<double *>(base);
    float *rl = reinterpret_cast<float *>(base + v8);
    float *cl = reinterpret_cast<float *>(base + v8 + v4);
    const long long l0 = ctx->launches;
    // own events: the inner GMRES times itself with the context's
    struct Ev {
        cudaEvent_t a = nullptr, b = nullptr;
        ~Ev()
        {
            if (a) cudaEventDestroy(a);
            if (b) cudaEventDestroy(b);
        }
    } ev;
    SK(cudaEventCreate(&ev.a));
    SK(cudaEventCreate(&ev.b));
    SK(cudaEventRecord(ev.a, ctx->stream));
    auto residual = [&](double *out) -> int {
        // r = b - A x in FP64 and ||r||   (mpir.cc:125-128, 271-273)
        SpmvOp op;
        op.epi = EPI_RESID;
        op.fin = FIN_STORE;
        op.x = x;
        op.y = r;
        op.b = b;
        op.dot_out = ctx->dscal;
        int r2 = spmv_run(ctx, A64, A64->all, op);
        if (r2) return r2;
        SK(cudaMemcpyAsync(ctx->hscal, ctx->dscal, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        SK(cudaStreamSynchronize(ctx->stream));
        *out = std::sqrt(ctx->hscal[0]);
        return B200LA_OK;
    };
    double rnorm;
    rc = residual(&rnorm);
    if (rc) return rc;
    const double res0 = rnorm;
    int n_outer = 0, inner_total = 0, inner_launches = 0;
    while (rnorm > outer->abstol && rnorm > outer->reltol * res0 && rnorm < outer->divtol && n_outer < max_outer) {
        ++n_outer;
        // resl = (float) resh; corl = 0   (mpir.cc:169-170)
        SK(launch_cast_residual(n, r, rl, cl, ctx->stream));
        ctx->launches += 1;
        // low-precision error correction: GMRES(m) on A32 with P32 (mpir.cc:193)
        b200la_result ir;
        std::memset(&ir, 0, sizeof ir);
        rc = b200la_gmres(ctx, A32, P32, m, rl, cl, inner, &ir);
        if (rc) return rc;
        inner_total += ir.iters;
        inner_launches += ir.launches;
        // x += (double) corl   (mpir.cc:223, 253)
        SK(launch_add_correction(n, cl, x, ctx->stream));
        ctx->launches += 1;
        rc = residual(&rnorm);
        if (rc) return rc;
    }
    SK(cudaEventRecord(ev.b, ctx->stream));
    SK(cudaEventSynchronize(ev.b));
    float ms = 0.f;
    SK(cudaEventElapsedTime(&ms, ev.a, ev.b));
    if (res) {
        res->iters = inner_total;
        res->outer = n_outer;
        res->res0 = res0;
        res->res = rnorm;
        res->status = rnorm < outer->abstol ? B200LA_SUCCESS_ABS
                      : rnorm < outer->reltol * res0 ? B200LA_SUCCESS_REL
                      : rnorm >= outer->divtol     ? B200LA_FAIL_DIV
                                                   : B200LA_FAIL_MAXITS;
        res->launches = (int)(ctx->launches - l0);
        res->solve_ms = ms;
    }
    (void)inner_launches;
    return ctx_check_device_error(ctx);
}

// ------------------------------------------------------------------ GMRES

namespace {

struct GmresDev {
    double *H;      // H(j, i) = H[j * (m + 1) + i]
    double *g, *cs, *sn, *y;
    int *jend;
};

__device__ __forceinline__ int check_dev(DevState *st, int step, double value)
{
    if (step == 0) st->res0 = value;
    if (value < st->abstol) return kSuccessAbs;
    if (value < st->reltol * st->res0) return kSuccessRel;
    if (value > st->divtol * st->res0) return kFailDiv;
    if (step >= st->maxits) return kFailMaxits;
    return kIterate;
}

// Givens part of one Arnoldi step (gmres.cc:380-402 with gmres.h:77-97).
__global__ void gmres_givens_kernel(int j, int m, GmresDev d, DevState *st)
{
    if (st->status != kIterate) return;
    const int ld = m + 1;
    double *Hj = d.H + (size_t)j * ld;
    for (int k = 0; k < j; ++k) {
        const double t = d.cs[k] * Hj[k] + d.sn[k] * Hj[k + 1];
        Hj[k + 1] = -d.sn[k] * Hj[k] + d.cs[k] * Hj[k + 1];
        Hj[k] = t;
    }
    const double beta = sqrt(Hj[j] * Hj[j] + Hj[j + 1] * Hj[j + 1]);
    d.cs[j] = Hj[j] / beta;
    d.sn[j] = Hj[j + 1] / beta;
    {
        const double t = d.cs[j] * Hj[j] + d.sn[j] * Hj[j + 1];
        Hj[j + 1] = -d.sn[j] * Hj[j] + d.cs[j] * Hj[j + 1];
        Hj[j] = t;
    }
    {
        const double t = d.cs[j] * d.g[j] + d.sn[j] * d.g[j + 1];
        d.g[j + 1] = -d.sn[j] * d.g[j] + d.cs[j] * d.g[j + 1];
        d.g[j] = t;
    }
    const double res = fabs(d.g[j + 1]);
    const int it = st->iter + 1;
    st->iter = it;
    st->res = res;
    const int s = check_dev(st, it, res);
    st->status = s;
    if (s != kIterate) *d.jend = j;
}

// Modified Gram-Schmidt of one Arnoldi step (gmres.cc:373-402) in one launch:
// w stays in registers (EV 16-byte vectors per thread), every product sums over
// the grid by a gather (grid_gather.cuh), v_{i+1} is loaded while the sum of
// v_i travels, the norm, V_{j+1} = w / ||w||, the Givens rotations (on CTA 0,
// while it waits) and the check follow in the same launch.
//   Bound by the j + 2 grid sums: the basis lies in L2 at these sizes.  A dot
// and an axpy launch per basis vector took 8.5 us at 2-D 512^2 (2.1 MB per
// vector).  GMRES(30) + ILU(0) 512^2 to 1e-10: 170 -> 145 ms; mixed 300^2: 25.8
// -> 20.9 ms; ILU(1) 200^2: 9.8 -> 8.3 ms.  The launches stay for vectors that
// do not fit the registers of one CTA per SM (1.2 million doubles), where their
// bytes outweigh the launches.
constexpr int kOrthThreads = 512;

template <typename T, int EV>
__global__ void __launch_bounds__(kOrthThreads) gmres_orth_kernel(int n, int j, int m, const T *__restrict__ w,
                                                                  T *__restrict__ V, size_t ld, GmresDev d,
                                                                  DevState *st, unsigned char *gmem, int *err, int first_poll)
{
    if (gate_closed(&st->status)) return;
    using V4 = std::conditional_t<sizeof(T) == 8, double2, float4>;
    constexpr int W = 16 / (int)sizeof(T);
    __shared__ typename GridGather<kOrthThreads>::Shared sh;
    GridGather<kOrthThreads> gg(gmem, sh, err, first_poll);
    const int stride = gridDim.x * kOrthThreads, first = blockIdx.x * kOrthThreads + threadIdx.x;
    const bool scribe = blockIdx.x == 0 && threadIdx.x == 0;
    double *Hj = d.H + (size_t)j * (m + 1);
    struct Vec {
        T e[W];
    };
    // vector iv of a basis vector, entries past n as zero (the vectors are padded to 256 bytes)
    auto load = [&](const T *p, Vec (&q)[EV]) {
#pragma unroll
        for (int u = 0; u < EV; ++u) {
            const int iv = first + u * stride;
            V4 t = {};
            if ((long long)iv * W < n) t = *reinterpret_cast<const V4 *>(p + (size_t)iv * W);
            q[u].e[0] = t.x;
            q[u].e[1] = t.y;
            if constexpr (W == 4) {
                q[u].e[2] = t.z;
                q[u].e[3] = t.w;
            }
#pragma unroll
            for (int k = 1; k < W; ++k)
                if ((long long)iv * W + k >= n) q[u].e[k] = T(0);
        }
    };
    auto dot = [&](const Vec (&a)[EV], const Vec (&b)[EV]) {
        double s = 0.0;
#pragma unroll
        for (int u = 0; u < EV; ++u) {
            T t = T(0);
#pragma unroll
            for (int k = 0; k < W; ++k) t += a[u].e[k] * b[u].e[k];
            s += (double)t;
        }
        return s;
    };
    Vec x[EV], v[EV], vn[EV] = {};
    load(w, x);
    load(V, v);
    // rotation k of the column (gmres.h:77-97), once H(j, k) and H(j, k + 1) are known
    double hk = 0.0;   // scribe: H(j, k) after the rotations before k
    auto rotate = [&](int k, double next) {
        const double t = d.cs[k] * hk + d.sn[k] * next;
        const double r = -d.sn[k] * hk + d.cs[k] * next;
        Hj[k] = t;
        hk = r;
    };
    double hlast = 0.0;   // H(j, i - 1), not yet rotated
    for (int i = 0; i <= j; ++i) {
        const double part[1] = {dot(x, v)};
        gg.template publish<1>(part);
        if (i < j) load(V + (size_t)(i + 1) * ld, vn);
        if (scribe) {
            if (i == 1) hk = hlast;
            if (i > 1) rotate(i - 2, hlast);
        }
        double h[1];
        gg.template total<1>(h);
        const T c = (T)(-1.0 * h[0]);
#pragma unroll
        for (int u = 0; u < EV; ++u) {
#pragma unroll
            for (int k = 0; k < W; ++k) {
                x[u].e[k] += c * v[u].e[k];
                v[u].e[k] = vn[u].e[k];
            }
        }
        hlast = h[0];
    }
    const double part[1] = {dot(x, x)};
    gg.template publish<1>(part);
    if (scribe) {
        if (j == 0) hk = hlast;
        else rotate(j - 1, hlast);
    }
    double nn[1];
    gg.template total<1>(nn);
    const double norm = sqrt(nn[0]);
    gg.close();
    // V_{j+1} = w / H(j, j+1)
    const T c = (T)(1.0 / norm);
    T *out = V + (size_t)(j + 1) * ld;
#pragma unroll
    for (int u = 0; u < EV; ++u) {
        const int iv = first + u * stride;
        if ((long long)iv * W + W <= n) {
            V4 t;
            t.x = c * x[u].e[0];
            t.y = c * x[u].e[1];
            if constexpr (W == 4) {
                t.z = c * x[u].e[2];
                t.w = c * x[u].e[3];
            }
            *reinterpret_cast<V4 *>(out + (size_t)iv * W) = t;
        } else {
#pragma unroll
            for (int k = 0; k < W; ++k)
                if ((long long)iv * W + k < n) out[(size_t)iv * W + k] = c * x[u].e[k];
        }
    }
    if (!scribe) return;
    // the new rotation (gmres.cc:380-402)
    const double beta = sqrt(hk * hk + norm * norm);
    const double cs = hk / beta, sn = norm / beta;
    d.cs[j] = cs;
    d.sn[j] = sn;
    Hj[j] = cs * hk + sn * norm;
    Hj[j + 1] = -sn * hk + cs * norm;
    const double gj = d.g[j], gn = d.g[j + 1];
    d.g[j + 1] = -sn * gj + cs * gn;
    d.g[j] = cs * gj + sn * gn;
    const double res = fabs(d.g[j + 1]);
    const int it = st->iter + 1;
    st->iter = it;
    st->res = res;
    const int s = check_dev(st, it, res);
    st->status = s;
    if (s != kIterate) *d.jend = j;
}

// CTAs of the one-launch orthogonalisation for vectors of n entries, and the
// 16-byte vectors per thread; 0: they do not fit.
static int orth_grid(int n, size_t es, int num_sms, int *ev)
{
    const long long nv = ((long long)n * (long long)es + 15) / 16;
    const int cap = gather_ctas(num_sms);
    for (int e = 1; e <= 8; e *= 2)
        if (nv <= (long long)cap * kOrthThreads * e) {
            *ev = e;
            return (int)std::max(1LL, (nv + (long long)kOrthThreads * e - 1) / ((long long)kOrthThreads * e));
        }
    return 0;
}

// f(the kernel instance for ev 16-byte vectors per thread)
template <typename T, class F>
static auto orth_dispatch(int ev, F f)
{
    switch (ev) {
    case 1: return f(gmres_orth_kernel<T, 1>);
    case 2: return f(gmres_orth_kernel<T, 2>);
    case 4: return f(gmres_orth_kernel<T, 4>);
    default: return f(gmres_orth_kernel<T, 8>);
    }
}

// Whether all CTAs of the grid can be on the device at once.  (Asked beforehand:
// in a captured graph the launch that would say so comes too late.)
template <typename T>
static bool orth_resident(const b200la_ctx *ctx, int grid, int ev)
{
    int per_sm = 0;
    const cudaError_t e = orth_dispatch<T>(ev, [&](auto kern) {
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kOrthThreads, 0);
    });
    return e == cudaSuccess && grid <= per_sm * ctx->num_sms;
}

template <typename T>
static cudaError_t launch_gmres_orth(int grid, int ev, int n, int j, int m, const void *w, void *V, size_t ld, GmresDev d,
                                     DevState *st, unsigned char *gmem, int *err, cudaStream_t stream)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = kOrthThreads;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return orth_dispatch<T>(ev, [&](auto kern) {
        return cudaLaunchKernelEx(&cfg, kern, n, j, m, (const T *)w, (T *)V, ld, d, st, gmem, err, gather_first());
    });
}

// Back substitution of UpdateSolution (gmres.cc:487-504) into y[0..k].
__global__ void gmres_backsub_kernel(int k, int m, GmresDev d)
{
    const int ld = m + 1;
    for (int i = 0; i <= m; ++i) d.y[i] = d.g[i];
    for (int i = k + 1; i--;) {
        d.y[i] /= d.H[(size_t)i * ld + i];
        const double t = d.y[i];
        for (int q = 0; q < i; ++q) d.y[q] -= d.H[(size_t)i * ld + q] * t;
    }
}

// Cycle start: H = 0, g = 0, g[0] = res (gmres.cc:344-350).  As in the
// reference, a restart normalises the new residual by the last Givens
// estimate |g[j+1]| held in res, not by a recomputed norm.
__global__ void gmres_cycle_kernel(int m, GmresDev d, const DevState *st)
{
    const int ld = m + 1;
    for (int i = threadIdx.x; i < m * ld; i += blockDim.x) d.H[i] = 0.0;
    for (int i = threadIdx.x; i <= m; i += blockDim.x) d.g[i] = 0.0;
    __syncthreads();
    if (threadIdx.x == 0) d.g[0] = st->res;
}

// z = sum_{i<=k} y_i V_i (the vectors V_i at stride ld elements).
template <typename T>
__global__ void lincomb_kernel(int n, int k, const T *__restrict__ V, size_t ld, const double *__restrict__ y,
                               T *__restrict__ z)
{
    for (int i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
        T s = T(0);
        for (int q = 0; q <= k; ++q) s += (T)y[q] * V[(size_t)q * ld + i];
        z[i] = s;
    }
}

}  // namespace

extern "C" int b200la_gmres(b200la_ctx *ctx, const b200la_csr *A, const b200la_precond *P, int m, const void *b,
                            void *x, const b200la_control *ctl, b200la_result *res)
{
    NvtxScope nvtx_range("b200la_gmres");
    if (!ctx || !A || !b || !x || !ctl || A->n != A->m || m < 1)
        return ctx_fail(ctx, B200LA_ERR_ARG, "gmres: invalid argument", cudaSuccess);
    if (P && (P->dtype != A->dtype || P->n != A->n))
        return ctx_fail(ctx, B200LA_ERR_ARG, "gmres: preconditioner does not match the operator", cudaSuccess);
    const int n = A->n, dt = A->dtype;
    const int mb = std::max(1, std::min(m, ctl->maxits));   // gmres.cc:301
    const size_t es = dt == B200LA_F64 ? 8 : 4;
    const size_t ldv = ((es * std::max(n, 1) + 255) / 256) * 256;   // bytes per basis vector
    const size_t small = sizeof(double) * ((size_t)mb * (mb + 1) + 4 * (mb + 1) + 8);
    void *wk;
    int rc = ctx_work(ctx, ldv * (mb + 1 + 2) + small, &wk);
    if (rc) return rc;
    char *base = static_cast<char *>(wk);
    auto V = [&](int k) { return (void *)(base + ldv * k); };
    void *w = base + ldv * (mb + 1), *z = base + ldv * (mb + 2);
    double *sm = reinterpret_cast<double *>(base + ldv * (mb + 3));
    GmresDev d;
    d.H = sm;
    d.g = sm + (size_t)mb * (mb + 1);
    d.cs = d.g + (mb + 1);
    d.sn = d.cs + (mb + 1);
    d.y = d.sn + (mb + 1);
    d.jend = reinterpret_cast<int *>(d.y + (mb + 1));
    const int *gate = &ctx->st->status;
    const Scratch sc = ctx_scratch(ctx);
    const long long l0 = ctx->launches;
    const size_t ld_el = ldv / es;
    int ev = 0;
    int orth = ctx->cooperative ? orth_grid(n, es, ctx->num_sms, &ev) : 0;
    if (orth && !(dt == B200LA_F64 ? orth_resident<double>(ctx, orth, ev) : orth_resident<float>(ctx, orth, ev)))
        orth = 0;

    DevState *hs = ctx->st_host;
    state_init(*hs, ctl, nullptr, 0);
    SK(cudaMemcpyAsync(ctx->st, hs, sizeof(DevState), cudaMemcpyHostToDevice, ctx->stream));
    SK(cudaEventRecord(ctx->ev0, ctx->stream));
    // V0 = b - A x; res = ||V0||; Check(0)   (gmres.cc:323-335)
    SpmvOp op;
    op.epi = EPI_RESID;
    op.fin = FIN_RES_INIT;
    op.x = x;
    op.y = V(0);
    op.b = b;
    op.st = ctx->st;
    rc = spmv_run(ctx, A, A->all, op);
    if (rc) return rc;
    long long graph_launches = 0;
    for (;;) {
        SK(cudaMemcpyAsync(hs, ctx->st, sizeof(DevState), cudaMemcpyDeviceToHost, ctx->stream));
        SK(cudaStreamSynchronize(ctx->stream));
        if (hs->status != kIterate) break;
        // one restart cycle: captured once, replayed per cycle
        auto cycle = [&]() -> int {
            gmres_cycle_kernel<<<1, 256, 0, ctx->stream>>>(mb, d, ctx->st);
            SK(cudaGetLastError());
            SK(launch_scale_dev(dt, n, d.g, true, V(0), V(0), nullptr, ctx->stream));
            ctx->launches += 2;
            for (int j = 0; j < mb; ++j) {
                const void *zin = V(j);
                if (P) {
                    int r2 = precond_apply_async(ctx, P, V(j), z, gate);
                    if (r2) return r2;
                    zin = z;
                }
                SpmvOp o;
                o.epi = EPI_SET;
                o.x = zin;
                o.y = w;
                o.gate = gate;
                int r2 = spmv_run(ctx, A, A->all, o);
                if (r2) return r2;
                if (orth) {
                    SK(dt == B200LA_F64 ? launch_gmres_orth<double>(orth, ev, n, j, mb, w, V(0), ld_el, d, ctx->st,
                                                                    ctx->gather, ctx->dev_err, ctx->stream)
                                        : launch_gmres_orth<float>(orth, ev, n, j, mb, w, V(0), ld_el, d, ctx->st,
                                                                   ctx->gather, ctx->dev_err, ctx->stream));
                    ctx->launches += 1;
                    continue;
                }
                // modified Gram-Schmidt (gmres.cc:373-377)
                for (int i = 0; i <= j; ++i) {
                    SK(launch_dot_to(sc, dt, n, w, V(i), d.H + (size_t)j * (mb + 1) + i, gate, ctx->stream));
                    SK(launch_axpy_dev(dt, n, d.H + (size_t)j * (mb + 1) + i, -1.0, V(i), w, gate, ctx->stream));
                    ctx->launches += 2;
                }
                // H(j, j+1) = ||w||; V_{j+1} = w / H(j, j+1)   (gmres.cc:379-383)
                SK(launch_dot_norm_to(sc, dt, n, w, d.H + (size_t)j * (mb + 1) + j + 1, gate, ctx->stream));
                SK(launch_scale_dev(dt, n, d.H + (size_t)j * (mb + 1) + j + 1, true, w, V(j + 1), gate, ctx->stream));
                gmres_givens_kernel<<<1, 1, 0, ctx->stream>>>(j, mb, d, ctx->st);
                SK(cudaGetLastError());
                ctx->launches += 3;
            }
            return B200LA_OK;
        };
        cudaGraphExec_t exec;
        int nodes = 0;
        const int kind = P ? P->kind : 0;
        ctx->last_cuda = cudaSuccess;
        rc = get_graph(ctx, {graph_key(A), graph_key(P), b, x, wk, (const void *)(intptr_t)mb,
                             (const void *)(intptr_t)(-7 - kind), ctx->stream, (const void *)(intptr_t)orth,
                             (const void *)(intptr_t)gather_first()}, cycle, &exec, &nodes);
        const cudaError_t le = rc ? ctx->last_cuda : cudaGraphLaunch(exec, ctx->stream);
        if (orth && le == cudaErrorCooperativeLaunchTooLarge) {   // (a stream limited to some of the SMs)
            cudaGetLastError();
            orth = 0;
            continue;
        }
        if (rc) return rc;
        SK(le);
        graph_launches += nodes;
        SK(cudaMemcpyAsync(hs, ctx->st, sizeof(DevState), cudaMemcpyDeviceToHost, ctx->stream));
        int jend = mb - 1;
        SK(cudaMemcpyAsync(&ctx->hscal[8], d.jend, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        volatile int *flag = reinterpret_cast<volatile int *>(ctx->hscal + 130);
        SK(cudaMemcpyAsync(const_cast<int *>(flag), ctx->dev_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        SK(cudaStreamSynchronize(ctx->stream));
        if (*flag != kDevOk) return ctx_check_device_error(ctx);   // a wait has run out: no further cycle
        if (hs->status != kIterate) std::memcpy(&jend, &ctx->hscal[8], sizeof(int));
        // UpdateSolution + preconditioner + x += w   (gmres.cc:404-445)
        gmres_backsub_kernel<<<1, 1, 0, ctx->stream>>>(jend, mb, d);
        SK(cudaGetLastError());
        const int g = std::max(1, std::min((n + kBlock * 4 - 1) / (kBlock * 4), ctx->num_sms * 8));
        if (dt == B200LA_F64)
            lincomb_kernel<double><<<g, kBlock, 0, ctx->stream>>>(n, jend, (const double *)V(0), ld_el, d.y, (double *)z);
        else
            lincomb_kernel<float><<<g, kBlock, 0, ctx->stream>>>(n, jend, (const float *)V(0), ld_el, d.y, (float *)z);
        SK(cudaGetLastError());
        ctx->launches += 2;
        const void *corr = z;
        if (P) {
            rc = precond_apply_async(ctx, P, z, w, nullptr);
            if (rc) return rc;
            corr = w;
        }
        SK(launch_axpy(dt, n, 1.0, corr, x, ctx->stream));
        ctx->launches += 1;
        if (hs->status != kIterate) break;
        // restart residual (gmres.cc:433-436)
        SpmvOp o;
        o.epi = EPI_RESID;
        o.fin = FIN_NONE;
        o.x = x;
        o.y = V(0);
        o.b = b;
        rc = spmv_run(ctx, A, A->all, o);
        if (rc) return rc;
    }
    SK(cudaEventRecord(ctx->ev1, ctx->stream));
    SK(cudaEventSynchronize(ctx->ev1));
    float ms = 0.f;
    SK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    rc = ctx_check_device_error(ctx);
    if (rc) return rc;
    if (res) {
        res->iters = hs->iter;
        res->status = hs->status;
        res->res0 = hs->res0;
        res->res = hs->res;
        res->outer = 0;
        res->launches = (int)(ctx->launches - l0 + graph_launches);
        res->solve_ms = ms;
    }
    ctx->launches += graph_launches;
    return B200LA_OK;
}

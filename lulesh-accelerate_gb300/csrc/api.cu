// api.cu -- the C ABI (include/lulesh_gb300.h): contexts, device memory,
// the captured run-loop graph and the step entry points.
#include "lulesh_internal.h"
#include "kernels.h"
#include "common.cuh"
#include "crossing.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

using namespace lulesh;

struct lulesh_ctx {
    int s = 0;
    long ne = 0, nn = 0;
    int precision = LULESH_PRECISION_FP64;
    int device = 0;
    cudaStream_t stream = nullptr;
    Dom dom{};
    std::vector<void *> allocs;
    DevScalars *h_sc = nullptr;      // pinned mirror for scalar reads
    int *d_active = nullptr;         // run-loop gate
    int *d_max_cycles = nullptr;
    int *h_stage = nullptr;          // pinned staging ints
    double *h_state = nullptr;       // mapped pinned buffer for the state of a small mesh, else null
    // What the host wrote into a pair field, null once a cycle has written the
    // field: the accessors give a double back as it came, not to a pair's 48
    // bits and range.
    std::unique_ptr<double[]> written[kPairFields];
    // run loop
    cudaGraphExec_t run_exec = nullptr;
    int run_mode = 0;                // 0 not built, 1 conditional while node, 2 host-driven chunks
    cudaGraphExec_t chunk_exec = nullptr;
    int status = LULESH_OK;          // sticky step error
    long long launches = 0;
    long origin = 0;                 // element holding the initial energy
    std::vector<int> regions;        // LULESH 2.0 region number per element (empty: none)
    int *d_mat_order = nullptr, *d_reps = nullptr;
    std::string err;
};

namespace {

// States of up to so many bytes pass through the pinned buffer when the host's
// arrays are pageable (s <= 25): the copy into the buffer takes ~35 us per MB,
// eleven copies from or to pageable arrays 90-110 us, and at 2.5 MB (s=30) the
// two are even.
constexpr size_t kStagedState = 1536 << 10;
constexpr int kChunkCycles = 16;     // cycles per graph in the host-driven fallback
constexpr int kUnroll = 4;           // cycles per pass of the while node, on meshes of up to
constexpr long kSmallElems = 150000; // so many elements
thread_local std::string g_err;

}  // namespace

void lulesh::set_last_error(const std::string &msg) { g_err = msg; }

namespace {

int fail(lulesh_ctx *c, int code, const std::string &msg)
{
    if (c) c->err = msg;
    else g_err = msg;
    return code;
}

#define CK(call)                                                                          \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess)                                                            \
            return fail(ctx, LULESH_ERR_CUDA,                                             \
                        std::string(#call) + ": " + cudaGetErrorString(e_));              \
    } while (0)

template <typename T>
int dalloc(lulesh_ctx *ctx, T **p, size_t n)
{
    void *q = nullptr;
    if (n == 0) n = 1;
    cudaError_t e = cudaMalloc(&q, n * sizeof(T));
    if (e != cudaSuccess)
        return fail(ctx, LULESH_ERR_CUDA, std::string("cudaMalloc: ") + cudaGetErrorString(e));
    ctx->allocs.push_back(q);
    *p = static_cast<T *>(q);
    return LULESH_OK;
}

struct FieldRef {
    const char *name;
    double *Dom::*member;
    bool node;
};

const FieldRef kFields[] = {
    {"x", &Dom::x, true},   {"y", &Dom::y, true},   {"z", &Dom::z, true},
    {"xd", &Dom::xd, true}, {"yd", &Dom::yd, true}, {"zd", &Dom::zd, true},
    {"fx", &Dom::fx, true}, {"fy", &Dom::fy, true}, {"fz", &Dom::fz, true},
    {"e", &Dom::e, false},  {"p", &Dom::p, false},  {"q", &Dom::q, false},
    {"ql", &Dom::ql, false}, {"qq", &Dom::qq, false}, {"v", &Dom::v, false},
    {"vnew", &Dom::vnew, false}, {"delv", &Dom::delv, false}, {"vdov", &Dom::vdov, false},
    {"arealg", &Dom::arealg, false}, {"ss", &Dom::ss, false},
    {"delv_xi", &Dom::delv_xi, false}, {"delv_eta", &Dom::delv_eta, false},
    {"delv_zeta", &Dom::delv_zeta, false}, {"delx_xi", &Dom::delx_xi, false},
    {"delx_eta", &Dom::delx_eta, false}, {"delx_zeta", &Dom::delx_zeta, false},
};

// Read-only mesh fields reachable by name.
double *const_field(lulesh_ctx *ctx, const char *name, bool *node)
{
    if (!strcmp(name, "volo")) { *node = false; return const_cast<double *>(ctx->dom.volo); }
    if (!strcmp(name, "elemMass")) { *node = false; return const_cast<double *>(ctx->dom.elem_mass); }
    if (!strcmp(name, "nodalMass")) { *node = true; return const_cast<double *>(ctx->dom.nodal_mass); }
    return nullptr;
}

double *find_field(lulesh_ctx *ctx, const char *name, bool *node, bool *writable)
{
    for (const FieldRef &f : kFields)
        if (!strcmp(name, f.name)) {
            *node = f.node;
            *writable = true;
            return ctx->dom.*(f.member);
        }
    *writable = false;
    return const_field(ctx, name, node);
}

// Status of the step after the stream drained: the first error site in
// program order wins (see ErrSite).
int read_status(lulesh_ctx *ctx)
{
    CK(cudaMemcpyAsync(ctx->h_sc, ctx->dom.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (ctx->h_sc->err_any) {
        static const int code[ERR_NUM] = {LULESH_VOLUME_ERROR, LULESH_VOLUME_ERROR, LULESH_VOLUME_ERROR,
                                          LULESH_QSTOP_ERROR, LULESH_VOLUME_ERROR};
        static const char *what[ERR_NUM] = {"IntegrateStressForElems: determ <= 0",
                                            "CalcHourglassControlForElems: v <= 0",
                                            "CalcLagrangeElements: vnew <= 0",
                                            "CalcQForElems: q > qstop",
                                            "ApplyMaterialPropertiesForElems: v <= 0"};
        for (int i = 0; i < ERR_NUM; ++i)
            if (ctx->h_sc->err[i]) {
                ctx->status = code[i];
                char buf[160];
                snprintf(buf, sizeof buf, "%s (element %d, cycle %d)", what[i], ctx->h_sc->err[i] - 1,
                         ctx->h_sc->cycle);
                ctx->err = buf;
                return code[i];
            }
    }
    return LULESH_OK;
}

// After cycles (the last of them perhaps stopped by an error) and read_status:
// the kinematics kernel has written the pair fields, unless the only cycle's
// force kernel stopped it.
void drop_written(lulesh_ctx *ctx, int cycles)
{
    const DevScalars *h = ctx->h_sc;
    const bool stopped = h->err_any && (h->err[ERR_K1_DETERM] || h->err[ERR_K1_VOLUME]);
    if (cycles < 1 || (cycles == 1 && stopped)) return;
    for (auto &w : ctx->written) w.reset();
}

// A run loop that ended with time < stoptime although the caller's own cap
// was not reached: the cycle budget ran out, or the time step stopped being
// positive.  Reported, not sticky: the state is valid and a further run
// continues from it.  Reads the scalars read_status just fetched.
int short_of_stoptime(lulesh_ctx *ctx, int max_cycles, int done)
{
    const DevScalars *h = ctx->h_sc;
    if (!(h->time < ctx->dom.prm.stoptime)) return LULESH_OK;
    if (max_cycles > 0 && max_cycles <= kRunCycleLimit && done >= max_cycles) return LULESH_OK;
    char buf[200];
    snprintf(buf, sizeof buf, "run stopped at time %.17g < stoptime %.17g after %d cycles: %s", h->time,
             ctx->dom.prm.stoptime, done,
             h->deltatime > 0.0 ? "the cycle budget (LULESH_RUN_CYCLE_BUDGET) ran out"
                                : "the time step is no longer positive");
    ctx->err = buf;
    return LULESH_ERR_TIMEOUT;
}

int check_launch(lulesh_ctx *ctx)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(ctx, LULESH_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
    return LULESH_OK;
}

// Clears the errors after the host replaced a field.
int clear_errors(lulesh_ctx *ctx)
{
    ScalarSet set{};
    set.moved = true;   // it may have been positions
    launch_set_scalars(ctx->dom.sc, set, ctx->stream);
    int rc = check_launch(ctx);
    if (rc) return rc;
    ctx->status = LULESH_OK;
    return LULESH_OK;
}

int upload(lulesh_ctx *ctx, double *dst, const double *src, long n)
{
    if (!src) return LULESH_OK;
    CK(cudaMemcpyAsync(dst, src, n * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    return LULESH_OK;
}

int download(lulesh_ctx *ctx, double *dst, const double *src, long n)
{
    if (!dst) return LULESH_OK;
    CK(cudaMemcpyAsync(dst, src, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    return LULESH_OK;
}

bool is_split(const lulesh_ctx *ctx) { return ctx->precision == LULESH_PRECISION_SPLIT; }

// After the host replaced FP64 node state, refresh the split path's hi/lo
// copies (nothing to do on the FP64 paths), and wait for all of it.
int refresh_split(lulesh_ctx *ctx)
{
    if (is_split(ctx)) {
        launch_split_sync(ctx->dom, ctx->stream);
        int rc = check_launch(ctx);
        if (rc) return rc;
    }
    CK(cudaStreamSynchronize(ctx->stream));
    return LULESH_OK;
}

// The fields of the Domain record in the order of the ABI's arguments.
StateView state_view(const Dom &d, const double *const host[11])
{
    StateView v{{d.x, d.y, d.z, d.xd, d.yd, d.zd, d.e, d.p, d.q, d.v, d.ss}, d.nn, d.ne, 0};
    for (int f = 0; f < 11; ++f) v.present |= (host[f] ? 1u : 0u) << f;
    return v;
}
size_t field_len(const StateView &v, int f) { return f < 6 ? v.nn : v.ne; }

// What the driver knows about a host array.  The runtime tells pinned memory
// from pageable; the extent of the piece that an address lies in, and whether
// a kernel may write it, only the driver API tells.
HostArray describe(const double *p, size_t n)
{
    HostArray a{reinterpret_cast<uintptr_t>(p), n * sizeof(double), HostMemory::kOther, 0, 0, 0, false};
    if (!p) return a;
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
        cudaGetLastError();
        return a;
    }
    if (attr.type == cudaMemoryTypeUnregistered) a.memory = HostMemory::kPageable;
    if (attr.type != cudaMemoryTypeHost) return a;
    a.memory = HostMemory::kPinned;
    using Query = CUresult (*)(unsigned, CUpointer_attribute *, void **, CUdeviceptr);
    static const Query query = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &found);
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess && found == cudaDriverEntryPointSuccess ? reinterpret_cast<Query>(f) : nullptr;
    }();
    CUdeviceptr start = 0;
    size_t bytes = 0;
    unsigned access = 0;
    CUpointer_attribute what[3] = {CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE,
                                   CU_POINTER_ATTRIBUTE_ACCESS_FLAGS};
    void *to[3] = {&start, &bytes, &access};
    // the range is of device addresses, which start where the piece does
    if (!query || query(3, what, to, reinterpret_cast<CUdeviceptr>(attr.devicePointer)) != CUDA_SUCCESS) return a;
    a.device = reinterpret_cast<uintptr_t>(attr.devicePointer);
    a.piece = a.at - (a.device - static_cast<uintptr_t>(start));
    a.piece_bytes = bytes;
    a.writable = access == CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE;
    return a;
}

Crossing crossing_of(const lulesh_ctx *ctx, const StateView &v, const double *const host[11], bool to_host, HostState *direct)
{
    HostArray a[11];
    for (int f = 0; f < 11; ++f) {
        a[f] = describe(host[f], field_len(v, f));
        direct->field[f] = reinterpret_cast<double *>(a[f].device);
    }
    return crossing(a, 11, to_host, ctx->h_state != nullptr);
}

void nodal(lulesh_ctx *ctx, const Dom &d)
{
    if (is_split(ctx)) launch_lagrange_nodal_split(d, ctx->stream);
    else launch_lagrange_nodal(d, ctx->stream);
}

void elements(lulesh_ctx *ctx, const Dom &d, const CycleEnd *end)
{
    if (is_split(ctx)) launch_lagrange_elements_split(d, ctx->stream, end);
    else launch_lagrange_elements(d, ctx->stream, end);
}

void run_body(lulesh_ctx *ctx, const Dom &d, cudaGraphConditionalHandle h)
{
    if (is_split(ctx)) launch_run_body_split(d, ctx->stream, h, ctx->d_active);
    else launch_run_body(d, ctx->stream, h, ctx->d_active);
}

// Cycles per pass of the while node.  A pass costs the node's own turn-round,
// 3-4 us, which on a small mesh is a noticeable part of a cycle (s=10 39.6 ->
// 36.5 us with four cycles, 36.1 with eight); the cycles after the
// first return at once when the run has ended, which is cheap there.  On a
// large mesh neither is worth having: one cycle per pass.
int body_cycles(const lulesh_ctx *ctx) { return ctx->ne <= kSmallElems ? kUnroll : 1; }

// Build the run-loop graph: prologue -> while(cond) { a few cycles }.  Falls
// back to a host-driven graph of kChunkCycles gated cycles when conditional
// nodes are not available.
int build_run_graph(lulesh_ctx *ctx)
{
    if (ctx->run_mode) return LULESH_OK;
    cudaGraph_t g = nullptr;
    cudaGraphConditionalHandle h = 0;
    bool ok = cudaGraphCreate(&g, 0) == cudaSuccess &&
              cudaGraphConditionalHandleCreate(&h, g, 0, 0) == cudaSuccess;
    if (ok) {
        // prologue, captured into g
        ok = cudaStreamBeginCaptureToGraph(ctx->stream, g, nullptr, nullptr, 0,
                                           cudaStreamCaptureModeThreadLocal) == cudaSuccess;
        if (ok) {
            launch_run_prologue(ctx->dom, ctx->stream, ctx->d_max_cycles, h, ctx->d_active);
            ok = cudaStreamEndCapture(ctx->stream, &g) == cudaSuccess;
        }
        size_t nnodes = 0;
        cudaGraphNode_t prologue = nullptr;
        if (ok) ok = cudaGraphGetNodes(g, nullptr, &nnodes) == cudaSuccess && nnodes == 1;
        if (ok) ok = cudaGraphGetNodes(g, &prologue, &nnodes) == cudaSuccess;
        cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t cnode = nullptr;
        if (ok) ok = cudaGraphAddNode(&cnode, g, &prologue, nullptr, 1, &cp) == cudaSuccess;
        if (ok) {
            cudaGraph_t body = cp.conditional.phGraph_out[0];
            ok = cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0,
                                               cudaStreamCaptureModeThreadLocal) == cudaSuccess;
            if (ok) {
                Dom d = ctx->dom;
                for (int i = 0; i < body_cycles(ctx); ++i) {
                    d.gate = i ? ctx->d_active : nullptr;
                    run_body(ctx, d, h);
                }
                cudaGraph_t out = nullptr;
                ok = cudaStreamEndCapture(ctx->stream, &out) == cudaSuccess;
            }
        }
        if (ok) ok = cudaGraphInstantiate(&ctx->run_exec, g, 0) == cudaSuccess;
    }
    if (g) cudaGraphDestroy(g);
    if (ok) {
        ctx->run_mode = 1;
        return LULESH_OK;
    }
    // conditional nodes unavailable: clear the sticky error and capture the
    // gated fallback
    cudaGetLastError();
    cudaStreamCaptureStatus cs;
    if (cudaStreamIsCapturing(ctx->stream, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
        cudaGraph_t junk = nullptr;
        cudaStreamEndCapture(ctx->stream, &junk);
        if (junk) cudaGraphDestroy(junk);
    }
    cudaGetLastError();
    cudaGraph_t cg = nullptr;
    CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    Dom d = ctx->dom;
    d.gate = ctx->d_active;
    for (int i = 0; i < kChunkCycles; ++i) run_body(ctx, d, 0);
    CK(cudaStreamEndCapture(ctx->stream, &cg));
    cudaError_t e = cudaGraphInstantiate(&ctx->chunk_exec, cg, 0);
    cudaGraphDestroy(cg);
    if (e != cudaSuccess) return fail(ctx, LULESH_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
    ctx->run_mode = 2;
    return LULESH_OK;
}

}  // namespace

extern "C" {

const char *lulesh_last_error(const lulesh_ctx *ctx)
{
    return ctx ? ctx->err.c_str() : g_err.c_str();
}

void lulesh_destroy(lulesh_ctx *ctx)
{
    if (!ctx) return;
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    if (ctx->run_exec) cudaGraphExecDestroy(ctx->run_exec);
    if (ctx->chunk_exec) cudaGraphExecDestroy(ctx->chunk_exec);
    for (void *p : ctx->allocs) cudaFree(p);
    if (ctx->h_sc) cudaFreeHost(ctx->h_sc);
    if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
    if (ctx->h_state) cudaFreeHost(ctx->h_state);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}

}  // extern "C"

namespace {

// A context: stream, device arrays, initial state.  m null: the s^3 cube of
// a Sedov problem, set up on the device (mesh_gpu.cu); else that host mesh.
int create_context(const HostMesh *m, int s, int init_mode, int precision, const lulesh_params *params, lulesh_ctx **out)
{
    *out = nullptr;
    lulesh_ctx *ctx = new lulesh_ctx;
    int rc = LULESH_OK;
    auto bail = [&](int code) { g_err = ctx->err; lulesh_destroy(ctx); return code; };

    ctx->s = s;
    ctx->origin = m ? m->origin : 0;
    ctx->ne = m ? m->ne : (long)s * s * s;
    ctx->nn = m ? m->nn : (long)(s + 1) * (s + 1) * (s + 1);
    ctx->precision = precision;
    if (cudaGetDevice(&ctx->device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) {
        ctx->err = std::string("no usable CUDA device: ") + cudaGetErrorString(cudaGetLastError());
        return bail(LULESH_ERR_CUDA);
    }
    const size_t state = (6 * (size_t)ctx->nn + 5 * (size_t)ctx->ne) * sizeof(double);
    if (cudaMallocHost(&ctx->h_sc, sizeof(DevScalars)) != cudaSuccess ||
        cudaMallocHost(&ctx->h_stage, 16 * sizeof(int)) != cudaSuccess) {
        ctx->err = "cudaMallocHost failed";
        return bail(LULESH_ERR_CUDA);
    }
    // without the buffer states are copied field by field
    if (state <= kStagedState && cudaMallocHost(&ctx->h_state, state) != cudaSuccess) {
        ctx->h_state = nullptr;
        cudaGetLastError();
    }

    Dom &d = ctx->dom;
    d.s = s;
    d.ne = (int)ctx->ne;
    d.nn = (int)ctx->nn;
    d.keep = 0;
    lulesh_params prm;
    default_params(&prm);
    set_params(d, params ? *params : prm);
    {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device) != cudaSuccess || sms < 1)
            sms = 1;
        choose_blocks(d, sms);
    }
    const size_t ne = ctx->ne, nn = ctx->nn;
    d.df = arith_of(precision);
    d.gate = nullptr;

    // All arrays in one allocation.  The lists that a cube's kernels form
    // from the indices exist only for a mesh given by its lists.
    int *nodelist, *cstart = nullptr, *clist = nullptr, *ebc, *nb[6] = {};
    unsigned char *nbc;
    double *volo, *emass, *nmass;
    auto layout = [&](Slab &b) {
        b.take(nodelist, 8 * ne);
        if (m) {
            b.take(cstart, nn + 1);
            b.take(clist, 8 * ne);
            for (int *&l : nb) b.take(l, ne);
        }
        b.take(nbc, nn);
        b.take(ebc, ne);
        b.take(volo, ne);
        b.take(emass, ne);
        b.take(nmass, nn);
        for (double **f : {&d.x, &d.y, &d.z, &d.xd, &d.yd, &d.zd, &d.fx, &d.fy, &d.fz, &d.inv_mass}) b.take(*f, nn);
        for (double **f : {&d.e, &d.p, &d.q, &d.v, &d.ss, &d.vnew, &d.delv, &d.vdov, &d.arealg, &d.ql, &d.qq, &d.delv_xi,
                           &d.delv_eta, &d.delv_zeta, &d.delx_xi, &d.delx_eta, &d.delx_zeta, &d.inv_volo})
            b.take(*f, ne);
        if (precision != LULESH_PRECISION_SPLIT) {
            for (double **f : {&d.fcx, &d.fcy, &d.fcz}) b.take(*f, 8 * ne);
            b.take(d.geo, geo_words(d.df) * ne);
        } else {
            for (float **f : {&d.f32x, &d.f32y, &d.f32z}) b.take(*f, 8 * ne);
            for (float2 **f : {&d.xs, &d.ys, &d.zs, &d.xds, &d.yds, &d.zds}) b.take(*f, nn);
            b.take(d.gq, 6 * ne);
        }
        b.take(d.sc, 1);
        b.take(ctx->d_active, 1);
        b.take(ctx->d_max_cycles, 1);
    };
    Slab slab;
    layout(slab);
    if ((rc = dalloc(ctx, &slab.base, slab.used)) != LULESH_OK) return bail(rc);
    const size_t bytes = slab.used;
    slab.used = 0;
    layout(slab);
    d.nodelist = nodelist;
    d.corner_start = cstart;
    d.corner_list = clist;
    d.node_bc = nbc;
    d.lxim = nb[0]; d.lxip = nb[1]; d.letam = nb[2]; d.letap = nb[3]; d.lzetam = nb[4]; d.lzetap = nb[5];
    d.elem_bc = ebc;
    d.volo = volo; d.elem_mass = emass; d.nodal_mass = nmass;

    cudaStream_t st = ctx->stream;
    auto up = [&](void *dst, const void *src, size_t n) {
        return cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st) == cudaSuccess;
    };
    double e0, dt0;
    bool ok = cudaMemsetAsync(slab.base, 0, bytes, st) == cudaSuccess;
    std::vector<double> e, ones, inv_volo, inv_mass;
    std::vector<int> start, slots;
    if (m) {
        e0 = m->e0;
        dt0 = m->dt0;
        // node -> corner slots, translated from the reference's 8*elem+corner
        // numbering to the corner-major slot corner*ne + elem
        start.assign(m->node_elem_start.begin(), m->node_elem_start.end());
        start.push_back((int)(8 * ne));
        slots.resize(8 * ne);
        for (size_t i = 0; i < 8 * ne; ++i) {
            const int k = m->node_elem_corner_list[i];
            slots[i] = (k & 7) * (int)ne + (k >> 3);
        }
        ones.assign(ne, 1.0);
        e.assign(ne, 0.0);
        e[m->origin] = e0;
        inv_volo.resize(ne);
        inv_mass.resize(nn);
        for (size_t i = 0; i < ne; ++i) inv_volo[i] = 1.0 / m->volo[i];
        for (size_t i = 0; i < nn; ++i) inv_mass[i] = 1.0 / m->nodal_mass[i];
        ok = ok && up(nodelist, m->nodelist.data(), 8 * ne * 4) && up(cstart, start.data(), (nn + 1) * 4) &&
             up(clist, slots.data(), 8 * ne * 4) && up(nbc, m->node_bc.data(), nn) && up(ebc, m->elem_bc.data(), ne * 4) &&
             up(volo, m->volo.data(), ne * 8) && up(emass, m->elem_mass.data(), ne * 8) &&
             up(nmass, m->nodal_mass.data(), nn * 8) && up(d.inv_mass, inv_mass.data(), nn * 8) &&
             up(d.inv_volo, inv_volo.data(), ne * 8) && up(d.x, m->x.data(), nn * 8) && up(d.y, m->y.data(), nn * 8) &&
             up(d.z, m->z.data(), nn * 8) && up(d.e, e.data(), ne * 8) && up(d.v, ones.data(), ne * 8);
        const std::vector<int> *lists[6] = {&m->lxim, &m->lxip, &m->letam, &m->letap, &m->lzetam, &m->lzetap};
        for (int i = 0; i < 6; ++i) ok = ok && up(nb[i], lists[i]->data(), ne * 4);
    } else {
        sedov_start(s, init_mode, cube_corner_volume(s), &e0, &dt0);
        if (ok) {
            launch_build_cube(d, CubeDesc{s, 0, 0, e0}, st);
            ok = cudaGetLastError() == cudaSuccess;
        }
    }
    DevScalars *h = ctx->h_sc;
    memset(h, 0, sizeof *h);
    h->time = 0.0;
    h->deltatime = dt0;
    h->dtcourant = 1.0e+20;
    h->dthydro = 1.0e+20;
    h->cycle = 0;
    h->courant_key = ~0ULL;
    h->hydro_key = ~0ULL;
    ok = ok && up(d.sc, h, sizeof *h);
    if (ok && precision == LULESH_PRECISION_SPLIT) {
        launch_split_sync(d, st);
        ok = cudaGetLastError() == cudaSuccess;
    }
    ok = ok && cudaStreamSynchronize(st) == cudaSuccess;
    if (!ok) {
        ctx->err = std::string("lulesh_create upload: ") + cudaGetErrorString(cudaGetLastError());
        return bail(LULESH_ERR_CUDA);
    }
    *out = ctx;
    return LULESH_OK;
}

int check_precision(int precision, const char *who)
{
    if (precision != LULESH_PRECISION_FP64 && precision != LULESH_PRECISION_SPLIT &&
        precision != LULESH_PRECISION_FP64_IEEE)
        return fail(nullptr, LULESH_ERR_ARG, std::string(who) + ": unknown precision");
    return LULESH_OK;
}

}  // namespace

extern "C" {

int lulesh_create(int s, int init_mode, int precision, const lulesh_params *params, lulesh_ctx **out)
{
    if (!out || s < 1 || s > kMaxEdge) return fail(nullptr, LULESH_ERR_ARG, "lulesh_create: bad size or output pointer");
    if (init_mode != LULESH_INIT_V1 && init_mode != LULESH_INIT_V2)
        return fail(nullptr, LULESH_ERR_ARG, "lulesh_create: init_mode must be LULESH_INIT_V1 or LULESH_INIT_V2");
    if (int rc = check_precision(precision, "lulesh_create")) return rc;
    return create_context(nullptr, s, init_mode, precision, params, out);
}

int lulesh_create_unstructured(const lulesh_unstructured_mesh *mesh, int precision, const lulesh_params *params,
                               lulesh_ctx **out)
{
    if (!out || !mesh) return fail(nullptr, LULESH_ERR_ARG, "lulesh_create_unstructured: NULL argument");
    *out = nullptr;
    if (int rc = check_precision(precision, "lulesh_create_unstructured")) return rc;
    HostMesh m;
    std::string err;
    if (m.build_unstructured(*mesh, &err) != LULESH_OK) return fail(nullptr, LULESH_ERR_ARG, err);
    return create_context(&m, m.s, 0, precision, params, out);
}

int lulesh_create_lmesh(const char *path, int precision, const lulesh_params *params, lulesh_ctx **out)
{
    if (!out) return fail(nullptr, LULESH_ERR_ARG, "lulesh_create_lmesh: NULL output pointer");
    *out = nullptr;
    if (int rc = check_precision(precision, "lulesh_create_lmesh")) return rc;
    LmeshFile f;
    std::string err;
    if (f.read(path, &err) != LULESH_OK) return fail(nullptr, LULESH_ERR_ARG, err);
    return lulesh_create_unstructured(&f.view, precision, params, out);
}

int lulesh_dump_domain(lulesh_ctx *ctx, const char *basename, int step)
{
    if (!ctx) return LULESH_ERR_ARG;
    const size_t ne = ctx->ne, nn = ctx->nn;
    std::vector<double> node(6 * nn), elem(4 * ne);
    std::vector<int> nodelist(8 * ne);
    const Dom &d = ctx->dom;
    double *const ndst[6] = {d.x, d.y, d.z, d.xd, d.yd, d.zd};
    double *const edst[4] = {d.e, d.p, d.v, d.q};
    for (int i = 0; i < 6; ++i)
        CK(cudaMemcpyAsync(node.data() + i * nn, ndst[i], nn * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    for (int i = 0; i < 4; ++i)
        CK(cudaMemcpyAsync(elem.data() + i * ne, edst[i], ne * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaMemcpyAsync(nodelist.data(), d.nodelist, 8 * ne * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaMemcpyAsync(ctx->h_sc, d.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    const double *fields[10] = {node.data(), node.data() + nn, node.data() + 2 * nn, node.data() + 3 * nn,
                                node.data() + 4 * nn, node.data() + 5 * nn, elem.data(), elem.data() + ne,
                                elem.data() + 2 * ne, elem.data() + 3 * ne};
    std::string err;
    const int rc = write_domain_file(basename, ctx->s, (long)ne, (long)nn, nodelist.data(), step, ctx->h_sc->time,
                                     fields, &err);
    return rc ? fail(ctx, rc, "lulesh_dump_domain: " + err) : LULESH_OK;
}

int lulesh_origin_element(lulesh_ctx *ctx, long *elem)
{
    if (!ctx || !elem) return LULESH_ERR_ARG;
    *elem = ctx->origin;
    return LULESH_OK;
}

int lulesh_sizes(lulesh_ctx *ctx, int *s, long *num_elem, long *num_node)
{
    if (!ctx) return LULESH_ERR_ARG;
    if (s) *s = ctx->s;
    if (num_elem) *num_elem = ctx->ne;
    if (num_node) *num_node = ctx->nn;
    return LULESH_OK;
}

void *lulesh_stream(lulesh_ctx *ctx) { return ctx ? (void *)ctx->stream : nullptr; }

long long lulesh_kernel_launches(lulesh_ctx *ctx) { return ctx ? ctx->launches : 0; }

int lulesh_keep_forces(lulesh_ctx *ctx, int keep)
{
    if (!ctx) return LULESH_ERR_ARG;
    ctx->dom.keep = keep ? 3 : 0;
    // the run graph bakes in the kernel arguments: rebuild on next run
    if (ctx->run_exec) { cudaGraphExecDestroy(ctx->run_exec); ctx->run_exec = nullptr; }
    if (ctx->chunk_exec) { cudaGraphExecDestroy(ctx->chunk_exec); ctx->chunk_exec = nullptr; }
    ctx->run_mode = 0;
    return LULESH_OK;
}

int lulesh_set_regions(lulesh_ctx *ctx, int num_regions, int balance, int cost)
{
    if (!ctx) return LULESH_ERR_ARG;
    if (num_regions < 0 || balance < 0 || cost < 0 || cost > 100)
        return fail(ctx, LULESH_ERR_ARG, "lulesh_set_regions: need num_regions >= 0, balance >= 0, 0 <= cost <= 100");
    double weights = 0.0;
    for (int i = 0; i < num_regions; ++i) weights += std::pow(double(i + 1), double(balance));
    if (weights > 2147483647.0) return fail(ctx, LULESH_ERR_ARG, "lulesh_set_regions: region weights overflow int");
    // the run graph bakes in the kernel arguments: rebuild on next run
    if (ctx->run_exec) { cudaGraphExecDestroy(ctx->run_exec); ctx->run_exec = nullptr; }
    if (ctx->chunk_exec) { cudaGraphExecDestroy(ctx->chunk_exec); ctx->chunk_exec = nullptr; }
    ctx->run_mode = 0;
    if (num_regions == 0) {
        ctx->regions.clear();
        ctx->dom.mat_order = nullptr;
        ctx->dom.reps = nullptr;
        return LULESH_OK;
    }
    const long ne = ctx->ne;
    region_numbers(ne, num_regions, balance, ctx->regions);
    std::vector<int> reps(ne), order(ne);
    for (long k = 0; k < ne; ++k) {
        reps[k] = region_reps(ctx->regions[k] - 1, num_regions, cost);
        order[k] = (int)k;
    }
    // costliest elements first, element order within a cost: warps see one
    // repetition count and the longest ones start earliest
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return reps[a] > reps[b]; });
    int rc;
    if (!ctx->d_mat_order && (rc = dalloc(ctx, &ctx->d_mat_order, ne)) != LULESH_OK) return rc;
    if (!ctx->d_reps && (rc = dalloc(ctx, &ctx->d_reps, ne)) != LULESH_OK) return rc;
    CK(cudaMemcpyAsync(ctx->d_mat_order, order.data(), ne * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(ctx->d_reps, reps.data(), ne * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    ctx->dom.mat_order = ctx->d_mat_order;
    ctx->dom.reps = ctx->d_reps;
    return LULESH_OK;
}

int lulesh_get_regions(lulesh_ctx *ctx, int *reg_num_list)
{
    if (!ctx || !reg_num_list) return LULESH_ERR_ARG;
    for (long k = 0; k < ctx->ne; ++k) reg_num_list[k] = ctx->regions.empty() ? 1 : ctx->regions[k];
    return LULESH_OK;
}

int lulesh_set_params(lulesh_ctx *ctx, const lulesh_params *params)
{
    if (!ctx || !params) return LULESH_ERR_ARG;
    set_params(ctx->dom, *params);
    if (ctx->run_exec) { cudaGraphExecDestroy(ctx->run_exec); ctx->run_exec = nullptr; }
    if (ctx->chunk_exec) { cudaGraphExecDestroy(ctx->chunk_exec); ctx->chunk_exec = nullptr; }
    ctx->run_mode = 0;
    return LULESH_OK;
}

int lulesh_get_params(lulesh_ctx *ctx, lulesh_params *params)
{
    if (!ctx || !params) return LULESH_ERR_ARG;
    *params = ctx->dom.prm;
    return LULESH_OK;
}

int lulesh_upload_domain(lulesh_ctx *ctx, const double *x, const double *y, const double *z,
                         const double *xd, const double *yd, const double *zd, const double *e,
                         const double *p, const double *q, const double *v, const double *ss,
                         double time, double deltatime)
{
    if (!ctx) return LULESH_ERR_ARG;
    const Dom &d = ctx->dom;
    const double *const host[11] = {x, y, z, xd, yd, zd, e, p, q, v, ss};
    const StateView view = state_view(d, host);
    ScalarSet set{};
    set.time = time;
    set.deltatime = deltatime;
    set.clock = set.moved = true;
    int rc;
    HostState direct;
    const Crossing how = crossing_of(ctx, view, host, false, &direct);
    if (how == Crossing::kStaged) {
        double *at = ctx->h_state;
        for (int f = 0; f < 11; at += field_len(view, f++))
            if (host[f]) memcpy(at, host[f], field_len(view, f) * sizeof(double));
        launch_state_in(view, ctx->h_state, d.sc, set, ctx->stream);
    } else if (how == Crossing::kDirect) {
        launch_state_from_host(view, direct, d.sc, set, ctx->stream);
    } else {
        for (int f = 0; f < 11; ++f)
            if ((rc = upload(ctx, view.field[f], host[f], field_len(view, f)))) return rc;
        launch_set_scalars(d.sc, set, ctx->stream);
    }
    if ((rc = check_launch(ctx))) return rc;
    ctx->status = LULESH_OK;
    return refresh_split(ctx);
}

int lulesh_download_domain(lulesh_ctx *ctx, double *x, double *y, double *z, double *xd, double *yd,
                           double *zd, double *e, double *p, double *q, double *v, double *ss,
                           double *time, double *deltatime)
{
    if (!ctx) return LULESH_ERR_ARG;
    const Dom &d = ctx->dom;
    double *const host[11] = {x, y, z, xd, yd, zd, e, p, q, v, ss};
    const StateView view = state_view(d, host);
    int rc;
    HostState direct;
    const Crossing how = crossing_of(ctx, view, host, true, &direct);
    if (how == Crossing::kStaged) {
        launch_state_out(view, ctx->h_state, d.sc, ctx->h_sc, ctx->stream);
        if ((rc = check_launch(ctx))) return rc;
    } else if (how == Crossing::kDirect) {
        launch_state_to_host(view, direct, d.sc, ctx->h_sc, ctx->stream);
        if ((rc = check_launch(ctx))) return rc;
    } else {
        for (int f = 0; f < 11; ++f)
            if ((rc = download(ctx, host[f], view.field[f], field_len(view, f)))) return rc;
        CK(cudaMemcpyAsync(ctx->h_sc, d.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, ctx->stream));
    }
    CK(cudaStreamSynchronize(ctx->stream));
    if (how == Crossing::kStaged) {
        const double *at = ctx->h_state;
        for (int f = 0; f < 11; at += field_len(view, f++))
            if (host[f]) memcpy(host[f], at, field_len(view, f) * sizeof(double));
    }
    if (time) *time = ctx->h_sc->time;
    if (deltatime) *deltatime = ctx->h_sc->deltatime;
    return LULESH_OK;
}

int lulesh_get_scalars(lulesh_ctx *ctx, lulesh_scalars *out)
{
    if (!ctx || !out) return LULESH_ERR_ARG;
    CK(cudaMemcpyAsync(ctx->h_sc, ctx->dom.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    out->time = ctx->h_sc->time;
    out->deltatime = ctx->h_sc->deltatime;
    out->dtcourant = ctx->h_sc->dtcourant;
    out->dthydro = ctx->h_sc->dthydro;
    out->cycle = ctx->h_sc->cycle;
    return LULESH_OK;
}

int lulesh_set_scalars(lulesh_ctx *ctx, const lulesh_scalars *in)
{
    if (!ctx || !in) return LULESH_ERR_ARG;
    launch_set_scalars(ctx->dom.sc, ScalarSet{in->time, in->deltatime, in->dtcourant, in->dthydro, in->cycle, true, true, false},
                       ctx->stream);
    if (int rc = check_launch(ctx)) return rc;
    CK(cudaStreamSynchronize(ctx->stream));
    ctx->status = LULESH_OK;
    return LULESH_OK;
}

int lulesh_get_field(lulesh_ctx *ctx, const char *name, double *host, long n)
{
    if (!ctx || !name || !host) return LULESH_ERR_ARG;
    bool node = false, writable = false;
    double *f = find_field(ctx, name, &node, &writable);
    if (!f) return fail(ctx, LULESH_ERR_ARG, std::string("unknown field ") + name);
    if (n != (node ? ctx->nn : ctx->ne)) return fail(ctx, LULESH_ERR_ARG, std::string("wrong length for field ") + name);
    if (is_split(ctx)) {
        // the split path keeps the monotonic-Q gradients in FP32
        static const char *gnames[6] = {"delv_xi", "delv_eta", "delv_zeta", "delx_xi", "delx_eta", "delx_zeta"};
        for (int g = 0; g < 6; ++g)
            if (!strcmp(name, gnames[g])) {
                std::vector<float> tmp((size_t)n);
                CK(cudaMemcpyAsync(tmp.data(), ctx->dom.gq + (size_t)g * ctx->ne, n * sizeof(float),
                                   cudaMemcpyDeviceToHost, ctx->stream));
                CK(cudaStreamSynchronize(ctx->stream));
                for (long i = 0; i < n; ++i) host[i] = tmp[(size_t)i];
                return LULESH_OK;
            }
    }
    const int pair = ctx->dom.df == kArithDF64 ? pair_field(name) : -1;
    if (pair >= 0 && ctx->written[pair]) {
        CK(cudaMemcpyAsync(host, ctx->written[pair].get(), n * sizeof(double), cudaMemcpyDefault, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        return LULESH_OK;
    }
    if (pair >= 0) {
        // through the corner forces' array, which holds nothing between calls
        launch_pairs_to_doubles(f, ctx->dom.fcx, n, ctx->stream);
        if (int rc = check_launch(ctx)) return rc;
        f = ctx->dom.fcx;
    }
    CK(cudaMemcpyAsync(host, f, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return LULESH_OK;
}

int lulesh_set_field(lulesh_ctx *ctx, const char *name, const double *host, long n)
{
    if (!ctx || !name || !host) return LULESH_ERR_ARG;
    bool node = false, writable = false;
    double *f = find_field(ctx, name, &node, &writable);
    if (!f) return fail(ctx, LULESH_ERR_ARG, std::string("unknown field ") + name);
    if (n != (node ? ctx->nn : ctx->ne)) return fail(ctx, LULESH_ERR_ARG, std::string("wrong length for field ") + name);
    const int pair = ctx->dom.df == kArithDF64 ? pair_field(name) : -1;
    CK(cudaMemcpyAsync(pair >= 0 ? ctx->dom.fcx : f, host, n * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    if (pair >= 0) {
        std::unique_ptr<double[]> &kept = ctx->written[pair];
        if (!kept) kept.reset(new (std::nothrow) double[n]);
        if (!kept) return fail(ctx, LULESH_ERR_ARG, std::string("no host memory for field ") + name);
        CK(cudaMemcpyAsync(kept.get(), ctx->dom.fcx, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        launch_doubles_to_pairs(ctx->dom.fcx, f, n, ctx->stream);
        if (int rc = check_launch(ctx)) return rc;
    }
    int rc = clear_errors(ctx);
    return rc ? rc : refresh_split(ctx);
}

int lulesh_time_increment(lulesh_ctx *ctx)
{
    if (!ctx) return LULESH_ERR_ARG;
    if (ctx->status) return ctx->status;
    launch_time_increment(ctx->dom, ctx->stream);
    ctx->launches += 1;
    // TimeIncrement has no error exit of its own and every other call reads
    // the status when it returns, so this one does not wait for the GPU
    return check_launch(ctx);
}

int lulesh_lagrange_nodal(lulesh_ctx *ctx)
{
    if (!ctx) return LULESH_ERR_ARG;
    if (ctx->status) return ctx->status;
    nodal(ctx, ctx->dom);
    ctx->launches += 2;
    int rc = check_launch(ctx);
    return rc ? rc : read_status(ctx);
}

int lulesh_lagrange_elements(lulesh_ctx *ctx)
{
    if (!ctx) return LULESH_ERR_ARG;
    if (ctx->status) return ctx->status;
    elements(ctx, ctx->dom, nullptr);
    ctx->launches += 2;
    int rc = check_launch(ctx);
    if (rc) return rc;
    rc = read_status(ctx);
    drop_written(ctx, 1);
    return rc;
}

int lulesh_calc_time_constraints(lulesh_ctx *ctx)
{
    if (!ctx) return LULESH_ERR_ARG;
    if (ctx->status) return ctx->status;
    launch_time_constraints(ctx->dom, ctx->stream);
    ctx->launches += 2;
    int rc = check_launch(ctx);
    return rc ? rc : read_status(ctx);
}

int lulesh_lagrange_leapfrog(lulesh_ctx *ctx)
{
    if (!ctx) return LULESH_ERR_ARG;
    if (ctx->status) return ctx->status;
    nodal(ctx, ctx->dom);
    const CycleEnd end{};
    elements(ctx, ctx->dom, &end);
    ctx->launches += 5;
    int rc = check_launch(ctx);
    if (rc) return rc;
    rc = read_status(ctx);
    drop_written(ctx, 1);
    return rc;
}

int lulesh_run(lulesh_ctx *ctx, int max_cycles, int *cycles_done)
{
    if (!ctx) return LULESH_ERR_ARG;
    if (cycles_done) *cycles_done = 0;
    if (ctx->status) return ctx->status;
    int rc = build_run_graph(ctx);
    if (rc) return rc;
    ctx->h_stage[0] = max_cycles;
    CK(cudaMemcpyAsync(ctx->d_max_cycles, ctx->h_stage, sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
    if (ctx->run_mode == 1) {
        CK(cudaGraphLaunch(ctx->run_exec, ctx->stream));
    } else {
        launch_run_prologue(ctx->dom, ctx->stream, ctx->d_max_cycles, 0, ctx->d_active);
        if ((rc = check_launch(ctx))) return rc;
        for (;;) {
            CK(cudaGraphLaunch(ctx->chunk_exec, ctx->stream));
            CK(cudaMemcpyAsync(ctx->h_stage + 1, ctx->d_active, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
            CK(cudaStreamSynchronize(ctx->stream));
            if (!ctx->h_stage[1]) break;
        }
    }
    rc = read_status(ctx);
    const int done = ctx->h_sc->run_cycles;
    drop_written(ctx, done);
    if (cycles_done) *cycles_done = done;
    ctx->launches += 1 + (long long)done * kernels_per_cycle();
    return rc ? rc : short_of_stoptime(ctx, max_cycles, done);
}

int lulesh_run_profiled(lulesh_ctx *ctx, int max_cycles, int *cycles_done, double *kernel_ms)
{
    if (!ctx) return LULESH_ERR_ARG;
    if (cycles_done) *cycles_done = 0;
    if (kernel_ms)
        for (int i = 0; i < kTimedKernels; ++i) kernel_ms[i] = 0.0;
    if (ctx->status) return ctx->status;
    cudaEvent_t ev[kTimedKernels + 1];
    for (auto &e : ev) CK(cudaEventCreate(&e));
    const int cap = (max_cycles > 0 && max_cycles < kRunCycleLimit) ? max_cycles : kRunCycleLimit;
    int done = 0, rc = LULESH_OK;
    Dom d = ctx->dom;
    d.gate = nullptr;
    for (;;) {
        if ((rc = read_status(ctx))) break;
        const DevScalars *h = ctx->h_sc;
        if (!(h->time < d.prm.stoptime) || !(h->deltatime > 0.0) || done >= cap) break;
        if (is_split(ctx)) launch_cycle_timed_split(d, ctx->stream, ev);
        else launch_cycle_timed(d, ctx->stream, ev);
        if ((rc = check_launch(ctx))) break;
        CK(cudaEventSynchronize(ev[kTimedKernels]));
        for (int i = 0; i < kTimedKernels && kernel_ms; ++i) {
            float ms = 0.f;
            CK(cudaEventElapsedTime(&ms, ev[i], ev[i + 1]));
            kernel_ms[i] += ms;
        }
        ++done;
        ctx->launches += kTimedKernels;
    }
    for (auto &e : ev) cudaEventDestroy(e);
    if (!rc) rc = read_status(ctx);
    drop_written(ctx, done);
    if (cycles_done) *cycles_done = done;
    return rc ? rc : short_of_stoptime(ctx, max_cycles, done);
}

int lulesh_probe_fp64_peak(double *tflops)
{
    lulesh_ctx *ctx = nullptr;
    if (!tflops) return LULESH_ERR_ARG;
    int dev = 0, sms = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    double *out = nullptr;
    CK(cudaMalloc(&out, sizeof(double)));
    cudaStream_t st;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    cudaEvent_t a, b;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    const int threads = 256, blocks = sms * 8, iters = 4096;
    launch_fp64_probe(out, blocks, threads, iters, st);   // warm-up
    CK(cudaEventRecord(a, st));
    launch_fp64_probe(out, blocks, threads, iters, st);
    CK(cudaEventRecord(b, st));
    CK(cudaEventSynchronize(b));
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, a, b));
    *tflops = 2.0 * 8.0 * (double)iters * threads * blocks / (ms * 1e-3) * 1e-12;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaStreamDestroy(st);
    cudaFree(out);
    return LULESH_OK;
}

int lulesh_probe_math(double errs[4])
{
    if (!errs) return LULESH_ERR_ARG;
    unsigned long long *keys = nullptr, h[4] = {0, 0, 0, 0};
    cudaStream_t st = nullptr;
    const int n = 1 << 20;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&keys, sizeof h) != cudaSuccess) {
        if (st) cudaStreamDestroy(st);
        return fail(nullptr, LULESH_ERR_CUDA, "lulesh_probe_math: no usable CUDA device");
    }
    cudaError_t e = cudaMemsetAsync(keys, 0, sizeof h, st);
    if (e == cudaSuccess) {
        launch_math_probe(keys, n, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, keys, sizeof h, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(keys);
    cudaStreamDestroy(st);
    if (e != cudaSuccess) return fail(nullptr, LULESH_ERR_CUDA, std::string("lulesh_probe_math: ") + cudaGetErrorString(e));
    for (int i = 0; i < 4; ++i) std::memcpy(&errs[i], &h[i], sizeof(double));
    return LULESH_OK;
}

int lulesh_probe_pairs(double errs[16])
{
    if (!errs) return LULESH_ERR_ARG;
    double *d = nullptr, h[16] = {};   // eight sums of squares, eight bit patterns
    cudaStream_t st = nullptr;
    const int n = 1 << 20;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess || cudaMalloc(&d, sizeof h) != cudaSuccess) {
        if (st) cudaStreamDestroy(st);
        return fail(nullptr, LULESH_ERR_CUDA, "lulesh_probe_pairs: no usable CUDA device");
    }
    cudaError_t e = cudaMemsetAsync(d, 0, sizeof h, st);
    if (e == cudaSuccess) {
        launch_pair_probe(d, reinterpret_cast<unsigned long long *>(d + 8), n, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof h, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    cudaStreamDestroy(st);
    if (e != cudaSuccess) return fail(nullptr, LULESH_ERR_CUDA, std::string("lulesh_probe_pairs: ") + cudaGetErrorString(e));
    for (int j = 0; j < 8; ++j) {
        errs[2 * j] = std::sqrt(h[j] / n);
        errs[2 * j + 1] = h[8 + j];
    }
    return LULESH_OK;
}

int lulesh_probe_pipe_rates(double *rates)
{
    lulesh_ctx *ctx = nullptr;
    if (!rates) return LULESH_ERR_ARG;
    int dev = 0, sms = 0, clk_khz = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaDeviceGetAttribute(&clk_khz, cudaDevAttrClockRate, dev));
    const int threads = 256, blocks = sms * 8;
    float *out = nullptr;
    CK(cudaMalloc(&out, sizeof(float) * threads * blocks));
    double *dout = nullptr;
    CK(cudaMalloc(&dout, sizeof(double)));
    cudaStream_t st;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    cudaEvent_t a, b;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    // ops per thread of each probe: FFMA, DFMA, D2F (+DADD), DDIV
    const int iters[4] = {4096, 1024, 1024, 64};
    const double ops[4] = {8.0 * 4096, 8.0 * 1024, 8.0 * 1024, 4.0 * 64};
    for (int w = 0; w < 4; ++w) {
        for (int rep = 0; rep < 2; ++rep) {     // the first launch warms up
            CK(cudaEventRecord(a, st));
            if (w == 1) launch_fp64_probe(dout, blocks, threads, iters[w], st);
            else launch_rate_probe(w == 0 ? 0 : (w == 2 ? 1 : 2), out, blocks, threads, iters[w], st);
            CK(cudaEventRecord(b, st));
        }
        CK(cudaEventSynchronize(b));
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, a, b));
        // operations per SM per clock at the nominal maximum clock
        rates[w] = ops[w] * threads * blocks / (ms * 1e-3) / ((double)clk_khz * 1e3) / sms;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaStreamDestroy(st);
    cudaFree(out);
    cudaFree(dout);
    return LULESH_OK;
}

int lulesh_origin_energy(lulesh_ctx *ctx, double *e0)
{
    if (!ctx || !e0) return LULESH_ERR_ARG;
    CK(cudaMemcpyAsync(ctx->h_sc, ctx->dom.e + ctx->origin, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    memcpy(e0, ctx->h_sc, sizeof(double));
    return LULESH_OK;
}

int lulesh_symmetry(lulesh_ctx *ctx, double *max_abs_diff, double *total_abs_diff, double *max_rel_diff)
{
    if (!ctx) return LULESH_ERR_ARG;
    const int s = ctx->s;
    if (s < 1) return fail(ctx, LULESH_ERR_ARG, "lulesh_symmetry: the plane-0 test needs the cube mesh");
    std::vector<double> plane((size_t)s * s);
    CK(cudaMemcpyAsync(plane.data(), ctx->dom.e, plane.size() * sizeof(double), cudaMemcpyDeviceToHost,
                       ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    double ma = 0.0, ta = 0.0, mr = 0.0;
    for (int j = 0; j < s; ++j)
        for (int k = j + 1; k < s; ++k) {
            const double a = std::fabs(plane[(size_t)j * s + k] - plane[(size_t)k * s + j]);
            ta += a;
            if (ma < a) ma = a;
            const double r = a / plane[(size_t)k * s + j];
            if (mr < r) mr = r;
        }
    if (max_abs_diff) *max_abs_diff = ma;
    if (total_abs_diff) *total_abs_diff = ta;
    if (max_rel_diff) *max_rel_diff = mr;
    return LULESH_OK;
}

}  // extern "C"

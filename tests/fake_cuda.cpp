// A CUDA runtime and kernel launchers that do nothing but keep books, for CPU tests of the host layer (capi.cpp):
// device memory is host memory with a limit, a launch is counted and advances a clock by a cost the test sets, a
// graph is the list of launches made while a stream captured, and any call can be made to fail.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "adjoint.h"
#include "batch_params.h"
#include "noalloc.h"
#include "state_io.h"
#include "step_pair.h"
#include "step_params.h"
#include "surface.h"

using namespace mrlbm;

namespace {
enum Kind { STEP = 0, PAIR, BATCH, OTHER, KINDS };
struct Launch { Kind kind; double us; std::vector<const void*> mem; };
struct Graph { std::vector<Launch> nodes; };

std::map<char*, size_t> live;
size_t used = 0, peak = 0, limit = (size_t)1 << 60;
std::map<std::string, std::pair<int, int>> failing; // call -> calls that still succeed, then times it fails
double now = 0.0, step_us[N_ALL_CFGS], pair_us = 1.0, batch_us = 1e9, graph_factor = 1.0;
long long done[KINDS], dangling = 0, captures = 0, graphs = 0;
Graph* capture = nullptr;
cudaError_t last = cudaSuccess;

bool is_live(const void* p) {
    auto it = live.upper_bound((char*)p);
    return it != live.begin() && (char*)p < (--it)->first + it->second;
}
cudaError_t report(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
bool fails(const char* call) {
    auto it = failing.find(call);
    if (it == failing.end() || it->second.second == 0) return false;
    if (it->second.first > 0) return --it->second.first, false;
    --it->second.second;
    return true;
}
void run(const Launch& l, double factor = 1.0) {
    ++done[l.kind];
    now += factor * l.us;
    for (const void* p : l.mem)
        if (!is_live(p)) ++dangling;
}
int launch(Kind kind, double us, std::vector<const void*> mem) {
    if (fails("launch") || (kind == PAIR && fails("pair"))) return -1;
    Launch l{kind, us, std::move(mem)};
    if (capture) capture->nodes.push_back(l);
    else run(l);
    return 0;
}
}  // namespace

extern "C" {
// ---- the tests' controls
void fake_reset() {
    failing.clear();
    limit = (size_t)1 << 60;
    peak = used;
    for (double& u : step_us) u = 1.0;
    pair_us = 1.0;
    batch_us = 1e9;
    graph_factor = 1.0;
    std::fill(done, done + KINDS, 0);
    dangling = captures = graphs = 0;
}
void fake_fail(const char* call, int times) { failing[call] = {0, times}; }
void fake_fail_after(const char* call, int calls, int times) { failing[call] = {calls, times}; }
void fake_mark() { peak = used; }
void fake_limit(int64_t bytes) { limit = (size_t)bytes; }
int64_t fake_used() { return (int64_t)used; }
int64_t fake_peak() { return (int64_t)peak; }
void fake_step_us(int cfg, double us) { step_us[cfg] = us; }
void fake_pair_us(double us) { pair_us = us; }
void fake_graph_factor(double f) { graph_factor = f; }
int64_t fake_done(int kind) { return done[kind]; }
int64_t fake_captures() { return captures; }
int64_t fake_graphs() { return graphs; }
int64_t fake_dangling() { return dangling; }

// ---- the runtime
cudaError_t cudaMalloc(void** p, size_t n) {
    if (fails("cudaMalloc") || used + n > limit) return report(cudaErrorMemoryAllocation);
    *p = std::calloc(1, n ? n : 1);
    live[(char*)*p] = n ? n : 1;
    used += n;
    peak = std::max(peak, used);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    auto it = live.find((char*)p);
    if (it != live.end()) {
        used -= it->second;
        live.erase(it);
        std::free(p);
    }
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = limit - used; *t = limit; return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::calloc(1, n ? n : 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (fails("cudaMemcpyAsync")) return report(cudaErrorUnknown);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamCreate(cudaStream_t* s) { *s = (cudaStream_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return cudaStreamCreate(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)std::calloc(1, sizeof(double)); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { *(double*)e = now; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) { *ms = (float)((*(double*)b - *(double*)a) * 1e-3); return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    if (fails("cudaStreamBeginCapture")) return report(cudaErrorStreamCaptureUnsupported);
    capture = new Graph();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = (cudaGraph_t)capture;
    capture = nullptr;
    ++captures;
    if (fails("cudaStreamEndCapture")) {
        delete (Graph*)*g;
        *g = nullptr;
        return report(cudaErrorStreamCaptureInvalidated);
    }
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    if (fails("cudaGraphInstantiate")) return report(cudaErrorMemoryAllocation);
    *e = (cudaGraphExec_t) new Graph(*(Graph*)g);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph*)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete (Graph*)e; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    if (fails("cudaGraphLaunch")) return report(cudaErrorMemoryAllocation);
    ++graphs;
    for (const Launch& l : ((Graph*)e)->nodes) run(l, graph_factor);
    return cudaSuccess;
}
static CUresult encode_tiled(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                             const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    return CUDA_SUCCESS;
}
#undef cudaGetDriverEntryPoint
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *fn = (void*)encode_tiled;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
}  // extern "C"

// ---- the kernels' launchers
namespace mrlbm {
int launch_step_f64(const StepParams<double>& p, int cfg, void*, int) { return launch(STEP, step_us[cfg], {p.src, p.dst}); }
int launch_step_f32(const StepParams<float>& p, int cfg, void*, int) { return launch(STEP, step_us[cfg], {p.src, p.dst}); }
int launch_pair_f64(const StepParams<double>& a, const StepParams<double>& b, const PairPlan&, bool, void*) {
    return launch(PAIR, pair_us, {a.src, a.dst, b.src, b.dst});
}
int launch_pair_f32(const StepParams<float>& a, const StepParams<float>& b, const PairPlan&, bool, void*) {
    return launch(PAIR, pair_us, {a.src, a.dst, b.src, b.dst});
}
int launch_batch_f64(const BatchArgs<double>& a, int, int, bool, void*) { return launch(BATCH, batch_us * a.nsteps, {}); }
int launch_batch_f32(const BatchArgs<float>& a, int, int, bool, void*) { return launch(BATCH, batch_us * a.nsteps, {}); }
int launch_batch_split_f64(const BatchArgs<double>&, int, int, int, void*) { return launch(BATCH, batch_us, {}); }
int launch_batch_split_f32(const BatchArgs<float>&, int, int, int, void*) { return launch(BATCH, batch_us, {}); }
int batch_split_blocks_per_sm(int, int) { return 4; }
int batch_blocks_per_sm(int, int) { return 4; }
int launch_finish_record(const double*, int, int, int, double*, int, void*) { return launch(OTHER, 0.0, {}); }
int launch_face_f64(const StepParams<double>&, bool, void*) { return launch(OTHER, 0.0, {}); }
int launch_face_f32(const StepParams<float>&, bool, void*) { return launch(OTHER, 0.0, {}); }
int tma_ctas_per_sm(int, int) { return 1; }
void tma_box(int, int, int* w, int* h, int* st) { *w = 32; *h = 8; *st = 2; }
int launch_surface_f64(const StepParams<double>&, const SurfaceTables&, double*, double*, cudaStream_t) { return launch(OTHER, 0.0, {}); }
int launch_surface_f32(const StepParams<float>&, const SurfaceTables&, double*, double*, cudaStream_t) { return launch(OTHER, 0.0, {}); }
int launch_adjoint_step(const StepParams<double>& p, const adj::AdjArgs&, cudaStream_t) { return launch(OTHER, 0.0, {p.src}); }
int launch_adjoint_step(const StepParams<float>& p, const adj::AdjArgs&, cudaStream_t) { return launch(OTHER, 0.0, {p.src}); }
cudaError_t launch_scatter_state(int, const double*, void*, void*, const Layout&, int, int, int, const double*, cudaStream_t, int, int) {
    return cudaSuccess;
}
cudaError_t launch_gather_state(int, const void*, double*, const Layout&, int, int, int, const double*, cudaStream_t, int, int) {
    return cudaSuccess;
}
cudaError_t launch_field_stats_finalize(const double*, double*, int64_t, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_copy_ring(int, const void*, void*, const Layout&, cudaStream_t) { return cudaSuccess; }
int noalloc_step(NaCase&, void*, const double*, int32_t, double*, int32_t*, void*, std::string&) { return -1; }
}  // namespace mrlbm

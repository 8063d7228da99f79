// The CUDA runtime and the kernel launchers as far as the host runtime of one simulation
// (nofluidx3d_gb300/csrc/nfx_api.cpp) calls them, for tests of that runtime without a GPU: device
// memory is host memory, every call is counted, a chosen allocation fails, and a launch with a null
// pointer where its kernel would read or write is an error. No kernel is run.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>

#include "nfx_internal.h"

namespace {
enum Count { MALLOCS, QUERIES, TETS, NODES, SIS, RUNS, ADVANCES, GRAPHS, CAPTURES, RUN_STEPS, COUNTS };
long counts[COUNTS];
long fail_in = -1;  // allocations until one fails; -1: none
int run_tiles[2] = {0, 0};
bool busy = false, capturing = false;

// a launch on a stream that is being captured happens when the graph is launched, not now
cudaError_t launched(Count what, bool ok) {
    if (!ok) return cudaErrorInvalidValue;
    if (!capturing) counts[what]++;
    return cudaSuccess;
}
}  // namespace

extern "C" {
long fake_count(int what) { return counts[what]; }
void fake_reset() { std::memset(counts, 0, sizeof(counts)); }
void fake_fail_malloc(long nth) { fail_in = nth; }
void fake_run_tiles(int a, int b) {
    run_tiles[0] = a;
    run_tiles[1] = b;
}
void fake_busy(int b) { busy = b != 0; }

cudaError_t CUDARTAPI cudaMalloc(void** p, size_t n) {
    counts[MALLOCS]++;
    if (fail_in >= 0 && fail_in-- == 0) return cudaErrorMemoryAllocation;
    *p = std::calloc(n, 1);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t CUDARTAPI cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t CUDARTAPI cudaHostAlloc(void** p, size_t n, unsigned) { return (*p = std::calloc(n, 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t CUDARTAPI cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t CUDARTAPI cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t CUDARTAPI cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    if (!d || !s) return cudaErrorInvalidValue;
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t CUDARTAPI cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    return d ? (std::memset(d, v, n), cudaSuccess) : cudaErrorInvalidValue;
}
cudaError_t CUDARTAPI cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t CUDARTAPI cudaSetDevice(int) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetLastError() { return cudaSuccess; }
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t CUDARTAPI cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)std::malloc(1), cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamDestroy(cudaStream_t s) { return std::free(s), cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamQuery(cudaStream_t) { return counts[QUERIES]++, busy ? cudaErrorNotReady : cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return capturing = true, cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return capturing = false, *g = (cudaGraph_t)std::malloc(1), cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    return counts[CAPTURES]++, *e = (cudaGraphExec_t)std::malloc(1), cudaSuccess;
}
cudaError_t CUDARTAPI cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return counts[GRAPHS]++, cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphDestroy(cudaGraph_t g) { return std::free(g), cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphExecDestroy(cudaGraphExec_t e) { return std::free(e), cudaSuccess; }
cudaError_t CUDARTAPI cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)std::malloc(1), cudaSuccess; }
cudaError_t CUDARTAPI cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t CUDARTAPI cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
cudaError_t CUDARTAPI cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { return *t = 0.f, cudaSuccess; }
}  // extern "C"

namespace nfx {

cudaError_t launch_tet_pass(const MeshDev& m, const StateDev& s, const BatchDev& b, int model, int, cudaStream_t, bool) {
    return launched(TETS, m.lconn && m.tile_inc && s.ua && s.facc && b.cells && (model != MODEL_VP || (s.vp_a && s.vp_b && s.vp_c && s.fields)));
}
cudaError_t launch_si_pass(const MeshDev& m, const StateDev& s, const BatchDev& b, int, bool, int, cudaStream_t, bool) {
    return launched(SIS, m.Xh && s.facc && b.cells);
}
cudaError_t launch_node_pass(const MeshDev& m, const StateDev& s, const BatchDev& b, int, int, int, int, cudaStream_t, bool) {
    return launched(NODES, m.block_box && s.va && s.vb && b.cells && s.force_out);
}
cudaError_t launch_advance_time(const StateDev& s, long long, long long, long long, cudaStream_t) {
    return launched(ADVANCES, s.clock);
}
cudaError_t run_tiles_max(const MeshDev&, int, int (&tiles)[2]) {
    tiles[0] = run_tiles[0];
    tiles[1] = run_tiles[1];
    return cudaSuccess;
}
int run_tiles_bound(const MeshDev&) { return run_tiles[1]; }
cudaError_t launch_run(const MeshDev& m, const StateDev& s, const BatchDev& b, int, int, unsigned* count, unsigned,
                       unsigned long long* acc, int nsteps, cudaStream_t, unsigned) {
    counts[RUN_STEPS] += nsteps;
    return launched(RUNS, m.lconn && s.ua && b.cells && count && acc);
}
cudaError_t launch_divide_check(const float*, const float*, float*, long long, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_points_to_user(const MeshDev&, const StateDev&, const int* u, double* out, cudaStream_t) {
    return u && out ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t launch_points_from_user(const MeshDev&, const StateDev&, const int* u, const double* in, cudaStream_t) {
    return u && in ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t launch_vec_to_user(const MeshDev&, const float4* a, const float2* b, int, const int* u, double* out, cudaStream_t) {
    return a && b && u && out ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t launch_vec_from_user(const MeshDev&, float4* a, float2* b, int, const int* u, const double* in, cudaStream_t) {
    return a && b && u && in ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t launch_field_to_user(int64_t, const int* u, const float2* src, int, double* out, cudaStream_t) {
    return u && src && out ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t launch_plastic_to_user(int64_t, int64_t, const StateDev& s, const int* u, double* out, cudaStream_t) {
    return u && s.vp_a && s.vp_b && s.vp_c && out ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t launch_plastic_from_user(int64_t, int64_t, const StateDev& s, const int* u, const double* in, cudaStream_t) {
    return u && s.vp_a && s.vp_b && s.vp_c && in ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace nfx

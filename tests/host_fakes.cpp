// The CUDA runtime and the kernel launchers, faked on the host, so that the library's host code
// (csrc/ch4_host.cpp) runs without a GPU: device memory is host memory, copies and clears happen
// at once, launchers do nothing.  What a test asks about is written down:
//   fake_log()     one line per launch or clear
//   fake_faults()  one line per call whose result a GPU would not promise
//   fake_fail(f)   the next call of f returns an error
//
// Work on the legacy stream is not ordered with the library's non-blocking streams, and a clear, a
// copy between device buffers and the last part of a copy from pageable memory may be unfinished
// when the call returns: a launch or an ordered copy before the host has waited is a fault.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <string>

#include "../include/ch4.h"
#include "launch.h"

namespace {
std::string g_log, g_faults, g_fail;
int g_longest = 0;       // what the deposit reports as its longest row list
size_t g_refused = 0;    // allocations of this size and more are refused
bool g_pending = false;  // unfinished work on the legacy stream
int g_streams = 0;

cudaError_t ordered(const char* what, cudaStream_t st) {
  if (st && g_pending) g_faults += std::string(what) + " beside unfinished work of the legacy stream\n";
  if (!st) g_pending = true;
  if (g_fail == what) {
    g_fail.clear();
    return cudaErrorUnknown;
  }
  return cudaSuccess;
}
cudaError_t launched(const char* what, cudaStream_t st, const std::string& detail = "") {
  g_log += std::string(what) + (detail.empty() ? "" : " " + detail) + "\n";
  return ordered(what, st);
}
void need(const char* what, const void* p) {
  if (!p) g_faults += std::string(what) + ": null buffer\n";
}
}  // namespace

extern "C" {
const char* fake_log() { return g_log.c_str(); }
const char* fake_faults() { return g_faults.c_str(); }
void fake_fail(const char* f) { g_fail = f; }
void fake_refuse(size_t n) { g_refused = n; }
void fake_longest(int n) { g_longest = n; }
void fake_reset() { g_log.clear(), g_faults.clear(), g_fail.clear(); }

cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_refused && n >= g_refused) return cudaErrorMemoryAllocation;
  return (*p = std::calloc(1, n ? n : 1)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemset(void* p, int v, size_t n) {
  std::memset(p, v, n);
  return ordered("cudaMemset", nullptr);
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
  std::memset(p, v, n);
  g_log += "clear " + std::to_string(n) + "\n";
  return ordered("cudaMemsetAsync", st);
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  std::memcpy(d, s, n);
  g_pending = k != cudaMemcpyDeviceToHost;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  std::memcpy(d, s, n);
  return ordered("cudaMemcpyAsync", st);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned) {
  *st = reinterpret_cast<cudaStream_t>((size_t)++g_streams);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  if (!st) g_pending = false;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = reinterpret_cast<cudaEvent_t>(1), cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->multiProcessorCount = 1;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = *t = (size_t)1 << 34, cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "faked error"; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) { return *g = reinterpret_cast<cudaGraphExec_t>(1), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) { return ordered("cudaGraphLaunch", st); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

ch4_status ch4_averages_noalloc(const double*, const double*, const double*, const double*, int, int, int, int, int,
                                double, double, double*, void*) {
  return CH4_ERR_UNSUPPORTED;
}
}

namespace ch4 {
using S = cudaStream_t;
#define BOTH(F) F(double) F(float)
#define FAKES(A)                                                                                                       \
  cudaError_t launch_step(const StepParams<A>&, LaunchShape, S st) { return launched("launch_step", st); }             \
  cudaError_t launch_sism(const StepParams<A>&, S st) { return launched("launch_sism", st); }                          \
  cudaError_t launch_init_prev(const StepParams<A>&, LaunchShape, S st) { return launched("launch_init_prev", st); }   \
  cudaError_t launch_hydro(const StepParams<A>&, LaunchShape, const A*, const A*, const A*, double*, double*, double*, \
                           double*, double*, A*, S st, A*, int) {                                                      \
    return launched("launch_hydro", st);                                                                               \
  }                                                                                                                    \
  cudaError_t launch_fields_chunk(const StepParams<A>&, LaunchShape, const A*, const A*, const A*, int, int, int, A*,  \
                                  S st) {                                                                              \
    return launched("launch_fields_chunk", st);                                                                        \
  }                                                                                                                    \
  cudaError_t launch_force_moments(const StepParams<A>&, LaunchShape, const A*, int, double*, int, double,             \
                                   const double*, A*, S st, int) {                                                     \
    return launched("launch_force_moments", st);                                                                       \
  }                                                                                                                    \
  cudaError_t launch_aos_to_soa(const StepParams<A>&, LaunchShape, int, const A*, void*, int, int, S st) {             \
    return launched("launch_aos_to_soa", st);                                                                          \
  }                                                                                                                    \
  cudaError_t launch_soa_to_aos(const StepParams<A>&, LaunchShape, int, const void*, A*, int, int, S st) {             \
    return launched("launch_soa_to_aos", st);                                                                          \
  }                                                                                                                    \
  cudaError_t launch_particle_reorder(const PartParams<A>&, const PartPlanes&, unsigned int*, int*, void*, size_t&,    \
                                      int, S st) {                                                                     \
    return launched("launch_particle_reorder", st);                                                                    \
  }                                                                                                                    \
  cudaError_t launch_particle_substep(const PartParams<A>&, S st) { return launched("launch_particle_substep", st); }  \
  cudaError_t launch_particle_leave(const PartParams<A>&, double* down, double* up, int, int* keep, int* counts,       \
                                    S st) {                                                                            \
    need("launch_particle_leave", down), need("launch_particle_leave", keep), need("launch_particle_leave", counts);   \
    return launched("launch_particle_leave", st);                                                                      \
  }                                                                                                                    \
  cudaError_t launch_particle_arrive(const PartParams<A>&, const int*, int, const double* fd, int, const double*, int, \
                                     S st) {                                                                           \
    need("launch_particle_arrive", fd);                                                                                \
    return launched("launch_particle_arrive", st);                                                                     \
  }                                                                                                                    \
  cudaError_t launch_particle_reinject(const PartParams<A>&, const double*, S st) {                                    \
    return launched("launch_particle_reinject", st);                                                                   \
  }                                                                                                                    \
  cudaError_t launch_deposit_scratch(const PartParams<A>&, unsigned int*, int*, size_t& bytes) {                       \
    return bytes = 64, cudaSuccess;                                                                                    \
  }                                                                                                                    \
  cudaError_t launch_deposit(const PartParams<A>& P, unsigned int*, int*, void* tmp, size_t&, S st, int stage) {       \
    if (P.nsort > 0) need("launch_deposit", tmp);                                                                      \
    if (P.nsort > 0 && !P.rows) need("launch_deposit", P.cell_rng), need("launch_deposit", P.srec);                    \
    if (P.row_longest && (P.rows ? g_longest > row_limit(P.segs) : P.row_watch && g_longest > P.row_watch))            \
      *P.row_longest = g_longest;                                                                                      \
    return launched("launch_deposit", st, "stage " + std::to_string(stage) + (P.rows_ready ? " ready" : "") +          \
                                              (P.nsort > 0 && P.row_count && !P.rows ? " cells" : ""));                \
  }                                                                                                                    \
  cudaError_t launch_ghosts_out(const PartParams<A>&, double* down, double* up, int, int* counts, S st) {              \
    need("launch_ghosts_out", down), need("launch_ghosts_out", counts);                                                \
    return launched("launch_ghosts_out", st);                                                                          \
  }                                                                                                                    \
  cudaError_t launch_ghosts_in(const PartParams<A>&, const double* fd, const double*, int, S st) {                     \
    need("launch_ghosts_in", fd);                                                                                      \
    return launched("launch_ghosts_in", st);                                                                           \
  }
BOTH(FAKES)

cudaError_t launch_halo_faces(const HaloFacesArgs& a, size_t bytes, S st) {
  if (a.word < 2 || a.word > bytes || ((size_t)a.down | (size_t)a.up) % a.word) g_faults += "launch_halo_faces: word\n";
  return launched("launch_halo_faces", st, "word " + std::to_string(a.word));
}
cudaError_t launch_halo_copy(const HaloCopy&, S st) { return launched("launch_halo_copy", st); }
cudaError_t launch_particle_records(const double*, int, int, int, double*, S st) { return launched("launch_particle_records", st); }
cudaError_t launch_particle_averages(const double*, int, int, double*, int, double*, S st) {
  return launched("launch_particle_averages", st);
}
cudaError_t launch_averages(const AvgParams&, int, double*, S st) { return launched("launch_averages", st); }
cudaError_t launch_diag(const AvgParams&, int, int, double*, double*, S st) { return launched("launch_diag", st); }
cudaError_t launch_ensemble_step(const StepParams<float>*, const EnsTile*, int, int*, LaunchShape, int, int, S st) {
  return launched("launch_ensemble_step", st);
}
int ensemble_blocks_per_sm(LaunchShape, int) { return 1; }
}  // namespace ch4

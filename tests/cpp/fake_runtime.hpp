// The C calls' host side (ae_mpm_api.cu) on a CUDA runtime and a world of the tests' own.  Copies are host
// copies that count as in flight until their stream (or an event after them) is waited for.
#pragma once
#include <math.h>
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }

#include "../../ae-engine_b200/csrc/ae_mpm_api.cu"

namespace {
std::vector<int> priorities;      // of the worlds' streams, in order
int in_flight = 0, countdown = -1;  // the step that counts down to zero fails
bool fails() { return countdown >= 0 && countdown-- == 0; }

struct FakeWorld : aemp::WorldBase {
  ae_mpm_exec_opts o{};
  int bad(const char* what) {
    err = what;
    return AE_MPM_ECUDA;
  }
  int upload(uint32_t, const void*, uint64_t, bool) override { return ++in_flight, fails() ? bad("upload") : 0; }
  int download(uint32_t, void*, bool) override {
    if (fails()) return bad("download");
    in_flight = 0;
    return 0;
  }
  int upload_motion(const float*, const float*, const float*, uint64_t) override {
    return ++in_flight, fails() ? bad("upload_motion") : 0;
  }
  int download_motion(float*, float*) override { return ++in_flight, fails() ? bad("download_motion") : 0; }
  int upload_many(uint32_t, const uint32_t*, const ae_mpm_particles*, const uint64_t*, cudaStream_t) override { return 0; }
  int download_many(uint32_t, const uint32_t*, ae_mpm_particles*, cudaStream_t, bool) override { return 0; }
  int step(uint32_t) override { return ++in_flight, fails() ? bad("step") : 0; }
  int sync() override { return 0; }
  int totals(uint32_t, double*) override { return 0; }
  int errors(uint32_t, uint32_t*, uint64_t*) override { return 0; }
  int set_scene_params(uint32_t, const ae_mpm_scene_desc&) override { return 0; }
  int grid_download(uint32_t, float*, float*, uint64_t) override { return 0; }
  int snapshot(bool) override { return 0; }
  uint64_t last_launches() const override { return 0; }
  uint64_t particles() const override { return 0; }
  cudaStream_t stream() const override { return nullptr; }
  int set_stream_priority(int p) override { return priorities.push_back(p), 0; }
  ae_mpm_exec_opts& opts() override { return o; }
  void invalidate_graph() override {}
  uint64_t device_bytes() const override { return 0; }
  int copy_scene_from(uint32_t, aemp::WorldBase*, uint32_t) override { return 0; }
  int assign_scene(uint32_t, const ae_mpm_scene_desc&, const void*, uint64_t) override { return 0; }
  int vacate_scene(uint32_t) override { return 0; }
  uint32_t scene_count(uint32_t) const override { return 0; }
  int precision() const override { return 32; }
  int stage_times(uint32_t, double*) override { return 0; }
};
}  // namespace

namespace aemp {
WorldBase* make_world(const ae_mpm_scene_desc*, uint32_t, const ae_mpm_exec_opts&, std::string&, int*, DevAlloc*) {
  return new FakeWorld;
}
}  // namespace aemp

extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return (*p = malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (fails()) return cudaErrorInvalidValue;
  memcpy(d, s, n);
  ++in_flight;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) { return *least = 0, *greatest = -5, cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return in_flight = 0, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(&in_flight);
  return fails() ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return fails() ? cudaErrorInvalidValue : cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return in_flight = 0, fails() ? cudaErrorInvalidValue : cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
}

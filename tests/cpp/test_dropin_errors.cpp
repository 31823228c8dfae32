// The drop-in calls' host side on a CUDA runtime of this file's own, whose copies are host copies that
// count as in flight until their stream (or an event after them) is waited for.  A call that fails at any
// of its steps must leave nothing in flight: the next call packs into the same staging areas.
#include <math.h>
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }

#include "../../ae-engine_b200/csrc/ae_mpm_api.cu"

#include <cassert>

namespace {
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
  int set_stream_priority(int) override { return 0; }
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
cudaError_t cudaStreamSynchronize(cudaStream_t) { return in_flight = 0, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(&in_flight);
  return fails() ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return fails() ? cudaErrorInvalidValue : cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return in_flight = 0, fails() ? cudaErrorInvalidValue : cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
}

int main() {
  const ae_mpm_grid grid{8, 8, 8, 0.5f, {0, 0, 0}};
  ae_mpm_config cfg{};
  cfg.substeps = 1;
  ae_mpm_material mat{};
  mat.density = 1.0f;
  const int32_t model = AE_MPM_NEO_HOOKEAN;
  int failed = 0;
  for (const uint64_t n : {uint64_t(100), uint64_t(60001)})  // one packed copy; pieces
    for (const bool full : {false, true}) {
      std::vector<float> a(105 * n, 1.0f);
      std::vector<uint16_t> mats(n);
      std::vector<uint64_t> idx(n);
      for (uint64_t k = 0; k < n; ++k) idx[k] = k;
      float* p = a.data();
      const ae_mpm_particles v{p, p + 3 * n, p + 6 * n, p + 15 * n, p + 16 * n, p + 25 * n, mats.data()};
      for (int at = 0;; ++at) {
        ae_mpm_ctx ctx{};
        countdown = at;
        in_flight = 0;
        const int rc = full ? ae_mpm_step_parallel_with_grid(&ctx, &v, n, &grid, &cfg, &mat, 1, &model, 1, 0.01f,
                                                             idx.data(), n)
                            : ae_mpm_step_velocity_only_parallel(&ctx, &v, n, &grid, &cfg, 0.01f, idx.data(), n);
        const bool reached = countdown < 0;
        if (reached != (rc != AE_MPM_OK)) return printf("n %d full %d step %d: rc %d\n", int(n), full, at, rc), 1;
        if (in_flight) {
          printf("n %d, full %d, failing step %d: returned %d with work in flight\n", int(n), full, at, rc);
          ++failed;
        }
        countdown = -1;
        delete ctx.dropin;
        cudaFree(ctx.dstage);
        cudaFreeHost(ctx.pin);
        if (!reached) break;  // the call has no more steps
        if (at > 200) return printf("no end\n"), 1;
      }
    }
  printf(failed ? "%d left work in flight\n" : "ok\n", failed);
  return failed != 0;
}

// A drop-in call that fails at any of its steps must leave nothing in flight: the next call packs into the
// same staging areas.
#include "fake_runtime.hpp"

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

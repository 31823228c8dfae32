// Stream priorities of a batch's groups: from the highest on, each group below the one before it; with more
// groups than levels the first ones share the highest, so that the last ones keep their order.
#include "fake_runtime.hpp"

int main() {
  ae_mpm_scene_desc d{};
  ae_mpm_material mat{};
  d.n[0] = d.n[1] = d.n[2] = 8;
  d.n_materials = 1;
  d.materials = &mat;
  d.max_particles = 10;
  const std::vector<ae_mpm_scene_desc> scenes(16, d);
  const std::vector<std::vector<int>> want = {{-5},
                                              {-5, -4},
                                              {-5, -4, -3, -2},
                                              {-5, -4, -3, -2, -1, 0},
                                              {-5, -5, -4, -3, -2, -1, 0},
                                              {-5, -5, -5, -5, -4, -3, -2, -1, 0}};
  for (const std::vector<int>& w : want) {
    ae_mpm_ctx ctx{};
    ae_mpm_batch* b = nullptr;
    priorities.clear();
    if (ae_mpm_batch_create(&ctx, scenes.data(), 16, nullptr, uint32_t(w.size()), &b)) return 2;
    ae_mpm_batch_destroy(b);
    if (priorities != w) {
      printf("%d groups:", int(w.size()));
      for (int p : priorities) printf(" %d", p);
      printf("\n");
      return 1;
    }
  }
  printf("ok\n");
  return 0;
}

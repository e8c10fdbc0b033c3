// prepare_scene's world sphere around positions from a file (argv[1]: floats, 9 a triangle): finite, and
// around every finite corner where its radius fits a float. argv[2]: the radius expected (0: any).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <string>

#include "scene_prep.h"

using namespace orion_gb300;

int main(int, char** argv) {
  HostScene s;
  std::FILE* f = std::fopen(argv[1], "rb");
  float x;
  while (f && std::fread(&x, sizeof x, 1, f) == 1) s.positions.push_back(x);
  const size_t n = s.positions.size() / 9;
  s.normals.assign(9 * n, 0.f);
  s.uvs.assign(6 * n, 0.f);
  s.material_of_prim.assign(n, 0);
  s.light_of_prim.assign(n, -1);
  s.materials.resize(1);
  s.materials[0] = orion_material{};
  s.camera.width = s.camera.height = 1;
  PreparedScene p;
  std::string err;
  if (!prepare_scene(s, &p, &err)) return std::puts(err.c_str()), 1;
  const float* c = p.world_center;
  std::printf("centre %g %g %g radius %g\n", c[0], c[1], c[2], p.world_radius);
  if (!(std::isfinite(c[0]) && std::isfinite(c[1]) && std::isfinite(c[2]) && std::isfinite(p.world_radius)))
    return std::puts("not finite"), 1;
  const float want = std::strtof(argv[2], nullptr);
  if (want > 0.f && !(std::fabs(p.world_radius - want) <= 1e-5f * want)) return std::puts("another radius"), 1;
  std::puts("ok");
  return 0;
}

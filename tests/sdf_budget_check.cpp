// Host check of sdf_cell_tables' size limit (myrt_b200/csrc/sdf_skip.hpp): many
// left folds whose first grids just fit together. Every program keeps its first
// grid, whatever the second grids of the programs before it took; one entry
// less and only the last loses its own. Prints the programs checked.
#include <cstdio>
#include <random>
#include <vector>

#include "../myrt_b200/csrc/sdf_skip.hpp"

using namespace myrt_b200;

int main() {
  int const n_programs = 12, n_prims = 40, cells = 8;
  std::vector<myrt_sdf_instr> instrs;
  std::vector<myrt_sdf_program> programs;
  std::vector<float> params;
  std::mt19937 rng(3);
  std::uniform_real_distribution<float> u(-1.f, 1.f);
  auto emit = [&](int op, std::initializer_list<float> values) {
    instrs.push_back({op, int(params.size())});
    params.insert(params.end(), values);
  };
  for (int p = 0; p < n_programs; ++p) {
    int const first = int(instrs.size());
    for (int g = 0; g < n_prims; ++g) {
      float const x = u(rng), y = u(rng), z = u(rng);
      emit(MYRT_SDF_TRANSLATE, {x, y, z});
      emit(MYRT_SDF_SPHERE, {0.1f, 0.f});
      if (g) emit(MYRT_SDF_SMOOTH_UNION, {0.05f});
    }
    programs.push_back({first, int(instrs.size()) - first});
  }
  myrt_sdf_view v{};
  v.instrs = instrs.data(), v.instr_count = instrs.size();
  v.programs = programs.data(), v.program_count = programs.size();
  v.params = params.data(), v.param_count = params.size();
  auto kept = [&](sdf_cells const& c, size_t& entries) {
    int n = 0;
    entries = 0;
    for (int p = 0; p < n_programs; ++p) {
      int4 const d = c.hdr[3 * p + 1];
      n += d.x > 0;
      if (d.x > 0) entries += size_t(c.start[d.w + d.x * d.y * d.z] - c.start[d.w]);
    }
    return n;
  };
  sdf_cells all, fit, less;
  size_t total = 0, got = 0;
  sdf_cell_tables(&v, cells, all);
  bool sound = kept(all, total) == n_programs && all.list.size() > total;  // second grids hold the rest
  sdf_cell_tables(&v, cells, fit, total);
  sound = sound && kept(fit, got) == n_programs && got == total && fit.list.size() <= total + total / 2;
  sdf_cell_tables(&v, cells, less, total - 1);
  sound = sound && kept(less, got) == n_programs - 1 && less.hdr[3 * (n_programs - 1) + 1].x == 0;
  if (!sound) {
    std::printf("first grids hold %zu entries, all %zu; kept %d\n", total, all.list.size(), kept(fit, got));
    return 1;
  }
  std::printf("%d\n", n_programs);
  return 0;
}

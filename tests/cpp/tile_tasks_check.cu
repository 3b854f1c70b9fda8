// The tile kernel's task lists (mfgpu::tile_tasks): every pivot and Schur tile
// of every front once, inside the front, and each task after the tasks whose
// finished block columns it waits for (block rows I and J at least J, or all
// the pivot block columns for a Schur tile; a pivot tile also the diagonal one).
#include <cstdio>
#include <map>
#include <set>
#include <tuple>
#include <vector>

#include "../../updating-multifrontal_b200/csrc/kernels_tile.cu"

namespace mfgpu {
std::atomic<long long> g_launches{0};
}

int main() {
  const std::vector<std::vector<std::pair<int, int>>> sets = {
      {{1, 1}}, {{64, 64}}, {{65, 65}}, {{63, 200}}, {{64, 200}}, {{100, 100}}, {{128, 129}},
      {{29, 89}, {49, 77}, {225, 285}, {253, 253}}, {{714, 1951}, {1, 300}, {640, 641}},
      std::vector<std::pair<int, int>>(700, {225, 285}), {{2045, 2045}, {33, 64}}, {{0, 70}, {5, 5}}};
  for (const auto& fr : sets) {
      std::vector<int> n, N, tasks, row;
      for (auto& p : fr) n.push_back(p.first), N.push_back(p.second);
      mfgpu::tile_tasks(n, N, tasks, row);
      const int nf = (int)n.size();
      if ((int)row.size() != nf + 1) return printf("row offsets\n"), 1;
      std::vector<int> done(row[nf], 0);
      std::set<std::tuple<int, int, int, int>> seen;
      size_t want = 0;
      for (int i = 0; i < nf; i++) {
        const int nb = (N[i] + 63) / 64, np = (n[i] + 63) / 64;
        if (row[i + 1] - row[i] != nb) return printf("block rows of front %d\n", i), 1;
        for (int J = 0; J < np; J++) want += nb - J;
        if (N[i] > n[i])
          for (int J = n[i] / 64; J < nb; J++) want += nb - J;
      }
      for (size_t t = 0; t < tasks.size(); t += 2) {
        const int i = tasks[t], I = tasks[t + 1] & 0x7fff, J = (tasks[t + 1] >> 15) & 0x7fff,
                  schur = tasks[t + 1] >> 30;
        const int nb = (N[i] + 63) / 64, np = (n[i] + 63) / 64;
        if (i < 0 || i >= nf || I >= nb || J > I || schur > 1) return printf("bad task\n"), 1;
        if (!seen.insert({i, I, J, schur}).second) return printf("task twice\n"), 1;
        int* d = done.data() + row[i];
        if (schur) {
          if (d[I] < np || d[J] < np) return printf("Schur tile before its panels\n"), 1;
        } else {
          if (J >= np || d[I] != J || d[J] < J + (I > J)) return printf("pivot tile too early\n"), 1;
          d[I] = J + 1;
        }
      }
      if (seen.size() != want) return printf("%zu tasks, %zu wanted\n", seen.size(), want), 1;
    }
  printf("ok\n");
  return 0;
}

// Host check of the cluster-resident lens's index arithmetic (lf_cluster.cuh): every layout is in bounds and
// one-to-one, splits into the lane part plus constants that the kernels use, keeps what must stay apart apart,
// and loads from the landing areas without bank conflicts.  Prints one line per configuration; exit status 1
// on any fault.
#include <cstdio>
#include <set>

#include "../../cmblensing_b200/csrc/lf_cluster.cuh"

using namespace lf;

template <typename T, int N, int CL> int check() {
  using G = ClGeo<T, N, CL>;
  using S = ClSystem<T, N, CL>;
  using RL = RowLay<T, N>;
  using CO = ColLay<T, N>;
  constexpr int E = G::E, TP = G::TP, step = lay_step<T, N>();
  int bad = 0;
  std::set<int> seen, kept;
  for (int q = 0; q < 2; ++q)
    for (int m = 0; m < N; ++m) {
      const int a = RL::at(m) + q * step;
      bad += a < 0 || a >= lay_group<T, N>();
      bad += RL::at(m % TP) + RL::at(m - m % TP) != RL::at(m);
      seen.insert(a);
      if (m < N / 2) kept.insert(a);
    }
  bad += (int)seen.size() != 2 * N;
  seen.clear();
  for (int m = 0; m < N; ++m) {  // the column scratch leaves the kept half spectra alone
    const int a = CO::at(m);
    bad += a < 0 || a >= lay_group<T, N>() || kept.count(a);
    bad += CO::at(m % TP) + CO::at(m - m % TP) - CO::at(0) != a;
    seen.insert(a);
  }
  bad += (int)seen.size() != N;
  seen.clear();
  for (int m = 0; m < N; ++m)
    for (int l = 0; l < G::KC; ++l) {
      const int a = col_at<T, N, G::KC>(m, l);
      bad += a < 0 || a >= S::kCol || col_at<T, N, G::KC>(m % TP, l) + G::KC * (m - m % TP) != a;
      seen.insert(a);
    }
  bad += (int)seen.size() != S::kCol;
  seen.clear();
  for (int k = 0; k < N / 2; ++k)
    for (int r = 0; r < G::RPC; ++r) {
      const int a = land_at<T, N, G::RPC>(k, r);
      bad += a < 0 || a >= S::kLand || land_at<T, N, G::RPC>(k % TP, r) + G::RPC * (k - k % TP) != a;
      seen.insert(a);
    }
  bad += (int)seen.size() != S::kLand;
  const int slots = sizeof(T) == 4 ? 16 : 8;  // accesses served together
  for (int w = 0; w < 32; w += slots) {
    std::set<int> c, d;
    for (int l = w; l < w + slots; ++l) {
      c.insert(col_at<T, N, G::KC>(l % TP, l / TP) % slots);
      d.insert(land_at<T, N, G::RPC>(l % TP, 2 * (l / TP)) % slots);
    }
    bad += (int)c.size() != slots || (int)d.size() != slots;
  }
  const int radices[2][3] = {{E, cl_r2(N, E), cl_r3(N, E)}, {cl_r3(N, E), cl_r2(N, E), E}};
  for (const auto& rad : radices) {  // a pass's outputs: a permutation, at lane part plus constant
    int ns = 1;
    for (int R : rad) {
      if (R == 1) continue;
      std::set<int> out;
      for (int l = 0; l < TP; ++l)
        for (int i = 0; i < E / R; ++i)
          for (int r = 0; r < R; ++r) {
            const int b = TP * i, bb = l + b;
            const int lp = (l / ns) * ns * R + l % ns, cp = (b / ns) * ns * R + b % ns + r * ns;
            const int want = (bb / ns) * ns * R + bb % ns + r * ns;
            bad += RL::at(lp) + RL::at(cp) != RL::at(want) || CO::at(lp) + CO::at(cp) - CO::at(0) != CO::at(want);
            out.insert(want);
          }
      bad += (int)out.size() != N;
      ns *= R;
    }
    bad += ns != N;
  }
  const size_t bytes = sizeof(c2<T>) * (S::kElems + cl_tw_size(N, E)) + 32;
  bad += bytes > 227 * 1024 || S::kElems * sizeof(c2<T>) % 16 != 0 || cl_tw_size(N, E) * sizeof(c2<T>) % 16 != 0;
  std::printf("T %zu N %d CL %d threads %d shared %zu faults %d\n", sizeof(T), N, CL, G::NT, bytes, bad);
  return bad;
}

int main() {
  int bad = 0;
  bad += check<float, 64, 4>() + check<float, 128, 8>() + check<float, 256, 16>();
  bad += check<double, 64, 4>() + check<double, 128, 8>() + check<double, 256, 16>();
  return bad != 0;
}

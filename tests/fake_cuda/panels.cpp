// One panel of the LU on the emulator: <kernel> <f|d> <N> <k0> <ncols> <CTAs> <drop_src> <drop_dst> <drop_from>
// <wait limit> <status word before> <odd value> <output file>.  odd value: 1 a NaN in the panel, 2 an infinity, 3 a
// column of NaN, 4 nothing but NaN, 5 a row of infinities.  kernel: reg, tall (its sub-panels, updates and placing) or
// grid (absent: its last CTA never runs).  Writes the sizes, the status words, pivots and interchange lists, the number of guard bytes that
// were written and of the emulator's faults, then the matrix before and after and the LU planes.
#include "emulate.h"
#include "panel.cuh"

using namespace hprmat;
constexpr int kNB = 32;

template <typename T>
int run(char** v) {
  const std::string kind = v[1];
  const int N = atoi(v[3]), k0 = atoi(v[4]), ncols = atoi(v[5]), G = atoi(v[6]);
  emu::drop_src = atoi(v[7]);
  emu::drop_dst = atoi(v[8]);
  emu::drop_from = (unsigned)atoi(v[9]);
  emu::wait_limit = (unsigned)atoi(v[10]);
  const int m = N - k0, ld = (N + 3) / 4 * 4;
  emu::Guarded<T> W((size_t)ld * N), cand((size_t)(2 * G + kNB) * kNB), rowj(2 * kNB), ubuf(kNB * kNB), xrows(kSubW * kSubW);
  emu::Guarded<int> lists(3 * kNB + 1), ipiv(N), status(SW_COUNT), pos(N), prow(kNB);
  emu::Guarded<unsigned long long> keys(kNB);
  emu::Guarded<float> lup((size_t)4 * ld * N);
  unsigned x = 12345u + N + k0;
  auto rnd = [&] { return (double)((x = x * 1664525u + 1013904223u) >> 8) / (1 << 24) - 0.5; };
  for (size_t i = 0; i < W.n; ++i) {
    W.p[i].x = rnd();
    W.p[i].y = rnd();
  }
  const int odd = atoi(v[12]);
  for (int c = k0; c < k0 + ncols; ++c)
    for (int r = k0; r < N; ++r) {
      auto& e = W.p[r + (size_t)c * ld];
      if ((odd <= 2 && odd > 0 && r == k0 + 7 && c == k0 + 3) || (odd == 3 && c == k0 + 5) || odd == 4 || (odd == 5 && r == k0 + 9))
        e.y = odd == 2 || odd == 5 ? INFINITY : NAN;
    }
  const std::vector<T> before(W.p, W.p + W.n);
  status.p[SW_TIMEOUT] = atoi(v[11]);
  for (int i = 0; i < 3 * kNB + 1; ++i) lists.p[i] = -(1 << 18);  // what an unwritten list may hold
  const StepSwaps sw{lists.p, lists.p + kNB, lists.p + 2 * kNB, lists.p + 3 * kNB};
  unsigned* growth = (unsigned*)(status.p + SW_COUNT - 1);
  const bool planes = sizeof(T) == sizeof(float2);
  if (kind == "tall") {
    SubArgs<T> a{};
    a.W = W.p;
    a.ld = ld;
    a.N = N;
    a.k0 = k0;
    a.ncols = ncols;
    a.rpc = (m + 15) / 16;
    a.G = 16;
    a.pos = pos.p;
    a.prow = prow.p;
    a.xrows = xrows.p;
    a.ubuf = ubuf.p;
    a.ldu = kNB;
    a.ipiv = ipiv.p;
    a.status = status.p;
    a.sw = sw;
    a.growth_bits = growth;
    a.lup = planes ? lup.p : nullptr;
    a.lup_ld = ld;
    a.lup_plane = (long)ld * N;
    for (a.c0 = 0; a.c0 < ncols; a.c0 += kSubW) {
      emu::launch(16, kSubThreads, true, [&] { panel_sub_kernel<T, 1>(a); });
      if (a.c0 + kSubW < ncols) emu::launch((m + kRestRows - 1) / kRestRows, 256, false, [&] { panel_rest_kernel<T, kNB>(a); });
    }
    if constexpr (sizeof(T) == sizeof(float2)) emu::launch((m + 31) / 32, 256, false, [&] { panel_planes_kernel<kNB>(a); });
    emu::launch((ncols + kPlaceCols - 1) / kPlaceCols, 256, false, [&] { panel_place_kernel<T, kNB>(a); });
  } else {
    PanelArgs<T> a{};
    a.W = W.p;
    a.ld = ld;
    a.N = N;
    a.k0 = k0;
    a.ncols = ncols;
    a.rpc = (m + G - 1) / G;
    a.G = G;
    a.ipiv = ipiv.p;
    a.cand_rows = cand.p;
    a.keys = keys.p;
    a.rowj = rowj.p;
    a.status = status.p;
    a.sw = sw;
    a.growth_bits = growth;
    a.lup = planes ? lup.p : nullptr;
    a.lup_ld = ld;
    a.lup_plane = (long)ld * N;
    if (kind == "reg")
      emu::launch(G, kRegPanelThreads, true, [&] { panel_reg_kernel<T, kNB>(a); });
    else
      emu::launch(kind == "absent" ? G - 1 : G, 256, true, [&] { panel_kernel<T, kNB, 256>(a); });
  }
  const size_t hits = W.hits() + cand.hits() + rowj.hits() + ubuf.hits() + xrows.hits() + lists.hits() + ipiv.hits() +
                      status.hits() + pos.hits() + prow.hits() + keys.hits() + lup.hits();
  FILE* f = fopen(v[13], "wb");
  const int head[4] = {ld, SW_TIMEOUT, (int)std::min<size_t>(hits, 1u << 30), emu::faults.load()};
  fwrite(head, sizeof(int), 4, f);
  fwrite(status.p, sizeof(int), SW_COUNT, f);
  fwrite(ipiv.p, sizeof(int), N, f);
  fwrite(lists.p, sizeof(int), 3 * kNB + 1, f);
  fwrite(before.data(), sizeof(T), W.n, f);
  fwrite(W.p, sizeof(T), W.n, f);
  fwrite(lup.p, sizeof(float), lup.n, f);
  return fclose(f);
}

int main(int argc, char** argv) {
  if (argc != 14) return 2;
  return argv[2][0] == 'd' ? run<double2>(argv) : run<float2>(argv);
}

// Prints the diagonal wavefront's layout of a matrix, as JSON, for the tests:
// diag_probe FILE FORM NLEVEL NSM SMEM, FILE: n, ptr[n + 1], col, all int32.
#include <chrono>
#include <cstdio>
#include <cstdlib>

#include "../mpk_gb300/csrc/diag.cuh"

int main(int argc, char **argv) {
  if (argc != 6) return 2;
  FILE *f = std::fopen(argv[1], "rb");
  int n = 0;
  if (!f || std::fread(&n, 4, 1, f) != 1) return 2;
  std::vector<int> ptr(n + 1);
  if (std::fread(ptr.data(), 4, n + 1, f) != (size_t)n + 1) return 2;
  std::vector<int> col(ptr[n]);
  if (std::fread(col.data(), 4, col.size(), f) != col.size()) return 2;
  std::fclose(f);
  const int nlevel = std::atoi(argv[3]);
  mpkg::DiagLayout l;
  const auto t0 = std::chrono::steady_clock::now();
  const int rc = mpkg::diag_layout(n, ptr.data(), col.data(), nlevel, std::atoi(argv[2]), std::atoi(argv[4]),
                                   std::atoi(argv[5]), &l);
  const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  std::printf("{\"rc\": %d, \"ms\": %.3f, \"fits\": %d, \"w\": %d, \"mode\": %d, \"depth\": %d, \"halo\": %d, \"grid\": %d, "
              "\"smem\": %d, \"win_at\": %d, \"irregular\": %ld, \"rows\": %ld, \"scanned\": %zu, \"patterns\": %zu}\n",
              rc, ms, (int)l.fits, l.w, l.mode, l.depth, l.halo, l.grid, l.smem, l.win_at, l.irregular, l.rows, l.pat.size(),
              l.mask.size() / 32);
}

// Diagonal wavefront: layout and launch interface (diag.cu).
#ifndef MPKG_DIAG_CUH
#define MPKG_DIAG_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include <memory>
#include <vector>

#include "host.h"

namespace mpkg {

// Arithmetic of the rows.
enum DiagForm {
  kDiagFma, kDiagFmaVal,  // FP64, 1/deg operator or matrix values
  kDiagSep, kDiagSepVal,
  kDiagDf, kDiagDfVal,    // double-float
  kDiagF32, kDiagBf16,    // mixed: FP32 or BF16 values
};

// How rows of other CTAs are read: from the halo; the outermost diagonal on
// either side from global memory and the others from the halo; from a halo for
// several levels.
enum DiagMode { kDiagAll, kDiagPair, kDiagDeep };

constexpr int kDiagMax = 9;  // diagonals
constexpr int kDiagMaxDepth = 8;

struct DiagArgs {
  int n, nlevel, nblk;
  uint32_t base, stall;   // as WaveArgs
  int d[kDiagMax];        // the diagonals, ascending column offsets ...
  int db[kDiagMax];       // ... and in bytes of a window
  int halo;               // rows kept of the CTAs on either side
  int depth, grow;        // levels per exchange; slices that a level takes more on either side for the next
  const int *row_lo, *dep_ptr, *dep_idx;
  unsigned int *flags;
  int *err;
  const unsigned short *pat;   // per slice: its pattern, kDiagIrregular for none
  const unsigned short *mask;  // pattern p, lane j: the diagonals that row has, at 32 p + j; pattern 0 has all
  const int2 *own;             // per CTA: slices [x, y) read own rows only
  const void *vals;            // [slice][diagonal][lane], in the form's type
  const int *nres;             // per CTA: its first slices whose values stay in shared memory
  // irregular slices: the CSR rows, their values (in the form's type) or 1/deg
  const int *ptr, *col;
  const void *coef;
  const double *lut;           // 1/d
  const float2 *lut2;          // ... in double-float
  double *vv;                  // FP64 levels (double-float: the rounded ones)
  float2 *ring;                // double-float levels l, l-1, l-2, n each
  int ring_all;                // rows of irregular slices may read any row there
  float *vf;                   // mixed levels, scaled by `scale`
  float scale;
  double *hv;                  // host mapping of vv, or null (as WaveArgs; double-float: vv is the host's)
  int smem;                    // dynamic shared memory
  int win_at, second;          // bytes: the own rows of window A, and of window B after those
};

constexpr unsigned short kDiagIrregular = 0xFFFF;
constexpr int kFlagStride = 32;  // flags lie in cache lines of their own

// Host side of a layout.
struct DiagLayout {
  bool fits = false;
  int w = 0, mode = kDiagAll;  // diagonals; DiagMode
  int d[kDiagMax] = {};
  int halo = 0, win_bytes = 0, halo_bytes = 0, grid = 0;
  int depth = 1, grow = 0, win_at = 0, second = 0;
  int smem = 0;                // dynamic shared memory that it needs
  int slices = 0;              // the most that a CTA computes at a level
  long reach = 0, irregular = 0, rows = 0;  // rows: computed by a call
  std::vector<int> lo, dptr, didx, nres;
  std::vector<int2> own;
  std::vector<unsigned short> pat, mask;
};

// The layout of the diagonal wavefront for `nsm` CTAs with up to `smem` bytes
// of dynamic shared memory; fits is false where the structure or the sizes do
// not suit it.
int diag_layout(int n, const int *ptr, const int *col, int nlevel, int form, int nsm, int smem, DiagLayout *out);

// Values along the layout's diagonals, [slice][diagonal][lane], zero where a
// row has no entry (and in irregular slices): conv(entry) in type T.  False
// for want of memory.
template <typename T, typename F>
bool diag_values(int n, const int *ptr, const int *col, const DiagLayout &l, T zero, F &&conv, T *out) {
  const int ns = (int)l.pat.size(), part = 256;  // slices a task
  return host_parallel((ns + part - 1) / part, ptr[n], 50000, [&](int t) {
    for (int sl = t * part; sl < std::min(ns, (t + 1) * part); sl++) {
      T *o = out + (size_t)sl * l.w * 32;
      std::fill(o, o + (size_t)l.w * 32, zero);
      if (l.pat[sl] == kDiagIrregular) continue;
      for (int i = sl * 32; i < std::min(n, sl * 32 + 32); i++) {
        int u = 0;
        for (int q = ptr[i]; q < ptr[i + 1]; q++) {
          while (l.d[u] != col[q] - i) u++;
          o[32 * u + i % 32] = conv(q);
        }
      }
    }
  });
}

const void *diag_kernel_ptr(int form, int w, int mode);
constexpr int kDiagThreads = 1024;
int diag_elem_bytes(int form);   // of a window element
int diag_value_bytes(int form);  // of a matrix value, 0 for 1/deg

}  // namespace mpkg

#endif

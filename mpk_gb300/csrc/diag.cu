// Diagonal wavefront (sm_103a): the wavefront executor for matrices whose
// rows keep to a few diagonals (meshes in their natural order).
//
// One CTA of 1024 threads per SM owns a contiguous, slice-aligned row range
// at every level and computes level l once the CTAs owning its columns have
// published level l-1, as the general wavefront does.  Two windows in shared
// memory hold its rows of the previous level and of the one being computed,
// so that a row reads its columns at constant distances from its own place: no
// index is loaded, and an entry is a shared-memory load and its arithmetic.
// Beside the window that is read lie `halo` rows of the CTAs before and after,
// fetched once those have published them; slices that read own rows only are
// computed before that wait.  Where the outermost diagonal on either side
// reaches further than the own rows (the planes of a 3-D mesh), that one entry
// is read from global memory instead, a slice ahead.  A slice of 32 rows that
// lacks some of the diagonals (mesh boundaries) has a pattern, a mask of
// diagonals per lane; slices with other columns run from the CSR.  Values lie
// [slice][diagonal][lane]; shared memory keeps as many slices of them as fit
// beside the windows for the whole call.
//
// A level costs some 4.5 K cycles of hand-over between CTAs, whatever its
// size.  Where the rows reach few slices a CTA exchanges every `depth` levels
// instead: it fetches depth times the halo and computes the levels between on
// so many slices of its neighbours too, as many levels as the cost below
// prefers (us with 1, 2, 3, 4 levels: 100^2 1/deg k = 4 12.4 / 8.7 / 10.2 /
// 8.4; 200 x 201 k = 6 18.5 / 14.4 / 15.0 / 16.4; mixed FP32 9-point 120 x 110
// k = 8 20.6 / 14.4 / 13.9 / 12.4; FP64 9-point 1023 x 769 k = 6 80 / 85 / 92 /
// 100).
//
// Row sums run over the entries in CSR order with the arithmetic of
// wave_kernel, wave_df_kernel and wave_mix_kernel: the same bits.
//
// What bounds it: in FP64 the FP64 pipe, 6 fused multiply-adds a 7-point row
// (47 K cycles a level on 128^3, 41 K of them that pipe's), else the
// instructions, about 100 a slice; and at every level some 5 K cycles of
// hand-over (release after the barrier 1.5-3 K, the neighbours' flags 1-2 K,
// the halo 1 K).  Against the general wavefront, which reads every index and
// its columns through L1 (us): 128^3 1/deg k = 8 228 / 249; 100^2 1/deg k = 4
// 8.2 / 15.2; 9-point FP64 1400 x 1300 k = 8 266 / 293; double-float 1/deg
// 101 x 97 x 89 k = 8 79 / 105; mixed FP32 120 x 110 x 100 k = 8 68 / 140, BF16
// 9-point 701 x 699 k = 4 17.4 / 40.8.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <map>
#include <string>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "diag.cuh"
#include "rows.cuh"

using namespace mpkg;

namespace {

template <int F>
struct Form;
template <int A, bool V>
struct Fp64Form {
  static constexpr int kArith = A;
  static constexpr bool kVal = V;
  using Elem = double;
  using Val = double;
};
template <>
struct Form<kDiagFma> : Fp64Form<MPKG_ARITH_FMA, false> {};
template <>
struct Form<kDiagFmaVal> : Fp64Form<MPKG_ARITH_FMA, true> {};
template <>
struct Form<kDiagSep> : Fp64Form<MPKG_ARITH_SEPARATE, false> {};
template <>
struct Form<kDiagSepVal> : Fp64Form<MPKG_ARITH_SEPARATE, true> {};
template <bool V>
struct DfForm {
  static constexpr int kArith = MPKG_ARITH_DF64;
  static constexpr bool kVal = V;
  using Elem = float2;
  using Val = float2;
};
template <>
struct Form<kDiagDf> : DfForm<false> {};
template <>
struct Form<kDiagDfVal> : DfForm<true> {};
template <typename VT>
struct MixForm {
  static constexpr int kArith = -1;
  static constexpr bool kVal = true;
  using Elem = float;
  using Val = VT;
};
template <>
struct Form<kDiagF32> : MixForm<float> {};
template <>
struct Form<kDiagBf16> : MixForm<__nv_bfloat16> {};

// A row's running sum.
template <int F>
struct Sum {  // FP64 and mixed
  using E = typename Form<F>::Elem;
  E s = 0;
  template <typename V>
  __device__ __forceinline__ void add(int u, V v, E x) {
    if constexpr (Form<F>::kArith < 0) s = __fmaf_rn(to_f32(v), x, s);
    else if (u == 0) s = row_first<Form<F>::kArith>(v, x);
    else if (u < kIntTerms) s = row_next<Form<F>::kArith>(s, v, x);
    else s = row_term<Form<F>::kArith>(s, v, x);
  }
};
template <>
struct Sum<kDiagDf> {
  float h = 0.f, l = 0.f;
  __device__ __forceinline__ void add(int, float2, float2 x) { df_acc(x, h, l); }
};
template <>
struct Sum<kDiagDfVal> {
  float h = 0.f, l = 0.f;
  __device__ __forceinline__ void add(int, float2 v, float2 x) { df_mac(v, x, h, l); }
};

// Waits (bounded) for the CTAs list[c0 .. c1) (or c0 .. c1 themselves) to
// publish `want`; every thread calls it.  One thread per flag polls: with every
// warp polling, the flags' lines are so busy that a wait of 1-2 thousand cycles
// takes 6-11 thousand.
__device__ __forceinline__ bool diag_wait(const DiagArgs &a, const int *list, int c0, int c1, unsigned want,
                                          int *s_abort) {
  for (int k = c0 + (int)threadIdx.x; k < c1; k += blockDim.x) {
    const int c = list ? list[k] : k;
    long spins = 0;
    while (ld_acquire(a.flags + kFlagStride * c) < want + a.stall) {
      if (++spins > kSpinLimit || *((volatile int *)a.err)) {
        atomicCAS(a.err, 0, kErrTimeout);
        *s_abort = 1;
        break;
      }
      __nanosleep(spins < 16 ? 32 : 256);
    }
  }
  __syncthreads();
  return *s_abort == 0;
}

__device__ __forceinline__ void diag_publish(const DiagArgs &a, int b, unsigned v) {
  __syncthreads();
  if (threadIdx.x == 0)
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(a.flags + kFlagStride * b), "r"(v) : "memory");
}

constexpr int kXGroups = 8;  // host execution: CTA groups that copy x in turn (as wave_kernel)

// MODE: kDiagAll, kDiagPair or kDiagDeep.
template <int F, int W, int MODE>
__global__ void __launch_bounds__(kDiagThreads, 1) diag_kernel(const __grid_constant__ DiagArgs a) {
  using FM = Form<F>;
  using E = typename FM::Elem;
  using V = typename FM::Val;
  constexpr bool kDf = FM::kArith == MPKG_ARITH_DF64, kMix = FM::kArith < 0;
  constexpr bool kPair = MODE == kDiagPair, kDeep = MODE == kDiagDeep;
  extern __shared__ __align__(128) unsigned char dg_smem[];
  __shared__ int s_abort;
  __shared__ __align__(8) unsigned long long s_bar;
  const int b = blockIdx.x, r0 = a.row_lo[b], r1 = a.row_lo[b + 1];
  const int s0 = r0 >> 5, ns = (r1 + 31 - r0) >> 5;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nt = blockDim.x, nw = nt >> 5;
  // shared memory: patterns, values, then the two windows at the end
  unsigned short *s_pat = reinterpret_cast<unsigned short *>(dg_smem);
  // slices before and after the own ones that it computes too at the first
  // level after an exchange
  const int depth = kDeep ? a.depth : 1, more = (depth - 1) * a.grow;
  const int xlo = min(s0, more), xhi = min(((a.n + 31) >> 5) - s0 - ns, more);
  s_pat += xlo;  // of the first own slice, as s_val and vals
  V *s_val = reinterpret_cast<V *>(dg_smem + ((2 * (xlo + ns + xhi) + 15) & ~15)) + xlo * W * 32;
  const V *vals = reinterpret_cast<const V *>(a.vals) + (size_t)s0 * W * 32;
  const int nres = FM::kVal ? a.nres[b] - xlo : 0;
  unsigned char *wins = dg_smem + a.win_at;
  const int w0 = max(0, r0 - a.halo), w1 = min(a.n, r1 + a.halo);
  if (threadIdx.x == 0) {
    s_abort = 0;
    if (FM::kVal) {  // the values stream in while the window is filled
      mbar_init(&s_bar);
      constexpr int kSlice = W * 32 * (int)sizeof(V);
      mbar_expect(&s_bar, (unsigned)((nres + xlo) * kSlice));
      for (int o = -xlo * kSlice; o < nres * kSlice; o += 32768)
        bulk_g2s(reinterpret_cast<unsigned char *>(s_val) + o, reinterpret_cast<const unsigned char *>(vals) + o,
                 (unsigned)min(32768, nres * kSlice - o), &s_bar);
    }
  }
  for (int k = (int)threadIdx.x - xlo; k < ns + xhi; k += nt) s_pat[k] = a.pat[s0 + k];
  auto level = [&](int l) -> const E * {  // where other CTAs' rows of level l are read
    if constexpr (kDf) return a.ring + (size_t)(l / depth % 3) * a.n;
    else if constexpr (kMix) return a.vf + (size_t)l * a.n;
    else return a.vv + (size_t)l * a.n;
  };
  // host execution: each CTA copies its rows of x to the device and publishes
  // level 0, in kXGroups groups of CTAs taken in order
  const bool host = !kMix && a.hv != nullptr;
  if constexpr (!kMix) {
    if (host) {
      const int grp = (int)((long)b * kXGroups / a.nblk);
      if (grp > 0) {
        const int c0 = (int)(((long)(grp - 1) * a.nblk + kXGroups - 1) / kXGroups);
        const int c1 = (int)(((long)grp * a.nblk + kXGroups - 1) / kXGroups);
        __syncthreads();
        if (!diag_wait(a, nullptr, c0, c1, a.base, &s_abort)) {
          if (FM::kVal) tr_wait(&s_bar, 0, a.err);  // the values are on their way
          return;
        }
      }
      for (int i = r0 + (int)threadIdx.x; i < r1; i += nt) {
        if constexpr (kDf) a.ring[i] = df_split(a.hv[i]);
        else a.vv[i] = a.hv[i];
      }
      diag_publish(a, b, a.base);
      if (!diag_wait(a, a.dep_idx, a.dep_ptr[b], a.dep_ptr[b + 1], a.base, &s_abort)) {
        if (FM::kVal) tr_wait(&s_bar, 0, a.err);
        return;
      }
    }
  }
  auto first = [&](int i) -> E {  // row i of level 0
    if constexpr (kDf) return host ? __ldcg(a.ring + i) : df_split(__ldg(a.vv + i));
    else if constexpr (kMix) return a.vf[i];
    else return __ldcg(a.vv + i);
  };
  {
    E *in = reinterpret_cast<E *>(wins) - r0;
    for (int i = w0 + (int)threadIdx.x; i < w1; i += nt) in[i] = first(i);
  }
  const int own0 = a.own[b].x, own1 = a.own[b].y;
  V coef{};  // of a row with all the diagonals
  if constexpr (!kDf && !kMix && !FM::kVal) coef = __ldg(a.lut + W);
  float2 coef2 = make_float2(0.f, 0.f);
  if constexpr (kDf && !FM::kVal) coef2 = __ldg(a.lut2 + W);
  __syncthreads();
  if (FM::kVal && !tr_wait(&s_bar, 0, a.err)) return;
  // the test hook's wait, also where no level waits
  if (kDeep && a.stall && !diag_wait(a, a.dep_idx, a.dep_ptr[b], a.dep_ptr[b + 1], a.base + 1, &s_abort)) return;
  for (int l = 1, left = -1; l <= a.nlevel; l++, left--) {
    // `left` levels follow before the next exchange; each needs a.grow slices
    // more of this one on either side
    const bool exchange = !kDeep || left < 0;
    if (exchange) left = min(depth, a.nlevel + 1 - l) - 1;
    const int lo = kDeep ? -min(xlo, left * a.grow) : 0, hi = ns + (kDeep ? min(xhi, left * a.grow) : 0);
    E *in = reinterpret_cast<E *>(wins + (l & 1 ? 0 : a.second)) - r0;
    E *out = reinterpret_cast<E *>(wins + (l & 1 ? a.second : 0)) - r0;
    const E *prev = level(l - 1);
    auto far = [&](int i) -> E { return kDf && l == 1 ? first(i) : __ldcg(prev + i); };
    const bool wait = exchange && l > 1;
    for (int part = 0; part < 2; part++) {
      // part 0: slices [own0, own1), which read own rows only; part 1: the others,
      // once the CTAs that own the rows around them have published those
      const int cut = part == 0 ? own1 : own0, end = part == 0 ? own1 : hi - (own1 - own0);
      auto at = [&](int j) { return j < cut ? j : j + (own1 - own0); };
      const int j0 = (part == 0 ? own0 : lo) + warp;
      E g0{}, g1{};
      auto fetch = [&](int j) {  // the far entries of slice j
        if (kPair && j < end) {
          const int i = r0 + 32 * at(j) + lane, c0 = i + a.d[0], c1 = i + a.d[W - 1];
          if (c0 >= 0 && i < a.n) g0 = far(c0);
          if (c1 < a.n) g1 = far(c1);  // c1 > i
        }
      };
      if (part == 1 && wait) {
        if (!diag_wait(a, a.dep_idx, a.dep_ptr[b], a.dep_ptr[b + 1], a.base + (unsigned)(l - 1), &s_abort)) return;
        fetch(j0);
        for (int i = w0 + (int)threadIdx.x; i < r0; i += nt) in[i] = __ldcg(prev + i);
        for (int i = r1 + (int)threadIdx.x; i < w1; i += nt) in[i] = __ldcg(prev + i);
        __syncthreads();
      } else {
        fetch(j0);
      }
      for (int j = j0; j < end; j += nw) {
        const int k = at(j), i = r0 + 32 * k + lane;
        const E x0 = g0, x1 = g1;
        fetch(j + nw);
        if (i >= a.n) continue;
        const int pat = s_pat[k];
        Sum<F> s;
        int len = W;
        if (pat != kDiagIrregular) {
          const int m = pat == 0 ? (1 << W) - 1 : __ldg(a.mask + 32 * pat + lane);
          const unsigned char *own = reinterpret_cast<const unsigned char *>(in + i);
          auto entry = [&](int u) -> E {
            return kPair && u == 0 ? x0 : kPair && u == W - 1 ? x1 : *reinterpret_cast<const E *>(own + a.db[u]);
          };
          auto row = [&](auto value) {  // value(u): from shared memory, or from global memory
            if (pat == 0) {
              E x[W];
#pragma unroll
              for (int u = 0; u < W; u++) x[u] = entry(u);
#pragma unroll
              for (int u = 0; u < W; u++) s.add(u, FM::kVal ? value(u) : coef, x[u]);
            } else {
              len = __popc(m);
              V c{};
              if constexpr (!kDf && !kMix && !FM::kVal) c = __ldg(a.lut + len);
#pragma unroll
              for (int u = 0; u < W; u++)
                if (m & (1 << u)) s.add(u, FM::kVal ? value(u) : c, entry(u));
            }
          };
          const V *v = s_val + k * W * 32 + lane;
          if (!FM::kVal || k < nres) {
            row([&](int u) { return v[32 * u]; });
          } else {
            const V *vg = vals + (ptrdiff_t)k * W * 32 + lane;
            V w[W];
#pragma unroll
            for (int u = 0; u < W; u++) w[u] = __ldg(vg + 32 * u);
            row([&](int u) { return w[u]; });
          }
        } else {  // any columns: the CSR row
          const int q0 = __ldg(a.ptr + i);
          len = __ldg(a.ptr + i + 1) - q0;
          const V *cf = static_cast<const V *>(a.coef);
          for (int q = 0; q < len; q++) {
            const int col = __ldg(a.col + q0 + q);
            const E x = col >= w0 && col < w1 ? in[col] : far(col);
            s.add(kIntTerms, kDf && !FM::kVal ? V{} : cf[FM::kVal ? q0 + q : i], x);
          }
        }
        if constexpr (kDf) {
          float2 r = df_norm(s.h, s.l);
          if (!FM::kVal)
            r = df_scale(pat == 0 ? coef2 : len < 256 ? __ldg(a.lut2 + len) : static_cast<const float2 *>(a.coef)[i], r);
          out[i] = r;
          if (kDeep && (unsigned)k >= (unsigned)ns) continue;
          // at an exchange others read the rows near the ends, with far diagonals any
          if ((!kDeep || left == 0) && l < a.nlevel && (kPair || i - r0 < a.halo || r1 - i <= a.halo || a.ring_all))
            a.ring[(size_t)(l / depth % 3) * a.n + i] = r;
          __stcs((host ? a.hv : a.vv) + (size_t)l * a.n + i, df_to_double(r));
        } else if constexpr (kMix) {
          const float y = s.s * a.scale;
          out[i] = y;
          if (kDeep && (unsigned)k >= (unsigned)ns) continue;
          __stcs(a.vf + (size_t)l * a.n + i, y);
        } else {
          out[i] = s.s;
          if (kDeep && (unsigned)k >= (unsigned)ns) continue;
          __stcs(a.vv + (size_t)l * a.n + i, s.s);
          if (host) a.hv[(size_t)l * a.n + i] = s.s;
        }
      }
    }
    if (kDeep && left > 0) __syncthreads();
    else if (l < a.nlevel) diag_publish(a, b, a.base + (unsigned)l);
  }
}

template <int F, int W>
const void *kernel_of(int mode) {
  if (mode == kDiagAll) return (const void *)diag_kernel<F, W, kDiagAll>;
  if (mode == kDiagDeep) return (const void *)diag_kernel<F, W, kDiagDeep>;
  if constexpr (W < 9) return (const void *)diag_kernel<F, W, kDiagPair>;
  return nullptr;
}
template <int F>
const void *kernel_of(int w, int mode) {
  return w == 5 ? kernel_of<F, 5>(mode) : w == 7 ? kernel_of<F, 7>(mode) : kernel_of<F, 9>(mode);
}

}  // namespace

namespace mpkg {

const void *diag_kernel_ptr(int form, int w, int mode) {
  switch (form) {
    case kDiagFma: return kernel_of<kDiagFma>(w, mode);
    case kDiagFmaVal: return kernel_of<kDiagFmaVal>(w, mode);
    case kDiagSep: return kernel_of<kDiagSep>(w, mode);
    case kDiagSepVal: return kernel_of<kDiagSepVal>(w, mode);
    case kDiagDf: return kernel_of<kDiagDf>(w, mode);
    case kDiagDfVal: return kernel_of<kDiagDfVal>(w, mode);
    case kDiagF32: return kernel_of<kDiagF32>(w, mode);
    case kDiagBf16: return kernel_of<kDiagBf16>(w, mode);
  }
  return nullptr;
}

int diag_elem_bytes(int form) { return form >= kDiagF32 ? 4 : 8; }
int diag_value_bytes(int form) {
  switch (form) {
    case kDiagFmaVal: case kDiagSepVal: case kDiagDfVal: return 8;
    case kDiagF32: return 4;
    case kDiagBf16: return 2;
  }
  return 0;
}

int diag_layout(int n, const int *ptr, const int *col, int nlevel, int form, int nsm, int smem, DiagLayout *out) {
  DiagLayout &l = *out;
  l.fits = false;
  const int nslice = (n + 31) / 32;
  const bool ring = form == kDiagDf || form == kDiagDfVal;
  const long eb = diag_elem_bytes(form), vb = diag_value_bytes(form);
  // the diagonals that more than half of 256 rows all over the matrix have
  std::map<int, int> seen;
  const int probes = std::min(n, 256);
  unsigned long long mix = 1;
  for (int t = 0; t < probes; t++) {
    // rows at random: a constant distance can keep to a mesh's planes
    mix = mix * 6364136223846793005ull + 1442695040888963407ull;
    const int i = n <= 256 ? t : (int)((mix >> 33) % (unsigned long long)n);
    if (ptr[i + 1] - ptr[i] > 2 * kDiagMax) return kOk;
    for (int q = ptr[i]; q < ptr[i + 1]; q++) seen[col[q] - i]++;
  }
  l.w = 0;
  for (const auto &s : seen)
    if (2 * s.second > probes) {
      if (l.w == kDiagMax) return kOk;
      l.d[l.w++] = s.first;
    }
  if (l.w != 5 && l.w != 7 && l.w != 9) return kOk;  // the kernels there are: 2-D and 3-D stencils
  const int W = l.w;
  // slice-aligned row ranges of equal length: a slice costs the same with
  // and without its holes
  const int grid = l.grid = std::min(nsm, nslice);
  l.lo.assign(grid + 1, 0);
  for (int b = 1; b <= grid; b++) l.lo[b] = (int)std::min<long>(n, 32L * ((long)nslice * b / grid));
  const int own = 32 * ((nslice + grid - 1) / grid);
  // Levels per exchange and the halo.  With one level, not 9 diagonals, the
  // halo holds all of them or all but the outermost pair: the first fetches 2
  // halo rows per CTA and level, the second two per own row, so a halo beyond
  // the own rows is taken only where the second does not do.  With more levels
  // it holds all.  A call's time in cycles, as measured: a hand-over 4500 and
  // the halo's rows, a barrier 200, a slice its share of the FP64 or issue
  // slots, a level at least the latency of one slice; once, the values of the
  // neighbours' slices.
  const bool pair = W < 9 && l.d[0] < 0 && l.d[W - 1] > 0;
  const bool fp64 = eb == 8 && !ring;
  const double per_slice = (fp64 ? 20.0 : ring ? 9.0 : 4.5) * W, least = fp64 ? 120.0 * W : ring ? 80.0 * W : 500.0;
  const long reach = std::max({0, -l.d[0], l.d[W - 1]}), ns_max = own / 32;
  l.win_bytes = (int)((own * eb + 15) / 16 * 16);
  l.grow = (int)((reach + 31) / 32);
  double best = -1;
  auto consider = [&](int depth, int g) {  // false: does not fit
    const long halo = 32L * (depth - 1) * l.grow + (g ? std::max({0, -l.d[1], l.d[W - 2]}) : reach);
    const long hb = (halo * eb + 15) / 16 * 16, most = ns_max + 2L * (depth - 1) * l.grow;
    if (2L * l.win_bytes + (depth > 1 ? 4 : 3) * hb + (2 * most + 16) > smem) return false;
    double cost = 0.4 * halo * ((nlevel + depth - 1) / depth) + 2.0 * (depth - 1) * l.grow * W * 32 * vb / 24;
    for (int lev = 0; lev < nlevel; lev++) {
      const int left = std::min(depth, nlevel - lev / depth * depth) - 1 - lev % depth;
      cost += (lev == 0 ? 0 : lev % depth == 0 ? 4500 : 200) +
              std::max(least, per_slice * std::min<long>(nslice, ns_max + 2L * left * l.grow));
    }
    if (best >= 0 && cost > 0.95 * best) return true;
    best = cost;
    l.depth = depth;
    l.mode = g ? kDiagPair : depth > 1 ? kDiagDeep : kDiagAll;
    l.halo = (int)std::min<long>(halo, n);
    l.halo_bytes = (int)hb;
    l.second = (int)(l.win_bytes + (depth > 1 ? 2 : 1) * hb);
    l.win_at = (int)(smem - l.second - l.win_bytes - hb);
    return true;
  };
  const bool near = !pair || reach <= own;
  if (!(near && consider(1, 0)) && !(pair && consider(1, 1)) && !consider(1, 0)) return kOk;  // too large
  // Rows of irregular slices run one entry after another, from the CSR, where
  // the general wavefront has 8 entries in flight.  That costs 350 cycles an
  // entry for these 8 (double-float 650, and 250 for each further one, which
  // the other forms take no slower than the general wavefront), and a CTA one
  // cycle for each of its irregular slices' entries (of a row's first 8), six
  // for those outside its window.  It has to stay below what the other slices
  // gain, of which columns beyond 16 bits, which the general wavefront reads
  // as 32, make 1.6 times as much; and one slice in twenty may be irregular.  us,
  // 5 levels, general / with any such rows / by this rule: 110^3 1/deg, every
  // 25th slice with one row of columns anywhere 168 / 104 / 104, the first 1 %
  // of the rows so 175 / 1024 / 175, the first 4 % with columns within 3000
  // 164 / 239 / 164; 100^2, 32 rows of columns anywhere 22.6 / 25.9 / 22.6;
  // double-float 110^3 212 / 116 / 116, 188 / 924 / 188, 197 / 295 / 197.
  const double spare = fp64 ? std::max(std::min(8000.0, 1900 + 130.0 * ns_max), 0.25 * per_slice * ns_max)
                            : std::max(std::min(12000.0, 2500 + 200.0 * ns_max), 0.45 * per_slice * ns_max);
  // every CTA's rows, on all host threads: the diagonals of each row, the
  // slices off them, the CTAs whose rows they read
  constexpr unsigned short kPartly = 1;  // for now: a slice that lacks some diagonals
  const unsigned short all = (unsigned short)((1 << W) - 1);
  std::vector<unsigned short> bits(n);
  l.pat.assign(nslice, 0);
  std::vector<std::vector<int>> waits(grid);
  auto owner = [&](int c) {
    int b = (int)((long)(c / 32) * grid / nslice);
    while (l.lo[b + 1] <= c) b++;
    while (l.lo[b] > c) b--;
    return b;
  };
  std::atomic<long> irregular{0}, worst{0};
  std::atomic<bool> wide{false}, refused{false};
  const bool scanned = host_parallel(grid, ptr[n], 50000, [&](int b) {
    const int r0 = l.lo[b], r1 = l.lo[b + 1];
    std::vector<char> seen(grid, 0);
    long loads = 0;
    for (int sl = r0 / 32; sl * 32 < r1 && !refused; sl++) {
      const int end = std::min(r1, sl * 32 + 32);
      bool ok = true, full = sl * 32 + 32 <= n;
      for (int i = sl * 32; i < end; i++) {
        if (ptr[i + 1] - ptr[i] > 65535) refused = true;  // by the general wavefront
        int u = 0;
        unsigned m = 0;
        for (int q = ptr[i]; q < ptr[i + 1]; q++) {
          const int c = col[q];
          if (c < r0 || c >= r1) {
            const int o = owner(c);
            if (!seen[o]) {
              seen[o] = 1;
              waits[b].push_back(o);
            }
          }
          while (u < W && l.d[u] != c - i) u++;
          if (u < W) m |= 1u << u++;
          else ok = false;
        }
        bits[i] = (unsigned short)m;
        full &= m == all;
      }
      if (ok) {
        l.pat[sl] = full ? 0 : kPartly;
        continue;
      }
      l.pat[sl] = kDiagIrregular;
      if (20 * ++irregular > nslice) refused = true;
      for (int i = sl * 32; i < end; i++) {
        const int len = ptr[i + 1] - ptr[i], ahead = std::min(len, 8);
        loads += ahead;
        for (int q = ptr[i]; q < ptr[i + 1]; q++) {
          if (q < ptr[i] + ahead && (col[q] < r0 - l.halo || col[q] >= r1 + l.halo)) loads += 5;
          if (std::abs(col[q] - i) > 32767) wide = true;
        }
        const long cost = std::max(loads, ahead * (ring ? 650L : 350L) + (ring ? (len - ahead) * 250L : 0L));
        for (long w = worst; cost > w && !worst.compare_exchange_weak(w, cost);) {
        }
      }
    }
  });
  if (!scanned) return fail(kENoMem, "diagonal layout");
  l.irregular = irregular;
  if (refused) return kOk;
  if (worst > (wide ? 1.6 : 1.0) * spare) return kOk;
  // patterns
  std::unordered_map<std::string, int> known;
  std::string m(64, 0);
  l.mask.assign(32, all);
  for (int sl = 0; sl < nslice; sl++) {
    if (l.pat[sl] != kPartly) continue;
    const int rows = std::min(32, n - sl * 32);
    std::fill(m.begin(), m.end(), 0);
    std::memcpy(&m[0], &bits[(size_t)sl * 32], 2 * rows);
    const auto f = known.emplace(m, (int)known.size() + 1);
    if (f.first->second >= kDiagIrregular) return kOk;
    l.pat[sl] = (unsigned short)f.first->second;
    if (f.second) {
      l.mask.resize(l.mask.size() + 32, 0);
      std::memcpy(&l.mask[l.mask.size() - 32], m.data(), 64);
    }
  }
  if (!irregular)  // more levels per exchange
    for (int depth = 2; depth <= std::min(nlevel, kDiagMaxDepth) && consider(depth, 0); depth++) {
    }
  // per CTA: slice ranges, resident values, dependencies
  l.own.assign(grid, make_int2(0, 0));
  l.nres.assign(grid, 0);
  long used = 0;  // bytes below the windows
  for (int b = 0; b < grid; b++) {
    const int r0 = l.lo[b], r1 = l.lo[b + 1], ns = (r1 - r0 + 31) / 32;
    const int reach_lo = std::max(0, -l.d[0]), reach_hi = std::max(0, l.d[W - 1]);
    int ka = (reach_lo + 31) / 32, kb = std::max(ka, (r1 - reach_hi - r0) / 32);
    if (ka > ns || kb > ns || ka >= kb) ka = kb = 0;
    for (int k = ka; k < kb; k++)
      if (l.pat[r0 / 32 + k] == kDiagIrregular) kb = k;
    l.own[b] = make_int2(ka, kb);
    const int s0 = r0 / 32, more = (l.depth - 1) * l.grow;
    const long all = std::min(s0, more) + ns + std::min(nslice - s0 - ns, more);
    l.slices = std::max(l.slices, (int)all);
    for (int lev = 0; lev < nlevel; lev++) {
      const int left = std::min(l.depth, nlevel - lev / l.depth * l.depth) - 1 - lev % l.depth, g = left * l.grow;
      l.rows += std::min<long>(n, 32L * (s0 + ns + std::min(nslice - s0 - ns, g))) - 32L * (s0 - std::min(s0, g));
    }
    const long pats = (2 * all + 15) / 16 * 16, room = l.win_at - l.halo_bytes - pats;
    if (vb) l.nres[b] = (int)std::min<long>(all, room / (vb * W * 32));
    used = std::max(used, pats + l.nres[b] * vb * W * 32);
    std::vector<int> &wt = waits[b];
    if (l.depth > 1)  // the rows of the halo
      for (const int end : {0, 1}) {
        const int c0 = end ? r1 : std::max(0, r0 - l.halo), c1 = end ? std::min(n, r1 + l.halo) : r0;
        if (c0 < c1)
          for (int o = owner(c0); o <= owner(c1 - 1); o++) wt.push_back(o);
      }
    std::sort(wt.begin(), wt.end());
    wt.erase(std::unique(wt.begin(), wt.end()), wt.end());
  }
  // what no CTA needs is left to other kernels
  const long slack = (l.win_at - l.halo_bytes - used) / 128 * 128;
  l.win_at -= (int)slack;
  l.smem = smem - (int)slack;
  if (ring) {  // a ring slot is reused: wait for the readers of the own rows too
    const std::vector<std::vector<int>> reads(waits);
    for (int c = 0; c < grid; c++)
      for (int b : reads[c]) waits[b].push_back(c);
  }
  l.dptr.assign(grid + 1, 0);
  l.didx.clear();
  for (int b = 0; b < grid; b++) {
    std::vector<int> &wt = waits[b];
    std::sort(wt.begin(), wt.end());
    wt.erase(std::unique(wt.begin(), wt.end()), wt.end());
    for (int c : wt) {
      l.didx.push_back(c);
      l.reach = std::max<long>(l.reach, std::abs(c - b));
    }
    l.dptr[b + 1] = (int)l.didx.size();
  }
  if (l.didx.empty()) l.didx.push_back(0);
  l.fits = true;
  return kOk;
}

}  // namespace mpkg

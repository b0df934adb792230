// pac_emu_vec.cpp -- TEST-ONLY host replay of the passes over 8-byte elements
// (pac_vec.cuh), sliced as pac_vec.cu: every tile's copy lands in a buffer
// that starts as NaN, then every step between two barriers runs for all
// threads in turn, with the per-thread registers kept in an array.
#include <algorithm>
#include <limits>
#include <vector>

#include "pac.h"
#include "pac_backend.h"
#include "pac_vec_list.h"

namespace pac {

int set_error(int status, const char* fmt, ...);

namespace {

#if PAC_VEC_SLICE % 2 == 0
using V = double;
constexpr int kBytes = 8;
#else
using V = F2;
constexpr int kBytes = 4;
#endif

template <class VP>
struct Exec {
  struct Regs {
    CV<V> v[VP::TPT];
    typename VP::Mid m;
  };
  std::vector<Regs> x;
  template <class F>
  void each(F&& f) {
    for (size_t t = 0; t < x.size(); ++t) f((int)t, x[t].v);
  }
  template <class F>
  void each_mid(F&& f) {
    for (size_t t = 0; t < x.size(); ++t) f((int)t, x[t].v, x[t].m);
  }
  void sync() {}
  void freed() {}
};

template <class VP>
void nan_fill(std::vector<CV<V>>& b) {
  double* p = (double*)b.data();
  std::fill(p, p + 2 * b.size(), std::numeric_limits<double>::quiet_NaN());
  if (kBytes == 4) {
    float* f = (float*)b.data();
    std::fill(f, f + 4 * b.size(), std::numeric_limits<float>::quiet_NaN());
  }
}

template <int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int OFFS, int PORD = 0>
int rows_as(const PassDesc& d) {
  using VP = VecPass<V, B2, MODE, SIGN, LOGL, 0, LOGW, NT, 0, OFFS, PORD>;
  using Real = typename VP::Real;
  std::vector<CV<V>> buf((size_t)VP::TILE);
  V* D = (V*)buf.data();
  std::vector<Cx<typename VP::Real>> tws((size_t)VP::TWN + 1);
  Exec<VP> ex;
  ex.x.resize(NT);
  for (int t = 0; t < NT; ++t) VP::tw_fill(d, t, tws.data());
  const long long wl = VP::W * VP::LPU, tiles = (d.nlines + wl - 1) / wl;
  for (long long tile = 0; tile < tiles; ++tile) {
    nan_fill<VP>(buf);
    const long long g0 = tile * wl, n = std::min(wl, d.nlines - g0) << LOGL;
    for (int t = 0; t < NT && d.unaligned; ++t) VP::copy_in(d, tile, t, buf.data());
    for (long long l = 0; l < n >> LOGL && !d.unaligned; ++l) {
      const long long o = VP::line_off(d, g0 + l);
      std::copy_n((const Real*)d.in_re + o, VP::L, (Real*)D + (l << LOGL));
      std::copy_n((const Real*)d.in_im + o, VP::L, (Real*)(D + VP::DIM) + (l << LOGL));
    }
    VP::template body<0>(d, tile, buf.data(), tws.data(), ex);
  }
  return PAC_SUCCESS;
}

template <int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int TW4, int DIR, int OFFS>
int cols_as(const PassDesc& d) {
  constexpr int T = DIR ? NT : (1 << (LOGL + LOGW)) / 16;
  using VP = VecPass<V, B2, MODE, SIGN, LOGL, 1, LOGW, T, DIR, OFFS>;
  std::vector<CV<V>> buf((size_t)VP::TILE);
  V* D = (V*)buf.data();
  std::vector<Cx<typename VP::Real>> tws((size_t)VP::TWN + 1);
  Exec<VP> ex;
  ex.x.resize(T);
  for (int t = 0; t < T; ++t) VP::tw_fill(d, t, tws.data());
  const int su = d.logS - ilog2(VP::LPU);
  if (LOGW > su || (d.nlines / VP::LPU) % VP::W)
    return set_error(PAC_ERROR_INTERNAL, "column tiles do not cover the lines");
  // the working layout is a bijection of the tile
  std::vector<char> seen(VP::TILE, 0);
  for (int e = 0; e < VP::L; ++e)
    for (int w = 0; w < VP::W; ++w) {
      const int q = VP::phys(w, e);
      if (q < 0 || q >= VP::TILE || seen[q]++)
        return set_error(PAC_ERROR_INTERNAL, "column layout is not a bijection");
    }
  const long long tiles = (d.nlines / VP::LPU) >> LOGW;
  const V* ire = (const V*)d.in_re;
  const V* iim = (const V*)d.in_im;
  for (long long tile = 0; tile < tiles; ++tile) {
    nan_fill<VP>(buf);
    int i0 = 0, o = 0;
    if (!VP::DIRECT) VP::tile_coords(d, tile, i0, o);
    for (int t = 0; t < T && d.unaligned && !VP::DIRECT; ++t) VP::copy_in(d, tile, t, buf.data());
    for (int e = 0; e < VP::L && !VP::DIRECT && !d.unaligned; ++e)
      for (int w = 0; w < VP::W; ++w) {
        const long long gi = ((long long)o << (LOGL + su)) + ((long long)e << su) + i0 + w;
        D[(e << LOGW) + w] = ire[gi];
        D[VP::DIM + (e << LOGW) + w] = iim[gi];
      }
    VP::template body<TW4>(d, tile, buf.data(), tws.data(), ex);
  }
  return PAC_SUCCESS;
}

template <int B2, int MODE, int SIGN, int LOGL, int TW4, int OFFS>
int small_as(const PassDesc& d) {
  for (long long u = 0; u < d.nlines / VT<V>::LPU; ++u)
    VecSmall<V, B2, MODE, SIGN, LOGL, OFFS>::template run<TW4>(d, u, [] {});
  return PAC_SUCCESS;
}

constexpr bool conv_mode(int mode, int sign) {
  return mode == MODE_CONV || (mode == MODE_DIF && sign < 0) || (mode == MODE_DIT && sign > 0);
}
int no_offsets() {
  return set_error(PAC_ERROR_INTERNAL, "a pass that takes no problem offsets");
}
template <int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT>
int go_rows(const PassDesc& d) {
  if constexpr (kBytes == 8 && MODE == MODE_DIF && SIGN < 0) {
    if (d.porder == 8) return rows_as<B2, MODE, SIGN, LOGL, LOGW, NT, 0, 8>(d);
    if (d.porder == 4) return rows_as<B2, MODE, SIGN, LOGL, LOGW, NT, 0, 4>(d);
  }
  if (!d.poff) return rows_as<B2, MODE, SIGN, LOGL, LOGW, NT, 0>(d);
  if constexpr (MODE == MODE_CONV) return rows_as<B2, MODE, SIGN, LOGL, LOGW, NT, 1>(d);
  else return no_offsets();
}
template <int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int TW4>
int go_cols(const PassDesc& d) {
  if (d.poff) {
    if constexpr (LOGL <= 8 && conv_mode(MODE, SIGN))
      return cols_as<B2, MODE, SIGN, LOGL, LOGW, NT, TW4, 1, 1>(d);
    else return no_offsets();
  }
  return cols_as<B2, MODE, SIGN, LOGL, LOGW, NT, TW4, vec_direct(MODE, LOGL, TW4), 0>(d);
}
template <int B2, int MODE, int SIGN, int LOGL, int TW4>
int go_small(const PassDesc& d) {
  if (!d.poff) return small_as<B2, MODE, SIGN, LOGL, TW4, 0>(d);
  if constexpr (conv_mode(MODE, SIGN)) return small_as<B2, MODE, SIGN, LOGL, TW4, 1>(d);
  else return no_offsets();
}

}  // namespace

#define PAC_CAT2(a, b) a##b
#define PAC_CAT(a, b) PAC_CAT2(a, b)

int PAC_CAT(replay_vec_, PAC_VEC_SLICE)(const PassDesc& d, int elem_bytes, int b2) {
  if (elem_bytes != kBytes) return -1;
  const int cols = d.logS > 0 ? 1 : 0;
  (void)cols;
#define PAC_MODES(GO, ...)                                                     \
  {                                                                            \
    if (d.mode == MODE_DIF && d.sign < 0) return GO(MODE_DIF, -1, __VA_ARGS__); \
    if (d.mode == MODE_DIF) return GO(MODE_DIF, +1, __VA_ARGS__);              \
    if (d.mode == MODE_DIT && d.sign > 0) return GO(MODE_DIT, +1, __VA_ARGS__); \
  }
#define PAC_TW4(GO, ...)                                \
  {                                                     \
    if (d.tw4_tab) PAC_MODES(GO, __VA_ARGS__, 2)        \
    else PAC_MODES(GO, __VA_ARGS__, 1)                  \
  }
#define PAC_ROW(MO, SG, B2_, LL, LW, NT_) go_rows<B2_, MO, SG, LL, LW, NT_>(d)
#define PAC_COL(MO, SG, B2_, LL, LW, NT_, TW) go_cols<B2_, MO, SG, LL, LW, NT_, TW>(d)
#define PAC_SML(MO, SG, B2_, LL, TW) go_small<B2_, MO, SG, LL, TW>(d)
#if PAC_VEC_SLICE / 2 == 0
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4)                      \
  if (d.mode == MODE_CONV && !cols && b2 == B2_ && d.logL == LL) \
    return PAC_ROW(MODE_CONV, -1, B2_, LL, LW, NT_);
  PAC_VEC_ROWS(PAC_X)
#elif PAC_VEC_SLICE / 2 == 1
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4) \
  if (!cols && b2 == B2_ && d.logL == LL) PAC_MODES(PAC_ROW, B2_, LL, LW, NT_)
  PAC_VEC_ROWS(PAC_X)
#elif PAC_VEC_SLICE / 2 == 2
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4) \
  if (cols && b2 == B2_ && d.logL == LL && !d.tw4) PAC_MODES(PAC_COL, B2_, LL, LW, NT_, 0)
  PAC_VEC_COLS2(PAC_X)
#elif PAC_VEC_SLICE / 2 == 3
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4) \
  if (cols && b2 == B2_ && d.logL == LL && d.tw4) PAC_TW4(PAC_COL, B2_, LL, LW, NT_)
  PAC_VEC_COLS2(PAC_X)
#else
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4)                                                   \
  if (cols && b2 == B2_ && d.logL == LL && !d.tw4) PAC_MODES(PAC_COL, B2_, LL, LW, NT_, 0)    \
  if (cols && b2 == B2_ && d.logL == LL && d.tw4) PAC_TW4(PAC_COL, B2_, LL, LW, NT_)
  PAC_VEC_COLS48(PAC_X)
#undef PAC_X
#define PAC_X(B2_, LL)                                                             \
  if (cols && b2 == B2_ && d.logL == LL && !d.tw4) PAC_MODES(PAC_SML, B2_, LL, 0)  \
  if (cols && b2 == B2_ && d.logL == LL && d.tw4) PAC_TW4(PAC_SML, B2_, LL)
  PAC_VEC_SMALL(PAC_X)
#endif
  return -1;
}

}  // namespace pac

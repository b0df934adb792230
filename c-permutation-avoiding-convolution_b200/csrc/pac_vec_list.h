// pac_vec_list.h -- the geometries of the passes over 8-byte elements
// (pac_vec.cuh), read by the planner, the sm_100a kernels and the test-only
// host replay.  One geometry serves FP64 lines and FP32 line pairs.
#pragma once

#include "pac_engine.cuh"
#include "pac_vec.cuh"

namespace pac {

// Tiles.  fields: log2 digit base, log2 L, columns, log2 W (line units of a
// tile), threads, CTAs per SM of the FP64 / FP32 kernel (register bound).
//
// Rows: 16 elements a thread at 128 registers, 16 warps per SM.  Lines of up
// to 512 points fit one warp, so a CTA is one warp and needs no CTA barrier:
// fused FP64 256-point rows of 2^24 elements (537 MB + H) take 95 us against
// 103 in four-warp CTAs, 512-point rows 121 against 128 (a copy: 84).  The
// scalar kernels took 105 (specialised) and 340 (generic, 1024 points).
// What bounds them: 256 points and fewer run at 88% of the copy rate; longer
// lines wait at barriers and on the FP pipes (FP64 4096 points: 57% busy at
// 159 us, 189 before).
//
// Columns of up to 256 points: rows of 128 bytes and more (64-byte rows cost
// 5-10%).  32 and 64 points hold 8 elements a thread at 24 warps per SM.
// 2^24 FP64 elements, DIF: 64 points 88 us, 128 points 89, 256 points 92
// (copied tiles: 97, 102, 108; generic kernels 163, 162, special 105).
// Longer columns get narrower rows, as the tile has to fit shared memory:
// 512 points 101, 1024 points 119 (generic 221).
#define PAC_VEC_ROWS(X)       \
  X(1, 5, 0, 4, 32, 16, 16)    \
  X(1, 6, 0, 3, 32, 16, 16)    \
  X(1, 7, 0, 2, 32, 16, 16)    \
  X(1, 8, 0, 1, 32, 16, 16)    \
  X(1, 9, 0, 0, 32, 16, 16)    \
  X(1, 10, 0, 0, 64, 8, 8)   \
  X(1, 11, 0, 0, 128, 4, 4)   \
  X(1, 12, 0, 0, 256, 2, 2)   \
  X(1, 13, 0, 0, 512, 1, 1)   \
  X(2, 6, 0, 3, 32, 16, 16)    \
  X(2, 8, 0, 1, 32, 16, 16)    \
  X(2, 10, 0, 0, 64, 8, 8)   \
  X(2, 12, 0, 0, 256, 2, 2)   \
  X(3, 6, 0, 3, 32, 16, 16)    \
  X(3, 9, 0, 0, 32, 16, 16)    \
  X(3, 12, 0, 0, 256, 2, 2)
#define PAC_VEC_COLS2(X)      \
  X(1, 5, 1, 6, 256, 3, 3)    \
  X(1, 6, 1, 5, 256, 3, 3)    \
  X(1, 7, 1, 4, 128, 4, 4)    \
  X(1, 8, 1, 4, 256, 2, 2)    \
  X(1, 9, 1, 3, 256, 2, 2)    \
  X(1, 10, 1, 2, 256, 2, 2)   \
  X(1, 11, 1, 2, 512, 1, 1)
#define PAC_VEC_COLS48(X)     \
  X(2, 6, 1, 5, 128, 4, 4)    \
  X(2, 8, 1, 4, 256, 2, 2)    \
  X(2, 10, 1, 2, 256, 2, 2)   \
  X(3, 6, 1, 5, 256, 3, 3)    \
  X(3, 9, 1, 3, 256, 2, 2)
// one-stage columns (registers only): log2 digit base, log2 L
#define PAC_VEC_SMALL(X) X(1, 1) X(1, 2) X(1, 3) X(1, 4) X(2, 2) X(2, 4) X(3, 3)

// The modes and signs that a pass of a factor can have: forward (A^T, FFT),
// the inverse FFT's DIF, conj(A), and the fused convolution (rows).  (A is
// conj(A) with real and imaginary parts exchanged.)
inline bool vec_mode(int mode, int sign, int cols) {
  if (mode == MODE_CONV) return !cols;
  return mode == MODE_DIF || (mode == MODE_DIT && sign > 0);
}

// 4-step twiddles of axes of up to this many points come from a whole table
// (FP64 16 MiB, FP32 8 MiB at 2^20), of longer ones from two-level tables
enum { PAC_TW4_TABLE_LOG = 20 };

// Columns of up to 256 points read global memory straight into registers (one
// tile a CTA); longer ones, and conj(A) passes with 4-step twiddles, whose
// twiddle loads would wait behind the data's, copy their tiles (persistent
// CTAs, 16 elements a thread).
PAC_HDC bool vec_direct(int mode, int logL, int tw4) {
  return logL <= 8 && !(mode == MODE_DIT && tw4);
}

// Dynamic shared memory of a launch of `tiles` CTAs of which `fit` fit the
// device.  On one stream fewer tiles than that are better spread over the SMs:
// CTAs that arrive while the kernel before still runs would otherwise pile up on
// the SMs that it leaves first, so each reserves its share of an SM's shared
// memory (1024 x 1024 FP32 21.6 us against 24.0, 64^3 FP64 14.2 against 17.0).
// But a reserved SM takes no CTA of another stream's either: eight plans on
// eight streams took 30.0 us a call with it against 18.6 (256 x 256 FP64), 122
// against 76 (8 x 2^16), more than the scalar kernels (20.6, 83).  So only
// launches on the legacy default stream, which other streams do not run beside
// unless they were made not to wait for it, reserve.
constexpr size_t kVecSmemSM = 228 * 1024;   // of an SM
constexpr size_t kVecSmemCTA = 226 * 1024;  // the most that a CTA may ask for (static kept)
inline size_t vec_smem(size_t smem, long long tiles, long long fit, int sms, bool legacy_stream) {
  if (!legacy_stream || fit <= 0 || tiles >= fit) return smem;
  const long long per_sm = (tiles + sms - 1) / sms;
  const size_t share = kVecSmemSM / (size_t)per_sm / 1024 * 1024 - 2048;
  if (share <= smem) return smem;
  return share < kVecSmemCTA ? share : kVecSmemCTA;
}

struct VecGeo {
  int logW = 0, nt = 0;
  size_t smem = 0;
  int small = 0;
};
inline bool vec_geometry(int b2, int mode, int sign, int logL, int cols, VecGeo* g) {
  if (!vec_mode(mode, sign, cols)) return false;
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4)                                             \
  if (b2 == B2_ && logL == LL && cols == CO) {                                          \
    g->logW = LW;                                                                       \
    g->nt = NT_;                                                                        \
    g->smem = VecPass<double, B2_, CO ? MODE_DIF : MODE_CONV, -1, LL, CO, LW, NT_>::SMEM; \
    g->small = 0;                                                                       \
    return true;                                                                        \
  }
  PAC_VEC_ROWS(PAC_X)
  PAC_VEC_COLS2(PAC_X)
  PAC_VEC_COLS48(PAC_X)
#undef PAC_X
#define PAC_X(B2_, LL)                   \
  if (cols && b2 == B2_ && logL == LL) { \
    g->logW = 0;                         \
    g->nt = 256;                         \
    g->smem = 0;                         \
    g->small = 1;                        \
    return true;                         \
  }
  PAC_VEC_SMALL(PAC_X)
#undef PAC_X
  return false;
}

// The passes are compiled in slices (PAC_VEC_SLICE, the Makefile): one
// translation unit per element type and group of lists.  A slice's launcher
// returns -1 for a pass that is not its own.
enum { PAC_VEC_SLICES = 10 };

}  // namespace pac

// pac_vec.cu -- launchers of the passes over 8-byte elements, one slice of
// them per translation unit (PAC_VEC_SLICE: element type x group).
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <mutex>

#include "pac.h"
#include "pac_backend.h"
#include "pac_vec_kernel.cuh"

namespace pac {

int set_error(int status, const char* fmt, ...);
void count_launch();

#define PAC_CU(call, what)                                                      \
  do {                                                                          \
    cudaError_t _e = (call);                                                    \
    if (_e != cudaSuccess)                                                      \
      return set_error(PAC_ERROR_CUDA, "%s: %s", what, cudaGetErrorString(_e)); \
  } while (0)

namespace {

#if PAC_VEC_SLICE % 2 == 0
using V = double;
constexpr int kBytes = 8;
#define PAC_VEC_MINB(M8, M4) M8
#else
using V = F2;
constexpr int kBytes = 4;
#define PAC_VEC_MINB(M8, M4) M4
#endif

// CTAs that fit the device with this kernel, its shared-memory limit raised
// (once per kernel and device)
struct Resident {
  std::mutex mu;
  int ctas[64] = {};
};
template <class K>
int resident(Resident& r, K kern, int nt, size_t smem, long long* out) {
  int dev = 0;
  PAC_CU(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> g(r.mu);
  const bool keep = dev >= 0 && dev < 64;
  if (keep && r.ctas[dev]) {
    *out = r.ctas[dev];
    return PAC_SUCCESS;
  }
  PAC_CU(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVecSmemCTA),
         "cudaFuncSetAttribute");
  int nb = 0, sms = 0;
  PAC_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, nt, smem),
         "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
  PAC_CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev),
         "cudaDeviceGetAttribute");
  if (nb < 1) return set_error(PAC_ERROR_INTERNAL, "pass over 8-byte elements does not fit an SM");
  if (keep) r.ctas[dev] = nb * sms;
  *out = (long long)nb * sms;
  return PAC_SUCCESS;
}

// A launch that may overlap the end of the work before it in the stream: the
// kernels set up (barriers, twiddles in shared memory) and then wait for that
// work (pdl_wait).  slots: CTAs that fit the device (negative: a CTA a tile,
// else persistent CTAs; 0 unknown); fewer tiles than that may reserve shared
// memory (vec_smem).
// (A pass that may not start early, PassDesc.dependent, is launched plainly.)
template <class K, class... A>
int pdl_launch(K kern, long long tiles, long long slots, int nt, size_t smem, cudaStream_t st,
               const PassDesc& d, const A&... args) {
  const long long fit = slots < 0 ? -slots : slots;
  long long grid = tiles;
  if (slots > 0 && tiles > slots) grid = slots;
  smem = vec_smem(smem, tiles, fit, be_num_sms(), st == nullptr || st == cudaStreamLegacy);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = d.dependent ? 1 : 0;
  PAC_CU(cudaLaunchKernelEx(&cfg, kern, d, args...), "pass over 8-byte elements");
  count_launch();
  return PAC_SUCCESS;
}

template <class VP>
int col_map(CUtensorMap* m, const void* base, const PassDesc& d) {
  auto enc = tensor_map_encoder();
  if (!enc) return set_error(PAC_ERROR_CUDA, "cuTensorMapEncodeTiled unavailable");
  const cuuint64_t S = (1ull << d.logS) / VP::LPU;
  cuuint64_t dims[3] = {S, (cuuint64_t)VP::L, (cuuint64_t)(d.nlines >> d.logS)};
  cuuint64_t strides[2] = {S * 8, S * VP::L * 8};
  cuuint32_t box[3] = {(cuuint32_t)VP::W, (cuuint32_t)VP::BOXR, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<void*>(base), dims, strides,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return set_error(PAC_ERROR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return PAC_SUCCESS;
}

template <int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int MINB, int OFFS, int PORD = 0>
int rows_as(const PassDesc& d, cudaStream_t st) {
  using VP = VecPass<V, B2, MODE, SIGN, LOGL, 0, LOGW, NT, 0, OFFS, PORD>;
  static Resident res;
  auto kern = pac_vec_rows_kernel<V, B2, MODE, SIGN, LOGL, LOGW, NT, MINB, OFFS, PORD>;
  long long slots = 0;
  int s = resident(res, kern, NT, VP::SMEM + 128, &slots);
  if (s != PAC_SUCCESS || d.vec == VEC_PREPARE) return s;
  const long long wl = VP::W * VP::LPU, tiles = (d.nlines + wl - 1) / wl;
  return pdl_launch(kern, tiles, slots, NT, VP::SMEM + 128, st, d);
}

// column tiles read straight from global memory
template <int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int MINB, int TW4, int OFFS>
int cols_direct(const PassDesc& d, cudaStream_t st) {
  using VP = VecPass<V, B2, MODE, SIGN, LOGL, 1, LOGW, NT, 1, OFFS>;
  static Resident res;
  auto kern = pac_vec_direct_kernel<V, B2, MODE, SIGN, LOGL, LOGW, NT, MINB, TW4, OFFS>;
  long long slots = 0;
  int s = resident(res, kern, NT, VP::TILE_BYTES, &slots);
  if (s != PAC_SUCCESS || d.vec == VEC_PREPARE) return s;
  const long long tiles = (d.nlines / VP::LPU) >> LOGW;
  if (tiles > 0x7fffffffLL) return set_error(PAC_ERROR_SIZE, "pass grid too large");
  return pdl_launch(kern, tiles, -slots, NT, VP::TILE_BYTES, st, d);
}

// column tiles brought in by tensor copies, 16 elements a thread
template <int B2, int MODE, int SIGN, int LOGL, int LOGW, int TW4>
int cols_copied(const PassDesc& d, cudaStream_t st) {
  constexpr int T = (1 << (LOGL + LOGW)) / 16, MB = 512 / T;
  using VP = VecPass<V, B2, MODE, SIGN, LOGL, 1, LOGW, T>;
  static Resident res;
  auto kern = pac_vec_cols_kernel<V, B2, MODE, SIGN, LOGL, LOGW, T, MB, TW4>;
  long long slots = 0;
  int s = resident(res, kern, T, VP::SMEM + 128, &slots);
  if (s != PAC_SUCCESS || d.vec == VEC_PREPARE) return s;
  CUtensorMap m[2] = {};
  if (!d.unaligned) {
    if ((s = col_map<VP>(&m[0], d.in_re, d)) != PAC_SUCCESS) return s;
    if ((s = col_map<VP>(&m[1], d.in_im, d)) != PAC_SUCCESS) return s;
  }
  const long long tiles = (d.nlines / VP::LPU) >> LOGW;
  if (tiles > 4 * slots) {
    // rounds enough to hide a launch; as a dependent launch these wide CTAs
    // cost 512 x 256 x 128 FP64 1.2%
    kern<<<(unsigned)slots, T, VP::SMEM + 128, st>>>(d, m[0], m[1]);
    PAC_CU(cudaGetLastError(), "pac_vec_cols_kernel launch");
    count_launch();
    return PAC_SUCCESS;
  }
  return pdl_launch(kern, tiles, slots, T, VP::SMEM + 128, st, d, m[0], m[1]);
}

template <int B2, int MODE, int SIGN, int LOGL, int TW4, int OFFS>
int small_as(const PassDesc& d, cudaStream_t st) {
  // few units in narrow CTAs, on more SMs (FFT of 64 FP32 problems of 16 x 16:
  // 5.7 us, in CTAs of 256 threads 7.1)
  const long long units = d.nlines / VT<V>::LPU;
  const int nt = units < 256LL * be_num_sms() ? 64 : 256;
  const long long grid = (units + nt - 1) / nt;
  if (grid > 0x7fffffffLL) return set_error(PAC_ERROR_SIZE, "pass grid too large");
  auto kern = pac_vec_small_kernel<V, B2, MODE, SIGN, LOGL, TW4, OFFS>;
  if (d.vec == VEC_PREPARE) {
    cudaFuncAttributes fa;
    PAC_CU(cudaFuncGetAttributes(&fa, kern), "cudaFuncGetAttributes");
    return PAC_SUCCESS;
  }
  return pdl_launch(kern, grid, 0, nt, 0, st, d);
}

// problems at any offset: convolutions only
constexpr bool conv_mode(int mode, int sign) {
  return mode == MODE_CONV || (mode == MODE_DIF && sign < 0) || (mode == MODE_DIT && sign > 0);
}
int no_offsets() {
  return set_error(PAC_ERROR_INTERNAL, "a pass that takes no problem offsets");
}

template <int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int MINB>
int go_rows(const PassDesc& d, cudaStream_t st) {
  if constexpr (kBytes == 8 && MODE == MODE_DIF && SIGN < 0) {
    if (d.porder == 8) return rows_as<B2, MODE, SIGN, LOGL, LOGW, NT, MINB, 0, 8>(d, st);
    if (d.porder == 4) return rows_as<B2, MODE, SIGN, LOGL, LOGW, NT, MINB, 0, 4>(d, st);
  }
  if (!d.poff) return rows_as<B2, MODE, SIGN, LOGL, LOGW, NT, MINB, 0>(d, st);
  if constexpr (MODE == MODE_CONV) return rows_as<B2, MODE, SIGN, LOGL, LOGW, NT, MINB, 1>(d, st);
  else return no_offsets();
}
template <int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int MINB, int TW4>
int go_cols(const PassDesc& d, cudaStream_t st) {
  if (d.poff) {
    if constexpr (LOGL <= 8 && conv_mode(MODE, SIGN))
      return cols_direct<B2, MODE, SIGN, LOGL, LOGW, NT, MINB, TW4, 1>(d, st);
    else return no_offsets();
  }
  if constexpr (vec_direct(MODE, LOGL, TW4))
    return cols_direct<B2, MODE, SIGN, LOGL, LOGW, NT, MINB, TW4, 0>(d, st);
  else return cols_copied<B2, MODE, SIGN, LOGL, LOGW, TW4>(d, st);
}
template <int B2, int MODE, int SIGN, int LOGL, int TW4>
int go_small(const PassDesc& d, cudaStream_t st) {
  if (!d.poff) return small_as<B2, MODE, SIGN, LOGL, TW4, 0>(d, st);
  if constexpr (conv_mode(MODE, SIGN)) return small_as<B2, MODE, SIGN, LOGL, TW4, 1>(d, st);
  else return no_offsets();
}

}  // namespace

// 0 no 4-step twiddles, 1 looked up, 2 from the whole table
static inline int vec_tw4(const PassDesc& d) { return d.tw4 ? (d.tw4_tab ? 2 : 1) : 0; }
#define PAC_CAT2(a, b) a##b
#define PAC_CAT(a, b) PAC_CAT2(a, b)

// groups: 0 fused rows; 1 DIF and DIT rows; 2 columns of base 2; 3 the same
// with 4-step twiddles; 4 columns of bases 4 and 8 and one-stage columns
int PAC_CAT(launch_vec_, PAC_VEC_SLICE)(const PassDesc& d, int elem_bytes, int b2, void* stream) {
  if (elem_bytes != kBytes) return -1;
  const int cols = d.logS > 0 ? 1 : 0;
  cudaStream_t st = (cudaStream_t)stream;
  (void)cols;
  (void)st;
#if PAC_VEC_SLICE / 2 == 0
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4)                \
  if (d.mode == MODE_CONV && !cols && b2 == B2_ && d.logL == LL) \
    return go_rows<B2_, MODE_CONV, -1, LL, LW, NT_, PAC_VEC_MINB(M8, M4)>(d, st);
  PAC_VEC_ROWS(PAC_X)
#undef PAC_X
#elif PAC_VEC_SLICE / 2 == 1
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4)                                              \
  if (!cols && b2 == B2_ && d.logL == LL) {                                              \
    if (d.mode == MODE_DIF && d.sign < 0)                                                \
      return go_rows<B2_, MODE_DIF, -1, LL, LW, NT_, PAC_VEC_MINB(M8, M4)>(d, st);       \
    if (d.mode == MODE_DIF)                                                              \
      return go_rows<B2_, MODE_DIF, +1, LL, LW, NT_, PAC_VEC_MINB(M8, M4)>(d, st);       \
    if (d.mode == MODE_DIT && d.sign > 0)                                                \
      return go_rows<B2_, MODE_DIT, +1, LL, LW, NT_, PAC_VEC_MINB(M8, M4)>(d, st);       \
  }
  PAC_VEC_ROWS(PAC_X)
#undef PAC_X
#else
#define PAC_COL(B2_, LL, LW, NT_, MB, TW)                                  \
  if (cols && b2 == B2_ && d.logL == LL && vec_tw4(d) == TW) {    \
    if (d.mode == MODE_DIF && d.sign < 0)                                  \
      return go_cols<B2_, MODE_DIF, -1, LL, LW, NT_, MB, TW>(d, st);       \
    if (d.mode == MODE_DIF)                                                \
      return go_cols<B2_, MODE_DIF, +1, LL, LW, NT_, MB, TW>(d, st);       \
    if (d.mode == MODE_DIT && d.sign > 0)                                  \
      return go_cols<B2_, MODE_DIT, +1, LL, LW, NT_, MB, TW>(d, st);       \
  }
#if PAC_VEC_SLICE / 2 == 2
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4) \
  PAC_COL(B2_, LL, LW, NT_, PAC_VEC_MINB(M8, M4), 0)
  PAC_VEC_COLS2(PAC_X)
#undef PAC_X
#elif PAC_VEC_SLICE / 2 == 3
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4) \
  PAC_COL(B2_, LL, LW, NT_, PAC_VEC_MINB(M8, M4), 1) \
  PAC_COL(B2_, LL, LW, NT_, PAC_VEC_MINB(M8, M4), 2)
  PAC_VEC_COLS2(PAC_X)
#undef PAC_X
#else
#define PAC_X(B2_, LL, CO, LW, NT_, M8, M4)          \
  PAC_COL(B2_, LL, LW, NT_, PAC_VEC_MINB(M8, M4), 0) \
  PAC_COL(B2_, LL, LW, NT_, PAC_VEC_MINB(M8, M4), 1) \
  PAC_COL(B2_, LL, LW, NT_, PAC_VEC_MINB(M8, M4), 2)
  PAC_VEC_COLS48(PAC_X)
#undef PAC_X
#define PAC_SM(B2_, LL, TW)                                               \
  if (cols && b2 == B2_ && d.logL == LL && vec_tw4(d) == TW) {   \
    if (d.mode == MODE_DIF && d.sign < 0)                                 \
      return go_small<B2_, MODE_DIF, -1, LL, TW>(d, st);                  \
    if (d.mode == MODE_DIF) return go_small<B2_, MODE_DIF, +1, LL, TW>(d, st); \
    if (d.mode == MODE_DIT && d.sign > 0)                                 \
      return go_small<B2_, MODE_DIT, +1, LL, TW>(d, st);                  \
  }
#define PAC_X(B2_, LL) PAC_SM(B2_, LL, 0) PAC_SM(B2_, LL, 1) PAC_SM(B2_, LL, 2)
  PAC_VEC_SMALL(PAC_X)
#undef PAC_X
#endif
#endif
  return -1;
}

}  // namespace pac

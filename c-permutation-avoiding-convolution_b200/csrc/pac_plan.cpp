// pac_plan.cpp -- plans and pass schedules behind pac.h.
//
// A plan splits every axis of the problem into "virtual axes" (factors) no
// longer than one CTA can hold in shared memory, and turns each operator
// into a sequence of passes (one kernel launch each):
//
//   A^T  (forward):  DIF passes over the factors in memory order; the outer
//                    factor of a split axis multiplies by the 4-step twiddle
//                    w_N^{i * rev(e)} after its stages.  Output: P_b order.
//   A, conj(A):      DIT passes in reverse order, 4-step twiddle before the
//                    stages of an outer factor.  Input: P_b order.
//   convolution:     DIF passes over all factors but the innermost, one fused
//                    pass (DIF stages, product with the filter spectrum at the
//                    same P_b positions, DIT stages) on the innermost factor,
//                    then the DIT passes back.  2m-1 launches for m factors;
//                    no pass ever permutes data in HBM.
//   fft / ifft:      DIF passes whose last factor per axis stores in natural
//                    order (self-sorting store of that pass).
//
// The reference performs the same factorisation with one stage per memory
// sweep (butterflies.c) and per-axis gather/scatter (butterflies_2d.c,
// butterflies_3d.c); the plan keeps its digit-reversal convention so the
// spectrum order is the reference's P_r F x.
#include <math.h>
#include <stdarg.h>
#include <stdlib.h>
#include <stdio.h>
#include <string.h>
#include <unistd.h>

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "pac.h"
#include "pac_backend.h"
#include "pac_host.h"
#include "pac_special.h"
#include "pac_vec_list.h"

namespace pac {

// ---------------------------------------------------------------------------
// error reporting
// ---------------------------------------------------------------------------
static thread_local char t_err[512];

int set_error(int status, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(t_err, sizeof(t_err), fmt, ap);
  va_end(ap);
  return status;
}

#define PAC_TRY(expr)                  \
  do {                                 \
    int _st = (expr);                  \
    if (_st != PAC_SUCCESS) return _st; \
  } while (0)

// ---------------------------------------------------------------------------
// schedules
// ---------------------------------------------------------------------------
struct VAx {
  int log;      // factor length 2^log
  int axis;     // real axis index
  int first;    // first factor of its axis
  int last;     // last (innermost) factor of its axis
  int b2;       // log2 of its axis's digit base
};

struct Schedule {
  int bytes = 8;  // element bytes of one real component
  int b2 = 1;     // log2 of the digit base
  int tc = 0;     // tensor-core form: radix-16 stages on the tensor cores
  // knobs (pac_tune_t): factor cap (0: built-in), largest stage radix (log2),
  // specialised kernels (-1 off, 0 default, k > 0 k-th candidate), tile shift
  int flog_cap = 0;
  int rlog_cap = 4;
  int special = 0;
  int w_shift = 0;
  int plane = 0;        // 3D: 1 plane schedule, -1 line schedule, 0 built-in
  int tables_fixed = 0; // the tables are complete and stay (allocating plans)
  int whole_tw4 = 1;    // whole 4-step tables for short axes (not for the FP32 forms' FP64
                        // schedule, which only set-up uses)
  int short_cols = 0;   // columns of at most 256 points (batches of problems at any offset)
  void* tcc = nullptr;  // its DFT operand table (tensor-core form)
  std::vector<VAx> vax;
  std::vector<std::vector<int>> rad;  // per factor: stage radix logs, DIF order
  void* pool = nullptr;               // stage twiddle tables
  std::map<std::pair<int, int>, int> tw_off;
  struct Tw4 {
    void* lo = nullptr;
    void* hi = nullptr;
    void* lo64 = nullptr;  // the same in FP64 (FP64 schedules: the same tables)
    void* hi64 = nullptr;
    int lolog = 0;
    // whole tables [k][i], keyed by the log of the factor (allocating plans)
    std::map<int, void*> tab;
  };
  std::map<int, Tw4> tw4;  // keyed by log N
  void* block = nullptr;  // the allocation that holds every table
  ~Schedule() {
    if (block) be_free(block);
    if (tcc) be_free(tcc);
  }
};

static const int kSmemBudget = 200 * 1024;

// stage radices of one factor of length 2^lg for digit base 2^b2: with
// stages of at most 4 bits the schedule the specialised kernels are compiled
// with (sched_n / sched_v, pac_stages.cuh); a tuned plan may cap them at 3
// bits (the same rule: fewest stages, bits spread evenly, larger first)
static std::vector<int> radix_schedule(int lg, int b2, int rlog_cap = 4) {
  std::vector<int> r;
  for (int i = 0; i < sched_n_cap(lg, b2, rlog_cap); ++i)
    r.push_back(sched_v_cap(lg, b2, rlog_cap, i));
  return r;
}

// Longest factor one CTA holds: 2^12 complex FP64 / 2^13 complex FP32
// (64 KiB per line).  PAC_MAX_FACTOR_LOG lowers it, which forces more
// factors per axis (used by the tests to reach 3- and 4-factor splits at
// small sizes).
static int max_factor_log(int bytes, int b2, int cap = 0) {
  int lmax = bytes == 8 ? 12 : 13;
  const char* env = getenv("PAC_MAX_FACTOR_LOG");
  if (cap > 0) {
    if (cap >= b2 && cap < lmax) lmax = cap;
  } else if (env) {
    int v = atoi(env);
    if (v >= b2 && v < lmax) lmax = v;
  }
  return lmax - lmax % b2;
}

// Device memory for a schedule's tables, carved into 256-byte aligned pieces
struct Arena {
  char* cur;
  char* end;
  void* take(size_t bytes) {
    size_t a = (bytes + 255) & ~(size_t)255;
    if (cur + a > end) return nullptr;
    void* p = cur;
    cur += a;
    return p;
  }
};

// Plans with the built-in knobs split every axis for the least time in the
// passes over 8-byte elements.  The costs are microseconds per 2^24 line-unit
// elements (537 MB moved) measured on HBM-sized arrays, FP64 and FP32 within
// 15% of each other: fused rows; columns; columns with 4-step twiddles (an
// outer factor of a split axis).  A column factor costs two passes of a
// convolution, the innermost factor one; a copy of the same bytes takes 84.
// Index: log2 of the factor; 0 where no kernel over 8-byte elements exists.
static const int kCostRow[14] = {0, 0, 0, 0, 0, 100, 96, 98, 98, 123, 130, 144, 162, 230};
static const int kCostCol[14] = {0, 84, 84, 84, 85, 87, 88, 90, 92, 101, 124, 140, 0, 0};
static const int kCostTw4[14] = {0, 90, 90, 90, 112, 92, 93, 97, 102, 108, 137, 165, 0, 0};

// The environment's kernel choices, looked up once per call (one getenv per
// choice and pass took 1 us of a call's 5).  PAC_PIPE=0 and
// PAC_SPECIAL_VARIANT=0 are the built-in choices, as if unset (PAC_COLTMA=0, no
// tensor copies, and PAC_CLUSTER_VARIANT=0, its first candidate, are not).
struct EnvChoice {
  const char *coltma = nullptr, *pipe = nullptr, *cluster = nullptr, *special = nullptr;
  // the passes run on the kernels over scalar elements
  bool scalar() const { return coltma || pipe || cluster || special; }
};
static EnvChoice env_choice() {
  EnvChoice c;
  for (char** e = environ; e && *e; ++e) {
    const char* v = *e;
    if (v[0] != 'P' || v[1] != 'A' || v[2] != 'C' || v[3] != '_') continue;
    auto is = [&](const char* name, const char** to) {
      const size_t n = strlen(name);
      if (strncmp(v + 4, name, n) == 0 && v[4 + n] == '=') *to = v + 5 + n;
    };
    is("COLTMA", &c.coltma);
    is("PIPE", &c.pipe);
    is("CLUSTER_VARIANT", &c.cluster);
    is("SPECIAL_VARIANT", &c.special);
  }
  if (c.pipe && atoi(c.pipe) == 0) c.pipe = nullptr;
  if (c.special && atoi(c.special) == 0) c.special = nullptr;
  return c;
}

// (under a kernel choice of the environment too the factors are those that the
// scalar kernels want: 64 FP64 lines of 2^16 points 96 us, 141 with these)
static bool builtin_split(const Schedule& s) {
  return !s.tc && s.flog_cap == 0 && s.rlog_cap >= 4 && s.special == 0 && s.w_shift == 0 &&
         s.plane == 0 && getenv("PAC_MAX_FACTOR_LOG") == nullptr && !env_choice().scalar();
}

// the cheapest split of an axis of 2^lg, digit base 2^b2, with 2^inner elements
// of later axes between its neighbours, into at most three factors.  Empty when
// some factor would have no kernel (short axes, long axes of large bases), and
// when a column tile of the cheapest one would not fit its stride: beside an axis
// of 2 or 4 points one pass over scalar elements is faster than more and
// shorter factors that fit (1024 problems of 1024 x 2 FP32: 55 us against 88).
static std::vector<int> cheapest_split(int lg, int b2, int inner, int bytes, bool short_cols,
                                       long long lines) {
  std::vector<int> best, cur;
  int best_cost = 1 << 30;
  bool best_fits = false;
  VecGeo g;
  // factor f at stride 2^logS
  auto cost = [&](int f, int logS, bool last) {
    const bool row = logS == 0;
    // one CTA takes 15 us for an 8192-point line: fewer lines than keep half
    // the SMs busy are faster in three passes of many tiles (one line 15 us
    // against 9.5)
    if (row && f == 13 && lines < 64) return 0;
    if (f > 13 || (short_cols && !row && f > 8)) return 0;
    if (!vec_geometry(b2, row ? MODE_CONV : MODE_DIF, -1, f, row ? 0 : 1, &g)) return 0;
    return row ? kCostRow[f] : 2 * (last ? kCostCol[f] : kCostTw4[f]);
  };
  for (int n = 1; n <= 3; ++n)
    for (int a = b2; a <= lg; a += b2)
      for (int b = n > 1 ? b2 : 0; a + b <= lg; b += b2) {
        const int c = lg - a - b;
        if ((n == 1 && a != lg) || (n == 2 && (c != 0 || b == 0)) || (n == 3 && c < b2)) {
          if (n < 2) break;
          continue;
        }
        cur.clear();
        for (int f : {a, b, c})
          if (f > 0) cur.push_back(f);
        int total = 0, logS = inner + lg;
        bool fits = true;
        for (size_t i = 0; i < cur.size() && total >= 0; ++i) {
          logS -= cur[i];
          const int v = cost(cur[i], logS, i + 1 == cur.size());
          total = v > 0 ? total + v : -1;
          fits = fits && (logS == 0 || g.logW + (bytes == 8 ? 0 : 1) <= logS);
        }
        if (total > 0 && total < best_cost) {
          best_cost = total;
          best = cur;
          best_fits = fits;
        }
        if (n < 2) break;
      }
  if (!best_fits) best.clear();
  return best;
}

// The factors of every axis and their stage radices -- the one rule every
// plan follows (allocating plans and the no-allocation entry point alike).
static int split_axes(Schedule& s, int rank, const int* logs, const int* b2s, int bytes,
                      long long batch, const Schedule* like = nullptr) {
  s.bytes = bytes;
  // lines of the innermost axis (pairs of them in FP32)
  long long lines = batch;
  int innermost = rank - 1;  // the last axis of more than one point
  while (innermost > 0 && logs[innermost] == 0) --innermost;
  for (int a = 0; a < innermost; ++a) lines <<= logs[a];
  lines = bytes == 8 ? lines : (lines + 1) / 2;
  s.b2 = b2s[rank - 1];
  if (like) s.vax = like->vax;
  for (int a = 0; a < rank && !like; ++a) {
    int lg = logs[a];
    if (lg == 0) continue;
    const int b2 = b2s[a];
    if (builtin_split(s)) {
      int inner = 0;
      for (int i = a + 1; i < rank; ++i) inner += logs[i];
      const std::vector<int> f = cheapest_split(lg, b2, inner, bytes, s.short_cols, lines);
      for (size_t i = 0; i < f.size(); ++i)
        s.vax.push_back({f[i], a, i == 0, i + 1 == f.size(), b2});
      if (!f.empty()) continue;
    }
    const int lmax = max_factor_log(bytes, b2, s.flog_cap);
    int digits = lg / b2;
    int dmax = lmax / b2;
    int nf = (digits + dmax - 1) / dmax;
    if (nf > PAC_MAX_FACTORS)
      return set_error(PAC_ERROR_SIZE, "axis %d needs %d factors (at most %d)", a, nf,
                       (int)PAC_MAX_FACTORS);
    // the innermost factor (contiguous lines, the fused pass of a
    // convolution) as long as one CTA holds; the outer factors (column
    // passes, whose tiles grow with the column length) share the rest evenly
    std::vector<int> parts(nf, 0);
    parts[nf - 1] = nf == 1 ? digits : dmax;
    const int rest = digits - parts[nf - 1];
    for (int f = 0; f < nf - 1; ++f) parts[f] = rest / (nf - 1) + (f < rest % (nf - 1) ? 1 : 0);
    for (int f = 0; f < nf; ++f) s.vax.push_back({parts[f] * b2, a, f == 0, f == nf - 1, b2});
  }
  for (auto& v : s.vax) {
    s.rad.push_back(radix_schedule(v.log, v.b2, s.rlog_cap));
    if (s.rad.back().size() > (size_t)PAC_MAX_STAGES)
      return set_error(PAC_ERROR_UNSUPPORTED_RADIX,
                       "a factor of 2^%d needs %zu stages of radix <= 2^%d (at most %d)", v.log,
                       s.rad.back().size(), s.rlog_cap, (int)PAC_MAX_STAGES);
  }
  return PAC_SUCCESS;
}

// Stage and 4-step twiddle tables of a split schedule, generated on `stream`,
// in one block: from `ar`, or allocated (s.block, with `extra` zeroed bytes
// at its start).  One cudaMalloc a schedule: each costs 10 to 100 us.
static int build_tables(Schedule& s, Arena* ar, void* stream, size_t extra = 0) {
  const int bytes = s.bytes;
  struct Piece {
    void** to;
    size_t bytes;
  };
  std::vector<Piece> pieces;
  std::vector<std::pair<int, int>> specs;
  long long total = 0;
  for (size_t i = 0; i < s.vax.size(); ++i) {
    int logK = s.vax[i].log;
    for (int rl : s.rad[i]) {
      std::pair<int, int> key(logK, rl);
      if (!s.tw_off.count(key) && logK > rl) {
        s.tw_off[key] = (int)total;
        specs.push_back(key);
        total += (1LL << (logK - rl)) * ((1LL << rl) - 1);
      }
      logK -= rl;
    }
  }
  if (total > 0) pieces.push_back({&s.pool, (size_t)total * 2 * bytes});
  // 4-step twiddles: for every non-last factor, N = L * (later factors of its axis)
  for (size_t i = 0; i < s.vax.size(); ++i) {
    if (s.vax[i].last) continue;
    int logN = 0;
    for (size_t j = i; j < s.vax.size() && s.vax[j].axis == s.vax[i].axis; ++j) logN += s.vax[j].log;
    const bool fresh = !s.tw4.count(logN);
    Schedule::Tw4& t = s.tw4[logN];  // (map nodes stay where they are)
    if (!ar && !s.tc && s.whole_tw4 && logN <= PAC_TW4_TABLE_LOG && !t.tab.count(s.vax[i].log)) {
      t.tab[s.vax[i].log] = nullptr;
      pieces.push_back({&t.tab[s.vax[i].log], (size_t)2 * bytes << logN});
    }
    if (!fresh) continue;
    t.lolog = (logN + 1) / 2;
    const size_t nlo = (size_t)1 << t.lolog, nhi = (size_t)1 << (logN - t.lolog);
    pieces.push_back({&t.lo, nlo * 2 * bytes});
    pieces.push_back({&t.hi, nhi * 2 * bytes});
    if (bytes != 8) {
      pieces.push_back({&t.lo64, nlo * 16});
      pieces.push_back({&t.hi64, nhi * 16});
    }
  }
  Arena own{nullptr, nullptr};
  if (!ar) {
    size_t need = extra;
    for (const Piece& p : pieces) need += (p.bytes + 255) & ~(size_t)255;
    if (need == 0) return PAC_SUCCESS;
    int st = be_malloc(&s.block, need);
    if (st == PAC_ERROR_ALLOC) {
      // without the whole 4-step tables, which only make passes faster
      size_t less = extra;
      std::vector<Piece> kept;
      for (const Piece& p : pieces) {
        bool whole = false;
        for (auto& kv : s.tw4)
          for (auto& f : kv.second.tab) whole = whole || p.to == &f.second;
        if (whole) continue;
        kept.push_back(p);
        less += (p.bytes + 255) & ~(size_t)255;
      }
      if (less < need) {
        pieces = kept;
        need = less;
        for (auto& kv : s.tw4) kv.second.tab.clear();
        st = be_malloc(&s.block, need);
      }
    }
    PAC_TRY(st);
    if (extra) PAC_TRY(be_memset(s.block, 0, extra, stream));
    own = {(char*)s.block + extra, (char*)s.block + need};
    ar = &own;
  }
  for (const Piece& p : pieces) {
    *p.to = ar->take(p.bytes);
    if (!*p.to) return set_error(PAC_ERROR_SIZE, "no-allocation scratch too small");
  }
  for (auto& k : specs)
    PAC_TRY(be_fill_stage_tw((char*)s.pool + (size_t)s.tw_off[k] * 2 * bytes, bytes, k.first,
                             k.second, stream));
  for (auto& kv : s.tw4) {
    const int logN = kv.first;
    Schedule::Tw4& t = kv.second;
    const long long nlo = 1LL << t.lolog, nhi = 1LL << (logN - t.lolog);
    PAC_TRY(be_fill_pow_tw(t.lo, bytes, nlo, 1, logN, stream));
    PAC_TRY(be_fill_pow_tw(t.hi, bytes, nhi, nlo, logN, stream));
    if (bytes == 8) {
      t.lo64 = t.lo;
      t.hi64 = t.hi;
    } else {
      PAC_TRY(be_fill_pow_tw(t.lo64, 8, nlo, 1, logN, stream));
      PAC_TRY(be_fill_pow_tw(t.hi64, 8, nhi, nlo, logN, stream));
    }
    for (auto& f : t.tab) PAC_TRY(be_fill_tw4(f.second, bytes, f.first, logN, stream));
  }
  return PAC_SUCCESS;
}

// The tables are filled on the legacy stream, which does not order against
// non-blocking streams: the caller finishes them before the plan is handed out.
static int build_schedule(Schedule& s, int rank, const int* logs, const int* b2s, int bytes,
                          long long batch, size_t extra = 0, const Schedule* like = nullptr) {
  PAC_TRY(split_axes(s, rank, logs, b2s, bytes, batch, like));
  PAC_TRY(build_tables(s, nullptr, nullptr, extra));
  s.tables_fixed = 1;
  return PAC_SUCCESS;
}

}  // namespace pac

// ---------------------------------------------------------------------------
// the plan object
// ---------------------------------------------------------------------------
struct pac_plan_s {
  int rank = 0;
  int dims[3] = {1, 1, 1};
  int logs[3] = {0, 0, 0};
  long long batch = 1;
  int b2 = 1;                // axis 0's digit base (log2)
  int b2s[3] = {1, 1, 1};    // every axis's
  int form = PAC_FORM_F64;
  long long N = 1;
  pac_tune_t tune = {0, 0, 0, 0, 0};      // knobs the plan was built with
  pac::Schedule main;                     // storage type of the form
  std::unique_ptr<pac::Schedule> s64;     // FP64 schedule (F32 form: filter spectrum)
  std::mutex ws_mu;
  void* ws = nullptr;  // workspace: 2 arrays of batch*N elements of the storage type
  size_t ws_bytes = 0;
  void* tmp64 = nullptr;  // FP64 temporary for the F32 filter spectrum
  size_t tmp64_bytes = 0;
  // device status word of the bounded waits (pac_plan_check_status) and
  // their spin limit in SM cycles (0: the kernels' default)
  int* status = nullptr;
  long long wait_limit = 0;
  // per-pass timing (pac_plan_set_pass_timing)
  int timing = 0;
  std::mutex t_mu;
  std::vector<void*> t_ev;
  std::vector<double> t_ms;
  long long t_calls = 0;
  ~pac_plan_s() {
    if (ws) pac::be_free(ws);
    if (tmp64) pac::be_free(tmp64);
    for (void* e : t_ev) pac::be_event_destroy(e);
  }
};

namespace pac {

struct PassSpec {
  PassDesc d;
  long long grid;
  int threads;
  size_t smem;
  bool oop;  // cannot run in place
  int b2;    // log2 digit base of the pass's axis
};

// geometry of a pass over factor vi for `batch` problems
static PassSpec make_pass(const Schedule& s, int vi, long long batch, long long N) {
  PassSpec p;
  PassDesc& d = p.d;
  memset(&d, 0, sizeof(d));
  const VAx& v = s.vax[vi];
  const int esz = s.bytes;
  const int SH = esz == 8 ? 4 : 5, NB = esz == 8 ? 16 : 32;
  d.L = 1 << v.log;
  d.logL = v.log;
  int logS = 0;
  for (size_t j = vi + 1; j < s.vax.size(); ++j) logS += s.vax[j].log;
  d.logS = logS;
  d.nlines = (batch * N) >> v.log;
  const int base_pitch = d.L + (d.L >> SH);
  long long target = (esz == 8 ? 4096 : 8192) >> v.log;
  long long W = target < 1 ? 1 : target;
  if (logS > 0) {
    if (W < 16) W = 16;
    if (W > (1LL << logS)) W = 1LL << logS;
  }
  if (s.w_shift > 0) W <<= s.w_shift;
  if (s.w_shift < 0) W >>= -s.w_shift;
  if (W < 1) W = 1;
  long long wmax = kSmemBudget / (2LL * esz * (base_pitch + NB));
  if (wmax < 1) wmax = 1;
  while (W > wmax) W >>= 1;
  if (W > 64) W = 64;
  // tiles must cover the lines exactly: W divides nlines (a batch that is
  // not a power of two makes nlines odd-factored)
  const long long lowbit = d.nlines & -d.nlines;
  if (W > lowbit) W = lowbit;
  if (W < 1) W = 1;
  d.W = (int)W;
  d.logW = 0;
  while ((1 << d.logW) < d.W) ++d.logW;
  d.pitch = pitch_for(esz, v.log, d.W);
  d.tc = s.tc;
  d.tcc = s.tcc;
  const std::vector<int>& rad = s.rad[vi];
  d.nst = (int)rad.size();
  int logK = v.log;
  int min_rl = 4;
  for (int i = 0; i < d.nst; ++i) {
    d.rlog[i] = rad[i];
    auto it = s.tw_off.find(std::make_pair(logK, rad[i]));
    d.tw_off[i] = it == s.tw_off.end() ? 0 : it->second;
    logK -= rad[i];
    if (rad[i] < min_rl) min_rl = rad[i];
  }
  d.tw = s.pool;
  long long bf = (long long)d.W << (v.log - 4 > 0 ? v.log - 4 : 0);
  int threads = (int)(bf < 32 ? 32 : bf > 256 ? 256 : bf);
  threads = (threads + 31) / 32 * 32;
  d.nthreads = threads;
  if (!v.last) {
    int logGin = 0, logSreal = 0;
    for (size_t j = vi + 1; j < s.vax.size(); ++j) {
      if (s.vax[j].axis == v.axis) logGin += s.vax[j].log;
      else logSreal += s.vax[j].log;
    }
    int logN = v.log + logGin;
    auto& t = s.tw4.at(logN);
    d.tw4_shift = logSreal;
    d.tw4_mask = (1LL << logGin) - 1;
    d.tw4_lolog = t.lolog;
    d.tw4_lo = t.lo;
    d.tw4_hi = t.hi;
    d.tw4_lo64 = t.lo64;
    d.tw4_hi64 = t.hi64;
    auto tab = t.tab.find(v.log);
    d.tw4_tab = tab == t.tab.end() ? nullptr : tab->second;
    d.tw4_logN = logN;
  }
  p.grid = d.nlines / d.W;
  p.threads = threads;
  p.smem = (size_t)2 * d.W * d.pitch * esz;
  p.oop = false;
  p.b2 = v.b2;
  return p;
}

// Switch a pass to the kernel over 8-byte elements (pac_vec.cuh) of its
// geometry.  Plans with knobs and the environment's kernel choices keep the
// kernels those select; a column tile has to lie within the stride.  Arrays that
// are not 16-byte aligned (slices of a larger one) stay here, without the copies
// that want them to be: 64 FP64 lines of 2^16 points 8 bytes off take 98 us, on
// the scalar kernels 150 (101 with the factors that those want).
static bool apply_vec(const Schedule& s, PassSpec& p, const EnvChoice& env) {
  PassDesc& d = p.d;
  if (s.special != 0 || s.w_shift != 0 || s.rlog_cap < 4 || d.plane) return false;
  // the tensor-core form's radix-16 stages have kernels of their own; a pass
  // without one is FP32 in either form
  if (d.tc)
    for (int i = 0; i < d.nst; ++i)
      if (d.rlog[i] == 4) return false;
  if (env.scalar()) return false;
  const int cols = d.logS > 0 ? 1 : 0;
  VecGeo g;
  if (!vec_geometry(p.b2, d.mode, d.sign, d.logL, cols, &g)) return false;
  if (!rads_match(d, d.logL, p.b2, 4)) return false;
  // 2048-point columns: the pipelined tensor-copy kernel (PAC_COLTMA_LIST)
  // prefetches through the whole tile (FP64 50 / 45 against 52 / 49 us on
  // 2048 x 2048, FP32 286 / 268 against 306 / 335 us on 16 of them)
  if (cols && d.logL == 11 && p.b2 == 1 && !d.nat && d.tw4 == 0 && (d.mode == MODE_DIT || d.sign < 0))
    return false;
  if (!cols && d.nat && d.nat_nf > 0) return false;
  const int logP = s.bytes == 8 ? 0 : 1;  // log2 lines of a unit
  if (cols && g.logW + logP > d.logS) return false;
  if (cols && (d.nlines >> d.logS) >= (1LL << 31)) return false;
  // (column passes load and store 8-byte values)
  const uintptr_t at = (uintptr_t)d.in_re | (uintptr_t)d.in_im | (uintptr_t)d.out_re |
                       (uintptr_t)d.out_im;
  if (cols && at % 8) return false;
  d.unaligned = at % 16 ? 1 : 0;
  d.vec = VEC_RUN;
  d.W = 1 << g.logW;
  d.logW = g.logW;
  d.nthreads = g.nt;
  p.threads = g.nt;
  const long long units = (d.nlines + logP) >> logP;
  p.grid = g.small ? (units + g.nt - 1) / g.nt : (units + d.W - 1) >> g.logW;
  p.smem = g.smem;
  return true;
}

// Switch a pass to its specialised kernel when pac_special.h has one for its
// geometry and the tile fits the lines (W divides nlines and the stride).
static void apply_special(const Schedule& s, PassSpec& p, const EnvChoice& env) {
  PassDesc& d = p.d;
  int logW = 0, nt = 0;
  if (apply_vec(s, p, env)) return;
  if (d.nat || d.plane) return;
  if (s.special < 0) return;  // tuned off
  // column pass whose tile a CTA cluster shares (W columns within the
  // stride, whole tiles), opt-in: PAC_CLUSTER_VARIANT=k picks the k-th
  // candidate geometry of the cluster list
  // (the cluster and pipelined variants have no tensor-core stages)
  // (the cluster and pipelined variants run the radix-16 schedule only)
  const char* cvar = d.tc || s.rlog_cap < 4 ? nullptr : env.cluster;
  if (d.logS > 0 && cvar != nullptr) {
    int logC = 0;
    if (cluster_geometry(s.bytes, p.b2, d.mode, d.sign, d.logL, &logW, &logC, &nt, atoi(cvar)) &&
        logW <= d.logS && (d.nlines & ((1LL << logW) - 1)) == 0) {
      d.W = 1 << logW;
      d.logW = logW;
      d.logC = logC;
      d.pitch = pitch_for(s.bytes, d.logL - logC, d.W);
      d.nthreads = nt;
      d.spec = 1;
      p.threads = nt;
      p.grid = (d.nlines >> logW) << logC;
      p.smem = (size_t)2 * d.W * d.pitch * s.bytes;
      return;
    }
  }
  // pipelined column pass, opt-in (PAC_PIPE=1): persistent CTAs, one per
  // SM, tensor-copy prefetch of the next tile (16-byte aligned input arrays
  // for the tensor maps)
  const char* pipe = d.tc || s.rlog_cap < 4 ? nullptr : env.pipe;
  if (d.logS > 0 && cvar == nullptr && pipe != nullptr &&
      pipe_geometry(s.bytes, p.b2, d.mode, d.sign, d.logL, &logW, &nt) && logW <= d.logS &&
      (d.nlines & ((1LL << logW) - 1)) == 0 && (d.nlines >> d.logS) < (1LL << 31) &&
      ((uintptr_t)d.in_re | (uintptr_t)d.in_im) % 16 == 0) {
    d.W = 1 << logW;
    d.logW = logW;
    d.pitch = pitch_for(s.bytes, d.logL, d.W);
    d.nthreads = nt;
    d.spec = 1;
    d.pipe = 1;
    const long long tiles = d.nlines >> logW;
    const long long sms = be_num_sms();
    p.threads = nt;
    p.grid = tiles < sms ? tiles : sms;
    p.smem = (size_t)2 * d.W * d.L * s.bytes + (size_t)d.W * d.pitch * s.bytes + 1024;
    return;
  }
  // column pass staged by tensor copies: PAC_COLTMA=k picks the k-th
  // candidate of its geometry, 0 none; unset, the geometry's default entry.
  // Plain DIF / DIT passes of the default radix schedule, 16-byte aligned
  // arrays; not with specialised kernels tuned off.
  const char* tv = env.coltma;
  const int tvar = (s.rlog_cap < 4 || s.special < 0) ? 0 : tv ? atoi(tv) : -1;
  int tminb = 1, tpipe = 0, tcand = 0;
  if (d.logS > 0 && cvar == nullptr && tvar != 0 && d.tw4 == 0 &&
      (d.mode == MODE_DIF || d.mode == MODE_DIT) &&
      coltma_geometry(s.bytes, p.b2, d.mode, d.sign, d.logL, d.tc, &logW, &nt, &tminb, &tpipe,
                      tvar > 0 ? tvar - 1 : -1, &tcand) &&
      rads_match(d, d.logL, p.b2, 4) && logW <= d.logS &&
      (d.nlines & ((1LL << logW) - 1)) == 0 && (d.nlines >> d.logS) < (1LL << 31) &&
      ((uintptr_t)d.in_re | (uintptr_t)d.in_im | (uintptr_t)d.out_re | (uintptr_t)d.out_im) %
              16 == 0) {
    d.W = 1 << logW;
    d.logW = logW;
    d.nthreads = nt;
    d.spec = 1;
    d.tma = tcand;
    const long long tiles = d.nlines >> logW;
    const long long slots = (long long)be_num_sms() * tminb;
    p.threads = nt;
    p.grid = tiles < slots ? tiles : slots;
    p.smem = (size_t)(tpipe ? 3 : 2) * d.W * d.L * s.bytes + 1024;
    // tensor-core form: per warpgroup two 8 KB operand tiles, and the DFT
    // operand's two 2 KB tiles
    if (d.tc) p.smem += (size_t)(nt / 128) * 16384 + 4096;
    return;
  }
  const char* var = env.special;
  int variant = s.special > 0 ? s.special : var ? atoi(var) : 0;
  const int cols = d.logS > 0 ? 1 : 0;
  const int rc = s.rlog_cap < 4 ? s.rlog_cap : 4;
  if (!special_geometry(s.bytes, p.b2, d.mode, d.sign, d.logL, cols, d.tc, rc, &logW, &nt,
                        variant)) {
    variant = 0;
    if (!special_geometry(s.bytes, p.b2, d.mode, d.sign, d.logL, cols, d.tc, rc, &logW, &nt))
      return;
  }
  const long long W = 1LL << logW;
  if ((d.nlines & (W - 1)) != 0) return;
  if (d.logS > 0 && logW > d.logS) return;
  d.W = (int)W;
  d.logW = logW;
  d.pitch = pitch_for(s.bytes, d.logL, d.W, cols, d.tc);
  d.nthreads = nt;
  d.spec = 1 + variant;
  p.threads = nt;
  p.grid = d.nlines / W;
  p.smem = (size_t)2 * d.W * d.pitch * s.bytes;
}

// A multi-plan pass whose geometry has a work-queue fast path
// (PAC_QUEUE_LIST): its tile width, and the mark that selects the
// compile-time body inside pac_queue_kernel.
static void apply_queue_special(const Schedule& s, PassSpec& p) {
  PassDesc& d = p.d;
  int logW = 0;
  const int cols = d.logS > 0 ? 1 : 0;
  if (d.nat || s.special < 0 || s.rlog_cap < 4) return;
  if (!queue_geometry(s.bytes, p.b2, d.mode, d.sign, d.logL, cols, d.tc, &logW)) return;
  const long long W = 1LL << logW;
  if ((d.nlines & (W - 1)) != 0 || (cols && logW > d.logS)) return;
  d.W = (int)W;
  d.logW = logW;
  d.pitch = pitch_for(s.bytes, d.logL, d.W, cols, d.tc);
  d.nthreads = PAC_QUEUE_THREADS;
  d.spec = 1;
  p.threads = PAC_QUEUE_THREADS;
  p.grid = d.nlines / W;
  p.smem = (size_t)2 * d.W * d.pitch * s.bytes;
}

// A pass of one stage reads global memory into registers and writes them
// back (no exchange through shared memory, unless it stores in natural order
// out of shared memory): it reserves none, so more CTAs fit per SM.
static size_t pass_smem(const PassSpec& p) {
  const PassDesc& d = p.d;
  return (d.nst == 1 && !d.nat && !d.pipe && d.logC == 0) ? 0 : p.smem;
}

// NVTX range name of a pass: its mode and line length, as bench.py names
// the passes of its per-pass breakdown ("DIF factor k", "fused innermost",
// "DIT factor k")
static void pass_range_name(const PassDesc& d, int index, char* buf, size_t n) {
  const char* mode = d.mode == MODE_CONV ? "fused innermost: DIF, x Hhat, DIT"
                     : d.mode == MODE_DIF ? "DIF" : "DIT";
  snprintf(buf, n, "pac pass %d %s 2^%d%s%s", index, mode, d.logL, d.logS > 0 ? " columns" : "",
           d.tma ? " (tensor copies)" : "");
}

static int launch(const Schedule& s, PassSpec& p, void* stream, int index = 0) {
  p.smem = pass_smem(p);
  char name[96];
  pass_range_name(p.d, index, name, sizeof(name));
  nvtxRangePushA(name);
  const int st = be_launch_pass(p.d, s.bytes, p.b2, p.grid, p.threads, p.smem, stream);
  nvtxRangePop();
  return st;
}

// Launch a pass list; with pass timing enabled, bracket every pass with
// events and accumulate the per-pass milliseconds in the plan.
static int exec_passes(pac_plan_s* pl, const Schedule& s, std::vector<PassSpec>& passes,
                       void* stream) {
  const EnvChoice env = env_choice();
  for (auto& p : passes) {
    p.d.status = pl->status;
    p.d.wait_limit = pl->wait_limit;
    // (the first pass over tables filled on this stream waits for them)
    p.d.dependent = s.tables_fixed || &p != &passes[0];
    apply_special(s, p, env);
  }
  if (!pl->timing) {
    for (size_t i = 0; i < passes.size(); ++i) PAC_TRY(launch(s, passes[i], stream, (int)i));
    return PAC_SUCCESS;
  }
  std::lock_guard<std::mutex> g(pl->t_mu);
  const size_t n = passes.size();
  while (pl->t_ev.size() < n + 1) {
    void* ev = nullptr;
    PAC_TRY(be_event_create(&ev));
    pl->t_ev.push_back(ev);
  }
  if (pl->t_ms.size() != n) {
    pl->t_ms.assign(n, 0.0);
    pl->t_calls = 0;
  }
  PAC_TRY(be_event_record(pl->t_ev[0], stream));
  for (size_t i = 0; i < n; ++i) {
    PAC_TRY(launch(s, passes[i], stream, (int)i));
    PAC_TRY(be_event_record(pl->t_ev[i + 1], stream));
  }
  for (size_t i = 0; i < n; ++i) {
    float ms = 0.f;
    PAC_TRY(be_event_elapsed(pl->t_ev[i], pl->t_ev[i + 1], &ms));
    pl->t_ms[i] += ms;
  }
  pl->t_calls++;
  return PAC_SUCCESS;
}

static int get_ws(pac_plan_s* pl, size_t bytes, void** out) {
  if (pl->ws_bytes < bytes) {
    if (pl->ws) be_free(pl->ws);
    pl->ws = nullptr;
    pl->ws_bytes = 0;
    PAC_TRY(be_malloc(&pl->ws, bytes));
    pl->ws_bytes = bytes;
  }
  *out = pl->ws;
  return PAC_SUCCESS;
}

// Run one operator of schedule s over `batch` problems.
static int run_transform(pac_plan_s* pl, const Schedule& s, int op, long long batch,
                         const void* in_re, const void* in_im, void* out_re, void* out_im,
                         double scale, int use_scale, void* stream) {
  const long long N = pl->N;
  const int m = (int)s.vax.size();
  const long long total = batch * N;
  // A x = swap(conj(A) swap(x)), swap exchanging real and imaginary parts: A
  // takes the inverse kernels with the arrays exchanged (kernels over 8-byte
  // elements; on the scalar ones of its own it took 62 us on 32 x 2^17 FP32
  // where conj(A) takes 28, and was slower than with their longer factors)
  if (op == PAC_OP_A || op == PAC_OP_UFFT) {
    std::swap(in_re, in_im);
    std::swap(out_re, out_im);
    op = PAC_OP_CONJ_A;
  }
  if (m == 0) {
    double sc = use_scale ? scale : 1.0;
    return be_scale_copy(total, s.bytes, in_re, in_im, out_re, out_im, sc, stream);
  }
  std::vector<PassSpec> passes;
  if (op == PAC_OP_AT || op == PAC_OP_FFT || op == PAC_OP_IFFT) {
    int sign = (op == PAC_OP_IFFT) ? +1 : -1;
    for (int vi = 0; vi < m; ++vi) {
      PassSpec p = make_pass(s, vi, batch, N);
      p.d.mode = MODE_DIF;
      p.d.sign = sign;
      p.d.tw4 = s.vax[vi].last ? 0 : 1;
      if (op != PAC_OP_AT && s.vax[vi].last) {
        // natural-order store of this axis
        p.d.nat = 1;
        int nf = 0, Mlog = 0;
        for (int j = vi - 1; j >= 0 && s.vax[j].axis == s.vax[vi].axis; --j) ++nf;
        for (int f = 0; f < nf; ++f) {
          p.d.nat_flog[f] = s.vax[vi - nf + f].log;
          Mlog += s.vax[vi - nf + f].log;
        }
        p.d.nat_nf = nf;
        p.d.nat_Mlog = Mlog;
        p.oop = nf > 0;
      }
      passes.push_back(p);
    }
  } else {
    for (int vi = m - 1; vi >= 0; --vi) {
      PassSpec p = make_pass(s, vi, batch, N);
      p.d.mode = MODE_DIT;
      p.d.sign = +1;
      p.d.tw4 = s.vax[vi].last ? 0 : 2;
      passes.push_back(p);
    }
  }
  if (use_scale) {
    passes.back().d.use_scale = 1;
    passes.back().d.scale = scale;
  }
  // buffer sequence: the last pass must write `out`
  const size_t arr_bytes = (size_t)total * s.bytes;
  int flips = 0;
  for (size_t i = 1; i < passes.size(); ++i) flips += passes[i].oop ? 1 : 0;
  void* ws = nullptr;
  bool need_ws = flips > 0 || (passes[0].oop && in_re == out_re);
  std::unique_lock<std::mutex> lk(pl->ws_mu, std::defer_lock);
  if (need_ws) {
    lk.lock();
    PAC_TRY(get_ws(pl, 2 * arr_bytes, &ws));
  }
  void* bre[2] = {out_re, ws};
  void* bim[2] = {out_im, ws ? (char*)ws + arr_bytes : nullptr};
  int cur = (flips % 2 == 0) ? 0 : 1;
  if (passes[0].oop && in_re == bre[cur]) cur ^= 1;  // only when in == out
  const void* src_re = in_re;
  const void* src_im = in_im;
  for (size_t i = 0; i < passes.size(); ++i) {
    PassSpec& p = passes[i];
    int dst = cur;
    if (i > 0 && p.oop) dst = cur ^ 1;
    p.d.in_re = src_re;
    p.d.in_im = src_im;
    p.d.out_re = bre[dst];
    p.d.out_im = bim[dst];
    cur = dst;
    src_re = bre[cur];
    src_im = bim[cur];
  }
  PAC_TRY(exec_passes(pl, s, passes, stream));
  if (cur != 0) PAC_TRY(be_memcpy(out_re, bre[cur], arr_bytes, CPY_D2D, stream));
  if (cur != 0) PAC_TRY(be_memcpy(out_im, bim[cur], arr_bytes, CPY_D2D, stream));
  return PAC_SUCCESS;
}

// The passes of one convolution call (2m - 1 for m factors): DIF over the
// outer factors, the fused innermost pass, DIT back; all in place in y.
// The plane schedule of a 3D convolution (pac_plane.cuh): the knob plane
// (or, at its built-in 0, PAC_PLANE=1/0; unset: off), one factor per axis,
// the default radix schedules, and a plane kernel compiled for the (N1, N2)
// planes.  Measured on FP32 256^3: 35% fewer DRAM bytes per convolution;
// against the line schedule with load/store-unit column passes the same
// time (and 13% faster on 512 x 256 x 128), but with the tensor-copy column
// passes the line schedule is faster on both (0.297 against 0.345 ms, 0.333
// against 0.350 ms), so it is the built-in choice and the tuner may still
// pick the plane schedule.
static bool plane_active(const Schedule& s, int* logC = nullptr, int* nt = nullptr) {
  int want = s.plane;
  if (want == 0) {
    const char* e = getenv("PAC_PLANE");
    want = e ? (atoi(e) ? 1 : -1) : -1;
  }
  if (want <= 0 || s.tc || s.rlog_cap < 4 || s.vax.size() != 3) return false;
  for (int i = 0; i < 3; ++i)
    if (!s.vax[i].first || !s.vax[i].last || s.vax[i].axis != i) return false;
  const int b2 = s.vax[1].b2;
  if (s.vax[2].b2 != b2) return false;
  int lc = 0, n = 0;
  if (!plane_geometry(s.bytes, b2, s.vax[1].log, s.vax[2].log, &lc, &n)) return false;
  if (s.rad[1] != radix_schedule(s.vax[1].log, b2) || s.rad[2] != radix_schedule(s.vax[2].log, b2))
    return false;
  if (logC) *logC = lc;
  if (nt) *nt = n;
  return true;
}

// The plane pass of a 3D plan over `batch` problems, in place in y: axes 1
// and 2 of every plane, stages of axis 1 then axis 2 in rlog / tw_off.
static PassSpec make_plane_pass(const Schedule& s, long long batch, long long N) {
  int logC = 0, nt = 0;
  plane_active(s, &logC, &nt);
  PassSpec p = make_pass(s, 2, batch, N);
  PassDesc& d = p.d;
  const int log1 = s.vax[1].log, log2 = s.vax[2].log;
  d.plane = 1;
  d.plane_logN1 = log1;
  d.plane_logN2 = log2;
  d.plane_n1s = (int)s.rad[1].size();
  d.nst = (int)(s.rad[1].size() + s.rad[2].size());
  int k = 0;
  for (int a = 1; a <= 2; ++a) {
    int logK = s.vax[a].log;
    for (int rl : s.rad[a]) {
      d.rlog[k] = rl;
      auto it = s.tw_off.find(std::make_pair(logK, rl));
      d.tw_off[k] = it == s.tw_off.end() ? 0 : it->second;
      logK -= rl;
      ++k;
    }
  }
  const int rc = 1 << (log1 - logC);
  d.W = rc;
  d.logW = log1 - logC;
  d.pitch = pitch_for(s.bytes, log2, rc);
  d.nthreads = nt;
  p.threads = nt;
  p.grid = ((batch * N) >> (log1 + log2)) << logC;
  p.smem = (size_t)2 * rc * d.pitch * s.bytes;
  return p;
}

static void build_conv_passes(pac_plan_s* pl, const void* x_re, const void* x_im,
                              const void* h_re, const void* h_im, int per_problem, void* y_re,
                              void* y_im, double scale, std::vector<PassSpec>& passes,
                              bool allow_plane = true, long long copies = 0) {
  const Schedule& s = pl->main;
  const long long batch = copies ? copies : pl->batch;
  const long long N = pl->N;
  const int m = (int)s.vax.size();
  const long long hmask = per_problem ? -1LL : (N - 1);
  if (allow_plane && plane_active(s)) {
    // DIF axis 0, the plane pass, DIT axis 0
    PassSpec a = make_pass(s, 0, batch, N);
    a.d.mode = MODE_DIF;
    a.d.sign = -1;
    a.d.in_re = x_re;
    a.d.in_im = x_im;
    a.d.out_re = y_re;
    a.d.out_im = y_im;
    passes.push_back(a);
    PassSpec p = make_plane_pass(s, batch, N);
    p.d.mode = MODE_CONV;
    p.d.h_re = h_re;
    p.d.h_im = h_im;
    p.d.h_mask = hmask;
    p.d.scale = scale;
    p.d.in_re = y_re;
    p.d.in_im = y_im;
    p.d.out_re = y_re;
    p.d.out_im = y_im;
    passes.push_back(p);
    PassSpec c = make_pass(s, 0, batch, N);
    c.d.mode = MODE_DIT;
    c.d.sign = +1;
    c.d.in_re = y_re;
    c.d.in_im = y_im;
    c.d.out_re = y_re;
    c.d.out_im = y_im;
    passes.push_back(c);
    return;
  }
  for (int vi = 0; vi < m - 1; ++vi) {
    PassSpec p = make_pass(s, vi, batch, N);
    p.d.mode = MODE_DIF;
    p.d.sign = -1;
    p.d.tw4 = s.vax[vi].last ? 0 : 1;
    p.d.in_re = vi == 0 ? x_re : y_re;
    p.d.in_im = vi == 0 ? x_im : y_im;
    p.d.out_re = y_re;
    p.d.out_im = y_im;
    passes.push_back(p);
  }
  {
    PassSpec p = make_pass(s, m - 1, batch, N);
    p.d.mode = MODE_CONV;
    p.d.h_re = h_re;
    p.d.h_im = h_im;
    p.d.h_mask = hmask;
    p.d.scale = scale;
    p.d.in_re = m == 1 ? x_re : y_re;
    p.d.in_im = m == 1 ? x_im : y_im;
    p.d.out_re = y_re;
    p.d.out_im = y_im;
    passes.push_back(p);
  }
  for (int vi = m - 2; vi >= 0; --vi) {
    PassSpec p = make_pass(s, vi, batch, N);
    p.d.mode = MODE_DIT;
    p.d.sign = +1;
    p.d.tw4 = s.vax[vi].last ? 0 : 2;
    p.d.in_re = y_re;
    p.d.in_im = y_im;
    p.d.out_re = y_re;
    p.d.out_im = y_im;
    passes.push_back(p);
  }
}

// The filter spectrum straight in plan order and storage type: A^T h by the
// FP64 schedule s, whose last pass stores it so (tmp: FP64 arrays of nfilters
// problems for the passes before it, may be hhat in FP64).  *done = 0 and
// nothing launched where that pass has no such kernel (pac_vec.cuh) or the
// plan's lines differ from s's.
static bool spectrum_direct(pac_plan_s* pl, const Schedule& s) {
  return s.bytes == 8 && !s.vax.empty() && !pl->main.vax.empty() &&
         s.vax.back().log == pl->main.vax.back().log && s.vax.back().b2 == pl->main.vax.back().b2;
}
static int run_spectrum(pac_plan_s* pl, const Schedule& s, long long nfilters, const double* h_re,
                        const double* h_im, void* hhat_re, void* hhat_im, double* tmp_re,
                        double* tmp_im, double scale, void* stream, int* done) {
  *done = 0;
  const int m = (int)s.vax.size();
  std::vector<PassSpec> passes;
  for (int vi = 0; vi < m; ++vi) {
    PassSpec p = make_pass(s, vi, nfilters, pl->N);
    p.d.mode = MODE_DIF;
    p.d.sign = -1;
    p.d.tw4 = s.vax[vi].last ? 0 : 1;
    p.d.in_re = vi == 0 ? h_re : tmp_re;
    p.d.in_im = vi == 0 ? h_im : tmp_im;
    p.d.out_re = vi == m - 1 ? hhat_re : tmp_re;
    p.d.out_im = vi == m - 1 ? hhat_im : tmp_im;
    passes.push_back(p);
  }
  PassDesc& d = passes.back().d;
  d.use_scale = 1;
  d.scale = scale;
  d.porder_logR = pl->main.rad.back().back();
  PassSpec probe = passes.back();
  if (!apply_vec(s, probe, env_choice())) return PAC_SUCCESS;
  d.porder = pl->main.bytes;
  *done = 1;
  return exec_passes(pl, s, passes, stream);
}

static int run_conv(pac_plan_s* pl, const void* x_re, const void* x_im, const void* h_re,
                    const void* h_im, int per_problem, void* y_re, void* y_im, double scale,
                    void* stream) {
  const Schedule& s = pl->main;
  if (s.vax.empty()) {
    const long long hmask = per_problem ? -1LL : (pl->N - 1);
    return be_pointwise(pl->batch * pl->N, s.bytes, x_re, x_im, h_re, h_im, hmask, y_re, y_im,
                        scale, stream);
  }
  std::vector<PassSpec> passes;
  build_conv_passes(pl, x_re, x_im, h_re, h_im, per_problem, y_re, y_im, scale, passes);
  return exec_passes(pl, s, passes, stream);
}

// For a batch of plans (pac_multi.cpp): the convolution pass descriptors of
// one problem in the generic kernel's geometry, with their CTA counts and
// shared-memory sizes.  A problem of one element (no factors) has none.
int plan_conv_descs(pac_plan_s* pl, const void* x_re, const void* x_im, const void* h_re,
                    const void* h_im, void* y_re, void* y_im, std::vector<PassDesc>& descs,
                    std::vector<long long>& ctas, std::vector<size_t>& smem) {
  std::vector<PassSpec> passes;
  if (!pl->main.vax.empty())  // (the work queue runs line passes only)
    build_conv_passes(pl, x_re, x_im, h_re, h_im, 0, y_re, y_im, 1.0, passes, false);
  for (auto& p : passes) apply_queue_special(pl->main, p);
  for (auto& p : passes) {
    p.smem = pass_smem(p);
    descs.push_back(p.d);
    ctas.push_back(p.grid);
    smem.push_back(p.smem);
  }
  return PAC_SUCCESS;
}
// For a batch of plans: the convolution passes of `copies` problems of the
// plan's shape at element offsets poff[0 ..] (device array) of packed arrays,
// a filter spectrum each.  Empty when some pass has no kernel that takes
// such offsets.
int plan_batch_passes(pac_plan_s* pl, long long copies, const long long* poff, const void* x_re,
                      const void* x_im, const void* h_re, const void* h_im, void* y_re,
                      void* y_im, std::vector<PassDesc>& descs, std::vector<long long>& tiles) {
  const Schedule& s = pl->main;
  const EnvChoice env = env_choice();
  descs.clear();
  tiles.clear();
  if (s.vax.empty()) return PAC_SUCCESS;
  std::vector<PassSpec> passes;
  build_conv_passes(pl, x_re, x_im, h_re, h_im, 1, y_re, y_im, 1.0, passes, false, copies);
  int logN = 0;
  for (const VAx& v : s.vax) logN += v.log;
  for (auto& p : passes) {
    if (!apply_vec(s, p, env) || (p.d.logS > 0 && p.d.logL > 8)) {
      descs.clear();
      tiles.clear();
      return PAC_SUCCESS;
    }
    p.d.poff = poff;
    p.d.logLP = logN - p.d.logL;
    p.d.status = pl->status;
    p.d.wait_limit = pl->wait_limit;
    p.d.dependent = s.tables_fixed;
    descs.push_back(p.d);
    tiles.push_back(p.grid);
  }
  return PAC_SUCCESS;
}
int plan_bytes(pac_plan_s* pl) { return pl->main.bytes; }
// the plan's waits report in *word (device memory of the caller's) from now on
void plan_set_status_word(pac_plan_s* pl, int* word) { pl->status = word; }

// Synchronise, read and clear a device status word.
int check_status_word(int* status, const char* what, void* stream) {
  int word = 0;
  PAC_TRY(be_stream_sync(stream));
  PAC_TRY(be_memcpy(&word, status, sizeof(int), CPY_D2H, stream));
  PAC_TRY(be_stream_sync(stream));
  if (word == PAC_SUCCESS) return PAC_SUCCESS;
  PAC_TRY(be_memset(status, 0, sizeof(int), stream));
  PAC_TRY(be_stream_sync(stream));
  return set_error(word, "a bounded device wait of %s gave up (status %d); the output of the "
                         "call it belongs to is incomplete", what, word);
}
// the factor lengths and stage radices of the plan (the autotuner skips a
// knob set whose schedule it has already timed)
std::string plan_signature(pac_plan_s* pl) {
  std::string sig = plane_active(pl->main) ? "plane|" : "";
  for (size_t i = 0; i < pl->main.vax.size(); ++i) {
    sig += std::to_string(pl->main.vax[i].log) + ":";
    for (int r : pl->main.rad[i]) sig += std::to_string(r) + ",";
    sig += ";";
  }
  return sig;
}
int plan_b2(pac_plan_s* pl) { return pl->b2; }

// P-order FP64 spectrum -> the plan's spectrum storage: every block of R
// positions (R the last stage radix of the innermost factor, the one the
// fused pass multiplies in) transposed to stride L/R, scaled, and rounded
// once to the plan's element type.  Plan set-up work, never part of a
// convolution.
static int to_plan_order(pac_plan_s* pl, const double* in_re, const double* in_im, int nfilters,
                         void* out_re, void* out_im, double scale, void* stream) {
  const Schedule& s = pl->main;
  const long long total = (long long)nfilters * pl->N;
  if (s.vax.empty()) {
    if (s.bytes == 8)
      return be_scale_copy(total, 8, in_re, in_im, out_re, out_im, scale, stream);
    PAC_TRY(be_round_to_f32(in_re, (float*)out_re, total, stream));
    return be_round_to_f32(in_im, (float*)out_im, total, stream);
  }
  const int logL = s.vax.back().log;
  const int logR = s.rad.back().back();
  return be_plan_order(in_re, in_im, out_re, out_im, s.bytes, logL, logR, total >> logL, scale,
                       stream);
}

// ---------------------------------------------------------------------------
// 1D convolution in caller-supplied device scratch (pac_convolve_1d_noalloc).
// The twiddle tables and the filter spectrum are carved out of `scratch` in
// 256-byte aligned pieces and regenerated on `stream` by every call, so a
// call never depends on what an earlier call left there.  Nothing here
// allocates device memory.
// ---------------------------------------------------------------------------
static int build_schedule_in_arena(Schedule& s, int logn, int batch, Arena& ar, void* stream) {
  const int logs[1] = {logn}, b2s[1] = {1};
  if (logn > 0) PAC_TRY(split_axes(s, 1, logs, b2s, 8, batch));
  return build_tables(s, &ar, stream);
}

int conv_in_scratch(void* scratch, size_t scratch_bytes, int logn, int batch, const double* x_re,
                    const double* x_im, const double* h_re, const double* h_im, double* y_re,
                    double* y_im, int* status, long long wait_limit, void* stream) {
  pac_plan_s pl;
  pl.status = status;
  pl.wait_limit = wait_limit;
  pl.rank = 1;
  pl.dims[0] = 1 << logn;
  pl.logs[0] = logn;
  pl.batch = batch;
  pl.b2 = 1;
  pl.form = PAC_FORM_F64;
  pl.N = 1LL << logn;
  Arena ar{(char*)scratch, (char*)scratch + scratch_bytes};
  int st = build_schedule_in_arena(pl.main, logn, batch, ar, stream);
  double* hre = (double*)ar.take((size_t)pl.N * 8);
  double* him = (double*)ar.take((size_t)pl.N * 8);
  if (st == PAC_SUCCESS && (!hre || !him))
    st = set_error(PAC_ERROR_SIZE, "no-allocation scratch too small");
  if (st == PAC_SUCCESS)
    st = run_transform(&pl, pl.main, PAC_OP_AT, 1, h_re, h_im, hre, him, 1.0 / (double)pl.N, 1,
                       stream);
  if (st == PAC_SUCCESS) st = to_plan_order(&pl, hre, him, 1, hre, him, 1.0, stream);
  if (st == PAC_SUCCESS) st = run_conv(&pl, x_re, x_im, hre, him, 0, y_re, y_im, 1.0, stream);
  return st;
}

}  // namespace pac

namespace pac {
// pac_noalloc.cu (the host replay: pac_emu.cpp): the status word of the
// no-allocation entry point on the current device
int noalloc_status_word(int** word);
}  // namespace pac

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace pac;

static int ilog2_exact(long long v, int b2) {
  if (v < 1) return -1;
  int lg = 0;
  while ((1LL << lg) < v) ++lg;
  if ((1LL << lg) != v) return -1;
  if (lg % b2) return -1;
  return lg;
}

namespace pac {
// pac_tune.cpp: the knobs PAC_TUNE_CACHE holds for this device and problem
bool tune_from_env_cache(int rank, const int* dims, const int* bases, int batch, int form,
                         pac_tune_t* tune);
}  // namespace pac

extern "C" {

static int create_plan(pac_plan_t* plan, int rank, const int* dims, const int* digit_bases,
                       int batch, int form, const pac_tune_t* tune, int short_cols = 0) {
  if (!plan || !dims || !digit_bases || rank < 1 || rank > 3 || batch < 1)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_plan_create: invalid rank/dims/batch");
  const pac_tune_t knobs = tune ? *tune : pac_tune_t{0, 0, 0, 0, 0};
  if (knobs.max_factor_log < 0 || knobs.max_factor_log > 13 || knobs.max_radix_log < 0 ||
      knobs.max_radix_log > 4 || knobs.special < -1 || knobs.w_shift < -6 || knobs.w_shift > 6 ||
      knobs.plane < -1 || knobs.plane > 1)
    return set_error(PAC_ERROR_INVALID_VALUE,
                     "pac_plan_create: knobs out of range (factor log %d, radix log %d, "
                     "special %d, w shift %d)",
                     knobs.max_factor_log, knobs.max_radix_log, knobs.special, knobs.w_shift);
  int b2s[3] = {1, 1, 1};
  for (int a = 0; a < rank; ++a) {
    const int base = digit_bases[a] == 0 ? 2 : digit_bases[a];
    b2s[a] = base == 2 ? 1 : base == 4 ? 2 : base == 8 ? 3 : 0;
    if (!b2s[a])
      return set_error(PAC_ERROR_UNSUPPORTED_RADIX,
                       "pac_plan_create: digit base %d (axis %d) not in {2,4,8}", base, a);
  }
  if (form != PAC_FORM_F64 && form != PAC_FORM_F32 && form != PAC_FORM_TC)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_plan_create: unknown form %d", form);
  int st = be_init();
  if (st != PAC_SUCCESS) return st;
  std::unique_ptr<pac_plan_s> p(new pac_plan_s());
  p->rank = rank;
  p->batch = batch;
  p->b2 = b2s[0];
  p->form = form;
  long long N = 1;
  for (int a = 0; a < rank; ++a) {
    int lg = ilog2_exact(dims[a], b2s[a]);
    if (lg < 0)
      return set_error(PAC_ERROR_NOT_POWER, "pac_plan_create: axis %d length %d is not a power of %d",
                       a, dims[a], 1 << b2s[a]);
    p->dims[a] = dims[a];
    p->logs[a] = lg;
    p->b2s[a] = b2s[a];
    N *= dims[a];
  }
  if (N * (long long)batch > (1LL << 40) || N > (1LL << 31))
    return set_error(PAC_ERROR_SIZE, "pac_plan_create: problem too large");
  p->N = N;
  p->tune = knobs;
  p->main.flog_cap = knobs.max_factor_log;
  p->main.rlog_cap = knobs.max_radix_log > 0 ? knobs.max_radix_log : 4;
  p->main.special = knobs.special;
  p->main.w_shift = knobs.w_shift;
  p->main.plane = knobs.plane;
  p->main.short_cols = short_cols;
  int bytes = form == PAC_FORM_F64 ? 8 : 4;
  p->main.tc = form == PAC_FORM_TC;
  // (the status word lies ahead of the tables)
  st = build_schedule(p->main, rank, p->logs, b2s, bytes, batch, 256);
  p->status = (int*)p->main.block;
  if (st != PAC_SUCCESS) return st;
  if (p->main.tc) {
    st = be_malloc(&p->main.tcc, sizeof(TcConst) * TC_CONST_SETS * 32);
    if (st == PAC_SUCCESS) st = be_fill_tc_const(p->main.tcc, nullptr);
    if (st != PAC_SUCCESS) return st;
  }
  if (bytes != 8) {
    p->s64.reset(new Schedule());
    p->s64->whole_tw4 = 0;
    // (the same factors, so that the spectrum's last pass can store plan order)
    st = build_schedule(*p->s64, rank, p->logs, b2s, 8, batch, 0,
                        builtin_split(p->main) ? &p->main : nullptr);
    if (st != PAC_SUCCESS) return st;
  }
  st = be_stream_sync(nullptr);
  if (st != PAC_SUCCESS) return st;
  *plan = p.release();
  return PAC_SUCCESS;
}

PAC_API int pac_plan_create_tuned(pac_plan_t* plan, int rank, const int* dims,
                                  const int* digit_bases, int batch, int form,
                                  const pac_tune_t* tune) {
  return create_plan(plan, rank, dims, digit_bases, batch, form, tune);
}

PAC_API int pac_plan_create_axes(pac_plan_t* plan, int rank, const int* dims,
                                 const int* digit_bases, int batch, int form) {
  pac_tune_t t;
  if (dims && digit_bases && rank >= 1 && rank <= 3 &&
      tune_from_env_cache(rank, dims, digit_bases, batch, form, &t))
    return create_plan(plan, rank, dims, digit_bases, batch, form, &t);
  return create_plan(plan, rank, dims, digit_bases, batch, form, nullptr);
}

PAC_API int pac_plan_create(pac_plan_t* plan, int rank, const int* dims, int batch,
                            int digit_base, int form) {
  const int bases[3] = {digit_base, digit_base, digit_base};
  return pac_plan_create_axes(plan, rank, dims, bases, batch, form);
}

}  // extern "C"
namespace pac {
// a multi-plan's plan of one shape: the built-in knobs (or, with `cached`, those
// of the tuning cache), factors whose passes can serve problems at any offset
int plan_create_for_batch(pac_plan_t* plan, int rank, const int* dims, const int* bases, int form,
                          int cached) {
  pac_tune_t t;
  if (cached && tune_from_env_cache(rank, dims, bases, 1, form, &t))
    return create_plan(plan, rank, dims, bases, 1, form, &t);
  return create_plan(plan, rank, dims, bases, 1, form, nullptr, 1);
}
}  // namespace pac
extern "C" {

PAC_API int pac_plan_destroy(pac_plan_t plan) {
  delete plan;
  return PAC_SUCCESS;
}

PAC_API int pac_plan_get_info(pac_plan_t plan, pac_plan_info_t* info) {
  if (!plan || !info) return set_error(PAC_ERROR_INVALID_VALUE, "pac_plan_get_info: NULL");
  memset(info, 0, sizeof(*info));
  info->n_elements = plan->N;
  info->batch = plan->batch;
  info->rank = plan->rank;
  for (int a = 0; a < 3; ++a) info->dims[a] = plan->dims[a];
  info->digit_base = 1 << plan->b2;
  for (int a = 0; a < 3; ++a) info->digit_bases[a] = a < plan->rank ? 1 << plan->b2s[a] : 0;
  info->form = plan->form;
  info->element_bytes = plan->main.bytes;
  int m = (int)plan->main.vax.size();
  info->conv_passes = m == 0 ? 1 : plane_active(plan->main) ? 3 : 2 * m - 1;
  info->transform_passes = m == 0 ? 1 : m;
  info->workspace_bytes = plan->ws_bytes + plan->tmp64_bytes;
  info->tune = plan->tune;
  return PAC_SUCCESS;
}

PAC_API int pac_filter_spectrum(pac_plan_t plan, const double* h_re, const double* h_im,
                                int nfilters, void* hhat_re, void* hhat_im, double scale,
                                pac_stream_t stream) {
  if (!plan || !h_re || !h_im || !hhat_re || !hhat_im)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_filter_spectrum: NULL argument");
  if (nfilters != 1 && nfilters != plan->batch)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_filter_spectrum: nfilters must be 1 or batch");
  if (plan->form == PAC_FORM_F64) {
    if (spectrum_direct(plan, plan->main)) {
      int done = 0;
      PAC_TRY(run_spectrum(plan, plan->main, nfilters, h_re, h_im, hhat_re, hhat_im,
                           (double*)hhat_re, (double*)hhat_im, scale, stream, &done));
      if (done) return PAC_SUCCESS;
    }
    // A^T h in P order straight into hhat, then reordered in place
    PAC_TRY(run_transform(plan, plan->main, PAC_OP_AT, nfilters, h_re, h_im, hhat_re, hhat_im,
                          scale, 1, stream));
    return to_plan_order(plan, (const double*)hhat_re, (const double*)hhat_im, nfilters, hhat_re,
                         hhat_im, 1.0, stream);
  }
  // F32 form: FP64 transform, reordered and rounded once
  std::lock_guard<std::mutex> g(plan->ws_mu);
  const bool direct = spectrum_direct(plan, *plan->s64);
  const bool one_pass = plan->s64->vax.size() == 1;
  // (one pass reads h while it writes hhat: not where they share memory.  Of
  // several passes the last reads the temporary)
  const size_t hb = (size_t)nfilters * plan->N;
  auto apart = [&](const double* a, void* b) {
    return (char*)b >= (char*)(a + hb) || (char*)a >= (char*)b + hb * sizeof(float);
  };
  if (direct && one_pass && apart(h_re, hhat_re) && apart(h_re, hhat_im) &&
      apart(h_im, hhat_re) && apart(h_im, hhat_im)) {
    int done = 0;
    PAC_TRY(run_spectrum(plan, *plan->s64, nfilters, h_re, h_im, hhat_re, hhat_im, nullptr,
                         nullptr, scale, stream, &done));
    if (done) return PAC_SUCCESS;
  }
  size_t need = (size_t)nfilters * plan->N * 2 * sizeof(double);
  if (plan->tmp64_bytes < need) {
    if (plan->tmp64) be_free(plan->tmp64);
    plan->tmp64 = nullptr;
    plan->tmp64_bytes = 0;
    PAC_TRY(be_malloc(&plan->tmp64, need));
    plan->tmp64_bytes = need;
  }
  double* tre = (double*)plan->tmp64;
  double* tim = tre + (size_t)nfilters * plan->N;
  if (direct && !one_pass) {
    int done = 0;
    PAC_TRY(run_spectrum(plan, *plan->s64, nfilters, h_re, h_im, hhat_re, hhat_im, tre, tim, scale,
                         stream, &done));
    if (done) return PAC_SUCCESS;
  }
  // the FP64 schedule never needs the workspace for A^T
  PAC_TRY(run_transform(plan, *plan->s64, PAC_OP_AT, nfilters, h_re, h_im, tre, tim, scale, 1,
                        stream));
  return to_plan_order(plan, tre, tim, nfilters, hhat_re, hhat_im, 1.0, stream);
}

PAC_API int pac_spectrum_to_plan_order(pac_plan_t plan, const double* p_re, const double* p_im,
                                       int nfilters, void* hhat_re, void* hhat_im, double scale,
                                       pac_stream_t stream) {
  if (!plan || !p_re || !p_im || !hhat_re || !hhat_im)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_spectrum_to_plan_order: NULL argument");
  if (nfilters != 1 && nfilters != plan->batch)
    return set_error(PAC_ERROR_INVALID_VALUE,
                     "pac_spectrum_to_plan_order: nfilters must be 1 or batch");
  if (plan->form != PAC_FORM_F64 && (p_re == hhat_re || p_im == hhat_im))
    return set_error(PAC_ERROR_INVALID_VALUE,
                     "pac_spectrum_to_plan_order: in place only for PAC_FORM_F64");
  return to_plan_order(plan, p_re, p_im, nfilters, hhat_re, hhat_im, scale, stream);
}

PAC_API int pac_convolve(pac_plan_t plan, const void* x_re, const void* x_im, const void* hhat_re,
                         const void* hhat_im, int hhat_per_problem, void* y_re, void* y_im,
                         double scale, pac_stream_t stream) {
  if (!plan || !x_re || !x_im || !hhat_re || !hhat_im || !y_re || !y_im)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_convolve: NULL argument");
  return run_conv(plan, x_re, x_im, hhat_re, hhat_im, hhat_per_problem ? 1 : 0, y_re, y_im, scale,
                  stream);
}

PAC_API int pac_transform(pac_plan_t plan, int op, const void* in_re, const void* in_im,
                          void* out_re, void* out_im, pac_stream_t stream) {
  if (!plan || !in_re || !in_im || !out_re || !out_im)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_transform: NULL argument");
  if (op < PAC_OP_AT || op > PAC_OP_UIFFT)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_transform: unknown op %d", op);
  bool scaled = op == PAC_OP_IFFT || op == PAC_OP_UIFFT;
  return run_transform(plan, plan->main, op, plan->batch, in_re, in_im, out_re, out_im,
                       scaled ? 1.0 / (double)plan->N : 1.0, scaled ? 1 : 0, stream);
}

PAC_API int pac_pointwise_product(long long n, const double* x_re, const double* x_im,
                                  const double* h_re, const double* h_im, double* y_re,
                                  double* y_im, double scale, pac_stream_t stream) {
  if (n < 0 || (n > 0 && (!x_re || !x_im || !h_re || !h_im || !y_re || !y_im)))
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_pointwise_product: bad argument");
  if (n == 0) return PAC_SUCCESS;
  PAC_TRY(be_init());
  return be_pointwise(n, 8, x_re, x_im, h_re, h_im, -1LL, y_re, y_im, scale, stream);
}

PAC_API int pac_scale(long long n, const double* x_re, const double* x_im, double* y_re,
                      double* y_im, double scale, pac_stream_t stream) {
  if (n < 0 || (n > 0 && (!x_re || !x_im || !y_re || !y_im)))
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_scale: bad argument");
  if (n == 0) return PAC_SUCCESS;
  PAC_TRY(be_init());
  return be_scale_copy(n, 8, x_re, x_im, y_re, y_im, scale, stream);
}

PAC_API int pac_permute(long long n, const int* rho, double* re, double* im, pac_stream_t stream) {
  if (n < 0 || (n > 0 && (!rho || !re)))
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_permute: bad argument");
  if (n == 0) return PAC_SUCCESS;
  PAC_TRY(be_init());
  return be_permute(n, rho, re, im, stream);
}

PAC_API int pac_reference_twiddles(int r, int n, double* re, double* im, pac_stream_t stream) {
  if ((r != 2 && r != 4 && r != 8) || n < 1 || !re || !im)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_reference_twiddles: bad argument");
  PAC_TRY(be_init());
  // the reference's level count (twiddle_factors.c:18, :40-45, :77-82)
  int t = 0;
  if (r == 2) {
    while (!((n >> t) & 1)) ++t;
  } else {
    int sh = r == 4 ? 2 : 3;
    for (int v = n; v > 1; v >>= sh) ++t;
  }
  if (t == 0) return PAC_SUCCESS;
  return be_fill_ref_tw(r, t, re, im, stream);
}

PAC_API int pac_malloc(void** ptr, size_t bytes) {
  if (!ptr) return set_error(PAC_ERROR_INVALID_VALUE, "pac_malloc: NULL");
  PAC_TRY(be_init());
  return be_malloc(ptr, bytes);
}
PAC_API int pac_free(void* ptr) { return ptr ? be_free(ptr) : PAC_SUCCESS; }
PAC_API int pac_memcpy_h2d(void* dst, const void* src, size_t bytes, pac_stream_t s) {
  return be_memcpy(dst, src, bytes, CPY_H2D, s);
}
PAC_API int pac_memcpy_d2h(void* dst, const void* src, size_t bytes, pac_stream_t s) {
  return be_memcpy(dst, src, bytes, CPY_D2H, s);
}
PAC_API int pac_memcpy_d2d(void* dst, const void* src, size_t bytes, pac_stream_t s) {
  return be_memcpy(dst, src, bytes, CPY_D2D, s);
}
PAC_API int pac_stream_create(pac_stream_t* s) {
  if (!s) return set_error(PAC_ERROR_INVALID_VALUE, "pac_stream_create: NULL");
  PAC_TRY(be_init());
  return be_stream_create(s);
}
PAC_API int pac_stream_destroy(pac_stream_t s) { return be_stream_destroy(s); }
PAC_API int pac_stream_synchronize(pac_stream_t s) { return be_stream_sync(s); }
PAC_API int pac_stream_set_l2_persisting(pac_stream_t stream, const void* base, size_t bytes) {
  if (bytes > 0 && !base)
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_stream_set_l2_persisting: NULL base");
  PAC_TRY(be_init());
  return be_l2_persist(stream, base, bytes);
}
PAC_API int pac_stream_wait_stream(pac_stream_t waiter, pac_stream_t waitee) {
  return be_stream_wait(waiter, waitee);
}
PAC_API long long pac_launch_count(void) { return be_launch_count(); }
PAC_API int pac_fma_peak(int elem_bytes, pac_stream_t stream, double* tflops) {
  if (!tflops || (elem_bytes != 8 && elem_bytes != 4))
    return set_error(PAC_ERROR_INVALID_VALUE, "pac_fma_peak: elem_bytes 8 or 4, tflops non-NULL");
  PAC_TRY(be_init());
  return be_fma_peak(elem_bytes, stream, tflops);
}

PAC_API int pac_plan_set_pass_timing(pac_plan_t plan, int enable) {
  if (!plan) return set_error(PAC_ERROR_INVALID_VALUE, "pac_plan_set_pass_timing: NULL");
  std::lock_guard<std::mutex> g(plan->t_mu);
  plan->timing = enable ? 1 : 0;
  plan->t_ms.clear();
  plan->t_calls = 0;
  return PAC_SUCCESS;
}

PAC_API int pac_plan_get_pass_timing(pac_plan_t plan, int max_passes, double* ms, long long* calls,
                                     int* npasses) {
  if (!plan || !npasses) return set_error(PAC_ERROR_INVALID_VALUE, "pac_plan_get_pass_timing: NULL");
  std::lock_guard<std::mutex> g(plan->t_mu);
  *npasses = (int)plan->t_ms.size();
  for (int i = 0; i < *npasses && i < max_passes; ++i) {
    if (ms) ms[i] = plan->t_ms[i];
  }
  if (calls) *calls = plan->t_calls;
  std::fill(plan->t_ms.begin(), plan->t_ms.end(), 0.0);
  plan->t_calls = 0;
  return PAC_SUCCESS;
}

PAC_API int pac_plan_set_wait_limit(pac_plan_t plan, long long cycles) {
  if (!plan) return set_error(PAC_ERROR_INVALID_VALUE, "pac_plan_set_wait_limit: NULL plan");
  plan->wait_limit = cycles > 0 ? cycles : 0;
  return PAC_SUCCESS;
}

PAC_API int pac_plan_check_status(pac_plan_t plan, pac_stream_t stream) {
  if (!plan) return set_error(PAC_ERROR_INVALID_VALUE, "pac_plan_check_status: NULL plan");
  return check_status_word(plan->status, "this plan", stream);
}

PAC_API int pac_noalloc_check_status(pac_stream_t stream) {
  PAC_TRY(be_init());
  int* word = nullptr;
  PAC_TRY(noalloc_status_word(&word));
  return check_status_word(word, "a no-allocation convolution", stream);
}

PAC_API const char* pac_status_string(int status) {
  switch (status) {
    case PAC_SUCCESS: return "success";
    case PAC_ERROR_INVALID_VALUE: return "invalid value";
    case PAC_ERROR_NOT_POWER: return "axis length is not a power of the radix";
    case PAC_ERROR_UNSUPPORTED_RADIX: return "unsupported radix";
    case PAC_ERROR_SIZE: return "problem too large";
    case PAC_ERROR_CUDA: return "CUDA error";
    case PAC_ERROR_NO_DEVICE: return "no usable sm_100 device";
    case PAC_ERROR_ALLOC: return "allocation failed";
    case PAC_ERROR_TIMEOUT: return "device wait timed out";
    default: return "internal error";
  }
}

PAC_API const char* pac_last_error(void) { return t_err; }

// pac_host.h
int pac_host_alloc(void** p, size_t bytes) { return be_host_alloc(p, bytes); }
void pac_host_free(void* p) { be_host_free(p); }
int pac_host_kind(const void* p) { return be_host_kind(p); }
int pac_host_device(void) { return be_get_device(); }
void pac_host_set_device(int device) { be_set_device(device); }
int pac_host_event_create(void** ev) { return be_sync_event_create(ev); }
void pac_host_event_destroy(void* ev) { be_event_destroy(ev); }
int pac_host_event_record(void* ev, pac_stream_t stream) { return be_event_record(ev, stream); }
int pac_host_event_wait(void* ev) { return be_event_wait(ev); }
int pac_host_fetch_status(pac_plan_t plan, int* word, pac_stream_t stream) {
  return be_memcpy(word, plan->status, sizeof(int), CPY_D2H, stream);
}

}  // extern "C"

// pac_vec.cuh -- passes over 8-byte elements: one FP64 line, or two FP32
// lines side by side.
//
// The unit of work is a "line unit": one line of doubles, or a pair of
// adjacent lines of floats whose elements travel together as a packed value
// (F2).  Both elements are 8 bytes, both run at 64 lanes per SM and clock
// (DFMA 112-124, FFMA2 / FADD2 123 G lane-instructions/s per SM measured,
// against 235 for scalar FFMA), so one set of geometries serves both types,
// and an FP32 pass issues half the arithmetic, shared-memory and twiddle
// instructions per element that a scalar one does.
//
// A tile of W line units x L elements passes through shared memory once:
//   bulk / tensor copy -> dense tile -> registers (16 elements a thread)
//   -> stages, exchanged through the same buffer in a padded (rows) or
//   swizzled (columns) layout -> registers -> global memory
// The buffer is free as soon as the last stage has read it, so the copy of
// the CTA's next tile runs under the last stage's arithmetic and stores; the
// other resident CTAs cover the rest of its latency.  Copies do not pass
// through L1, which is left to the twiddle tables.
//
// Columns of up to 256 points skip the copy: their first step reads global
// memory into registers, one tile a CTA, which keeps more loads in flight.
//
// Measured (B200, a convolution's three passes, 1024 x 2^16 FP32): 652 us,
// 1460 with the scalar kernels; 2^22 FP64 141 against 220, 5 x 1024 x 512
// FP64 transform pairs 104 against 186.
//
// The member functions are per-thread work between two CTA barriers; the
// sm_100a kernel (pac_vec_kernel.cuh) puts __syncthreads() between them, the
// host replay (pac_emu_vec.cpp) runs each for every thread in turn.
#pragma once

namespace pac {

// ---------------------------------------------------------------------------
// 8-byte values: double, and two floats (F2; lane 0 is the first line)
// ---------------------------------------------------------------------------
struct alignas(8) F2 {
  uint64_t u;
};
PAC_HD F2 f2_make(float a, float b) {
  F2 r;
#if defined(__CUDA_ARCH__)
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.u) : "f"(a), "f"(b));
#else
  r.u = (uint64_t)f32_bits(a) | ((uint64_t)f32_bits(b) << 32);
#endif
  return r;
}
PAC_HD void f2_split(F2 v, float& a, float& b) {
#if defined(__CUDA_ARCH__)
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v.u));
#else
  const uint32_t lo = (uint32_t)v.u, hi = (uint32_t)(v.u >> 32);
  __builtin_memcpy(&a, &lo, 4);
  __builtin_memcpy(&b, &hi, 4);
#endif
}
#if defined(__CUDA_ARCH__)
#define PAC_F2_BINARY(name, op, expr)                                       \
  PAC_HD F2 name(F2 a, F2 b) {                                              \
    F2 r;                                                                   \
    asm(op ".rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));       \
    return r;                                                               \
  }
#else
#define PAC_F2_BINARY(name, op, expr)      \
  PAC_HD F2 name(F2 a, F2 b) {             \
    float x0, x1, y0, y1;                  \
    f2_split(a, x0, x1);                   \
    f2_split(b, y0, y1);                   \
    return f2_make(x0 expr y0, x1 expr y1); \
  }
#endif
PAC_F2_BINARY(vadd, "add", +)
PAC_F2_BINARY(vsub, "sub", -)
PAC_F2_BINARY(vmul, "mul", *)
#undef PAC_F2_BINARY
PAC_HD F2 vneg(F2 a) {
  float x, y;
  f2_split(a, x, y);
  return f2_make(-x, -y);
}
// a * b + c
PAC_HD F2 vfma(F2 a, F2 b, F2 c) {
#if defined(__CUDA_ARCH__)
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(a.u), "l"(b.u), "l"(c.u));
  return r;
#else
  return vadd(vmul(a, b), c);
#endif
}
PAC_HD double vadd(double a, double b) { return a + b; }
PAC_HD double vsub(double a, double b) { return a - b; }
PAC_HD double vmul(double a, double b) { return a * b; }
PAC_HD double vneg(double a) { return -a; }
PAC_HD double vfma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return fma(a, b, c);
#else
  return a * b + c;
#endif
}
// c - a * b
template <class V>
PAC_HD V vnfma(V a, V b, V c) {
  return vfma(vneg(a), b, c);
}

// Loads of signals, intermediates and filter spectra.  These passes may start
// before the launch ahead of them has ended (pac_vec.cu), so what they read may
// still be written while they run: ordinary loads, after pdl_wait.  (The
// read-only path, __ldg, is for memory that nothing writes during the kernel:
// the compiler may move such a load ahead of the wait, and its cache need not
// see the writes.  It is left to the twiddle tables.)
template <class V>
PAC_HD V ld_data(const V* p) {
  return *p;
}
// the same, staying where it is written (ahead of a barrier)
template <class T>
PAC_HD T ld_now(const T* p) {
#if defined(__CUDA_ARCH__)
  T v;
  if constexpr (sizeof(T) == 8) asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  else asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
#else
  return *p;
#endif
}

template <class V>
struct VT;
template <>
struct VT<double> {
  using Real = double;
  enum { LPU = 1 };  // lines of a unit
  static PAC_HD double set(double c) { return c; }
};
template <>
struct VT<F2> {
  using Real = float;
  enum { LPU = 2 };
  static PAC_HD F2 set(double c) { return f2_make((float)c, (float)c); }
};

// complex value of V; also a twiddle (both lanes of an F2 the same)
template <class V>
struct alignas(16) CV {
  V re, im;
};
// a complex value of shared memory as one 16-byte access
template <class V>
PAC_HD CV<V> vget(const CV<V>* p) {
#if defined(__CUDA_ARCH__)
  const double2 v = *reinterpret_cast<const double2*>(p);
  CV<V> r;
  if constexpr (sizeof(typename VT<V>::Real) == 8) r = {v.x, v.y};
  else {
    r.re.u = (uint64_t)__double_as_longlong(v.x);
    r.im.u = (uint64_t)__double_as_longlong(v.y);
  }
  return r;
#else
  return *p;
#endif
}
template <class V>
PAC_HD void vput(CV<V>* p, CV<V> v) {
#if defined(__CUDA_ARCH__)
  if constexpr (sizeof(typename VT<V>::Real) == 8) {
    *reinterpret_cast<double2*>(p) = make_double2(v.re, v.im);
  } else {
    *reinterpret_cast<double2*>(p) = make_double2(__longlong_as_double((long long)v.re.u),
                                                  __longlong_as_double((long long)v.im.u));
  }
#else
  *p = v;
#endif
}
template <class V>
PAC_HD CV<V> vcadd(CV<V> a, CV<V> b) {
  return {vadd(a.re, b.re), vadd(a.im, b.im)};
}
template <class V>
PAC_HD CV<V> vcsub(CV<V> a, CV<V> b) {
  return {vsub(a.re, b.re), vsub(a.im, b.im)};
}
// a + SIGN i b, a - SIGN i b
template <int SIGN, class V>
PAC_HD CV<V> vcaddi(CV<V> a, CV<V> b) {
  if constexpr (SIGN > 0) return {vsub(a.re, b.im), vadd(a.im, b.re)};
  else return {vadd(a.re, b.im), vsub(a.im, b.re)};
}
// a * w (SIGN < 0) or a * conj(w)
template <int SIGN, class V>
PAC_HD CV<V> vctw(CV<V> a, CV<V> w) {
  const V t = vmul(a.re, w.re), s = vmul(a.im, w.re);
  if constexpr (SIGN < 0) return {vnfma(a.im, w.im, t), vfma(a.re, w.im, s)};
  else return {vfma(a.im, w.im, t), vnfma(a.re, w.im, s)};
}

// ---------------------------------------------------------------------------
// R-point DFTs in registers, natural order in and out, SIGN -1 forward.
// Radix-4 steps; a factor (1 +- i) / sqrt 2 is applied as two additions and
// the multiplication is folded into the following butterfly's FMA: 52 and
// 152 operations for R = 8 and 16 (56 and 168 for plain radix-2 steps).
// ---------------------------------------------------------------------------
template <int SIGN, class V>
PAC_HD void vdft4(CV<V>& a, CV<V>& b, CV<V>& c, CV<V>& d) {
  const CV<V> s0 = vcadd(a, c), s1 = vcsub(a, c), s2 = vcadd(b, d), s3 = vcsub(b, d);
  a = vcadd(s0, s2);
  c = vcsub(s0, s2);
  b = vcaddi<SIGN>(s1, s3);
  d = vcaddi<-SIGN>(s1, s3);
}
// 4-point DFT of (a, b w, c w^2, d w^3), w = exp(SIGN i pi / 4)
template <int SIGN, class V>
PAC_HD void vdft4_w8(CV<V>& a, CV<V>& b, CV<V>& c, CV<V>& d) {
  const V H = VT<V>::set(0.70710678118654752440);
  const CV<V> s0 = vcaddi<SIGN>(a, c), s1 = vcaddi<-SIGN>(a, c);
  const CV<V> p = vcaddi<SIGN>(b, d), q = vcaddi<-SIGN>(b, d);
  const CV<V> P = vcaddi<SIGN>(p, p), Q = vcaddi<SIGN>(q, q);  // sqrt 2 w p, sqrt 2 w q
  a = {vfma(P.re, H, s0.re), vfma(P.im, H, s0.im)};
  c = {vnfma(P.re, H, s0.re), vnfma(P.im, H, s0.im)};
  if constexpr (SIGN > 0) {
    b = {vnfma(Q.im, H, s1.re), vfma(Q.re, H, s1.im)};
    d = {vfma(Q.im, H, s1.re), vnfma(Q.re, H, s1.im)};
  } else {
    b = {vfma(Q.im, H, s1.re), vnfma(Q.re, H, s1.im)};
    d = {vnfma(Q.im, H, s1.re), vfma(Q.re, H, s1.im)};
  }
}
// 4-point DFT of (a, b u, c u^2, d u^3), u = exp(SIGN i pi / 8) (Q = 1) or
// its cube (Q = 3)
template <int SIGN, int Q, class V>
PAC_HD void vdft4_w16(CV<V>& a, CV<V>& b, CV<V>& c, CV<V>& d) {
  constexpr double C1 = 0.92387953251128675613, S1 = 0.38268343236508977173;
  const V H = VT<V>::set(0.70710678118654752440);
  // u = cb + SIGN i sb, u^3 = cd + SIGN i sd
  const V cb = VT<V>::set(Q == 1 ? C1 : S1), sb = VT<V>::set(SIGN * (Q == 1 ? S1 : C1));
  const V cd = VT<V>::set(Q == 1 ? S1 : -C1), sd = VT<V>::set(SIGN * (Q == 1 ? C1 : -S1));
  // c u^2: (1 + SIGN i) H (Q = 1), (-1 + SIGN i) H (Q = 3)
  CV<V> s0, s1;
  if constexpr (Q == 1) {
    const CV<V> P = vcaddi<SIGN>(c, c);
    s0 = {vfma(P.re, H, a.re), vfma(P.im, H, a.im)};
    s1 = {vnfma(P.re, H, a.re), vnfma(P.im, H, a.im)};
  } else {
    const CV<V> P = vcaddi<-SIGN>(c, c);  // -(-1 + SIGN i) c = (1 - SIGN i) c
    s0 = {vnfma(P.re, H, a.re), vnfma(P.im, H, a.im)};
    s1 = {vfma(P.re, H, a.re), vfma(P.im, H, a.im)};
  }
  const CV<V> z = {vnfma(b.im, sb, vmul(b.re, cb)), vfma(b.re, sb, vmul(b.im, cb))};
  const CV<V> p = {vfma(d.re, cd, vnfma(d.im, sd, z.re)), vfma(d.im, cd, vfma(d.re, sd, z.im))};
  const CV<V> q = {vnfma(d.re, cd, vfma(d.im, sd, z.re)), vnfma(d.im, cd, vnfma(d.re, sd, z.im))};
  a = vcadd(s0, p);
  c = vcsub(s0, p);
  b = vcaddi<SIGN>(s1, q);
  d = vcaddi<-SIGN>(s1, q);
}

template <int R, int SIGN, class V>
PAC_HD void vdft(CV<V> (&x)[R]) {
  static_assert(R == 2 || R == 4 || R == 8 || R == 16, "radix");
  if constexpr (R == 2) {
    const CV<V> s = vcadd(x[0], x[1]), t = vcsub(x[0], x[1]);
    x[0] = s;
    x[1] = t;
  } else if constexpr (R == 4) {
    vdft4<SIGN>(x[0], x[1], x[2], x[3]);
  } else if constexpr (R == 8) {
    CV<V> s[4], t[4];
    static_for<4>([&](auto jj) {
      constexpr int j = jj.value;
      s[j] = vcadd(x[j], x[j + 4]);
      t[j] = vcsub(x[j], x[j + 4]);
    });
    vdft4<SIGN>(s[0], s[1], s[2], s[3]);
    vdft4_w8<SIGN>(t[0], t[1], t[2], t[3]);
    static_for<4>([&](auto kk) {
      x[2 * kk.value] = s[kk.value];
      x[2 * kk.value + 1] = t[kk.value];
    });
  } else {
    static_for<4>([&](auto jj) {
      constexpr int j = jj.value;
      vdft4<SIGN>(x[j], x[j + 4], x[j + 8], x[j + 12]);
    });
    // x[j + 4 q] now holds sub-sequence q at j; its 4-point DFT over j
    // (twiddled by exp(SIGN 2 pi i j q / 16)) gives outputs q + 4 k
    vdft4<SIGN>(x[0], x[1], x[2], x[3]);
    vdft4_w16<SIGN, 1>(x[4], x[5], x[6], x[7]);
    vdft4_w8<SIGN>(x[8], x[9], x[10], x[11]);
    vdft4_w16<SIGN, 3>(x[12], x[13], x[14], x[15]);
    CV<V> y[16];
    static_for<16>([&](auto ii) {
      constexpr int q = ii.value >> 2, k = ii.value & 3;
      y[q + 4 * k] = x[ii.value];
    });
    static_for<16>([&](auto ii) { x[ii.value] = y[ii.value]; });
  }
}

// ---------------------------------------------------------------------------
// Twiddles
// ---------------------------------------------------------------------------
PAC_HD CV<double> vtw(const Cx<double>& w) { return {w.re, w.im}; }
PAC_HD CV<F2> vtw(const Cx<float>& w) { return {f2_make(w.re, w.re), f2_make(w.im, w.im)}; }
// x[s] *= w_K^{j s} (SIGN < 0) or its conjugate, s = 1 .. R-1, from rows of
// ell entries of a CTA's copy of the stage table (VecPass::tw_fill), tw at
// entry j of row 0.  FP64 at radix >= 4 keeps the rows of w^1, w^2, w^4, w^8
// and forms the other powers (w^3 = w^2 w, w^12 = w^8 w^4, the rest one
// product more; as deep as stage_twiddles); FP32 has a row for every power
// and uses the entries as they were rounded.
template <int R, int SIGN, bool TABLE, class V>
PAC_HD void vtwiddle(CV<V> (&x)[R], const Cx<typename VT<V>::Real>* tw, int ell) {
  if constexpr (sizeof(typename VT<V>::Real) == 8 && R >= 4) {
    CV<V> w[4], w4;
    auto row = [&](int r) { return TABLE ? vtw(ld_tw(tw + ((1 << r) - 1) * ell)) : vtw(tw[r * ell]); };
    w[1] = row(0);
    w[2] = row(1);
    w[3] = vctw<-1>(w[2], w[1]);
    static_for<3>([&](auto ss) { x[ss.value + 1] = vctw<SIGN>(x[ss.value + 1], w[ss.value + 1]); });
    static_for<R / 4>([&](auto qq) {
      constexpr int q = qq.value;  // powers 4q .. 4q + 3
      if constexpr (q > 0) {
        CV<V> b;
        if constexpr (q == 3) b = vctw<-1>(w[0], w4);
        else b = row(q + 1);
        if constexpr (q == 1) w4 = b;
        if constexpr (q == 2) w[0] = b;
        x[4 * q] = vctw<SIGN>(x[4 * q], b);
        static_for<3>([&](auto ss) {
          constexpr int s = ss.value + 1;
          x[4 * q + s] = vctw<SIGN>(x[4 * q + s], vctw<-1>(b, w[s]));
        });
      }
    });
  } else {
    static_for<R - 1>([&](auto ss) {
      constexpr int s = ss.value + 1;
      x[s] = vctw<SIGN>(x[s], TABLE ? vtw(ld_tw(tw + (s - 1) * ell)) : vtw(tw[(s - 1) * ell]));
    });
  }
}

// The 4-step twiddles w_N^{iG (r0 + t L/R)}, t = 0 .. R-1, of an innermost
// butterfly (ell = 1): iG is the line's index among the later factors, r0 the
// reversed block index, t the reversed slot.  With b = w^{iG r0} and z =
// w^{iG L/R} they are (b z^{4q}) z^r, t = 4q + r: five values looked up in the
// two-level FP64 tables instead of one per element (32 gathers a butterfly),
// and products, which an HBM-bound column pass has the pipe for.  FP32 forms
// the factors b z^{4q} and z^r in FP64 and rounds them once, so a twiddle
// takes three FP32 roundings, as the product of two FP32 table entries does.
struct Tw4Look {
  const Cx<double>*lo, *hi;
  uint32_t mask;
  int lolog;
  PAC_HD CV<double> operator()(uint32_t E) const {
    return vctw<-1>(vtw(ld_tw(lo + (E & mask))), vtw(ld_tw(hi + (E >> lolog))));
  }
};
// the values of the unit's lines (a pair of FP32 lines has two) as one
PAC_HD void vjoin(const CV<double> (&v)[1], CV<double>& o) { o = v[0]; }
PAC_HD void vjoin(const CV<double> (&v)[2], CV<F2>& o) {
  o = {f2_make((float)v[0].re, (float)v[1].re), f2_make((float)v[0].im, (float)v[1].im)};
}
// register s of a butterfly (of block blk in a line of 2^logL, unit's first
// line g0) is at slot rev(s), so its t is s
//
// TW4 = 2: axes of up to 2^PAC_TW4_TABLE_LOG points have the whole table
// w_N^{k i} in [k][i] order, rounded once from FP64: one coalesced load per
// element (an FP32 pair's two entries are adjacent), out of L2.
PAC_HD CV<double> vtw4_entry(const Cx<double>* p, bool) { return vtw(ld_tw(p)); }
PAC_HD CV<F2> vtw4_entry(const Cx<float>* p, bool pair) {
  if (!pair) return vtw(ld_tw(p));  // both lines have the same index
#if defined(__CUDA_ARCH__)
  const float4 v = __ldg(reinterpret_cast<const float4*>(p));
  return {f2_make(v.x, v.z), f2_make(v.y, v.w)};
#else
  return {f2_make(p[0].re, p[1].re), f2_make(p[0].im, p[1].im)};
#endif
}
template <int R, int SIGN, int B2, class V>
PAC_HD void vtw4_table(const PassDesc& d, long long g0, int blk, int logL, CV<V> (&y)[R]) {
  constexpr int LR = ilog2(R);
  const long long i = g0 & ((1LL << d.logS) - 1);
  const uint32_t iG = (uint32_t)((i >> d.tw4_shift) & d.tw4_mask);
  const uint32_t r0 = drev<B2>((uint32_t)blk, logL - LR);
  const int logM = d.tw4_logN - logL;  // later factors of the axis
  const Cx<typename VT<V>::Real>* tab =
      (const Cx<typename VT<V>::Real>*)d.tw4_tab + ((size_t)r0 << logM) + iG;
  const bool pair = d.tw4_shift == 0;
  static_for<R>([&](auto ss) {
    y[ss.value] = vctw<SIGN>(
        y[ss.value], vtw4_entry(tab + ((size_t)ss.value << (logM + logL - LR)), pair));
  });
}
template <int TW4, int R, int SIGN, int B2, bool ONEBLK, class V>
PAC_HD void vtw4_apply(const PassDesc& d, long long g0, int blk, int logL, CV<V> (&y)[R]) {
  constexpr int LR = ilog2(R), LPU = VT<V>::LPU;
  if constexpr (TW4 == 2) {
    vtw4_table<R, SIGN, B2>(d, g0, blk, logL, y);
    return;
  }
  const Tw4Look look{(const Cx<double>*)d.tw4_lo64, (const Cx<double>*)d.tw4_hi64,
                     (1u << d.tw4_lolog) - 1, d.tw4_lolog};
  const long long i = g0 & ((1LL << d.logS) - 1);
  const uint32_t r0 = ONEBLK ? 0 : drev<B2>((uint32_t)blk, logL - LR);
  CV<double> b[LPU], z4[LPU], z8[LPU];
  CV<V> z[4], f;
  {
    CV<double> z1[LPU], z2[LPU], z3[LPU];
    static_for<LPU>([&](auto ll) {
      constexpr int l = ll.value;
      // E stays below N: iG < N / L, r0 < L / R, t < R
      const uint32_t iG = (uint32_t)(((i + l) >> d.tw4_shift) & d.tw4_mask);
      const uint32_t E = iG << (logL - LR);
      if constexpr (!ONEBLK) b[l] = look(iG * r0);
      z1[l] = look(E);
      if constexpr (R >= 4) {
        z2[l] = look(2 * E);
        z3[l] = vctw<-1>(z2[l], z1[l]);
      }
      if constexpr (R >= 8) z4[l] = look(4 * E);
      if constexpr (R >= 16) z8[l] = look(8 * E);
    });
    vjoin(z1, z[1]);
    if constexpr (R >= 4) {
      vjoin(z2, z[2]);
      vjoin(z3, z[3]);
    }
  }
  static_for<(R + 3) / 4>([&](auto qq) {
    constexpr int q = qq.value;
    constexpr bool one = ONEBLK && q == 0;
    CV<double> c[LPU];
    static_for<LPU>([&](auto ll) {
      constexpr int l = ll.value;
      if constexpr (q == 0) {
        if constexpr (!ONEBLK) c[l] = b[l];
      } else {
        const CV<double> p = q == 1 ? z4[l] : q == 2 ? z8[l] : vctw<-1>(z8[l], z4[l]);
        if constexpr (ONEBLK) c[l] = p;
        else c[l] = vctw<-1>(p, b[l]);
      }
    });
    if constexpr (!one) {
      vjoin(c, f);
      y[4 * q] = vctw<SIGN>(y[4 * q], f);
    }
    static_for<(R < 4 ? R : 4) - 1>([&](auto ss) {
      constexpr int r = ss.value + 1;
      if constexpr (one) y[r] = vctw<SIGN>(y[r], z[r]);
      else y[4 * q + r] = vctw<SIGN>(y[4 * q + r], vctw<-1>(f, z[r]));
    });
  });
}

// offset, in units, of column unit u's first element
template <int LOGL, int LPU, int OFFS>
PAC_HD long long unit_base(const PassDesc& d, long long u) {
  const int su = d.logS - ilog2(LPU);
  long long b = 0;
  if constexpr (OFFS != 0) {
    const int lp = d.logLP - ilog2(LPU);
    b = d.poff[u >> lp] >> ilog2(LPU);
    u &= (1LL << lp) - 1;
  }
  return b + ((u >> su) << (LOGL + su)) + (u & ((1LL << su) - 1));
}

// ---------------------------------------------------------------------------
// The pass
// ---------------------------------------------------------------------------
template <class V, int B2, int MODE, int SIGN, int LOGL, int COLS, int LOGW, int NT, int DIR = 0,
          int OFFS = 0, int PORD = 0>
struct VecPass {
  using Real = typename VT<V>::Real;
  using RS = RadsFor<LOGL, B2>;
  static constexpr int LPU = VT<V>::LPU;
  static constexpr int kThreads = NT;
  static constexpr int L = 1 << LOGL, W = 1 << LOGW;
  static constexpr int NS = RS::n;
  static constexpr int TPT = (W << LOGL) / NT;  // elements of a thread
  static constexpr bool CONV = MODE == MODE_CONV;
  static constexpr int STEPS = CONV ? 2 * NS - 1 : NS;
  static constexpr int VIN = RS::v[NS - 1];  // innermost stage radix (log)
  // The working layout holds complex values of 16 bytes (one access each;
  // eight lanes take 128 bytes).  Rows: one pad value every 8, or every 16
  // where the innermost radix is 16, and a pitch that keeps short lines of
  // eight lanes on different banks: conflict-free in every stage.  Columns:
  // rows of W values; 2^SB rows per 128 bytes, whose low row bits the
  // innermost stage's block index flips.
  static constexpr int PS = VIN == 4 ? 4 : 3;
  static constexpr int PITCH = L + (L >> PS) + (LOGL == 5 ? 4 : 0);
  static constexpr int SB = LOGW >= 3 ? 0 : 3 - LOGW;
  static constexpr int TILE = COLS ? W << LOGL : W * PITCH;  // complex values
  static constexpr size_t TILE_BYTES = (size_t)TILE * 16;
  static constexpr int DIM = W << LOGL;  // the dense tile: W L real, W L imaginary parts
  // the first step reads global memory, not a copy
  static constexpr bool DIRECT = DIR != 0;
  static constexpr int BOXR = L < 256 ? L : 256;  // rows of one tensor-copy box
  // DIT rows would read R consecutive elements a thread from the dense tile:
  // they copy it into the padded layout first.  DIF rows leave through the
  // buffer, so that a warp stores consecutive elements.
  static constexpr bool RELAY_IN = !COLS && MODE == MODE_DIT;
  static constexpr bool RELAY_OUT = !COLS && MODE == MODE_DIF;
  static_assert(TPT * NT == (W << LOGL) && TPT % (1 << RS::v[0]) == 0, "whole butterflies");
  static_assert(NS >= 2, "one-stage passes exchange nothing");
  static_assert(!CONV || !COLS, "the fused pass runs on rows");
  static_assert(!COLS || VIN + SB <= LOGL, "the swizzle bits lie inside a line");
  static_assert(TILE_BYTES >= (size_t)16 * DIM, "the dense tile fits the buffer");

  static PAC_HDC int stage_at(int s) {
    return MODE == MODE_DIF ? s : MODE == MODE_DIT ? NS - 1 - s : s < NS ? s : 2 * NS - 2 - s;
  }
  // DIF (twiddle after the DFT) or DIT (before)
  static PAC_HDC bool dif_step(int s) { return MODE == MODE_DIF || (CONV && s < NS); }
  static PAC_HDC int sign_of(int s) { return CONV ? (s < NS ? -1 : +1) : SIGN; }

  // The stage twiddles in shared memory: a persistent CTA copies the table
  // rows that its butterflies read once, at its start (the loads of a stage
  // would otherwise wait for L1 or L2 in every tile: 3.3 of the 10.5 cycles
  // between two instructions of a warp on fused 4096-point rows).  Stage I
  // with ell > 1 has tw_rows(I) rows of ell entries; row r is the power 2^r
  // (FP64 at radix >= 4) or r + 1.
  static constexpr bool kPow2 = sizeof(Real) == 8;
  static PAC_HDC int tw_ell(int I) { return 1 << (RS::logK(LOGL, I) - RS::v[I]); }
  static PAC_HDC int tw_rows(int I) {
    return kPow2 && RS::v[I] >= 2 ? RS::v[I] : (1 << RS::v[I]) - 1;
  }
  static PAC_HDC int tw_base(int I) {
    int o = 0;
    for (int i = 0; i < I; ++i)
      if (tw_ell(i) > 1) o += tw_rows(i) * tw_ell(i);
    return o;
  }
  static constexpr int TWN = tw_base(NS);  // entries
  static constexpr size_t SMEM = TILE_BYTES + (size_t)TWN * 2 * sizeof(Real);
  static PAC_HD void tw_fill(const PassDesc& d, int t, Cx<Real>* tws) {
    static_for<NS>([&](auto ii) {
      constexpr int I = ii.value, ell = tw_ell(I), n = tw_rows(I) * ell, base = tw_base(I);
      constexpr bool pow2 = kPow2 && RS::v[I] >= 2;
      if constexpr (ell > 1) {
        const Cx<Real>* src = (const Cx<Real>*)d.tw + d.tw_off[I];
        if constexpr (kPow2) {
          for (int q = t; q < n; q += NT) {
            const int r = q / ell, j = q - r * ell;
            tws[base + q] = src[((pow2 ? 1 << r : r + 1) - 1) * ell + j];
          }
        } else {
          // four times the rows: eight loads in flight (one line of 1024
          // points 6.3 -> 5.2 us; FP64 4096 points 7.1 -> 7.6, so not there)
#pragma unroll 8
          for (int q = t; q < n; q += NT) {
            const int r = q / ell, j = q - r * ell;
            tws[base + q] = ld_tw(src + r * ell + j);
          }
        }
      }
    });
  }

  // working layout, and the position of slot SL of a butterfly of stage I
  // whose first element e0 (of unit w) is at p0: rows are p0 plus a constant,
  // as the low bits that e0 adds never carry into the pad count
  template <int I, int SL>
  static PAC_HD int phys_at(int p0, int w, int e0) {
    constexpr int off = SL << (RS::logK(LOGL, I) - RS::v[I]);
    if constexpr (COLS) return phys(w, e0 + off);
    else return p0 + off + (off >> PS);
  }
  static PAC_HD int phys(int w, int e) {
    if constexpr (COLS) {
      return ((e ^ ((e >> VIN) & ((1 << SB) - 1))) << LOGW) + w;
    } else {
      return w * PITCH + e + (e >> PS);
    }
  }
  // element e of unit w of the dense tile that the copies bring in: columns
  // [e][w]; rows line after line (an F2 joins two lines)
  static PAC_HD V dense(const V* B, int w, int e) {
    if constexpr (COLS) {
      return B[(e << LOGW) + w];
    } else if constexpr (LPU == 1) {
      return B[(w << LOGL) + e];
    } else {
      const float* f = reinterpret_cast<const float*>(B) + (w << (LOGL + 1)) + e;
      return f2_make(f[0], f[L]);
    }
  }
  // butterfly k of thread t in stage I: unit w, first element e0, index j
  template <int I>
  static PAC_HD void coords(int t, int k, int& w, int& e0, int& j) {
    constexpr int LR = RS::v[I];
    constexpr int LK = RS::logK(LOGL, I), logell = LK - LR;
    const int u = t + k * NT;
    int v;
    if constexpr (COLS) {
      w = u & (W - 1);
      v = u >> LOGW;
    } else {
      w = u >> (LOGL - LR);
      v = u & ((1 << (LOGL - LR)) - 1);
    }
    j = v & ((1 << logell) - 1);
    e0 = ((v >> logell) << LK) + j;
  }
  // inputs of step S; DENSE reads the copies' layout
  template <int S, bool DENSE>
  static PAC_HD void read(int t, const CV<V>* B, CV<V> (&x)[TPT]) {
    const V* D = reinterpret_cast<const V*>(B);
    constexpr int I = stage_at(S), LR = RS::v[I], R = 1 << LR;
    constexpr int logell = RS::logK(LOGL, I) - LR;
    static_for<TPT / R>([&](auto kk) {
      int w, e0, j;
      coords<I>(t, kk.value, w, e0, j);
      const int p0 = phys(w, e0);
      static_for<R>([&](auto mm) {
        constexpr int m = mm.value;
        constexpr int sl = dif_step(S) ? m : drev_c(m, LR, B2);
        if constexpr (DENSE) {
          const int e = e0 + (sl << logell);
          x[kk.value * R + m] = {dense(D, w, e), dense(D + DIM, w, e)};
        } else {
          x[kk.value * R + m] = vget(B + phys_at<I, sl>(p0, w, e0));
        }
      });
    });
  }
  // the first step's inputs from global memory
  static PAC_HD void read_g(const PassDesc& d, long long tile, int t, CV<V> (&x)[TPT]) {
    constexpr int I = stage_at(0), LR = RS::v[I], R = 1 << LR;
    constexpr int logell = RS::logK(LOGL, I) - LR;
    const int rowsh = d.logS - ilog2(LPU);
    const long long base = tile_base(d, tile);
    const V* ire = (const V*)d.in_re;
    const V* iim = (const V*)d.in_im;
    static_for<TPT / R>([&](auto kk) {
      int w, e0, j;
      coords<I>(t, kk.value, w, e0, j);
      static_for<R>([&](auto mm) {
        constexpr int m = mm.value;
        constexpr int sl = dif_step(0) ? m : drev_c(m, LR, B2);
        const long long gi = base + ((long long)(e0 + (sl << logell)) << rowsh) + w;
        x[kk.value * R + m] = {ld_data(ire + gi), ld_data(iim + gi)};
      });
    });
  }
  // outputs of step S into the working layout: register s of a DIF step is
  // frequency s at slot rev(s), register m of a DIT step (and of the middle
  // one) is element m
  template <int S>
  static PAC_HD void write(int t, CV<V>* B, const CV<V> (&x)[TPT]) {
    constexpr int I = stage_at(S), LR = RS::v[I], R = 1 << LR;
    constexpr bool digit = dif_step(S) && !(CONV && S == NS - 1);
    static_for<TPT / R>([&](auto kk) {
      int w, e0, j;
      coords<I>(t, kk.value, w, e0, j);
      const int p0 = phys(w, e0);
      static_for<R>([&](auto mm) {
        constexpr int m = mm.value;
        vput(B + phys_at<I, digit ? drev_c(m, LR, B2) : m>(p0, w, e0), x[kk.value * R + m]);
      });
    });
  }

  // the arithmetic of step S (not the middle one of a convolution)
  template <int S, int TW4>
  static PAC_HD void compute(const PassDesc& d, long long tile, int t, const Cx<Real>* tws,
                             CV<V> (&x)[TPT]) {
    constexpr int I = stage_at(S), LR = RS::v[I], R = 1 << LR;
    constexpr int logell = RS::logK(LOGL, I) - LR;
    constexpr int SG = sign_of(S);
    constexpr bool DIF = dif_step(S);
    const Cx<Real>* tw = DIRECT ? (const Cx<Real>*)d.tw + d.tw_off[I] : tws + tw_base(I);
    static_for<TPT / R>([&](auto kk) {
      int w, e0, j;
      coords<I>(t, kk.value, w, e0, j);
      CV<V> y[R];
      static_for<R>([&](auto mm) { y[mm.value] = x[kk.value * R + mm.value]; });
      if constexpr (!DIF && TW4 && logell == 0)
        vtw4_apply<TW4, R, SG, B2, NS == 1>(d, ((tile << LOGW) + w) * LPU, e0 >> LR, LOGL, y);
      if constexpr (!DIF && logell > 0) vtwiddle<R, SG, DIRECT>(y, tw + j, 1 << logell);
      vdft<R, SG>(y);
      if constexpr (DIF && logell > 0) vtwiddle<R, SG, DIRECT>(y, tw + j, 1 << logell);
      if constexpr (DIF && TW4 && logell == 0)
        vtw4_apply<TW4, R, SG, B2, NS == 1>(d, ((tile << LOGW) + w) * LPU, e0 >> LR, LOGL, y);
      static_for<R>([&](auto mm) { x[kk.value * R + mm.value] = y[mm.value]; });
    });
  }
  // the middle step of a convolution: last DIF stage, the product with the
  // filter spectrum (plan order: position blk*R + t of a line at t*(L/R) +
  // blk), first DIT stage.  The last line of an odd count stands in for the
  // missing partner of its pair.
  // It runs in groups of four frequencies, which the last radix-4 step of the
  // forward DFT yields together and the first one of the inverse DFT takes
  // together; the spectrum values of a group are loaded one group ahead (of
  // the first group before the barrier that the step waits at: hload).
  static constexpr int RM = 1 << VIN;                        // its radix
  static constexpr int GPB = RM >= 4 ? RM / 4 : 1;           // groups of a butterfly
  static constexpr int GF = RM >= 4 ? 4 : RM;                // frequencies of a group
  static constexpr int GROUPS = CONV ? (TPT / RM) * GPB : 1;
  struct Mid {
    CV<V> h[GF];
  };
  // frequency f of group q of a butterfly
  template <int Q, int F>
  static PAC_HDC int freq() {
    return RM == 16 ? Q + 4 * F : RM == 8 ? 2 * F + Q : F;
  }
  template <int G>
  static PAC_HD void hload(const PassDesc& d, long long tile, int t, Mid& m) {
    constexpr int k = G / GPB, Q = G % GPB;
    const Real* hre = (const Real*)d.h_re;
    const Real* him = (const Real*)d.h_im;
    int w, e0, j;
    coords<NS - 1>(t, k, w, e0, j);
    const int blk = e0 >> VIN;
    const long long l0 = ((tile << LOGW) + w) * LPU;
    const long long last = d.nlines - 1;
    const long long h0 = (line_off(d, l0 < last ? l0 : last) & d.h_mask) + blk;
    const long long h1 =
        LPU == 2 ? (line_off(d, l0 + 1 < last ? l0 + 1 : last) & d.h_mask) + blk : h0;
    static_for<GF>([&](auto ff) {
      constexpr int off = drev_c(freq<Q, ff.value>(), VIN, B2) << (LOGL - VIN);
      if constexpr (LPU == 1) {
        m.h[ff.value] = {ld_now(hre + h0 + off), ld_now(him + h0 + off)};
      } else {
        m.h[ff.value] = {f2_make(ld_now(hre + h0 + off), ld_now(hre + h1 + off)),
                         f2_make(ld_now(him + h0 + off), ld_now(him + h1 + off))};
      }
    });
  }
  static PAC_HD void middle(const PassDesc& d, long long tile, int t, Mid& first,
                            CV<V> (&x)[TPT]) {
    const bool scaled = d.scale != 1.0;
    const V sc = VT<V>::set(d.scale);
    Mid m[2];
    m[0] = first;
    static_for<TPT / RM>([&](auto kk) {
      constexpr int o = kk.value * RM;
      if constexpr (RM == 16) {
        static_for<4>([&](auto jj) {
          constexpr int j = o + jj.value;
          vdft4<-1>(x[j], x[j + 4], x[j + 8], x[j + 12]);
        });
      } else if constexpr (RM == 8) {
        static_for<4>([&](auto jj) {
          constexpr int j = o + jj.value;
          const CV<V> a = vcadd(x[j], x[j + 4]), b = vcsub(x[j], x[j + 4]);
          x[j] = a;
          x[j + 4] = b;
        });
      }
      static_for<GPB>([&](auto qq) {
        constexpr int q = qq.value, G = kk.value * GPB + q;
        if constexpr (G + 1 < GROUPS) hload<G + 1>(d, tile, t, m[(G + 1) & 1]);
        // the last forward step: frequencies freq<q, 0 .. 3> in registers
        // o + 4 q + 0 .. 3
        CV<V>* y = x + o + GF * q;
        if constexpr (RM == 2) {
          const CV<V> a = vcadd(y[0], y[1]), b = vcsub(y[0], y[1]);
          y[0] = a;
          y[1] = b;
        } else if constexpr (q == 0) {
          vdft4<-1>(y[0], y[1], y[2], y[3]);
        } else if constexpr (RM == 8 || q == 2) {
          vdft4_w8<-1>(y[0], y[1], y[2], y[3]);
        } else {
          vdft4_w16<-1, q>(y[0], y[1], y[2], y[3]);
        }
        static_for<GF>([&](auto ff) {
          y[ff.value] = vctw<-1>(y[ff.value], m[G & 1].h[ff.value]);
          if (scaled) y[ff.value] = {vmul(y[ff.value].re, sc), vmul(y[ff.value].im, sc)};
        });
        // the first inverse step over the same four
        if constexpr (RM == 2) {
          const CV<V> a = vcadd(y[0], y[1]), b = vcsub(y[0], y[1]);
          y[0] = a;
          y[1] = b;
        } else if constexpr (RM == 8) {
          // frequencies 2 f + q: pairs (f, f + 2)
          const CV<V> a = vcadd(y[0], y[2]), b = vcadd(y[1], y[3]);
          const CV<V> c = vcsub(y[0], y[2]), e = vcsub(y[1], y[3]);
          y[0] = a;
          y[1] = b;
          y[2] = c;
          y[3] = e;
        } else {
          vdft4<+1>(y[0], y[1], y[2], y[3]);
        }
      });
      if constexpr (RM == 16) {
        // register o + 4 j + q': sub-sequence q' of the inverse at j
        CV<V> z[16];
        static_for<16>([&](auto ii) { z[(ii.value & 3) * 4 + (ii.value >> 2)] = x[o + ii.value]; });
        vdft4<+1>(z[0], z[1], z[2], z[3]);
        vdft4_w16<+1, 1>(z[4], z[5], z[6], z[7]);
        vdft4_w8<+1>(z[8], z[9], z[10], z[11]);
        vdft4_w16<+1, 3>(z[12], z[13], z[14], z[15]);
        static_for<16>([&](auto ii) {
          x[o + (ii.value >> 2) + 4 * (ii.value & 3)] = z[ii.value];
        });
      } else if constexpr (RM == 8) {
        // group q left sums s[q], s[q + 2] in its registers 0, 1 and
        // differences t[q], t[q + 2] in 2, 3
        CV<V> s0 = x[o], s2 = x[o + 1], t0 = x[o + 2], t2 = x[o + 3];
        CV<V> s1 = x[o + 4], s3 = x[o + 5], t1 = x[o + 6], t3 = x[o + 7];
        vdft4<+1>(s0, s1, s2, s3);
        vdft4_w8<+1>(t0, t1, t2, t3);
        x[o] = s0;
        x[o + 2] = s1;
        x[o + 4] = s2;
        x[o + 6] = s3;
        x[o + 1] = t0;
        x[o + 3] = t1;
        x[o + 5] = t2;
        x[o + 7] = t3;
      }
    });
  }

  // element offset of row l (OFFS: of problems that do not lie back to back,
  // PassDesc.poff; a variant of its own, as the look-up cost the others 4%)
  static PAC_HD long long line_off(const PassDesc& d, long long l) {
    if constexpr (!OFFS) return l << LOGL;
    return d.poff[l >> d.logLP] + ((l & ((1LL << d.logLP) - 1)) << LOGL);
  }

  // ---- the dense tile of a pass whose arrays the copies cannot take ------------
  static PAC_HD void copy_in(const PassDesc& d, long long tile, int t, CV<V>* B) {
    if constexpr (COLS) {
      const long long base = tile_base(d, tile);
      const int rowsh = d.logS - ilog2(LPU);
      V* D = reinterpret_cast<V*>(B);
#if defined(__CUDACC__)
#pragma unroll 4
#endif
      for (int q = t; q < DIM; q += NT) {
        const long long gi = base + ((long long)(q >> LOGW) << rowsh) + (q & (W - 1));
        D[q] = ld_data((const V*)d.in_re + gi);
        D[DIM + q] = ld_data((const V*)d.in_im + gi);
      }
    } else {
      constexpr long long WL = W * LPU;
      const long long g0 = tile * WL, left = d.nlines - g0;
      const int n = (int)(left < WL ? left : WL) << LOGL;
      Real* D = reinterpret_cast<Real*>(B);
#if defined(__CUDACC__)
#pragma unroll 4
#endif
      for (int q = t; q < n; q += NT) {
        const long long gi = line_off(d, g0 + (q >> LOGL)) + (q & (L - 1));
        D[q] = ld_data((const Real*)d.in_re + gi);
        D[LPU * DIM + q] = ld_data((const Real*)d.in_im + gi);
      }
    }
  }

  // ---- DIT rows: the dense tile through registers into the padded layout --
  static PAC_HD void relay_read(int t, const CV<V>* B, CV<V> (&x)[TPT]) {
    const V* D = reinterpret_cast<const V*>(B);
    static_for<TPT>([&](auto kk) {
      const int q = t + kk.value * NT;
      x[kk.value] = {dense(D, q >> LOGL, q & (L - 1)), dense(D + DIM, q >> LOGL, q & (L - 1))};
    });
  }
  static PAC_HD void relay_write(int t, CV<V>* B, const CV<V> (&x)[TPT]) {
    static_for<TPT>([&](auto kk) {
      const int q = t + kk.value * NT;
      vput(B + phys(q >> LOGL, q & (L - 1)), x[kk.value]);
    });
  }

  // ---- stores ------------------------------------------------------------
  // rows: the unit's line(s) in the output, and which of them exist
  struct RowOut {
    Real *re, *im;
    long long next;  // from the first line to the second
    bool first, second;
  };
  static PAC_HD RowOut row_out(const PassDesc& d, long long tile, int w, int e0) {
    const long long l0 = ((tile << LOGW) + w) * LPU;
    const bool first = l0 < d.nlines, second = LPU == 2 && l0 + 1 < d.nlines;
    const long long o = !OFFS || first ? line_off(d, l0) + e0 : 0;
    const long long next = OFFS && second ? line_off(d, l0 + 1) + e0 - o : L;
    return {(Real*)d.out_re + o, (Real*)d.out_im + o, next, first, second};
  }
  static PAC_HD void put_row(const RowOut& r, int off, CV<V> v) {
    if constexpr (LPU == 1) {
      if (r.first) {
        r.re[off] = v.re;
        r.im[off] = v.im;
      }
    } else {
      float a, b, c, e;
      f2_split(v.re, a, b);
      f2_split(v.im, c, e);
      if (r.first) {
        r.re[off] = a;
        r.im[off] = c;
      }
      if (r.second) {
        r.re[r.next + off] = b;
        r.im[r.next + off] = e;
      }
    }
  }
  // tile -> first column unit i0 and outer index o of a column tile
  static PAC_HD void tile_coords(const PassDesc& d, long long tile, int& i0, int& o) {
    const long long g0 = tile << LOGW;  // in units; the stride is S / LPU units
    const int logSU = d.logS - ilog2(LPU);
    i0 = (int)(g0 & ((1LL << logSU) - 1));
    o = (int)(g0 >> logSU);
  }
  // unit offset of a column tile's first row
  static PAC_HD long long tile_base(const PassDesc& d, long long tile) {
    return unit_base<LOGL, LPU, OFFS>(d, tile << LOGW);
  }
  // the last step's outputs from the registers to global memory: whole rows
  // of W elements (columns; at their natural index when the pass ends a
  // natural-order transform), consecutive elements of a line (rows)
  static PAC_HD void store(const PassDesc& d, long long tile, int t, const CV<V> (&x)[TPT]) {
    constexpr int S = STEPS - 1;
    constexpr int I = stage_at(S), LR = RS::v[I], R = 1 << LR;
    constexpr int logell = RS::logK(LOGL, I) - LR;
    constexpr bool digit = dif_step(S);
    const bool scaled = d.use_scale && !CONV;
    const V sc = VT<V>::set(d.scale);
    V* cre = (V*)d.out_re;
    V* cim = (V*)d.out_im;
    long long base = 0;
    int rowsh = d.logS - ilog2(LPU);
    if constexpr (COLS) {
      if (d.nat) {
        long long in_base, out_base;
        nat_line<B2>(d, (tile << LOGW) * LPU, &in_base, &out_base);
        base = out_base >> ilog2(LPU);
        rowsh += d.nat_Mlog;
      } else {
        base = tile_base(d, tile);
      }
    }
    static_for<TPT / R>([&](auto kk) {
      int w, e0, j;
      coords<I>(t, kk.value, w, e0, j);
      RowOut r;
      if constexpr (!COLS) r = row_out(d, tile, w, e0);
      static_for<R>([&](auto mm) {
        constexpr int m = mm.value;
        constexpr int off = (digit ? drev_c(m, LR, B2) : m) << logell;
        CV<V> v = x[kk.value * R + m];
        if (scaled) v = {vmul(v.re, sc), vmul(v.im, sc)};
        if constexpr (COLS) {
          const int row = MODE == MODE_DIF && d.nat ? (int)drev<B2>((uint32_t)(e0 + off), LOGL)
                                                    : e0 + off;
          const long long gi = base + ((long long)row << rowsh) + w;
          cre[gi] = v.re;
          cim[gi] = v.im;
        } else {
          put_row(r, off, v);
        }
      });
    });
  }
  // DIF rows: out of the buffer, consecutive elements of a line by
  // consecutive threads, in digit-reversed (the slots), natural or plan order
  // (a filter spectrum: the pass after the transform that reordered and
  // rounded it is gone)
  static PAC_HD void relay_store(const PassDesc& d, long long tile, int t, const CV<V>* B) {
    const V sc = VT<V>::set(d.scale);
    static_for<TPT>([&](auto kk) {
      const int q = t + kk.value * NT;
      const int w = q >> LOGL, e = q & (L - 1);
      int slot = e;
      if constexpr (PORD != 0) {
        const int lq = LOGL - d.porder_logR;
        slot = ((e & ((1 << lq) - 1)) << d.porder_logR) + (e >> lq);
      } else if (d.nat) {
        slot = (int)drev<B2>((uint32_t)e, LOGL);
      }
      CV<V> v = vget(B + phys(w, slot));
      if (d.use_scale) v = {vmul(v.re, sc), vmul(v.im, sc)};
      if constexpr (PORD == 4) {  // FP64 lines, rounded once
        const long long l = (tile << LOGW) + w;
        if (l < d.nlines) {
          ((float*)d.out_re)[(l << LOGL) + e] = (float)v.re;
          ((float*)d.out_im)[(l << LOGL) + e] = (float)v.im;
        }
        return;
      }
      put_row(row_out(d, tile, w, e), 0, v);
    });
  }

  // the order of the steps, over an executor: X.each(f) runs f(t, x) for
  // every thread and X.sync() is the CTA barrier after it; X.freed() is a
  // barrier too, after which nothing reads the buffer any more
  template <int TW4, class X>
  static PAC_HD void body(const PassDesc& d, long long tile, CV<V>* B, const Cx<Real>* tws, X& ex) {
    if constexpr (RELAY_IN) {
      ex.each([&](int t, CV<V>(&x)[TPT]) { relay_read(t, B, x); });
      ex.sync();
      ex.each([&](int t, CV<V>(&x)[TPT]) { relay_write(t, B, x); });
      ex.sync();
    }
    static_for<STEPS>([&](auto ss) {
      constexpr int S = ss.value;
      ex.each([&](int t, CV<V>(&x)[TPT]) {
        if constexpr (S == 0 && DIRECT) read_g(d, tile, t, x);
        else read<S, S == 0 && !RELAY_IN>(t, B, x);
      });
      if constexpr (S == STEPS - 1 && !RELAY_OUT) ex.freed();
      if constexpr (CONV && S == NS - 1) {
        ex.each_mid([&](int t, CV<V>(&x)[TPT], auto& m) { middle(d, tile, t, m, x); });
      } else {
        ex.each([&](int t, CV<V>(&x)[TPT]) { compute<S, TW4>(d, tile, t, tws, x); });
      }
      if constexpr (S < STEPS - 1 || RELAY_OUT) {
        // the dense tile and the working layout differ: everything is read
        // before anything is written; later steps write the slots they read
        if constexpr (S == 0 && !RELAY_IN && !DIRECT) ex.sync();
        ex.each([&](int t, CV<V>(&x)[TPT]) { write<S>(t, B, x); });
        if constexpr (CONV && S == NS - 2)
          ex.each_mid([&](int t, CV<V>(&)[TPT], auto& m) { hload<0>(d, tile, t, m); });
        ex.sync();
      }
    });
    if constexpr (RELAY_OUT) {
      ex.each([&](int t, CV<V>(&)[TPT]) { relay_store(d, tile, t, B); });
      ex.freed();
    } else {
      ex.each([&](int t, CV<V>(&x)[TPT]) { store(d, tile, t, x); });
    }
  }
};

// Columns of 2 to 16 elements: one unit a thread, registers only.
template <class V, int B2, int MODE, int SIGN, int LOGL, int OFFS = 0>
struct VecSmall {
  static constexpr int L = 1 << LOGL, LPU = VT<V>::LPU;
  static_assert(LOGL >= 1 && LOGL <= 4 && LOGL % B2 == 0 && (B2 != 3 || LOGL == 3), "one stage");
  // unit u of nlines / LPU
  // loaded() runs once the unit is in registers
  template <int TW4, class F>
  static PAC_HD void run(const PassDesc& d, long long u, F&& loaded) {
    const int su = d.logS - ilog2(LPU);
    const V* ire = (const V*)d.in_re;
    const V* iim = (const V*)d.in_im;
    V* ore = (V*)d.out_re;
    V* oim = (V*)d.out_im;
    const long long in0 = unit_base<LOGL, LPU, OFFS>(d, u);
    long long out0 = in0;
    int osh = su;
    if (MODE == MODE_DIF && d.nat) {
      long long ib, ob;
      nat_line<B2>(d, u * LPU, &ib, &ob);
      out0 = ob >> ilog2(LPU);
      osh += d.nat_Mlog;
    }
    CV<V> x[L];
    static_for<L>([&](auto mm) {
      constexpr int m = mm.value;
      const long long gi = in0 + ((long long)(MODE == MODE_DIF ? m : drev_c(m, LOGL, B2)) << su);
      x[m] = {ld_data(ire + gi), ld_data(iim + gi)};
    });
    loaded();
    if constexpr (TW4 && MODE == MODE_DIT) vtw4_apply<TW4, L, SIGN, B2, true>(d, u * LPU, 0, LOGL, x);
    vdft<L, SIGN>(x);
    if constexpr (TW4 && MODE == MODE_DIF) vtw4_apply<TW4, L, SIGN, B2, true>(d, u * LPU, 0, LOGL, x);
    const V sc = VT<V>::set(d.scale);
    const bool nat = MODE == MODE_DIF && d.nat;
    static_for<L>([&](auto mm) {
      constexpr int m = mm.value;
      constexpr int rev = drev_c(m, LOGL, B2);
      CV<V> v = x[m];
      if (d.use_scale) v = {vmul(v.re, sc), vmul(v.im, sc)};
      const long long gi = out0 + ((long long)(MODE == MODE_DIF && !nat ? rev : m) << osh);
      ore[gi] = v.re;
      oim[gi] = v.im;
    });
  }
};

}  // namespace pac

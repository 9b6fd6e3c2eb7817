// sipg_fx.cuh -- the FP64 operator's sums on the integer pipe.
//
// GB300 issues 2 FP64 operations per SM per cycle but 64 32 x 32-bit products
// added to a 64-bit sum (IMAD.WIDE; both rates measured with independent
// chains).  The operator's contractions -- the stiffness sums, the lifted
// jumps, the face derivatives, ~18 of its ~21 FP64 operations per DoF at p = 4
// -- have constant coefficients, so they are taken in fixed point: an
// element's values share one power-of-two scale, and each value and each
// coefficient is an integer held as two limbs,
//     F = h 2^29 + l.
// A product adds h h' to one 64-bit sum and h l' + l h' to another (three
// IMAD.WIDE; l l' is left out, up to half a unit of the total).  The kept products
// are summed without rounding, so their order is free, and a result is rounded
// once more on its way back to a double.
//
// The LGL nodes are symmetric, so every 1-D matrix here maps even functions
// of the node index to even ones and odd to odd: values are kept as sums and
// differences of mirrored nodes in both directions ("parity form"), which
// halves the products (n^3 instead of 2 n^3 an element for the stiffness) and
// costs integer additions only.
//
// Face terms.  In parity form along a face the trace of an element is the sum
// (0 side) or difference (N side) of its even and odd values of index 0 along
// the normal, and w times the normal derivative is a contraction with the face
// rows; the LGL weights are symmetric, so jump, derivative sum and penalty
// combine component by component and enter the output's parity components of
// index 0.  Face values stay integers all the way.
//
// Large penalties (fx_large_nu).  A jump's integer is rounded at the quantum of
// the face's larger element, and nu multiplies that; so beyond some tens of
// units the integer sums leave the penalty out, and it joins the outputs of the
// face nodes as nu w (u - u_across) in FP64 (fx_penalty).  Relative 2-norm
// error on sin(2 pi x) sin(3 pi y), 12^2 elements, p = 4, penalty 100 p^2: 9.0e-14
// with integer jumps, 1.4e-14 with FP64 ones, 1.8e-14 with FP64 chains.
//
// Accuracy.  A value's quantum is 2^-55 of its element's scale (a value within 1/4
// of the largest one is exact), a coefficient's 2^-58 of the largest (the tables
// are built in extended precision), and a total's unit is 2^(3 - sk) of the scale
// (sk: fx_scale; 2^-56, 2^-54, 2^-53, 2^-52, 2^-53, 2^-52, 2^-53, 2^-52 for p = 1..8), to which each
// parity component is rounded and of which each dropped l l' is up to a half.  A
// plain FP64 chain rounds each of its 2n + 4 steps at 2^-53 of the partial sum.  The
// integer coefficients of a zero-sum row (stiffness, derivative) sum to zero; the
// dropped products leave a constant's result within some units of zero.  An element
// whose neighbour is more than 2^kFxRoom times larger takes a coarser scale.
// That is accuracy relative to the element's (and its neighbours') largest
// values.  An output sums its own row and column of the element, its face terms
// and the traces across, and where those are all small, chains keep it accurate
// relative to them and one scale for the element does not.  So the elements
// that one scale does not fit take FP64 chains instead (chain_node), each by
// itself: those where some node's row and column both stay below 2^-kFxSpread of
// the scale, which an element far smaller than a neighbour is too, and zeros
// beside non-zeros.  The others' entry-wise error is bounded by the scale;
// against the sum of the entry's terms it reaches 900 2^-53 (a load vector,
// whose corner nodes carry small weights, p = 8; chains: 4 2^-53), 15 2^-53 on
// uniform values (chains 13).  Of the elements of CG directions (means over a solve,
// p = 2..8) 0.1 to 1.2 in 1000 lie beyond 2^-4, 9 to 29 beyond 2^-2.
//
// Range.  The scale is the element's own, so vectors of any magnitude keep
// this accuracy.  An element with an infinity, a NaN, or a magnitude near the
// ends of the exponent range (kFxMinExp, kFxMaxExp) has no scale: it and its
// neighbours take the chains.  Which elements do depends on the element and its
// four neighbours alone.
#pragma once

#include <cmath>
#include <cstring>

#include "sipg_internal.cuh"

namespace sipg {

constexpr int kFxLimb = 29;                       // bits of a low limb
constexpr int kFxBits = 55;                       // a value's integer is below 2^kFxBits
constexpr int kFxRoom = 2;                        // bits a neighbour's scale may exceed the element's
constexpr int kFxSpread = 4;                      // bits a node's row and column may both stay below the scale
constexpr int kFxMinExp = 200, kFxMaxExp = 1983;  // an element's largest value's biased exponent lies between
constexpr int kFxNoScale = 2047;                  // the scale of an element where it does not

// Fixed-point tables of degree P in parity form (limb pairs, .x = h, .y = l).
// Mirrored nodes i and N - i have the even index i and the odd index i (< NO);
// the middle node of an odd n has the even index NE - 1 alone.  HB(b) is 1/2
// for a mirrored pair and 1 for the middle node: the inverse of the sum and
// difference along the other direction.
template <int P>
struct FxTab {
  static constexpr int N1 = P + 1, NE = (N1 + 1) / 2, NO = N1 / 2;
  int2 ke[NE * NE * NE];  // [(i * NE + k) * NE + b]: HB(b) w_b (K[i][k] + K[i][N-k]) / 2 (K[i][k] for the middle k)
  int2 ko[NO * NO * NE];  // [(i * NO + k) * NE + b]: HB(b) w_b (K[i][k] - K[i][N-k]) / 2
  // the face rows [i * NE + b]: HB(b) w_b (D[i][0] +- D[N-i][0]) / 4.  As a
  // lift: times J_0side -+ J_Nside.  As a derivative: HB w_b times the 0 side's
  // is twice (even + odd), HB w_b times the N side's twice (odd - even).
  int2 le[NE * NE], lo[NO * NE];
  double wl[N1];  // the weights beyond Tab::w
  double w[NE];   // HB(b) w_b, and the largest
  double wmax;
  int sk;  // coefficient = F 2^-sk
};

inline int2 fx_limbs(long long f) {
  const long long h = (f + (1ll << (kFxLimb - 1))) >> kFxLimb;
  return make_int2((int)h, (int)(f - h * (1ll << kFxLimb)));
}

// The scale exponent for coefficients up to cmax in magnitude whose rows (in
// parity form, for values of up to four nodes each) sum to at most l1: F <
// 2^58 and row sums below 2^59, so that no 64-bit sum passes 2^62.  A total's
// unit is 2^(3 - scale) of the element's largest value.  From degree 3 on that
// is a fraction of the rounding of FP64 chains, whose length grows with the
// degree; the short chains of degrees 1 and 2 round less, so there F < 2^58 and
// 2^59 and rows up to 2^61 (a middle value's coefficient at degree 2 is 32
// times a corner's).  Their components then stay below 2^61 and limbs below
// 2^30, and a node's output below 2^62.  Error against extended precision,
// relative 2-norm over smooth, uniform and normal values at degree 2: 2.2e-16,
// 8.0e-17, 9.6e-17; with the bounds of degree 3: 1.6e-15, 2.7e-16, 4.3e-16; FP64
// chains: 2.2e-16, 1.7e-16, 1.5e-16.  The time is the same.
template <int P>
inline int fx_scale(double cmax, double l1) {
  int ec = 0, el = 0;
  std::frexp(cmax, &ec);  // cmax < 2^ec
  std::frexp(P <= 2 ? l1 * (1 - 1e-12) : l1, &el);  // (their l1 are powers of two: l1 <= 2^el)
  const int a = (P == 2 ? 59 : 58) - ec, b = (P <= 2 ? 61 : 59) - el;
  return a < b ? a : b;
}

// LGL weights w, the derivative column d0[i] = D[i][0] and the stiffness K in
// extended precision (the double nodes polished by Newton steps on
// (1 - x^2) P_N').
template <int P>
inline void fx_reference(const HostTables& h, long double* w, long double* d0, long double* K) {
  constexpr int n = P + 1, N = P;
  long double x[n], pn[n];
  auto legendre = [](long double xx, long double* p1) {  // P_N; *p1 = P_(N-1)
    long double a = 1, b = xx;
    for (int k = 2; k <= N; ++k) {
      const long double c = ((2 * k - 1) * xx * b - (k - 1) * a) / k;
      a = b;
      b = c;
    }
    *p1 = a;
    return b;
  };
  for (int i = 0; i < n; ++i) {
    x[i] = h.nodes[i];
    long double p1 = 0;
    if (i > 0 && i < N)
      for (int it = 0; it < 3; ++it) {  // (1 - x^2) P_N' = N (P_(N-1) - x P_N), its derivative -N (N + 1) P_N
        const long double p = legendre(x[i], &p1);
        x[i] += (p1 - x[i] * p) / ((N + 1) * p);
      }
  }
  for (int i = 0; i < n; ++i) {
    long double p1 = 0;
    pn[i] = legendre(x[i], &p1);
    w[i] = 2 / (N * (N + 1) * pn[i] * pn[i]);
  }
  auto D = [&](int i, int k) -> long double {
    if (i == k) return k == 0 ? -0.25L * N * (N + 1) : (k == N ? 0.25L * N * (N + 1) : 0.0L);
    return pn[k] / (pn[i] * (x[k] - x[i]));
  };
  for (int a = 0; a < n; ++a) {
    d0[a] = D(a, 0);
    for (int b = 0; b < n; ++b) {
      long double s = 0;
      for (int k = 0; k < n; ++k) s += w[k] * D(a, k) * D(b, k);
      K[a * n + b] = s;
    }
  }
}

template <int P>
inline FxTab<P> make_fxtab(const HostTables& h) {
  using Tb = FxTab<P>;
  constexpr int n = P + 1, N = P, NE = Tb::NE, NO = Tb::NO;
  long double w[n], d0[n], K[n * n];
  fx_reference<P>(h, w, d0, K);
  Tb t;
  std::memset(&t, 0, sizeof(t));
  auto hw = [&](int b) { return (2 * b == N ? 1.0L : 0.5L) * w[b]; };
  auto ke = [&](int i, int k) { return 2 * k == N ? K[i * n + k] : 0.5L * (K[i * n + k] + K[i * n + N - k]); };
  auto ko = [&](int i, int k) { return 0.5L * (K[i * n + k] - K[i * n + N - k]); };
  double cmax = 0, l1 = 0;
  for (int i = 0; i < NE; ++i)
    for (int b = 0; b < NE; ++b) {
      auto big = [&](int r, int k) {
        return std::fmax(std::fabs((double)ke(r, k)), k < NO && r < NO ? std::fabs((double)ko(r, k)) : 0.0);
      };
      double row = 0;
      for (int k = 0; k < NE; ++k) {
        cmax = std::fmax(cmax, (double)hw(b) * big(i, k));
        row += (double)hw(b) * big(i, k) + (double)hw(i) * big(b, k);
      }
      auto lift = [&](int r) { return 0.25 * (std::fabs((double)d0[r]) + std::fabs((double)d0[N - r])); };
      cmax = std::fmax(cmax, (double)hw(b) * lift(i));
      // a jump's integer may be twice a value's
      l1 = std::fmax(l1, row + 2 * ((double)hw(b) * lift(i) + (double)hw(i) * lift(b)));
    }
  t.sk = fx_scale<P>(cmax, l1);
  auto fix = [&](long double c) { return (long long)std::llrintl(std::ldexp(c, t.sk)); };
  // a zero-sum row f(k) of even indices: the middle entry (even n: entry z)
  // takes what the others leave, times the sum of two mirrored values
  auto zero_sum = [&](auto f, auto out, int z) {
    if (NE > NO) z = NE - 1;
    long long sum = 0;
    for (int k = 0; k < NE; ++k) {
      if (k == z) continue;
      *out(k) = fx_limbs(fix(f(k)));
      sum += fix(f(k));
    }
    *out(z) = fx_limbs(NE > NO ? -2 * sum : -sum);
  };
  for (int b = 0; b < NE; ++b) {
    for (int i = 0; i < NE; ++i)
      zero_sum([&](int k) { return hw(b) * ke(i, k); }, [&](int k) { return &t.ke[(i * NE + k) * NE + b]; }, i);
    zero_sum([&](int k) { return 0.25L * hw(b) * (d0[k] + d0[N - k]); }, [&](int k) { return &t.le[k * NE + b]; }, 0);
    for (int i = 0; i < NO; ++i) {
      for (int k = 0; k < NO; ++k) t.ko[(i * NO + k) * NE + b] = fx_limbs(fix(hw(b) * ko(i, k)));
      t.lo[i * NE + b] = fx_limbs(fix(0.25L * hw(b) * (d0[i] - d0[N - i])));
    }
  }
  for (int i = 0; i < NE; ++i) {
    t.w[i] = (double)hw(i);
    t.wmax = std::fmax(t.wmax, t.w[i]);
  }
  for (int i = 0; i < n; ++i) t.wl[i] = (double)(w[i] - (long double)h.w[i]);
  return t;
}

__device__ __forceinline__ int fx_biased(double v) { return (int)(((unsigned)__double2hiint(v) << 1) >> 21); }

// v 2^kFxBits / 2^(be - 1022) towards zero (be: the scale's biased exponent,
// at least v's; a zero's or denormal's hidden bit is shifted out, as
// be >= kFxMinExp).
__device__ __forceinline__ long long fx_fix(double v, int be) {
  constexpr int kUp = kFxBits - 53;
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = (__funnelshift_l(lo, hi, kUp) & ((1u << (20 + kUp)) - 1u)) | (1u << (20 + kUp));
  const int s = min(be - fx_biased(v), 63);
  long long m = (long long)((((unsigned long long)mh << 32) | (lo << kUp)) >> s);
  // (predicated: the compiler's select takes two instructions more)
  asm("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %1, 0;\n\t@p neg.s64 %0, %0;\n\t}" : "+l"(m) : "r"((int)hi));
  return m;
}
__device__ __forceinline__ int2 fx_limbs_of(long long f) {
  return make_int2((int)(f >> kFxLimb), (int)((unsigned)f & ((1u << kFxLimb) - 1u)));
}
// The same value at a scale 2^sh larger.
__device__ __forceinline__ int2 fx_shift(int2 f, int sh) {
  return fx_limbs_of((((long long)f.x << kFxLimb) + f.y) >> sh);
}

// The two sums of a fixed-point contraction; the total rounds to nearest.
struct FxAcc {
  long long hh, mid;
};
__device__ __forceinline__ FxAcc fx_zero() { return FxAcc{0, 1ll << (kFxLimb - 1)}; }
// (the empty asm statements keep the compiler from splitting the chains of
// sums, which costs an addition per product)
__device__ __forceinline__ void fx_mac(FxAcc& s, int2 c, int2 u) {
  s.hh += (long long)c.x * u.x;
  s.mid += (long long)c.y * u.x;
  asm("" : "+l"(s.hh), "+l"(s.mid));
  s.mid += (long long)c.x * u.y;
  asm("" : "+l"(s.mid));
}
__device__ __forceinline__ long long fx_total(const FxAcc& s) { return s.hh + (s.mid >> kFxLimb); }

// The exponent of a total whose values had scale be: it counts 2^(2 kFxLimb)
// units of a value times a coefficient.
__device__ __forceinline__ int fx_exp(int be, int sk) { return be - 1022 - kFxBits - sk + 2 * kFxLimb; }

// r 2^ex as a double, rounded to nearest (kFxMinExp and kFxMaxExp keep the
// exponent in range).  The conversion instruction runs on the FP64 pipe,
// which has room for the one per output it takes here; converting with
// integer instructions instead (17 of them) measured no faster.
__device__ __forceinline__ double fx_double(long long r, int ex) {
  const double d = (double)r;
  const int hi = __double2hiint(d);
  return __hiloint2double(hi != 0 ? hi + (ex << 20) : 0, __double2loint(d));  // r != 0: hi != 0
}

// For the running maximum of magnitudes: the high word less its sign.
__device__ __forceinline__ unsigned fx_mag(double v) { return (unsigned)__double2hiint(v) << 1; }
// The scale of an element whose largest fx_mag is m: kFxMinExp for zeros only.
__device__ __forceinline__ int fx_be(unsigned m, bool nonzero) {
  const int e = (int)(m >> 21);
  if (e >= kFxMaxExp || (e <= kFxMinExp && nonzero)) return kFxNoScale;
  return max(e, kFxMinExp);
}
// Whether an element takes the chains: its outputs' scale be, the largest of its
// and its faces' scales (faces), and the exponent low that every node's row or
// column reaches.
__device__ __forceinline__ bool fx_chains(int be, int faces, int low) {
  return be >= kFxMaxExp || (low < be - kFxSpread && faces > kFxMinExp);
}
// The high word of a double as an integer of the same order, and back.
__device__ __forceinline__ int fx_ordered(int hi) { return hi ^ ((hi >> 31) & 0x7fffffff); }
// How far apart two values are whose ordered high words are lo <= hi, as fx_mag.
__device__ __forceinline__ unsigned fx_apart(int lo, int hi) {
  return fx_mag(__dadd_rn(__hiloint2double(fx_ordered(hi), 0), -__hiloint2double(fx_ordered(lo), 0)));
}
// Twice the trace of an element: its even value of index 0 along the normal plus
// (0 side) or less (N side) the odd one.
__device__ __forceinline__ long long fx_trace0(int2 e, int2 o) {
  return (long long)(e.x + o.x) * (1 << kFxLimb) + ((long long)e.y + o.y);
}
__device__ __forceinline__ long long fx_traceN(int2 e, int2 o) {
  return (long long)(e.x - o.x) * (1 << kFxLimb) + (e.y - o.y);
}
// v, at a scale 2^sh smaller, at this one (sh >= -kFxRoom).
__device__ __forceinline__ long long fx_scaled(long long v, int sh) {
  if (sh != 0) v = (v * (1 << kFxRoom)) >> min(sh + kFxRoom, 63);
  return v;
}

// The parity form of the four values at mirrored nodes: v[0] = (i, j), v[1] =
// (N - i, j), v[2] = (i, N - j), v[3] = (N - i, N - j) become even-even,
// odd-even, even-odd, odd-odd (first word: the i direction).
__device__ __forceinline__ void fx_quad(long long (&v)[4]) {
  const long long a = v[0] + v[1], b = v[0] - v[1], c = v[2] + v[3], d = v[2] - v[3];
  v[0] = a + c;
  v[1] = b + d;
  v[2] = a - c;
  v[3] = b - d;
}

// HB w times the normal derivatives on a pair of opposite faces, at component b
// (weight index wb) along them, from the element's values get(k, odd) of index
// k and parity odd along the normal: r0 half the 0 side's, rN minus half the N
// side's, in units of 2^fx_exp(be, sk).
template <int P, typename Get>
__device__ __forceinline__ void fx_derivatives(const FxTab<P>& fx, int wb, Get get, long long& r0, long long& rN) {
  using Tb = FxTab<P>;
  FxAcc ev = fx_zero(), od = fx_zero();
#pragma unroll
  for (int k = 0; k < Tb::NE; ++k) fx_mac(ev, fx.le[k * Tb::NE + wb], get(k, false));
#pragma unroll
  for (int k = 0; k < Tb::NO; ++k) fx_mac(od, fx.lo[k * Tb::NE + wb], get(k, true));
  const long long e = fx_total(ev), o = fx_total(od);
  r0 = e + o;
  rN = e - o;
}

// Whether the penalty's coefficients nu HB(b) w_b, scaled as the tables, pass
// 2^60: the integer terms of the largest jumps (components below 2^(kFxBits + 2),
// times 2^kFxRoom from a larger neighbour, from two faces at a corner node) could
// then pass 2^63 units: from penalties of 4.0, 1.5, 4.3, 2.8, 2.3, 1.8, 1.6 and 1.4
// p^2 on for p = 1..8.
__device__ __forceinline__ bool fx_large_nu(double nu_wmax, int sk) { return fx_biased(nu_wmax) - 1022 + sk > 60; }
__device__ __forceinline__ int2 fx_nu(double wnu, int sk) {
  return fx_limbs_of(__double2ll_rn(wnu * __hiloint2double((1023 + sk) << 20, 0)));
}

// One face component: the jump J (0 side less N side, in units of a value at
// the face's scale max(b0, bN)) and half of HB Q, Q = w (kappa (d0 + dN) + nu
// J), in units of a total at that scale.  nu: nu HB w as limbs (zero if
// fx_large_nu); t0, tN: twice the traces, r0, rN as fx_derivatives; a boundary
// face has only one side (in0 or inN), kappa = 1, and a doubled J (the lift's
// table has kappa = 1/2 folded in).  kPivot: delta the difference of the sides'
// pivots, which the component takes mult times (its scale joins the face's).
template <bool kPivot>
__device__ __forceinline__ void fx_face(int2 nu, bool in0, bool inN, long long t0, long long r0, int b0, long long tN,
                                        long long rN, int bN, double delta, int mult, long long& J, long long& Q) {
  if (!in0) t0 = 0, r0 = 0, b0 = bN;
  if (!inN) tN = 0, rN = 0, bN = b0;
  int b = max(b0, bN);
  if (kPivot) b = max(b, fx_biased(delta));
  if (b != b0 || b != bN) {
    const int s0 = min(b - b0, 62), sN = min(b - bN, 62);
    t0 = (t0 >> s0) & ~1ll;
    r0 >>= s0;
    tN = (tN >> sN) & ~1ll;
    rN >>= sN;
  }
  J = (t0 - tN) >> 1;  // (both are even)
  long long r = r0 - rN;
  if (!(in0 && inN)) r *= 2;
  if (kPivot) J += mult * fx_fix(delta, b);
  FxAcc s = fx_zero();
  s.hh = 1;  // the half rounds to nearest (rounded down: 3.3e-16 for smooth values at degree 2, now 2.2e-16)
  fx_mac(s, nu, fx_limbs_of(J));
  Q = (r + fx_total(s)) >> 1;
  if (!(in0 && inN)) J *= 2;
}

// A large penalty's coefficient nu w, w = wh + wl, in two doubles: rounded to
// one, its error is the same at every node of a line and does not average out
// (uniform values, p = 6, 100 p^2: 2-norm error 1.08 2^-52 of the terms, here
// 0.21; FP64 chains 1.43).  And its FP64 term added to an output v on a face, whose value exceeds the
// one across by jump.  (Explicitly rounded: the same bits wherever they are
// inlined.)
__device__ __forceinline__ double2 fx_penalty(double wh, double wl, double nu) {
  const double c = __dmul_rn(wh, nu);
  return make_double2(c, __fma_rn(wl, nu, __fma_rn(wh, nu, -c)));
}
__device__ __forceinline__ double fx_add_penalty(double v, double2 c, double jump) {
  return __fma_rn(c.x, jump, __fma_rn(c.y, jump, v));
}

}  // namespace sipg

// sipg_apply_fx.cuh -- the FP64 element-per-thread apply with its sums in
// fixed point (sipg_fx.cuh), on the tiles of sipg_apply.cuh.  Phases of a CTA:
//   0  each thread loads its element's n^2 values and finds their scale; the
//      scales of the elements around the tile, dealt out over the warps;
//   1  the values' parity form into the thread's column of shared memory, and w
//      times the normal derivative on each face; the same for the one face of
//      each element around the tile, a pair of face components per thread;
//   1b the N side of each face (for the faces below and left of the tile the 0
//      side) combines both sides into the jump J and Q;
//   2  per pair of mirrored output columns: the lifted jumps and both
//      stiffness sums as one fixed-point sum per parity component, the face
//      terms of index 0 added, back to the nodes, and rounded to a double; then
//      the epilogue (store; in the CG modes a deterministic grid reduction).
// Every output depends on the element and its four neighbours alone, through
// integers, so every tile shape gives the same bits.
//
// Bound by integer issue and its latency: 183 instructions per DoF at p = 4 (29
// of them the products; the rest conversions, parity form, limbs, 64-bit
// additions and shared memory); ncu: multiply-add pipe 54 %, 46 % of the issue
// slots with the 16 warps per SM that registers and shared memory allow, where FP64 chains are bound by an FP64
// pipe of 2 operations per SM and cycle (21 per DoF).  Measured, FP64 chains
// against this: 1024^2, p = 4 1080 -> 266 us (388 -> 1577 GB/s of the 16 bytes
// per DoF); 443^2, p = 8 977 -> 288 us; ~16 M DoF, p = 1..8: 25, 26, 25, 24, 22,
// 20, 18, 16 -> 81, 97, 94, 98, 79, 70, 67, 55 GDoF/s.  The error
// against extended precision fell with it (p = 4, uniform values, relative
// 2-norm: 2.8e-16 -> 1.1e-16).
#pragma once

#include <type_traits>

#include "sipg_apply.cuh"
#include "sipg_fx.cuh"

namespace sipg {

template <int P>
struct FxForm {
  static constexpr bool regs = P <= 4;  // raw values in registers between load and conversion
  static constexpr int load_unroll = (P >= 5) ? 2 * (P + 1) : (P + 1) * (P + 1);
  static constexpr int col_unroll = (P >= 5) ? 1 : (P + 1);
  static constexpr int face_unroll = (P >= 5) ? 1 : (P + 1);
};

// Address of value k of the element whose value 0 is at p: one wide product.
__device__ __forceinline__ const double* fx_addr(const double* p, unsigned noe, int k) {
  return reinterpret_cast<const double*>(reinterpret_cast<const char*>(p) + (unsigned long long)noe * (8u * (unsigned)k));
}

// Value k of element e as the operator sees it (CG: p = r + beta p_old).
// (Passed by value: a closure over the tile's variables, handed to a function
// that is not inlined, puts them in memory: 443^2, p = 8: 377 us, here 270.)
template <bool CG>
struct FxLoad {
  const double *in, *pold;
  unsigned noe;
  double beta;
  bool first;
  __device__ __forceinline__ double operator()(int k, size_t e) const {
    const double r = __ldg(fx_addr(in + e, noe, k));
    if (CG) return first ? r : fma(beta, __ldg(fx_addr(pold + e, noe, k)), r);
    return r;
  }
};

// The plain FP64 code, for tiles whose values are out of the fixed-point range
// (sipg_fx.cuh): one thread computes all outputs of element (gx, gy) with FP64
// sums, reading it and its neighbours through ld(k, element).  Rolled and
// unshared: it is as slow as it is rare.  Returns the thread's share of the
// reduction.
template <int P, int MODE, typename Ld>
__device__ __noinline__ double plain_element(const ApplyArgs<double>& a, const Tab<double, P>& tb, int gx, int gy,
                                             Ld ld, double* pnew) {
  constexpr int N = P, N1 = P + 1, BASE = apply_base_mode(MODE);
  constexpr bool kDot = (BASE == APPLY_CG || BASE == APPLY_DOT);
  const int dim = a.dim;
  const size_t noe = (size_t)dim * dim, e = (size_t)gy * dim + gx;
  // J and Q of the LEFT, RIGHT, DOWN and UP face
  double J[4][N1], Q[4][N1];
#pragma unroll 1
  for (int f = 0; f < 4; ++f) {
    const bool x = f < 2, zero = (f & 1) == 0;  // zero: this element is the 0 side
    const bool in = f == 0 ? gx > 0 : (f == 1 ? gx < dim - 1 : (f == 2 ? gy < dim - 1 : gy > 0));
    const size_t ne = f == 0 ? e - 1 : (f == 1 ? e + 1 : (f == 2 ? e + dim : e - dim));
#pragma unroll 1
    for (int j = 0; j < N1; ++j) {
      double u0 = 0, d0 = 0, uN = 0, dN = 0;
      if (zero || in)
#pragma unroll 1
        for (int i = 0; i < N1; ++i) {
          const double v = ld(x ? i * N1 + j : j * N1 + i, zero ? e : ne);
          if (i == 0) u0 = v;
          d0 = fma(tb.D0[i], v, d0);
        }
      if (!zero || in)
#pragma unroll 1
        for (int i = 0; i < N1; ++i) {
          const double v = ld(x ? i * N1 + j : j * N1 + i, zero ? ne : e);
          if (i == N) uN = v;
          dN = fma(tb.DN[i], v, dN);
        }
      face_combine<double>(tb.w[j], tb.WH[j], a.nu, in, u0, d0, uN, dN, J[f][j], Q[f][j]);
    }
  }
  double acc = 0.0;
#pragma unroll 1
  for (int i1 = 0; i1 < N1; ++i1)
#pragma unroll 1
    for (int j = 0; j < N1; ++j) {
      double v = face_seed<double, N>(i1, j, Q[0][j], Q[1][j], Q[2][i1], Q[3][i1]);
      v = fma(tb.D0[i1], J[0][j], fma(tb.DN[i1], J[1][j], v));
#pragma unroll 1
      for (int i = 0; i < N1; ++i) v = fma(tb.KW[(i1 * N1 + i) * N1 + j], ld(i * N1 + j, e), v);
#pragma unroll 1
      for (int i = 0; i < N1; ++i) v = fma(tb.KW[(j * N1 + i) * N1 + i1], ld(i1 * N1 + i, e), v);
      v = fma(tb.D0[j], J[2][i1], v);
      v = fma(tb.DN[j], J[3][i1], v);
      const size_t gk = (size_t)(i1 * N1 + j) * noe + e;
      if (BASE == APPLY_RESID) {
        const double rv = __ldg(a.b + gk) - v;
        a.out[gk] = rv;
        acc = fma(rv, rv, acc);
      } else {
        a.out[gk] = v;
        if (kDot) {
          const double c = ld(i1 * N1 + j, e);
          if (BASE == APPLY_CG) pnew[gk] = c;
          acc = fma(c, v, acc);
        }
      }
    }
  return acc;
}

// A large penalty's terms into the outputs that this thread (z of ZS) has
// stored for element (gx, gy); returns its share of the reduction.  (A pass of
// its own, off the path of the other penalties: as conditions on it, 5 % there.)
template <int P, int MODE, int ZS, typename Ld>
__device__ __noinline__ double add_penalty(const ApplyArgs<double>& a, const Tab<double, P>& tb, int gx, int gy, int z,
                                           Ld ld, const double* pnew) {
  constexpr int N = P, N1 = P + 1, BASE = apply_base_mode(MODE);
  const size_t noe = (size_t)a.dim * a.dim, e = (size_t)gy * a.dim + gx;
  double acc = 0.0;
#pragma unroll 1
  for (int i1 = 0; i1 < N1; ++i1) {
    if (ZS > 1 && min(i1, N - i1) % ZS != z) continue;  // its columns
#pragma unroll 1
    for (int j = 0; j < N1; ++j) {
      const bool face = i1 == 0 || i1 == N || j == 0 || j == N;
      if (BASE == APPLY_PLAIN && !face) continue;
      const size_t gk = (size_t)(i1 * N1 + j) * noe + e;
      double v = a.out[gk];
      if (face) {
        const double q = fx_penalty<P>(tb, a.nu, a.dim, gx, gy, i1, j, ld);
        v = __dadd_rn(v, BASE == APPLY_RESID ? -q : q);
        a.out[gk] = v;
      }
      if (BASE == APPLY_RESID) acc = fma(v, v, acc);
      else if (BASE == APPLY_CG) acc = fma(pnew[gk], v, acc);
      else if (BASE == APPLY_DOT) acc = fma(ld(i1 * N1 + j, e), v, acc);
    }
  }
  return acc;
}

template <int P, int TX, int TY, int MODE>
__device__ __forceinline__ void apply_tile_fx(const ApplyArgs<double>& a, const ApplyTab<double, P>& tabs, int bx,
                                              int by, int bid, int nblocks) {
  constexpr int N = P, N1 = P + 1, NN = N1 * N1, TE = TX * TY;
  constexpr int NE = FxTab<P>::NE, NO = FxTab<P>::NO;
  constexpr int BASE = apply_base_mode(MODE);
  // *_PIVOT modes: the sums over differences from the element's first value
  // (exact zero-sum rows make that the same sum), so that the scale, and with
  // it the rounding, is that of the element's variation
  constexpr bool kPivot = MODE != BASE;
  constexpr bool kDot = (BASE == APPLY_CG || BASE == APPLY_DOT);
  constexpr bool kRegs = FxForm<P>::regs;
  constexpr int ZS = fx_split(P), NT = TE * ZS;  // threads per element, per CTA
  constexpr int kHalo = FxSmem<P, TX, TY>::HALO, RS = FxSmem<P, TX, TY>::RS, kWarps = NT / 32;
  const FxTab<P>& fx = tabs.fx;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red_sh[32];
  __shared__ int2 s_nu[NE];                                   // nu HB(b) w_b
  __shared__ unsigned s_mag[ZS > 1 ? ZS * TE : 1];
  __shared__ int s_be[(TY + 2) * (TX + 2)];                   // the elements' scales, halo ring included
  __shared__ double s_v0[kPivot ? (TY + 2) * (TX + 2) : 1];   // and pivots
  int2* uf = reinterpret_cast<int2*>(smem_raw);  // values (low word, high word), then limb pairs, in place
  long long* rf = reinterpret_cast<long long*>(smem_raw) + NN * TE;
  long long* ht_ = rf + 4 * N1 * RS;  // the halo elements' traces (doubled)

  if (kDot) {
    if (*(volatile int*)&a.st->done) return;  // converged: the launch is a no-op
  }
  const int tx = threadIdx.x, ty = threadIdx.y, t = ty * TX + tx;  // the element
  const int z = ZS > 1 ? threadIdx.z : 0, lt = z * TE + t;         // which of its threads; linear id
  const int dim = a.dim;
  const int x0 = bx * TX, y0 = a.row0 + by * TY;
  const int gx = x0 + tx, gy = y0 + ty;
  const bool act = (gx < dim) && (gy < dim);
  const unsigned noe = (unsigned)dim * (unsigned)dim;  // (dim <= 65535)
  const size_t e = (size_t)gy * dim + gx;

  bool first = true;
  double beta = 0.0;
  int par = 0;
  if (BASE == APPLY_CG) {
    first = a.st->first != 0;
    beta = a.st->beta;
    par = a.st->parity;
  }
  const double* __restrict__ pold = par ? a.pbuf1 : a.pbuf0;
  double* __restrict__ pnew = par ? a.pbuf0 : a.pbuf1;
  auto addr = [&](const double* p, int k) { return fx_addr(p, noe, k); };
  const FxLoad<BASE == APPLY_CG> ld{a.in, pold, noe, beta, first};
  // the slot of x index (i, odd) and y index (j, odd): even indices at their
  // node, odd ones at the mirrored node
  auto at = [&](int i, bool io, int j, bool jo) -> int { return ((io ? N - i : i) * N1 + (jo ? N - j : j)) * TE + t; };
  auto Be = [&](int row, int col) -> int& { return s_be[(row + 1) * (TX + 2) + col + 1]; };
  auto V0 = [&](int row, int col) -> double& { return s_v0[kPivot ? (row + 1) * (TX + 2) + col + 1 : 0]; };
  auto R = [&](int face, int b, int tt) -> long long& { return rf[(face * N1 + b) * RS + tt]; };  // LEFT, RIGHT, DOWN, UP
  // the 2 (TX + TY) elements around the tile: above, below, right, left of it
  auto halo_at = [&](int h, int& hx, int& hy) {
    const int q = h < 2 * TX ? h % TX : (h - 2 * TX) % TY;
    hx = h < 2 * TX ? x0 + q : (h < 2 * TX + TY ? x0 + TX : x0 - 1);
    hy = h < TX ? y0 - 1 : (h < 2 * TX ? y0 + TY : y0 + q);
    return hx >= 0 && hx < dim && hy >= 0 && hy < dim;
  };
  const bool large = fx_large_nu(a.nu * fx.wmax, fx.sk);
  bool bad = false;
  if (lt < NE) {
    s_nu[lt] = large ? make_int2(0, 0) : fx_nu(fx.w[lt] * a.nu, fx.sk);
  }

  // ---- phase 0 --------------------------------------------------------------
  // (raw values in registers where they fit, else in the shared column)
  unsigned mag = 0;
  double rv_[kRegs ? NN : 1];
  auto raw = [&](int k) -> double {
    if (kRegs) return rv_[kRegs ? k : 0];
    const int2 v = uf[k * TE + t];
    return __hiloint2double(v.y, v.x);
  };
  auto put_raw = [&](int k, double v) {
    if (kRegs) rv_[kRegs ? k : 0] = v;
    else uf[k * TE + t] = make_int2(__double2loint(v), __double2hiint(v));
  };
  const double pv = kPivot && act ? ld(0, e) : 0.0;
  if constexpr (ZS == 1) {
#pragma unroll(FxForm<P>::load_unroll)
    for (int k = 0; k < NN; ++k) put_raw(k, act ? ld(k, e) : 0.0);
  } else {
#pragma unroll(FxForm<P>::load_unroll / ZS)
    for (int k = z; k < NN; k += ZS) put_raw(k, act ? ld(k, e) : 0.0);
  }
  // the halo elements: element h to lane h / kWarps of warp h % kWarps
  for (int h = (lt & 31) * kWarps + (lt >> 5); h < kHalo; h += NT) {
    int hx, hy;
    if (!halo_at(h, hx, hy)) continue;
    const size_t he = (size_t)hy * dim + hx;
    const double v0 = kPivot ? ld(0, he) : 0.0;
    unsigned hm = 0;
#pragma unroll(N1)
    for (int k = 0; k < NN; ++k) hm = max(hm, fx_mag(kPivot ? __dadd_rn(ld(k, he), -v0) : ld(k, he)));
    bad = bad || (hm >> 21) >= (unsigned)kFxMaxExp;
    if ((hm >> 21) < (unsigned)kFxMinExp) {
      for (int k = 0; k < NN; ++k) bad = bad || (kPivot ? __dadd_rn(ld(k, he), -v0) : ld(k, he)) != 0.0;
    }
    Be(hy - y0, hx - x0) = fx_be(hm);
    if (kPivot) V0(hy - y0, hx - x0) = v0;
  }
#pragma unroll(kRegs ? NN : N1)
  for (int k = z; k < NN; k += ZS) {
    if (kPivot) put_raw(k, __dadd_rn(raw(k), -pv));
    mag = max(mag, fx_mag(raw(k)));
  }
  // out of the fixed-point range: this tile takes the plain code (a value
  // below kFxMinExp only where the whole element is)
  bool small = false;
  if ((mag >> 21) < (unsigned)kFxMinExp) {
#pragma unroll(kRegs ? NN : 1)
    for (int k = z; k < NN; k += ZS) small = small || raw(k) != 0.0;
  }
  if constexpr (ZS > 1) {
    s_mag[lt] = mag;
    __syncthreads();  // the other threads' values, and their magnitude
    mag = max(mag, s_mag[lt ^ TE]);
    static_assert(ZS == 2, "one other thread");
  }
  bad = bad || (mag >> 21) >= (unsigned)kFxMaxExp || (small && (mag >> 21) < (unsigned)kFxMinExp);
  const int bs = fx_be(mag);
  Be(ty, tx) = bs;
  if (kPivot) {
    V0(ty, tx) = pv;
    bad = bad || (fx_mag(pv) >> 21) >= (unsigned)kFxMaxExp;
  }
#pragma unroll
  for (int i = 0; i < NE; ++i)
#pragma unroll
    for (int j = 0; j < NE; ++j) {  // mirrored nodes: the quad's slots are its own
      if (ZS > 1 && (i + j) % ZS != z) continue;
      const bool mi = 2 * i == N, mj = 2 * j == N;
      long long q[4];
      q[0] = fx_fix(raw(i * N1 + j), bs);
      q[1] = mi ? 0 : fx_fix(raw((N - i) * N1 + j), bs);
      q[2] = mj ? 0 : fx_fix(raw(i * N1 + N - j), bs);
      q[3] = mi || mj ? 0 : fx_fix(raw((N - i) * N1 + N - j), bs);
      fx_quad(q);
      uf[at(i, false, j, false)] = fx_limbs_of(q[0]);
      if (!mi) uf[at(i, true, j, false)] = fx_limbs_of(q[1]);
      if (!mj) uf[at(i, false, j, true)] = fx_limbs_of(q[2]);
      if (!mi && !mj) uf[at(i, true, j, true)] = fx_limbs_of(q[3]);
    }
  double acc = 0.0;
  const bool plain = __syncthreads_or(bad);
  if (plain) {
    if (act && z == 0) acc = plain_element<P, MODE>(a, tabs.t, gx, gy, ld, pnew);
  } else {

  // ---- phase 1 --------------------------------------------------------------
  // w times the normal derivatives of the element's four faces, component b of
  // the face in slot b (odd components at the mirrored node)
#pragma unroll(FxForm<P>::face_unroll)
  for (int b = z; b < N1; b += ZS) {
    const int wb = b < NE ? b : N - b;
    long long r0, rN;
    fx_derivatives<P>(fx, wb, [&](int k, bool odd) { return uf[((odd ? N - k : k) * N1 + b) * TE + t]; }, r0, rN);
    R(0, b, t) = r0;
    R(1, b, t) = rN;
    fx_derivatives<P>(fx, wb, [&](int k, bool odd) { return uf[(b * N1 + (odd ? N - k : k)) * TE + t]; }, r0, rN);
    R(2, b, t) = r0;
    R(3, b, t) = rN;
  }
  // the faces of the elements around the tile, one pair of mirrored components
  // per thread: above and right of the tile the 0 side, below and left the N
  // side
  for (int task = lt; task < kHalo * NE; task += NT) {
    const int j = task / kHalo, h = task - j * kHalo;
    int hx, hy;
    if (!halo_at(h, hx, hy)) continue;
    const size_t he = (size_t)hy * dim + hx;
    const bool yface = h < 2 * TX;
    const bool nside = (h >= TX && h < 2 * TX) || h >= 2 * TX + TY;
    const int di = yface ? 1 : N1, dj = yface ? N1 : 1;  // strides along the normal and the face
    const bool mid = 2 * j == N;
    const double v0 = kPivot ? ld(0, he) : 0.0;
    const int hbe = Be(hy - y0, hx - x0);
    auto hv = [&](int i, int jj) {
      const double v = ld(i * di + jj * dj, he);
      return fx_fix(kPivot ? __dadd_rn(v, -v0) : v, hbe);
    };
    int2 q[NE][4];
#pragma unroll
    for (int k = 0; k < NE; ++k) {
      const bool mk = 2 * k == N;
      long long f[4];
      f[0] = hv(k, j);
      f[1] = mk ? 0 : hv(N - k, j);
      f[2] = mid ? 0 : hv(k, N - j);
      f[3] = mk || mid ? 0 : hv(N - k, N - j);
      fx_quad(f);
#pragma unroll
      for (int c = 0; c < 4; ++c) q[k][c] = fx_limbs_of(f[c]);
    }
    // (at the middle component both halves of q hold the same values)
#pragma unroll
    for (int odd_b = 0; odd_b < 2; ++odd_b) {
      const int b = odd_b ? N - j : j;
      long long r0, rN;
      fx_derivatives<P>(fx, j, [&](int k, bool odd) { return q[k][(odd ? 1 : 0) + 2 * odd_b]; }, r0, rN);
      const int2 ev = q[0][2 * odd_b], od = q[0][1 + 2 * odd_b];
      ht_[b * kHalo + h] = nside ? fx_traceN(ev, od) : fx_trace0(ev, od);
      const int f = h < TX ? 2 : (h < 2 * TX ? 3 : (h < 2 * TX + TY ? 0 : 1));
      const int q0 = h < TX ? 0 : (h < 2 * TX ? TX : (h < 2 * TX + TY ? 2 * TX : 2 * TX + TY));
      R(f, b, TE + h - q0) = nside ? rN : r0;
    }
  }
  __syncthreads();

  // ---- phase 1b -------------------------------------------------------------
  // A face's J replaces its N side's derivative, its Q the 0 side's (of a side
  // outside the tile: the entry behind the tile's).
  auto X0 = [&](int b, int tt) { return fx_trace0(uf[b * TE + tt], uf[(N * N1 + b) * TE + tt]); };
  auto XN = [&](int b, int tt) { return fx_traceN(uf[b * TE + tt], uf[(N * N1 + b) * TE + tt]); };
  auto Y0 = [&](int b, int tt) { return fx_trace0(uf[(b * N1) * TE + tt], uf[(b * N1 + N) * TE + tt]); };
  auto YN = [&](int b, int tt) { return fx_traceN(uf[(b * N1) * TE + tt], uf[(b * N1 + N) * TE + tt]); };
  auto mult = [](int b) { return b >= NE ? 0 : (2 * b == N ? 1 : 2); };  // how often component b takes a constant
  // *_PIVOT: the 0 side's pivot less the N side's (a missing side: zero)
  auto delta = [&](bool in0, int r0, int c0, bool inN, int rN, int cN) -> double {
    return kPivot ? __dadd_rn(in0 ? V0(r0, c0) : 0.0, inN ? -V0(rN, cN) : 0.0) : 0.0;
  };
  if (act) {
    const bool rint = gx < dim - 1, uint_ = gy > 0;
    const bool rt = tx < TX - 1, ut = ty > 0;
    const int tr = rt ? t + 1 : TE + ty, tu = ut ? t - TX : TE + tx;
    const int ber = rint ? Be(ty, tx + 1) : bs, beu = uint_ ? Be(ty - 1, tx) : bs;
    const double dr = delta(rint, ty, tx + 1, true, ty, tx), du = delta(uint_, ty - 1, tx, true, ty, tx);
#pragma unroll(FxForm<P>::face_unroll)
    for (int b = 0; b < N1; ++b) {
      const int wb = b < NE ? b : N - b;
      const int2 nu = s_nu[wb];
      long long J, Q;
      if (ZS == 1 || z == 0) {
        const long long t0 = rt ? X0(b, t + 1) : ht_[b * kHalo + 2 * TX + ty];
        fx_face<kPivot>(nu, rint, true, t0, R(0, b, tr), ber, XN(b, t), R(1, b, t), bs, dr, mult(b),
                        J, Q);
        R(1, b, t) = J;
        R(0, b, tr) = Q;
      }
      if (ZS == 1 || z == 1) {
        const long long t0 = ut ? Y0(b, t - TX) : ht_[b * kHalo + tx];
        fx_face<kPivot>(nu, uint_, true, t0, R(2, b, tu), beu, YN(b, t), R(3, b, t), bs, du, mult(b),
                        J, Q);
        R(3, b, t) = J;
        R(2, b, tu) = Q;
      }
    }
  }
  // the faces without an N side in the tile: below it (or below the mesh's last row) ...
  const int rows_in = min(TY, dim - y0);
  for (int q = lt; q < TX * N1; q += NT) {
    const int b = q / TX, c = q - b * TX, wb = b < NE ? b : N - b, el = (rows_in - 1) * TX + c;
    if (x0 + c >= dim) continue;
    const bool in = y0 + rows_in < dim;
    const int eN = rows_in < TY ? el + TX : TE + c;
    long long J, Q;
    fx_face<kPivot>(s_nu[wb], true, in, Y0(b, el), R(2, b, el), Be(rows_in - 1, c),
                    ht_[b * kHalo + TX + c], R(3, b, eN), in ? Be(TY, c) : 0, delta(true, rows_in - 1, c, in, TY, c),
                    mult(b), J, Q);
    R(3, b, eN) = J;
    R(2, b, el) = Q;
  }
  // ... and left of it
  for (int q = lt; q < TY * N1; q += NT) {
    const int b = q / TY, r = q - b * TY, wb = b < NE ? b : N - b, el = r * TX;
    if (y0 + r >= dim) continue;
    const bool in = x0 > 0;
    long long J, Q;
    fx_face<kPivot>(s_nu[wb], true, in, X0(b, el), R(0, b, el), Be(r, 0),
                    ht_[b * kHalo + 2 * TX + TY + r], R(1, b, TE + r), in ? Be(r, -1) : 0,
                    delta(true, r, 0, in, r, -1), mult(b), J, Q);
    R(1, b, TE + r) = J;
    R(0, b, el) = Q;
  }
  __syncthreads();

  // ---- phase 2 --------------------------------------------------------------
  {
    // the four faces: where J and Q are (component b at + b * RS), and the face's scale
    struct Face {
      const long long *pj, *pq;
      int be;
    };
    auto scale = [&](bool in, int row, int col) {
      const int b = in ? max(bs, Be(row, col)) : bs;
      return kPivot ? max(b, fx_biased(delta(true, ty, tx, in, row, col))) : b;
    };
    const Face fl{&R(1, 0, tx > 0 ? t - 1 : TE + ty), &R(0, 0, t), scale(gx > 0, ty, tx - 1)};
    const Face fr{&R(1, 0, t), &R(0, 0, tx < TX - 1 ? t + 1 : TE + ty), scale(gx < dim - 1, ty, tx + 1)};
    const Face fd{&R(3, 0, ty < TY - 1 ? t + TX : TE + tx), &R(2, 0, t), scale(gy < dim - 1, ty + 1, tx)};
    const Face fu{&R(3, 0, t), &R(2, 0, ty > 0 ? t - TX : TE + tx), scale(gy > 0, ty - 1, tx)};
    // the outputs' scale; where it is not the element's own, its values move to it
    const int be = max(bs, max(max(fl.be, fr.be), max(fd.be, fu.be)) - (kPivot ? 1 : kFxRoom));
    if (be > bs)
      for (int k = z; k < NN; k += ZS) uf[k * TE + t] = fx_shift(uf[k * TE + t], min(be - bs, 63));
    if (ZS > 1) __syncthreads();
    const int ex = fx_exp(be, fx.sk);
    auto jump = [&](const Face& f, int b) { return fx_scaled(f.pj[b * RS], be - f.be); };
    auto half_q = [&](const Face& f, int b) { return fx_scaled(f.pq[b * RS], be - f.be); };
    // what the even / odd columns lift from the x faces
    int2 xm[N1], xp[N1];
#pragma unroll
    for (int b = 0; b < N1; ++b) {
      const long long jl = jump(fl, b), jr = jump(fr, b);
      xm[b] = fx_limbs_of(jl - jr);
      xp[b] = fx_limbs_of(jl + jr);
    }
    // one pair of mirrored columns i, N - i (mi: the middle column alone)
    auto columns = [&](int i, auto mid_c) {
      constexpr bool mi = decltype(mid_c)::value;
      asm volatile("" ::: "memory");  // the values are read again for each pair: registers
      FxAcc oe[N1], oo[N1];           // the even and the odd column, y in parity form
#pragma unroll
      for (int j = 0; j < N1; ++j) {
        const int b = j < NE ? j : N - j;
        oe[j] = fx_zero();
        oo[j] = fx_zero();
        fx_mac(oe[j], fx.le[i * NE + b], xm[j]);
        if (!mi) fx_mac(oo[j], fx.lo[i * NE + b], xp[j]);
      }
      // x sums
#pragma unroll
      for (int k = 0; k < NE; ++k)
#pragma unroll
        for (int j = 0; j < N1; ++j)
          fx_mac(oe[j], fx.ke[(i * NE + k) * NE + (j < NE ? j : N - j)], uf[(k * N1 + j) * TE + t]);
      if (!mi) {
#pragma unroll
        for (int k = 0; k < NO; ++k)
#pragma unroll
          for (int j = 0; j < N1; ++j)
            fx_mac(oo[j], fx.ko[(i * NO + k) * NE + (j < NE ? j : N - j)], uf[((N - k) * N1 + j) * TE + t]);
      }
      // y sums and the y faces' lifts
#pragma unroll
      for (int s = 0; s < (mi ? 1 : 2); ++s) {
        const int row = s ? N - i : i;
        int2 c[N1];
#pragma unroll
        for (int j = 0; j < N1; ++j) c[j] = uf[(row * N1 + j) * TE + t];
        const long long jd = jump(fd, row), ju = jump(fu, row);
        const int2 ym = fx_limbs_of(jd - ju), yp = fx_limbs_of(jd + ju);
#pragma unroll
        for (int j = 0; j < NE; ++j) {
          FxAcc& o = s ? oo[j] : oe[j];
#pragma unroll
          for (int k = 0; k < NE; ++k) fx_mac(o, fx.ke[(j * NE + k) * NE + i], c[k]);
          fx_mac(o, fx.le[j * NE + i], ym);
        }
#pragma unroll
        for (int j = 0; j < NO; ++j) {
          FxAcc& o = s ? oo[N - j] : oe[N - j];
#pragma unroll
          for (int k = 0; k < NO; ++k) fx_mac(o, fx.ko[(j * NO + k) * NE + i], c[N - k]);
          fx_mac(o, fx.lo[j * NE + i], yp);
        }
      }
      // the totals, with the face terms: Q enters node 0, less Q node N
      long long re[N1], ro[N1];
#pragma unroll
      for (int j = 0; j < N1; ++j) {
        re[j] = fx_total(oe[j]);
        ro[j] = mi ? 0 : fx_total(oo[j]);
      }
      if (!mi && i == 0) {
#pragma unroll
        for (int b = 0; b < N1; ++b) {
          const long long ql = half_q(fl, b), qr = half_q(fr, b);
          re[b] += ql - qr;
          ro[b] += ql + qr;
        }
      }
#pragma unroll
      for (int s = 0; s < (mi ? 1 : 2); ++s) {
        const long long qd = half_q(fd, s ? N - i : i), qu = half_q(fu, s ? N - i : i);
        (s ? ro[0] : re[0]) += qd - qu;
        (s ? ro[N] : re[N]) += qd + qu;
      }
      // back to the nodes
      auto emit = [&](int i1, int j, long long r) {
        const double v = fx_double(r, ex);
        const int k = i1 * N1 + j;
        double* out = const_cast<double*>(addr(a.out + e, k));
        if (BASE == APPLY_RESID) {
          const double rv = __ldg(addr(a.b + e, k)) - v;
          *out = rv;
          acc = fma(rv, rv, acc);
        } else {
          *out = v;
          if (kDot) {
            const double pk = ld(k, e);
            if (BASE == APPLY_CG) *const_cast<double*>(addr(pnew + e, k)) = pk;
            acc = fma(pk, v, acc);
          }
        }
      };
      auto emit_row = [&](int j, long long ve, long long vo) {
        if (mi) {
          emit(i, j, ve);
        } else {
          emit(i, j, ve + vo);
          emit(N - i, j, ve - vo);
        }
      };
#pragma unroll
      for (int j = 0; j < NE; ++j) {
        if (2 * j == N) {
          emit_row(j, re[j], ro[j]);
        } else {
          emit_row(j, re[j] + re[N - j], ro[j] + ro[N - j]);
          emit_row(N - j, re[j] - re[N - j], ro[j] - ro[N - j]);
        }
      }
    };
#pragma unroll(FxForm<P>::col_unroll)
    for (int i = z; i < NO; i += ZS)
      if (act) columns(i, std::false_type{});
    if constexpr (NE > NO)
      if (act && z == NO % ZS) columns(NE - 1, std::true_type{});
  }
    if (large && act) acc = add_penalty<P, MODE, ZS>(a, tabs.t, gx, gy, z, ld, pnew);
  }  // !plain
  if (BASE != APPLY_PLAIN) {
    const double bt = block_sum<double, NT>(acc, red_sh);
    double total;
    if (grid_sum_last<double, NT>(bt, a.red, bid, nblocks, red_sh, &total) && lt == 0)
      apply_finish<double, BASE>(a.st, total, par);
  }
}

}  // namespace sipg

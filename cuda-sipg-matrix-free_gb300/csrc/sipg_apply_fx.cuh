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
//   3  the elements that one scale does not fit (sipg_fx.cuh), by FP64 chains.
// Every output depends on the element and its four neighbours alone, through
// integers or through the chain of chain_node, so every tile shape gives the
// same bits.
//
// Bound by integer issue and its latency: 180 instructions per DoF at p = 4 (29
// of them the products; the rest conversions, parity form, limbs, 64-bit
// additions and shared memory); ncu: multiply-add pipe 57 %, 46 % of the issue
// slots with the 16 warps per SM that registers and shared memory allow, where FP64 chains are bound by an FP64
// pipe of 2 operations per SM and cycle (21 per DoF).  Measured, FP64 chains
// against this: 1024^2, p = 4 1080 -> 262 us (388 -> 1604 GB/s of the 16 bytes
// per DoF); 443^2, p = 8 977 -> 249 us; ~16 M DoF, p = 1..8: 25, 26, 25, 24, 22,
// 20, 18, 16 -> 84, 104, 103, 95, 87, 77, 74, 64 GDoF/s.  The 2-norm error against
// extended precision fell with it (p = 4, uniform values: 2.8e-16 -> 1.1e-16);
// entry by entry see sipg_fx.cuh.
#pragma once

#include <type_traits>

#include "sipg_apply.cuh"
#include "sipg_fx.cuh"

namespace sipg {

template <int P>
struct FxForm {
  static constexpr bool regs = P <= 4;  // raw values in registers between load and conversion
  static constexpr int row_unroll = fx_split(P) > 1 ? 1 : 2;  // rows of loads in flight, beyond that
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
template <bool CG, bool COHERENT>
struct FxLoad {
  const double *in, *pold;
  unsigned noe;
  double beta;
  bool first;
  __device__ __forceinline__ double at(const double* p) const { return COHERENT ? __ldcg(p) : __ldg(p); }
  __device__ __forceinline__ double operator()(int k, size_t e) const {
    const double r = at(fx_addr(in + e, noe, k));
    if (CG) return first ? r : fma(beta, at(fx_addr(pold + e, noe, k)), r);
    return r;
  }
};

// v + sum_i c(i) l(i) as one FP64 chain; PIVOT: over the differences l(i) - l(0).
// U: terms whose loads are in flight together.
template <int P, bool PIVOT, int U, typename C, typename V>
__device__ __forceinline__ double chain_sum(double v, C c, V l) {
  const double p0 = PIVOT ? l(0) : 0.0;
#pragma unroll(U)
  for (int i = 0; i <= P; ++i) v = fma(c(i), PIVOT ? l(i) - p0 : l(i), v);
  return v;
}

// One side of a face for the FP64 chains: its trace and normal derivative (D) at
// node q of the face of element e (x: an x face; last: the N side).
template <int P, bool PIVOT, int U, typename Ld>
__device__ __forceinline__ void chain_side(const double* D, bool x, bool last, int q, size_t e, Ld ld, double& u,
                                           double& d) {
  auto line = [&](int i) { return ld(x ? i * (P + 1) + q : q * (P + 1) + i, e); };
  u = line(last ? P : 0);
  d = chain_sum<P, PIVOT, U>(0.0, [&](int i) { return D[i]; }, line);
}

// The neighbour across face f (LEFT, RIGHT, DOWN, UP) of element (gx, gy) = e.
__device__ __forceinline__ bool chain_across(int f, int dim, int gx, int gy, size_t e, size_t& ne) {
  ne = f == 0 ? e - 1 : (f == 1 ? e + 1 : (f == 2 ? e + dim : e - dim));
  return f == 0 ? gx > 0 : (f == 1 ? gx < dim - 1 : (f == 2 ? gy < dim - 1 : gy > 0));
}

// Output (i1, j) of element (gx, gy) as one FP64 chain: the face terms, the x
// faces' lift, the row's and the column's stiffness sums, the y faces' lift.
// PIVOT: zero-sum rows over differences from the line's first value.
template <int P, bool PIVOT, int U, typename Ld>
__device__ __forceinline__ double chain_node(const Tab<double, P>* tb, double nu, int dim, int gx, int gy, int i1,
                                             int j, Ld ld) {
  constexpr int N = P, N1 = P + 1;
  const size_t e = (size_t)gy * dim + gx;
  double J[4], Q[4];  // at the node's line
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    const bool x = f < 2, zero = (f & 1) == 0;  // zero: this element is the 0 side
    const int q = x ? j : i1, k0 = x ? q : q * N1, kN = x ? N * N1 + q : q * N1 + N;
    size_t ne;
    const bool in = chain_across(f, dim, gx, gy, e, ne);
    const double own = ld(zero ? k0 : kN, e), other = in ? ld(zero ? kN : k0, ne) : 0.0;
    J[f] = mul_rn(in ? tb->WH[q] : tb->w[q], zero ? own - other : other - own);
    Q[f] = 0.0;
  }
#pragma unroll
  for (int d = 0; d < 2; ++d) {  // the x face, the y face that the node lies on
    const bool x = d == 0;
    const int at = x ? i1 : j, q = x ? j : i1, f = 2 * d + (at == 0 ? 0 : 1);
    if (at != 0 && at != N) continue;
    const bool zero = at == 0;
    size_t ne;
    const bool in = chain_across(f, dim, gx, gy, e, ne);
    double u0 = 0.0, d0 = 0.0, uN = 0.0, dN = 0.0, unused, v;
    chain_side<P, PIVOT, U>(zero ? tb->D0 : tb->DN, x, !zero, q, e, ld, zero ? u0 : uN, zero ? d0 : dN);
    if (in) chain_side<P, PIVOT, U>(zero ? tb->DN : tb->D0, x, zero, q, ne, ld, zero ? uN : u0, zero ? dN : d0);
    face_combine<double>(tb->w[q], tb->WH[q], nu, in, u0, d0, uN, dN, unused, v);
    Q[2 * d + 0] = zero ? v : 0.0;
    Q[2 * d + 1] = zero ? 0.0 : v;
  }
  double v = face_seed<double, N>(i1, j, Q[0], Q[1], Q[2], Q[3]);
  v = fma(tb->D0[i1], J[0], fma(tb->DN[i1], J[1], v));
  v = chain_sum<P, PIVOT, U>(v, [&](int i) { return tb->KW[(i1 * N1 + i) * N1 + j]; },
                             [&](int i) { return ld(i * N1 + j, e); });
  v = chain_sum<P, PIVOT, U>(v, [&](int i) { return tb->KW[(j * N1 + i) * N1 + i1]; },
                             [&](int i) { return ld(i1 * N1 + i, e); });
  v = fma(tb->D0[j], J[2], v);
  return fma(tb->DN[j], J[3], v);
}

// A generic pointer to the tables in the kernel's parameters: lanes that index
// them differently read them like global memory, where the constant bank would
// serve one address at a time.
template <int P>
__device__ __forceinline__ const Tab<double, P>* generic_tab(const Tab<double, P>& tb) {
  const Tab<double, P>* p = &tb;
  asm volatile("" : "+l"(p));
  return p;
}

// Stores output k of element e, whose value is v, as the mode does, and adds
// its share of the reduction.
template <int MODE, typename Ld>
__device__ __forceinline__ void chain_emit(const ApplyArgs<double>& a, size_t noe, int k, size_t e, double v, Ld ld,
                                           double* pnew, double& acc) {
  constexpr int BASE = apply_base_mode(MODE);
  const size_t gk = (size_t)k * noe + e;
  if (BASE == APPLY_RESID) {
    const double rv = __ldg(a.b + gk) - v;
    a.out[gk] = rv;
    acc = fma(rv, rv, acc);
  } else {
    a.out[gk] = v;
    if (BASE == APPLY_CG || BASE == APPLY_DOT) {
      const double c = ld(k, e);
      if (BASE == APPLY_CG) pnew[gk] = c;
      acc = fma(c, v, acc);
    }
  }
}

// The elements x0 + b of row gy for the bits b of todo, by the warp; every
// ZS-th part of the work for the z-th of the elements' threads.  Returns the
// lane's share of the reduction.
//
// Few elements: one output per lane, as many elements at a time as that fills
// (the latency of some 4 n FP64 operations each).  Many: one element per lane,
// its faces' values first; bound by the FP64 pipe.  1024^2, p = 4, and 443^2,
// p = 8, one element in 1000 uneven (and four neighbours each): 310 and 308 us,
// none: 264 and 250; all uneven: 1617 and 1571 us (an element per lane alone: the
// same; an output per lane alone: 3860 and 2706; a kernel of FP64 chains: 1083
// and 980).
template <int P, int MODE, int ZS, typename Ld>
__device__ __noinline__ double chain_elements(const ApplyArgs<double>& a, const Tab<double, P>& tabs, int x0, int gy,
                                              unsigned todo, int z, Ld ld, double* pnew) {
  constexpr int N = P, N1 = P + 1, NN = N1 * N1;
  constexpr bool kPivot = MODE != apply_base_mode(MODE);
  constexpr int G = NN <= 32 ? 32 / NN : 1;
  constexpr int kMany = 8 * G > 16 ? 16 : 8 * G;
  const int lane = threadIdx.x & 31, dim = a.dim;
  const size_t noe = (size_t)dim * dim;
  double acc = 0.0;
  if (__popc(todo) < kMany) {
    const Tab<double, P>* tb = generic_tab<P>(tabs);
    const int slot = NN <= 32 ? lane / NN : 0;
    for (int pick = 0; todo; pick ^= 1) {
      int gx = -1;  // the slot's element
#pragma unroll 1
      for (int g = 0; g < G; ++g, todo &= todo - 1)
        if (g == slot && todo) gx = x0 + __ffs(todo) - 1;
      if ((ZS > 1 && pick != z) || gx < 0) continue;
#pragma unroll 1
      for (int k = NN <= 32 ? lane % NN : lane; k < NN; k += 32)
        chain_emit<MODE>(a, noe, k, (size_t)gy * dim + gx,
                         chain_node<P, kPivot, N1>(tb, a.nu, dim, gx, gy, k / N1, k % N1, ld), ld, pnew, acc);
    }
    return acc;
  }
  if (!(todo >> lane & 1)) return acc;
  const int gx = x0 + lane;
  const size_t e = (size_t)gy * dim + gx;
  double J[4][N1], Q[4][N1];
#pragma unroll 1
  for (int f = 0; f < 4; ++f) {
    const bool x = f < 2, zero = (f & 1) == 0;
    size_t ne;
    const bool in = chain_across(f, dim, gx, gy, e, ne);
#pragma unroll 1
    for (int q = 0; q < N1; ++q) {
      double u0 = 0.0, d0 = 0.0, uN = 0.0, dN = 0.0;
      if (zero || in) chain_side<P, kPivot, N1>(tabs.D0, x, false, q, zero ? e : ne, ld, u0, d0);
      if (!zero || in) chain_side<P, kPivot, N1>(tabs.DN, x, true, q, zero ? ne : e, ld, uN, dN);
      face_combine<double>(tabs.w[q], tabs.WH[q], a.nu, in, u0, d0, uN, dN, J[f][q], Q[f][q]);
    }
  }
#pragma unroll 1
  for (int i1 = z; i1 < N1; i1 += ZS) {
#pragma unroll 1
    for (int j = 0; j < N1; ++j) {
      double v = face_seed<double, N>(i1, j, Q[0][j], Q[1][j], Q[2][i1], Q[3][i1]);
      v = fma(tabs.D0[i1], J[0][j], fma(tabs.DN[i1], J[1][j], v));
      v = chain_sum<P, kPivot, N1>(v, [&](int i) { return tabs.KW[(i1 * N1 + i) * N1 + j]; },
                                   [&](int i) { return ld(i * N1 + j, e); });
      v = chain_sum<P, kPivot, N1>(v, [&](int i) { return tabs.KW[(j * N1 + i) * N1 + i1]; },
                                   [&](int i) { return ld(i1 * N1 + i, e); });
      v = fma(tabs.D0[j], J[2][i1], v);
      v = fma(tabs.DN[j], J[3][i1], v);
      chain_emit<MODE>(a, noe, i1 * N1 + j, e, v, ld, pnew, acc);
    }
  }
  return acc;
}

// A large penalty's terms into the outputs that this thread (z of ZS) has
// stored for element (gx, gy), pen[q] the coefficient at node q of a face; acc:
// its share of the reduction so far.  (A pass
// of its own, off the path of the other penalties: as conditions on it, 5 % there.)
template <int P, int MODE, int ZS, typename Ld>
__device__ __noinline__ double add_penalty(const ApplyArgs<double>& a, const double2* pen, int gx, int gy, int z, Ld ld,
                                           double acc) {
  constexpr int N = P, N1 = P + 1, BASE = apply_base_mode(MODE);
  const size_t noe = (size_t)a.dim * a.dim, e = (size_t)gy * a.dim + gx;
  auto mine = [&](int i1) { return ZS == 1 || min(i1, N - i1) % ZS == z; };  // the columns it stored
#pragma unroll 1
  for (int f = 0; f < 4; ++f) {
    const bool x = f < 2, zero = (f & 1) == 0;
    size_t ne;
    const bool in = chain_across(f, a.dim, gx, gy, e, ne);
    double own[N1], other[N1], v[N1];
#pragma unroll
    for (int q = 0; q < N1; ++q) {
      if (!mine(x ? 0 : q)) continue;
      const int k0 = x ? q : q * N1, kN = x ? N * N1 + q : q * N1 + N;
      own[q] = ld(zero ? k0 : kN, e);
      other[q] = in ? ld(zero ? kN : k0, ne) : 0.0;
      v[q] = a.out[(size_t)(zero ? k0 : kN) * noe + e];
    }
#pragma unroll
    for (int q = 0; q < N1; ++q) {
      if (!mine(x ? 0 : q)) continue;
      const int k0 = x ? q : q * N1, kN = x ? N * N1 + q : q * N1 + N;
      const double2 c = pen[q];
      const double jump = BASE == APPLY_RESID ? __dadd_rn(other[q], -own[q]) : __dadd_rn(own[q], -other[q]);
      a.out[(size_t)(zero ? k0 : kN) * noe + e] = fx_add_penalty(v[q], c, jump);
      if (BASE == APPLY_CG || BASE == APPLY_DOT) acc = fma(own[q], fma(c.x, jump, c.y * jump), acc);
    }
  }
  if (BASE == APPLY_RESID) {
    acc = 0.0;
#pragma unroll 1
    for (int i1 = 0; i1 < N1; ++i1) {
      if (!mine(i1)) continue;
#pragma unroll
      for (int j = 0; j < N1; ++j) {
        const double v = a.out[(size_t)(i1 * N1 + j) * noe + e];
        acc = fma(v, v, acc);
      }
    }
  }
  return acc;
}

template <int P, int TX, int TY, int MODE>
__device__ __forceinline__ void apply_tile_fx(const ApplyArgs<double>& a, const ApplyTab<double, P>& tabs, int bx,
                                              int by, int bid, int nblocks) {
  constexpr int N = P, N1 = P + 1, NN = N1 * N1, TE = TX * TY;
  static_assert(TX == 32, "a warp is a row of elements");
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
  __shared__ double2 s_pen[N1];                               // nu w, if large
  __shared__ int s_be[(TY + 2) * (TX + 2)];                   // the elements' scales, halo ring included
  __shared__ double s_v0[kPivot ? (TY + 2) * (TX + 2) : 1];   // and pivots
  int2* uf = reinterpret_cast<int2*>(smem_raw);  // values (low word, high word), then limb pairs, in place
  long long* rf = reinterpret_cast<long long*>(smem_raw) + NN * TE;
  long long* ht_ = rf + 4 * N1 * RS;  // the halo elements' traces (doubled)
  unsigned* lines = reinterpret_cast<unsigned*>(rf);  // phase 0, ZS > 1: what the element's threads know of its lines

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
  const FxLoad<BASE == APPLY_CG, false> ld{a.in, pold, noe, beta, first};
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
  if (large && lt < N1) s_pen[lt] = fx_penalty(tabs.t.w[lt], fx.wl[lt], a.nu);
  if (lt < NE) s_nu[lt] = large ? make_int2(0, 0) : fx_nu(fx.w[lt] * a.nu, fx.sk);

  // ---- phase 0 --------------------------------------------------------------
  // (raw values in registers where they fit, else in the shared column)
  double rv_[kRegs ? NN : 1];
  auto raw = [&](int k) -> double {
    if (kRegs) return rv_[kRegs ? k : 0];
    const int2 v = uf[k * TE + t];
    return __hiloint2double(v.y, v.x);
  };
  // The element's largest magnitude, and the exponent that every node's row (i1
  // fixed) or column reaches: in the *_PIVOT modes of the differences along the
  // line, else of the values.
  unsigned mag = 0, rows = ~0u, low_words = 0;  // rows: the smallest of them
  unsigned cmax[N1];                            // columns: largest magnitude, or (pivot) ordered high word
  int cmin[kPivot ? N1 : 1];
#pragma unroll
  for (int j = 0; j < N1; ++j) {
    cmax[j] = kPivot ? 0x80000000u : 0u;
    if (kPivot) cmin[j] = 0x7fffffff;
  }
  auto row = [&](auto value) {  // value(j): one row
    unsigned rmax = 0;
    int rlo = 0x7fffffff, rhi = (int)0x80000000;
#pragma unroll
    for (int j = 0; j < N1; ++j) {
      const double v = value(j);
      low_words |= (unsigned)__double2loint(v);
      if (kPivot) {
        const int o = fx_ordered(__double2hiint(v));
        rlo = min(rlo, o), rhi = max(rhi, o);
        cmin[kPivot ? j : 0] = min(cmin[kPivot ? j : 0], o), cmax[j] = (unsigned)max((int)cmax[j], o);
      } else {
        const unsigned m = fx_mag(v);
        rmax = max(rmax, m);
        cmax[j] = max(cmax[j], m);
      }
    }
    rows = min(rows, kPivot ? fx_apart(rlo, rhi) : rmax);
  };
  const double pv = kPivot && act ? ld(0, e) : 0.0;
  auto load = [&](int k) {
    const double v = act ? ld(k, e) : 0.0;
    return kPivot ? __dadd_rn(v, -pv) : v;
  };
  if constexpr (kRegs) {
#pragma unroll
    for (int k = 0; k < NN; ++k) rv_[k] = act ? ld(k, e) : 0.0;
  } else {
#pragma unroll(FxForm<P>::row_unroll)
    for (int i = z; i < N1; i += ZS)
      row([&](int j) {
        const double v = load(i * N1 + j);
        uf[(i * N1 + j) * TE + t] = make_int2(__double2loint(v), __double2hiint(v));
        return v;
      });
  }
  // the halo elements: element h to lane h / kWarps of warp h % kWarps
  for (int h = (lt & 31) * kWarps + (lt >> 5); h < kHalo; h += NT) {
    int hx, hy;
    if (!halo_at(h, hx, hy)) continue;
    const size_t he = (size_t)hy * dim + hx;
    const double v0 = kPivot ? ld(0, he) : 0.0;
    unsigned hm = 0, hl = 0;
#pragma unroll(N1)
    for (int k = 0; k < NN; ++k) {
      const double v = kPivot ? __dadd_rn(ld(k, he), -v0) : ld(k, he);
      hm = max(hm, fx_mag(v));
      hl |= (unsigned)__double2loint(v);
    }
    Be(hy - y0, hx - x0) = fx_be(hm, (hm | hl) != 0);
    if (kPivot) V0(hy - y0, hx - x0) = v0;
  }
  if constexpr (kRegs) {
#pragma unroll
    for (int i = 0; i < N1; ++i)
      row([&](int j) {
        double& v = rv_[kRegs ? i * N1 + j : 0];
        if (kPivot) v = __dadd_rn(v, -pv);
        return v;
      });
  }
  if constexpr (ZS > 1) {
    static_assert(ZS == 2, "one other thread");
    auto mine = [&](int q, int tt) -> unsigned& { return lines[q * NT + tt]; };
#pragma unroll
    for (int j = 0; j < N1; ++j) {
      mine(j, lt) = cmax[j];
      if (kPivot) mine(N1 + 2 + j, lt) = (unsigned)cmin[kPivot ? j : 0];
    }
    mine(N1, lt) = rows;
    mine(N1 + 1, lt) = low_words;
    __syncthreads();  // the other thread's rows
    const int other = z ? lt - TE : lt + TE;
#pragma unroll
    for (int j = 0; j < N1; ++j) {
      cmax[j] = kPivot ? (unsigned)max((int)cmax[j], (int)mine(j, other)) : max(cmax[j], mine(j, other));
      if (kPivot) cmin[kPivot ? j : 0] = min(cmin[kPivot ? j : 0], (int)mine(N1 + 2 + j, other));
    }
    rows = min(rows, mine(N1, other));
    low_words |= mine(N1 + 1, other);
  }
  unsigned cols = ~0u;
#pragma unroll
  for (int j = 0; j < N1; ++j) {
    if (kPivot) {
      const int lo = cmin[kPivot ? j : 0], hi = (int)cmax[j];
      cols = min(cols, fx_apart(lo, hi));
      mag = max(mag, max((unsigned)fx_ordered(lo) << 1, (unsigned)fx_ordered(hi) << 1));
    } else {
      cols = min(cols, cmax[j]);
      mag = max(mag, cmax[j]);
    }
  }
  const int low = (int)(max(rows, cols) >> 21);
  const int bs = fx_be(mag, (mag | low_words) != 0);
  Be(ty, tx) = bs;
  if (kPivot) V0(ty, tx) = pv;
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
  __syncthreads();

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
      if (!kPivot) return b;
      const double d = delta(true, ty, tx, in, row, col);
      return max(b, d != 0.0 && fx_biased(d) <= kFxMinExp ? kFxNoScale : fx_biased(d));
    };
    const Face fl{&R(1, 0, tx > 0 ? t - 1 : TE + ty), &R(0, 0, t), scale(gx > 0, ty, tx - 1)};
    const Face fr{&R(1, 0, t), &R(0, 0, tx < TX - 1 ? t + 1 : TE + ty), scale(gx < dim - 1, ty, tx + 1)};
    const Face fd{&R(3, 0, ty < TY - 1 ? t + TX : TE + tx), &R(2, 0, t), scale(gy < dim - 1, ty + 1, tx)};
    const Face fu{&R(3, 0, t), &R(2, 0, ty > 0 ? t - TX : TE + tx), scale(gy > 0, ty - 1, tx)};
    // the outputs' scale; where it is not the element's own, its values move to it
    const int faces = max(max(fl.be, fr.be), max(fd.be, fu.be));
    const int be = max(bs, faces - (kPivot ? 1 : kFxRoom));
    const bool fits = act && !fx_chains(be, faces, low);  // one scale fits the element
    const unsigned todo = __ballot_sync(0xffffffffu, act && !fits);
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
      if (fits) columns(i, std::false_type{});
    if constexpr (NE > NO)
      if (fits && z == NO % ZS) columns(NE - 1, std::true_type{});
    if (large && fits) acc = add_penalty<P, MODE, ZS>(a, s_pen, gx, gy, z, ld, acc);

    // ---- phase 3 ------------------------------------------------------------
    if (todo) acc += chain_elements<P, MODE, ZS>(a, tabs.t, x0, gy, todo, z, ld, pnew);
  }
  if (BASE != APPLY_PLAIN) {
    const double bt = block_sum<double, NT>(acc, red_sh);
    double total;
    if (grid_sum_last<double, NT>(bt, a.red, bid, nblocks, red_sh, &total) && lt == 0)
      apply_finish<double, BASE>(a.st, total, par);
  }
}

}  // namespace sipg

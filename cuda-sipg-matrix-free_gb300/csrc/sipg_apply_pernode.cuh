// sipg_apply_pernode.cuh -- the FP64 apply for small meshes: one thread per
// output node.
//
// GB300 issues FP64 at a small fraction of its FP32 rate: a warp instruction of
// 32 conversions or sums occupies a sub-partition's FP64 unit for 64 cycles.
// The element-per-thread apply (sipg_apply_fx.cuh) gives every thread the whole
// (p+1)^2 outputs of one element, so a mesh with few elements -- 256 at 16 x 16
// -- runs a few warps, each through thousands of instructions, on a handful of
// SMs.  Here a CTA holds EX x EY elements and gives each output node its own
// thread: the same operations spread over (p+1)^2 times more warps, on more SMs.
//
// The sums are the fixed-point ones of sipg_apply_fx.cuh (sipg_fx.cuh): the
// same integers, whose sums do not depend on their order, so the result is
// bit-identical to every other FP64 tile shape; only the CG reductions (p.Ap,
// r.r) group their partial sums differently.
//
// A CTA works through tiles blockIdx.x, blockIdx.x + gridDim.x, ... with the
// grid at most the resident CTAs, so a mesh of any size has at most a few
// thousand reduction partials.  Phases per tile (static shared memory, tens of
// KB at most):
//   0  the values of the EX x EY elements and of the 2 (EX + EY) halo elements
//      around them (from L2: small meshes live there), with p = r + beta p_old
//      formed on the fly in the CG mode, and the elements' scales;
//   1  their parity form, four mirrored nodes per thread;
//   2  w times the normal derivatives, one face component per thread;
//   3  J and Q, one face component per thread;
//   4  one parity component of the output per thread;
//   5  one output node per thread, then the epilogue (store, direction store
//      in the CG mode, deterministic grid reduction in the CG / DOT / residual
//      modes).
// An element that one scale does not fit (sipg_fx.cuh) takes FP64 chains in
// phase 5, its nodes' threads one each.
#pragma once

#include <algorithm>
#include <atomic>

#include "sipg_apply_fx.cuh"

namespace sipg {

template <int P, int SHAPE>
struct PernodeShape {
  static constexpr int N1 = P + 1, NN = N1 * N1;
  static constexpr int EX = pernode_ex(P, SHAPE), EY = pernode_ey(P), NE = EX * EY;
  static constexpr int NT = (NE * NN + 31) / 32 * 32;  // threads: whole warps, the tail idle in phase 2
  // resident CTAs the registers are limited for: what 80 to 128 a thread allow,
  // two up to 512 threads (128^2, p = 1, at 128 registers: 10.3 us, at 80: 8.2;
  // p = 4, shape 1: 45 us with one CTA, 29 with two; p = 6: 53 and 39)
  static constexpr int MIN_BLOCKS =
      NT >= 512 ? 1 : (NT > 256 ? 2 : 65536 / (NT * (P == 1 ? 80 : 128)));
  static constexpr int SX = EX + 2, SY = EY + 2;       // element slots, halo ring included
  static constexpr int NX = EY * (EX + 1) * N1;        // x-face nodes: [EY][EX+1][N1]
  static constexpr int NY = EX * (EY + 1) * N1;        // y-face nodes: [EY+1][EX][N1]
};

// The CTA's shared memory.
template <int P, int SHAPE>
struct PernodeFxSmem {
  using S = PernodeShape<P, SHAPE>;
  static constexpr int NSLOT = S::SX * S::SY;
  int2 us[NSLOT * S::NN];     // slot (sy, sx) = element (y0 - 1 + sy, x0 - 1 + sx): values, then parity form
  double own[S::NE * S::NN];  // the tile's values [node][element]
  static constexpr int RX = S::EY * S::SX * S::N1, RY = S::SY * S::EX * S::N1;
  long long r0[RX + RY], rN[RX + RY];  // derivatives of the x faces, then the y faces: 0 side, N side
  long long xj[S::NX], xq[S::NX], yj[S::NY], yq[S::NY];
  long long tot[S::NE * S::NN];  // the output's parity components
  unsigned mag[NSLOT];           // zero between tiles
  unsigned lines[2 * S::NE];     // the smallest of an element's rows' and columns' largest magnitudes
  int be[NSLOT], bo[S::NE];      // scales of the slots' values, of the outputs
  int xbe[S::EY * (S::EX + 1)], ybe[S::EX * (S::EY + 1)];  // of the faces
  FxTab<P> fx;
  int2 nu[FxTab<P>::NE];
  bool large;
};

// The fixed-point tables into shared memory (indexed per thread below: a
// constant-bank read whose address differs across the warp would serialise),
// the penalty's coefficients, and cleared magnitudes.
template <int P, int SHAPE>
__device__ __forceinline__ void pernode_fx_tables(PernodeFxSmem<P, SHAPE>& sm, const FxTab<P>& fx, double nu) {
  const int t = threadIdx.x;
  static_assert(sizeof(FxTab<P>) % 8 == 0, "copied as 8-byte words");
  for (int k = t; k < (int)(sizeof(FxTab<P>) / 8); k += PernodeShape<P, SHAPE>::NT)
    reinterpret_cast<long long*>(&sm.fx)[k] = reinterpret_cast<const long long*>(&fx)[k];
  for (int k = t; k < PernodeFxSmem<P, SHAPE>::NSLOT; k += PernodeShape<P, SHAPE>::NT) sm.mag[k] = 0;
  const bool large = fx_large_nu(nu * fx.wmax, fx.sk);
  if (t < FxTab<P>::NE) {
    sm.nu[t] = large ? make_int2(0, 0) : fx_nu(fx.w[t] * nu, fx.sk);
  }
  if (t == 0) sm.large = large;
  __syncthreads();
}

// (Three terms in flight: with all of them the call's registers cost every
// per-node tile; 128^2, p = 5: 34 us instead of 29.)
template <int P, typename Ld>
__device__ __noinline__ double chain_node_call(const Tab<double, P>& tabs, double nu, int dim, int gx, int gy, int i1,
                                               int j, Ld ld) {
  return chain_node<P, false, 3>(generic_tab<P>(tabs), nu, dim, gx, gy, i1, j, ld);
}

// One tile (origin x0, y0): phases 0-5, returning this thread's share of the
// reduction (p.Ap in the CG / DOT modes, r.r in the residual mode).
// kCoherent: read a.in and pold through L2 only -- for a caller that runs
// while other CTAs of the same grid write them (the persistent CG).
template <int P, int SHAPE, int MODE, bool kCoherent>
__device__ __forceinline__ double pernode_tile_fx(const ApplyArgs<double>& a, PernodeFxSmem<P, SHAPE>& sm,
                                                  const ApplyTab<double, P>& tabs, int x0, int y0, bool first,
                                                  double beta, const double* __restrict__ pold,
                                                  double* __restrict__ pnew) {
  using S = PernodeShape<P, SHAPE>;
  using Tb = FxTab<P>;
  constexpr int N = P, N1 = S::N1, NN = S::NN, EX = S::EX, EY = S::EY, NE = S::NE, NT = S::NT;
  constexpr int SX = S::SX, SY = S::SY, NX = S::NX, NY = S::NY, NSLOT = SX * SY;
  constexpr int HE = Tb::NE, HO = Tb::NO;
  constexpr bool kDot = (MODE == APPLY_CG || MODE == APPLY_DOT);
  const FxTab<P>& fx = sm.fx;
  const int t = threadIdx.x;
  const int dim = a.dim;
  const size_t noe = (size_t)dim * dim;
  auto ldin = [&](const double* p) -> double { return kCoherent ? __ldcg(p) : __ldg(p); };
  auto ld = [&](int k, size_t e) -> double {
    const double v = ldin(a.in + (size_t)k * noe + e);
    return MODE == APPLY_CG && !first ? fma(beta, ldin(pold + (size_t)k * noe + e), v) : v;
  };
  auto corner = [](int sx, int sy) { return (sx == 0 || sx == SX - 1) && (sy == 0 || sy == SY - 1); };
  auto in_mesh = [&](int sx, int sy) {
    const int gx = x0 - 1 + sx, gy = y0 - 1 + sy;
    return gx >= 0 && gx < dim && gy >= 0 && gy < dim;
  };
  // ---- phase 0: values and magnitudes ----------------------------------------
  // (every load of the thread first, so that they are in flight together)
  if (t < 2 * NE) sm.lines[t] = ~0u;
  constexpr int IT = (NSLOT * NN + NT - 1) / NT;
  double vr[IT], vp[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int idx = t + it * NT, k = idx / NSLOT, sl = idx - k * NSLOT;
    const int sy = sl / SX, sx = sl - sy * SX;
    vr[it] = vp[it] = 0.0;
    if (idx < NSLOT * NN && !corner(sx, sy) && in_mesh(sx, sy)) {
      const size_t gk = (size_t)k * noe + (size_t)(y0 - 1 + sy) * dim + (x0 - 1 + sx);
      vr[it] = ldin(a.in + gk);
      if (MODE == APPLY_CG && !first) vp[it] = ldin(pold + gk);
    }
  }
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int idx = t + it * NT, k = idx / NSLOT, sl = idx - k * NSLOT;
    const int sy = sl / SX, sx = sl - sy * SX;
    if (idx >= NSLOT * NN) break;
    const double v = MODE == APPLY_CG && !first ? fma(beta, vp[it], vr[it]) : vr[it];
    const unsigned m = fx_mag(v) | min((unsigned)__double2loint(v), 1u);  // zero for zeros only
    if (m != 0) atomicMax(&sm.mag[sl], m);
    sm.us[sl * NN + k] = make_int2(__double2loint(v), __double2hiint(v));
    if (sx > 0 && sx < SX - 1 && sy > 0 && sy < SY - 1) sm.own[k * NE + (sy - 1) * EX + sx - 1] = v;
  }
  __syncthreads();
  // ---- phase 1: parity form ---------------------------------------------------
  auto scale = [&](int sl) { return fx_be(sm.mag[sl], sm.mag[sl] != 0); };
  for (int sl = t; sl < NSLOT; sl += NT) sm.be[sl] = scale(sl);
  for (int task = t; task < NSLOT * HE * HE; task += NT) {
    const int sl = task / (HE * HE), q2 = task - sl * (HE * HE), i = q2 / HE, j = q2 - i * HE;
    const int be = scale(sl);
    const bool mi = 2 * i == N, mj = 2 * j == N;
    int2* u = sm.us + sl * NN;
    const int k0 = i * N1 + j, k1 = (N - i) * N1 + j, k2 = i * N1 + N - j, k3 = (N - i) * N1 + N - j;
    auto raw = [&](int k) { return __hiloint2double(u[k].y, u[k].x); };
    long long q[4];
    q[0] = fx_fix(raw(k0), be);
    q[1] = mi ? 0 : fx_fix(raw(k1), be);
    q[2] = mj ? 0 : fx_fix(raw(k2), be);
    q[3] = mi || mj ? 0 : fx_fix(raw(k3), be);
    fx_quad(q);
    u[k0] = fx_limbs_of(q[0]);
    if (!mi) u[k1] = fx_limbs_of(q[1]);
    if (!mj) u[k2] = fx_limbs_of(q[2]);
    if (!mi && !mj) u[k3] = fx_limbs_of(q[3]);
  }
  __syncthreads();
  // ---- phase 2: normal derivatives -------------------------------------------
  constexpr int TX_ = EY * SX * N1, TY_ = SY * EX * N1;
  for (int task = t; task < TX_ + TY_; task += NT) {
    const bool x = task < TX_;
    const int q = x ? task : task - TX_;
    const int b = q % N1, r = q / N1, wb = b < HE ? b : N - b;
    // x: tile row r / SX, slot column r % SX; y: slot row r / EX, tile column r % EX
    const int sl = x ? (r / SX + 1) * SX + r % SX : (r / EX) * SX + r % EX + 1;
    const int2* u = sm.us + sl * NN;
    long long r0, rN;
    fx_derivatives<P>(fx, wb, [&](int k, bool odd) {
      const int kk = odd ? N - k : k;
      return x ? u[kk * N1 + b] : u[b * N1 + kk];
    }, r0, rN);
    sm.r0[task] = r0;
    sm.rN[task] = rN;
  }
  for (int sl = t; sl < NSLOT; sl += NT) sm.mag[sl] = 0;  // for the next tile
  __syncthreads();
  // ---- phase 3: J and Q ---------------------------------------------------------
  for (int f = t; f < NX + NY; f += NT) {
    const bool x = f < NX;
    const int q = x ? f : f - NX, b = q % N1, r = q / N1, wb = b < HE ? b : N - b;
    int s0, sN, i0, iN, face;  // slots of the two sides, their derivatives
    bool zv, nv;
    if (x) {  // x face c of tile row ey: the left slot is the N side, the right one the 0 side
      const int c = r % (EX + 1), ey = r / (EX + 1);
      sN = (ey + 1) * SX + c, s0 = sN + 1;
      iN = (ey * SX + c) * N1 + b, i0 = iN + N1;
      nv = in_mesh(c, ey + 1), zv = in_mesh(c + 1, ey + 1);
      face = ey * (EX + 1) + c;
    } else {  // y face c of tile column ex: the upper slot is the 0 side, the lower one the N side
      const int ex = r % EX, c = r / EX;
      s0 = c * SX + ex + 1, sN = s0 + SX;
      i0 = TX_ + (c * EX + ex) * N1 + b, iN = i0 + EX * N1;
      zv = in_mesh(ex + 1, c), nv = in_mesh(ex + 1, c + 1);
      face = c * EX + ex;
    }
    if (!zv && !nv) continue;
    const int2 *u0 = sm.us + s0 * NN, *uN = sm.us + sN * NN;
    const int ke = x ? b : b * N1, ko = x ? N * N1 + b : b * N1 + N;
    const int be0 = sm.be[s0], beN = sm.be[sN];
    long long J, Q;
    fx_face<false>(sm.nu[wb], zv, nv, fx_trace0(u0[ke], u0[ko]),
                   sm.r0[i0], be0, fx_traceN(uN[ke], uN[ko]), sm.rN[iN], beN, 0.0, 0, J, Q);
    const int bf = !zv ? beN : (!nv ? be0 : max(be0, beN));
    if (x) {
      sm.xj[q] = J;
      sm.xq[q] = Q;
      if (b == 0) sm.xbe[face] = bf;
    } else {
      sm.yj[q] = J;
      sm.yq[q] = Q;
      if (b == 0) sm.ybe[face] = bf;
    }
  }
  __syncthreads();
  // ---- phase 4: the output's parity components -----------------------------------
  int be_out = 0, faces = 0;  // the scales of the thread's element
  if (t < NE * NN) {
    const int le = t % NE, k = t / NE, ex = le % EX, ey = le / EX;
    const int ka = k / N1, kb = k - ka * N1;  // slot indices along x and y
    if (x0 + ex < dim && y0 + ey < dim) {
      const int sl = (ey + 1) * SX + ex + 1;
      const int2* u = sm.us + sl * NN;
      const int bs = sm.be[sl];
      const int fL = ey * (EX + 1) + ex, fR = fL + 1, fU = ey * EX + ex, fD = fU + EX;  // faces
      const int bL = sm.xbe[fL], bR = sm.xbe[fR], bU = sm.ybe[fU], bD = sm.ybe[fD];
      faces = max(max(bL, bR), max(bD, bU));
      const int be = be_out = max(bs, faces - kFxRoom);
      if (k < N1) {  // one row and one column each
        unsigned row = 0, col = 0;
#pragma unroll
        for (int i = 0; i < N1; ++i) {
          row = max(row, fx_mag(sm.own[(i * N1 + k) * NE + le]));
          col = max(col, fx_mag(sm.own[(k * N1 + i) * NE + le]));
        }
        atomicMin(&sm.lines[2 * le], row);
        atomicMin(&sm.lines[2 * le + 1], col);
      }
      const int so = be - bs, xp = fx_exp(be, fx.sk);
      auto own = [&](int kk) { return so > 0 ? fx_shift(u[kk], min(so, 63)) : u[kk]; };
      const bool oa = ka >= HE, ob = kb >= HE;  // odd indices sit at the mirrored slots
      const int ia = oa ? N - ka : ka, ib = ob ? N - kb : kb;
      FxAcc s = fx_zero();
      // x sums and lift, then y
      const int na = oa ? HO : HE, nb = ob ? HO : HE;
      const int2 *ta = oa ? fx.ko + ia * HO * HE + ib : fx.ke + ia * HE * HE + ib;
      const int2 *tb = ob ? fx.ko + ib * HO * HE + ia : fx.ke + ib * HE * HE + ia;
#pragma unroll
      for (int q = 0; q < HE; ++q)
        if (q < na) fx_mac(s, ta[q * HE], own((oa ? N - q : q) * N1 + kb));
#pragma unroll
      for (int q = 0; q < HE; ++q)
        if (q < nb) fx_mac(s, tb[q * HE], own(ka * N1 + (ob ? N - q : q)));
      const long long jl = fx_scaled(sm.xj[fL * N1 + kb], be - bL), jr = fx_scaled(sm.xj[fR * N1 + kb], be - bR);
      const long long jd = fx_scaled(sm.yj[fD * N1 + ka], be - bD), ju = fx_scaled(sm.yj[fU * N1 + ka], be - bU);
      fx_mac(s, (oa ? fx.lo : fx.le)[ia * HE + ib], fx_limbs_of(oa ? jl + jr : jl - jr));
      fx_mac(s, (ob ? fx.lo : fx.le)[ib * HE + ia], fx_limbs_of(ob ? jd + ju : jd - ju));
      long long r = fx_total(s);
      auto half_q = [&](long long q, int bf) { return fx_scaled(q, be - bf); };
      if (ia == 0) {
        const long long ql = half_q(sm.xq[fL * N1 + kb], bL), qr = half_q(sm.xq[fR * N1 + kb], bR);
        r += oa ? ql + qr : ql - qr;
      }
      if (ib == 0) {
        const long long qd = half_q(sm.yq[fD * N1 + ka], bD), qu = half_q(sm.yq[fU * N1 + ka], bU);
        r += ob ? qd + qu : qd - qu;
      }
      sm.tot[le * NN + k] = r;
      if (k == 0) sm.bo[le] = xp;
    }
  }
  __syncthreads();
  // ---- phase 5: one output node per thread ---------------------------------------
  double acc = 0.0;
  if (t < NE * NN) {
    const int le = t % NE, k = t / NE;  // element fastest: neighbouring threads store neighbouring elements
    const int ex = le % EX, ey = le / EX, i1 = k / N1, j = k - i1 * N1;
    const int gx = x0 + ex, gy = y0 + ey;
    if (gx < dim && gy < dim) {
      const long long* T = sm.tot + le * NN;
      const int i = i1 < N - i1 ? i1 : N - i1, jj = j < N - j ? j : N - j;
      auto row = [&](int ka) -> long long {  // the component at y node j
        if (2 * jj == N) return T[ka * N1 + jj];
        const long long ev = T[ka * N1 + jj], od = T[ka * N1 + N - jj];
        return j == jj ? ev + od : ev - od;
      };
      long long r = row(i);
      if (2 * i != N) r = i1 == i ? r + row(N - i) : r - row(N - i);
      double v = fx_double(r, sm.bo[le]);
      if (fx_chains(be_out, faces, (int)(max(sm.lines[2 * le], sm.lines[2 * le + 1]) >> 21))) {
        v = chain_node_call<P>(tabs.t, a.nu, dim, gx, gy, i1, j,
                               FxLoad<MODE == APPLY_CG, kCoherent>{a.in, pold, (unsigned)noe, beta, first});
      } else if (sm.large) {
        const size_t e = (size_t)gy * dim + gx;
        const double own = sm.own[k * NE + le];
        auto face = [&](int q, bool in, int ka, size_t ne) {
          v = fx_add_penalty(v, fx_penalty(tabs.t.w[q], fx.wl[q], a.nu), __dadd_rn(own, in ? -ld(ka, ne) : 0.0));
        };
        if (i1 == 0) face(j, gx > 0, N * N1 + j, e - 1);
        if (i1 == N) face(j, gx < dim - 1, j, e + 1);
        if (j == 0) face(i1, gy < dim - 1, i1 * N1 + N, e + dim);
        if (j == N) face(i1, gy > 0, i1 * N1, e - dim);
      }
      const size_t gk = (size_t)k * noe + (size_t)gy * dim + gx;
      if (MODE == APPLY_RESID) {
        const double rv = __ldg(a.b + gk) - v;
        a.out[gk] = rv;
        acc = fma(rv, rv, acc);
      } else {
        a.out[gk] = v;
        const double c = sm.own[k * NE + le];
        if (MODE == APPLY_CG) pnew[gk] = c;
        if (kDot) acc = fma(c, v, acc);
      }
    }
  }
  __syncthreads();  // the next tile overwrites the shared memory
  return acc;
}

template <typename T, int P, int SHAPE, int MODE>
__global__ void __launch_bounds__(PernodeShape<P, SHAPE>::NT, PernodeShape<P, SHAPE>::MIN_BLOCKS)
    k_sipg_apply_pernode(const __grid_constant__ ApplyArgs<T> a, const __grid_constant__ ApplyTab<T, P> tb) {
  using S = PernodeShape<P, SHAPE>;
  constexpr int EX = S::EX, EY = S::EY, NT = S::NT;
  __shared__ PernodeFxSmem<P, SHAPE> sm;
  __shared__ T red_sh[32];

  constexpr bool kDot = (MODE == APPLY_CG || MODE == APPLY_DOT);
  if (kDot) {
    if (*(volatile int*)&a.st->done) return;  // converged: the launch is a no-op
  }
  const int t = threadIdx.x;
  const int dim = a.dim;
  const int rows = a.nrows > 0 ? a.nrows : dim;  // a band of element rows from a.row0
  const int tiles_x = (dim + EX - 1) / EX, ntiles = tiles_x * ((rows + EY - 1) / EY);

  bool first = true;
  T beta = T(0);
  int par = 0;
  if (MODE == APPLY_CG) {
    first = a.st->first != 0;
    beta = a.st->beta;
    par = a.st->parity;
  }
  const T* __restrict__ pold = par ? a.pbuf1 : a.pbuf0;
  T* __restrict__ pnew = par ? a.pbuf0 : a.pbuf1;
  pernode_fx_tables<P, SHAPE>(sm, tb.fx, a.nu);
  T acc = T(0);
  // the CTA's tiles: blockIdx.x, + gridDim.x, ... (the grid is at most the
  // resident CTAs, so the reduction has few partials on any mesh)
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int x0 = (tile % tiles_x) * EX, y0 = a.row0 + (tile / tiles_x) * EY;
    acc += pernode_tile_fx<P, SHAPE, MODE, false>(a, sm, tb, x0, y0, first, beta, pold, pnew);
  }

  if (MODE != APPLY_PLAIN) {
    const T bt = block_sum<T, NT>(acc, red_sh);
    T total;
    if (grid_sum_last<T, NT>(bt, a.red, (int)blockIdx.x, (int)gridDim.x, red_sh, &total) && t == 0)
      apply_finish<T, MODE>(a.st, total, par);
  }
}

// Resident CTAs of a per-node kernel on the current device (occupancy x SMs),
// computed once per kernel and device.  (The kernel is a template argument: the
// shapes and modes of a degree share one function type, and a count kept per
// type was the first one's for all, so that the CTAs of a reduction depended on
// what had run before.)
template <auto KERNEL>
int pernode_resident_blocks(int threads) {
  constexpr int kDevices = 64;
  static std::atomic<int> cached[kDevices];
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
  const bool keep = dev >= 0 && dev < kDevices;
  if (keep && cached[dev].load(std::memory_order_relaxed) > 0) return cached[dev].load(std::memory_order_relaxed);
  if (dev < 0 || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERNEL, threads, 0) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return 152;  // one CTA per SM of a GB300
  }
  if (keep) cached[dev].store(sms * per_sm, std::memory_order_relaxed);
  return sms * per_sm;
}

template <typename T, int P, int SHAPE>
cudaError_t launch_apply_pernode_shape(int mode, const ApplyArgs<T>& a, const ApplyTab<T, P>& tb, cudaStream_t s) {
  using S = PernodeShape<P, SHAPE>;
  if (mode == APPLY_PREPARE) return cudaSuccess;  // static shared memory: no attribute to set
  const int rows = a.nrows > 0 ? a.nrows : a.dim;
  const long long ntiles = (long long)((a.dim + S::EX - 1) / S::EX) * ((rows + S::EY - 1) / S::EY);
  // at most the resident CTAs, and in a reducing mode at most one partial per
  // scratch entry
  auto grid_for = [&](int resident, bool reduces) {
    long long g = std::min<long long>(ntiles, resident);
    if (reduces) g = std::min<long long>(g, a.red.capacity);
    return (int)std::max<long long>(g, 1);
  };
  auto launch = [&](auto mode_c) {
    constexpr int MODE = decltype(mode_c)::value;
    constexpr auto kernel = k_sipg_apply_pernode<T, P, SHAPE, MODE>;
    kernel<<<grid_for(pernode_resident_blocks<kernel>(S::NT), MODE != APPLY_PLAIN), dim3(S::NT), 0, s>>>(a, tb);
  };
  switch (mode) {
    case APPLY_PLAIN: launch(std::integral_constant<int, APPLY_PLAIN>{}); break;
    case APPLY_CG: launch(std::integral_constant<int, APPLY_CG>{}); break;
    case APPLY_RESID: launch(std::integral_constant<int, APPLY_RESID>{}); break;
    case APPLY_DOT: launch(std::integral_constant<int, APPLY_DOT>{}); break;
    default: return cudaErrorInvalidValue;
  }
  count_launch();
  return cudaGetLastError();
}

// The per-node tile named by cfg (tpe = (p+1)^2; tx x ty one of the two
// compiled shapes).
template <typename T, int P>
cudaError_t launch_apply_pernode(const TileCfg& cfg, int mode, const ApplyArgs<T>& a, const HostTables& h,
                                 cudaStream_t s) {
  if (cfg.ty != pernode_ey(P)) return cudaErrorInvalidConfiguration;
  const ApplyTab<T, P>& tb = apply_tabs<T, P>(h);
  if (cfg.tx == pernode_ex(P, 0)) return launch_apply_pernode_shape<T, P, 0>(mode, a, tb, s);
  if (cfg.tx == pernode_ex(P, 1)) return launch_apply_pernode_shape<T, P, 1>(mode, a, tb, s);
  return cudaErrorInvalidConfiguration;
}

}  // namespace sipg

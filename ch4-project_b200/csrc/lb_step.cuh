// The fused step kernel (included by lb_kernels.cuh inside namespace ch4).
//
// One launch = one iteration of the reference loop for the populations: BGK
// collision (src/fluid.c:1033-1226) with the equilibrium of src/lb.c:382-415,
// the build_forcing terms (src/forcing.c:360-707), Guo forcing
// (src/forcing.c:1423-1435), the wall rules of src/boundary_conditions.c:419-1524
// and streaming (src/lb.c:544-584), for p, g and h.  Each population is read once
// and written once.
//
// EXACT (the FP64 instantiation) keeps every operation of the reference in its
// order, so the result is bit-identical.  The FP32 instantiation evaluates the
// same quantities as the even and odd parts of pairs of directions; its error
// against FP64 is reported, not zero.

template <typename S, typename A>
__device__ __forceinline__ void load_full(const StepParams<A>& P, int set, const S* p, A* f) {
#pragma unroll
  for (int q = 0; q < Q; q++) f[q] = Codec<S, A>::load(p, q * POP_BLOCK, P.w[q], P.shift[set]);
}
template <typename S, typename A, int set>
__device__ __forceinline__ void load_set(const StepParams<A>& P, long long idx, A* f) {
  load_full(P, set, pop_at<S>(P.fin[set], P.bstride, idx), f);
}

// The stored values of a cell as they are: f itself, or for the half-precision store the
// deviation f - w * shift.
template <typename S, typename A>
__device__ __forceinline__ void load_raw(const S* p, A* f) {
#pragma unroll
  for (int q = 0; q < Q; q++) f[q] = Codec<S, A>::load_raw(p, q * POP_BLOCK);
}

// the first direction q of pair k = 0 .. 8 of opposite directions (q, qinv(q))
__host__ __device__ constexpr int pair_q(int k) { return k < 3 ? 2 * k + 1 : k < 5 ? k + 4 : k < 7 ? k + 6 : k + 8; }

// Linear-index deltas to the neighbour at c = -1 / +1 along each axis, with the
// periodic wrap folded in (computed once per cell instead of once per direction).
struct Nbr {
  int xm, xp, ym, yp, zm, zp;
};

__device__ __forceinline__ Nbr neighbours(int x, int y, int z, int NX, int NY, int NZ) {
  const int sxy = NX * NY;
  Nbr n;
  n.xm = x == 0 ? NX - 1 : -1;
  n.xp = x == NX - 1 ? -(NX - 1) : 1;
  n.ym = y == 0 ? (NY - 1) * NX : -NX;
  n.yp = y == NY - 1 ? -(NY - 1) * NX : NX;
  n.zm = z == 0 ? (NZ - 1) * sxy : -sxy;
  n.zp = z == NZ - 1 ? -(NZ - 1) * sxy : sxy;
  return n;
}

template <int q, bool WITH_Y>
__device__ __forceinline__ int nbr_delta(const Nbr& n) {
  int d = 0;
  if constexpr (cx(q) < 0) d += n.xm;
  if constexpr (cx(q) > 0) d += n.xp;
  if constexpr (WITH_Y && cy(q) < 0) d += n.ym;
  if constexpr (WITH_Y && cy(q) > 0) d += n.yp;
  if constexpr (cz(q) < 0) d += n.zm;
  if constexpr (cz(q) > 0) d += n.zp;
  return d;
}

// The walls one set meets at this cell: per axis (0 x, 1 y, 2 z) whether a direction with
// c_a = +1 (hp) or -1 (hm) leaves through a wall of this set, and per side the fluid's slip
// flag or the value walls' fac.  Built only for cells on a wall row, column or plane.
struct Walls {
  uint32_t hit;   // bit a: a wall of this set at the upper end of axis a at this cell, bit 3 + a: lower
  uint32_t slip;  // the same bits for the fluid's specular walls
};

// fac = 2((T_wall - T_ref) - t) of a value wall of set 1 (temperature) or 2 (scalar) on
// axis a, upper (plus) or lower side, src/boundary_conditions.c:966-1236, 1249-1520: y walls
// T_top / T_bot with the fixed-flux and no-flux variants, x walls T_top on both sides (as
// the reference has it), z walls T_top / T_bot; scalar walls S_top / S_bot on every axis
template <int set, typename A>
__device__ __forceinline__ A wall_fac(const StepParams<A>& P, int a, bool plus, A tt, A ss) {
  const uint32_t F = P.feat, WL = P.walls;
  if constexpr (set == 2) return A(2) * (((plus ? P.S_top : P.S_bot) - P.S_ref) - ss);
  if (a == 1) {
    A T_wall = plus ? P.T_top : P.T_bot;
    if (plus && (F & K_TFLUX_P)) T_wall = A(0.5) * P.grad_T_top + tt + P.T_ref;
    if (!plus && (F & K_TFLUX_M)) T_wall = A(-0.5) * P.grad_T_bot + tt + P.T_ref;
    if (F & (plus ? K_TNOFLUX_P : K_TNOFLUX_M)) return A(0);
    return A(2) * ((T_wall - P.T_ref) - tt);
  }
  if (a == 0) {
    if (WL & (plus ? W_TNOFLUX_XP : W_TNOFLUX_XM)) return A(0);
    return A(2) * ((P.T_top - P.T_ref) - tt);
  }
  if (WL & (plus ? W_TNOFLUX_ZP : W_TNOFLUX_ZM)) return A(0);
  return A(2) * (((plus ? P.T_top : P.T_bot) - P.T_ref) - tt);
}

// direction q of the cell at p
template <typename S, typename A, bool RAW>
__device__ __forceinline__ void put(S* p, int q, A v, A w, A shift) {
  if constexpr (RAW) Codec<S, A>::store_raw(p, q * POP_BLOCK, v);
  else Codec<S, A>::store(p, q * POP_BLOCK, v, w, shift);
}

// The push of a cell that meets no wall: every value streams to x + c_q, the sets of a
// direction to one address.
template <typename S, typename A, bool THERM, bool SCAL, bool RAW, int q>
__device__ __forceinline__ void push_bulk_one(const StepParams<A>& P, int idx, const Nbr& nb, const A* f, const A* g,
                                              const A* h) {
  constexpr int sets = 1 + (THERM ? 1 : 0) + (SCAL ? 1 : 0);
  S* p = pop_at<S>(P.fout[0], sets * Q * POP_BLOCK, idx + nbr_delta<q, true>(nb));
  put<S, A, RAW>(p, q, f[q], P.w[q], RAW ? A(0) : A(P.shift[0]));
  if constexpr (THERM) put<S, A, RAW>(p, Q + q, g[q], P.w[q], RAW ? A(0) : A(P.shift[1]));
  if constexpr (SCAL) put<S, A, RAW>(p, (sets - 1) * Q + q, h[q], P.w[q], RAW ? A(0) : A(P.shift[2]));
}
template <typename S, typename A, bool THERM, bool SCAL, bool RAW>
__device__ __forceinline__ void push_bulk(const StepParams<A>& P, int idx, const Nbr& nb, const A* f, const A* g,
                                          const A* h) {
#define CH4_PUSH(Q_) push_bulk_one<S, A, THERM, SCAL, RAW, Q_>(P, idx, nb, f, g, h);
  CH4_PUSH(0) CH4_PUSH(1) CH4_PUSH(2) CH4_PUSH(3) CH4_PUSH(4) CH4_PUSH(5) CH4_PUSH(6) CH4_PUSH(7) CH4_PUSH(8)
  CH4_PUSH(9) CH4_PUSH(10) CH4_PUSH(11) CH4_PUSH(12) CH4_PUSH(13) CH4_PUSH(14) CH4_PUSH(15) CH4_PUSH(16)
  CH4_PUSH(17) CH4_PUSH(18)
#undef CH4_PUSH
}

// The push of one set of a cell on a wall; wallmode: 0 no walls of this set, 1 fluid walls,
// 2 value walls (temperature or scalar).
// RAW: `post` holds values as they are stored (a wall rule moves a value between directions
// of the same weight, so the deviation form passes through it unchanged).
template <typename S, typename A, int set, int q, bool RAW>
__device__ __forceinline__ void push_one(const StepParams<A>& P, int idx, const Nbr& nb, const A* post, int wallmode,
                                         const Walls& W, A tt, A ss) {
  const A sh = RAW ? A(0) : A(P.shift[set]);
  // the wall bit of each axis this direction leaves through (compile-time masks: q is fixed)
  constexpr uint32_t mx = cx(q) > 0 ? 1u : cx(q) < 0 ? 8u : 0u;
  constexpr uint32_t my = cy(q) > 0 ? 2u : cy(q) < 0 ? 16u : 0u;
  constexpr uint32_t mz = cz(q) > 0 ? 4u : cz(q) < 0 ? 32u : 0u;
  const bool hx = (W.hit & mx) != 0, hy = (W.hit & my) != 0, hz = (W.hit & mz) != 0;
  if (wallmode != 0 && (hx || hy || hz)) {
    if (wallmode == 1) {
      // a slip wall stands alone on its axis (the other axes are periodic), so a direction
      // that meets it meets no other wall
      if (int(hx) + int(hy) + int(hz) == 1) {
        const bool sx = (W.slip & mx) != 0, sy = (W.slip & my) != 0, sz = (W.slip & mz) != 0;
        // specular reflection: the hit axis keeps the cell's coordinate, the others stream
        // (src/boundary_conditions.c:606-610 (x), 751-753 (y), 895-899 (z))
        if (hx && sx) {
          constexpr int r = qmirror(q, 0);
          const int d = (cy(q) < 0 ? nb.ym : cy(q) > 0 ? nb.yp : 0) + (cz(q) < 0 ? nb.zm : cz(q) > 0 ? nb.zp : 0);
          put<S, A, RAW>(pop_at<S>(P.fout[set], P.bstride, idx + d), r, post[q], P.w[r], sh);
          return;
        }
        if (hy && sy) {
          constexpr int r = qmirror(q, 1);
          put<S, A, RAW>(pop_at<S>(P.fout[set], P.bstride, idx + nbr_delta<q, false>(nb)), r, post[q], P.w[r], sh);
          return;
        }
        if (hz && sz) {
          constexpr int r = qmirror(q, 2);
          const int d = (cx(q) < 0 ? nb.xm : cx(q) > 0 ? nb.xp : 0) + (cy(q) < 0 ? nb.ym : cy(q) > 0 ? nb.yp : 0);
          put<S, A, RAW>(pop_at<S>(P.fout[set], P.bstride, idx + d), r, post[q], P.w[r], sh);
          return;
        }
      }
      // halfway bounce-back, src/boundary_conditions.c:623,775,917
      constexpr int r = qinv(q);
      put<S, A, RAW>(pop_at<S>(P.fout[set], P.bstride, idx), r, post[q], P.w[r], sh);
    } else {
      // fixed value / flux walls: the reference's loops run y, then x, then z, each writing
      // the slot the cell pulls as inv[q]; the last wall the direction crosses decides
      // (src/boundary_conditions.c:1019-1027, 1118-1151, 1186-1224).  Temperature walls on
      // x store rhs(x).p[q] + w[inv q] fac, every other value wall rhs(x).p[inv q] + ...
      constexpr int r = qinv(q);
      const int a = hz ? 2 : hx ? 0 : 1;
      const bool plus = a == 2 ? cz(q) > 0 : a == 0 ? cx(q) > 0 : cy(q) > 0;
      const A fac = wall_fac<set>(P, a, plus, tt, ss);
      const A base = (set == 1 && a == 0) ? post[q] : post[r];
      put<S, A, RAW>(pop_at<S>(P.fout[set], P.bstride, idx), r, base + P.w[r] * fac, P.w[r], sh);
    }
    return;
  }
  put<S, A, RAW>(pop_at<S>(P.fout[set], P.bstride, idx + nbr_delta<q, true>(nb)), q, post[q], P.w[q], sh);
}

template <typename S, typename A, int set, bool RAW>
__device__ __forceinline__ void push_set(const StepParams<A>& P, int idx, const Nbr& nb, const A* post, int wallmode,
                                         const Walls& W, A tt, A ss) {
#define CH4_PUSH(Q_) push_one<S, A, set, Q_, RAW>(P, idx, nb, post, wallmode, W, tt, ss);
  CH4_PUSH(0) CH4_PUSH(1) CH4_PUSH(2) CH4_PUSH(3) CH4_PUSH(4) CH4_PUSH(5) CH4_PUSH(6) CH4_PUSH(7) CH4_PUSH(8)
  CH4_PUSH(9) CH4_PUSH(10) CH4_PUSH(11) CH4_PUSH(12) CH4_PUSH(13) CH4_PUSH(14) CH4_PUSH(15) CH4_PUSH(16)
  CH4_PUSH(17) CH4_PUSH(18)
#undef CH4_PUSH
}

// The push of a cell on a wall row, column or plane, out of line: wall cells are a thin
// shell of the lattice, and keeping their case in its own function keeps the registers of
// the bulk path (every other cell) at what the bulk needs.  `post` is the caller's copy of
// the post-collision values; P is a kernel or shared-memory parameter block.
template <typename S, typename A, int set, bool RAW>
__device__ __noinline__ void push_walled(const StepParams<A>& P, int idx, Nbr nb, const A* post, int wallmode,
                                         Walls W, A tt, A ss) {
  push_set<S, A, set, RAW>(P, idx, nb, post, wallmode, W, tt, ss);
}

// Per-cell quantities shared by the collision of every direction.
template <typename A>
struct CellState {
  A rho, ux, uy, uz, u2, tt, ss;
  A dr, dt, ds;  // sums of the values as loaded: rho, tt, ss less the shift of a deviation store
  A ts;          // temperature source of the particles (K_TSRC), else 0
  A Fx, Fy, Fz;
  A invtau, it, is;
  A base, uF;  // METHOD_TRT in FP32: 1 - u2/(2 cs^2), u.F
};

// ---- FP64: BGK and Guo's forcing, every operation in the reference's order
// (equilibrium src/lb.c:408, forcing src/forcing.c:1423-1435), a pair (q, -q) at a time.
// c_{-q}.u is -(c_q.u) exactly, so the products of c.u serve both directions with their signs,
// and the products with the weight serve the directions that share it: the same values with
// half the operations.  Measured, us a step: Kolmogorov 64^3 (FP64 pipe and latency) 20.5 ->
// 16.4, 128^3 116 -> 107; Rayleigh-Benard 256x256x64 (HBM, 93 % of a copy's rate) 449 -> 419.
// With two or three sets the constants of Guo's factors are formed again per pair (12 % more
// operations) instead of kept: 18 registers that the 128 of the memory-bound kernels lack.
template <bool KEEP, typename A>
struct Guo64 {
  A p[3], m[3], z[3];  // (1 - u)/cs^2, (-1 - u)/cs^2, -u/cs^2
  A u[3], invcs2;
  __device__ __forceinline__ Guo64(const A* v, A i2) : invcs2(i2) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      u[a] = v[a];
      p[a] = (A(1) - v[a]) * i2;
      m[a] = (A(-1) - v[a]) * i2;
      z[a] = (-v[a]) * i2;
    }
  }
  // (c_a - u_a)/cs^2 + c_a (c.u)/cs^4, ci = (c.u)/cs^4
  __device__ __forceinline__ A d(int a, int c, A ci) const {
    if (c == 0) return KEEP ? z[a] : (-u[a]) * invcs2;
    if (c > 0) return (KEEP ? p[a] : (A(1) - u[a]) * invcs2) + ci;
    return (KEEP ? m[a] : (A(-1) - u[a]) * invcs2) - ci;
  }
  __device__ __forceinline__ void add(A& r, const A* kF, int c0, int c1, int c2, A ci) const {
    r += kF[0] * d(0, c0, ci);
    r += kF[1] * d(1, c1, ci);
    r += kF[2] * d(2, c2, ci);
  }
};

// one value relaxed towards t w poly, as the reference writes it
template <typename A>
__device__ __forceinline__ void relax64(A& v, A invtau, A eq) {
  v += -invtau * (v - eq);
}

// the pairs [K0, K1) of one weight class; kF = (1 - dt/2tau) w rho F
template <int K0, int K1, bool THERM, bool SCAL, bool KEEP, typename A>
__device__ __forceinline__ void exact_pairs(const StepParams<A>& P, const CellState<A>& c, bool forced, bool tsrc,
                                            const Guo64<KEEP, A>& G, const A* kF, A w, A p2, A* f, A* g, A* h) {
  const A rw = c.rho * w, tw = c.tt * w, sw = c.ss * w, ts = w * c.ts;
#pragma unroll
  for (int k = K0; k < K1; k++) {
    const int q = pair_q(k), b = qinv(q);
    const A cu = cdot_rt(q, c.ux, c.uy, c.uz);
    const A t1 = P.invcs2 * cu, t2 = P.invtwocs4 * cu * cu;
    const A pq = A(1) + t1 + t2 - p2, pb = A(1) - t1 + t2 - p2;
    relax64(f[q], c.invtau, rw * pq);
    relax64(f[b], c.invtau, rw * pb);
    if (forced) {
      const A ci = cu * P.invcs4;
      G.add(f[q], kF, cx(q), cy(q), cz(q), ci);
      G.add(f[b], kF, cx(b), cy(b), cz(b), -ci);
    }
    if constexpr (THERM) {
      relax64(g[q], c.it, tw * pq);
      relax64(g[b], c.it, tw * pb);
      if (tsrc) g[q] += ts, g[b] += ts;  // add_forcing's w t_source, src/forcing.c:1475
    }
    if constexpr (SCAL) {
      relax64(h[q], c.is, sw * pq);
      relax64(h[b], c.is, sw * pb);
    }
  }
}

template <bool THERM, bool SCAL, typename A>
__device__ __forceinline__ void collide_exact(const StepParams<A>& P, const CellState<A>& c, bool forced, A* f, A* g,
                                              A* h) {
  constexpr bool KEEP = !THERM && !SCAL;
  const A u[3] = {c.ux, c.uy, c.uz};
  const A p2 = P.invtwocs2 * c.u2;
  const bool tsrc = THERM && (P.feat & K_TSRC);
  const Guo64<KEEP, A> G(u, P.invcs2);
  A kF[3];
  auto coefficients = [&](int q) {
    const A k = P.facw[q] * c.rho;
    kF[0] = k * c.Fx, kF[1] = k * c.Fy, kF[2] = k * c.Fz;
  };
  {  // rest: c.u = 0
    const A poly = A(1) - p2;
    relax64(f[0], c.invtau, c.rho * P.w[0] * poly);
    if (forced) {
      coefficients(0);
      G.add(f[0], kF, 0, 0, 0, A(0));
    }
    if constexpr (THERM) {
      relax64(g[0], c.it, c.tt * P.w[0] * poly);
      if (tsrc) g[0] += P.w[0] * c.ts;
    }
    if constexpr (SCAL) relax64(h[0], c.is, c.ss * P.w[0] * poly);
  }
  if (forced) coefficients(1);
  exact_pairs<0, 3, THERM, SCAL, KEEP>(P, c, forced, tsrc, G, kF, P.w[1], p2, f, g, h);
  if (forced) coefficients(7);
  exact_pairs<3, 9, THERM, SCAL, KEEP>(P, c, forced, tsrc, G, kF, P.w[7], p2, f, g, h);
}

// ---- FP32: BGK and Guo's forcing, f' = (1 - om) f + w (E +- O) for a pair (q, -q), with the
// even part E = r1 + (c.u)(c.b) and the odd part O = c.a:
//   a  = 3 rho (om u + k F),  b = rho (9/2 om u + 9 k F)                  (k = 1 - dt/2tau)
//   r1 = om rho - 3/2 om rho u^2 - 3 k rho u.F
// and for a passive set E = r1 + 9/2 om t (c.u)^2, O = 3 om t (c.u).  The weights are folded
// into the coefficients (1/36; twice that on the straight pairs), so a pair costs 8 (fluid)
// and 5 (passive set) operations.  What the rounded weights would add to a cell's mass and
// momentum every step (1/12 in FP32 is 3e-8 off: 4e-5 of u after 600 steps) is closed: the
// rest population takes r1 less what the other eighteen received, and the straight pairs take
// of O what the diagonal ones leave of the momentum, (m_i - 8 a_i) / 2.  In the deviation form
// (half-precision store) om rho becomes om (rho - shift) and nothing else changes: no shift is
// added or taken off per population.
// Every product that feeds a sum is an explicit fma or a rounded product: all kernels that
// inline this round the same way.
// Warp instructions per 32 cells of Rayleigh-Benard, against 19 separate polynomials: F32
// 1,090 -> 902, F16 1,260 -> 826.  us a step at 256x256x128: F16 360 -> 335, F32 (HBM) 448 ->
// 439; three sets 110x96x100 F32 136 -> 109 (with the flat cell index).
struct Set32 {
  float omf, r1, r1d, kA, kT;  // 1 - om; r1, w r1; w 3 om t, w 9/2 om t (w = 1/36)
};

__device__ __forceinline__ Set32 set32(float om, float sum, float t, float u2, float src) {
  Set32 s;
  const float ot = __fmul_rn(om, t);
  s.omf = 1.0f - om;
  s.r1 = fmaf(__fmul_rn(-1.5f, ot), u2, fmaf(om, sum, src));
  s.r1d = __fmul_rn(s.r1, 1.0f / 36.0f);
  s.kA = __fmul_rn(ot, 3.0f / 36.0f);
  s.kT = __fmul_rn(ot, 4.5f / 36.0f);
  return s;
}

// what the rest direction receives: r1 - 24 w r1 (6 straight directions of 2 w, 12 diagonal of w)
__device__ __forceinline__ float rest32(float omf, float r1, float r1d, float f) {
  return fmaf(omf, f, fmaf(-24.0f, r1d, r1));
}

template <int k>
__device__ __forceinline__ void pair32(const Set32& s, float cu, float q2, float* f) {
  constexpr int q = pair_q(k), b = qinv(q);
  constexpr float m = k < 3 ? 2.0f : 1.0f;  // weight 1/18 on the straight pairs
  const float ev = fmaf(m * s.kT, q2, m * s.r1d);
  f[q] = fmaf(s.omf, f[q], fmaf(m * s.kA, cu, ev));
  f[b] = fmaf(s.omf, f[b], fmaf(-m * s.kA, cu, ev));
}

// c_q . v of pair k, the zero components dropped
template <int k>
__device__ __forceinline__ float pdot32(const float* v) {
  return cdot<pair_q(k)>(v[0], v[1], v[2]);
}

template <int k, bool THERM, bool SCAL>
__device__ __forceinline__ void collide32_pair(const float* u, const float* a, const float* b, float omf, float r1d,
                                               const Set32& tg, const Set32& th, float* f, float* g, float* h) {
  constexpr int q = pair_q(k), qb = qinv(q);
  const float cu = pdot32<k>(u), od = pdot32<k>(a), cb = pdot32<k>(b);
  const float ev = fmaf(cu, cb, r1d);
  f[q] = fmaf(omf, f[q], ev + od);
  f[qb] = fmaf(omf, f[qb], ev - od);
  if constexpr (THERM || SCAL) {
    const float q2 = __fmul_rn(cu, cu);
    if constexpr (THERM) pair32<k>(tg, cu, q2, g);
    if constexpr (SCAL) pair32<k>(th, cu, q2, h);
  }
}

template <bool THERM, bool SCAL>
__device__ __forceinline__ void collide32(const StepParams<float>& P, const CellState<float>& c, bool forcing, float* f,
                                          float* g, float* h) {
  constexpr float w = 1.0f / 36.0f;
  const float u[3] = {c.ux, c.uy, c.uz};
  const float om = c.invtau;
  float r1 = fmaf(__fmul_rn(-1.5f, __fmul_rn(om, c.rho)), c.u2, __fmul_rn(om, c.dr));
  const float r8 = __fmul_rn(0.125f, c.rho);  // 9/2 w rho
  float a[3], as[3], b[3];  // diagonal weight; a also on the straight pairs
  float m[3] = {__fmul_rn(om, u[0]), __fmul_rn(om, u[1]), __fmul_rn(om, u[2])};
#pragma unroll
  for (int i = 0; i < 3; i++) b[i] = __fmul_rn(r8, m[i]);
  if (forcing) {
    const float F[3] = {c.Fx, c.Fy, c.Fz};
    r1 = fmaf(__fmul_rn(-3.0f, __fmul_rn(P.gfac, c.rho)), fmaf(c.uz, c.Fz, fmaf(c.uy, c.Fy, __fmul_rn(c.ux, c.Fx))), r1);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const float kF = __fmul_rn(P.gfac, F[i]);
      m[i] = m[i] + kF;
      b[i] = __fmul_rn(r8, m[i] + kF);
    }
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    m[i] = __fmul_rn(c.rho, m[i]);
    a[i] = __fmul_rn(m[i], 3.0f * w);
    as[i] = fmaf(-4.0f, a[i], 0.5f * m[i]);
  }
  const float omf = 1.0f - om, r1d = __fmul_rn(r1, w);
  const Set32 tg = set32(c.it, c.dt, c.tt, c.u2, c.ts), th = set32(c.is, c.ds, c.ss, c.u2, 0.0f);
  f[0] = rest32(omf, r1, r1d, f[0]);
  if constexpr (THERM) g[0] = rest32(tg.omf, tg.r1, tg.r1d, g[0]);
  if constexpr (SCAL) h[0] = rest32(th.omf, th.r1, th.r1d, h[0]);
  {
    const float b2[3] = {2.0f * b[0], 2.0f * b[1], 2.0f * b[2]}, r2 = 2.0f * r1d;
    collide32_pair<0, THERM, SCAL>(u, as, b2, omf, r2, tg, th, f, g, h);
    collide32_pair<1, THERM, SCAL>(u, as, b2, omf, r2, tg, th, f, g, h);
    collide32_pair<2, THERM, SCAL>(u, as, b2, omf, r2, tg, th, f, g, h);
  }
  collide32_pair<3, THERM, SCAL>(u, a, b, omf, r1d, tg, th, f, g, h);
  collide32_pair<4, THERM, SCAL>(u, a, b, omf, r1d, tg, th, f, g, h);
  collide32_pair<5, THERM, SCAL>(u, a, b, omf, r1d, tg, th, f, g, h);
  collide32_pair<6, THERM, SCAL>(u, a, b, omf, r1d, tg, th, f, g, h);
  collide32_pair<7, THERM, SCAL>(u, a, b, omf, r1d, tg, th, f, g, h);
  collide32_pair<8, THERM, SCAL>(u, a, b, omf, r1d, tg, th, f, g, h);
}

// sum and momentum of one set's loaded values by pairs (sums f_q + f_-q, differences f_q - f_-q)
__device__ __forceinline__ void moments32(const float* f, float& m, float& mx, float& my, float& mz) {
  float s[9], d[9];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    s[k] = f[pair_q(k)] + f[qinv(pair_q(k))];
    d[k] = f[pair_q(k)] - f[qinv(pair_q(k))];
  }
  m = f[0] + (((s[0] + s[1]) + (s[2] + s[3])) + (((s[4] + s[5]) + (s[6] + s[7])) + s[8]));
  // pairs: x, y, z, (x+y), (x-y), (x+z), (-x+z), (y+z), (y-z)
  mx = (d[0] + d[3]) + (d[4] + (d[5] - d[6]));
  my = (d[1] + d[3]) + ((d[7] + d[8]) - d[4]);
  mz = (d[2] + d[5]) + (d[6] + (d[7] - d[8]));
}
__device__ __forceinline__ float sum32(const float* f) {
  float s[9];
#pragma unroll
  for (int k = 0; k < 9; k++) s[k] = f[pair_q(k)] + f[qinv(pair_q(k))];
  return f[0] + (((s[0] + s[1]) + (s[2] + s[3])) + (((s[4] + s[5]) + (s[6] + s[7])) + s[8]));
}

// METHOD_TRT's antisymmetric rate from a rate w (src/fluid.c:1141-1143, magic gamma 1/4)
template <typename A>
__device__ __forceinline__ A trt_minus(A w) {
  return (A(4) - A(2) * w) / (A(2) + (A(4) * A(0.25) - A(1)) * w);
}

// Two-relaxation-time collision of METHOD_TRT (src/fluid.c:1140-1160) of one set, in
// place: per direction the symmetric part (f_q + f_-q)/2 relaxes towards that of the
// equilibrium with wm, the antisymmetric part (f_q - f_-q)/2 with w.  The reference picks
// the rates by which_pop == 'f', a name no set is called with ('p', 'g', 'h'), so every
// set takes this form, as here.  Operations in the reference's order.
template <typename A>
__device__ __forceinline__ void trt_set(A* f, const A* eq, A w, A wm) {
  A out[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const int qb = qinv(q);
    const A fp = A(0.5) * (f[q] + f[qb]), fm = A(0.5) * (f[q] - f[qb]);
    const A ep = A(0.5) * (eq[q] + eq[qb]), em = A(0.5) * (eq[q] - eq[qb]);
    const A fcoll = -wm * (fp - ep) - w * (fm - em);
    out[q] = f[q] + fcoll;
  }
#pragma unroll
  for (int q = 0; q < Q; q++) f[q] = out[q];
}

// METHOD_TRT collision of all enabled sets, then Guo's forcing of the fluid
template <bool EXACT, bool THERM, bool SCAL, typename A>
__device__ __forceinline__ void collide_trt(const StepParams<A>& P, const CellState<A>& c, bool forcing, A wm, A* f,
                                            A* g, A* h) {
  A poly[Q], eq[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const A cu = cdot_rt(q, c.ux, c.uy, c.uz);
    poly[q] = EXACT ? A(1) + P.invcs2 * cu + P.invtwocs4 * cu * cu - P.invtwocs2 * c.u2
                    : c.base + cu * (P.invcs2 + P.invtwocs4 * cu);
    eq[q] = EXACT ? c.rho * P.w[q] * poly[q] : (c.rho * P.w[q]) * poly[q];
  }
  trt_set(f, eq, c.invtau, wm);
  if (forcing) {
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const A cu = cdot_rt(q, c.ux, c.uy, c.uz);
      if constexpr (EXACT) {  // src/forcing.c:1423-1435, three separate additions
        const A dx = guo_d_rt(cx(q), c.ux, cu, P.invcs2, P.invcs4);
        const A dy = guo_d_rt(cy(q), c.uy, cu, P.invcs2, P.invcs4);
        const A dz = guo_d_rt(cz(q), c.uz, cu, P.invcs2, P.invcs4);
        f[q] += P.facw[q] * c.rho * c.Fx * dx;
        f[q] += P.facw[q] * c.rho * c.Fy * dy;
        f[q] += P.facw[q] * c.rho * c.Fz * dz;
      } else {
        const A cF = cdot_rt(q, c.Fx, c.Fy, c.Fz);
        f[q] += (P.facw[q] * c.rho) * ((cF - c.uF) * P.invcs2 + (cu * cF) * P.invcs4);
      }
    }
  }
  if constexpr (THERM) {
#pragma unroll
    for (int q = 0; q < Q; q++) eq[q] = EXACT ? c.tt * P.w[q] * poly[q] : (c.tt * P.w[q]) * poly[q];
    trt_set(g, eq, c.it, (P.feat & K_TLES) ? trt_minus(c.it) : P.invtau_m[1]);
    if (P.feat & K_TSRC)
#pragma unroll
      for (int q = 0; q < Q; q++) g[q] += P.w[q] * c.ts;
  }
  if constexpr (SCAL) {
#pragma unroll
    for (int q = 0; q < Q; q++) eq[q] = EXACT ? c.ss * P.w[q] * poly[q] : (c.ss * P.w[q]) * poly[q];
    trt_set(h, eq, c.is, (P.feat & K_SLES) ? trt_minus(c.is) : P.invtau_m[2]);
  }
}

// The step for one cell (x, y, z) of the lattice described by P.
// Kernel variants (separate instantiations, so that the plain BGK kernels keep their
// registers): bit 0 METHOD_TRT, bit 1 LES (eddy-viscosity relaxation times).
constexpr int V_TRT = 1, V_LES = 2;

template <typename S, typename A, bool THERM, bool SCAL, int V = 0>
__device__ __forceinline__ void lb_cell(const StepParams<A>& P, int x, int y, int z) {
  constexpr bool TRT = (V & V_TRT) != 0, LES = (V & V_LES) != 0;
  constexpr bool EXACT = sizeof(A) == 8;
  const int idx = (z * P.NY + y) * P.NX + x;
  const uint32_t F = P.feat;
  const bool forcing = (F & K_FORCING) != 0;

  // FP32 BGK works on the values as stored (deviations for the half-precision store)
  constexpr bool RAW = !EXACT && !TRT;
  A f[Q], g[Q], h[Q];
  CellState<A> c;
  A mx, my, mz;
  [[maybe_unused]] A ul[4], tl = A(0);
  if constexpr (LES) {
    // u^n is at hand in the vectors the gradients are taken from.  The relaxation time comes
    // before the populations are loaded, so that no population is held through the gradients
    // (the stress form reads its own copy): 48 registers instead of 64 with one set.  Measured
    // at 128^3 FP32, us a step: Kolmogorov LES 115.5 -> 103.7, Rayleigh-Benard LES 185 -> 171.
    ld4(P.ules, idx, ul);
    const A u2 = ul[0] * ul[0] + ul[1] * ul[1] + ul[2] * ul[2];
    A rho = A(1);
    if (F & K_LSTRAIN) {
      load_set<S, A, 0>(P, idx, f);
      rho = mom0(f);
    }
    tl = les_tau<EXACT>(P, x, y, z, idx, f, rho, ul[0], ul[1], ul[2], u2);
    if (P.feat & K_LSTRAIN) P.tau_les[idx] = tl;  // the only reader: the stress form, next step
  }
  constexpr int sets = 1 + (THERM ? 1 : 0) + (SCAL ? 1 : 0);
  const S* p = pop_at<S>(P.fin[0], sets * Q * POP_BLOCK, idx);
  if constexpr (RAW) {
    load_raw(p, f);
    if constexpr (THERM) load_raw(p + Q * POP_BLOCK, g);
    if constexpr (SCAL) load_raw(p + (sets - 1) * Q * POP_BLOCK, h);
    constexpr bool DEV = Codec<S, A>::deviation;
    moments32(f, c.dr, mx, my, mz);
    c.dt = THERM ? sum32(g) : A(0);
    c.ds = SCAL ? sum32(h) : A(0);
    c.rho = DEV ? c.dr + P.shift[0] : c.dr;
    c.tt = DEV && THERM ? c.dt + P.shift[1] : c.dt;
    c.ss = DEV && SCAL ? c.ds + P.shift[2] : c.ds;
  } else {
    load_full(P, 0, p, f);
    if constexpr (THERM) load_full(P, 1, p + Q * POP_BLOCK, g);
    if constexpr (SCAL) load_full(P, 2, p + (sets - 1) * Q * POP_BLOCK, h);
    c.rho = c.dr = mom0(f);
    mx = momx(f), my = momy(f), mz = momz(f);
    c.tt = c.dt = THERM ? mom0(g) : A(0);
    c.ss = c.ds = SCAL ? mom0(h) : A(0);
  }
  c.ts = (THERM && (F & K_TSRC)) ? P.tsrc[idx] : A(0);

  // u^n = mv/rho + dt/2 F^{n-1} (src/lb.c:464-466); F^n for Guo (src/forcing.c:1423-1435)
  A px = A(0), py = A(0), pz = A(0);
  c.Fx = c.Fy = c.Fz = A(0);
  if (forcing) {
    if constexpr (!LES) {
      const A tp = THERM ? P.tprev[idx] : A(0);
      const A sp = SCAL ? P.sprev[idx] : A(0);
      cell_force(P, x, y, z, idx, tp, sp, P.hit_prev, (F & K_TWOWAY) ? P.dprev : nullptr, P.fm_prev, px, py, pz);
    }
    cell_force(P, x, y, z, idx, c.tt, c.ss, P.hit_cur, (F & K_TWOWAY) ? P.dcur : nullptr, P.fm_cur, c.Fx, c.Fy, c.Fz);
  }
  if constexpr (LES) {
    c.ux = ul[0], c.uy = ul[1], c.uz = ul[2];
    c.u2 = EXACT ? c.ux * c.ux + c.uy * c.uy + c.uz * c.uz
                 : A(fmaf(float(c.uz), float(c.uz), fmaf(float(c.uy), float(c.uy), __fmul_rn(float(c.ux), float(c.ux)))));
  } else if constexpr (EXACT) {
    c.ux = mx / c.rho + P.hdt * px;
    c.uy = my / c.rho + P.hdt * py;
    c.uz = mz / c.rho + P.hdt * pz;
    c.u2 = c.ux * c.ux + c.uy * c.uy + c.uz * c.uz;
  } else {
    const A ir = __frcp_rn(c.rho);  // 1 / rho, rounded to nearest
    c.ux = fmaf(P.hdt, px, __fmul_rn(mx, ir));
    c.uy = fmaf(P.hdt, py, __fmul_rn(my, ir));
    c.uz = fmaf(P.hdt, pz, __fmul_rn(mz, ir));
    c.u2 = fmaf(c.uz, c.uz, fmaf(c.uy, c.uy, __fmul_rn(c.ux, c.ux)));
  }
  if constexpr (THERM) P.tprev[idx] = c.tt;
  if constexpr (SCAL) P.sprev[idx] = c.ss;

  c.invtau = P.invtau[0];
  c.it = P.invtau[1];
  c.is = P.invtau[2];
  if constexpr (LES) {
    c.invtau = A(1) / tl;
    // tau_t_les / tau_s_les (src/les.c:273-326, turbulent Prandtl and Schmidt numbers 1)
    if (THERM && (F & K_TLES)) c.it = A(1) / (A(3) * (P.kappa + (tl - A(0.5) - A(3) * P.nu) / (A(3) * A(1))) + A(0.5));
    if (SCAL && (F & K_SLES)) c.is = A(1) / (A(3) * (P.chi + (tl - A(0.5) - A(3) * P.nu) / (A(3) * A(1))) + A(0.5));
  }

  if constexpr (TRT) {
    c.base = A(1) - P.invtwocs2 * c.u2;
    c.uF = c.ux * c.Fx + c.uy * c.Fy + c.uz * c.Fz;
    // the antisymmetric rate from the cell's own rate (LES) or the set's
    const A wm = LES ? trt_minus(c.invtau) : P.invtau_m[0];
    collide_trt<EXACT, THERM, SCAL>(P, c, forcing, wm, f, g, h);
  } else if constexpr (EXACT) {
    collide_exact<THERM, SCAL>(P, c, forcing, f, g, h);
  } else {
    collide32<THERM, SCAL>(P, c, forcing, f, g, h);
  }

  const Nbr nb = neighbours(x, y, z, P.NX, P.NY, P.NZ);
  const uint32_t WL = P.walls;
  const bool toprow = y == P.NY - 1, botrow = y == 0;
  const bool xedge = (WL & (W_FX | W_TX | W_SX)) && (x == 0 || x == P.NX - 1);
  const bool yedge = (F & (K_FWALL | K_TWALL | K_SWALL)) && (toprow || botrow);
  const bool zedge = (WL & (W_FZ | W_TZ | W_SZ)) && (z == 0 || z == P.NZ - 1);
  Walls W{0u, 0u};
  // cells that touch no wall stream every value (periodic y rows too: Kolmogorov 32^3 FP32, where
  // the rows' out-of-line push ended the step, 6.2 -> 4.6 us)
  if (!(xedge || yedge || zedge)) {
    push_bulk<S, A, THERM, SCAL, RAW>(P, idx, nb, f, g, h);
    return;
  }
  // the wall bits of this cell for walls on the axes (x, y, z) of a set
  const uint32_t at = (x == P.NX - 1 ? 1u : 0u) | (toprow ? 2u : 0u) | (z == P.NZ - 1 ? 4u : 0u) |
                      (x == 0 ? 8u : 0u) | (botrow ? 16u : 0u) | (z == 0 ? 32u : 0u);
  auto on = [&](bool wx, bool wy, bool wz) { return at & ((wx ? 9u : 0u) | (wy ? 18u : 0u) | (wz ? 36u : 0u)); };
  A tmp[Q];
  {
    W.hit = on((WL & W_FX) != 0, (F & K_FWALL) != 0, (WL & W_FZ) != 0);
    W.slip = W.hit & (((WL & W_FSLIP_XP) ? 1u : 0u) | ((F & K_FSLIP_P) ? 2u : 0u) | ((WL & W_FSLIP_ZP) ? 4u : 0u) |
                      ((WL & W_FSLIP_XM) ? 8u : 0u) | ((F & K_FSLIP_M) ? 16u : 0u) | ((WL & W_FSLIP_ZM) ? 32u : 0u));
#pragma unroll
    for (int q = 0; q < Q; q++) tmp[q] = f[q];
    push_walled<S, A, 0, RAW>(P, idx, nb, tmp, W.hit ? 1 : 0, W, c.tt, c.ss);
  }
  if constexpr (THERM) {
    W.hit = on((WL & W_TX) != 0, (F & K_TWALL) != 0, (WL & W_TZ) != 0);
#pragma unroll
    for (int q = 0; q < Q; q++) tmp[q] = g[q];
    push_walled<S, A, 1, RAW>(P, idx, nb, tmp, W.hit ? 2 : 0, W, c.tt, c.ss);
  }
  if constexpr (SCAL) {
    W.hit = on((WL & W_SX) != 0, (F & K_SWALL) != 0, (WL & W_SZ) != 0);
#pragma unroll
    for (int q = 0; q < Q; q++) tmp[q] = h[q];
    push_walled<S, A, 2, RAW>(P, idx, nb, tmp, W.hit ? 2 : 0, W, c.tt, c.ss);
  }
}

// One thread per cell, consecutive cells in consecutive threads whatever NX is: with rows cut
// into blocks of 128 a lattice 129 wide left 127 threads of every second block idle, one 32
// wide three quarters of every block.  Two divisions by multiplication replace the block
// coordinates.  Rayleigh-Benard 129x97x75 FP64: 142 -> 112 us a step (with the pairs above).
template <typename S, typename A, bool THERM, bool SCAL, int V>
__device__ __forceinline__ void lb_thread(const StepParams<A>& P) {
  grid_chain();
  const unsigned int i = blockIdx.x * (unsigned)blockDim.x + threadIdx.x;
  if (i >= P.zcells) return;
  const unsigned int k = fast_div(i, P.div_nxy), r = i - k * (unsigned)(P.NX * P.NY);
  const unsigned int y = fast_div(r, P.div_nx);
  lb_cell<S, A, THERM, SCAL, V>(P, (int)(r - y * (unsigned)P.NX), (int)y, P.zfirst + (int)k * P.zstride);
}

template <typename S, typename A, bool THERM, bool SCAL, int V = 0>
__global__ void __launch_bounds__(128) lb_step_kernel(const __grid_constant__ StepParams<A> P) {
  lb_thread<S, A, THERM, SCAL, V>(P);
}

// Resident 128-thread blocks per SM that a form is held to, 0 where the compiler's own choice
// stands (a hint then raises the registers).  The forms run at the HBM roofline or wait for
// it, and lose with fewer warps; at these bounds none spills more than 8 bytes.  us a step:
//   FP64, two sets: 4 (128 registers), 13 % over the 3 that a few registers more leave
//   FP32, fluid only 250^3: 390.3 -> 386.5 at 10 blocks (48 registers); at 8: 409.7
//   FP32, two sets 256x256x128: 414.1 -> 412.1 at 7 blocks (72); at 5: 429.7; F16 301.6 ->
//   296.7; with LES 128^3 156.2 -> 151.7; three sets: 5
template <typename A, bool THERM, bool SCAL, int V>
constexpr int step_blocks() {
  constexpr int sets = 1 + (THERM ? 1 : 0) + (SCAL ? 1 : 0);
  if (V & V_TRT) return 0;
  if (sizeof(A) == 8) return V == 0 && sets == 2 ? 4 : 0;
  return sets == 1 ? (V == 0 ? 10 : 0) : sets == 2 ? 7 : 5;
}
template <typename S, typename A, bool THERM, bool SCAL, int V>
__global__ void __launch_bounds__(128, step_blocks<A, THERM, SCAL, V>()) lb_step_kernel_blocks(
    const __grid_constant__ StepParams<A> P) {
  lb_thread<S, A, THERM, SCAL, V>(P);
}

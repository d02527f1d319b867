// small.cuh -- small walkers (up to 8 electrons, 4 of a spin, one determinant, FP64): moves and E_L with 8
// lanes per walker, 4 walkers to a warp.
//
// A warp per walker leaves most lanes idle on such systems (7 pairs, 2 centres, 4 orbitals, 24
// shells): the 8-electron dimer's DMC step took 102 thousand warp instructions per walker, at a third of
// the issue rate.  With 8 lanes a proposal's shells are 3 to a lane and its pairs one to a lane; an
// evaluation has an electron per lane, a quadrature point per lane.  Orbital values are summed per lane
// over its shells straight into the (at most 4) orbitals and shared by shuffles, so no basis row is
// stored, and the determinant ratio at a quadrature point needs no projection on the basis.  The orbital
// rows of the electrons' positions are kept through the moves: neither the drift at the current
// position nor the evaluation after the moves forms them again.
// Everything is FP64; sums differ in order from the warp-per-walker kernels (full_eval, propose).
// What bounds it: latency between dependent FP64 instructions at 12 warps per SM (168 registers; an issue in
// every 2.5 cycles).  At 128 registers for 14 to 16 warps the spills cost more than the warps give: 8192 walkers
// of the dimer 1.00 -> 1.05 ms per evaluation, DMC step 3.44 -> 4.31 ms.  Two electrons at a time in point_psi
// filled the evaluation's chains (0.91 -> 0.90 ms) but spilled in the DMC step (3.18 -> 3.33 ms).
// A single walker takes longer on 8 lanes than on 32, so few walkers stay with a warp each (small_serves).
// Measured (B200) against a warp per walker: dimer of 8 electrons, order 4, 8192 walkers, evaluation
// 1.04 -> 0.90 ms; DMC step of about the same population 10.0 -> 3.2 ms; C2, order 5, DMC step 1.33 -> 0.69 ms,
// T-moves 1.28 -> 0.82 ms; its accelerated sweep of 8192 walkers 8.0 -> 5.1 ms (k_small_accel, whose sums are those
// of a warp per walker).
#pragma once
#include "jastile.cuh"

namespace sm {

using jt::sfor;

constexpr int GS = 8;  // lanes of a walker
constexpr int NO = 4;  // most electrons (= orbitals) of a spin
constexpr int NE = 8;  // most electrons
constexpr int RCAP = 96;  // radial values of the tasks' centres kept per walker
constexpr int ACH = 24;   // basis functions formed at a time by k_small_accel

// Doubles of a walker in shared memory.
struct Lay {
  int N, C, qm, ext;  // ext: basis functions beside the rows (k_small_accel)
  __host__ __device__ Lay(int N_, int C_, int nord, int ext_ = 0) : N(N_), C(C_), qm(nord > 1 ? nord - 1 : 1), ext(ext_) {}
  __host__ __device__ int ai() const { return 3 * N; }
  __host__ __device__ int f() const { return ai() + 2 * NO * NO; }
  __host__ __device__ int a() const { return f() + N * N; }
  __host__ __device__ int h() const { return a() + N * C; }
  __host__ __device__ int z() const { return h() + N * C; }
  __host__ __device__ int pa() const { return z() + N * qm; }
  __host__ __device__ int ph() const { return pa() + C; }
  __host__ __device__ int pr() const { return ph() + C; }        // proposed row [5][NO]
  __host__ __device__ int pl() const { return pr() + 5 * NO; }   // [C][GS] a point's scaled distances per lane
  __host__ __device__ int row() const { return pl() + C * GS; }  // rows [N][5][NO]; then the tasks
  __host__ __device__ int rlen() const {
    const int t = N * C * NLT + RCAP, r = N * 5 * NO + ext, u = 2 * MAXQ;  // u: a T-move's elements and ratios
    return t > r ? (t > u ? t : u) : (r > u ? r : u);
  }
  // odd, so that the walkers of a warp start in different banks
  __host__ __device__ int total() const { return (row() + rlen()) | 1; }
};

struct Args {
  int nsweep = 1;
  uint64_t seed = 0, sweep0 = 0;
  double step = 0;
  ElRot rot{};
  const int *order = nullptr;  // shells by l, so that the lanes of a round mostly share it
  // accelerated moves: whole shells of up to ACH functions (first shell, shells, first function, functions), and
  // every how many sweeps the inverses are formed anew
  const int4 *chunk = nullptr;
  int nchunk = 0, reinv = 1;
  Mover mv{1, 5.0, 1.0, 1.0};
  DmcPar P{};
  DmcData D{};
  double tau = 0;
  int variant = 0;
  const int *nw = nullptr;
  const long long *step_dev = nullptr;
  int *moved = nullptr;
};

__device__ __forceinline__ unsigned gmask() { return 0xffu << (threadIdx.x & 24); }
__device__ __forceinline__ double gsum(double v, unsigned m) {
  v += __shfl_xor_sync(m, v, 4);
  v += __shfl_xor_sync(m, v, 2);
  v += __shfl_xor_sync(m, v, 1);
  return v;
}

using stab::Rad;

// Adds a shell's functions times the orbital coefficients cf [2l + 1][no] into o.
template <int l, int NCH>
__device__ __forceinline__ void add_shell(const Rad &R, double d0, double d1, double d2, const double *cf, int no, double (&o)[NCH][NO]) {
  double S[9], G[9][3];
  solid_all<double, NCH == 5>(l, d0, d1, d2, S, G);
#pragma unroll
  for (int i = 0; i < 2 * l + 1; i++) {
    const double st = S[i] * R.t;
    const double f0 = S[i] * R.q, f1 = G[i][0] * R.q + st * d0, f2 = G[i][1] * R.q + st * d1, f3 = G[i][2] * R.q + st * d2,
                 f4 = S[i] * R.lap;
#pragma unroll
    for (int k = 0; k < NO; k++) {
      const double c = k < no ? cf[i * no + k] : 0.0;
      o[0][k] += c * f0;
      if constexpr (NCH == 5) {
        o[1][k] += c * f1;
        o[2][k] += c * f2;
        o[3][k] += c * f3;
        o[4][k] += c * f4;
      }
    }
  }
}

// Values (NCH 1) or values, gradients and Laplacians (NCH 5) of the spin's orbitals at a point into
// out[NCH][NO] (shared memory), the walker's lanes over the shells.
template <int NCH>
__device__ __noinline__ void orb_row(const Sys<double> &s, const stab::Tab &T, const int *order, int sp, double x, double y, double z,
                                     double *out) {
  const int sub = threadIdx.x & 7;
  const unsigned m = gmask();
  const int no = s.nocc[sp];
  const double *cf = s.cocc[sp];
  double o[NCH][NO];
#pragma unroll
  for (int c = 0; c < NCH; c++)
#pragma unroll
    for (int k = 0; k < NO; k++) o[c][k] = 0;
  for (int q = sub; q < s.nshell; q += GS) {
    const int ish = order[q];
    const ShellRec h = T.rec[ish];
    const double *cc = s.cent + 3 * h.cen, *cr = cf + (size_t)h.b0 * no;
    const double d0 = x - cc[0], d1 = y - cc[1], d2 = z - cc[2], r2 = d0 * d0 + d1 * d1 + d2 * d2;
    Rad R;
    if (NCH == 1) R = Rad{stab::factor(s, T, ish, h, r2), 0.0, 0.0};
    else if (h.kind == 1) R = stab::gauss_rad(T, h, r2);
    else R = stab::general_rad(s, ish, r2);
    switch (h.l) {
    case 0: add_shell<0, NCH>(R, d0, d1, d2, cr, no, o); break;
    case 1: add_shell<1, NCH>(R, d0, d1, d2, cr, no, o); break;
    case 2: add_shell<2, NCH>(R, d0, d1, d2, cr, no, o); break;
    case 3: add_shell<3, NCH>(R, d0, d1, d2, cr, no, o); break;
    default: add_shell<4, NCH>(R, d0, d1, d2, cr, no, o);
    }
  }
#pragma unroll
  for (int c = 0; c < NCH; c++)
#pragma unroll
    for (int k = 0; k < NO; k++) {
      const double v = gsum(o[c][k], m);
      if (((c * NO + k) & 7) == sub) out[c * NO + k] = v;
    }
  __syncwarp(m);
}

template <int NORD>
struct Tab {
  static constexpr jt::Combos cb = jt::make_combos(NORD);
  static constexpr Terms tl = make_terms(NORD);
};

// e-e-n terms of a pair as a function of its electron e, whose scaled distances are pa and
// ph = -k a^2 / r, with the other's aj and power sums zj: value, d/du and d2/du2, and (LEVEL > 0) the gradient
// over a (w/o the pair's own), its product with d/du along r, and the Laplacian.  The coefficients of
// u^k are summed first; at each centre they make a polynomial in the electron's own a, so that the gradient
// is one factor per centre and nothing is kept per power but the three polynomials.
struct Een {
  double f = 0, w1 = 0, w2 = 0, g0 = 0, g1 = 0, g2 = 0, tt = 0, lp = 0;
};
template <int NORD, int LEVEL>
__device__ __forceinline__ void een_pair(const Sys<double> &s, const JasPar<double> &J, double du, const double *xe, const double *pa,
                                         const double *ph, const double *aj, const double *zj, double r0, double r1, double r2, Een &o) {
  using TB = Tab<NORD>;
  constexpr int NC = jt::make_combos(NORD).n, NT = make_terms(NORD).n, NCA = NC > 0 ? NC : 1, QM = NORD - 1;
  const double sk = J.scalek;
  double u[NORD + 1];
  u[0] = 1;
#pragma unroll
  for (int q = 1; q <= NORD; q++) u[q] = u[q - 1] * du;
  double b0[QM + 1], b1[QM + 1], b2[QM + 1], cu[NCA], ct[NCA], c2[NCA];
#pragma unroll
  for (int q = 0; q <= QM; q++) b0[q] = b1[q] = b2[q] = 0;
  sfor<NT>([&](auto LL) {
    constexpr int ll = decltype(LL)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
    if constexpr (TB::tl.m[ll] == 0) {
      const double c = J.c[0][ll];
      b0[l] += c * u[k];
      if constexpr (LEVEL > 0 && k > 0) b1[l] += (c * k) * u[k - 1];
      if constexpr (LEVEL > 1 && k > 1) b2[l] += (c * (k * (k - 1))) * u[k - 2];
    }
  });
  sfor<NC>([&](auto YY) {
    constexpr int y = decltype(YY)::v, l = TB::cb.l[y], nk = TB::cb.nk[y];
    double x0 = 0, x1 = 0, x2 = 0;
    sfor<nk>([&](auto K) {
      constexpr int k = decltype(K)::v, ik = TB::cb.ll[y][k];
      const double c = l ? J.c[0][ik] : 2 * J.c[0][ik];
      x0 += c * u[k];
      if constexpr (LEVEL > 0 && k > 0) x1 += (c * k) * u[k - 1];
      if constexpr (LEVEL > 1 && k > 1) x2 += (c * (k * (k - 1))) * u[k - 2];
    });
    cu[y] = x0;
    ct[y] = x1;
    c2[y] = x2;
  });
  o.f = 2.0 * s.C * b0[0];
  o.w1 = 2.0 * s.C * b1[0];
  o.w2 = 2.0 * s.C * b2[0];
#pragma unroll
  for (int q = 1; q <= QM; q++) {
    o.f += b0[q] * zj[q - 1];
    if (LEVEL > 0) o.w1 += b1[q] * zj[q - 1];
    if (LEVEL > 1) o.w2 += b2[q] * zj[q - 1];
  }
  for (int c = 0; c < s.C; c++) {
    const double a = pa[c], b = aj[c];
    double bp[QM + 1], P0[QM + 1], P1[QM + 1], P2[QM + 1];
    bp[0] = 1;
#pragma unroll
    for (int q = 1; q <= QM; q++) {
      bp[q] = bp[q - 1] * b;
      P0[q] = b0[q];
      P1[q] = b1[q];
      P2[q] = b2[q];
    }
    sfor<2 * NC>([&](auto Y) {
      constexpr int yv = decltype(Y)::v, y = yv / 2, l = TB::cb.l[y], m = TB::cb.m[y];
      if constexpr (yv % 2 == 0 || l > 0) {
        constexpr int p = yv % 2 ? m : l + m, q = yv % 2 ? l + m : m, nk = TB::cb.nk[y];
        P0[p] += cu[y] * bp[q];
        if constexpr (LEVEL > 0 && nk > 1) P1[p] += ct[y] * bp[q];
        if constexpr (LEVEL > 1 && nk > 2) P2[p] += c2[y] * bp[q];
      }
    });
    // the polynomials without their constant term over a, and derivatives with respect to a
    double p0 = P0[QM], p1 = P1[QM], p2 = P2[QM], d0 = QM * P0[QM], d1 = QM * P1[QM], e0 = QM * (QM - 1) * P0[QM];
#pragma unroll
    for (int q = QM - 1; q >= 1; q--) {
      p0 = p0 * a + P0[q];
      if (LEVEL > 0) {
        p1 = p1 * a + P1[q];
        d0 = d0 * a + q * P0[q];
        d1 = d1 * a + q * P1[q];
      }
      if (LEVEL > 1) {
        p2 = p2 * a + P2[q];
        if (q > 1) e0 = e0 * a + q * (q - 1) * P0[q];
      }
    }
    o.f += a * p0;
    if (LEVEL > 0) {
      o.w1 += a * p1;
      const double h = ph[c], dx = xe[0] - s.cent[3 * c], dy = xe[1] - s.cent[3 * c + 1], dz = xe[2] - s.cent[3 * c + 2];
      const double t = d0 * h;
      o.g0 += t * dx;
      o.g1 += t * dy;
      o.g2 += t * dz;
      if (LEVEL > 1) {
        const double s2 = sk * a;
        o.w2 += a * p2;
        o.tt += d1 * h * (r0 * dx + r1 * dy + r2 * dz);
        o.lp += (e0 * a * (s2 * s2) + 2 * h * d0) * a;
      }
    }
  }
}

// The value alone, centre by centre.
template <int NORD>
struct EenValue {
  using TB = Tab<NORD>;
  static constexpr int NC = jt::make_combos(NORD).n, NT = make_terms(NORD).n, QM = NORD > 1 ? NORD - 1 : 1;
  double b[QM + 1], cu[NC > 0 ? NC : 1], f;
  __device__ __forceinline__ void start(const Sys<double> &s, const JasPar<double> &J, double du, const double *zj) {
    double u[NORD + 1];
    u[0] = 1;
#pragma unroll
    for (int q = 1; q <= NORD; q++) u[q] = u[q - 1] * du;
#pragma unroll
    for (int q = 0; q <= QM; q++) b[q] = 0;
    sfor<NT>([&](auto LL) {
      constexpr int ll = decltype(LL)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
      if constexpr (TB::tl.m[ll] == 0) b[l] += J.c[0][ll] * u[k];
    });
    sfor<NC>([&](auto YY) {
      constexpr int y = decltype(YY)::v, l = TB::cb.l[y], nk = TB::cb.nk[y];
      double x = 0;
      sfor<nk>([&](auto K) {
        constexpr int k = decltype(K)::v, ik = TB::cb.ll[y][k];
        x += (l ? J.c[0][ik] : 2 * J.c[0][ik]) * u[k];
      });
      cu[y] = x;
    });
    f = 2.0 * s.C * b[0];
#pragma unroll
    for (int q = 1; q <= QM; q++) f += b[q] * zj[q - 1];
  }
  __device__ __forceinline__ void add(double a, double r) {
    double rp[QM + 1], P[QM + 1];
    rp[0] = 1;
#pragma unroll
    for (int q = 1; q <= QM; q++) {
      rp[q] = rp[q - 1] * r;
      P[q] = b[q];
    }
    sfor<2 * NC>([&](auto Y) {
      constexpr int yv = decltype(Y)::v, y = yv / 2, l = TB::cb.l[y], m = TB::cb.m[y];
      if constexpr (yv % 2 == 0 || l > 0) {
        constexpr int p = yv % 2 ? m : l + m, q = yv % 2 ? l + m : m;
        P[p] += cu[y] * rp[q];
      }
    });
    double t = P[QM];
#pragma unroll
    for (int q = QM - 1; q >= 1; q--) t = t * a + P[q];
    f += a * t;
  }
};

// e-e and e-e-n terms of electron e (position xe, scaled distances pa, ph = -k a^2 / r) with
// electron j (xj, aj, power sums zj): value, gradient (LEVEL 1) and Laplacian (2) with respect to e.
template <int NORD, int LEVEL>
__device__ __forceinline__ double pair_terms(const Sys<double> &s, const JasPar<double> &J, int e, int j, const double *xe,
                                             const double *pa, const double *ph, const double *xj, const double *aj,
                                             const double *zj, double *g, double &lap, double &rin) {
  const double sk = J.scalek;
  const double r0 = xe[0] - xj[0], r1 = xe[1] - xj[1], r2 = xe[2] - xj[2];
  const double rij = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
  const double du = 1.0 / (1.0 + sk * rij);
  int isb, ipar;
  double ss;
  pair_class(J, s.nup, e, j, isb, ss, ipar);
  double fu = 0, fuu = 0;
  const double f = jas_ee<double, (LEVEL > 0)>(J, isb, ss, ipar, rij, du, fu, fuu);
  rin = LEVEL > 0 ? 1.0 / rij : 0.0;
  Een o;
  if constexpr (NORD > 1) een_pair<NORD, LEVEL>(s, J, du, xe, pa, ph, aj, zj, r0, r1, r2, o);
  if constexpr (LEVEL > 0) {
    const double u1 = -sk * du * du;  // du/dr; u'' + 2 u'/r = -2 k du^3 / r
    const double fr = fu + o.w1 * u1 * rin;
    g[0] = fr * r0 + o.g0;
    g[1] = fr * r1 + o.g1;
    g[2] = fr * r2 + o.g2;
    if constexpr (LEVEL > 1) lap = fuu + 2 * fu + o.w2 * u1 * u1 + 2 * u1 * rin * (o.w1 * du + o.tt) + o.lp;
  }
  return f + o.f;
}

// Jastrow of electron e at xe with the others where they are: its scaled distances (v + pa, ph), this
// lane's pair value pf (lane = other electron; lane e: the e-n term), the sum over all of them minus
// the pair table's row, and with GRAD the gradient.
template <int NORD, bool GRAD>
__device__ __noinline__ void electron_jastrow(const Sys<double> &s, const JasPar<double> &J, double *v, int e, const double *xe,
                                              double &pf, double &dj, double *g) {
  const Lay L(s.N, s.C, NORD);
  const int sub = threadIdx.x & 7, N = s.N, C = s.C;
  const unsigned m = gmask();
  double *pa = v + L.pa(), *ph = v + L.ph();
  const double sk = J.scalek;
  double en = 0, g0 = 0, g1 = 0, g2 = 0;
  for (int c = sub; c < C; c += GS) {
    const double dx = xe[0] - s.cent[3 * c], dy = xe[1] - s.cent[3 * c + 1], dz = xe[2] - s.cent[3 * c + 2];
    const double r = sqrt(dx * dx + dy * dy + dz * dz), a = 1.0 / (1.0 + sk * r);
    double fi = 0, fii = 0;
    en += jas_en<double, GRAD>(J, s.ctype[c], r, a, fi, fii);
    pa[c] = a;
    if (GRAD) {
      ph[c] = -sk * a * a / r;
      g0 += fi * dx;
      g1 += fi * dy;
      g2 += fi * dz;
    }
  }
  __syncwarp(m);
  double d = en, f = 0;
  if (sub < N && sub != e) {
    double gp[3], lap, rin;
    f = pair_terms<NORD, GRAD ? 1 : 0>(s, J, e, sub, xe, pa, ph, v + 3 * sub, v + L.a() + sub * C, v + L.z() + sub * L.qm, gp, lap, rin);
    d += f;
    if (GRAD) {
      g0 += gp[0];
      g1 += gp[1];
      g2 += gp[2];
    }
  }
  if (sub < N) d -= v[L.f() + e * N + sub];
  dj = gsum(d, m);
  en = gsum(en, m);
  pf = sub == e ? en : f;
  if (GRAD) {
    g[0] = gsum(g0, m);
    g[1] = gsum(g1, m);
    g[2] = gsum(g2, m);
  }
}

// Determinant ratio and, with GRAD, gradient of the ratio over it, of electron e with the orbital row
// r [5][NO] (every lane of the walker).
template <bool GRAD>
__device__ __forceinline__ double det_ratio(const Sys<double> &s, const double *v, const Lay &L, int e, const double *r, double *g) {
  const int sp = e < s.nup ? 0 : 1, n = sp ? s.ndn : s.nup, eo = sp ? e - s.nup : e;
  const double *A = v + L.ai() + sp * NO * NO + eo;
  double rho = 0, g0 = 0, g1 = 0, g2 = 0;
#pragma unroll
  for (int k = 0; k < NO; k++)
    if (k < n) {
      const double a = A[k * NO];
      rho += a * r[k];
      if (GRAD) {
        g0 += a * r[NO + k];
        g1 += a * r[2 * NO + k];
        g2 += a * r[3 * NO + k];
      }
    }
  if (GRAD) {
    const double ri = 1.0 / rho;
    g[0] += g0 * ri;
    g[1] += g1 * ri;
    g[2] += g2 * ri;
  }
  return rho;
}

// Accepts electron e at xn: inverse (Sherman-Morrison), pair table, distances, position and row.
template <int NORD>
__device__ __forceinline__ void accept(const Sys<double> &s, double *v, const Lay &L, int e, const double *xn, double pf, double rho,
                                       int nrow) {
  const int sub = threadIdx.x & 7, N = s.N, C = s.C;
  const unsigned m = gmask();
  const int sp = e < s.nup ? 0 : 1, n = sp ? s.ndn : s.nup, eo = sp ? e - s.nup : e;
  double *A = v + L.ai() + sp * NO * NO;
  const double *r = v + L.pr();
  double nv[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int i = sub + GS * h, k = i / NO, j = i & (NO - 1);
    double vb = 0;
#pragma unroll
    for (int q = 0; q < NO; q++)
      if (q < n) vb += r[q] * A[q * NO + j];
    vb -= j == eo ? 1.0 : 0.0;
    nv[h] = A[k * NO + j] - A[k * NO + eo] * vb / rho;
  }
  __syncwarp(m);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int i = sub + GS * h;
    if (i / NO < n && (i & (NO - 1)) < n) A[i] = nv[h];
  }
  if (sub < N) {
    v[L.f() + e * N + sub] = pf;
    v[L.f() + sub * N + e] = pf;
  }
  for (int c = sub; c < C; c += GS) v[L.a() + e * C + c] = v[L.pa() + c];
  if (NORD > 1)
    for (int q = sub; q < L.qm; q += GS) {
      double z = 0;
      for (int c = 0; c < C; c++) {
        double p = 1;
        for (int k = 0; k <= q; k++) p *= v[L.pa() + c];
        z += p;
      }
      v[L.z() + e * L.qm + q] = z;
    }
  if (sub < 3) v[3 * e + sub] = xn[sub];
  for (int i = sub; i < nrow; i += GS) v[L.row() + e * 5 * NO + i] = r[i];
  __syncwarp(m);
}

// Inverses of both spins' Slater matrices from the rows' values: lanes 0-3 the up rows, 4-7 the down
// rows (k_inv_reg's elimination).  Returns ln|D| and sign(D) (0 when singular).
__device__ __forceinline__ void invert(const Sys<double> &s, double *v, const Lay &L, double &lnd, double &sgn) {
  const int sub = threadIdx.x & 7, sp = sub >> 2, r = sub & 3;
  const unsigned m = gmask(), h4 = 0xfu << (threadIdx.x & 28);
  const int n = sp ? s.ndn : s.nup, e = (sp ? s.nup : 0) + r, base = threadIdx.x & 28;
  double a[NO];
#pragma unroll
  for (int j = 0; j < NO; j++) a[j] = (r < n && j < n) ? v[L.row() + e * 5 * NO + j] : 0.0;
  bool used = r >= n, fail = false;
  double piv = 1.0;
  int mycol = 0, pv[NO];
#pragma unroll
  for (int k = 0; k < NO; k++) {
    pv[k] = 0;
    if (k >= n || fail) continue;
    double best = used ? -1.0 : fabs(a[0]);
    if (!(best > -1.0)) best = -1.0;
    int bi = r;
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(h4, best, o);
      const int oi = __shfl_xor_sync(h4, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (!(best > 0.0)) { fail = true; continue; }
    pv[k] = bi;
    if (r == bi) {
      used = true;
      piv = a[0];
      mycol = k;
      const double pi = 1.0 / a[0];
#pragma unroll
      for (int j = 1; j < NO; j++) a[j - 1] = a[j] * pi;
      a[NO - 1] = pi;
    }
    double p[NO];
#pragma unroll
    for (int j = 0; j < NO; j++) p[j] = __shfl_sync(h4, a[j], base + bi);
    if (r != bi) {
      const double f = a[0];
#pragma unroll
      for (int j = 0; j < NO; j++) a[j] = (j + 1 < NO ? a[j + 1] : 0.0) - f * p[j];
    }
  }
  if (fail && r < n)  // a singular matrix stays as it is, as in k_inv_reg
#pragma unroll
    for (int j = 0; j < NO; j++)
      if (j < n) v[L.ai() + sp * NO * NO + r * NO + j] = v[L.row() + e * 5 * NO + j];
  double ln = (r < n && !fail) ? log(fabs(piv)) : 0.0;
  int neg = (r < n && piv < 0) ? 1 : 0;
  if (!fail && r < n) {
#pragma unroll
    for (int j = 0; j < NO; j++) {
      const int mm = j - (NO - n);
      if (mm >= 0) {
        int p = 0;
#pragma unroll
        for (int q = 0; q < NO; q++)
          if (q == mm) p = pv[q];
        v[L.ai() + sp * NO * NO + mycol * NO + p] = a[j];
        if (mm < mycol) neg += p > r;
      }
    }
  }
  const unsigned bad = __ballot_sync(m, fail) & m;
  lnd = gsum(ln, m);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) neg += __shfl_xor_sync(m, neg, o);
  sgn = bad ? 0.0 : ((neg & 1) ? -1.0 : 1.0);
  __syncwarp(m);
}

// psi(electron e at xn) / psi for one lane's own point: determinant ratio times the exponential of the
// Jastrow change.  tab: radial factors of centre tc's shells, or null.
template <int NORD>
__device__ __noinline__ double point_psi(const Sys<double> &s, const stab::Tab &T, const JasPar<double> &J, double *v, int e, const double *xn, int tc,
                                         const double *tab) {
  const Lay L(s.N, s.C, NORD);
  const int sub = threadIdx.x & 7, N = s.N, C = s.C;
  const int sp = e < s.nup ? 0 : 1, n = sp ? s.ndn : s.nup, eo = sp ? e - s.nup : e, no = s.nocc[sp];
  const double *cf = s.cocc[sp];
  double o[NO], g[NO];
#pragma unroll
  for (int k = 0; k < NO; k++) {
    o[k] = 0;
    g[k] = k < n ? v[L.ai() + sp * NO * NO + k * NO + eo] : 0.0;
  }
  const int t0 = tab ? s.cshell0[tc] : 0, t1 = tab ? s.cshell0[tc + 1] : 0;
  double dr = 0, d0 = 0, d1 = 0, d2 = 0, r2 = 0;
  int cen = -1;
  for (int ish = 0; ish < s.nshell; ish++) {
    const ShellRec h = T.rec[ish];
    if (h.cen != cen) {
      cen = h.cen;
      d0 = xn[0] - s.cent[3 * cen];
      d1 = xn[1] - s.cent[3 * cen + 1];
      d2 = xn[2] - s.cent[3 * cen + 2];
      r2 = d0 * d0 + d1 * d1 + d2 * d2;
    }
    double rad;
    if (ish >= t0 && ish < t1) rad = tab[ish - t0];
    else rad = stab::factor(s, T, ish, h, r2);
    double S[9], G[9][3];
    const double *r = cf + (size_t)h.b0 * no;
    auto add = [&](int sl, double val) {
#pragma unroll
      for (int k = 0; k < NO; k++)
        if (k < no) o[k] += val * r[sl * no + k];
    };
    switch (h.l) {
    case 0: add(0, rad); break;
    case 1: add(0, d2 * rad); add(1, d0 * rad); add(2, d1 * rad); break;
    case 2:
      solid_all<double, false>(2, d0, d1, d2, S, G);
#pragma unroll
      for (int i = 0; i < 5; i++) add(i, S[i] * rad);
      break;
    case 3:
      solid_all<double, false>(3, d0, d1, d2, S, G);
#pragma unroll
      for (int i = 0; i < 7; i++) add(i, S[i] * rad);
      break;
    default:
      solid_all<double, false>(4, d0, d1, d2, S, G);
#pragma unroll
      for (int i = 0; i < 9; i++) add(i, S[i] * rad);
    }
  }
#pragma unroll
  for (int k = 0; k < NO; k++) dr += o[k] * g[k];
  double *pl = v + L.pl() + sub;
  double f = 0;
  for (int c = 0; c < C; c++) {
    const double a0 = xn[0] - s.cent[3 * c], a1 = xn[1] - s.cent[3 * c + 1], a2 = xn[2] - s.cent[3 * c + 2];
    const double r = sqrt(a0 * a0 + a1 * a1 + a2 * a2), a = 1.0 / (1.0 + J.scalek * r);
    double fi, fii;
    f += jas_en<double, false>(J, s.ctype[c], r, a, fi, fii);
    pl[c * GS] = a;
  }
  f -= v[L.f() + e * N + e];
  for (int j = 0; j < N; j++) {
    if (j == e) continue;
    const double *xj = v + 3 * j;
    const double r0 = xn[0] - xj[0], r1 = xn[1] - xj[1], q2 = xn[2] - xj[2];
    const double rij = sqrt(r0 * r0 + r1 * r1 + q2 * q2);
    int isb, ipar;
    double ss, du;
    pair_class(J, s.nup, e, j, isb, ss, ipar);
    f += pt::ee_value(J, isb, ss, ipar, rij, du) - v[L.f() + e * N + j];
    if constexpr (NORD > 1) {
      const double *aj = v + L.a() + j * C;
      EenValue<NORD> o;
      o.start(s, J, du, v + L.z() + j * L.qm);
      for (int c = 0; c < C; c++) o.add(pl[c * GS], aj[c]);
      f += o.f;
    }
  }
  return dr * exp(f);
}

// E_L and everything it leaves behind (full_eval) from the rows and positions in shared memory.
struct Res {
  double eloc, v2, lnd, sgn;
};
template <int NORD>
__device__ __forceinline__ Res evaluate(const Sys<double> &s, const stab::Tab &T, const JasPar<double> &J, const EcpPar &E, const State<double> &st,
                                        int w, double *v, const Lay &L, const ElRot &rot, bool anew = true, double lnd = 0,
                                        double sgn = 1) {
  const int sub = threadIdx.x & 7, N = s.N, C = s.C;
  const unsigned m = gmask();
  const double sk = J.scalek;
  if (anew) invert(s, v, L, lnd, sgn);  // else the inverses, ln|D| and sign as the moves left them
  const bool ok = sgn != 0.0 && (anew || isfinite(lnd));
  if (!ok) sgn = 0.0;
  // ---- distances and power sums, lane = electron
  double pe_en = 0, fen = 0, vj[3] = {0, 0, 0}, d2j = 0, pe_ee = 0, fsum = 0;
  const bool act = sub < N;
  const int i = act ? sub : 0;
  const double xi[3] = {v[3 * i], v[3 * i + 1], v[3 * i + 2]};
  double *pa = v + L.a() + i * C, *ph = v + L.h() + i * C;
  if (act) {
    double z[ZQ];
    z[0] = (double)C;
#pragma unroll
    for (int q = 1; q < ZQ; q++) z[q] = 0;
    for (int c = 0; c < C; c++) {
      const double dx = xi[0] - s.cent[3 * c], dy = xi[1] - s.cent[3 * c + 1], dz = xi[2] - s.cent[3 * c + 2];
      const double r = sqrt(dx * dx + dy * dy + dz * dz), a = 1.0 / (1.0 + sk * r);
      double fi, fii;
      fen += jas_en<double, true>(J, s.ctype[c], r, a, fi, fii);
      vj[0] += fi * dx;
      vj[1] += fi * dy;
      vj[2] += fi * dz;
      d2j += fii + 2 * fi;
      pa[c] = a;
      ph[c] = -sk * a * a / r;
      double *ren = st.ren + ((size_t)w * N * C + i * C + c) * 2;
      ren[0] = r;
      ren[1] = a;
      if (s.nloc == 0) pe_en -= s.zc[c] / r;
      double p = a;
#pragma unroll
      for (int q = 1; q < ZQ; q++) { z[q] += p; p *= a; }
    }
    if (NORD > 1)
#pragma unroll
      for (int q = 1; q < (NORD > 1 ? NORD : 2); q++) v[L.z() + i * L.qm + q - 1] = z[q];
    double *zg = st.zq + ((size_t)w * N + i) * ZQ;
#pragma unroll
    for (int q = 0; q < ZQ; q++) zg[q] = z[q];
    v[L.f() + i * N + i] = fen;
    fsum = fen;
  }
  __syncwarp(m);
  double dvd = 0, vx = 0, vy = 0, vz = 0;
  if (act) {
    for (int j = 0; j < N; j++) {
      if (j == i) continue;
      double g[3], lap, rin;
      const double f = pair_terms<NORD, 2>(s, J, i, j, xi, pa, ph, v + 3 * j, v + L.a() + j * C, v + L.z() + j * L.qm, g, lap, rin);
      vj[0] += g[0];
      vj[1] += g[1];
      vj[2] += g[2];
      d2j += lap;
      v[L.f() + i * N + j] = f;
      if (j < i) {
        fsum += f;
        pe_ee += rin;
      }
    }
    const int sp = i < s.nup ? 0 : 1, n = sp ? s.ndn : s.nup, eo = sp ? i - s.nup : i;
    const double *A = v + L.ai() + sp * NO * NO + eo, *r = v + L.row() + i * 5 * NO;
    double g0 = 0, g1 = 0, g2 = 0, lp = 0;
#pragma unroll
    for (int k = 0; k < NO; k++)
      if (k < n) {
        const double a = A[k * NO];
        g0 += a * r[NO + k];
        g1 += a * r[2 * NO + k];
        g2 += a * r[3 * NO + k];
        lp += a * r[4 * NO + k];
      }
    dvd = lp - (g0 * g0 + g1 * g1 + g2 * g2);
    vx = vj[0] + g0;
    vy = vj[1] + g1;
    vz = vj[2] + g2;
  }
  __syncwarp(m);
  const double v2 = gsum(act ? vx * vx + vy * vy + vz * vz : 0.0, m), d2lnd = gsum(dvd, m);
  fsum = gsum(fsum, m);
  d2j = gsum(d2j, m);
  pe_ee = gsum(pe_ee, m);
  pe_en = gsum(pe_en, m);
  // ---- pseudopotential
  double vloc = 0, vnl = 0;
  if (s.nloc > 0 && ok) {
    double *rec = v + L.row(), *tab = rec + N * C * NLT;  // the rows are no longer read
    double R[9];
    if (rot.random) random_rotation(rot.seed, (uint32_t)w, rot.sweep, R);
    else
#pragma unroll
      for (int k = 0; k < 9; k++) R[k] = rot.R[k];
    int ntask = 0;
    for (int base = 0; base < N * C; base += GS) {
      const int j = base + sub;
      bool nl = false;
      double vps[MAXLCH], r = 0;
      int c = 0, e = 0;
      if (j < N * C) {
        c = j / N;
        e = j - c * N;
        const double dx = v[3 * e] - s.cent[3 * c], dy = v[3 * e + 1] - s.cent[3 * c + 1], dz = v[3 * e + 2] - s.cent[3 * c + 2];
        r = sqrt(dx * dx + dy * dy + dz * dz);
        const int it = s.ctype[c];
        ecp_vps(E, it, r, vps);
        vloc += vps[E.lpotp1[it] - 1];
        for (int l = 0; l < E.npotd[it]; l++)
          if (l + 1 != E.lpotp1[it] && fabs(vps[l]) > 1e-4) nl = true;
      }
      const unsigned b = (__ballot_sync(m, nl) >> (threadIdx.x & 24)) & 0xffu;
      if (nl) {
        double *q = rec + (ntask + __popc(b & ((1u << sub) - 1u))) * NLT;
        q[0] = (double)(e * C + c);
        q[1] = r;
        for (int l = 0; l < MAXLCH; l++) q[2 + l] = l < E.npotd[s.ctype[c]] ? vps[l] : 0.0;
      }
      ntask += __popc(b);
    }
    __syncwarp(m);
    const int nsh = (s.nshc > 0 && ntask * s.nshc <= RCAP) ? s.nshc : 0;
    for (int k = sub; k < ntask * nsh; k += GS) {
      const int t = k / nsh, q = k - t * nsh, c = (int)rec[t * NLT] % C, ish = s.cshell0[c] + q;
      if (ish < s.cshell0[c + 1]) tab[k] = stab::factor(s, T, ish, T.rec[ish], rec[t * NLT + 1] * rec[t * NLT + 1]);
    }
    __syncwarp(m);
    const int nq = E.nquad, npts = ntask * nq;
    for (int t = sub; t < npts; t += GS) {
      const int task = t / nq, q = t - task * nq;
      const double *rc = rec + task * NLT;
      const int idx = (int)rc[0], e = idx / C, c = idx - e * C, it = s.ctype[c];
      const double r = rc[1], *q0 = s.quad->q0[q];
      const double qx = R[0] * q0[0] + R[1] * q0[1] + R[2] * q0[2], qy = R[3] * q0[0] + R[4] * q0[1] + R[5] * q0[2],
                   qz = R[6] * q0[0] + R[7] * q0[1] + R[8] * q0[2];
      const double *cc = s.cent + 3 * c;
      const double costh = ((v[3 * e] - cc[0]) * qx + (v[3 * e + 1] - cc[1]) * qy + (v[3 * e + 2] - cc[2]) * qz) / r;
      const double xn[3] = {cc[0] + r * qx, cc[1] + r * qy, cc[2] + r * qz};
      const double ratio = point_psi<NORD>(s, T, J, v, e, xn, c, nsh ? tab + task * nsh : nullptr);
      double vp = 0;
      for (int l = 0; l < E.npotd[it]; l++)
        if (l + 1 != E.lpotp1[it]) vp += rc[2 + l] * yl0(l, costh);
      vnl += s.quad->wq[q] * vp * ratio;
    }
    __syncwarp(m);
    vloc = gsum(vloc, m);
    vnl = gsum(vnl, m);
  }
  const double pe = s.pecent + pe_ee + (s.nloc > 0 ? vloc + vnl : pe_en), d2 = d2lnd + d2j;
  Res res;
  res.v2 = v2;
  res.lnd = ok ? lnd : -INFINITY;
  res.sgn = sgn;
  res.eloc = ok ? pe - HB * (d2 + v2) : nan("");
  if (sub == 0) {
    const double lnpsi = lnd + fsum;
    st.fsum[w] = fsum;
    st.lnd[w] = res.lnd;
    st.sgn[w] = sgn;
    uint32_t flag = 0;
    if (!ok) flag |= CHAMP_WS_SINGULAR;
    if (!isfinite(res.eloc) || !isfinite(lnpsi)) flag |= CHAMP_WS_NONFINITE;
    st.status[w] = flag;
  }
  return res;
}

// What a walker keeps between kernels: positions, inverses and pair table (distances and power sums are
// written by evaluate); for a mixed-precision state the FP32 move tables.
__device__ __forceinline__ void store(const Sys<double> &s, const State<double> &st, int w, const double *v, const Lay &L) {
  const int sub = threadIdx.x & 7, N = s.N, C = s.C;
  __syncwarp(gmask());
  for (int i = sub; i < 3 * N; i += GS) st.x[(size_t)w * 3 * N + i] = v[i];
  for (int sp = 0; sp < 2; sp++) {
    const int n = sp ? s.ndn : s.nup;
    double *A = st.ainv + (size_t)w * st.astride + (sp ? s.nup * s.nup : 0);
    for (int i = sub; i < n * n; i += GS) A[i] = v[L.ai() + sp * NO * NO + (i / n) * NO + i % n];
  }
  if (st.m_fso) {
    const double *rn = st.ren + (size_t)w * N * C * 2, *zz = st.zq + (size_t)w * N * ZQ;
    for (int i = sub; i < N * N; i += GS) st.m_fso[(size_t)w * N * N + i] = (float)v[L.f() + i];
    for (int i = sub; i < N * C * 2; i += GS) st.m_ren[(size_t)w * N * C * 2 + i] = (float)rn[i];
    for (int i = sub; i < N * ZQ; i += GS) st.m_zq[(size_t)w * N * ZQ + i] = (float)zz[i];
    if (st.m_rtd)
      for (int i = sub; i < N * C; i += GS) {
        const int c = i / N, e = i - c * N;
        st.m_rtd[(size_t)w * N * C + i] = (float)rn[2 * (e * C + c) + 1];
      }
  } else {
    for (int i = sub; i < N * N; i += GS) st.fso[(size_t)w * N * N + i] = v[L.f() + i];
  }
}

enum { EVAL = 0, GAUSS = 1, DMC = 7, DMC_EL = 8 };

// EVAL: E_L of the walkers after a sweep; GAUSS: sweeps of Gaussian moves, each followed by E_L; DMC: a
// drift-diffusion step with E_L, reweighting and copy counts (k_dmc_move); DMC_EL: its second half.
template <int NORD, int MODE>
__global__ void __launch_bounds__(128, 3) k_small(const __grid_constant__ Sys<double> s, const __grid_constant__ State<double> st,
                                                  const __grid_constant__ Args A) {
  __shared__ JasPar<double> J;
  __shared__ EcpPar E;
  extern __shared__ __align__(16) char dsm[];
  const stab::Tab T = stab::stage(s, dsm);
  load_params(s, J, E);
  const Lay L(s.N, s.C, NORD);
  const int N = s.N, C = s.C, sub = threadIdx.x & 7, grp = threadIdx.x >> 3;
  const unsigned m = gmask();
  double *v = (double *)(dsm + stab::tab_smem(s.nshell, s.nprim)) + (size_t)grp * L.total();
  constexpr bool dmc = MODE == DMC || MODE == DMC_EL, moves = MODE == GAUSS || MODE == DMC;
  const int W = dmc ? *A.D.nw : st.W;
  const uint64_t step0 = dmc ? (uint64_t)A.D.ctr[0] : A.sweep0;
  const double et = dmc ? *A.D.et : 0, eest = dmc ? *A.D.eest : 0, esigma = dmc ? energy_sigma(A.P, A.D.esg, N) : 0,
               sqt = dmc ? sqrt(A.P.tau) : 0;
  const int w = blockIdx.x * (blockDim.x / GS) + grp;
  double sw = 0, swe = 0;
  if (w < W) {
    for (int i = sub; i < 3 * N; i += GS) v[i] = st.x[(size_t)w * 3 * N + i];
    if (moves) {
      for (int sp = 0; sp < 2; sp++) {
        const int n = sp ? s.ndn : s.nup;
        const double *a = st.ainv + (size_t)w * st.astride + (sp ? s.nup * s.nup : 0);
        for (int i = sub; i < n * n; i += GS) v[L.ai() + sp * NO * NO + (i / n) * NO + i % n] = a[i];
      }
      for (int i = sub; i < N * N; i += GS) v[L.f() + i] = st.fso[(size_t)w * N * N + i];
      for (int i = sub; i < N * C; i += GS) v[L.a() + i] = st.ren[((size_t)w * N * C + i) * 2 + 1];
      for (int i = sub; i < N * L.qm; i += GS) v[L.z() + i] = st.zq[((size_t)w * N + i / L.qm) * ZQ + 1 + i % L.qm];
    }
    __syncwarp(m);
    double es = 0, e2 = 0, acc = 0, el = 0;
    const int nsw = MODE == GAUSS ? A.nsweep : 1;
    for (int isw = 0; isw < nsw; isw++) {
      const uint64_t sweep = step0 + (uint64_t)isw;
      for (int e = 0; e < N; e++)
        orb_row<5>(s, T, A.order, e < s.nup ? 0 : 1, v[3 * e], v[3 * e + 1], v[3 * e + 2], v + L.row() + e * 5 * NO);
      double sdd = 0, spd = 0;
      for (int e = 0; moves && e < N; e++) {
        const int sp = e < s.nup ? 0 : 1;
        const double xo[3] = {v[3 * e], v[3 * e + 1], v[3 * e + 2]};
        double *pr = v + L.pr();
        double pf, d0, go[3], gn[3], dj, rho, p, ua, xn[3];
        if constexpr (MODE == GAUSS) {
          double g[3];
          move_randoms(A.seed, (uint32_t)w, sweep, (uint32_t)e, g, &ua);
          for (int k = 0; k < 3; k++) xn[k] = xo[k] + A.step * g[k];
          orb_row<5>(s, T, A.order, sp, xn[0], xn[1], xn[2], pr);
          electron_jastrow<NORD, false>(s, J, v, e, xn, pf, dj, gn);
          rho = det_ratio<false>(s, v, L, e, pr, gn);
          p = rho * rho * exp(2.0 * dj);
        } else {
          electron_jastrow<NORD, true>(s, J, v, e, xo, pf, d0, go);
          det_ratio<true>(s, v, L, e, v + L.row() + e * 5 * NO, go);
          double vo[3], vn[3], g[3], db[3];
          avg_drift(go, A.P.tau, A.P.adrift, vo);
          move_randoms(A.P.seed, (uint32_t)w, sweep, (uint32_t)e, g, &ua);
          for (int k = 0; k < 3; k++) xn[k] = xo[k] + A.P.tau * vo[k] + sqt * g[k];
          orb_row<5>(s, T, A.order, sp, xn[0], xn[1], xn[2], pr);
          electron_jastrow<NORD, true>(s, J, v, e, xn, pf, dj, gn);
          rho = det_ratio<true>(s, v, L, e, pr, gn);
          avg_drift(gn, A.P.tau, A.P.adrift, vn);
          const double lgf = -0.5 * (g[0] * g[0] + g[1] * g[1] + g[2] * g[2]);
          for (int k = 0; k < 3; k++) db[k] = xo[k] - xn[k] - A.P.tau * vn[k];
          const double lgb = -(db[0] * db[0] + db[1] * db[1] + db[2] * db[2]) / (2 * A.P.tau);
          p = (rho > 0) ? rho * rho * exp(2.0 * dj + lgb - lgf) : 0.0;  // fixed node
          const double dd = A.P.tau * (g[0] * g[0] + g[1] * g[1] + g[2] * g[2]);
          sdd += dd;
          spd += (p < 1.0 ? p : 1.0) * dd;
        }
        if (ua < p) {
          accept<NORD>(s, v, L, e, xn, pf, rho, 5 * NO);
          acc += 1;
        }
        __syncwarp(m);
      }
      ElRot rot = A.rot;  // EVAL: the sweep's
      if (MODE != EVAL) {
        rot.random = 1;
        rot.seed = dmc ? A.P.seed : A.seed;
        rot.sweep = sweep;
      }
      const Res res = evaluate<NORD>(s, T, J, E, st, w, v, L, rot);
      el = res.eloc;
      es += el;
      e2 += el * el;
      if (dmc && sub == 0) {
        const double teff = MODE == DMC ? (sdd > 0 ? A.P.tau * spd / sdd : A.P.tau) : A.D.teff[w];
        const double eint = integrated_energy(A.P, A.D.el[w], A.D.v2[w], el, res.v2, N, eest, et, esigma, teff);
        double wn = A.D.wt[w] * exp(-eint * teff);
        if (!isfinite(wn) || !isfinite(el)) wn = 0.0;  // a walker with a non-finite energy dies
        A.D.wt[w] = wn;
        A.D.el[w] = el;
        A.D.v2[w] = res.v2;
        A.D.ncopy[w] = copy_count(A.P, wn, w, sweep);
        sw = wn;
        if (wn > 0) swe = wn * el;
      }
    }
    store(s, st, w, v, L);
    if (!dmc && sub == 0) {
      st.s_esum[w] += es;
      st.s_e2sum[w] += e2;
      st.s_acc[w] += acc;
      st.s_elast[w] = el;
    }
  }
  if (dmc) {
    __syncwarp();
    sw = warp_sum(sw);
    swe = warp_sum(swe);
    if ((threadIdx.x & 31) == 0 && sw != 0) {
      atomicAdd(&A.D.red[0], sw);
      atomicAdd(&A.D.red[1], swe);
    }
    for (int i = W + blockIdx.x * blockDim.x + (int)threadIdx.x; i < A.P.wmax; i += gridDim.x * blockDim.x) A.D.ncopy[i] = 0;
  }
}

// ---- accelerated Metropolis moves (metrop_slat_mov1.f90:82-546).  A proposal follows the drift, and each move
// changes the next electron's drift: a walk magnifies the last bit of whatever it is formed from, 1e-16 to 6e-3 bohr
// within four sweeps for the worst of 8192 walkers of the dimer.  So everything a proposal depends on is formed
// here by the operations, in the order, of a warp per walker (propose, accept_move, k_vmc): basis functions
// and their interleaved sums, the drift and its sums over lanes, the inverse's updates and when it is formed anew.
// With Gaussian shells up to d the walks are the same to the bit; with others (shell_eval_put as compiled here) to
// rounding, which their examples magnify little: positions of C2 3e-10 bohr after 15 sweeps, of Be 1e-12.
// k_small's cheaper sums took 2.6 ms for a sweep of 8192 walkers of C2, a warp per walker takes 8.0, this 5.1.

// A Gaussian shell with n = l + 1, l <= 2, [slot][channel]: the operations of shell_eval_put with those products
// fused with their sums that the compiler fuses in k_vmc.
template <int l>
__device__ __forceinline__ void gauss_shell5(const Sys<double> &s, int2 pr, double d0, double d1, double d2, double *o) {
  double r = sqrt(__fma_rn(d2, d2, __fma_rn(d0, d0, __dmul_rn(d1, d1))));
  if (r == 0.0) { r = 1e-30; d0 = r; }
  const double ri = 1.0 / r, rm1 = l == 0 ? 1.0 : l == 1 ? r : __dmul_rn(r, r), rm2 = __dmul_rn(rm1, ri), rm3 = __dmul_rn(rm2, ri);
  double R0 = 0, R1 = 0, R2 = 0;
#pragma unroll 2
  for (int p = pr.x; p < pr.x + pr.y; p++) {
    const double zr = __dmul_rn(__dmul_rn(2 * s.pz[p], r), r), ex = __dmul_rn(s.pc[p], exp(-0.5 * zr));
    R0 = __fma_rn(rm1, ex, R0);
    R1 = __dadd_rn(R1, __dmul_rn(__dmul_rn(rm2, __dadd_rn(l, -zr)), ex));
    R2 = __dadd_rn(R2, __dmul_rn(__dmul_rn(rm3, __dadd_rn(l * (l - 1), -__dmul_rn(__dadd_rn(2 * l + 1, -zr), zr))), ex));
  }
  const double ril = l == 0 ? 1.0 : l == 1 ? ri : __dmul_rn(ri, ri), d[3] = {d0, d1, d2};
  const double lap = __fma_rn(-__dmul_rn(__dmul_rn(l * (l + 1), ri), ri), R0, __fma_rn(2 * ri, R1, R2));
  // function S, its gradient G (zero where Z says so)
  auto put = [&](int sl, double S, const double *G, const int *Z) {
    const double Y = __dmul_rn(S, ril), lr = __dmul_rn(__dmul_rn(__dmul_rn(l * S, ril), ri), ri);
    o[sl * 5] = __dmul_rn(Y, R0);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double a = __dmul_rn(__dmul_rn(Y, d[k]), ri);
      double v = __dmul_rn(a, R1);
      if (l > 0) {
        const double q = -__dmul_rn(lr, d[k]);
        v = __fma_rn(a, R1, __dmul_rn(Z[k] ? __fma_rn(G[k], ril, q) : q, R0));
      }
      o[sl * 5 + k + 1] = v;
    }
    o[sl * 5 + 4] = __dmul_rn(Y, lap);
  };
  if constexpr (l == 0) {
    put(0, 1.0, nullptr, nullptr);
  } else if constexpr (l == 1) {
    const double G[3] = {1.0, 1.0, 1.0};
    const int Z[3][3] = {{0, 0, 1}, {1, 0, 0}, {0, 1, 0}};
    put(0, d2, G, Z[0]);
    put(1, d0, G, Z[1]);
    put(2, d1, G, Z[2]);
  } else {
    const double s3 = 1.7320508075688772, x2 = __dmul_rn(d0, d0);
    const double sx = __dmul_rn(s3, d0), sy = __dmul_rn(s3, d1), sz = __dmul_rn(s3, d2);
    const double G[5][3] = {{-d0, -d1, 2 * d2}, {sz, 0.0, sx}, {0.0, sz, sy}, {sx, -sy, 0.0}, {sy, sx, 0.0}};
    const int Z[5][3] = {{1, 1, 1}, {1, 0, 1}, {0, 1, 1}, {1, 1, 0}, {1, 1, 0}};
    put(0, 0.5 * __dadd_rn(2 * __dmul_rn(d2, d2), -__fma_rn(d1, d1, x2)), G[0], Z[0]);
    put(1, __dmul_rn(sx, d2), G[1], Z[1]);
    put(2, __dmul_rn(sy, d2), G[2], Z[2]);
    put(3, __dmul_rn(0.5 * s3, __fma_rn(-d1, d1, x2)), G[3], Z[3]);
    put(4, __dmul_rn(sx, d1), G[4], Z[4]);
  }
}
static __device__ __noinline__ void general_shell5(const Sys<double> &s, int ish, double x, double y, double z, double *o) {
  const double pt[3] = {x, y, z};
  shell_eval_put<double, 5>(s, ish, pt, [o](int sl, int c, double v) { o[sl * 5 + c] = v; });
}

// The orbital row at a point into out [5][NO]: warp_orbitals' sums of up to LM orbitals, 32 / LM interleaved ones
// per orbital -- G = 4 / LM of them in each lane -- and their tree.  phi: ACH basis functions.
template <int LM>
__device__ __noinline__ void accel_row(const Sys<double> &s, const int4 *chunk, int nchunk, int sp, double x, double y, double z, double *phi,
                                       double *out) {
  constexpr int G = 4 / LM;
  const int sub = threadIdx.x & 7, no = s.nocc[sp];
  const unsigned m = gmask();
  const double *cf = s.cocc[sp];
  double o[5][4];
#pragma unroll
  for (int c = 0; c < 5; c++)
#pragma unroll
    for (int k = 0; k < 4; k++) o[c][k] = 0;
  for (int q = 0; q < nchunk; q++) {
    const int4 ch = chunk[q];
    for (int h = sub; h < ch.y; h += GS) {
      const int ish = ch.x + h;
      const int4 sh = s.shell[ish];
      double *f = phi + (s.shb0[ish] - ch.z) * 5;
      if (sh.w != 1 || sh.y != sh.z + 1 || sh.z > 2) {
        general_shell5(s, ish, x, y, z, f);
        continue;
      }
      const int2 pr = s.shprim[ish];
      const double *cc = s.cent + 3 * sh.x;
      if (sh.z == 0) gauss_shell5<0>(s, pr, x - cc[0], y - cc[1], z - cc[2], f);
      else if (sh.z == 1) gauss_shell5<1>(s, pr, x - cc[0], y - cc[1], z - cc[2], f);
      else gauss_shell5<2>(s, pr, x - cc[0], y - cc[1], z - cc[2], f);
    }
    __syncwarp(m);
    for (int b = ch.z + ((sub - ch.z) & 7); b < ch.z + ch.w; b += GS) {
      const double *p = phi + (b - ch.z) * 5;
#pragma unroll
      for (int g = 0; g < G; g++)
        if (((b >> 3) & (G - 1)) == g)
#pragma unroll
          for (int k = 0; k < LM; k++)
            if (k < no) {
              const double c = cf[(size_t)b * no + k];
#pragma unroll
              for (int i = 0; i < 5; i++) o[i][g * LM + k] += c * p[i];
            }
    }
    __syncwarp(m);
  }
#pragma unroll
  for (int c = 0; c < 5; c++) {
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int d = 1; d < 8; d <<= 1) o[c][k] += __shfl_xor_sync(m, o[c][k], d);
#pragma unroll
    for (int d = 1; d < G; d <<= 1)
#pragma unroll
      for (int g = 0; g < G; g += 2 * d)
#pragma unroll
        for (int k = 0; k < LM; k++) o[c][g * LM + k] += o[c][(g + d) * LM + k];
#pragma unroll
    for (int k = 0; k < NO; k++)
      if (((c * NO + k) & 7) == sub) out[c * NO + k] = k < LM ? o[c][k < LM ? k : 0] : 0.0;
  }
  __syncwarp(m);
}
__device__ __forceinline__ void accel_orbitals(const Sys<double> &s, const Args &A, int e, const double *x, double *phi, double *out) {
  const int sp = e < s.nup ? 0 : 1, no = s.nocc[sp];
  if (no > 2) accel_row<4>(s, A.chunk, A.nchunk, sp, x[0], x[1], x[2], phi, out);
  else if (no > 1) accel_row<2>(s, A.chunk, A.nchunk, sp, x[0], x[1], x[2], phi, out);
  else accel_row<1>(s, A.chunk, A.nchunk, sp, x[0], x[1], x[2], phi, out);
}

// propose() of electron e at xn with the orbital row r: determinant ratio, Jastrow change and drift; this lane's
// pair value in pf (lane e: the e-n term).  Distances: ren [N][C][2] in the place of a and h, rnew [C][2] of pa and ph.
template <int NORD>
__device__ __noinline__ void accel_propose(const Sys<double> &s, const JasPar<double> &J, double *v, int e, const double *xn, const double *r,
                                           double &rho, double &dj, double &pf, double *grad) {
  const Lay L(s.N, s.C, NORD);
  const int sub = threadIdx.x & 7, N = s.N, C = s.C;
  const unsigned m = gmask();
  double *rnew = v + L.pa();
  const double *ren = v + L.a(), *fso = v + L.f();
  for (int c = sub; c < C; c += GS) {
    double q, d;
    cen_dist(s, J.scalek, xn, c, q, d);
    rnew[2 * c] = q;
    rnew[2 * c + 1] = d;
  }
  __syncwarp(m);
  const int sp = e < s.nup ? 0 : 1, n = sp ? s.ndn : s.nup, eo = sp ? e - s.nup : e;
  const double *Ai = v + L.ai() + sp * NO * NO + eo;
  double t[4];  // lanes k = 0 .. 3 of the warp's sums, which add k and k + 2 first
#pragma unroll
  for (int c = 0; c < 4; c++) {
    double q[NO];
#pragma unroll
    for (int k = 0; k < NO; k++) q[k] = k < n ? __dmul_rn(Ai[k * NO], r[c * NO + k]) : 0.0;
    t[c] = (q[0] + q[2]) + (q[1] + q[3]);
  }
  rho = t[0];
  double d = 0, g[4][3], fen[4];  // of this lane and those 8, 16 and 24 above it
#pragma unroll
  for (int i = 0; i < 4; i++) fen[i] = g[i][0] = g[i][1] = g[i][2] = 0;
  double f = 0;
  if (sub < N && sub != e) {
    f = pair_value<double, NORD, true>(s, J, e, sub, xn, rnew, v + 3 * sub, ren + 2 * C * sub, g[0]);
    d = f - fso[e * N + sub];
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
    for (int c = sub + 8 * i; c < C; c += 32) {
      double fi = 0, fii = 0;
      fen[i] += jas_en<double, true>(J, s.ctype[c], rnew[2 * c], rnew[2 * c + 1], fi, fii);
      const double *cc = s.cent + 3 * c;
      g[i][0] += fi * (xn[0] - cc[0]);
      g[i][1] += fi * (xn[1] - cc[1]);
      g[i][2] += fi * (xn[2] - cc[2]);
    }
  const double fent = gsum((fen[0] + fen[2]) + (fen[1] + fen[3]), m);
  if (sub == 0) d += fent - fso[e * N + e];
  dj = gsum(d, m);
  pf = sub == e ? fent : f;
#pragma unroll
  for (int k = 0; k < 3; k++) grad[k] = gsum((g[0][k] + g[2][k]) + (g[1][k] + g[3][k]), m) + t[1 + k] / rho;
}

// accept_move() of electron e at xn.
__device__ __forceinline__ void accel_accept(const Sys<double> &s, double *v, const Lay &L, int e, const double *xn, double pf) {
  const int sub = threadIdx.x & 7, N = s.N, C = s.C;
  const unsigned m = gmask();
  const int sp = e < s.nup ? 0 : 1, n = sp ? s.ndn : s.nup, eo = sp ? e - s.nup : e;
  double *A = v + L.ai() + sp * NO * NO;
  const double *r = v + L.pr();
  auto vb = [&](int j) {
    double a = 0;
#pragma unroll
    for (int k = 0; k < NO; k++)
      if (k < n) a += r[k] * A[k * NO + j];
    return a - (j == eo ? 1.0 : 0.0);
  };
  const double rinv = 1.0 / (vb(eo) + 1.0);
  double nv[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int i = sub + GS * h, k = i / NO, j = i & (NO - 1);
    nv[h] = A[i] - A[k * NO + eo] * vb(j) * rinv;
  }
  __syncwarp(m);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int i = sub + GS * h;
    if (i / NO < n && (i & (NO - 1)) < n) A[i] = nv[h];
  }
  if (sub < N) {
    v[L.f() + e * N + sub] = pf;
    v[L.f() + sub * N + e] = pf;
  }
  for (int i = sub; i < 2 * C; i += GS) v[L.a() + 2 * C * e + i] = v[L.pa() + i];
  if (sub < 3) v[3 * e + sub] = xn[sub];
  for (int i = sub; i < 5 * NO; i += GS) v[L.row() + e * 5 * NO + i] = r[i];
  __syncwarp(m);
}

template <int NORD>
__global__ void __launch_bounds__(128, 3) k_small_accel(const __grid_constant__ Sys<double> s, const __grid_constant__ State<double> st,
                                                        const __grid_constant__ Args A) {
  __shared__ JasPar<double> J;
  __shared__ EcpPar E;
  extern __shared__ __align__(16) char dsm[];
  const stab::Tab T = stab::stage(s, dsm);
  load_params(s, J, E);
  const Lay L(s.N, s.C, NORD, 5 * ACH);
  const int N = s.N, C = s.C, sub = threadIdx.x & 7, grp = threadIdx.x >> 3;
  const unsigned m = gmask();
  double *v = (double *)(dsm + stab::tab_smem(s.nshell, s.nprim)) + (size_t)grp * L.total();
  double *phi = v + L.row() + N * 5 * NO, *pr = v + L.pr();
  const int w = blockIdx.x * (blockDim.x / GS) + grp;
  if (w >= st.W) return;
  for (int i = sub; i < 3 * N; i += GS) v[i] = st.x[(size_t)w * 3 * N + i];
  for (int sp = 0; sp < 2; sp++) {
    const int n = sp ? s.ndn : s.nup;
    const double *a = st.ainv + (size_t)w * st.astride + (sp ? s.nup * s.nup : 0);
    for (int i = sub; i < n * n; i += GS) v[L.ai() + sp * NO * NO + (i / n) * NO + i % n] = a[i];
  }
  for (int i = sub; i < N * N; i += GS) v[L.f() + i] = st.fso[(size_t)w * N * N + i];
  double lnd = st.lnd[w], sgn = st.sgn[w], es = 0, e2 = 0, acc = 0, el = 0;
  __syncwarp(m);
  for (int isw = 0; isw < A.nsweep; isw++) {
    const uint64_t sweep = A.sweep0 + (uint64_t)isw;
    for (int i = sub; i < N * C; i += GS) cen_dist(s, J.scalek, v + 3 * (i / C), i % C, v[L.a() + 2 * i], v[L.a() + 2 * i + 1]);
    for (int e = 0; e < N; e++) accel_orbitals(s, A, e, v + 3 * e, phi, v + L.row() + e * 5 * NO);
    for (int e = 0; e < N; e++) {
      const double xo[3] = {v[3 * e], v[3 * e + 1], v[3 * e + 2]};
      double rho, dj, pf, go[3], gn[3], xn[3], fxop, areao, rtry, p = 0;
      accel_propose<NORD>(s, J, v, e, xo, v + L.row() + e * 5 * NO, rho, dj, pf, go);
      MoveRng rng{A.seed, (uint32_t)w, (uint32_t)sweep, (uint32_t)(sweep >> 32), (uint32_t)e, 0u, {0.0, 0.0}, 0};
      slat_forward(s, A.mv, xo, go, rng, xn, fxop, areao, rtry);
      SlatBack b;
      if (slat_geometry(s, A.mv, xo, xn, b)) {
        double fxnp, arean;
        __syncwarp(m);
        accel_orbitals(s, A, e, xn, phi, pr);
        accel_propose<NORD>(s, J, v, e, xn, pr, rho, dj, pf, gn);
        slat_reverse(s, A.mv, b, gn, fxnp, arean);
        const double rr = rtry / b.rminon;
        p = rr * rr * rho * rho * exp(2.0 * dj) * fabs((fxnp * areao) / (fxop * arean));
      }
      if (rng.next() < p) {
        accel_accept(s, v, L, e, xn, pf);
        lnd += log(fabs(rho));
        if (rho < 0) sgn = -sgn;
        acc += 1;
      }
      __syncwarp(m);
    }
    ElRot rot{};
    rot.random = 1;
    rot.seed = A.seed;
    rot.sweep = sweep;
    const bool anew = A.reinv <= 1 || sweep % (uint64_t)A.reinv == 0;
    const Res res = evaluate<NORD>(s, T, J, E, st, w, v, L, rot, anew, lnd, sgn);
    lnd = res.lnd;
    sgn = res.sgn;
    el = res.eloc;
    es += el;
    e2 += el * el;
    __syncwarp(m);
  }
  store(s, st, w, v, L);
  if (sub == 0) {
    st.s_esum[w] += es;
    st.s_e2sum[w] += e2;
    st.s_acc[w] += acc;
    st.s_elast[w] = el;
  }
}

// T-moves of every electron (tmove_electron): a quadrature point per lane for the ratios, the heat-bath
// choice in order by every lane.
template <int NORD>
__device__ __forceinline__ int tmove(const Sys<double> &s, const stab::Tab &T, const JasPar<double> &J, const EcpPar &E, const State<double> &st, double *v,
                                     const Lay &L, int w, int e, const Args &A, uint64_t step, double *gp) {
  const int sub = threadIdx.x & 7, nq = E.nquad, C = s.C;
  const unsigned m = gmask();
  MoveRng rng{A.seed, (uint32_t)w, (uint32_t)step, (uint32_t)(step >> 32), 256u + (uint32_t)e, 0u, {0.0, 0.0}, 0};
  double R[9];
  rotation_from(rng, R);
  const double xo[3] = {v[3 * e], v[3 * e + 1], v[3 * e + 2]};
  auto point = [&](const double *Rm, const double *cc, double r, int q, double *qv, double *xq) {
    const double *q0 = s.quad->q0[q];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      qv[k] = Rm[3 * k] * q0[0] + Rm[3 * k + 1] * q0[1] + Rm[3 * k + 2] * q0[2];
      xq[k] = cc[k] + r * qv[k];
    }
  };
  // T elements to the points of centre c about position rv + c, with this lane's points into gp
  auto elements = [&](const double *Rm, int c, const double *rv, double r, const double *vps, double div, double *rat) {
    const int it = s.ctype[c];
    for (int q = sub; q < nq; q += GS) {
      double qv[3], xq[3];
      point(Rm, s.cent + 3 * c, r, q, qv, xq);
      const double costh = (rv[0] * qv[0] + rv[1] * qv[1] + rv[2] * qv[2]) / r;
      const double psi = point_psi<NORD>(s, T, J, v, e, xq, c, nullptr), ratio = psi / div;
      double t = 0;
      for (int l = 0; l < E.npotd[it]; l++)
        if (l + 1 != E.lpotp1[it]) t += s.quad->wq[q] * (exp(-A.tau * vps[l]) - 1) * yl0(l, costh) * ratio;
      gp[q] = t;
      if (rat) rat[q] = psi;
    }
    __syncwarp(m);
  };
  double *rat = gp + MAXQ;
  double S = 1.0, pratio = 0.0;
  int pc = -1, pq = -1;
  for (int c = 0; c < C; c++) {
    const double *cc = s.cent + 3 * c;
    const double rv[3] = {xo[0] - cc[0], xo[1] - cc[1], xo[2] - cc[2]};
    const double r = sqrt(rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2]);
    const int it = s.ctype[c];
    double vps[MAXLCH];
    ecp_vps(E, it, r, vps);
    bool skip = true;
    for (int l = 0; l < E.npotd[it]; l++)
      if (l + 1 != E.lpotp1[it] && fabs(vps[l]) > 1e-4) skip = false;
    if (skip) continue;
    elements(R, c, rv, r, vps, 1.0, rat);
    for (int q = 0; q < nq; q++)
      if (gp[q] > 0) {
        S += gp[q];
        if (rng.next() < gp[q] / S) { pc = c; pq = q; pratio = rat[q]; }
      }
    __syncwarp(m);
  }
  if (pc < 0) return 0;
  const double *cc = s.cent + 3 * pc;
  const double r = sqrt((xo[0] - cc[0]) * (xo[0] - cc[0]) + (xo[1] - cc[1]) * (xo[1] - cc[1]) + (xo[2] - cc[2]) * (xo[2] - cc[2]));
  double qn[3], xn[3];
  point(R, cc, r, pq, qn, xn);
  double p = 1.0;
  if (A.variant == 2) {
    double vps[MAXLCH], R2[9];
    ecp_vps(E, s.ctype[pc], r, vps);
    rotation_from(rng, R2);
    const double xe[3] = {xn[0] - cc[0], xn[1] - cc[1], xn[2] - cc[2]};
    elements(R2, pc, xe, r, vps, pratio, nullptr);
    double Sb = 1.0;
    for (int q = 0; q < nq; q++)
      if (gp[q] > 0) Sb += gp[q];
    p = S / Sb < 1.0 ? S / Sb : 1.0;
    __syncwarp(m);
  }
  if (rng.next() >= p) return 0;
  double pf, dj, g[3];
  orb_row<1>(s, T, A.order, e < s.nup ? 0 : 1, xn[0], xn[1], xn[2], v + L.pr());
  electron_jastrow<NORD, false>(s, J, v, e, xn, pf, dj, g);
  const double rho = det_ratio<false>(s, v, L, e, v + L.pr(), g);
  accept<NORD>(s, v, L, e, xn, pf, rho, 0);
  if (sub == 0) {
    st.fsum[w] += dj;
    st.lnd[w] += log(fabs(rho));
    if (rho < 0) st.sgn[w] = -st.sgn[w];
  }
  return 1;
}

// What a T-move pass leaves besides the positions: log-determinant, sign and Jastrow sum as updated by
// the accepted moves, pair table, distances and power sums.
template <int NORD>
__global__ void __launch_bounds__(128, 3) k_small_tmove(const __grid_constant__ Sys<double> s, const __grid_constant__ State<double> st,
                                                        const __grid_constant__ Args A) {
  __shared__ JasPar<double> J;
  __shared__ EcpPar E;
  extern __shared__ __align__(16) char dsm[];
  const stab::Tab T = stab::stage(s, dsm);
  load_params(s, J, E);
  const Lay L(s.N, s.C, NORD);
  const int N = s.N, C = s.C, sub = threadIdx.x & 7, grp = threadIdx.x >> 3;
  const unsigned m = gmask();
  double *v = (double *)(dsm + stab::tab_smem(s.nshell, s.nprim)) + (size_t)grp * L.total();
  const int W = A.nw ? *A.nw : st.W, w = blockIdx.x * (blockDim.x / GS) + grp;
  const uint64_t step = A.step_dev ? (uint64_t)A.step_dev[0] : A.sweep0;
  if (w >= W) return;
  for (int i = sub; i < 3 * N; i += GS) v[i] = st.x[(size_t)w * 3 * N + i];
  for (int sp = 0; sp < 2; sp++) {
    const int n = sp ? s.ndn : s.nup;
    const double *a = st.ainv + (size_t)w * st.astride + (sp ? s.nup * s.nup : 0);
    for (int i = sub; i < n * n; i += GS) v[L.ai() + sp * NO * NO + (i / n) * NO + i % n] = a[i];
  }
  for (int i = sub; i < N * N; i += GS) v[L.f() + i] = st.fso[(size_t)w * N * N + i];
  for (int i = sub; i < N * C; i += GS) v[L.a() + i] = st.ren[((size_t)w * N * C + i) * 2 + 1];
  for (int i = sub; i < N * L.qm; i += GS) v[L.z() + i] = st.zq[((size_t)w * N + i / L.qm) * ZQ + 1 + i % L.qm];
  __syncwarp(m);
  int n = 0;
  double *gp = v + L.row();
  for (int e = 0; e < N; e++) {
    const int got = tmove<NORD>(s, T, J, E, st, v, L, w, e, A, step, gp);
    if (got) {
      // the electron's distances and power sums
      for (int c = sub; c < C; c += GS) {
        const double dx = v[3 * e] - s.cent[3 * c], dy = v[3 * e + 1] - s.cent[3 * c + 1], dz = v[3 * e + 2] - s.cent[3 * c + 2];
        double *ren = st.ren + ((size_t)w * N * C + e * C + c) * 2;
        ren[0] = sqrt(dx * dx + dy * dy + dz * dz);
        ren[1] = v[L.a() + e * C + c];
      }
      for (int q = 1 + sub; q < ZQ; q += GS) {
        double z = 0;
        for (int c = 0; c < C; c++) z += ipow(v[L.a() + e * C + c], q);
        st.zq[((size_t)w * N + e) * ZQ + q] = z;
      }
    }
    n += got;
    __syncwarp(m);
  }
  store(s, st, w, v, L);
  if (A.moved && sub == 0) A.moved[w] = n;
}

}  // namespace sm

// nlpoints.cuh -- the last part of the staged evaluation: velocities, nonlocal pseudopotential, E_L and
// the FP32 move tables, WPW warps per walker; and the projection of G onto the basis before it.
//
// The Jastrow ratio at a quadrature point p of electron e is, beside e-e and e-n terms, the e-e-n sum
// over the other electrons j and the centres.  Its terms are u_pj^k a_pc^p r_jc^q:
//   k = 0 does not depend on the pair: sum_c a_pc^p (sum_j r_jc^q - r_ec^q) from per-centre sums;
//   terms of one electron alone (q = 0 or p = 0) need only sum_j u^k and sum_j u^k S_l(j);
//   the rest is sum_c a_pc^p T_kq(p, c) with T_kq(p, c) = sum_j u_pj^k r_jc^q, products [p][j] x [j][c]
//   issued as mma m8n8k4 -- 3 of them for order 4 (6 for order 5), where the sums over centres
//   X_pq(p, j) of the same terms took 6 (10).
// A lane's fragment element is one (point, electron) pair, so each lane forms its pair's distance
// and powers once, in place.  The determinant ratio sums the basis functions at the point (lane =
// point) with the electron's projected G; a primitive whose exponent exceeds the shell's smallest weighing one
// by more than 70 / r^2 is not formed (gauss_radial).
// What bounds it: latency between dependent FP64 instructions and mma (an issue in every third cycle; a
// third of the FP64 pipe), hence the most warps that the registers allow.  Blocks of 8 warps on one walker from 65
// electrons on put 16 warps on an SM where shared memory holds two such walkers only: 21.0 -> 19.1 ms at 128
// electrons, against 4 warps and 168 registers.  With 33 to 64 electrons 4 warps at 128 registers, 1.42 -> 1.19 ms; a
// warp per walker below that keeps 168 registers with one determinant (0.53 against 0.55 ms), and takes 128
// with several, whose tables add to the wait for memory (1.07 -> 0.91 ms).
// Measured (B200), the part of an evaluation from the inverses on, projection included, against k_el_fin:
// 4096 walkers of 128 electrons and 32 centres, order 4, 46.2 -> 20.2 ms (projection 0.95); 1001 of 51
// and 13, order 5, 4.57 -> 1.23 ms; 3001 of 20 and 5, 0.96 -> 0.56 ms; the multi-determinant dimer (200
// determinants), 3.8 -> 0.9 ms.  k_el_fin stays for several centre types with e-e-n terms.
#pragma once
#include "jastile.cuh"
#include "shelltab.cuh"

namespace pt {

using jt::sfor;

// G projected onto the basis, gproj[e][b] = sum_k coef[b][k] G[k][e]: a block per (walker, spin), G
// staged in shared memory, 8 x 2 tiles of m8n8k4 per warp and 64 basis functions per block pass.
constexpr int GP_LD = 68;  // = 4 mod 16 doubles
template <bool MD>
__global__ void __launch_bounds__(128, 4) k_gproj(const __grid_constant__ Sys<double> s, const __grid_constant__ State<double> st) {
  extern __shared__ __align__(16) double G[];  // [nocc][GP_LD]
  const int w = blockIdx.x >> 1, sp = blockIdx.x & 1, n = sp ? s.ndn : s.nup, no = s.nocc[sp], e0 = sp ? s.nup : 0;
  if (n == 0) return;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5, rr = lane >> 2, kq = lane & 3, B = s.nbasis;
  const double *g = MD ? st.gam + (size_t)w * st.gstride + (sp ? s.nocc[0] * s.nup : 0)
                       : st.ainv + (size_t)w * st.astride + (sp ? s.nup * s.nup : 0);
  const int no4 = (no + 3) & ~3;
  for (int i = tid; i < no4 * 64; i += 128) {
    const int k = i >> 6, e = i & 63;
    G[k * GP_LD + e] = (k < no && e < n) ? g[k * n + e] : 0.0;
  }
  __syncthreads();
  const double *ct = s.coccT[sp];
  double *out = st.gproj + ((size_t)w * s.N + e0) * B;
  for (int b0 = 16 * wib; b0 < B; b0 += 64) {
    const int ba = min(b0 + rr, B - 1), bb = min(b0 + 8 + rr, B - 1);  // spare columns repeat the last (not stored)
    for (int m0 = 0; m0 < n; m0 += 32) {
      double c[4][2][2];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) c[i][j][0] = c[i][j][1] = 0;
#pragma unroll 4
      for (int k0 = 0; k0 < no4; k0 += 4) {
        const int k = min(k0 + kq, no - 1);  // past the orbitals G is zero
        const double x0 = ct[(size_t)k * B + ba], x1 = ct[(size_t)k * B + bb];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const double a = G[(k0 + kq) * GP_LD + m0 + 8 * i + rr];
          dmma_884(c[i][0][0], c[i][0][1], a, x0);
          dmma_884(c[i][1][0], c[i][1][1], a, x1);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int e = m0 + 8 * i + rr;
        if (e >= n) continue;
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int b = b0 + 8 * j + 2 * kq + h;
            if (b < B) out[(size_t)e * B + b] = c[i][j][h];
          }
      }
    }
  }
}

// (k, q) of the products T_kq, k >= 1, q >= 1, that the mixed terms of one electron pair need.
struct KQ {
  int n;
  int k[16], q[16];
};
__host__ __device__ constexpr KQ make_kq(int nord) {
  KQ x{};
  const jt::Combos c = jt::make_combos(nord);
  for (int k = 1; k <= nord; k++)
    for (int q = 1; q <= nord; q++) {
      bool need = false;
      for (int y = 0; y < c.n; y++)
        if (k < c.nk[y] && (c.m[y] == q || c.l[y] + c.m[y] == q)) need = true;
      if (need) { x.k[x.n] = k; x.q[x.n] = q; x.n++; }
    }
  return x;
}
__host__ __device__ constexpr int kq_index(const KQ &x, int k, int q) {
  for (int i = 0; i < x.n; i++)
    if (x.k[i] == k && x.q[i] == q) return i;
  return -1;
}
template <int NORD>
struct Tab {
  static constexpr jt::Combos cb = jt::make_combos(NORD);
  static constexpr Terms tl = make_terms(NORD);
  static constexpr KQ kq = make_kq(NORD);
};

// Shared memory of a walker (doubles): scaled distances [Ct][Np], positions, V_k [NORD][N], per-centre
// sums [NORD - 1][C], rows of the pair table summed [N], the tasks' radial values [nrow], reductions,
// per 32 (electron, centre) pairs the mask of those in range and the number in range before them, and
// (lane) the distances of lane_jastrow; and per electron what the velocities add to the energy [2][N].
struct Dims {
  int N, C, Ct, Np, nord, nrow, lane;
  __host__ __device__ Dims(int N_, int C_, int nord_, int nrow_, bool lane_ = false)
      : N(N_), C(C_), Ct(nord_ > 1 ? (C_ + 7) & ~7 : 0), Np(0), nord(nord_ > 1 ? nord_ : 0), nrow(nrow_), lane(nord_ > 1 && lane_) {
    const int p = (N_ + 3) & ~3;
    Np = p + ((4 - p % 16) + 16) % 16;
  }
  __host__ __device__ int x() const { return Ct * Np; }
  __host__ __device__ int v() const { return x() + 3 * N; }
  __host__ __device__ int z() const { return v() + nord * N; }
  __host__ __device__ int f() const { return z() + nord * Ct; }
  __host__ __device__ int row() const { return f() + N; }
  __host__ __device__ int red() const { return row() + nrow; }
  __host__ __device__ int msk() const { return red() + 32; }
  __host__ __device__ int lanes() const { return msk() + (N * C + 31) / 32 + 1; }
  __host__ __device__ int vel() const { return lanes() + (lane ? 32 * C : 0); }
  __host__ __device__ int total() const { return vel() + 2 * N; }
  __host__ __device__ size_t bytes() const { return sizeof(double) * (size_t)((total() + 1) & ~1); }
};

// e-e value with one division: u / (1 + b2 u) = r / (1 + k r + b2 r), du = 1 / (1 + k r).
__device__ __forceinline__ double ee_value(const JasPar<double> &J, int isb, double ss, int ipar, double r, double &du) {
  const double d1 = 1.0 + J.scalek * r, d2 = d1 + J.b[isb][1] * r, inv = 1.0 / (d1 * d2);
  du = d2 * inv;
  const double u = r * du;
  double p = 0;
  for (int i = J.nordb; i >= 2; i--) p = p * u + J.b[isb][i];
  return ss * J.b[isb][0] * r * (d1 * inv) - J.asymp_b[ipar] + p * u * u;
}

// Jastrow of electron e at 32 points (one per lane, lanes without one: act false), minus that of the
// electron where it is.
template <int NORD>
__device__ __forceinline__ double point_jastrow(const Sys<double> &s, const JasPar<double> &J, const Dims &D, const double *sm,
                                             const double *xn, int e, bool act, int lane) {
  using TB = Tab<NORD>;
  constexpr int NQ = make_kq(NORD).n > 0 ? make_kq(NORD).n : 1, NC = jt::make_combos(NORD).n, NT = make_terms(NORD).n;
  constexpr int QM = NORD > 1 ? NORD - 1 : 1, KM = NORD > 1 ? NORD : 1;
  const int N = s.N, C = s.C, Np = D.Np;
  const double *sd = sm, *xs = sm + D.x(), *V = sm + D.v(), *Z = sm + D.z(), *F = sm + D.f();
  const unsigned full = 0xffffffffu, am = __ballot_sync(full, act);
  const int kq = lane & 3, rr = lane >> 2;
  const double sk = J.scalek;
  double mine = 0;
#pragma unroll 1
  for (int mt = 0; mt < 4; mt++) {
    if (((am >> (8 * mt)) & 0xffu) == 0u) continue;
    const int prow = 8 * mt + rr;
    const double p0 = __shfl_sync(full, xn[0], prow), p1 = __shfl_sync(full, xn[1], prow), p2 = __shfl_sync(full, xn[2], prow);
    const int pe = __shfl_sync(full, e, prow);
    const bool pact = (am >> prow) & 1u;
    double f = 0;
    for (int c0 = 0; c0 < C; c0 += 32) {
      double T[NQ][4][2];
#pragma unroll
      for (int i = 0; i < NQ; i++)
#pragma unroll
        for (int t = 0; t < 4; t++) T[i][t][0] = T[i][t][1] = 0;
      double U[KM];
#pragma unroll
      for (int k = 0; k < KM; k++) U[k] = 0;
#pragma unroll 2
      for (int j0 = 0; j0 < N; j0 += 4) {
        const int j = j0 + kq;
        double u[KM + 1];
        u[0] = 1;
#pragma unroll
        for (int k = 1; k <= KM; k++) u[k] = 0;
        if (pact && j < N && j != pe) {
          const double a0 = p0 - xs[3 * j], a1 = p1 - xs[3 * j + 1], a2 = p2 - xs[3 * j + 2];
          const double rij = sqrt(a0 * a0 + a1 * a1 + a2 * a2);
          int isb, ipar;
          double ss, du;
          pair_class(J, s.nup, pe, j, isb, ss, ipar);
          const double ee = ee_value(J, isb, ss, ipar, rij, du);
          if (c0 == 0) f += ee;
          if constexpr (NORD > 1) {
#pragma unroll
            for (int k = 1; k <= KM; k++) u[k] = u[k - 1] * du;
            if (c0 == 0) {
#pragma unroll
              for (int k = 1; k <= KM; k++) {
                f += u[k] * V[(k - 1) * N + j];
                U[k - 1] += u[k];
              }
            }
          }
        }
        if constexpr (NORD > 1) {
#pragma unroll
          for (int t = 0; t < 4; t++) {
            if (c0 + 8 * t >= C) break;
            const double b = sd[(c0 + 8 * t + rr) * Np + j];
            double bp[QM + 1];
            bp[0] = 1;
#pragma unroll
            for (int q = 1; q <= QM; q++) bp[q] = bp[q - 1] * b;
            sfor<make_kq(NORD).n>([&](auto I) {
              constexpr int i = decltype(I)::v, k = TB::kq.k[i], q = TB::kq.q[i];
              dmma_884(T[i][t][0], T[i][t][1], u[k], bp[q]);
            });
          }
        }
      }
      // this lane's (point, centre) elements: e-n term, k = 0 terms, the T sums; and S_l of the point
      double S[QM];
#pragma unroll
      for (int q = 0; q < QM; q++) S[q] = 0;
#pragma unroll
      for (int t = 0; t < 4; t++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int c = c0 + 8 * t + 2 * kq + h;
          if (c >= C || !pact) continue;
          const double *cc = s.cent + 3 * c;
          const double a0 = p0 - cc[0], a1 = p1 - cc[1], a2 = p2 - cc[2];
          const double r = sqrt(a0 * a0 + a1 * a1 + a2 * a2), a = 1.0 / (1.0 + sk * r);
          double fi, fii;
          f += jas_en<double, false>(J, s.ctype[c], r, a, fi, fii);
          if constexpr (NORD > 1) {
            const double re = sd[c * Np + pe];
            double ap[QM + 1], rp[QM + 1];
            ap[0] = rp[0] = 1;
#pragma unroll
            for (int q = 1; q <= QM; q++) {
              ap[q] = ap[q - 1] * a;
              rp[q] = rp[q - 1] * re;
              S[q - 1] += ap[q];
            }
            sfor<2 * NC>([&](auto Y) {
              constexpr int yv = decltype(Y)::v, y = yv / 2, l = TB::cb.l[y], m = TB::cb.m[y], nk = TB::cb.nk[y];
              constexpr int p = yv % 2 ? m : l + m, q = yv % 2 ? l + m : m, i0 = TB::cb.ll[y][0];
              double v = J.c[0][i0] * (Z[(q - 1) * C + c] - rp[q]);
              sfor<nk - 1>([&](auto K) {
                constexpr int k = decltype(K)::v + 1, ik = TB::cb.ll[y][k], it = kq_index(TB::kq, k, q);
                v += J.c[0][ik] * T[it][t][h];
              });
              f += ap[p] * v;
            });
          }
        }
      if constexpr (NORD > 1) {
        // S_l of these centres is spread over the row's lanes, sum_j u^k is complete only with all
        // its lanes: share the latter, then each lane adds its centres' part
        if (c0 == 0) {
#pragma unroll
          for (int k = 0; k < KM; k++) {
            U[k] += __shfl_xor_sync(full, U[k], 1);
            U[k] += __shfl_xor_sync(full, U[k], 2);
          }
        }
        if (C <= 32) {
          sfor<NT>([&](auto L) {
            constexpr int ll = decltype(L)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
            if constexpr (TB::tl.m[ll] == 0 && l > 0) f += J.c[0][ll] * U[k - 1] * S[l - 1];
          });
        } else {
          // more than 32 centres: sum_j u^k again for this block of centres' S_l
          double Uk[KM];
#pragma unroll
          for (int k = 0; k < KM; k++) Uk[k] = 0;
          for (int j = kq; j < N; j += 4)
            if (pact && j != pe) {
              const double a0 = p0 - xs[3 * j], a1 = p1 - xs[3 * j + 1], a2 = p2 - xs[3 * j + 2];
              const double du = 1.0 / (1.0 + sk * sqrt(a0 * a0 + a1 * a1 + a2 * a2));
              double u = 1;
#pragma unroll
              for (int k = 0; k < KM; k++) { u *= du; Uk[k] += u; }
            }
#pragma unroll
          for (int k = 0; k < KM; k++) {
            Uk[k] += __shfl_xor_sync(full, Uk[k], 1);
            Uk[k] += __shfl_xor_sync(full, Uk[k], 2);
          }
          sfor<NT>([&](auto L) {
            constexpr int ll = decltype(L)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
            if constexpr (TB::tl.m[ll] == 0 && l > 0) f += J.c[0][ll] * Uk[k - 1] * S[l - 1];
          });
        }
      }
    }
    f += __shfl_xor_sync(full, f, 1);
    f += __shfl_xor_sync(full, f, 2);
    const double got = __shfl_sync(full, f, 4 * (lane & 7));
    if ((lane >> 3) == mt) mine = got;
  }
  return act ? mine - F[e] : 0.0;
}

// The same with a point per lane and no tiles: up to 32 electrons the tiles' rows and their centre part leave
// most of a warp idle.  pl: [C][32] doubles of the warp.
template <int NORD>
__device__ __forceinline__ double lane_jastrow(const Sys<double> &s, const JasPar<double> &J, const Dims &D, const double *sm, double *pl,
                                            const double *xn, int e, int lane) {
  using TB = Tab<NORD>;
  constexpr int NC = jt::make_combos(NORD).n, NT = make_terms(NORD).n, ND = jt::make_combos(NORD).nd;
  constexpr int QM = NORD > 1 ? NORD - 1 : 1, KM = NORD > 1 ? NORD : 1, NDA = ND > 0 ? ND : 1;
  const int N = s.N, C = s.C, Np = D.Np;
  const double *sd = sm, *xs = sm + D.x(), *V = sm + D.v(), *Z = sm + D.z(), *F = sm + D.f();
  const double sk = J.scalek;
  double f = -F[e], S[QM], U[KM];
#pragma unroll
  for (int q = 0; q < QM; q++) S[q] = 0;
#pragma unroll
  for (int k = 0; k < KM; k++) U[k] = 0;
  for (int c = 0; c < C; c++) {
    const double a0 = xn[0] - s.cent[3 * c], a1 = xn[1] - s.cent[3 * c + 1], a2 = xn[2] - s.cent[3 * c + 2];
    const double r = sqrt(a0 * a0 + a1 * a1 + a2 * a2), a = 1.0 / (1.0 + sk * r);
    double fi, fii;
    f += jas_en<double, false>(J, s.ctype[c], r, a, fi, fii);
    if constexpr (NORD > 1) {
      pl[32 * c + lane] = a;
      const double re = sd[c * Np + e];
      double ap[QM + 1], rp[QM + 1];
      ap[0] = rp[0] = 1;
#pragma unroll
      for (int q = 1; q <= QM; q++) {
        ap[q] = ap[q - 1] * a;
        rp[q] = rp[q - 1] * re;
        S[q - 1] += ap[q];
      }
      sfor<2 * NC>([&](auto Y) {
        constexpr int yv = decltype(Y)::v, y = yv / 2, l = TB::cb.l[y], m = TB::cb.m[y], i0 = TB::cb.ll[y][0];
        constexpr int p = yv % 2 ? m : l + m, q = yv % 2 ? l + m : m;
        f += J.c[0][i0] * ap[p] * (Z[(q - 1) * C + c] - rp[q]);
      });
    }
  }
  for (int j = 0; j < N; j++) {
    if (j == e) continue;
    const double a0 = xn[0] - xs[3 * j], a1 = xn[1] - xs[3 * j + 1], a2 = xn[2] - xs[3 * j + 2];
    int isb, ipar;
    double ss, du;
    pair_class(J, s.nup, e, j, isb, ss, ipar);
    f += ee_value(J, isb, ss, ipar, sqrt(a0 * a0 + a1 * a1 + a2 * a2), du);
    if constexpr (NORD > 1) {
      double X[NDA];
#pragma unroll
      for (int y = 0; y < ND; y++) X[y] = 0;
#pragma unroll 2
      for (int c = 0; c < C; c++) {
        const double a = pl[32 * c + lane], b = sd[c * Np + j];
        double ap[QM + 1], bp[QM + 1];
        ap[0] = bp[0] = 1;
#pragma unroll
        for (int q = 1; q <= QM; q++) { ap[q] = ap[q - 1] * a; bp[q] = bp[q - 1] * b; }
        sfor<NC>([&](auto Y) {
          constexpr int y = decltype(Y)::v, l = TB::cb.l[y], m = TB::cb.m[y], dv = TB::cb.dv[y];
          if constexpr (dv >= 0) {
            X[dv] += ap[l + m] * bp[m];
            if constexpr (l > 0) X[dv] += ap[m] * bp[l + m];
          }
        });
      }
      double u[KM + 1];
      u[0] = 1;
#pragma unroll
      for (int k = 1; k <= KM; k++) {
        u[k] = u[k - 1] * du;
        U[k - 1] += u[k];
        f += u[k] * V[(k - 1) * N + j];
      }
      sfor<NC>([&](auto Y) {
        constexpr int y = decltype(Y)::v, l = TB::cb.l[y], nk = TB::cb.nk[y], dv = TB::cb.dv[y];
        if constexpr (dv >= 0) {
          double cu = 0;
          sfor<nk - 1>([&](auto K) {
            constexpr int k = decltype(K)::v + 1, ik = TB::cb.ll[y][k];
            cu += J.c[0][ik] * u[k];
          });
          f += (l ? cu : 2 * cu) * X[dv];
        }
      });
    }
  }
  if constexpr (NORD > 1)
    sfor<NT>([&](auto L) {
      constexpr int ll = decltype(L)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
      if constexpr (TB::tl.m[ll] == 0 && l > 0) f += J.c[0][ll] * U[k - 1] * S[l - 1];
    });
  return f;
}

// Determinant ratio at a point: sum_b phi_b(point) g_b.  c0: the centre whose shells' radial
// factors are tabulated in tab (null: none).
__device__ __forceinline__ double point_ratio(const Sys<double> &s, const stab::Tab &T, const double *xn, const double *g,
                                             int c0, const double *tab) {
  double dr = 0, d0 = 0, d1 = 0, d2 = 0, r2 = 0;
  int cen = -1;
  const int t0 = tab ? s.cshell0[c0] : 0, t1 = tab ? s.cshell0[c0 + 1] : 0;
#pragma unroll 1
  for (int ish = 0; ish < s.nshell; ish++) {
    const ShellRec h = T.rec[ish];
    if (h.cen != cen) {
      cen = h.cen;
      const double *cc = s.cent + 3 * cen;
      d0 = xn[0] - cc[0];
      d1 = xn[1] - cc[1];
      d2 = xn[2] - cc[2];
      r2 = d0 * d0 + d1 * d1 + d2 * d2;
    }
    double rad;
    if (ish >= t0 && ish < t1) rad = tab[ish - t0];
    else rad = stab::factor(s, T, ish, h, r2);
    const double *gb = g + h.b0;
    double S[9], G[9][3], acc = 0;
    switch (h.l) {
    case 0: acc = gb[0]; break;
    case 1: acc = d2 * gb[0] + d0 * gb[1] + d1 * gb[2]; break;
    case 2:
      solid_all<double, false>(2, d0, d1, d2, S, G);
#pragma unroll
      for (int i = 0; i < 5; i++) acc += S[i] * gb[i];
      break;
    case 3:
      solid_all<double, false>(3, d0, d1, d2, S, G);
#pragma unroll
      for (int i = 0; i < 7; i++) acc += S[i] * gb[i];
      break;
    default:
      solid_all<double, false>(4, d0, d1, d2, S, G);
#pragma unroll
      for (int i = 0; i < 9; i++) acc += S[i] * gb[i];
    }
    dr += acc * rad;
  }
  return dr;
}

// What the forward pass of the parameter gradient keeps (null otherwise): velocities [4N], points'
// coefficients [N C][nq], E_L and the number of tasks; the task records are the evaluation's.  b (may be
// null; walkers bstride apart): the coefficients without the determinant ratio, for the nonlocal part of
// the orbital-resolved local energy.
struct Tape {
  double *v = nullptr, *c = nullptr, *el = nullptr, *b = nullptr;
  int *n = nullptr;
  size_t bstride = 0;
};

template <int NORD, bool MD, int WPW>
__global__ void __launch_bounds__(WPW == 8 ? 256 : 128, WPW == 8 ? 2 : WPW == 4 || MD ? 4 : 3) k_fin_points(const __grid_constant__ Sys<double> s,
                                                       const __grid_constant__ State<double> st, int nrow,
                                                       int outputs, int stats, ElRot rot, int tables_only, Tape tape) {
  using TB = Tab<NORD>;
  __shared__ JasPar<double> J;
  __shared__ EcpPar E;
  extern __shared__ __align__(16) char dsm[];
  load_params(s, J, E);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpos = WPW == 1 ? 0 : wib;
  const int tid = WPW == 1 ? lane : (int)threadIdx.x, tpw = 32 * WPW, per = WPW == 1 ? 4 : 1;
  const int N = s.N, C = s.C, nomax = s.nomax;
  const Dims D(N, C, NORD, nrow, WPW == 1);
  const stab::Tab T = stab::stage(s, dsm);
  __syncthreads();
  double *sm = (double *)(dsm + stab::tab_smem(s.nshell, s.nprim) + (WPW == 1 ? D.bytes() * wib : 0));
  double *sd = sm, *xs = sm + D.x(), *V = sm + D.v(), *Z = sm + D.z(), *F = sm + D.f(), *row = sm + D.row(), *red = sm + D.red(), *vel = sm + D.vel();
  for (int w = blockIdx.x * per + (WPW == 1 ? wib : 0); w < st.W; w += gridDim.x * per) {
    View<double> v{};
    v.xs = xs;
    v.vacc = st.el_vj + (size_t)w * 4 * N;
    v.divj = v.vacc + 3 * N;
    v.ainv = st.ainv + (size_t)w * st.astride;
    v.fso = st.fso + (size_t)w * N * N;
    v.ren = st.ren + (size_t)w * N * C * 2;
    v.zq = st.zq + (size_t)w * N * ZQ;
    v.orb5 = st.orb5 + (size_t)w * N * 5 * nomax;
    v.gproj = st.gproj ? st.gproj + (size_t)w * N * s.nbasis : nullptr;
    v.nlt = st.nlt ? st.nlt + (size_t)w * N * C * NLT : nullptr;
    v.tv = st.tv + (size_t)w * st.tvstride;
    v.gam = st.gam + (size_t)w * st.gstride;
    v.ymd = st.ymd + (size_t)w * st.tvstride;
    v.wdet = st.wdet + (size_t)w * st.wstride;
    const double *rt = st.el_rt + (size_t)w * 2 * C * N, *sc = st.el_sc + (size_t)w * EL_SC;
    for (int i = tid; i < 3 * N; i += tpw) xs[i] = st.x[(size_t)w * 3 * N + i];
    double lnd = sc[4] + sc[6], sgn = sc[5] * sc[7];
    const bool ok = sc[5] != 0.0 && sc[7] != 0.0;
    if (MD && ok) {
      lnd += sc[8];
      sgn *= sc[9];
    }
    const bool points = s.nloc > 0 && ok && !tables_only;
    double d2lnd = 0, v2 = 0, vloc = 0, vnl = 0;
    if (!tables_only) {
      // velocities: 8 lanes per electron, the sums in the order of det_velocities (a lane's orbitals are those of
      // 4 lanes there).  Near a node grad psi / psi and lap psi / psi grow as 1 / d and their squares cancel in
      // E_L, which keeps the last bits of these sums: in another order the energies of a few thousand
      // unequilibrated walkers differed by 1e-8.
      for (int e4 = 4 * wpos; e4 < N; e4 += 4 * WPW) {
        const int e = e4 + (lane >> 3), l8 = lane & 7;
        double q[4][4];
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
          for (int i = 0; i < 4; i++) q[c][i] = 0;
        if (e < N) {
          const int sp = e < s.nup ? 0 : 1, n = sp ? s.ndn : s.nup, eo = sp ? e - s.nup : e, no = s.nocc[sp];
          const double *G = gam_ptr<double, MD>(s, v, sp), *oe = v.orb5 + (size_t)e * 5 * nomax;
          for (int k0 = l8; k0 < no; k0 += 32)
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const int k = k0 + 8 * i;
              if (k < no) {
                const double a = G[k * n + eo];
#pragma unroll
                for (int c = 0; c < 4; c++) q[c][i] += a * oe[(c + 1) * nomax + k];
              }
            }
        }
        double g[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          g[c] = (q[c][0] + q[c][2]) + (q[c][1] + q[c][3]);
#pragma unroll
          for (int o = 4; o >= 1; o >>= 1) g[c] += __shfl_xor_sync(0xffffffffu, g[c], o);
        }
        if (e < N && l8 == 0) {
          const double dvd = g[3] - (g[0] * g[0] + g[1] * g[1] + g[2] * g[2]);
          const double vx = v.vacc[3 * e] + g[0], vy = v.vacc[3 * e + 1] + g[1], vz = v.vacc[3 * e + 2] + g[2];
          vel[e] = dvd;
          vel[N + e] = vx * vx + vy * vy + vz * vz;
          if (outputs) {
            double *ov = st.o_vel + ((size_t)w * N + e) * 3;
            ov[0] = vx; ov[1] = vy; ov[2] = vz;
            st.o_divv[(size_t)w * N + e] = v.divj[e] + dvd;
          }
          if (tape.v) {
            double *ov = tape.v + (size_t)w * 4 * N + 3 * e;
            ov[0] = vx; ov[1] = vy; ov[2] = vz;
          }
        }
      }
    }
    int ntask = 0;
    if (points) {
      // ---- tables of the walker: scaled distances, per-centre sums, rows of the pair table, V_k
      if constexpr (NORD > 1) {
        for (int c = wpos; c < D.Ct; c += WPW) {
          double z[NORD - 1];
#pragma unroll
          for (int q = 0; q < NORD - 1; q++) z[q] = 0;
          for (int e = lane; e < D.Np; e += 32) {
            const double d = (c < C && e < N) ? rt[(C + c) * N + e] : 0.0;
            sd[c * D.Np + e] = d;
            double p = d;
#pragma unroll
            for (int q = 0; q < NORD - 1; q++) { z[q] += p; p *= d; }
          }
#pragma unroll
          for (int q = 0; q < NORD - 1; q++) {
            const double a = warp_sum(z[q]);
            if (lane == 0 && c < C) Z[q * C + c] = a;
          }
        }
        for (int e = tid; e < N; e += tpw) {
          double vk[NORD];
#pragma unroll
          for (int k = 0; k < NORD; k++) vk[k] = 0;
          sfor<make_terms(NORD).n>([&](auto L) {
            constexpr int ll = decltype(L)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
            if constexpr (TB::tl.m[ll] == 0) vk[k - 1] += J.c[0][ll] * (l ? v.zq[e * ZQ + l] : 2.0 * C);
          });
#pragma unroll
          for (int k = 0; k < NORD; k++) V[k * N + e] = vk[k];
        }
      }
      for (int e = wpos; e < N; e += WPW) {
        double a = 0;
        for (int j = lane; j < N; j += 32) a += v.fso[(size_t)e * N + j];
        a = warp_sum(a);
        if (lane == 0) F[e] = a;
      }
      // ---- (electron, centre) pairs in range, centre-major, so that the points of a round mostly share
      // their centre: first their masks (and the local part), then the records in order
      const int np = N * C, nch = (np + 31) / 32;
      unsigned *msk = (unsigned *)(sm + D.msk());
      int *moff = (int *)(msk + nch);
      for (int ch = wpos; ch < nch; ch += WPW) {
        const int j = 32 * ch + lane;
        bool nl = false;
        if (j < np) {
          double vps[MAXLCH];
          const int it = s.ctype[j / N];
          ecp_vps(E, it, rt[j], vps);
          vloc += vps[E.lpotp1[it] - 1];
          for (int l = 0; l < E.npotd[it]; l++)
            if (l + 1 != E.lpotp1[it] && fabs(vps[l]) > 1e-4) nl = true;
        }
        const unsigned m = __ballot_sync(0xffffffffu, nl);
        if (lane == 0) msk[ch] = m;
      }
      if (tid == 0) {
        double R[9];
        if (rot.random) random_rotation(rot.seed, (uint32_t)w, rot.sweep, R);
        else
          for (int i = 0; i < 9; i++) R[i] = rot.R[i];
        for (int i = 0; i < 9; i++) red[16 + i] = R[i];
      }
      jt::walker_sync<WPW>();
      if (wpos == 0) {
        int run = 0;
        for (int base = 0; base < nch; base += 32) {
          const int n1 = base + lane < nch ? __popc(msk[base + lane]) : 0;
          int inc = n1;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += x;
          }
          if (base + lane < nch) moff[base + lane] = run + inc - n1;
          run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) red[25] = (double)run;
      }
      jt::walker_sync<WPW>();
      ntask = (int)red[25];
      for (int ch = wpos; ch < nch; ch += WPW) {
        const unsigned m = msk[ch];
        if ((m >> lane) & 1u) {
          const int j = 32 * ch + lane, c = j / N, it = s.ctype[c];
          double vps[MAXLCH], *rec = v.nlt + (size_t)(moff[ch] + __popc(m & ((1u << lane) - 1u))) * NLT;
          ecp_vps(E, it, rt[j], vps);
          rec[0] = (double)((j - c * N) * C + c);
          rec[1] = rt[j];
          for (int l = 0; l < MAXLCH; l++) rec[2 + l] = (l < E.npotd[it]) ? vps[l] : 0.0;
        }
      }
      jt::walker_sync<WPW>();
      const int nshc = (s.nshc > 0 && ntask * s.nshc <= nrow) ? s.nshc : 0;
      for (int i = tid; i < ntask * nshc; i += tpw) {
        const int tk = i / nshc, k = i - tk * nshc;
        const double *rc = v.nlt + (size_t)tk * NLT;
        const int ish = s.cshell0[(int)rc[0] % C] + k;
        if (ish < s.cshell0[(int)rc[0] % C + 1])
          row[i] = stab::factor(s, T, ish, T.rec[ish], rc[1] * rc[1]);
      }
      jt::walker_sync<WPW>();
      const int nq = E.nquad, npts = ntask * nq;
      const double *R = red + 16;
      for (int t0 = 32 * wpos; t0 < npts; t0 += 32 * WPW) {
        const bool act = t0 + lane < npts;
        const int t = act ? t0 + lane : t0, task = t / nq, q = t - task * nq;
        const double *rec = v.nlt + (size_t)task * NLT;
        const int idx = (int)rec[0], e = idx / C, c = idx - e * C;
        const double r = rec[1], *cc = s.cent + 3 * c, *xe = xs + 3 * e, *q0 = s.quad->q0[q];
        double qv[3];
#pragma unroll
        for (int k = 0; k < 3; k++) qv[k] = R[3 * k] * q0[0] + R[3 * k + 1] * q0[1] + R[3 * k + 2] * q0[2];
        const double costh = ((xe[0] - cc[0]) * qv[0] + (xe[1] - cc[1]) * qv[1] + (xe[2] - cc[2]) * qv[2]) / r;
        const double xn[3] = {cc[0] + r * qv[0], cc[1] + r * qv[1], cc[2] + r * qv[2]};
        const double dr = point_ratio(s, T, xn, v.gproj + (size_t)e * s.nbasis, c, nshc ? row + task * nshc : nullptr);
        double dj;
        if constexpr (WPW == 1) dj = lane_jastrow<NORD>(s, J, D, sm, sm + D.lanes(), xn, e, lane);
        else dj = point_jastrow<NORD>(s, J, D, sm, xn, e, act, lane);
        if (!act) continue;
        const int it = s.ctype[c];
        double vp = 0;
        for (int l = 0; l < E.npotd[it]; l++)
          if (l + 1 != E.lpotp1[it]) vp += rec[2 + l] * yl0(l, costh);
        const double cb = s.quad->wq[q] * exp(dj) * vp, coeff = cb * dr;
        vnl += coeff;
        if (tape.c) tape.c[(size_t)w * N * C * nq + t] = coeff;
        if (tape.b) tape.b[(size_t)w * tape.bstride + t] = cb;
      }
    }
    vloc = warp_sum(vloc);
    vnl = warp_sum(vnl);
    if (WPW > 1) {
      __syncthreads();
      if (lane == 0) {
        double *o = red + 2 * wpos;  // the task counts and the rotation are no longer read
        o[0] = vloc; o[1] = vnl;
      }
      __syncthreads();
      vloc = vnl = 0;
      for (int k = 0; k < WPW; k++) {
        vloc += red[2 * k];
        vnl += red[2 * k + 1];
      }
    } else {
      __syncwarp();
    }
    if (wpos == 0) {
      for (int e = 0; e < N && !tables_only; e++) {  // in det_velocities' order, too
        d2lnd += vel[e];
        v2 += vel[N + e];
      }
      EvalRes res;
      finish_eval(s, st, w, v, lane, outputs != 0, ok, lnd, sgn, sc[0], sc[1], sc[2], sc[3], d2lnd, v2, vloc, vnl, ntask, res);
      if (stats && lane == 0) {
        st.s_esum[w] += res.eloc;
        st.s_e2sum[w] += res.eloc * res.eloc;
        st.s_elast[w] = res.eloc;
      }
      if (tape.el && lane == 0) {
        tape.el[w] = res.eloc;
        tape.n[w] = ntask;
        double *o = st.el_sc + (size_t)w * EL_SC;  // what the local part of the orbital energies needs
        o[10] = (res.d2j + res.vj2) / N;
        o[11] = (res.pe - res.pe_nl) / N;
      }
    }
    if (st.m_fso) {  // FP32 move tables of a mixed-precision state (mirror_store)
      const double *f = v.fso, *rn = v.ren, *zz = v.zq;
      for (int i = tid; i < N * N; i += tpw) st.m_fso[(size_t)w * N * N + i] = (float)f[i];
      for (int i = tid; i < N * C * 2; i += tpw) st.m_ren[(size_t)w * N * C * 2 + i] = (float)rn[i];
      for (int i = tid; i < N * ZQ; i += tpw) st.m_zq[(size_t)w * N * ZQ + i] = (float)zz[i];
      if (st.m_rtd)
        for (int i = tid; i < N * C; i += tpw) st.m_rtd[(size_t)w * C * N + i] = (float)rt[(size_t)C * N + i];
    }
    jt::walker_sync<WPW>();
  }
}

// Multi-determinant tables of every walker (a warp each): T, Y, G, and ln|chi|, sign(chi) to sc[8], sc[9].
static __global__ void __launch_bounds__(128, 4) k_md_tables(const __grid_constant__ Sys<double> s, const __grid_constant__ State<double> st) {
  const int lane = threadIdx.x & 31;
  for (int w = blockIdx.x * 4 + (threadIdx.x >> 5); w < st.W; w += gridDim.x * 4) {
    View<double> v{};
    v.ainv = st.ainv + (size_t)w * st.astride;
    v.orb5 = st.orb5 + (size_t)w * s.N * 5 * s.nomax;
    v.tv = st.tv + (size_t)w * st.tvstride;
    v.gam = st.gam + (size_t)w * st.gstride;
    v.ymd = st.ymd + (size_t)w * st.tvstride;
    v.wdet = st.wdet + (size_t)w * st.wstride;
    double *sc = st.el_sc + (size_t)w * EL_SC;
    if (sc[5] == 0.0 || sc[7] == 0.0) continue;
    double lc, sg;
    md_tables(s, v, lane, lc, sg);
    if (lane == 0) { sc[8] = lc; sc[9] = sg; }
    __syncwarp();
  }
}

}  // namespace pt

// pgtile.cuh -- parameter derivatives of walkers whose state lives in HBM, FP64, one centre type with
// e-e-n terms: the forward pass after the staged evaluation, and the reverse sweep of the Jastrow
// parameters with its sums over centres as tensor-core products.
//
// k_pgrad runs a warp per walker, adds every pair's and point's parameter values through shared-memory
// atomics and keeps per-electron sums of every parameter; here the seeds (-1/2 on the Laplacians, the
// velocities, each electron's sum of point coefficients) multiply a pair's contribution where it is formed,
// so a parameter has two sums in registers (value, local energy) and nothing is stored per electron.
// The e-e-n parameters are the terms of k_jas_tile (pairs) and point_jastrow (points), each with
// its own sum instead of being weighted by its coefficient.
// What bounds it: FP64 issue.  Measured (B200), 1024 walkers of 128 electrons, 32 centres, 2064 parameters: the
// forward pass 122 -> 15 ms (k_pg_nl 3.3, rows of all orbitals 2.9, the evaluation the rest), the reverse sweep
// 212 -> 4.5 ms (points 3.0, pairs 1.2).
#pragma once
#include "nlpoints.cuh"
#include "orbtile.cuh"

namespace pg {

using jt::sfor;

// Forward pass, nonlocal part: per electron the sum of its points' coefficients (tape_v + 3N), and
// phis[e][b], the points' basis functions weighted by their coefficients without the determinant ratio
// (tb): a warp per electron, lanes over shells, so that a row is summed in shared memory by its owner lanes.
static __global__ void __launch_bounds__(128, 6) k_pg_nl(const __grid_constant__ Sys<double> s, const __grid_constant__ State<double> st,
                                                  double *tape_v, const int *tape_n, const double *tape_c, double *scr,
                                                  size_t stride, const double *tape_b, ElRot rot, const int *order) {
  extern __shared__ __align__(16) char dsm[];
  const stab::Tab T = stab::stage(s, dsm);
  __syncthreads();
  double *rows = (double *)(dsm + stab::tab_smem(s.nshell, s.nprim));  // [4][nbasis]
  const int w = blockIdx.x, lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int N = s.N, C = s.C, B = s.nbasis, nq = s.ecp->nquad;
  double *row = rows + (size_t)wib * B;
  const int ntask = tape_n[w];
  const double *rec0 = st.nlt + (size_t)w * N * C * NLT, *tc = tape_c + (size_t)w * N * C * nq;
  for (int e = wib; e < N; e += 4) {
    for (int b = lane; b < B; b += 32) row[b] = 0;
    __syncwarp();
    double csum = 0;
    for (int t = 0; t < ntask; t++) {
      const double *rec = rec0 + (size_t)t * NLT;
      const int idx = (int)rec[0];
      if (idx / C != e) continue;
      const int c = idx - e * C;
      const double *cc = s.cent + 3 * c;
      for (int q = 0; q < nq; q++) {
        csum += tc[(size_t)t * nq + q];
        if (!scr) continue;
        const double cf = tape_b[(size_t)w * stride + (size_t)t * nq + q], *q0 = s.quad->q0[q];
        double xn[3];
#pragma unroll
        for (int k = 0; k < 3; k++) xn[k] = cc[k] + rec[1] * (rot.R[3 * k] * q0[0] + rot.R[3 * k + 1] * q0[1] + rot.R[3 * k + 2] * q0[2]);
        for (int h = lane; h < s.nshell; h += 32) {
          const int ish = order[h];
          const ShellRec r = T.rec[ish];
          const double *cs = s.cent + 3 * r.cen;
          const double d0 = xn[0] - cs[0], d1 = xn[1] - cs[1], d2 = xn[2] - cs[2];
          const double f = cf * stab::factor(s, T, ish, r, d0 * d0 + d1 * d1 + d2 * d2);
          double *o = row + r.b0;
          double S[9], G[9][3];
          switch (r.l) {
          case 0: o[0] += f; break;
          case 1: o[0] += f * d2; o[1] += f * d0; o[2] += f * d1; break;
          case 2:
            solid_all<double, false>(2, d0, d1, d2, S, G);
#pragma unroll
            for (int i = 0; i < 5; i++) o[i] += f * S[i];
            break;
          case 3:
            solid_all<double, false>(3, d0, d1, d2, S, G);
#pragma unroll
            for (int i = 0; i < 7; i++) o[i] += f * S[i];
            break;
          default:
            solid_all<double, false>(4, d0, d1, d2, S, G);
#pragma unroll
            for (int i = 0; i < 9; i++) o[i] += f * S[i];
          }
        }
      }
    }
    __syncwarp();
    if (lane == 0) tape_v[(size_t)w * 4 * N + 3 * N + e] = csum;
    if (scr)
      for (int b = lane; b < B; b += 32) scr[(size_t)w * stride + (size_t)e * B + b] = row[b];
    __syncwarp();
  }
}

// Local part of the orbital-resolved local energy (orbital_local_energy) from the orbitals in scr.
static __global__ void __launch_bounds__(256) k_pg_blocal(const __grid_constant__ Sys<double> s, const __grid_constant__ State<double> st,
                                                   double *scr, size_t stride) {
  const int N = s.N, M = s.norb;
  const long long n = (long long)st.W * N * M;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const int w = (int)(q / (N * M)), i = (int)(q - (long long)w * N * M), e = i / M, m = i - e * M;
    double *b = scr + (size_t)w * stride + (size_t)N * s.nbasis;
    const double *o = b + (size_t)e * 5 * M + m, *vj = st.el_vj + (size_t)w * 4 * N + 3 * e, *sc = st.el_sc + (size_t)w * EL_SC;
    b[(size_t)N * 5 * M + i] = -HB * (o[4 * M] + 2 * (vj[0] * o[M] + vj[1] * o[2 * M] + vj[2] * o[3 * M]) + sc[10] * o[0]) + sc[11] * o[0];
  }
}

constexpr int KB = MAXORD;  // e-e (k = 1 ..) and e-n (k = 2 ..) parameters of a set, at most
template <int NORD>
__host__ __device__ constexpr int nterms() { return make_terms(NORD).n; }

// Sums a lane's arrays over the walker's lanes and warps and adds them to dst.
template <int WPW>
__device__ __forceinline__ void reduce_add(double v, double *dst, int lane) {
  const double a = warp_sum(v);
  if (lane == 0) {
    if (WPW == 1) *dst += a;
    else atomicAdd(dst, a);
  }
}

// Reverse sweep, quadrature points: dst[P] = sum over the points of coefficient times the parameter's basis
// function with the electron there.  Shared memory as k_fin_points (pt::Dims; V holds the power sums).
template <int NORD, int WPW>
__global__ void __launch_bounds__(128, NORD > 4 ? 2 : 3) k_pg_points(const __grid_constant__ Sys<double> s,
                                                                     const __grid_constant__ State<double> st, const int *tape_n,
                                                                     const double *tape_c, double *raw, int P, ElRot rot) {
  using TB = pt::Tab<NORD>;
  constexpr int NT = nterms<NORD>(), NC = jt::make_combos(NORD).n, NQ = pt::make_kq(NORD).n, QM = NORD - 1, KM = NORD;
  __shared__ JasPar<double> J;
  __shared__ EcpPar E;
  extern __shared__ __align__(16) char dsm[];
  load_params(s, J, E);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpos = WPW == 1 ? 0 : wib;
  const int tid = WPW == 1 ? lane : (int)threadIdx.x, tpw = 32 * WPW, per = WPW == 1 ? 4 : 1;
  const int N = s.N, C = s.C;
  const pt::Dims D(N, C, NORD, 0);
  double *sm = (double *)(dsm + (WPW == 1 ? D.bytes() * wib : 0));
  double *sd = sm, *xs = sm + D.x(), *S = sm + D.v(), *Z = sm + D.z();
  const int kq = lane & 3, rr = lane >> 2, Np = D.Np;
  const double sk = J.scalek, ar = 1.0 / sk, b1 = J.b[0][0], b2 = J.b[0][1], ba = 1.0 + b2 * ar, r1c = ar * ar / (ba * ba);
  const unsigned full = 0xffffffffu;
  for (int w = blockIdx.x * per + (WPW == 1 ? wib : 0); w < st.W; w += gridDim.x * per) {
    const double *rt = st.el_rt + (size_t)w * 2 * C * N;
    for (int i = tid; i < 3 * N; i += tpw) xs[i] = st.x[(size_t)w * 3 * N + i];
    for (int c = wpos; c < D.Ct; c += WPW) {
      double z[QM];
#pragma unroll
      for (int q = 0; q < QM; q++) z[q] = 0;
      for (int e = lane; e < Np; e += 32) {
        const double d = (c < C && e < N) ? rt[(C + c) * N + e] : 0.0;
        sd[c * Np + e] = d;
        double p = d;
#pragma unroll
        for (int q = 0; q < QM; q++) { z[q] += p; p *= d; }
      }
#pragma unroll
      for (int q = 0; q < QM; q++) {
        const double a = warp_sum(z[q]);
        if (lane == 0 && c < C) Z[q * C + c] = a;
      }
    }
    for (int i = tid; i < QM * N; i += tpw) S[i] = st.zq[((size_t)w * N + i % N) * ZQ + 1 + i / N];
    jt::walker_sync<WPW>();
    double da[NT], eb[KB], ea[KB];
#pragma unroll
    for (int i = 0; i < NT; i++) da[i] = 0;
#pragma unroll
    for (int i = 0; i < KB; i++) eb[i] = ea[i] = 0;
    const int nq = E.nquad, npts = tape_n[w] * nq;
    const double *rec0 = st.nlt + (size_t)w * N * C * NLT, *tc = tape_c + (size_t)w * N * C * nq;
    for (int t0 = 32 * wpos; t0 < npts; t0 += 32 * WPW) {
      const int t = min(t0 + lane, npts - 1), task = t / nq, q = t - task * nq;
      const double cfl = t0 + lane < npts ? tc[t] : 0.0;
      const double *rec = rec0 + (size_t)task * NLT, *q0 = s.quad->q0[q];
      const int idx = (int)rec[0], el = idx / C;
      const double *cc0 = s.cent + 3 * (idx - el * C);
      double xn[3];
#pragma unroll
      for (int k = 0; k < 3; k++) xn[k] = cc0[k] + rec[1] * (rot.R[3 * k] * q0[0] + rot.R[3 * k + 1] * q0[1] + rot.R[3 * k + 2] * q0[2]);
      const unsigned am = __ballot_sync(full, cfl != 0.0);
#pragma unroll 1
      for (int mt = 0; mt < 4; mt++) {
        if (((am >> (8 * mt)) & 0xffu) == 0u) continue;
        const int prow = 8 * mt + rr;
        const double p0 = __shfl_sync(full, xn[0], prow), p1 = __shfl_sync(full, xn[1], prow), p2 = __shfl_sync(full, xn[2], prow);
        const int pe = __shfl_sync(full, el, prow);
        const double cw = __shfl_sync(full, cfl, prow);
        const bool pact = cw != 0.0;
        double U[KM];
#pragma unroll
        for (int k = 0; k < KM; k++) U[k] = 0;
        for (int c0 = 0; c0 < C; c0 += 32) {
          double T[NQ][4][2];
#pragma unroll
          for (int i = 0; i < NQ; i++)
#pragma unroll
            for (int x = 0; x < 4; x++) T[i][x][0] = T[i][x][1] = 0;
          for (int j0 = 0; j0 < N; j0 += 4) {
            const int j = j0 + kq;
            double u[KM + 1];
            u[0] = 1;
#pragma unroll
            for (int k = 1; k <= KM; k++) u[k] = 0;
            if (pact && j < N && j != pe) {
              const double a0 = p0 - xs[3 * j], a1 = p1 - xs[3 * j + 1], a2 = p2 - xs[3 * j + 2];
              const double rij = sqrt(a0 * a0 + a1 * a1 + a2 * a2), du = 1.0 / (1.0 + sk * rij);
#pragma unroll
              for (int k = 1; k <= KM; k++) u[k] = u[k - 1] * du;
              if (c0 == 0) {
                int isb, ipar;
                double ss;
                pair_class(J, s.nup, pe, j, isb, ss, ipar);
                const double x = rij * du, bu = 1.0 / (1.0 + b2 * x);
                double xp = x, ap = ar;
#pragma unroll
                for (int k = 1; k < KB; k++) {
                  if (k > J.nordb) break;
                  if (k == 1) eb[0] -= cw * ss * b1 * (x * x * bu * bu - r1c);
                  else eb[k - 1] += cw * (xp - ap);
                  xp *= x;
                  ap *= ar;
                }
#pragma unroll
                for (int k = 1; k <= KM; k++) U[k - 1] += u[k];
                sfor<NT>([&](auto L) {
                  constexpr int ll = decltype(L)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
                  if constexpr (TB::tl.m[ll] == 0) da[ll] += cw * u[k] * (l ? S[(l ? l - 1 : 0) * N + j] : 2.0 * C);
                });
              }
            }
#pragma unroll
            for (int x = 0; x < 4; x++) {
              if (c0 + 8 * x >= C) break;
              const double b = sd[(c0 + 8 * x + rr) * Np + j];
              double bp[QM + 1];
              bp[0] = 1;
#pragma unroll
              for (int k = 1; k <= QM; k++) bp[k] = bp[k - 1] * b;
              sfor<NQ>([&](auto I) {
                constexpr int i = decltype(I)::v, k = TB::kq.k[i], qq = TB::kq.q[i];
                dmma_884(T[i][x][0], T[i][x][1], u[k], bp[qq]);
              });
            }
          }
          if (c0 == 0) {
#pragma unroll
            for (int k = 0; k < KM; k++) {
              U[k] += __shfl_xor_sync(full, U[k], 1);
              U[k] += __shfl_xor_sync(full, U[k], 2);
            }
          }
          double Sp[QM];
#pragma unroll
          for (int k = 0; k < QM; k++) Sp[k] = 0;
#pragma unroll
          for (int x = 0; x < 4; x++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int c = c0 + 8 * x + 2 * kq + h;
              if (c >= C || !pact) continue;
              const double *cc = s.cent + 3 * c;
              const double a0 = p0 - cc[0], a1 = p1 - cc[1], a2 = p2 - cc[2];
              const double r = sqrt(a0 * a0 + a1 * a1 + a2 * a2), a = 1.0 / (1.0 + sk * r), y = r * a;
              double yp = y * y, rp2 = ar * ar;
#pragma unroll
              for (int k = 2; k < KB; k++) {
                if (k > J.norda) break;
                ea[k - 2] += cw * (yp - rp2);
                yp *= y;
                rp2 *= ar;
              }
              const double re = sd[c * Np + pe];
              double ap[QM + 1], rp[QM + 1];
              ap[0] = rp[0] = 1;
#pragma unroll
              for (int k = 1; k <= QM; k++) {
                ap[k] = ap[k - 1] * a;
                rp[k] = rp[k - 1] * re;
                Sp[k - 1] += ap[k];
              }
              sfor<2 * NC>([&](auto Y) {
                constexpr int yv = decltype(Y)::v, yy = yv / 2, l = TB::cb.l[yy], m = TB::cb.m[yy], nk = TB::cb.nk[yy];
                constexpr int p = yv % 2 ? m : l + m, qq = yv % 2 ? l + m : m, i0 = TB::cb.ll[yy][0];
                const double ca = cw * ap[p];
                da[i0] += ca * (Z[(qq - 1) * C + c] - rp[qq]);
                sfor<nk - 1>([&](auto K) {
                  constexpr int k = decltype(K)::v + 1, ik = TB::cb.ll[yy][k], it = pt::kq_index(TB::kq, k, qq);
                  da[ik] += ca * T[it][x][h];
                });
              });
            }
          sfor<NT>([&](auto L) {
            constexpr int ll = decltype(L)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
            if constexpr (TB::tl.m[ll] == 0 && l > 0) da[ll] += cw * U[k - 1] * Sp[l - 1];
          });
        }
      }
    }
    double *dst = raw + (size_t)w * 3 * P;
    const int na = J.norda - 1 > 0 ? J.norda - 1 : 0, nb = J.nordb;
#pragma unroll
    for (int k = 0; k < KB; k++) {
      if (k < na) reduce_add<WPW>(ea[k], dst + k, lane);
      if (k < nb) reduce_add<WPW>(eb[k], dst + na + k, lane);
    }
#pragma unroll
    for (int k = 0; k < NT; k++) reduce_add<WPW>(da[k], dst + na + nb + k, lane);
    jt::walker_sync<WPW>();
  }
}

// Reverse sweep, pairs and e-n terms: raw[1][P] = d ln psi / dp, raw[2][P] = -1/2 sum_e (lap_e + 2 v_e .
// grad_e) of the parameter's basis function minus the sum over e of its value times e's sum of
// point coefficients.  k_jas_tile's tiles; shared memory jt::Dims.
template <int NORD, int WPW>
__global__ void __launch_bounds__(128, 2) k_pg_pairs(const __grid_constant__ Sys<double> s, const __grid_constant__ State<double> st,
                                                     const double *tape_v, double *raw, int P) {
  using TB = jt::Tab<NORD>;
  constexpr int NC = jt::make_combos(NORD).n, NT = nterms<NORD>(), ND = jt::make_combos(NORD).nd, QM = NORD - 1;
  __shared__ JasPar<double> J;
  __shared__ EcpPar E;
  extern __shared__ __align__(16) char dsm[];
  load_params(s, J, E);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int N = s.N, C = s.C;
  const jt::Dims D(N, C, WPW);
  const int wpos = WPW == 1 ? 0 : wib;
  double *sm = (double *)(dsm + (WPW == 1 ? D.bytes() * wib : 0));
  double *sd = sm + D.d(), *sh = sm + D.h() + wpos * D.KS * 32, *xs = sm + D.x(), *ss = sm + D.s(), *cen = sm + D.cen(), *zs = sm + D.z();
  const int Np = D.Np, Cp = 4 * D.KS, KS = D.KS;
  const double sk = J.scalek, ar = 1.0 / sk, b1 = J.b[0][0], b2 = J.b[0][1], ba = 1.0 + b2 * ar, r1c = ar * ar / (ba * ba);
  const int tpw = 32 * WPW, tid = WPW == 1 ? lane : (int)threadIdx.x;
  const int rr = lane >> 2, kq = lane & 3, per = WPW == 1 ? 4 : 1;
  for (int w = blockIdx.x * per + (WPW == 1 ? wib : 0); w < st.W; w += gridDim.x * per) {
    const double *rt = st.el_rt + (size_t)w * 2 * C * N, *tv = tape_v + (size_t)w * 4 * N;
    for (int i = tid; i < 3 * N; i += tpw) xs[i] = st.x[(size_t)w * 3 * N + i];
    for (int i = tid; i < 3 * Cp; i += tpw) cen[i] = i < 3 * C ? s.cent[i] : 0.0;
    for (int c = wpos; c < Cp; c += WPW) {
      double z[QM];
#pragma unroll
      for (int q = 0; q < QM; q++) z[q] = 0;
      for (int e = lane; e < Np; e += 32) {
        const double d = (c < C && e < N) ? rt[(C + c) * N + e] : 0.0;
        sd[c * Np + e] = d;
        double p = d;
#pragma unroll
        for (int q = 0; q < QM; q++) { z[q] += p; p *= d; }
      }
#pragma unroll
      for (int q = 0; q < QM; q++) {
        const double a = warp_sum(z[q]);
        if (lane == 0) zs[q * Cp + c] = a;
      }
    }
    for (int i = tid; i < QM * N; i += tpw) ss[i] = st.zq[((size_t)w * N + i % N) * ZQ + 1 + i / N];
    jt::walker_sync<WPW>();
    // gv: value sums over ordered pairs (halved at the end); ge: local-energy sums
    double gv[NT], ge[NT], bv[KB], be[KB], av[KB], ae[KB];
#pragma unroll
    for (int i = 0; i < NT; i++) gv[i] = ge[i] = 0;
#pragma unroll
    for (int i = 0; i < KB; i++) bv[i] = be[i] = av[i] = ae[i] = 0;
    for (int i0 = 8 * wpos; i0 < N; i0 += 8 * WPW) {
      const int i = i0 + rr;
      const bool iok = i < N;
      const int ic = iok ? i : N - 1;
      const double xi0 = xs[3 * ic], xi1 = xs[3 * ic + 1], xi2 = xs[3 * ic + 2];
      const double vi0 = tv[3 * ic], vi1 = tv[3 * ic + 1], vi2 = tv[3 * ic + 2], ci = tv[3 * N + ic];
      double gs[QM][3], ls[QM];  // gradients of the power sums; -1/2 (lap + 2 v . grad) of them
#pragma unroll
      for (int q = 0; q < QM; q++) gs[q][0] = gs[q][1] = gs[q][2] = ls[q] = 0;
      for (int ks = 0; ks < KS; ks++) {
        const int c = 4 * ks + kq;
        double h = 0;
        if (c < C && iok) {
          const double a = sd[c * Np + i];
          const double dx = xi0 - cen[3 * c], dy = xi1 - cen[3 * c + 1], dz = xi2 - cen[3 * c + 2];
          const double r = rt[c * N + i], vr = vi0 * dx + vi1 * dy + vi2 * dz;
#pragma unroll
          for (int k = 2; k < KB; k++) {
            if (k > J.norda) break;
            double t, t1, t2;
            en_param_terms(J, r, a, k, t, t1, t2, true);
            av[k - 2] += t;
            ae[k - 2] -= HB * ((t2 + 2 * t1) + 2 * t1 * vr) + ci * t;
          }
          h = -sk * a * a / r;
          const double s2 = sk * sk * a * a;
          double ap[QM + 1], kp[QM + 1];
          ap[0] = 1;
          kp[0] = 0;
#pragma unroll
          for (int q = 1; q <= QM; q++) {
            ap[q] = ap[q - 1] * a;
            const double t = q * ap[q - 1] * h, lp = q * ap[q] * ((q - 1) * s2 + 2 * h);
            gs[q - 1][0] += t * dx;
            gs[q - 1][1] += t * dy;
            gs[q - 1][2] += t * dz;
            kp[q] = -HB * (lp + 2 * t * vr);
            ls[q - 1] += kp[q];
          }
          sfor<2 * NC>([&](auto Y) {  // k = 0: summed over the other electrons at once
            constexpr int yv = decltype(Y)::v, y = yv / 2, l = TB::cb.l[y], m = TB::cb.m[y], i0c = TB::cb.ll[y][0];
            constexpr int p = yv % 2 ? m : l + m, q = yv % 2 ? l + m : m;
            const double zr = zs[(q - 1) * Cp + c] - ap[q];
            gv[i0c] += ap[p] * zr;
            ge[i0c] += (kp[p] - ci * ap[p]) * zr;
          });
        }
        sh[ks * 32 + lane] = h;
      }
#pragma unroll
      for (int o = 1; o <= 2; o <<= 1)
#pragma unroll
        for (int q = 0; q < QM; q++) {
          gs[q][0] += __shfl_xor_sync(0xffffffffu, gs[q][0], o);
          gs[q][1] += __shfl_xor_sync(0xffffffffu, gs[q][1], o);
          gs[q][2] += __shfl_xor_sync(0xffffffffu, gs[q][2], o);
          ls[q] += __shfl_xor_sync(0xffffffffu, ls[q], o);
        }
      __syncwarp();
      for (int j0 = 0; j0 < N; j0 += 8) {
        double ax[ND][2], ag[ND][3][2], al[ND][2];
#pragma unroll
        for (int y = 0; y < ND; y++) {
          ax[y][0] = ax[y][1] = al[y][0] = al[y][1] = 0;
#pragma unroll
          for (int k = 0; k < 3; k++) ag[y][k][0] = ag[y][k][1] = 0;
        }
#pragma unroll 1
        for (int ks = 0; ks < KS; ks++) {
          const int c = 4 * ks + kq;
          const double a = sd[c * Np + i0 + rr], b = sd[c * Np + j0 + rr];
          double ap[QM + 1], bp[QM + 1];
          ap[0] = bp[0] = 1;
#pragma unroll
          for (int q = 1; q <= QM; q++) { ap[q] = ap[q - 1] * a; bp[q] = bp[q - 1] * b; }
          const double h = sh[ks * 32 + lane], s2 = sk * sk * a * a;
          const double dx = xi0 - cen[3 * c], dy = xi1 - cen[3 * c + 1], dz = xi2 - cen[3 * c + 2];
          sfor<2 * NC>([&](auto Y) {
            constexpr int yv = decltype(Y)::v, y = yv / 2, l = TB::cb.l[y], m = TB::cb.m[y], dv = TB::cb.dv[y];
            if constexpr (dv >= 0 && (yv % 2 == 0 || l > 0)) {
              constexpr int p = yv % 2 ? m : l + m, q = yv % 2 ? l + m : m;
              const double t = p * ap[p - 1] * h;
              dmma_884(ax[dv][0], ax[dv][1], ap[p], bp[q]);
              dmma_884(ag[dv][0][0], ag[dv][0][1], t * dx, bp[q]);
              dmma_884(ag[dv][1][0], ag[dv][1][1], t * dy, bp[q]);
              dmma_884(ag[dv][2][0], ag[dv][2][1], t * dz, bp[q]);
              dmma_884(al[dv][0], al[dv][1], p * ap[p] * ((p - 1) * s2 + 2 * h), bp[q]);
            }
          });
        }
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          const int j = j0 + 2 * kq + hh;
          if (!iok || j >= N || j == i) continue;
          const double r0 = xi0 - xs[3 * j], r1 = xi1 - xs[3 * j + 1], r2 = xi2 - xs[3 * j + 2];
          const double rij = sqrt(r0 * r0 + r1 * r1 + r2 * r2), rin = 1.0 / rij, du = 1.0 / (1.0 + sk * rij);
          const double vr = vi0 * r0 + vi1 * r1 + vi2 * r2;
          int isb, ipar;
          double sc;
          pair_class(J, s.nup, i, j, isb, sc, ipar);
          {
            const double x = rij * du, bu = 1.0 / (1.0 + b2 * x), d2 = du * du, dd2 = -2 * sk * du * d2, d4 = d2 * d2, d2r = d2 * rin;
            double xm2 = 0, xm1 = 1, xp = x, ap = ar;
#pragma unroll
            for (int k = 1; k < KB; k++) {
              if (k > J.nordb) break;
              double t, tu, tuu;
              if (k == 1) {
                t = -sc * b1 * (x * x * bu * bu - r1c);
                tu = -sc * b1 * 2 * x * bu * bu * bu;
                tuu = -sc * b1 * 2 * (1.0 - 2 * b2 * x) * bu * bu * bu * bu;
              } else {
                t = xp - ap;
                tu = k * xm1;
                tuu = k * (k - 1) * xm2;
              }
              xm2 = xm1;
              xm1 = xp;
              xp *= x;
              ap *= ar;
              const double t1 = tu * d2r, t2 = tuu * d4 + tu * dd2;
              bv[k - 1] += t;
              be[k - 1] -= HB * ((t2 + 2 * t1) + 2 * t1 * vr) + ci * t;
            }
          }
          double u[NORD + 1];
          u[0] = 1;
#pragma unroll
          for (int q = 1; q <= NORD; q++) u[q] = u[q - 1] * du;
          const double u1 = -sk * du * du, u1r = u1 * rin;
          // of u^k Y: -1/2 (lap + 2 v . grad) - c_i value
          auto add = [&](int ll, int k, double Y, double gY, double kY) {
            const double d1 = k * u[k - 1], d2u = k > 1 ? k * (k - 1) * u[k - 2 > 0 ? k - 2 : 0] : 0.0;
            gv[ll] += u[k] * Y;
            ge[ll] += -HB * ((d2u * u1 * u1 + 2 * d1 * u1r * (du + vr)) * Y + 2 * d1 * u1r * gY) + u[k] * (kY - ci * Y);
          };
          sfor<NT>([&](auto LL) {
            constexpr int ll = decltype(LL)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
            if constexpr (TB::tl.m[ll] == 0) {
              if constexpr (l == 0) add(ll, k, 2.0 * C, 0.0, 0.0);
              else add(ll, k, ss[(l - 1) * N + i] + ss[(l - 1) * N + j], r0 * gs[l - 1][0] + r1 * gs[l - 1][1] + r2 * gs[l - 1][2], ls[l - 1]);
            }
          });
          sfor<NC>([&](auto YY) {
            constexpr int y = decltype(YY)::v, dv = TB::cb.dv[y], l = TB::cb.l[y], nk = TB::cb.nk[y];
            if constexpr (dv >= 0) {
              const double f2 = l ? 1.0 : 2.0;
              const double gx = f2 * ag[dv][0][hh], gy = f2 * ag[dv][1][hh], gz = f2 * ag[dv][2][hh], Y = f2 * ax[dv][hh];
              const double gY = r0 * gx + r1 * gy + r2 * gz;
              const double kY = -HB * (f2 * al[dv][hh] + 2 * (vi0 * gx + vi1 * gy + vi2 * gz));
              sfor<nk - 1>([&](auto K) {
                constexpr int k = decltype(K)::v + 1, ik = TB::cb.ll[y][k];
                add(ik, k, Y, gY, kY);
              });
            }
          });
        }
      }
      __syncwarp();
    }
    double *g = raw + (size_t)w * 3 * P + P, *d = g + P;
    const int na = J.norda - 1 > 0 ? J.norda - 1 : 0, nb = J.nordb;
#pragma unroll
    for (int k = 0; k < KB; k++) {
      if (k < na) {
        reduce_add<WPW>(av[k], g + k, lane);
        reduce_add<WPW>(ae[k], d + k, lane);
      }
      if (k < nb) {
        reduce_add<WPW>(0.5 * bv[k], g + na + k, lane);
        reduce_add<WPW>(be[k], d + na + k, lane);
      }
    }
#pragma unroll
    for (int k = 0; k < NT; k++) {
      reduce_add<WPW>(0.5 * gv[k], g + na + nb + k, lane);
      reduce_add<WPW>(ge[k], d + na + nb + k, lane);
    }
    jt::walker_sync<WPW>();
  }
}

// Free Jastrow parameters from the raw ones (pg_finish): a, b as they are, c through the cusp projection.
static __global__ void __launch_bounds__(128) k_pg_out(const __grid_constant__ Sys<double> s, int W, const double *raw, int P, int nab, int nt,
                                                int nfree, int jo, double *dl, double *de) {
  const int n = nfree - jo;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < (long long)W * n; q += (long long)gridDim.x * blockDim.x) {
    const int w = (int)(q / n), f = (int)(q - (long long)w * n);
    const double *r = raw + (size_t)w * 3 * P;
    double g = 0, d = 0;
    if (f < nab) {
      g = r[P + f];
      d = r[f] + r[2 * P + f];
    } else {
      const int jf = f - nab;
      for (int ll = 0; ll < nt; ll++) {
        const double pm = s.cproj[ll * s.ncfree + jf];
        g += pm * r[P + nab + ll];
        d += pm * (r[nab + ll] + r[2 * P + nab + ll]);
      }
    }
    dl[(size_t)w * nfree + jo + f] = g;
    de[(size_t)w * nfree + jo + f] = d;
  }
}

}  // namespace pg

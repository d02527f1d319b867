// jastile.cuh -- the Jastrow part of the staged evaluation with its sums over centres as FP64
// tensor-core products (one centre type, e-e-n terms present).
//
// The e-e-n term of a pair, sum_c sum_klm c_klm u^k (a^l + r^l)(a r)^m with a = 1/(1 + k r_ic) and
// r = 1/(1 + k r_jc), needs for every ordered pair the sums over centres
//   Y_lm      = sum_c a^(l+m) r^m + a^m r^(l+m)
//   grad_i Y_lm, lap_i Y_lm   (only for the (l, m) that some k >= 1 multiplies)
// (the terms with m = 0 are sums over one electron alone).  For tiles of 8 electrons i by 8
// electrons j these are products over the centres, [i][c] x [c][j], issued as mma m8n8k4: a lane
// forms its fragment's powers and gradients in registers from a and h = -k a^2 / r, so only the
// scaled distances (one [C][N] table in shared memory) are loaded.  The terms with k = 0 do not
// depend on r_ij: their gradients and Laplacians summed over j need only sum_j r_jc^q per centre,
// so they are added once per electron instead of once per pair.
//
// What bounds it: the FP64 pipe (DMMA and scalar FMA share one rate).  Per ordered pair and centre
// 18 products for order 4 (value 6, gradient and Laplacian 12) against ~100 scalar operations per
// unordered pair and centre of the term-by-term sum of k_el_jas, which stays for several centre types
// and for no e-e-n term.  Measured (B200): 4096 walkers of 128 electrons and 32 centres, order 4,
// 33.2 -> 5.1 ms; 1001 walkers of 51 electrons and 13 centres, order 5, 1.35 -> 0.37 ms; 3001 walkers
// of 20 electrons and 5 centres, 0.17 -> 0.12 ms.
#pragma once
#include <utility>

#include "kernels.cuh"

namespace jt {

template <int I>
struct Ic {
  static constexpr int v = I;
};
// f(Ic<0>), ..., f(Ic<N - 1>): loops over the term tables
// whose indices stay compile-time constants (the tables then never reach memory)
template <class F, int... I>
__device__ __forceinline__ void sfor_seq(F &&f, std::integer_sequence<int, I...>) {
  (f(Ic<I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void sfor(F &&f) {
  sfor_seq(static_cast<F &&>(f), std::make_integer_sequence<int, N>{});
}

// The (l, m), m >= 1, of the e-e-n terms: k runs over 0 .. nk-1; the term's index in the c array
// for each k; dv: index among the ones with k >= 1 terms (whose gradients are needed per pair) or -1.
struct Combos {
  int n, nd;
  int l[12], m[12], nk[12], dv[12];
  int ll[12][8];
};
__host__ __device__ constexpr int term_index(const Terms &t, int k, int l, int m) {
  for (int i = 0; i < t.n; i++)
    if (t.k[i] == k && t.l[i] == l && t.m[i] == m) return i;
  return -1;
}
__host__ __device__ constexpr Combos make_combos(int nord) {
  Combos x{};
  const Terms t = make_terms(nord);
  for (int m = 1; 2 * m <= nord; m++)
    for (int l = 0; l + 2 * m <= nord; l++) {
      x.l[x.n] = l;
      x.m[x.n] = m;
      x.nk[x.n] = nord - l - 2 * m + 1;
      for (int k = 0; k < x.nk[x.n]; k++) x.ll[x.n][k] = term_index(t, k, l, m);
      x.dv[x.n] = x.nk[x.n] > 1 ? x.nd++ : -1;
      x.n++;
    }
  return x;
}

constexpr int WARPS = 4;  // warps of a block of a walker of more than 32 electrons
constexpr int SP = 6;     // per-electron power sums kept in shared memory: sum_c a^q, q = 1 .. SP

// Shared memory of one walker (doubles): scaled distances [4 KS][Np], h fragments per warp
// [KS][32], positions, power sums [SP][N], column sums of the pair Laplacians per warp, centres,
// per-centre sums of powers and of their Laplacians.
struct Dims {
  int KS, Np, N, C, warps;
  __host__ __device__ Dims(int N_, int C_, int w) : KS((C_ + 3) / 4), Np(0), N(N_), C(C_), warps(w) {
    // row stride = 4 mod 16 doubles: the fragment loads (4 rows by 4 columns per half warp) hit
    // 16 different banks
    const int p = (N_ + 7) & ~7;
    Np = p + ((4 - p % 16) + 16) % 16;
  }
  __host__ __device__ int d() const { return 0; }
  __host__ __device__ int h() const { return 4 * KS * Np; }
  __host__ __device__ int x() const { return h() + warps * KS * 32; }
  __host__ __device__ int s() const { return x() + 3 * N; }
  __host__ __device__ int col() const { return s() + SP * N; }
  __host__ __device__ int cen() const { return col() + warps * N; }
  __host__ __device__ int z() const { return cen() + 3 * 4 * KS; }
  __host__ __device__ int red() const { return z() + 2 * SP * 4 * KS; }
  __host__ __device__ int total() const { return red() + 4 * warps; }
  __host__ __device__ size_t bytes() const { return sizeof(double) * (size_t)((total() + 1) & ~1); }
};

template <int WPW>
__device__ __forceinline__ void walker_sync() {
  if (WPW == 1) __syncwarp();
  else __syncthreads();
}

template <int NORD>
struct Tab {
  static constexpr Combos cb = make_combos(NORD);
  static constexpr Terms tl = make_terms(NORD);
};

// WPW warps per walker (1: every warp of a block its own walker; WARPS: the block shares one).
// VO: values only (pair table, distances, Jastrow sum).
template <int NORD, int WPW, bool VO>
__global__ void __launch_bounds__(128, NORD > 4 ? 2 : 3) k_jas_tile(Sys<double> s, State<double> st) {
  using TB = Tab<NORD>;
  constexpr int NC = make_combos(NORD).n, NT = make_terms(NORD).n;
  constexpr int ND = VO ? 0 : make_combos(NORD).nd, NDA = ND > 0 ? ND : 1;
  constexpr int QM = NORD - 1;  // largest power of a scaled distance in the mixed terms
  __shared__ JasPar<double> J;
  __shared__ EcpPar E;
  extern __shared__ __align__(16) char dsm[];
  load_params(s, J, E);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int N = s.N, C = s.C;
  const Dims D(N, C, WPW);
  const int wpos = WPW == 1 ? 0 : wib;  // this warp's place among its walker's warps
  double *sm = (double *)(dsm + (WPW == 1 ? D.bytes() * wib : 0));
  double *sd = sm + D.d(), *sh = sm + D.h() + wpos * D.KS * 32, *xs = sm + D.x(), *ss = sm + D.s(),
         *col = sm + D.col() + wpos * N, *cen = sm + D.cen(), *zs = sm + D.z(), *red = sm + D.red();
  double *lz = zs + SP * 4 * D.KS;
  const int Np = D.Np, Cp = 4 * D.KS, KS = D.KS;
  const double sk = J.scalek;
  const int tpw = 32 * WPW, tid = WPW == 1 ? lane : (int)threadIdx.x;  // this walker's threads
  const int rr = lane >> 2, kq = lane & 3;
  const int per = WPW == 1 ? WARPS : 1;
  for (int w = blockIdx.x * per + (WPW == 1 ? wib : 0); w < st.W; w += gridDim.x * per) {
    for (int i = tid; i < 3 * N; i += tpw) xs[i] = st.x[(size_t)w * 3 * N + i];
    for (int i = tid; i < 3 * Cp; i += tpw) cen[i] = i < 3 * C ? s.cent[i] : 0.0;
    for (int i = tid; i < WPW * N; i += tpw) (sm + D.col())[i] = 0.0;
    walker_sync<WPW>();
    // distances to the centres (lanes over electrons, a warp per centre), and per centre the sums
    // over the electrons of the powers and of their Laplacians
    double pe_en = 0;
    double *rt = st.el_rt + (size_t)w * 2 * C * N, *ren = st.ren + (size_t)w * N * C * 2;
    for (int c = wpos; c < Cp; c += WPW) {
      double zq[QM], lq[QM];
#pragma unroll
      for (int q = 0; q < QM; q++) zq[q] = lq[q] = 0;
      for (int e = lane; e < Np; e += 32) {
        double d = 0;
        if (c < C && e < N) {
          const double *cc = s.cent + 3 * c;
          const double a0 = xs[3 * e] - cc[0], a1 = xs[3 * e + 1] - cc[1], a2 = xs[3 * e + 2] - cc[2];
          const double r = sqrt(a0 * a0 + a1 * a1 + a2 * a2);
          d = 1.0 / (1.0 + sk * r);
          rt[c * N + e] = r;
          rt[(C + c) * N + e] = d;
          *(double2 *)(ren + 2 * (e * C + c)) = make_double2(r, d);
          if (s.nloc == 0) pe_en -= s.zc[c] / r;
          if (!VO) {
            const double h = -sk * d * d / r, s2 = sk * sk * d * d;
            double p = d;
#pragma unroll
            for (int q = 0; q < QM; q++) {
              zq[q] += p;
              lq[q] += (q + 1) * p * (q * s2 + 2 * h);
              p *= d;
            }
          }
        }
        sd[c * Np + e] = d;
      }
      if (!VO) {
#pragma unroll
        for (int q = 0; q < QM; q++) {
          const double a = warp_sum(zq[q]), b = warp_sum(lq[q]);
          if (lane == 0) {
            zs[q * Cp + c] = a;
            lz[q * Cp + c] = b;
          }
        }
      }
    }
    walker_sync<WPW>();
    for (int e = tid; e < N; e += tpw) {
      double z[ZQ];
      z[0] = (double)C;
#pragma unroll
      for (int q = 1; q < ZQ; q++) z[q] = 0;
      for (int c = 0; c < C; c++) {
        const double d = sd[c * Np + e];
        double p = d;
#pragma unroll
        for (int q = 1; q < ZQ; q++) { z[q] += p; p *= d; }
      }
      double *g = st.zq + ((size_t)w * N + e) * ZQ;
#pragma unroll
      for (int q = 0; q < ZQ; q++) g[q] = z[q];
#pragma unroll
      for (int q = 0; q < SP; q++) ss[q * N + e] = z[q + 1];
    }
    walker_sync<WPW>();
    double fsum = 0, d2j = 0, pe_ee = 0;
    double *vj = st.el_vj + (size_t)w * 4 * N, *fso = st.fso + (size_t)w * N * N;
    for (int i0 = 8 * wpos; i0 < N; i0 += 8 * WPW) {
      const int i = i0 + rr;
      const bool iok = i < N;
      const double xi0 = iok ? xs[3 * i] : 0.0, xi1 = iok ? xs[3 * i + 1] : 0.0, xi2 = iok ? xs[3 * i + 2] : 0.0;
      // ---- the row's one-electron parts, lanes over (electron, centre): e-n term, gradients and
      // Laplacians of the power sums, and the k = 0 e-e-n terms summed over all other electrons
      double v0 = 0, v1 = 0, v2 = 0, div = 0, fen = 0;
      double gs[QM][3], ls[QM];
#pragma unroll
      for (int q = 0; q < QM; q++) gs[q][0] = gs[q][1] = gs[q][2] = ls[q] = 0;
      for (int ks = 0; ks < KS; ks++) {
        const int c = 4 * ks + kq;
        double h = 0;
        if (c < C && iok) {
          const double a = sd[c * Np + i];
          const double dx = xi0 - cen[3 * c], dy = xi1 - cen[3 * c + 1], dz = xi2 - cen[3 * c + 2];
          const double r = rt[c * N + i];
          double fi = 0, fii = 0;
          fen += jas_en<double, !VO>(J, 0, r, a, fi, fii);
          if (!VO) {
            h = -sk * a * a / r;
            v0 += fi * dx;
            v1 += fi * dy;
            v2 += fi * dz;
            div += fii + 2 * fi;
            const double s2 = sk * sk * a * a;
            double ap[QM + 1], lp[QM + 1], tp[QM + 1];
            ap[0] = 1;
            lp[0] = tp[0] = 0;
#pragma unroll
            for (int q = 1; q <= QM; q++) {
              ap[q] = ap[q - 1] * a;
              tp[q] = q * ap[q - 1] * h;
              lp[q] = q * ap[q] * ((q - 1) * s2 + 2 * h);
              gs[q - 1][0] += tp[q] * dx;
              gs[q - 1][1] += tp[q] * dy;
              gs[q - 1][2] += tp[q] * dz;
              ls[q - 1] += lp[q];
            }
            double tg = 0, lown = 0, loth = 0;
            sfor<2 * NC>([&](auto Y) {
              constexpr int Yv = decltype(Y)::v, y = Yv / 2, l = TB::cb.l[y], m = TB::cb.m[y];
              constexpr int p = Yv % 2 ? m : l + m, q = Yv % 2 ? l + m : m;
              constexpr int i0c = TB::cb.ll[y][0];
              const double c0 = J.c[0][i0c], zr = c0 * (zs[(q - 1) * Cp + c] - ap[q]);
              tg += tp[p] * zr;
              lown += lp[p] * zr;
              loth += c0 * (lz[(p - 1) * Cp + c] - lp[p]) * ap[q];
            });
            v0 += tg * dx;
            v1 += tg * dy;
            v2 += tg * dz;
            div += 0.5 * (lown + loth);  // a pair's Laplacian is halved between its electrons
            d2j += lown + fii + 2 * fi;
          }
        }
        sh[ks * 32 + lane] = h;
      }
      // the four lanes of a row share its sums
#pragma unroll
      for (int o = 1; o <= 2; o <<= 1) {
        fen += __shfl_xor_sync(0xffffffffu, fen, o);
        if (!VO) {
#pragma unroll
          for (int q = 0; q < QM; q++) {
            gs[q][0] += __shfl_xor_sync(0xffffffffu, gs[q][0], o);
            gs[q][1] += __shfl_xor_sync(0xffffffffu, gs[q][1], o);
            gs[q][2] += __shfl_xor_sync(0xffffffffu, gs[q][2], o);
            ls[q] += __shfl_xor_sync(0xffffffffu, ls[q], o);
          }
        }
      }
      if (kq == 0 && iok) fsum += fen;
      double si[SP];
#pragma unroll
      for (int q = 0; q < SP; q++) si[q] = iok ? ss[q * N + i] : 0.0;
      __syncwarp();
      // ---- pair tiles
      for (int j0 = 0; j0 < N; j0 += 8) {
        double ax[NC][2], ag[NDA][3][2], al[NDA][2];
#pragma unroll
        for (int y = 0; y < NC; y++) ax[y][0] = ax[y][1] = 0;
#pragma unroll
        for (int y = 0; y < NDA; y++) {
          al[y][0] = al[y][1] = 0;
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
          sfor<NC>([&](auto Y) {
            constexpr int y = decltype(Y)::v, l = TB::cb.l[y], m = TB::cb.m[y];
            dmma_884(ax[y][0], ax[y][1], ap[l + m], bp[m]);
            if constexpr (l > 0) dmma_884(ax[y][0], ax[y][1], ap[m], bp[l + m]);
          });
          if constexpr (!VO) {
            const double h = sh[ks * 32 + lane], s2 = sk * sk * a * a;
            const double dx = xi0 - cen[3 * c], dy = xi1 - cen[3 * c + 1], dz = xi2 - cen[3 * c + 2];
            sfor<2 * NC>([&](auto Y) {
              constexpr int Yv = decltype(Y)::v, y = Yv / 2, l = TB::cb.l[y], m = TB::cb.m[y], dv = TB::cb.dv[y];
              if constexpr (dv >= 0 && (Yv % 2 == 0 || l > 0)) {
                constexpr int p = Yv % 2 ? m : l + m, q = Yv % 2 ? l + m : m;
                const double t = p * ap[p - 1] * h;
                dmma_884(ag[dv][0][0], ag[dv][0][1], t * dx, bp[q]);
                dmma_884(ag[dv][1][0], ag[dv][1][1], t * dy, bp[q]);
                dmma_884(ag[dv][2][0], ag[dv][2][1], t * dz, bp[q]);
                dmma_884(al[dv][0], al[dv][1], p * ap[p] * ((p - 1) * s2 + 2 * h), bp[q]);
              }
            });
          }
        }
        double lsum[2] = {0, 0};
        double fo[2] = {0, 0};
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          const int j = j0 + 2 * kq + hh;
          if (!iok || j >= N) continue;
          if (j == i) {
            fo[hh] = fen;  // the table's diagonal: the electron's e-n term
            continue;
          }
          const double r0 = xi0 - xs[3 * j], r1 = xi1 - xs[3 * j + 1], r2 = xi2 - xs[3 * j + 2];
          const double rij = sqrt(r0 * r0 + r1 * r1 + r2 * r2), rin = 1.0 / rij;
          const double du = 1.0 / (1.0 + sk * rij);
          int isb, ipar;
          double sc;
          pair_class(J, s.nup, i, j, isb, sc, ipar);
          double fu, fuu;
          double f = jas_ee<double, !VO>(J, isb, sc, ipar, rij, du, fu, fuu);
          double u[NORD + 1];
          u[0] = 1;
#pragma unroll
          for (int q = 1; q <= NORD; q++) u[q] = u[q - 1] * du;
          // w0 = sum c u^k Y, w1 = sum c k u^(k-1) Y, w2 = sum c k (k-1) u^(k-2) Y; the gradient of Y
          // with the weights c u^k (g) and c k u^(k-1) (t, only along r_ij), its Laplacian with c u^k (lp)
          double w0 = 0, w1 = 0, w2 = 0, g0 = 0, g1 = 0, g2 = 0, tt = 0, lp = 0;
          sfor<NT>([&](auto LL) {
            constexpr int ll = decltype(LL)::v, k = TB::tl.k[ll], l = TB::tl.l[ll];
            if constexpr (TB::tl.m[ll] == 0) {
              const double c = J.c[0][ll];
              double Y = 2.0 * C;
              if constexpr (l > 0) Y = si[l - 1] + ss[(l - 1) * N + j];
              w0 += c * u[k] * Y;
              if constexpr (!VO) {
                w1 += (c * k) * u[k - 1] * Y;
                if constexpr (k > 1) w2 += (c * (k * (k - 1))) * u[k - 2] * Y;
                if constexpr (l > 0) {
                  const double cu = c * u[k], ct = (c * k) * u[k - 1];
                  g0 += cu * gs[l - 1][0];
                  g1 += cu * gs[l - 1][1];
                  g2 += cu * gs[l - 1][2];
                  tt += ct * (r0 * gs[l - 1][0] + r1 * gs[l - 1][1] + r2 * gs[l - 1][2]);
                  lp += cu * ls[l - 1];
                }
              }
            }
          });
          sfor<NC>([&](auto YY) {
            constexpr int y = decltype(YY)::v, dv = TB::cb.dv[y], l = TB::cb.l[y], nk = TB::cb.nk[y];
            const double Y = (l ? 1.0 : 2.0) * ax[y][hh];
            double cu = 0, ct = 0;
            sfor<nk>([&](auto K) {
              constexpr int k = decltype(K)::v, ik = TB::cb.ll[y][k];
              const double c = J.c[0][ik];
              w0 += c * u[k] * Y;
              if constexpr (!VO && k > 0) {
                cu += c * u[k];
                ct += (c * k) * u[k - 1];
                if constexpr (k > 1) w2 += (c * (k * (k - 1))) * u[k - 2] * Y;
              }
            });
            if constexpr (!VO && dv >= 0) {
              w1 += ct * Y;
              if constexpr (l == 0) { cu *= 2; ct *= 2; }
              g0 += cu * ag[dv][0][hh];
              g1 += cu * ag[dv][1][hh];
              g2 += cu * ag[dv][2][hh];
              tt += ct * (r0 * ag[dv][0][hh] + r1 * ag[dv][1][hh] + r2 * ag[dv][2][hh]);
              lp += cu * al[dv][hh];
            }
          });
          f += w0;
          fo[hh] = f;
          if (j < i) {
            fsum += f;
            pe_ee += rin;
          }
          if (!VO) {
            const double u1 = -sk * du * du;  // du/dr; u'' + 2 u'/r = -2 k du^3 / r
            const double fr = fu + w1 * u1 * rin;
            v0 += fr * r0 + g0;
            v1 += fr * r1 + g1;
            v2 += fr * r2 + g2;
            const double lap = fuu + 2 * fu + w2 * u1 * u1 + 2 * u1 * rin * (w1 * du + tt) + lp;
            d2j += lap;
            div += 0.5 * lap;
            lsum[hh] = 0.5 * lap;
          }
        }
        if (iok) {
          const int j = j0 + 2 * kq;
          if (j + 1 < N && (N & 1) == 0) *(double2 *)(fso + (size_t)i * N + j) = make_double2(fo[0], fo[1]);
          else {
            if (j < N) fso[(size_t)i * N + j] = fo[0];
            if (j + 1 < N) fso[(size_t)i * N + j + 1] = fo[1];
          }
        }
        if (!VO) {
#pragma unroll
          for (int o = 4; o <= 16; o <<= 1) {
            lsum[0] += __shfl_xor_sync(0xffffffffu, lsum[0], o);
            lsum[1] += __shfl_xor_sync(0xffffffffu, lsum[1], o);
          }
          if (rr == 0) {
            if (j0 + 2 * kq < N) col[j0 + 2 * kq] += lsum[0];
            if (j0 + 2 * kq + 1 < N) col[j0 + 2 * kq + 1] += lsum[1];
          }
        }
      }
#pragma unroll
      for (int o = 1; o <= 2; o <<= 1) {
        v0 += __shfl_xor_sync(0xffffffffu, v0, o);
        v1 += __shfl_xor_sync(0xffffffffu, v1, o);
        v2 += __shfl_xor_sync(0xffffffffu, v2, o);
        div += __shfl_xor_sync(0xffffffffu, div, o);
      }
      if (iok && kq == 0) {
        vj[3 * i] = v0;
        vj[3 * i + 1] = v1;
        vj[3 * i + 2] = v2;
        vj[3 * N + i] = div;
      }
      __syncwarp();
    }
    fsum = warp_sum(fsum);
    d2j = warp_sum(d2j);
    pe_ee = warp_sum(pe_ee);
    pe_en = warp_sum(pe_en);
    if (lane == 0) {
      red[4 * wpos] = fsum;
      red[4 * wpos + 1] = d2j;
      red[4 * wpos + 2] = pe_ee;
      red[4 * wpos + 3] = pe_en;
    }
    walker_sync<WPW>();
    if (!VO)
      for (int e = tid; e < N; e += tpw) {
        double a = 0;
        for (int k = 0; k < WPW; k++) a += (sm + D.col())[k * N + e];
        vj[3 * N + e] += a;
      }
    if (tid < 4) {
      double a = 0;
      for (int k = 0; k < WPW; k++) a += red[4 * k + tid];
      st.el_sc[(size_t)w * EL_SC + tid] = a;
    }
    walker_sync<WPW>();
  }
}

}  // namespace jt

// movebatch.cuh -- a sweep of Gaussian single-electron moves of single-determinant walkers whose
// state lives in HBM, with everything but the accept decisions taken out of the serial chain.
//
// In a sweep every electron is proposed once, at x_e + step g_e, so all N proposals of a walker are
// known before the first decision.  What a decision needs of the earlier ones is little:
//   psi'/psi of the determinant: with M = Phi' A (row a: proposed orbital row of electron a; A the
//     spin's inverse at the start of the sweep) the ratio of electron e is M[e][e], and accepting e
//     is one elimination step of M with that pivot (the Sherman-Morrison update of A carried over
//     to M), of which only the rows and columns after e matter;
//   the Jastrow change dJ_e = sum_j u(x'_e, x_j) - u(x_e, x_j) with the current x_j: its value with
//     nobody moved, plus for every accepted j < e the correction
//     [u(x'_e, x'_j) - u(x'_j, x_e)] - [u(x'_e, x_j) - u(x_e, x_j)].
// So four kernels replace the warp-per-walker chain of proposals:
//   k_mv_draw   proposals and accept uniforms;
//   k_mv_prop   orbital rows of all proposals, a tiled product with the coefficients;
//   k_mv_pairs  for every pair the three pair values above, summed and differenced;
//   k_mv_walk   M by tensor-core products, then the N decisions.
// The pair values, orbitals and e-n terms are formed by the operations, in the order, of propose(), in
// the compute type T; ratios and sums are FP64 as there.  The evaluation that follows every sweep
// rebuilds the inverses and tables from the positions, so nothing but the positions is written back.
//
// Measured (B200), one sweep: 4096 walkers of 128 electrons, mixed precision, 19.4 -> 5.2 ms (pairs 2.6,
// orbital rows 1.6, decisions 1.0); 2048 in FP64, 22.7 -> 4.1 ms; 1001 walkers of 51 electrons,
// order 5, FP64, 1.48 -> 0.39 ms.
//
// The scratch is the walker's place in the orbital rows of the FP64 evaluation (5 N nomax doubles,
// free between evaluations): corrections [N][N], orbital rows [N][nomax], dJ [N], x' [N][3], uniforms [N].
#pragma once
#include "kernels.cuh"
#include "shelltab.cuh"

namespace mv {

struct Scr {
  double *base;
  size_t stride;
  int N, nomax;
  __host__ __device__ size_t need() const { return (size_t)N * N + (size_t)N * nomax + 5 * (size_t)N; }
  __device__ double *delta(int w) const { return base + (size_t)w * stride; }
  __device__ double *phi(int w) const { return delta(w) + (size_t)N * N; }
  __device__ double *dj(int w) const { return phi(w) + (size_t)N * nomax; }
  __device__ double *xn(int w) const { return dj(w) + N; }
  __device__ double *ua(int w) const { return xn(w) + 3 * N; }
};

static __global__ void __launch_bounds__(256) k_mv_draw(const double *x, int W, int N, Scr q, uint64_t seed, uint64_t sweep,
                                                 double step) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)W * N) return;
  const int w = (int)(i / N), e = (int)(i - (long long)w * N);
  double g[3], ua;
  move_randoms(seed, (uint32_t)w, sweep, (uint32_t)e, g, &ua);
  const double *xo = x + 3 * i;
  double *xn = q.xn(w) + 3 * e;
  xn[0] = xo[0] + step * g[0];
  xn[1] = xo[1] + step * g[1];
  xn[2] = xo[2] + step * g[2];
  q.ua(w)[e] = ua;
}

constexpr int PB = 128;  // proposals of a block
constexpr int KB = 32;   // basis functions of a chunk (whole shells)
template <class T, int NT>
__host__ __device__ constexpr int ldb() { return sizeof(T) == 4 ? 16 * NT : 16 * NT + 4; }
template <class T>
__host__ __device__ constexpr int lda() { return sizeof(T) == 4 ? PB : PB + 4; }
template <class T, int NT>
__host__ __device__ constexpr size_t prop_smem() { return sizeof(T) * (size_t)KB * (lda<T>() + ldb<T, NT>()); }

static __device__ __noinline__ void general_shell1(const Sys<double> &s, int ish, double x, double y, double z, double *o) {
  const double pt[3] = {x, y, z};
  shell_eval_put<double, 1>(s, ish, pt, [o](int sl, int, double v) { o[sl * lda<double>()] = v; });
}
__device__ __forceinline__ void put_shell(const Sys<double> &s, const stab::Tab &T, int ish, const double *pt, double *o) {
  const ShellRec h = T.rec[ish];
  if (h.kind == 1 && h.l <= 2) {
    const double *cc = s.cent + 3 * h.cen;
    const double d0 = pt[0] - cc[0], d1 = pt[1] - cc[1], d2 = pt[2] - cc[2];
    const double g = stab::gauss_radial(T, h, d0 * d0 + d1 * d1 + d2 * d2);
    constexpr int ld = lda<double>();
    if (h.l == 0) o[0] = g;
    else if (h.l == 1) {
      o[0] = d2 * g;
      o[ld] = d0 * g;
      o[2 * ld] = d1 * g;
    } else {
      double S[9], G[9][3];
      solid_all<double, false>(2, d0, d1, d2, S, G);
#pragma unroll
      for (int i = 0; i < 5; i++) o[i * ld] = S[i] * g;
    }
  } else {
    general_shell1(s, ish, pt[0], pt[1], pt[2], o);
  }
}
__device__ __forceinline__ void put_shell(const Sys<float> &s, const stab::Tab &, int ish, const double *pt, float *o) {
  shell_eval_put<float, 1>(s, ish, pt, [o](int sl, int, float v) { o[sl * lda<float>()] = v; });
}

// Orbital rows of 128 proposals of one spin (grid.y) per block: chunks of basis functions in shared
// memory (lane = proposal, a warp per shell) times the spin's coefficients, which arrive by
// cp.async and serve all 128 proposals.  FP32: every thread sums 8 x NT orbital values over the basis
// functions in order, as warp_orbitals does (the same sums); FP64: mma m8n8k4.
template <class T, int NT>
__global__ void __launch_bounds__(256, 2) k_mv_prop(const __grid_constant__ Sys<T> s, int W, Scr q, const int4 *chunk,
                                                    int nchunk) {
  extern __shared__ __align__(16) char dsm[];
  constexpr int LDA = lda<T>(), LDB = ldb<T, NT>(), NC = 16 * NT;
  T *phi = (T *)dsm, *cf = phi + KB * LDA;
  stab::Tab Tb{};
  if constexpr (sizeof(T) == 8) Tb = stab::stage(s, dsm + prop_smem<T, NT>());
  const int sp = blockIdx.y, n = sp ? s.ndn : s.nup, no = s.nocc[sp], e0 = sp ? s.nup : 0;
  const long long items = (long long)W * n, i0 = (long long)blockIdx.x * PB;
  if (i0 >= items) return;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const T *coef = s.cocc[sp];
  const int grp = wib & 3;  // this warp forms basis functions of proposals 32 grp ..
  double px[3];
  {
    long long it = i0 + 32 * grp + lane;
    if (it >= items) it = items - 1;
    const int w = (int)(it / n), e = e0 + (int)(it - (long long)w * n);
    const double *xn = q.xn(w) + 3 * e;
    px[0] = xn[0]; px[1] = xn[1]; px[2] = xn[2];
  }
  constexpr int EV = 16 / sizeof(T);
  const bool vec = no % EV == 0 && (reinterpret_cast<uintptr_t>(coef) & 15) == 0;
  // FP32: rows 8 (tid / 16) + 0..7, orbitals NT (tid % 16) + 0..NT-1; FP64: 4 x 2 warps of 4 x NT tiles
  const int rr = lane >> 2, kq = lane & 3, wm = wib >> 1, wn = wib & 1, tr = tid >> 4, tc = tid & 15;
  T acc[8][NT];
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < NT; j++) acc[i][j] = T(0);
  __syncthreads();  // the shell tables are in place
  for (int k = 0; k < nchunk; k++) {
    const int4 ch = chunk[k];
    const int nk = sizeof(T) == 4 ? ch.w : (ch.w + 3) & ~3;
    if (vec) {
      constexpr int V = NC / EV;
      for (int i = tid; i < nk * V; i += 256) {
        const int r = i / V, c = EV * (i - r * V);
        T *dst = cf + r * LDB + c;
        if (r < ch.w && c < no) cp_async16(dst, coef + (size_t)(ch.z + r) * no + c);
        else
#pragma unroll
          for (int v = 0; v < EV; v++) dst[v] = T(0);
      }
    } else {
      for (int i = tid; i < nk * NC; i += 256) {
        const int r = i / NC, c = i - r * NC;
        cf[r * LDB + c] = (r < ch.w && c < no) ? coef[(size_t)(ch.z + r) * no + c] : T(0);
      }
    }
    cp_async_commit();
    for (int r = ch.w + (wib >> 2); r < nk; r += 2) phi[r * LDA + 32 * grp + lane] = T(0);
    for (int h = wib >> 2; h < ch.y; h += 2) {
      const int ish = ch.x + h;
      put_shell(s, Tb, ish, px, phi + (s.shb0[ish] - ch.z) * LDA + 32 * grp + lane);
    }
    cp_async_wait<0>();
    __syncthreads();
    if constexpr (sizeof(T) == 4) {
#pragma unroll 4
      for (int u = 0; u < nk; u++) {
        float a[8], b[NT];
        *(float4 *)&a[0] = *(const float4 *)(phi + u * LDA + 8 * tr);
        *(float4 *)&a[4] = *(const float4 *)(phi + u * LDA + 8 * tr + 4);
        if constexpr (NT == 4) *(float4 *)&b[0] = *(const float4 *)(cf + u * LDB + 4 * tc);
        else
#pragma unroll
          for (int j = 0; j < NT; j++) b[j] = cf[u * LDB + NT * tc + j];
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int j = 0; j < NT; j++) acc[i][j] = fmaf(b[j], a[i], acc[i][j]);
      }
    } else {
      const T *ap = phi + kq * LDA + wm * 32 + rr, *bp = cf + kq * LDB + wn * 8 * NT + rr;
      for (int ks = 0; ks < nk; ks += 4) {
        T a[4], b[NT];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = ap[ks * LDA + 8 * i];
#pragma unroll
        for (int j = 0; j < NT; j++) b[j] = bp[ks * LDB + 8 * j];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < NT; j++) dmma_884((double &)acc[2 * i][j], (double &)acc[2 * i + 1][j], a[i], b[j]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < NT; j++) {
      int row, c;
      if constexpr (sizeof(T) == 4) {
        row = 8 * tr + i;
        c = NT * tc + j;
      } else {
        row = wm * 32 + 8 * (i >> 1) + rr;
        c = wn * 8 * NT + 8 * j + 2 * kq + (i & 1);
      }
      const long long it = i0 + row;
      if (it >= items || c >= no) continue;
      const int w = (int)(it / n), e = e0 + (int)(it - (long long)w * n);
      ((T *)q.phi(w))[(size_t)e * s.nomax + c] = acc[i][j];
    }
}

template <int WPW>
__device__ __forceinline__ void wsync() {
  if (WPW == 1) __syncwarp();
  else __syncthreads();
}

// Shared memory of a walker in k_mv_pairs: scaled distances to the centres of the proposed and the
// current positions [C][Np] (T), their power sums [NORD][Np] (T), positions [3 N] each and dJ sums per
// warp [WPW][Np] (double).
template <class T, int NORD>
struct PairDims {
  int Np, C, N;
  __host__ __device__ PairDims(int N_, int C_) : Np((N_ + 15) & ~15), C(NORD > 1 ? C_ : 0), N(N_) {}
  __host__ __device__ size_t t_elems() const { return (size_t)2 * C * Np + 2 * (NORD > 1 ? NORD : 0) * Np; }
  __host__ __device__ size_t bytes(int wpw) const {
    return align16(sizeof(T) * t_elems()) + sizeof(double) * (size_t)((6 * N + 1) / 2 * 2 + wpw * Np);
  }
};

// The pair values of every proposal, WPW warps per walker.  A warp takes 8 electrons i by 16
// electrons j at a time, a lane 2 x 2 pairs with i > j: u(x'_i, x_j), u(x'_j, x_i) and
// u(x'_i, x'_j), each from its sums over the centres (een_xsums' products, in its order).
// What bounds it: the FMA rate of T (6 products per pair value and centre for order 4).
template <class T, int NORD, int WPW>
__global__ void __launch_bounds__(128, 4) k_mv_pairs(const __grid_constant__ Sys<T> s, const __grid_constant__ State<T> st,
                                                     Scr q) {
  __shared__ JasPar<T> J;
  __shared__ EcpPar E;
  extern __shared__ __align__(16) char dsm[];
  load_params(s, J, E);
  constexpr MixedPQ mx = make_mixed(NORD);
  constexpr int NM = mx.n > 0 ? mx.n : 1;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpos = WPW == 1 ? 0 : wib;
  const int tid = WPW == 1 ? lane : (int)threadIdx.x, tpw = 32 * WPW, per = WPW == 1 ? 4 : 1;
  const int N = s.N, C = s.C;
  const PairDims<T, NORD> D(N, C);
  const int Np = D.Np;
  char *sm = dsm + (WPW == 1 ? D.bytes(1) * wib : 0);
  T *an = (T *)sm, *ao = an + (size_t)D.C * Np, *zn = ao + (size_t)D.C * Np, *zo = zn + (NORD > 1 ? NORD : 0) * Np;
  double *xo = (double *)(sm + align16(sizeof(T) * D.t_elems())), *xn = xo + 3 * N,
         *dall = xo + (6 * N + 1) / 2 * 2, *dw = dall + (size_t)wpos * Np;
  const T sk = J.scalek;
  const int ii = lane >> 3, jj = lane & 7;
  for (int w = blockIdx.x * per + (WPW == 1 ? wib : 0); w < st.W; w += gridDim.x * per) {
    const double *xg = st.x + (size_t)w * 3 * N, *xng = q.xn(w);
    for (int i = tid; i < 3 * N; i += tpw) {
      xo[i] = xg[i];
      xn[i] = xng[i];
    }
    for (int i = tid; i < WPW * Np; i += tpw) dall[i] = 0;
    wsync<WPW>();
    // e-n terms of the proposals and, for the e-e-n sums, both sets of scaled distances
    const T *ren = st.ren + (size_t)w * N * C * 2, *fso = st.fso + (size_t)w * N * N, *zq = st.zq + (size_t)w * N * ZQ;
    if constexpr (NORD > 1) {
      for (int i = tid; i < C * Np; i += tpw) {
        const int e = i / C, c = i - e * C;
        T d = 0, dold = 0;
        if (e < N) {
          T r;
          cen_dist(s, sk, xn + 3 * e, c, r, d);
          dold = ren[2 * (e * C + c) + 1];
        }
        an[c * Np + e] = d;
        ao[c * Np + e] = dold;
      }
      wsync<WPW>();
    }
    for (int e = tid; e < Np; e += tpw) {
      T z[NORD > 1 ? NORD : 1];
#pragma unroll
      for (int k = 0; k < (NORD > 1 ? NORD : 1); k++) z[k] = T(0);
      double en = 0;
      if (e < N) {
        for (int c0 = 0; c0 < 32 && c0 < C; c0++) {
          T fen = 0;
          for (int c = c0; c < C; c += 32) {  // as propose() sums them: a lane per 32 centres
            T r, d, fi = 0, fii = 0;
            cen_dist(s, sk, xn + 3 * e, c, r, d);
            fen += jas_en<T, false>(J, s.ctype[c], r, d, fi, fii);
          }
          en += (double)fen;
        }
        en -= (double)fso[(size_t)e * N + e];
        if constexpr (NORD > 1) {
          for (int c = 0; c < C; c++) {
            const T d = an[c * Np + e];
            T p = d;
#pragma unroll
            for (int k = 1; k < NORD; k++) {
              z[k] += p;
              // rounded by itself: the power sums add complete powers
              if constexpr (sizeof(T) == 4) p = __fmul_rn(p, d);
              else p = p * d;
            }
          }
          z[0] = T(C);
        }
      }
      dall[e] += en;
      if constexpr (NORD > 1)
#pragma unroll
        for (int k = 0; k < NORD; k++) {
          zn[k * Np + e] = z[k];
          zo[k * Np + e] = e < N ? zq[e * ZQ + k] : T(0);
        }
    }
    wsync<WPW>();
    double *delta = q.delta(w);
    const int nr = (N + 7) / 8;
    int t = 0;
    for (int r = 0; r < nr; r++)
      for (int c16 = 0; 16 * c16 < 8 * r + 8; c16++, t++) {
        if (t % WPW != wpos) continue;
        const int i0 = 8 * r + 2 * ii, j0 = 16 * c16 + 2 * jj;
        T val[3][2][2];
#pragma unroll 1
        for (int set = 0; set < 3; set++) {
          // proposed electron a (value set 1: j, else i), other electron b, at its old (sets 0, 1) or
          // proposed (set 2) position
          const int pe = set == 1 ? j0 : i0, oe = set == 1 ? i0 : j0;
          const T *po = set == 2 ? an : ao;
          T X[NM][2][2];
          if constexpr (NORD > 1) {
#pragma unroll
            for (int m = 0; m < mx.n; m++) X[m][0][0] = X[m][0][1] = X[m][1][0] = X[m][1][1] = T(0);
            const T *pa = an + pe, *pb = po + oe;
#pragma unroll 2
            for (int c = 0; c < C; c++) {
              T ap[2][NORD], bp[2][NORD];
#pragma unroll
              for (int h = 0; h < 2; h++) {
                ap[h][0] = bp[h][0] = T(1);
                ap[h][1] = pa[c * Np + h];
                bp[h][1] = pb[c * Np + h];
#pragma unroll
                for (int k = 2; k < NORD; k++) {
                  ap[h][k] = ap[h][k - 1] * ap[h][1];
                  bp[h][k] = bp[h][k - 1] * bp[h][1];
                }
              }
#pragma unroll
              for (int m = 0; m < mx.n; m++)
#pragma unroll
                for (int a = 0; a < 2; a++)
#pragma unroll
                  for (int b = 0; b < 2; b++) X[m][a][b] += ap[a][mx.p[m]] * bp[b][mx.q[m]];
            }
          }
#pragma unroll
          for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 2; b++) {
              const int e = pe + a, j = oe + b;
              T f = 0;
              if (e < N && j < N && e != j) {
                int isb, ipar;
                T ss;
                pair_class(J, s.nup, e, j, isb, ss, ipar);
                const double *xe = xn + 3 * e, *xj = (set == 2 ? xn : xo) + 3 * j;
                T rv[3] = {T(xe[0] - xj[0]), T(xe[1] - xj[1]), T(xe[2] - xj[2])};
                T rij = tsqrt(rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2]);
                T du = T(1) / (T(1) + sk * rij);
                T fu = 0, fuu = 0;
                f = jas_ee<T, false>(J, isb, ss, ipar, rij, du, fu, fuu);
                if constexpr (NORD > 1) {
                  T ai[NORD], zj[NORD], Xp[NM];
                  const T *zb = set == 2 ? zn : zo;
#pragma unroll
                  for (int k = 0; k < NORD; k++) {
                    ai[k] = zn[k * Np + e];
                    zj[k] = zb[k * Np + j];
                  }
#pragma unroll
                  for (int m = 0; m < mx.n; m++) Xp[m] = X[m][a][b];
                  f += een_from_x<T, NORD>(J.c[0], du, ai, zj, Xp);
                }
              }
              if (set == 0) val[0][a][b] = f;
              else if (set == 1) val[1][b][a] = f;
              else val[2][a][b] = f;
            }
        }
        double rs[2] = {0, 0}, cs[2] = {0, 0};
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
          for (int b = 0; b < 2; b++) {
            const int i = i0 + a, j = j0 + b;
            if (i >= N || j >= i) continue;
            const double q1 = (double)val[0][a][b] - (double)fso[(size_t)i * N + j],
                         q2 = (double)val[1][a][b] - (double)fso[(size_t)j * N + i];
            rs[a] += q1;
            cs[b] += q2;
            delta[(size_t)j * N + i] = ((double)val[2][a][b] - (double)val[1][a][b]) - q1;
          }
#pragma unroll
        for (int o = 1; o <= 4; o <<= 1) {
          rs[0] += __shfl_xor_sync(0xffffffffu, rs[0], o);
          rs[1] += __shfl_xor_sync(0xffffffffu, rs[1], o);
        }
#pragma unroll
        for (int o = 8; o <= 16; o <<= 1) {
          cs[0] += __shfl_xor_sync(0xffffffffu, cs[0], o);
          cs[1] += __shfl_xor_sync(0xffffffffu, cs[1], o);
        }
        if (jj == 0) {
          dw[i0] += rs[0];
          dw[i0 + 1] += rs[1];
        }
        __syncwarp();
        if (ii == 0) {
          dw[j0] += cs[0];
          dw[j0 + 1] += cs[1];
        }
        __syncwarp();
      }
    wsync<WPW>();
    double *dj = q.dj(w);
    for (int e = tid; e < N; e += tpw) {
      double a = 0;
      for (int k = 0; k < WPW; k++) a += dall[k * Np + e];
      dj[e] = a;
    }
    wsync<WPW>();
  }
}

// M = Phi' A of one spin by FP64 tensor-core products, then the spin's decisions in order; thread e
// keeps dJ of electron e.  The corrections of the next PF electrons are loaded ahead of their
// decisions.  One barrier per electron.
constexpr int PF = 4;
template <class T, int WPW>
__global__ void __launch_bounds__(128, 4) k_mv_walk(State<T> st, Scr q, int N, int nup, int nmax) {
  extern __shared__ __align__(16) char dsm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpos = WPW == 1 ? 0 : wib;
  const int tid = WPW == 1 ? lane : (int)threadIdx.x, tpw = 32 * WPW, per = WPW == 1 ? 4 : 1;
  const int rr = lane >> 2, kq = lane & 3;
  const int md = nmax * nmax, dw = md + 3 * N;  // doubles of a walker
  double *M = (double *)dsm + (WPW == 1 ? (size_t)dw * wib : 0), *sua = M + md, *sdj = sua + N;
  for (int w = blockIdx.x * per + (WPW == 1 ? wib : 0); w < st.W; w += gridDim.x * per) {
    const double *delta = q.delta(w);
    for (int i = tid; i < N; i += tpw) sua[i] = q.ua(w)[i];
    double dj = tid < N ? q.dj(w)[tid] : 0.0;
    bool taken = false;
    int acc = 0;
    double pf[PF];
#pragma unroll
    for (int k = 0; k < PF; k++) pf[k] = (k < N && tid > k && tid < N) ? delta[(size_t)k * N + tid] : 0.0;
    if (tid == 0) sdj[0] = dj;
    for (int sp = 0; sp < 2; sp++) {
      const int n = sp ? N - nup : nup, e0 = sp ? nup : 0;
      if (n == 0) continue;
      const T *phi = (const T *)q.phi(w) + (size_t)e0 * q.nomax;
      const double *A = st.ainv + (size_t)w * st.astride + (sp ? nup * nup : 0);
      wsync<WPW>();  // the other spin's M is no longer read
      for (int m0 = 16 * wpos; m0 < n; m0 += 16 * WPW)
        for (int n0 = 0; n0 < n; n0 += 32) {
          double c[2][4][2];
#pragma unroll
          for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) c[a][b][0] = c[a][b][1] = 0;
          for (int k0 = 0; k0 < n; k0 += 4) {
            const int k = k0 + kq;
            double av[2], bv[4];
#pragma unroll
            for (int a = 0; a < 2; a++) {
              const int r = m0 + 8 * a + rr;
              av[a] = (r < n && k < n) ? (double)phi[(size_t)r * q.nomax + k] : 0.0;
            }
#pragma unroll
            for (int b = 0; b < 4; b++) {
              const int cc = n0 + 8 * b + rr;
              bv[b] = (k < n && cc < n) ? A[k * n + cc] : 0.0;
            }
#pragma unroll
            for (int a = 0; a < 2; a++)
#pragma unroll
              for (int b = 0; b < 4; b++) dmma_884(c[a][b][0], c[a][b][1], av[a], bv[b]);
          }
#pragma unroll
          for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 4; b++)
#pragma unroll
              for (int h = 0; h < 2; h++) {
                const int r = m0 + 8 * a + rr, cc = n0 + 8 * b + 2 * kq + h;
                if (r < n && cc < n) M[r * nmax + cc] = c[a][b][h];
              }
        }
      for (int eo = 0; eo < n; eo++) {
        const int e = e0 + eo;
        wsync<WPW>();  // M and dJ of electron e are complete
        const double rho = M[eo * nmax + eo], d = sdj[e & 1];
        const double p = rho * rho * exp(2.0 * d);
        const double de = pf[0];
#pragma unroll
        for (int k = 0; k + 1 < PF; k++) pf[k] = pf[k + 1];
        const int en = e + PF;
        pf[PF - 1] = (en < N && tid > en && tid < N) ? delta[(size_t)en * N + tid] : 0.0;
        if (sua[e] < p) {
          acc++;
          if (tid == e) taken = true;
          dj += de;
          const double ri = 1.0 / rho;
          // rows and columns after e: M -= M[:, e] M[e, :] / rho
          const int nc = n - eo - 1;
          const int wc = nc > 32 ? 64 : nc > 16 ? 32 : 16;  // threads along a row
          const int c0 = tid & (wc - 1), r0 = tid / wc, rs = tpw / wc;
          if (c0 < nc) {
            const double me = M[eo * nmax + eo + 1 + c0] * ri;
            for (int r = eo + 1 + r0; r < n; r += rs) M[r * nmax + eo + 1 + c0] -= M[r * nmax + eo] * me;
          }
        }
        if (tid == e + 1) sdj[(e + 1) & 1] = dj;
      }
    }
    if (taken) {
      const double *xn = q.xn(w) + 3 * tid;
      double *x = st.x + (size_t)w * 3 * N + 3 * tid;
      x[0] = xn[0]; x[1] = xn[1]; x[2] = xn[2];
    }
    if (tid == 0) st.s_acc[w] += (double)acc;
    wsync<WPW>();
  }
}

}  // namespace mv

// orbtile.cuh -- basis functions and orbitals of every electron (value, gradient, Laplacian) for the
// staged evaluation, as FP64 tensor-core products, and the Slater-matrix inversion in registers.
#pragma once
#include "kernels.cuh"

namespace ot {

constexpr int EB = 32;      // electrons of a block (one per lane while the basis is formed)
constexpr int ROWS = 5 * EB;
constexpr int LDA = ROWS + 4;  // = 4 mod 16 doubles: the fragment loads hit different banks
constexpr int KB = 32;      // basis functions of a chunk (whole shells, padded to a multiple of 4)
constexpr int THREADS = 256;

template <int NT>
__host__ __device__ constexpr int ldb() { return 16 * NT + 4; }
template <int NT>
__host__ __device__ constexpr size_t smem_bytes() { return sizeof(double) * (size_t)KB * (LDA + ldb<NT>()); }

// A Gaussian shell with n = l + 1, l <= 2, of one electron: the operations of shell_eval_put with the products fused
// with their sums as the compiler fuses them in warp_basis, written out, so that the bits are the same
// wherever it is inlined and l is a constant.
template <int l>
__device__ __forceinline__ void gauss_shell5(const Sys<double> &s, int2 pr, double d0, double d1, double d2, double *o) {
  double r = sqrt(__dadd_rn(__fma_rn(d0, d0, __dmul_rn(d1, d1)), __dmul_rn(d2, d2)));
  if (r == 0.0) { r = 1e-30; d0 = r; }
  const double ri = 1.0 / r, rm1 = l == 0 ? 1.0 : l == 1 ? r : __dmul_rn(r, r), rm2 = __dmul_rn(rm1, ri), rm3 = __dmul_rn(rm2, ri);
  double R0 = 0, R1 = 0, R2 = 0;
#pragma unroll 2
  for (int p = pr.x; p < pr.x + pr.y; p++) {
    const double zr = __dmul_rn(__dmul_rn(2 * s.pz[p], r), r), ex = __dmul_rn(s.pc[p], exp(-0.5 * zr));
    R0 = __fma_rn(rm1, ex, R0);
    R1 = __dadd_rn(R1, __dmul_rn(__dmul_rn(rm2, __dadd_rn(l, -zr)), ex));
    R2 = __dadd_rn(R2, __dmul_rn(__dmul_rn(rm3, __fma_rn(__dadd_rn(zr, -(2 * l + 1)), zr, l * (l - 1))), ex));
  }
  const double ril = l == 0 ? 1.0 : l == 1 ? ri : __dmul_rn(ri, ri), d[3] = {d0, d1, d2};
  const double lap = __fma_rn(-__dmul_rn(__dmul_rn(l * (l + 1), ri), ri), R0, __fma_rn(2 * ri, R1, R2));
  // function S, its gradient G (zero where Z says so)
  auto put = [&](int sl, double S, const double *G, const int *Z) {
    const double Y = __dmul_rn(S, ril), lr = __dmul_rn(__dmul_rn(__dmul_rn(l * S, ril), ri), ri);
    o[sl * LDA] = __dmul_rn(Y, R0);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double a = __dmul_rn(__dmul_rn(Y, d[k]), ri);
      double v = __dmul_rn(a, R1);
      if (l > 0) {
        const double q = -__dmul_rn(lr, d[k]);
        v = __fma_rn(a, R1, __dmul_rn(Z[k] ? __fma_rn(G[k], ril, q) : q, R0));
      }
      o[sl * LDA + (k + 1) * EB] = v;
    }
    o[sl * LDA + 4 * EB] = __dmul_rn(Y, lap);
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
    const double s3 = 1.7320508075688772, x2 = __dmul_rn(d0, d0), y2 = __dmul_rn(d1, d1);
    const double sx = __dmul_rn(s3, d0), sy = __dmul_rn(s3, d1), sz = __dmul_rn(s3, d2);
    const double G[5][3] = {{-d0, -d1, 2 * d2}, {sz, 0.0, sx}, {0.0, sz, sy}, {sx, -sy, 0.0}, {sy, sx, 0.0}};
    const int Z[5][3] = {{1, 1, 1}, {1, 0, 1}, {0, 1, 1}, {1, 1, 0}, {1, 1, 0}};
    put(0, 0.5 * __dadd_rn(2 * __dmul_rn(d2, d2), -__dadd_rn(x2, y2)), G[0], Z[0]);
    put(1, __dmul_rn(sx, d2), G[1], Z[1]);
    put(2, __dmul_rn(sy, d2), G[2], Z[2]);
    put(3, __dmul_rn(0.5 * s3, __dadd_rn(x2, -y2)), G[3], Z[3]);
    put(4, __dmul_rn(sx, d1), G[4], Z[4]);
  }
}
// Any other shell (out of line: its registers are not those of the contraction, and the compiler fuses there
// what it fuses in warp_basis).
static __device__ __noinline__ void general_shell5(const Sys<double> &s, int ish, double x, double y, double z, double *o) {
  const double pt[3] = {x, y, z};
  shell_eval_put<double, 5>(s, ish, pt, [o](int sl, int c, double v) { o[sl * LDA + c * EB] = v; });
}

// Orbitals of 32 electrons of one spin (sp0 + blockIdx.y) per block: chunks of basis functions are formed in
// shared memory (lane = electron, a warp per shell, so that every lane runs the same shell) and
// contracted with the spin's coefficients by mma m8n8k4: 160 rows (5 channels x 32 electrons) by
// 16 NT orbitals, 8 warps as 4 (rows) x 2 (orbitals), 5 x NT tiles each.  The coefficients of a
// chunk arrive by cp.async while its basis functions are formed and are shared by the 32
// electrons (the warp-per-electron contraction streamed them from L2 once per 4 electrons).
// The rows are those of warp_basis and warp_orbitals to the last bit: the same basis functions, and the mma
// adds its four products in order, each by a fused multiply-add, so an orbital is summed over b as there --
// in order above 16 orbitals, in LB interleaved sums and their pairwise tree up to 16 (SPLIT = LB).  It has to
// be so: where psi nearly vanishes the inverse magnifies the last bit of a row by the condition number (ratios
// of an 80-electron cluster's first moves then differ by 3e-9), and the accelerated mover, whose proposals follow
// the drift, magnifies it again with every sweep (its walks came apart).
// What bounds it: the FP64 pipe (about a fourth of it the basis functions).  Measured (B200): 4096
// walkers of 128 electrons, 416 basis functions, 15.6 -> 7.2 ms; two sweeps of 1001 of 51 electrons 1.25 -> 0.42; 3001 of 20
// electrons, 65 functions, 0.32 -> 0.18.  Basis functions by shelltab.cuh's exponential and formulas took 6.0, 0.33 and
// 0.13 ms, and split the walks; shell_eval_put out of line 9.2 ms (indexed arrays in local memory).
// k_el_orb stays for more than 64 orbitals of a spin, and for one or two (32 or 16 interleaved sums each).
// chunk[k]: first shell, shells, first basis function, basis functions.
// ALL: the columns blockIdx.y * 16 NT onwards of all orbitals (s.call), for every electron, into all + w
// stride as [N][5][norb] instead, without the Slater matrices.
template <int NT, int SPLIT, bool ALL>
__global__ void __launch_bounds__(THREADS, 2) k_orb_tile(const __grid_constant__ Sys<double> s, State<double> st, const int4 *chunk, int nchunk,
                                                         int sp0, double *all, size_t stride) {
  static_assert(SPLIT == 1 || (NT == 1 && !ALL), "interleaved sums: up to 16 orbitals");
  extern __shared__ __align__(16) double sm[];
  double *phi = sm, *cf = sm + KB * LDA;
  constexpr int LDB = ldb<NT>();
  // sums of a warp: above 8 orbitals both warps of a row tile hold all of theirs, below they share them
  constexpr int NS = SPLIT <= 2 ? SPLIT : SPLIT / 2;
  const int sp = ALL ? 0 : sp0 + blockIdx.y, n = ALL ? s.N : (sp ? s.ndn : s.nup), e0 = sp ? s.nup : 0;
  const int col0 = ALL ? (int)blockIdx.y * 16 * NT : 0, ld = ALL ? s.norb : s.nocc[sp], no = ld - col0;
  const long long items = (long long)st.W * n, i0 = (long long)blockIdx.x * EB;
  if (i0 >= items) return;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5, rr = lane >> 2, kq = lane & 3;
  const int wm = wib >> 1, wn = wib & 1;
  const double *coef = ALL ? s.call + col0 : s.cocc[sp];
  double px[3] = {0, 0, 0};
  {
    long long it = i0 + lane;
    if (it >= items) it = items - 1;  // the last block's spare lanes repeat its last electron
    const int w = (int)(it / n), e = e0 + (int)(it - (long long)w * n);
    const double *x = st.x + ((size_t)w * s.N + e) * 3;
    px[0] = x[0]; px[1] = x[1]; px[2] = x[2];
  }
  const bool vec = ld % 2 == 0 && (reinterpret_cast<uintptr_t>(coef) & 15) == 0;
  double acc[5][NT * NS][2];
#pragma unroll
  for (int i = 0; i < 5; i++)
#pragma unroll
    for (int j = 0; j < NT * NS; j++) acc[i][j][0] = acc[i][j][1] = 0;
  for (int k = 0; k < nchunk; k++) {
    const int4 ch = chunk[k];
    const int nk4 = (ch.w + 3) & ~3;
    // coefficients of the chunk: rows [k][16 NT], zero past the orbitals and the basis functions
    if (vec) {
      constexpr int V = 8 * NT;
      for (int i = tid; i < nk4 * V; i += THREADS) {
        const int r = i / V, c = 2 * (i - r * V);
        double *dst = cf + r * LDB + c;
        if (r < ch.w && c < no) cp_async16(dst, coef + (size_t)(ch.z + r) * ld + c);
        else dst[0] = dst[1] = 0.0;
      }
    } else {
      for (int i = tid; i < nk4 * 16 * NT; i += THREADS) {
        const int r = i / (16 * NT), c = i - r * (16 * NT);
        cf[r * LDB + c] = (r < ch.w && c < no) ? coef[(size_t)(ch.z + r) * ld + c] : 0.0;
      }
    }
    cp_async_commit();
    for (int r = ch.w + wib; r < nk4; r += 8)
#pragma unroll
      for (int c = 0; c < 5; c++) phi[r * LDA + c * EB + lane] = 0.0;
    for (int q = wib; q < ch.y; q += 8) {
      const int ish = ch.x + q;
      const int4 sh = s.shell[ish];
      double *o = phi + (s.shb0[ish] - ch.z) * LDA + lane;
      if (sh.w != 1 || sh.y != sh.z + 1 || sh.z > 2) {
        general_shell5(s, ish, px[0], px[1], px[2], o);
        continue;
      }
      const int2 pr = s.shprim[ish];
      const double *cc = s.cent + 3 * sh.x;
      const double d0 = px[0] - cc[0], d1 = px[1] - cc[1], d2 = px[2] - cc[2];
      if (sh.z == 0) gauss_shell5<0>(s, pr, d0, d1, d2, o);
      else if (sh.z == 1) gauss_shell5<1>(s, pr, d0, d1, d2, o);
      else gauss_shell5<2>(s, pr, d0, d1, d2, o);
    }
    cp_async_wait<0>();
    __syncthreads();
    if constexpr (SPLIT == 1) {
      const double *ap = phi + kq * LDA + wm * 40 + rr, *bp = cf + kq * LDB + wn * 8 * NT + rr;
      for (int ks = 0; ks < nk4; ks += 4) {
        double a[5], b[NT];
#pragma unroll
        for (int i = 0; i < 5; i++) a[i] = ap[ks * LDA + 8 * i];
#pragma unroll
        for (int j = 0; j < NT; j++) b[j] = bp[ks * LDB + 8 * j];
#pragma unroll
        for (int i = 0; i < 5; i++)
#pragma unroll
          for (int j = 0; j < NT; j++) dmma_884(acc[i][j][0], acc[i][j][1], a[i], b[j]);
      }
    } else {
      // sum q takes the basis functions b = q mod SPLIT, four of them to an mma (zeros past the chunk)
      const double *ap = phi + wm * 40 + rr, *bp = cf + (SPLIT == 2 ? 8 * wn : 0) + rr;
      const int q0 = SPLIT == 2 ? 0 : NS * wn;
#pragma unroll
      for (int j = 0; j < NS; j++) {
        const int r0 = (q0 + j - ch.z) & (SPLIT - 1);
        for (int t = r0; t < ch.w; t += 4 * SPLIT) {
          const int r = t + SPLIT * kq;
          const bool in = r < ch.w;
          const double b = in ? bp[r * LDB] : 0.0;
#pragma unroll
          for (int i = 0; i < 5; i++) dmma_884(acc[i][j][0], acc[i][j][1], in ? ap[r * LDA + 8 * i] : 0.0, b);
        }
      }
    }
    __syncthreads();
  }
  // the interleaved sums by their pairwise tree; the second half of them from the other warp of the row tile
  if constexpr (SPLIT > 1) {
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int d = 1; d < NS; d <<= 1)
#pragma unroll
          for (int j = 0; j < NS; j += 2 * d) acc[i][j][h] += acc[i][j + d][h];
    if constexpr (SPLIT > 2) {
      double *ex = sm + (size_t)(32 * wm + lane) * 10;
      if (wn == 1)
#pragma unroll
        for (int i = 0; i < 5; i++) {
          ex[2 * i] = acc[i][0][0];
          ex[2 * i + 1] = acc[i][0][1];
        }
      __syncthreads();
      if (wn == 1) return;
#pragma unroll
      for (int i = 0; i < 5; i++) {
        acc[i][0][0] += ex[2 * i];
        acc[i][0][1] += ex[2 * i + 1];
      }
    }
  }
  const int nomax = s.nomax;
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const int row = wm * 40 + 8 * i + rr, ch = row / EB;
    const long long it = i0 + (row - ch * EB);
    if (it >= items) continue;
    const int w = (int)(it / n), eo = (int)(it - (long long)w * n);
    double *o = ALL ? all + (size_t)w * stride + ((size_t)eo * 5 + ch) * ld + col0
                    : st.orb5 + (((size_t)w * s.N + e0 + eo) * 5 + ch) * nomax;
    double *A = st.ainv + (size_t)w * st.astride + (sp ? s.nup * s.nup : 0) + (size_t)eo * n;
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = wn * 8 * NT + 8 * j + 2 * kq + h;
        if (c < no) o[c] = acc[i][j][h];
        if (!ALL && ch == 0 && c < n) A[c] = acc[i][j][h];
      }
  }
}

// Inversion of the Slater matrices (matinv, qmc/vmc/matinv.f90) in registers: a block of NM threads
// per (walker, spin), a thread per row, Gauss-Jordan with partial pivoting.  Step k eliminates the
// column that sits at register 0 and every row then shifts left by one with the new column of the
// inverse entering on the right, so no register is indexed at run time; rows are not exchanged (the
// pivot row of step k ends as row k of the inverse, its electron as that row's column).  The
// pivot row goes through shared memory once per step.  Rows and columns past n are those of the
// identity.  Replaces the elimination in shared memory, which read and wrote the whole matrix there
// in each of the n steps: 3.4 -> 1.0 ms for 4096 walkers with 64 x 64 matrices (now the latency of the
// n pivot steps), 0.087 -> 0.037 ms for 3001 with 10 x 10.
template <int NM>
__global__ void __launch_bounds__(NM) k_inv_reg(double *ainv, int astride, int nup, int ndn, int W, double *scr) {
  constexpr int NW = NM / 32;
  __shared__ __align__(16) double prow[2][NM];
  __shared__ double s_best[2][NW], s_ln[NW];
  __shared__ int s_bi[2][NW], s_piv[NM];
  const int w = blockIdx.x >> 1, sp = blockIdx.x & 1;
  if (w >= W) return;
  const int n = sp ? ndn : nup, t = threadIdx.x, lane = t & 31, wib = t >> 5;
  double *out = scr + (size_t)w * EL_SC + 4 + 2 * sp;
  if (n == 0) {
    if (t == 0) { out[0] = 0.0; out[1] = 1.0; }
    return;
  }
  double *g = ainv + (size_t)w * astride + (sp ? nup * nup : 0);
  double a[NM];
#pragma unroll
  for (int j = 0; j < NM; j++) a[j] = (t < n && j < n) ? g[t * n + j] : 0.0;
  bool used = t >= n;
  double mypiv = 1.0;
  int mycol = -1;
  for (int k = 0; k < n; k++) {
    const int b = k & 1;
    double best = used ? -1.0 : fabs(a[0]);
    if (!(best > -1.0)) best = -1.0;  // a NaN is no pivot
    int bi = t;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (NW > 1) {
      if (lane == 0) { s_best[b][wib] = best; s_bi[b][wib] = bi; }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < NW; q++)
        if (s_best[b][q] > best || (s_best[b][q] == best && s_bi[b][q] < bi)) { best = s_best[b][q]; bi = s_bi[b][q]; }
    }
    if (!(best > 0.0)) {  // singular (every thread sees the same): the matrix stays as it is
      if (t == 0) { out[0] = 0.0; out[1] = 0.0; }
      return;
    }
    if (t == bi) {
      used = true;
      mypiv = a[0];
      mycol = k;
      s_piv[k] = t;
      const double pinv = 1.0 / a[0];
#pragma unroll
      for (int j = 1; j < NM; j++) a[j - 1] = a[j] * pinv;
      a[NM - 1] = pinv;
#pragma unroll
      for (int j = 0; j < NM; j += 2) *(double2 *)&prow[b][j] = make_double2(a[j], a[j + 1]);
    }
    __syncthreads();
    if (t != bi) {
      const double f = a[0];
#pragma unroll
      for (int j = 0; j < NM; j += 2) {
        const double2 p = *(const double2 *)&prow[b][j];
        a[j] = (j + 1 < NM ? a[j + 1] : 0.0) - f * p.x;
        a[j + 1] = (j + 2 < NM ? a[j + 2] : 0.0) - f * p.y;
      }
    }
  }
  __syncthreads();
  // row of step mycol: inverse[mycol][electron of step m] = a[NM - n + m]
  if (t < n) {
#pragma unroll
    for (int j = 0; j < NM; j++) {
      const int m = j - (NM - n);
      if (m >= 0) g[mycol * n + s_piv[m]] = a[j];
    }
  }
  // ln|D| = sum ln|pivot|; sign: pivots below zero and the parity of the row order
  double ln = t < n ? log(fabs(mypiv)) : 0.0;
  int neg = (t < n && mypiv < 0) ? 1 : 0;
  if (t < n)
    for (int m = 0; m < mycol; m++) neg += s_piv[m] > t;  // inversions of the permutation
  ln = warp_sum(ln);
  neg = warp_sum(neg);
  if (lane == 0) { s_ln[wib] = ln; s_bi[0][wib] = neg; }
  __syncthreads();
  if (t == 0) {
    double l = 0;
    int q = 0;
    for (int i = 0; i < NW; i++) { l += s_ln[i]; q += s_bi[0][i]; }
    out[0] = l;
    out[1] = (q & 1) ? -1.0 : 1.0;
  }
}

}  // namespace ot

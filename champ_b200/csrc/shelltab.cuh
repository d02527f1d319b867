// shelltab.cuh -- the basis shells as the tiled FP64 kernels read them: packed records and primitives staged in
// shared memory, and an exponential for their Gaussians.
//
// Every warp of these kernels walks all shells once per point or electron.  From the tables in global
// memory that was a chain of dependent loads per shell which the small L1 beside their shared memory kept
// missing, and about 200 integer and control instructions per shell for 50 in FP64.
#pragma once
#include "kernels.cuh"

namespace stab {

// exp(x) for x <= 0 by table and polynomial (P. T. P. Tang, Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic, ACM TOMS 15, 1989): x = (64 m + j) ln2 / 64 + r, |r| <= ln2 / 128,
// exp(x) = 2^m t[j] (1 + r + r^2/2 + ... + r^5/120); the omitted term is below 4e-17.  Below -700 it
// returns 0: 1e-304 there, short of the -708 where the result would leave the normal range.
__device__ __forceinline__ double fast_exp(double x, const double *t) {
  const double magic = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer in the low word
  const double f = fma(x, 92.332482616893656877, magic);  // 64 / ln 2
  const int n = __double2loint(f);
  const double k = f - magic;
  // ln2 / 64 in two parts, the first short enough that k times it is exact
  const double r = fma(k, -2.8447437476627285e-11, fma(k, -0.010830424667801708, x));
  const double r2 = r * r;
  const double p = fma(r2, fma(r2, fma(8.3333333333333332e-3, r, 4.1666666666666664e-2), fma(0.16666666666666666, r, 0.5)), r);
  const double s = t[n & 63];
  const double e = __hiloint2double(__double2hiint(s) + ((n >> 6) << 20), __double2loint(s));
  return x < -700.0 ? 0.0 : fma(e, p, e);
}

struct Tab {
  const ShellRec *rec;
  const double2 *prim;
  const double *ex;
};
constexpr size_t TAB_MAX = 24 * 1024;  // larger tables stay in global memory
__host__ __device__ inline size_t tab_smem(int nshell, int nprim) {
  const size_t b = sizeof(ShellRec) * nshell + sizeof(double2) * nprim + sizeof(double) * 64;
  return b <= TAB_MAX ? b : 0;
}
// Copies the tables to base (shared memory, 16-byte aligned; tab_smem bytes) by the whole block, which must
// synchronise before it reads them; or points to global memory where they are too large.
__device__ inline Tab stage(const Sys<double> &s, void *base) {
  if (!tab_smem(s.nshell, s.nprim)) return Tab{s.srec, s.sprim, s.sexp};
  int4 *d = (int4 *)base;
  const int n0 = 2 * s.nshell, n1 = n0 + s.nprim, n2 = n1 + 32;
  for (int i = threadIdx.x; i < n2; i += blockDim.x)
    d[i] = i < n0 ? ((const int4 *)s.srec)[i] : i < n1 ? ((const int4 *)s.sprim)[i - n0] : ((const int4 *)s.sexp)[i - n1];
  return Tab{(const ShellRec *)d, (const double2 *)(d + n0), (const double *)(d + n1)};
}

// Radial factor of a shell over r^l (so that a basis function is S_lm(d) times it).
static __device__ __noinline__ double general_radial(const Sys<double> &s, int ish, double r) {
  double R[3];
  if (r == 0.0) r = 1e-30;
  shell_radial<double, false>(s, ish, r, R);
  return R[0] * ipow(1.0 / r, s.shell[ish].z);
}
// Gaussian shells (exponents ascending): a primitive is not formed (but for the second of a pair) where its
// exponential is below e^-70 = 4e-31 of that of the widest primitive that weighs -- at least 1e-8 of the shell's
// largest weight -- hence below 4e-23 of that primitive's value.  Two primitives at a time: an exponential is a chain of ten dependent FP64
// operations, and the callers have too few warps in flight to fill it.  Small walkers' evaluation 0.97 -> 0.91 ms
// (8192 of 8 electrons), their DMC step 3.28 -> 3.18 ms; the projected points of 3001 walkers of 20 electrons
// 0.53 -> 0.52 ms.
__device__ __forceinline__ double gauss_radial(const Tab &T, const ShellRec &h, double r2) {
  double g = 0;
  int p = h.p0;
  const int end = p + h.np;
  if (h.np & 1) {
    const double2 q = T.prim[p++];
    g = q.y * fast_exp(-q.x * r2, T.ex);
  }
#pragma unroll 1
  for (; p < end; p += 2) {
    const double2 q0 = T.prim[p], q1 = T.prim[p + 1];
    if ((q0.x - h.zmin) * r2 > 70.0) break;
    const double e0 = fast_exp(-q0.x * r2, T.ex), e1 = fast_exp(-q1.x * r2, T.ex);
    g += q0.y * e0;
    g += q1.y * e1;
  }
  return g;
}
__device__ __forceinline__ double factor(const Sys<double> &s, const Tab &T, int ish, const ShellRec &h, double r2) {
  return h.kind == 1 ? gauss_radial(T, h, r2) : general_radial(s, ish, sqrt(r2));
}

// The radial part with what gradients and Laplacians need: q (the factor above), q'/r and q'' + (2l + 2) q'/r, so
// that a function S_lm(d) q has the gradient grad S q + S d (q'/r) and the Laplacian S times the third.
struct Rad {
  double q, t, lap;
};
static __device__ __noinline__ Rad general_rad(const Sys<double> &s, int ish, double r2) {
  const int l = s.shell[ish].z;
  double r = sqrt(r2), R[3];
  if (r == 0.0) r = 1e-30;
  shell_radial<double, true>(s, ish, r, R);
  const double ri = 1.0 / r, ril = ipow(ri, l);
  return Rad{R[0] * ril, (R[1] - l * R[0] * ri) * ri * ril, (R[2] + 2 * ri * R[1] - l * (l + 1) * ri * ri * R[0]) * ril};
}
__device__ __forceinline__ Rad gauss_rad(const Tab &T, const ShellRec &h, double r2) {
  double g = 0, gp = 0, gpp = 0;
  int p = h.p0;
  const int end = p + h.np;
  if (h.np & 1) {
    const double2 q = T.prim[p++];
    g = q.y * fast_exp(-q.x * r2, T.ex);
    gp = -q.x * g;
    gpp = -q.x * gp;
  }
#pragma unroll 1
  for (; p < end; p += 2) {
    const double2 q0 = T.prim[p], q1 = T.prim[p + 1];
    if ((q0.x - h.zmin) * r2 > 70.0) break;
    const double e0 = q0.y * fast_exp(-q0.x * r2, T.ex), e1 = q1.y * fast_exp(-q1.x * r2, T.ex);
    const double z0 = q0.x * e0, z1 = q1.x * e1;
    g += e0;
    gp -= z0;
    gpp += q0.x * z0;
    g += e1;
    gp -= z1;
    gpp += q1.x * z1;
  }
  return Rad{g, 2 * gp, 4 * r2 * gpp + (4 * h.l + 6) * gp};
}

}  // namespace stab

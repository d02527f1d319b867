// eltile.cu -- launchers of the staged evaluation's tensor-core parts (jastile.cuh, orbtile.cuh).
#include <algorithm>

#include "ctx.h"
#include "jastile.cuh"
#include "orbtile.cuh"
#include "nlpoints.cuh"
#include "pgtile.cuh"

static size_t gproj_smem(const champ_ctx *c) { return sizeof(double) * pt::GP_LD * (size_t)((c->nomax + 3) & ~3); }

// The attributes of the kernels that the context launches.
template <int NORD, bool MD>
static int fin_attrs(const champ_ctx *c) {
  int rc = c->fin_wpw == 1   ? kernel_smem(pt::k_fin_points<NORD, MD, 1>, 128, c->fin_smem)
           : c->fin_wpw == 8 ? kernel_smem(pt::k_fin_points<NORD, MD, 8>, 256, c->fin_smem)
           : c->fin_wpw      ? kernel_smem(pt::k_fin_points<NORD, MD, 4>, 128, c->fin_smem)
                             : CHAMP_OK;
  if (!rc && c->fin_wpw && c->nloc > 0) rc = kernel_smem(pt::k_gproj<MD>, 128, gproj_smem(c));
  return rc;
}
template <int NORD>
static int el_attrs(const champ_ctx *c) {
  int rc = c->md.multidet ? fin_attrs<NORD, true>(c) : fin_attrs<NORD, false>(c);
  if constexpr (NORD > 1) {
    if (c->jas_wpw == 1) {
      if (!rc) rc = kernel_smem(jt::k_jas_tile<NORD, 1, false>, 128, c->jas_smem);
      if (!rc) rc = kernel_smem(jt::k_jas_tile<NORD, 1, true>, 128, c->jas_smem);
    } else if (c->jas_wpw) {
      if (!rc) rc = kernel_smem(jt::k_jas_tile<NORD, jt::WARPS, false>, 128, c->jas_smem);
      if (!rc) rc = kernel_smem(jt::k_jas_tile<NORD, jt::WARPS, true>, 128, c->jas_smem);
    }
  }
  return rc;
}
static int orb_class(int nocc) { return nocc > 32 ? 5 : nocc > 16 ? 4 : nocc > 8 ? 3 : nocc > 4 ? 2 : nocc > 2 ? 1 : 0; }
static int orb_attrs(int k) {
  return k == 5   ? kernel_smem(ot::k_orb_tile<4, 1, false>, ot::THREADS, ot::smem_bytes<4>())
         : k == 4 ? kernel_smem(ot::k_orb_tile<2, 1, false>, ot::THREADS, ot::smem_bytes<2>())
         : k == 3 ? kernel_smem(ot::k_orb_tile<1, 2, false>, ot::THREADS, ot::smem_bytes<1>())
         : k == 2 ? kernel_smem(ot::k_orb_tile<1, 4, false>, ot::THREADS, ot::smem_bytes<1>())
         : k == 1 ? kernel_smem(ot::k_orb_tile<1, 8, false>, ot::THREADS, ot::smem_bytes<1>())
                  : CHAMP_OK;
}

// Which parts serve the context's system, their shared memory, and the chunks of whole shells that
// the orbital part forms at a time.
int el_tile_setup(champ_ctx *c) {
  const int nmax = std::max(c->nup, c->ndn), nomax = c->nomax;
  c->inv_nm = nmax <= 32 ? 32 : 64;
  if ((c->nordc == 4 || c->nordc == 5) && c->nct == 1) {
    // one warp per walker up to 32 electrons (4 tiles of rows, so that a block's warps would have one each
    // and wait for one another), else a block per walker
    const int wpw = c->N <= 32 ? 1 : jt::WARPS;
    const size_t b = jt::Dims(c->N, c->C, wpw).bytes() * (wpw == 1 ? jt::WARPS : 1);
    if (b <= 200 * 1024) {
      c->jas_wpw = wpw;
      c->jas_smem = b;
    }
  }
  if (nomax <= 64) {
    std::vector<int4> sh(c->nshell), ch;
    std::vector<int> b0(c->nshell);
    CK(cudaMemcpy(sh.data(), c->sd.shell, sizeof(int4) * c->nshell, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(b0.data(), c->sd.shb0, sizeof(int) * c->nshell, cudaMemcpyDeviceToHost));
    for (int i = 0; i < c->nshell; i++) {
      const int nb = 2 * sh[i].z + 1;
      if (ch.empty() || ch.back().w + nb > ot::KB) ch.push_back(make_int4(i, 0, b0[i], 0));
      ch.back().y++;
      ch.back().w += nb;
    }
    int4 *d = nullptr;
    CK(cudaMalloc(&d, sizeof(int4) * ch.size()));
    c->allocs.push_back(d);
    CK(cudaMemcpy(d, ch.data(), sizeof(int4) * ch.size(), cudaMemcpyHostToDevice));
    c->orb_chunk = d;
    c->orb_nchunk = (int)ch.size();
    c->orb_nt = nomax <= 16 ? 1 : nomax <= 32 ? 2 : 4;
    // one or two orbitals of a spin: 32 or 16 interleaved sums each (k_orb_tile holds up to 8)
    auto served = [&](int no) { return no == 0 || no > 2; };
    c->orb_tile = served(c->sd.nocc[0]) && served(c->sd.nocc[1]);
  }
  if (c->nordc <= 1 || c->nct == 1) {
    const int wpw = c->N <= 32 ? 1 : c->N <= 64 ? 4 : 8;
    c->fin_nrow = std::min(c->N * c->C * std::max(c->sd.nshc, 1), wpw == 1 ? 256 : 768);
    const size_t b = pt::Dims(c->N, c->C, c->nordc, c->fin_nrow, wpw == 1).bytes() * (wpw == 1 ? 4 : 1) +
                     stab::tab_smem(c->sd.nshell, c->sd.nprim);
    if (b <= 200 * 1024) {
      c->fin_wpw = wpw;
      c->fin_smem = b;
    }
  }
  int rc = c->nordc == 4 ? el_attrs<4>(c) : c->nordc == 5 ? el_attrs<5>(c) : el_attrs<0>(c);
  for (int sp = 0; sp < 2; sp++)
    if (!rc && c->orb_tile) rc = orb_attrs(orb_class(c->sd.nocc[sp]));
  return rc;
}

template <int NORD>
static int jas(champ_ctx *c, const State<double> &st, bool vo) {
  const int W = st.W;
  if (c->jas_wpw == 1) {
    const dim3 g((W + jt::WARPS - 1) / jt::WARPS);
    if (vo) jt::k_jas_tile<NORD, 1, true><<<g, 32 * jt::WARPS, c->jas_smem, c->stream>>>(c->sd, st);
    else jt::k_jas_tile<NORD, 1, false><<<g, 32 * jt::WARPS, c->jas_smem, c->stream>>>(c->sd, st);
  } else {
    if (vo) jt::k_jas_tile<NORD, jt::WARPS, true><<<W, 32 * jt::WARPS, c->jas_smem, c->stream>>>(c->sd, st);
    else jt::k_jas_tile<NORD, jt::WARPS, false><<<W, 32 * jt::WARPS, c->jas_smem, c->stream>>>(c->sd, st);
  }
  CK(cudaGetLastError());
  return CHAMP_OK;
}
int el_tile_jas(champ_ctx *c, const State<double> &st, bool vo) {
  return c->nordc == 4 ? jas<4>(c, st, vo) : jas<5>(c, st, vo);
}

// Spins sp0 .. sp0 + ns - 1, which have orbitals of the same class (orb_class).
template <int NT, int SPLIT>
static int orb(champ_ctx *c, const State<double> &st, int sp0, int ns) {
  const int n = std::max(sp0 ? 0 : c->nup, sp0 + ns > 1 ? c->ndn : 0);
  const long long items = (long long)st.W * n;
  if (items == 0) return CHAMP_OK;
  const dim3 g((unsigned)((items + ot::EB - 1) / ot::EB), ns);
  ot::k_orb_tile<NT, SPLIT, false><<<g, ot::THREADS, ot::smem_bytes<NT>(), c->stream>>>(c->sd, st, c->orb_chunk, c->orb_nchunk, sp0, nullptr, 0);
  CK(cudaGetLastError());
  return CHAMP_OK;
}
static int orb_spins(champ_ctx *c, const State<double> &st, int k, int sp0, int ns) {
  return k == 5 ? orb<4, 1>(c, st, sp0, ns) : k == 4 ? orb<2, 1>(c, st, sp0, ns) : k == 3 ? orb<1, 2>(c, st, sp0, ns)
       : k == 2 ? orb<1, 4>(c, st, sp0, ns) : orb<1, 8>(c, st, sp0, ns);
}
int el_tile_orb(champ_ctx *c, const State<double> &st) {
  const int k0 = orb_class(c->sd.nocc[0]), k1 = orb_class(c->sd.nocc[1]);
  if (k0 == k1) return orb_spins(c, st, k0, 0, 2);
  int rc = orb_spins(c, st, k0, 0, 1);
  if (!rc) rc = orb_spins(c, st, k1, 1, 1);
  return rc;
}

int el_tile_inv(champ_ctx *c, const State<double> &st) {
  const unsigned g = 2 * (unsigned)st.W;
  if (c->inv_nm == 32) ot::k_inv_reg<32><<<g, 32, 0, c->stream>>>(st.ainv, st.astride, c->nup, c->ndn, st.W, st.el_sc);
  else ot::k_inv_reg<64><<<g, 64, 0, c->stream>>>(st.ainv, st.astride, c->nup, c->ndn, st.W, st.el_sc);
  CK(cudaGetLastError());
  return CHAMP_OK;
}

template <int NORD, bool MD>
static int fin(champ_ctx *c, const State<double> &st, bool outputs, bool stats, const ElRot &rot, bool tables_only, const pt::Tape &tape) {
  const int W = st.W;
  if (MD) {
    pt::k_md_tables<<<(W + 3) / 4, 128, 0, c->stream>>>(c->sd, st);
    CK(cudaGetLastError());
  }
  if (c->nloc > 0 && !tables_only) {
    pt::k_gproj<MD><<<2 * W, 128, gproj_smem(c), c->stream>>>(c->sd, st);
    CK(cudaGetLastError());
  }
  if (c->fin_wpw == 1)
    pt::k_fin_points<NORD, MD, 1><<<(W + 3) / 4, 128, c->fin_smem, c->stream>>>(c->sd, st, c->fin_nrow, outputs, stats, rot, tables_only, tape);
  else if (c->fin_wpw == 8)
    pt::k_fin_points<NORD, MD, 8><<<W, 256, c->fin_smem, c->stream>>>(c->sd, st, c->fin_nrow, outputs, stats, rot, tables_only, tape);
  else
    pt::k_fin_points<NORD, MD, 4><<<W, 128, c->fin_smem, c->stream>>>(c->sd, st, c->fin_nrow, outputs, stats, rot, tables_only, tape);
  CK(cudaGetLastError());
  return CHAMP_OK;
}
template <int NORD>
static int fin_n(champ_ctx *c, const State<double> &st, bool outputs, bool stats, const ElRot &rot, bool tables_only, const pt::Tape &tape) {
  return c->md.multidet ? fin<NORD, true>(c, st, outputs, stats, rot, tables_only, tape)
                        : fin<NORD, false>(c, st, outputs, stats, rot, tables_only, tape);
}
int el_tile_fin(champ_ctx *c, const State<double> &st, bool outputs, bool stats, const ElRot &rot, bool tables_only) {
  const pt::Tape t{};
  return c->nordc == 4 ? fin_n<4>(c, st, outputs, stats, rot, tables_only, t)
       : c->nordc == 5 ? fin_n<5>(c, st, outputs, stats, rot, tables_only, t) : fin_n<0>(c, st, outputs, stats, rot, tables_only, t);
}

// ---- parameter gradient (pgtile.cuh) -----------------------------------------------------------
// The forward pass as the staged evaluation with a tape: e-e-n terms on the tensor cores.
// (The points' coefficients for the orbital-resolved local energy wait in the place of its orbitals, which
// are formed after their use.)  One determinant: the orbital and CSF derivatives of a multi-determinant
// state go through the reference determinant's inverse, which near its nodes amplifies any change of
// rounding beyond the derivatives themselves.
bool pg_tile_fwd_ok(const champ_ctx *c) {
  const bool room = c->ncsfp + c->norbp == 0 || c->C * c->nquad <= 5 * c->norb;
  return c->el_staged && c->jas_wpw && c->fin_wpw && c->orb_tile && !c->md.multidet && room;
}
// The reverse sweep in FP64: one e-e parameter set.
bool pg_tile_bwd_ok(const champ_ctx *c) {
  return pg_tile_fwd_ok(c) && c->prec == CHAMP_PREC_FP64 && c->par.nspin2b == 1 && c->pg_raw;
}

static size_t pgnl_smem(const champ_ctx *c) {
  return sizeof(double) * 4 * (size_t)c->nbasis + stab::tab_smem(c->sd.nshell, c->sd.nprim);
}

template <int NORD>
static int bwd_attrs(const champ_ctx *c) {
  const bool one = c->jas_wpw == 1;
  const size_t b = pt::Dims(c->N, c->C, NORD, 0).bytes() * (one ? 4 : 1);
  int rc = one ? kernel_smem(pg::k_pg_points<NORD, 1>, 128, b) : kernel_smem(pg::k_pg_points<NORD, 4>, 128, b);
  if (!rc) rc = one ? kernel_smem(pg::k_pg_pairs<NORD, 1>, 128, c->jas_smem) : kernel_smem(pg::k_pg_pairs<NORD, 4>, 128, c->jas_smem);
  return rc;
}

int pg_tile_setup(champ_ctx *c) {
  if (!pg_tile_fwd_ok(c)) return CHAMP_OK;
  std::vector<int4> sh(c->nshell);
  CK(cudaMemcpy(sh.data(), c->sd.shell, sizeof(int4) * c->nshell, cudaMemcpyDeviceToHost));
  std::vector<int> order(c->nshell);
  for (int i = 0; i < c->nshell; i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return sh[a].z < sh[b].z; });
  CK(cudaMalloc(&c->shell_order, sizeof(int) * c->nshell));
  c->allocs.push_back(c->shell_order);
  CK(cudaMemcpy(c->shell_order, order.data(), sizeof(int) * c->nshell, cudaMemcpyHostToDevice));
  int rc = kernel_smem(ot::k_orb_tile<4, 1, true>, ot::THREADS, ot::smem_bytes<4>());
  if (!rc) rc = kernel_smem(pg::k_pg_nl, 128, pgnl_smem(c));
  if (rc || c->prec != CHAMP_PREC_FP64 || c->par.nspin2b != 1) return rc;
  rc = c->nordc == 4 ? bwd_attrs<4>(c) : bwd_attrs<5>(c);
  if (rc) return rc;
  CK(cudaMalloc(&c->pg_raw, sizeof(double) * 3 * (size_t)c->np_raw * c->wmax));
  c->allocs.push_back(c->pg_raw);
  return CHAMP_OK;
}

static ElRot fixed_rotation(const champ_ctx *c) {
  ElRot r{};
  for (int i = 0; i < 9; i++) r.R[i] = c->rot[i];
  return r;
}

int pg_tile_fwd(champ_ctx *c) {
  State<double> st = c->std_;
  st.W = c->W;
  const int W = c->W;
  const ElRot rot = fixed_rotation(c);
  int rc = el_tile_jas(c, st, false);
  if (!rc) rc = el_tile_orb(c, st);
  if (!rc) rc = el_tile_inv(c, st);
  pt::Tape t;
  t.v = c->pg_tv;
  t.c = c->pg_tc;
  t.el = c->pg_el;
  t.n = c->pg_tn;
  t.b = c->pg_scr ? c->pg_scr + (size_t)c->N * c->nbasis : nullptr;
  t.bstride = c->scr_stride;
  if (!rc) rc = c->nordc == 4 ? fin_n<4>(c, st, false, false, rot, false, t) : fin_n<5>(c, st, false, false, rot, false, t);
  if (rc) return rc;
  c->orb5_valid = true;
  if (c->nloc > 0) {
    pg::k_pg_nl<<<W, 128, pgnl_smem(c), c->stream>>>(c->sd, st, c->pg_tv, c->pg_tn, c->pg_tc, c->pg_scr,
                                                                             c->scr_stride, t.b, rot, c->shell_order);
  } else {
    CK(cudaMemset2DAsync(c->pg_tv + 3 * c->N, sizeof(double) * 4 * c->N, 0, sizeof(double) * c->N, W, c->stream));
    if (c->pg_scr)
      CK(cudaMemset2DAsync(c->pg_scr, sizeof(double) * c->scr_stride, 0, sizeof(double) * (size_t)c->N * c->nbasis, W, c->stream));
  }
  CK(cudaGetLastError());
  if (c->pg_scr) {
    const long long items = (long long)W * c->N;
    const dim3 g((unsigned)((items + ot::EB - 1) / ot::EB), (c->norb + 63) / 64);
    double *all = c->pg_scr + (size_t)c->N * c->nbasis;
    ot::k_orb_tile<4, 1, true><<<g, ot::THREADS, ot::smem_bytes<4>(), c->stream>>>(c->sd, st, c->orb_chunk, c->orb_nchunk, 0, all, c->scr_stride);
    CK(cudaGetLastError());
    const long long el = items * c->norb;
    pg::k_pg_blocal<<<(unsigned)std::min<long long>((el + 255) / 256, 148 * 32), 256, 0, c->stream>>>(c->sd, st, c->pg_scr, c->scr_stride);
    CK(cudaGetLastError());
  }
  return CHAMP_OK;
}

template <int NORD>
static int bwd(champ_ctx *c) {
  State<double> st = c->std_;
  st.W = c->W;
  const int W = c->W, P = c->np_raw, wpw = c->jas_wpw;
  CK(cudaMemsetAsync(c->pg_raw, 0, sizeof(double) * 3 * (size_t)P * W, c->stream));
  const dim3 g(wpw == 1 ? (W + 3) / 4 : W);
  if (c->nloc > 0) {
    const size_t b = pt::Dims(c->N, c->C, NORD, 0).bytes() * (wpw == 1 ? 4 : 1);
    if (wpw == 1) pg::k_pg_points<NORD, 1><<<g, 128, b, c->stream>>>(c->sd, st, c->pg_tn, c->pg_tc, c->pg_raw, P, fixed_rotation(c));
    else pg::k_pg_points<NORD, 4><<<g, 128, b, c->stream>>>(c->sd, st, c->pg_tn, c->pg_tc, c->pg_raw, P, fixed_rotation(c));
    CK(cudaGetLastError());
  }
  if (wpw == 1) pg::k_pg_pairs<NORD, 1><<<g, 128, c->jas_smem, c->stream>>>(c->sd, st, c->pg_tv, c->pg_raw, P);
  else pg::k_pg_pairs<NORD, 4><<<g, 128, c->jas_smem, c->stream>>>(c->sd, st, c->pg_tv, c->pg_raw, P);
  CK(cudaGetLastError());
  const int nt = make_terms(NORD).n, nab = P - nt, jo = c->nfree - c->nparm_jas;
  const long long n = (long long)W * c->nparm_jas;
  if (n > 0)
    pg::k_pg_out<<<(unsigned)std::min<long long>((n + 127) / 128, 148 * 32), 128, 0, c->stream>>>(c->sd, W, c->pg_raw, P, nab, nt, c->nfree, jo,
                                                                                               c->pg_dl, c->pg_de);
  CK(cudaGetLastError());
  return CHAMP_OK;
}
int pg_tile_bwd(champ_ctx *c) { return c->nordc == 4 ? bwd<4>(c) : bwd<5>(c); }

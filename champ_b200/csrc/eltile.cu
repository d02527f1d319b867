// eltile.cu -- launchers of the staged evaluation's tensor-core parts (jastile.cuh, orbtile.cuh).
#include <algorithm>

#include "ctx.h"
#include "jastile.cuh"
#include "orbtile.cuh"
#include "nlpoints.cuh"

template <class K>
static int big_smem(K kern, size_t bytes) {
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
  return CHAMP_OK;
}

template <int NORD>
static int fin_attrs_n() {
  int rc = big_smem(pt::k_fin_points<NORD, false, 1>, 200 * 1024);
  if (!rc) rc = big_smem(pt::k_fin_points<NORD, false, 4>, 200 * 1024);
  if (!rc) rc = big_smem(pt::k_fin_points<NORD, true, 1>, 200 * 1024);
  if (!rc) rc = big_smem(pt::k_fin_points<NORD, true, 4>, 200 * 1024);
  return rc;
}
static int fin_attrs(champ_ctx *c) {
  int rc = c->nordc == 4 ? fin_attrs_n<4>() : c->nordc == 5 ? fin_attrs_n<5>() : fin_attrs_n<0>();
  if (!rc) rc = big_smem(pt::k_gproj<false>, 200 * 1024);
  if (!rc) rc = big_smem(pt::k_gproj<true>, 200 * 1024);
  return rc;
}

// Which parts serve the context's system, their shared memory, and the chunks of whole shells that
// the orbital part forms at a time.
int el_tile_setup(champ_ctx *c) {
  const int nmax = std::max(c->nup, c->ndn), nomax = c->nomax;
  c->inv_nm = nmax <= 32 ? 32 : 64;
  if ((c->nordc == 4 || c->nordc == 5) && c->nct == 1) {
    // one warp per walker up to 32 electrons (4 tiles of rows), else a block per walker
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
  }
  if (c->nordc <= 1 || c->nct == 1) {
    // every shell's smallest exponent among the primitives that weigh in it
    std::vector<int2> pr(c->nshell);
    CK(cudaMemcpy(pr.data(), c->sd.shprim, sizeof(int2) * c->nshell, cudaMemcpyDeviceToHost));
    int np = 0;
    for (const int2 &p : pr) np = std::max(np, p.x + p.y);
    std::vector<double> z(np), wt(np), zm(c->nshell, 0.0);
    CK(cudaMemcpy(z.data(), c->sd.pz, sizeof(double) * np, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(wt.data(), c->sd.pc, sizeof(double) * np, cudaMemcpyDeviceToHost));
    for (int i = 0; i < c->nshell; i++) {
      double wmax = 0, m = 1e300;
      for (int p = pr[i].x; p < pr[i].x + pr[i].y; p++) wmax = std::max(wmax, std::fabs(wt[p]));
      for (int p = pr[i].x; p < pr[i].x + pr[i].y; p++)
        if (std::fabs(wt[p]) >= 1e-8 * wmax) m = std::min(m, z[p]);
      zm[i] = m < 1e300 ? m : 0.0;
    }
    double *d = nullptr;
    CK(cudaMalloc(&d, sizeof(double) * c->nshell));
    c->allocs.push_back(d);
    CK(cudaMemcpy(d, zm.data(), sizeof(double) * c->nshell, cudaMemcpyHostToDevice));
    c->shell_zmin = d;
    const int wpw = c->N <= 32 ? 1 : 4;
    c->fin_nrow = std::min(c->N * c->C * std::max(c->sd.nshc, 1), wpw == 1 ? 256 : 768);
    const size_t b = pt::Dims(c->N, c->C, c->nordc, c->fin_nrow).bytes() * (wpw == 1 ? 4 : 1);
    if (b <= 200 * 1024) {
      c->fin_wpw = wpw;
      c->fin_smem = b;
    }
  }
  int rc = fin_attrs(c);
  for (auto k : {jt::k_jas_tile<4, 1, false>, jt::k_jas_tile<4, 1, true>, jt::k_jas_tile<4, jt::WARPS, false>,
                 jt::k_jas_tile<4, jt::WARPS, true>, jt::k_jas_tile<5, 1, false>, jt::k_jas_tile<5, 1, true>,
                 jt::k_jas_tile<5, jt::WARPS, false>, jt::k_jas_tile<5, jt::WARPS, true>})
    if (!rc) rc = big_smem(k, 200 * 1024);
  if (!rc) rc = big_smem(ot::k_orb_tile<1>, ot::smem_bytes<1>());
  if (!rc) rc = big_smem(ot::k_orb_tile<2>, ot::smem_bytes<2>());
  if (!rc) rc = big_smem(ot::k_orb_tile<4>, ot::smem_bytes<4>());
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

int el_tile_orb(champ_ctx *c, const State<double> &st) {
  const int nmax = std::max(c->nup, c->ndn);
  const long long items = (long long)st.W * nmax;
  const dim3 g((unsigned)((items + ot::EB - 1) / ot::EB), 2);
  switch (c->orb_nt) {
  case 1: ot::k_orb_tile<1><<<g, ot::THREADS, ot::smem_bytes<1>(), c->stream>>>(c->sd, st, c->orb_chunk, c->orb_nchunk); break;
  case 2: ot::k_orb_tile<2><<<g, ot::THREADS, ot::smem_bytes<2>(), c->stream>>>(c->sd, st, c->orb_chunk, c->orb_nchunk); break;
  default: ot::k_orb_tile<4><<<g, ot::THREADS, ot::smem_bytes<4>(), c->stream>>>(c->sd, st, c->orb_chunk, c->orb_nchunk);
  }
  CK(cudaGetLastError());
  return CHAMP_OK;
}

int el_tile_inv(champ_ctx *c, const State<double> &st) {
  const unsigned g = 2 * (unsigned)st.W;
  if (c->inv_nm == 32) ot::k_inv_reg<32><<<g, 32, 0, c->stream>>>(st.ainv, st.astride, c->nup, c->ndn, st.W, st.el_sc);
  else ot::k_inv_reg<64><<<g, 64, 0, c->stream>>>(st.ainv, st.astride, c->nup, c->ndn, st.W, st.el_sc);
  CK(cudaGetLastError());
  return CHAMP_OK;
}

template <int NORD, bool MD>
static int fin(champ_ctx *c, const State<double> &st, bool outputs, bool stats, const ElRot &rot, bool tables_only) {
  const int W = st.W;
  if (MD) {
    pt::k_md_tables<<<(W + 3) / 4, 128, 0, c->stream>>>(c->sd, st);
    CK(cudaGetLastError());
  }
  if (c->nloc > 0 && !tables_only) {
    const size_t sm = sizeof(double) * pt::GP_LD * (size_t)((c->nomax + 3) & ~3);
    pt::k_gproj<MD><<<2 * W, 128, sm, c->stream>>>(c->sd, st);
    CK(cudaGetLastError());
  }
  if (c->fin_wpw == 1)
    pt::k_fin_points<NORD, MD, 1><<<(W + 3) / 4, 128, c->fin_smem, c->stream>>>(c->sd, st, c->shell_zmin, c->fin_nrow, outputs, stats, rot, tables_only);
  else
    pt::k_fin_points<NORD, MD, 4><<<W, 128, c->fin_smem, c->stream>>>(c->sd, st, c->shell_zmin, c->fin_nrow, outputs, stats, rot, tables_only);
  CK(cudaGetLastError());
  return CHAMP_OK;
}
template <int NORD>
static int fin_n(champ_ctx *c, const State<double> &st, bool outputs, bool stats, const ElRot &rot, bool tables_only) {
  return c->md.multidet ? fin<NORD, true>(c, st, outputs, stats, rot, tables_only)
                        : fin<NORD, false>(c, st, outputs, stats, rot, tables_only);
}
int el_tile_fin(champ_ctx *c, const State<double> &st, bool outputs, bool stats, const ElRot &rot, bool tables_only) {
  return c->nordc == 4 ? fin_n<4>(c, st, outputs, stats, rot, tables_only)
       : c->nordc == 5 ? fin_n<5>(c, st, outputs, stats, rot, tables_only) : fin_n<0>(c, st, outputs, stats, rot, tables_only);
}

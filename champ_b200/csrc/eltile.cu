// eltile.cu -- launchers of the staged evaluation's tensor-core parts (jastile.cuh, orbtile.cuh).
#include <algorithm>

#include "ctx.h"
#include "jastile.cuh"
#include "orbtile.cuh"

template <class K>
static int big_smem(K kern, size_t bytes) {
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
  return CHAMP_OK;
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
  int rc = CHAMP_OK;
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

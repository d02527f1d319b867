// eltile.cu -- launchers of the staged evaluation's tensor-core parts (jastile.cuh, orbtile.cuh).
#include <algorithm>

#include "ctx.h"
#include "jastile.cuh"

template <class K>
static int big_smem(K kern, size_t bytes) {
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
  return CHAMP_OK;
}

// Which parts serve the context's system, and their shared memory.
int el_tile_setup(champ_ctx *c) {
  if ((c->nordc == 4 || c->nordc == 5) && c->nct == 1) {
    // one warp per walker up to 32 electrons (4 tiles of rows), else a block per walker
    const int wpw = c->N <= 32 ? 1 : jt::WARPS;
    const size_t b = jt::Dims(c->N, c->C, wpw).bytes() * (wpw == 1 ? jt::WARPS : 1);
    if (b <= 200 * 1024) {
      c->jas_wpw = wpw;
      c->jas_smem = b;
    }
  }
  int rc = CHAMP_OK;
  for (auto k : {jt::k_jas_tile<4, 1, false>, jt::k_jas_tile<4, 1, true>, jt::k_jas_tile<4, jt::WARPS, false>,
                 jt::k_jas_tile<4, jt::WARPS, true>, jt::k_jas_tile<5, 1, false>, jt::k_jas_tile<5, 1, true>,
                 jt::k_jas_tile<5, jt::WARPS, false>, jt::k_jas_tile<5, jt::WARPS, true>})
    if (!rc) rc = big_smem(k, 200 * 1024);
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

// movebatch.cu -- launchers of the batched single-electron moves (movebatch.cuh).
#include <algorithm>

#include "ctx.h"
#include "movebatch.cuh"

namespace {

// up to 32 electrons a warp per walker, else a block per walker
int warps_per_walker(const champ_ctx *c) { return c->N <= 32 ? 1 : 4; }
size_t walk_smem(const champ_ctx *c) {
  return sizeof(double) * ((size_t)c->nmax * c->nmax + 3 * c->N) * (warps_per_walker(c) == 1 ? 4 : 1);
}
template <class T, int NORD>
size_t pairs_smem(const champ_ctx *c) {
  const int wpw = warps_per_walker(c);
  return mv::PairDims<T, NORD>(c->N, c->C).bytes(wpw) * (wpw == 1 ? 4 : 1);
}
template <class T, int NT>
size_t prop_smem(const champ_ctx *c) {
  return mv::prop_smem<T, NT>() + (sizeof(T) == 8 ? stab::tab_smem(c->sd.nshell, c->sd.nprim) : 0);
}
mv::Scr scratch(const champ_ctx *c) { return mv::Scr{c->std_.orb5, 5 * (size_t)c->N * c->nomax, c->N, c->nomax}; }

template <class T, int NORD>
int setup(champ_ctx *c) {
  const size_t sp = pairs_smem<T, NORD>(c), sw = walk_smem(c);
  if (sp > 200 * 1024 || sw > 200 * 1024) return CHAMP_OK;
  const bool one = warps_per_walker(c) == 1;
  int rc = one ? kernel_smem(mv::k_mv_pairs<T, NORD, 1>, 128, sp) : kernel_smem(mv::k_mv_pairs<T, NORD, 4>, 128, sp);
  if (!rc) rc = one ? kernel_smem(mv::k_mv_walk<T, 1>, 128, sw) : kernel_smem(mv::k_mv_walk<T, 4>, 128, sw);
  if (!rc)
    rc = c->orb_nt == 1   ? kernel_smem(mv::k_mv_prop<T, 1>, 256, prop_smem<T, 1>(c))
         : c->orb_nt == 2 ? kernel_smem(mv::k_mv_prop<T, 2>, 256, prop_smem<T, 2>(c))
                          : kernel_smem(mv::k_mv_prop<T, 4>, 256, prop_smem<T, 4>(c));
  if (!rc) c->move_batch = 1;
  return rc;
}

template <class T, int NORD>
int sweep(champ_ctx *c, const State<T> &st, uint64_t seed, uint64_t isweep, double step) {
  const int W = st.W, N = c->N, wpw = warps_per_walker(c);
  const mv::Scr q = scratch(c);
  const Sys<T> &s = sysof<T>(c);
  const long long items = (long long)W * N, per = (long long)W * c->nmax;
  mv::k_mv_draw<<<(unsigned)((items + 255) / 256), 256, 0, c->stream>>>(st.x, W, N, q, seed, isweep, step);
  CK(cudaGetLastError());
  const dim3 g((unsigned)((per + mv::PB - 1) / mv::PB), 2);
  switch (c->orb_nt) {
  case 1: mv::k_mv_prop<T, 1><<<g, 256, prop_smem<T, 1>(c), c->stream>>>(s, W, q, c->orb_chunk, c->orb_nchunk); break;
  case 2: mv::k_mv_prop<T, 2><<<g, 256, prop_smem<T, 2>(c), c->stream>>>(s, W, q, c->orb_chunk, c->orb_nchunk); break;
  default: mv::k_mv_prop<T, 4><<<g, 256, prop_smem<T, 4>(c), c->stream>>>(s, W, q, c->orb_chunk, c->orb_nchunk);
  }
  CK(cudaGetLastError());
  const size_t sp = pairs_smem<T, NORD>(c), sw = walk_smem(c);
  if (wpw == 1) {
    mv::k_mv_pairs<T, NORD, 1><<<(W + 3) / 4, 128, sp, c->stream>>>(s, st, q);
    CK(cudaGetLastError());
    mv::k_mv_walk<T, 1><<<(W + 3) / 4, 128, sw, c->stream>>>(st, q, N, c->nup, c->nmax);
  } else {
    mv::k_mv_pairs<T, NORD, 4><<<W, 128, sp, c->stream>>>(s, st, q);
    CK(cudaGetLastError());
    mv::k_mv_walk<T, 4><<<W, 128, sw, c->stream>>>(st, q, N, c->nup, c->nmax);
  }
  CK(cudaGetLastError());
  return CHAMP_OK;
}

}  // namespace

// Whether the context's Gaussian sweeps run as batched moves: a staged evaluation to follow, one
// determinant, one centre type (and at most MAXC_NL centres) where there are e-e-n terms, and in mixed
// precision more than 16 orbitals per spin (with fewer, propose() splits the basis functions of an
// orbital among lanes: other FP32 sums).
int move_batch_setup(champ_ctx *c) {
  const bool een = c->nordc > 1;
  if (!c->el_staged || c->md.multidet || !c->orb_chunk || (een && (c->nct != 1 || c->C > MAXC_NL))) return CHAMP_OK;
  if (scratch(c).need() > scratch(c).stride || c->N > 128) return CHAMP_OK;
  if (c->prec == CHAMP_PREC_MIXED) {
    if (c->nup <= 16 || c->ndn <= 16) return CHAMP_OK;
    return c->nordc == 4 ? setup<float, 4>(c) : c->nordc == 5 ? setup<float, 5>(c) : setup<float, 0>(c);
  }
  return c->nordc == 4 ? setup<double, 4>(c) : c->nordc == 5 ? setup<double, 5>(c) : setup<double, 0>(c);
}

int move_batch_sweep(champ_ctx *c, uint64_t seed, uint64_t isweep, double step) {
  c->orb5_valid = false;  // the scratch is the FP64 state's orbital rows
  if (c->prec == CHAMP_PREC_MIXED) {
    State<float> st = c->stf;
    st.W = c->W;
    return c->nordc == 4 ? sweep<float, 4>(c, st, seed, isweep, step)
         : c->nordc == 5 ? sweep<float, 5>(c, st, seed, isweep, step) : sweep<float, 0>(c, st, seed, isweep, step);
  }
  State<double> st = c->std_;
  st.W = c->W;
  return c->nordc == 4 ? sweep<double, 4>(c, st, seed, isweep, step)
       : c->nordc == 5 ? sweep<double, 5>(c, st, seed, isweep, step) : sweep<double, 0>(c, st, seed, isweep, step);
}

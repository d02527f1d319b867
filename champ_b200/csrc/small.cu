// small.cu -- launchers of the small walkers' kernels (small.cuh).
#include <algorithm>

#include "ctx.h"
#include "nlpoints.cuh"
#include "small.cuh"

namespace {

template <int NORD>
int attrs(const champ_ctx *c) {
  const size_t b = sizeof(double) * (size_t)sm::Lay(c->N, c->C, c->nordc).total() * 16 + stab::tab_smem(c->sd.nshell, c->sd.nprim);
  int rc = CHAMP_OK;
  for (auto k : {sm::k_small<NORD, sm::EVAL>, sm::k_small<NORD, sm::GAUSS>, sm::k_small<NORD, sm::DMC>, sm::k_small<NORD, sm::DMC_EL>,
                 sm::k_small_tmove<NORD>})
    if (!rc) rc = kernel_smem(k, 128, b);
  if (!rc) rc = kernel_smem(sm::k_small_accel<NORD>, 128, b + sizeof(double) * 16 * 5 * sm::ACH);
  return rc;
}

// Threads of a block: 128 (16 walkers), fewer while the walkers would not reach every SM.
int threads(const champ_ctx *c, int W) {
  const int sm = c->num_sms > 0 ? c->num_sms : 148;
  int t = 128;
  while (t > 32 && (W * sm::GS + t - 1) / t < sm) t >>= 1;
  return t;
}

constexpr int ACCEL = 6, TMOVE = 100;  // beside k_small's modes
template <int NORD>
int run(champ_ctx *c, const State<double> &st, int mode, const sm::Args &A, int W) {
  const int t = threads(c, W), per = t / sm::GS;
  const size_t smem = sizeof(double) * (size_t)sm::Lay(c->N, c->C, c->nordc, mode == ACCEL ? 5 * sm::ACH : 0).total() * per +
                      stab::tab_smem(c->sd.nshell, c->sd.nprim);
  const dim3 g((W + per - 1) / per);
  switch (mode) {
  case sm::EVAL: sm::k_small<NORD, sm::EVAL><<<g, t, smem, c->stream>>>(c->sd, st, A); break;
  case sm::GAUSS: sm::k_small<NORD, sm::GAUSS><<<g, t, smem, c->stream>>>(c->sd, st, A); break;
  case sm::DMC: sm::k_small<NORD, sm::DMC><<<g, t, smem, c->stream>>>(c->sd, st, A); break;
  case ACCEL: sm::k_small_accel<NORD><<<g, t, smem, c->stream>>>(c->sd, st, A); break;
  case sm::DMC_EL: sm::k_small<NORD, sm::DMC_EL><<<g, t, smem, c->stream>>>(c->sd, st, A); break;
  default: sm::k_small_tmove<NORD><<<g, t, smem, c->stream>>>(c->sd, st, A);
  }
  CK(cudaGetLastError());
  return CHAMP_OK;
}
int run(champ_ctx *c, const State<double> &st, int mode, const sm::Args &A, int W) {
  return c->nordc == 4 ? run<4>(c, st, mode, A, W) : c->nordc == 5 ? run<5>(c, st, mode, A, W) : run<0>(c, st, mode, A, W);
}

}  // namespace

// Small walkers: state resident in shared memory (kd), one determinant, at most 8 electrons and 4 of a
// spin, one centre type where there are e-e-n terms.
int small_setup(champ_ctx *c) {
  if (!c->kd.lay.resident || c->md.multidet || c->nmax > sm::NO || c->N > sm::NE || (c->nordc > 1 && c->nct != 1)) return CHAMP_OK;
  if (sizeof(double) * (size_t)sm::Lay(c->N, c->C, c->nordc).total() * 16 + sizeof(double) * 16 * 5 * sm::ACH + stab::TAB_MAX > 200 * 1024) return CHAMP_OK;
  std::vector<int4> sh(c->nshell);
  CK(cudaMemcpy(sh.data(), c->sd.shell, sizeof(int4) * c->nshell, cudaMemcpyDeviceToHost));
  std::vector<int> order(c->nshell);
  for (int i = 0; i < c->nshell; i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return sh[a].z < sh[b].z; });
  int *d = nullptr;
  CK(cudaMalloc(&d, sizeof(int) * std::max(c->nshell, 1)));
  c->allocs.push_back(d);
  CK(cudaMemcpy(d, order.data(), sizeof(int) * c->nshell, cudaMemcpyHostToDevice));
  c->small_order = d;
  std::vector<int> b0(c->nshell);
  CK(cudaMemcpy(b0.data(), c->sd.shb0, sizeof(int) * c->nshell, cudaMemcpyDeviceToHost));
  std::vector<int4> ch;
  for (int i = 0; i < c->nshell; i++) {
    const int nb = 2 * sh[i].z + 1;
    if (ch.empty() || ch.back().w + nb > sm::ACH) ch.push_back(make_int4(i, 0, b0[i], 0));
    ch.back().y++;
    ch.back().w += nb;
  }
  int4 *dc = nullptr;
  CK(cudaMalloc(&dc, sizeof(int4) * std::max<size_t>(ch.size(), 1)));
  c->allocs.push_back(dc);
  CK(cudaMemcpy(dc, ch.data(), sizeof(int4) * ch.size(), cudaMemcpyHostToDevice));
  c->small_chunk = dc;
  c->small_nchunk = (int)ch.size();
  const int rc = c->nordc == 4 ? attrs<4>(c) : c->nordc == 5 ? attrs<5>(c) : attrs<0>(c);
  if (!rc) c->small = 1;
  return rc;
}

// How many walkers.  A walker on 8 lanes takes longer than on 32 (an evaluation with nonlocal points 440 us
// against 230), so the kernels pay where a warp per walker fills the SMs more than once: walkers above a number
// per SM, by what the operation spends on points, which split worst.  Measured (B200, 148 SMs; dimer and C2
// of 8 electrons, calls of 2 sweeps or 4 steps, us here against a warp per walker):
//   evaluation      2400 walkers 1325 / 1084, 3600 1492 / 1395, 8192 with mixed-precision sweeps 2790 / 3100;
//   Gaussian moves  1800 1142 / 1035, 2400 1250 / 1379;
//   accelerated     600 1897 / 1631 and 2091 / 1672, 900 1985 / 2430 and 2226 / 2273, 8192 9354 / 27012 and 10026 / 20893;
//   DMC, T-moves    1800 2776 / 2571 and 2351 / 2294, 2400 2834 / 4399 and 2557 / 3881; T-moves 1800 5758 / 4956 and
//                   5234 / 6122, 2400 5946 / 7552 and 5448 / 9157 (a warp per walker holds 16 per SM at once).
// Without a pseudopotential there are no points: Gaussian moves of the Be-like atom 120 / 139 at 60 walkers,
// 154 / 276 at 2400.
// Evaluations of walkers that a caller supplies, and the E_L after accelerated sweeps in FP32, stay with a warp per
// walker for their bits: near a node the inverse magnifies the rounding of its rows (drifts of 8192 unequilibrated
// walkers to 5e-11), and the moves start from it.
bool small_serves(const champ_ctx *c, SmallOp op, int W) {
  if (!c->small) return false;
  if (c->nloc == 0 && op == SmallOp::Gauss) return true;
  const int sm = c->num_sms > 0 ? c->num_sms : 148;
  const int per = op == SmallOp::Eval ? 32 : op == SmallOp::Gauss ? 14 : op == SmallOp::Accel ? 6 : 16;
  return W > per * sm;
}

// the E_L after a sweep of Gaussian moves, and its statistics
int small_eval(champ_ctx *c, const State<double> &st, const ElRot &rot) {
  sm::Args A;
  A.order = c->small_order;
  A.rot = rot;
  return run(c, st, sm::EVAL, A, st.W);
}
int small_vmc(champ_ctx *c, const State<double> &st, const OpArgs &a) {
  sm::Args A;
  A.order = c->small_order;
  A.nsweep = a.nsweep;
  A.seed = a.seed;
  A.sweep0 = a.sweep0;
  A.step = a.step;
  A.mv = c->mover;
  A.chunk = c->small_chunk;
  A.nchunk = c->small_nchunk;
  A.reinv = c->reinv_every;
  return run(c, st, c->mover.kind == 6 ? ACCEL : sm::GAUSS, A, st.W);
}
int small_dmc(champ_ctx *c, const State<double> &st, bool moves) {
  sm::Args A;
  A.order = c->small_order;
  A.P = c->dpar;
  A.D = c->dA;
  return run(c, st, moves ? sm::DMC : sm::DMC_EL, A, c->dpar.wmax);
}
int small_tmove(champ_ctx *c, const State<double> &st, const OpArgs &a) {
  sm::Args A;
  A.order = c->small_order;
  A.tau = a.tau;
  A.variant = a.variant;
  A.seed = a.seed;
  A.sweep0 = a.sweep0;
  A.nw = a.dmc ? c->dA.nw : nullptr;
  A.step_dev = a.dmc ? c->dA.ctr : nullptr;
  A.moved = a.moved;
  return run(c, st, TMOVE, A, a.dmc ? c->dpar.wmax : st.W);
}

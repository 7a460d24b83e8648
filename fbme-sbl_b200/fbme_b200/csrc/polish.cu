// Active-set polish of the FBME plans: top-K support from the UAMP score,
// exact reduced posterior with the Type-II evidence, evidence gate, EM
// updates of the active variances and the noise, the residual support
// exchange, fixed-budget diagnostics and the outputs.
//
// Follows torch_sbl/solver.py:1926-2021 (driver), 3961-4510
// (_uamp_active_em_polish, the branches the plans reach), 3591-3779
// (_active_posterior_with_evidence), 2898-2931 (Cholesky loading),
// 3219-3317 (deletion gain), 3408-3496 (fixed-budget residuals),
// 2081-2126 (effective DOF, support mask).
//
// Everything except the exchange scoring is K-dimensional (K <= 32): one
// block per scene, lane i owning row i.  Fourier atoms are never
// materialised:
//   Gram      G[k][l] = D1[(n1k-n1l) mod N1] * D2[(n2k-n2l) mod N2]
//             (Dirichlet kernels summed in FP64 once per plan),
//   A_S^H y   = (A^H y)[S], a gather of the backprojection,
//   ||y - A_S mu||^2 = ||y||^2 - 2 Re(c^H mu) + mu^H G mu   (FP64),
//   A^H(y - A_S mu)[n] = (A^H y)[n] - sum_k mu_k D(n - n_k)  (exchange).
// The evidence (log-determinant + quadratic form) is accumulated in FP64.
#include <math.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "topk.cuh"

namespace fbme {

constexpr float kTinyP = 1.17549435e-38f;
constexpr float kEpsP = 1.1920929e-07f;
constexpr int kMaxEval = 8;

struct PolishScene {
  int active[kMaxPolish];      // base active set (best accepted)
  int work_active[kMaxPolish]; // active set of the next evaluation
  float work_gamma[kMaxPolish];
  float work_noise;
  float2 best_mean[kMaxPolish];
  float best_pv[kMaxPolish];
  float best_dd[kMaxPolish];
  float best_gamma[kMaxPolish];
  float best_noise;
  double best_nle;
  float trace[kMaxEval];
  int evals;        // evaluations done
  int pending;      // exchange proposed at the previous transition
  int exch_acc;     // accepted exchanges
  int has_best;
};

size_t polish_state_bytes() { return sizeof(PolishScene); }

struct PolishArgs {
  BatchShape s;
  DevConfig c;
  PolishBuffers p;
};

FBME_DEV float2 dirichlet2(const float2* d1, const float2* d2, int n1, int n2, int a1, int a2,
                           int b1, int b2) {
  int i1 = a1 - b1, i2 = a2 - b2;
  if (i1 < 0) i1 += n1;
  if (i2 < 0) i2 += n2;
  return cmul(d1[i1], d2[i2]);
}

// Gram entry G[i][j] of atoms (a1, a2) and (b1, b2): the separable
// Dirichlet product for the full prefix block, or the 2-D table of an
// observation mask (global memory, L2-resident).
FBME_DEV float2 gram_at(const PolishArgs& A, const float2* d1, const float2* d2, int a1, int a2, int b1,
                        int b2) {
  if (A.p.gram2d) {
    int i1 = a1 - b1, i2 = a2 - b2;
    if (i1 < 0) i1 += A.s.n1;
    if (i2 < 0) i2 += A.s.n2;
    return __ldg(A.p.gram2d + static_cast<long long>(i1) * A.s.n2 + i2);
  }
  return dirichlet2(d1, d2, A.s.n1, A.s.n2, a1, a2, b1, b2);
}

// Copy the Dirichlet tables of a scene shape into shared memory: 8-byte
// asynchronous copies, all in flight before the one wait (a warp copying
// one element per lane at a time waited on every round trip).
FBME_DEV void load_dirichlet(const PolishArgs& A, float2* d1, float2* d2) {
  for (int i = threadIdx.x; i < A.s.n1; i += blockDim.x)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(d1 + i)), "l"(A.p.dir1 + i) : "memory");
  for (int i = threadIdx.x; i < A.s.n2; i += blockDim.x)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(d2 + i)), "l"(A.p.dir2 + i) : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
}

// One scene's K-dimensional algebra runs on a block of kPolishWarps warps:
// lane i owns row i, warp w the columns w, w + 8, w + 16, w + 24 of every
// row.  Its cost is the serial chain of the factorisation, so the block is
// there to shorten a step, not to add throughput: four entries of a row and
// of the inverse a thread instead of up to 32 each.  Measured (B200, K = 32):
// the three polish launches of one Stable scene 138 us in a single warp, 60 us
// so; of a 512-scene replay 157 -> 128 us.  Every entry of the factorisation
// keeps its operations and their order; the FP64 sums of the residual energy
// are added per warp first (residual_energy).
constexpr int kPolishWarps = 8;
constexpr int kPolishThreads = 32 * kPolishWarps;
constexpr int kPolishCols = kMaxPolish / kPolishWarps;  // columns of a row per thread

struct PolishShared {
  float2 M[kMaxPolish][kMaxPolish + 1];  // the system, for its transpose
  float2 L[kMaxPolish][kMaxPolish + 1];  // its Cholesky factor by columns: L[q][i] is entry (i, q)
  float rl[kMaxPolish];                  // 1 / L[q][q]
  float eqv[kMaxPolish];                 // squared column norms of L^-1
  float2 mean[kMaxPolish];
  double ev[3][kMaxPolish];              // logarithms of the evidence
  double log_nu;
  double2 gm[kPolishWarps][kMaxPolish];  // G mu, one partial sum per warp
  int status;
};

// Column q of the factorisation: its owner warp arrives, the others wait.
FBME_DEV void column_arrive(int q) {
  asm volatile("bar.arrive %0, %1;" ::"r"(1 + (q & 1)), "n"(kPolishThreads) : "memory");
}
FBME_DEV void column_sync(int q) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + (q & 1)), "n"(kPolishThreads) : "memory");
}

// Exact reduced posterior + negative log evidence for the work set, on the
// whole block; every warp returns the same values: in lane k mean_k, pv_k,
// dd_k; nle (all lanes).  Factorisation failures go to S.status.
struct EvalOut {
  float2 mean;
  float pv, dd;
  double nle;
  float dscale;  // equilibration scale sqrt(S_kk) of lane k's row
};

// Complex updates of the factorisation with their rounding spelled out (the
// first product fused, then one rounded sum), so that every kernel holding
// them gives the same bits however the compiler contracts; the reduced
// systems of close atoms are ill-conditioned enough to show the difference.
FBME_DEV float2 add_mul(float2 v, float2 a, float2 b) {  // v + a b
  return make_float2(__fadd_rn(v.x, fmaf(a.x, b.x, -__fmul_rn(a.y, b.y))),
                     __fadd_rn(v.y, fmaf(a.x, b.y, __fmul_rn(a.y, b.x))));
}
FBME_DEV float2 sub_mul(float2 v, float2 a, float2 b) {  // v - a b
  return make_float2(__fsub_rn(v.x, fmaf(a.x, b.x, -__fmul_rn(a.y, b.y))),
                     __fsub_rn(v.y, fmaf(a.x, b.y, __fmul_rn(a.y, b.x))));
}
FBME_DEV float2 sub_mulc(float2 v, float2 a, float2 b) {  // v - a conj(b)
  return make_float2(__fsub_rn(v.x, fmaf(a.x, b.x, __fmul_rn(a.y, b.y))),
                     __fsub_rn(v.y, fmaf(a.y, b.x, -__fmul_rn(a.x, b.y))));
}
FBME_DEV float2 sub_cmul(float2 v, float2 a, float2 b) {  // v - conj(a) b
  return make_float2(__fsub_rn(v.x, fmaf(a.x, b.x, __fmul_rn(a.y, b.y))),
                     __fsub_rn(v.y, fmaf(a.x, b.y, -__fmul_rn(a.y, b.x))));
}

FBME_DEV EvalOut evaluate(const PolishArgs& A, PolishShared& S, const float2* d1, const float2* d2, int K,
                          int my_idx, float my_gamma, float nu, float2 my_c, float data_energy) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const BatchShape& s = A.s;
  const bool on = lane < K;
  const int n1i = my_idx / s.n2, n2i = my_idx % s.n2;
  // One reciprocal per scale, reused by multiplication: a division here is
  // a full IEEE sequence with a slow-path branch, on the critical path.
  const float inv_nu = 1.0f / nu, inv_g = 1.0f / my_gamma;
  // system S = diag(1/gamma) + G / nu, Hermitian-symmetrised
  float2 r[kPolishCols];
#pragma unroll
  for (int u = 0; u < kPolishCols; ++u) {
    const int j = w + kPolishWarps * u;
    const int n1j = __shfl_sync(0xffffffffu, n1i, j), n2j = __shfl_sync(0xffffffffu, n2i, j);
    r[u] = make_float2(0.f, 0.f);
    if (on && j < K) {
      const float2 g = gram_at(A, d1, d2, n1i, n2i, n1j, n2j);
      r[u] = make_float2(g.x * inv_nu, g.y * inv_nu);
      if (j == lane) r[u].x = __fadd_rn(r[u].x, inv_g);
      S.M[lane][j] = r[u];
    }
  }
  __syncthreads();
  const float diag = on ? S.M[lane][lane].x : 1.0f;
  const float dscale = on ? sqrtf(fmaxf(diag, kTinyP)) : 1.0f;
  const float inv_d = 1.0f / dscale;
  // deterministic diagonal loading: multiplier * eps * mean|Re diag|
  float dsum = on ? fabsf(diag * (inv_d * inv_d)) : 0.f;
  dsum = warp_sum(dsum);
  const float scale = fmaxf(dsum / static_cast<float>(K), kTinyP);
  const float jitter = A.c.jitter * (kEpsP * scale);
  // equilibrate: E[i][j] = S[i][j] / (d_i d_j).  S is exactly Hermitian
  // after its symmetrisation and the scale is the same product for (i, j)
  // and (j, i), so E is exactly Hermitian as well.
#pragma unroll
  for (int u = 0; u < kPolishCols; ++u) {
    const int j = w + kPolishWarps * u;
    const float f = inv_d * __shfl_sync(0xffffffffu, inv_d, j);
    if (on && j < K) {
      const float2 b = S.M[j][lane];
      r[u] = make_float2(0.5f * (r[u].x + b.x) * f, 0.5f * (r[u].y - b.y) * f);
      if (j == lane) r[u].x = __fadd_rn(r[u].x, jitter);
    }
  }
  // Cholesky, lower, right-looking, and in the same pass over q the inverse
  // factor X = L^-1 and the forward solve L z = c / nu / d (in every warp).  A
  // thread's entry r[u] is first the system's, updated by the columns left
  // of its own, then (once its column is posted) the sum over k of
  // L[lane][k] X[k][j], final for row q at step q, when row q of X lies in
  // lane q of the same warp.  The chain that sets the time is column q ->
  // entry (q+1, q+1) -> square root, reciprocal -> column q+1, so the warp
  // that owns column q+1 takes it first, posts it, arrives at the column's
  // barrier without waiting there, and makes the step's other updates after
  // it (one barrier a step for all: 75 us for those three launches).  Columns
  // stay where they are posted and the barrier ids alternate: a warp can
  // reach the barrier of column q+2 only after every warp passed column q's.
  const float2 rhs = on ? make_float2(my_c.x * inv_nu, my_c.y * inv_nu) : make_float2(0.f, 0.f);
  float2 z = make_float2(rhs.x * inv_d, rhs.y * inv_d);
  float eqv[kPolishCols];
#pragma unroll
  for (int u = 0; u < kPolishCols; ++u) eqv[u] = 0.f;
  int failed = 0;
  auto post = [&](int q, float2& v) {
    const float sdiag = __shfl_sync(0xffffffffu, v.x, q);
    const float piv = sqrtf(sdiag > 0.f ? sdiag : kTinyP);
    const float rq = 1.0f / piv;
    const float2 a = make_float2(lane == q ? piv : lane > q ? v.x * rq : 0.f, lane > q ? v.y * rq : 0.f);
    S.L[q][lane] = a;
    S.rl[q] = rq;  // the same value from every lane
    __syncwarp();  // this warp reads the column without waiting at its barrier
    column_arrive(q);
    v = make_float2(0.f, 0.f);
    failed |= sdiag > 0.f ? 0 : isfinite(sdiag) ? FBME_STATUS_CHOLESKY : FBME_STATUS_NONFINITE;
  };
  if (w == 0) post(0, r[0]);
#pragma unroll
  for (int uq = 0; uq < kPolishCols; ++uq) {
#pragma unroll 1
    for (int wq = 0; wq < kPolishWarps; ++wq) {
      const int q = kPolishWarps * uq + wq;
      if (q >= K) break;
      if (w != wq) column_sync(q);
      const float2 a = S.L[q][lane];  // column q: L[lane][q]
      const float rlq = S.rl[q];
      const int next = q + 1 < K ? q + 1 : -1;
      if (wq + 1 < kPolishWarps) {
        if (w == wq + 1 && next > 0) {
          if (lane >= next) r[uq] = sub_mulc(r[uq], a, S.L[q][next]);
          post(next, r[uq]);
        }
      } else if (uq + 1 < kPolishCols) {
        if (w == 0 && next > 0) {
          if (lane >= next) r[uq + 1] = sub_mulc(r[uq + 1], a, S.L[q][next]);
          post(next, r[uq + 1]);
        }
      }
      // the rest of the step, without branches: right of column q the
      // system's update, else the inverse's (u == uq: by warp)
#pragma unroll
      for (int u = 0; u < kPolishCols; ++u) {
        const int j = w + kPolishWarps * u;
        const bool right = u > uq || (u == uq && w > wq);
        float2 v = r[u];
        if (u >= uq) {
          const float2 t = sub_mulc(r[u], a, S.L[q][j]);
          if (right && j != next && lane >= j) v = t;
        }
        if (u <= uq) {
          float2 xq = make_float2(__shfl_sync(0xffffffffu, r[u].x, q), __shfl_sync(0xffffffffu, r[u].y, q));
          xq = j == q ? make_float2(rlq, 0.f) : make_float2(-xq.x * rlq, -xq.y * rlq);
          const float e = __fadd_rn(eqv[u], fmaf(xq.x, xq.x, __fmul_rn(xq.y, xq.y)));
          const float2 t = add_mul(r[u], a, xq);
          eqv[u] = right ? eqv[u] : e;
          if (!right && lane > q) v = t;
        }
        r[u] = v;
      }
      const float2 zs = make_float2(z.x * rlq, z.y * rlq);
      const float2 zq = make_float2(__shfl_sync(0xffffffffu, zs.x, q), __shfl_sync(0xffffffffu, zs.y, q));
      const float2 zt = sub_mul(z, a, zq);
      z = lane == q ? zs : lane > q ? zt : z;
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int u = 0; u < kPolishCols; ++u) S.eqv[w + kPolishWarps * u] = eqv[u];
  }
  if (failed && lane == 0) atomicOr(&S.status, failed);
  // warp 7: L^H w = z, mu = w / d; warps 0-3 the evidence's logarithms
  if (w == kPolishWarps - 1) {
    const float rl = on ? S.rl[lane] : 1.0f;
    float2 v = z;
#pragma unroll 1
    for (int q0 = kMaxPolish - 8; q0 >= 0; q0 -= 8) {
      float2 l[8];  // L[q][lane], ahead of the chain
#pragma unroll
      for (int i = 0; i < 8; ++i) l[i] = S.L[lane][q0 + i];
#pragma unroll
      for (int i = 7; i >= 0; --i) {
        const int q = q0 + i;
        if (lane == q) v = make_float2(v.x * rl, v.y * rl);
        const float2 vq = make_float2(__shfl_sync(0xffffffffu, v.x, q), __shfl_sync(0xffffffffu, v.y, q));
        if (lane < q && q < K) v = sub_cmul(v, l[i], vq);
      }
    }
    S.mean[lane] = make_float2(v.x * inv_d, v.y * inv_d);
  } else if (w == 0) {
    S.ev[0][lane] = on ? log(static_cast<double>(fmaxf(S.L[lane][lane].x, kTinyP))) : 0.0;
  } else if (w == 1) {
    S.ev[1][lane] = on ? log(static_cast<double>(dscale)) : 0.0;
  } else if (w == 2) {
    S.ev[2][lane] = on ? log(static_cast<double>(my_gamma)) : 0.0;
  } else if (w == 3) {
    const double l = log(static_cast<double>(nu));
    if (lane == 0) S.log_nu = l;
  }
  __syncthreads();
  EvalOut o;
  o.dscale = dscale;
  o.mean = on ? S.mean[lane] : make_float2(0.f, 0.f);
  o.pv = on ? fmaxf(S.eqv[lane] * (inv_d * inv_d), 0.f) : 0.f;
  o.dd = on ? fmaxf((my_gamma - o.pv) * (inv_g * inv_g), 0.f) : 0.f;
  // evidence (FP64 accumulation)
  double ld = S.ev[0][lane] + S.ev[1][lane], lg = S.ev[2][lane];
  double qd = on ? static_cast<double>(rhs.x) * o.mean.x + static_cast<double>(rhs.y) * o.mean.y : 0.0;
  ld = warp_sum(ld);
  lg = warp_sum(lg);
  qd = warp_sum(qd);
  const double logdet = observed_samples(s, A.c) * S.log_nu + lg + 2.0 * ld;
  double quad = static_cast<double>(data_energy) / nu - qd;
  if (quad < 0.0) quad = 0.0;
  o.nle = logdet + quad;
  if (!isfinite(o.nle) && threadIdx.x == 0) atomicOr(&S.status, FBME_STATUS_NONFINITE);
  return o;
}

// ||y - A_S mu||^2 by the Gram identity, FP64, on the whole block (every
// warp returns the sum): warp w adds the columns j = w, w + 8, ... of G mu.
using GramSums = double2[kPolishWarps][kMaxPolish];
FBME_DEV double residual_energy(const PolishArgs& A, GramSums& gm, const float2* d1, const float2* d2, int K,
                                int my_idx, float2 my_mu, float2 my_c, float data_energy) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const BatchShape& s = A.s;
  const int n1i = my_idx / s.n2, n2i = my_idx % s.n2;
  double gr = 0.0, gi = 0.0;  // (G mu)_i
#pragma unroll
  for (int u = 0; u < kPolishCols; ++u) {
    const int j = w + kPolishWarps * u;
    const int n1j = __shfl_sync(0xffffffffu, n1i, j), n2j = __shfl_sync(0xffffffffu, n2i, j);
    const float mjx = __shfl_sync(0xffffffffu, my_mu.x, j);
    const float mjy = __shfl_sync(0xffffffffu, my_mu.y, j);
    if (lane < K && j < K) {
      const float2 g = gram_at(A, d1, d2, n1i, n2i, n1j, n2j);
      gr += static_cast<double>(g.x) * mjx - static_cast<double>(g.y) * mjy;
      gi += static_cast<double>(g.x) * mjy + static_cast<double>(g.y) * mjx;
    }
  }
  __syncthreads();  // an earlier call's sums have been read
  gm[w][lane] = make_double2(gr, gi);
  __syncthreads();
  double cross = 0.0, quad = 0.0;
  if (lane < K) {
    cross = static_cast<double>(my_c.x) * my_mu.x + static_cast<double>(my_c.y) * my_mu.y;
    gr = gi = 0.0;
#pragma unroll
    for (int v = 0; v < kPolishWarps; ++v) {
      const double2 t = gm[v][lane];
      gr += t.x;
      gi += t.y;
    }
    quad = my_mu.x * gr + my_mu.y * gi;  // Re(conj(mu_i) (G mu)_i)
  }
  cross = warp_sum(cross);
  quad = warp_sum(quad);
  double e = static_cast<double>(data_energy) - 2.0 * cross + quad;
  return e > 0.0 ? e : 0.0;
}

// Deletion gain of one active atom (solver.py:3247-3276).
FBME_DEV float deletion_gain(float2 mean, float pv, float gamma) {
  const float g = fmaxf(gamma, kTinyP);
  const float2 q = make_float2(mean.x / g, mean.y / g);
  const float down = fminf(fmaxf(pv / g, kTinyP), 1.0f);
  return -logf(down) - g * abs_sq(q) / down;
}

// Warp bitonic sort of (value desc, position asc); returns this lane's
// position after sorting.
FBME_DEV int warp_sort_desc(float val, int pos, float* out_val) {
  const int lane = threadIdx.x & 31;
  for (int size = 2; size <= 32; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, val, stride);
      const int op = __shfl_xor_sync(0xffffffffu, pos, stride);
      const bool other_first = (ov > val) || (ov == val && op < pos);
      const bool lower = (lane & stride) == 0;
      const bool asc = (lane & size) == 0;
      if (lower == asc ? other_first : !other_first) {
        val = ov;
        pos = op;
      }
    }
  *out_val = val;
  return pos;
}

// Evaluations p in [state.evals, P) until done or an exchange is needed,
// one block per scene.  phase 0: initialise from the top-K; phase 1: apply
// the exchange whose candidate lists are in p.cand_*, then continue.  Every
// warp holds the same lane values (active set, variances, best model), so
// the decisions need no broadcast; warp 0 writes the state.
FBME_DEV void polish_body(const PolishArgs& A, PolishShared& S, TopkMergeShared& T, int phase, int lists, int scene) {
  extern __shared__ float2 dtab[];  // D1 (n1) then D2 (n2)
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (scene >= A.s.B) return;
  const BatchShape& s = A.s;
  const DevConfig& c = A.c;
  const int K = c.polish_size;
  const bool on = lane < K;
  PolishScene* ps = reinterpret_cast<PolishScene*>(A.p.pstate) + scene;
  const float fl = A.p.sc.floor_[scene];
  const float data_energy = A.p.sc.data_energy[scene];
  const float Mf = static_cast<float>(observed_samples(s, c));
  const long long N = s.n();
  const float2* bp = A.p.bp + scene * N;
  float2* d1 = dtab;
  float2* d2 = dtab + s.n1;
  if (threadIdx.x == 0) S.status = 0;

  // the selection this phase starts from: the active set or the exchange's
  // additions, merged from the candidate lists (S.M and S.L are free here)
  static_assert(sizeof(S.M) + sizeof(S.L) >= kMergeMax * sizeof(unsigned long long), "merge scratch");
  const int nsel = phase == 0 ? K : c.exchange;
  {
    const size_t off = static_cast<size_t>(scene) * lists * nsel;
    block_topk_merge<kMergeMax / kPolishThreads>(A.p.cand_key + off, A.p.cand_idx + off, lists, nsel,
                                                 reinterpret_cast<unsigned long long*>(&S), T);
  }

  // the work set of the next evaluation and the best model so far
  int idx = 0, bidx = 0, pending = 0, exch_acc = 0, has_best = 0, evals = 0;
  float gam = 1.0f, nu = 0.f, bnoise = 0.f, bpv = 0.f, bdd = 0.f, bg = 1.0f;
  float2 bmu = make_float2(0.f, 0.f);
  double best_nle = 0.0;
  if (phase == 0) {
    // prune + reinitialise (solver.py:4087-4106)
    if (on) {
      idx = merge_index(T.best[lane]);
      const float g0 = A.p.gamma[scene * N + idx];
      gam = c.reinit ? fmaxf(key_to_float(merge_key(T.best[lane])), fl) : g0;
    }
    nu = A.p.sc.noise[scene];
    load_dirichlet(A, d1, d2);
  } else {
    evals = ps->evals;
    has_best = ps->has_best;
    exch_acc = ps->exch_acc;
    nu = ps->work_noise;
    bnoise = ps->best_noise;
    best_nle = ps->best_nle;
    if (on) {
      idx = ps->work_active[lane];
      gam = ps->work_gamma[lane];
      bidx = ps->active[lane];
      bmu = ps->best_mean[lane];
      bpv = ps->best_pv[lane];
      bdd = ps->best_dd[lane];
      bg = ps->best_gamma[lane];
    }
    load_dirichlet(A, d1, d2);
    // residual support exchange (solver.py:4397-4494), using the best
    // state after evaluation 0 as the base.
    const int E = c.exchange;
    const float del = on ? deletion_gain(bmu, bpv, bg) : -INFINITY;
    float sval;
    const int rem_pos = warp_sort_desc(on ? del : -INFINITY, on ? lane : 0x7fffffff, &sval);
    // lane r < E: removal position rem_pos, addition candidate r
    int repl_idx = -1;
    float repl_gamma = 0.f;
    int xmask = 0;
    if (lane < E) {
      const float add_e = key_to_float(merge_key(T.best[lane]));
      const int add_i = merge_index(T.best[lane]);
      const float ce = Mf;
      const float ratio = add_e / fmaxf(bnoise * ce, kTinyP);
      const float add_gain = ratio > 1.0f ? ratio - 1.0f - logf(fmaxf(ratio, kTinyP)) : 0.0f;
      xmask = (add_gain + sval) > 0.0f;
      float ag = fmaxf(add_e - bnoise * ce, 0.0f) / (ce * ce);
      ag = fminf(fmaxf(ag, fl), c.max_prec);
      repl_idx = add_i;
      repl_gamma = ag;
    }
    // apply: position rem_pos takes the addition where exchanged
    for (int r = 0; r < E; ++r) {
      const int pr = __shfl_sync(0xffffffffu, rem_pos, r);
      const int xm = __shfl_sync(0xffffffffu, xmask, r);
      const int ri = __shfl_sync(0xffffffffu, repl_idx, r);
      const float rg = __shfl_sync(0xffffffffu, repl_gamma, r);
      if (xm && lane == pr) {
        idx = ri;
        gam = rg;
      }
    }
    pending = __any_sync(0xffffffffu, xmask != 0);
  }

  const int P = c.polish_iters;
  for (int p = evals; p < P; ++p) {
    const float2 cvec = on ? bp[idx] : make_float2(0.f, 0.f);
    const EvalOut o = evaluate(A, S, d1, d2, K, idx, gam, nu, cvec, data_energy);
    // evidence gate (solver.py:4168-4298)
    bool accept = true;
    if (c.gate && has_best) {
      const double margin = static_cast<double>(c.margin_factor) * kEpsP *
                            (1.0 + fabs(o.nle) + fabs(best_nle));
      accept = isfinite(o.nle) && (!isfinite(best_nle) || o.nle <= best_nle - margin);
      if (pending && accept) exch_acc += 1;
      pending = 0;
    }
    if (accept) {
      bidx = idx;
      bmu = o.mean;
      bpv = o.pv;
      bdd = o.dd;
      bg = gam;
      bnoise = nu;
      best_nle = o.nle;
      has_best = 1;
    }
    if (threadIdx.x == 0) ps->trace[p] = static_cast<float>(best_nle);
    evals = p + 1;
    if (p + 1 == P) break;
    // EM between evaluations (solver.py:4320-4391), from the best state
    const float ng = fminf(fmaxf(abs_sq(bmu) + bpv, fl), c.max_prec);
    const float keep = c.polish_damping;
    const float upd_g = keep * bg + (1.0f - keep) * ng;
    const float2 bc = on ? bp[bidx] : make_float2(0.f, 0.f);
    const double er = residual_energy(A, S.gm, d1, d2, K, bidx, bmu, bc, data_energy);
    float dof = on ? fminf(fmaxf(1.0f - bpv / fmaxf(bg, kTinyP), 0.f), 1.f) : 0.f;
    dof = warp_sum(dof);
    float un;
    if (c.fixed_noise > 0.f) {
      un = c.fixed_noise;
    } else if (!c.noise_evidence) {
      un = static_cast<float>((er + static_cast<double>(bnoise) * dof + c.noise_rate) /
                              (static_cast<double>(Mf) + c.noise_shape));
    } else {
      un = static_cast<float>((er + c.noise_rate) /
                              fmax(static_cast<double>(Mf) - dof + c.noise_shape, kEpsP));
    }
    un = fmaxf(un, fl);
    nu = c.fixed_noise > 0.f ? un : keep * bnoise + (1.0f - keep) * un;
    idx = bidx;
    gam = upd_g;
    const int E = c.exchange;
    if (E > 0 && p == 0) break;  // exchange candidates are scored over the grid next
  }
  if (w == 0) {
    if (on) {
      ps->active[lane] = bidx;
      ps->best_mean[lane] = bmu;
      ps->best_pv[lane] = bpv;
      ps->best_dd[lane] = bdd;
      ps->best_gamma[lane] = bg;
      ps->work_active[lane] = idx;
      ps->work_gamma[lane] = gam;
    }
    if (lane == 0) {
      ps->best_noise = bnoise;
      ps->best_nle = best_nle;
      ps->has_best = has_best;
      ps->work_noise = nu;
      ps->evals = evals;
      ps->pending = pending;
      ps->exch_acc = exch_acc;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && S.status) atomicOr(&A.p.status[scene], S.status);
}
__global__ void __launch_bounds__(kPolishThreads) polish_kernel(PolishArgs A, int phase, int lists) {
  dep_sync();
  __shared__ PolishShared S;
  __shared__ TopkMergeShared T;
  polish_body(A, S, T, phase, lists, blockIdx.x);
}

// Residual exchange scoring (solver.py:4398-4412) without the M-space
// residual: score[n] = |A^H y[n] - sum_k mu_k D1[n1-a_k] D2[n2-b_k]|^2 over
// the grid, active atoms excluded.  A CTA covers TY*RPT grid rows; thread
// (tx, ty) accumulates RPT rows x CPT columns, the columns in pairs
// 2tx + {0, 1} + 2*TX*c.  One paired FP32 FMA then serves two columns: with
// RE, IM the real and imaginary accumulators of the pair,
//   RE += ux*Dx;  IM += ux*Dy;  RE += uy*(-Dy);  IM += uy*Dx
// (per element the rounding sequence of a complex MAC).  D2 sits in shared
// memory split into re, im and -im, unrolled past the wrap, and twice, at
// even and at odd offset, so that the pair at any shift is one aligned
// 8-byte load with no index arithmetic.  Each CTA emits its E best
// (key, index) candidates.
template <int RPT_, int CPT, int TX_, int THREADS, int N2MAX>
struct ExTile {
  static constexpr int RPT = RPT_, TX = TX_, threads = THREADS, n2_max = N2MAX;
  static constexpr int ty = THREADS / TX;
  static constexpr int rows = ty * RPT;     // grid rows per CTA
  static constexpr int span = TX * CPT;     // columns of the thread grid
  static constexpr int pairs = CPT / 2;
  static constexpr int kpt = RPT * CPT;     // scores per thread
  static_assert(span >= N2MAX, "the thread grid spans the widest row");
  // floats per D2 table: index e + 1 <= N2 + span must be in range
  __host__ __device__ static constexpr int table_len(int n2) { return (n2 + span + 2) & ~1; }
  static size_t smem_bytes(int n2) {
    return static_cast<size_t>(rows) * n2 * sizeof(float2) + 6ull * table_len(n2) * sizeof(float);
  }
};

// Two CTAs per SM (128 registers a thread): a persistent single CTA per SM
// with double-buffered rows measured slower, its 8 warps too few to keep
// the FMA pipes fed.
template <typename T>
FBME_DEV void exchange_body(const PolishArgs& A, uint32_t* cand_key, int* cand_idx, int scene, int bx, int nbx) {
  constexpr int RPT = T::RPT, TX = T::TX;
  extern __shared__ float4 ex_shm4[];
  __shared__ TopkPrunedShared S;
  __shared__ float4 u4[kMaxPolish][T::rows];  // {ux, ux, uy, uy}
  __shared__ uint32_t excl[T::rows][16];      // active-atom bitmap per row (N2 <= 512)
  __shared__ int atom_a[kMaxPolish], atom_b[kMaxPolish];
  __shared__ float2 atom_mu[kMaxPolish];
  const BatchShape& s = A.s;
  const int r0 = bx * T::rows;
  const int K = A.c.polish_size, E = A.c.exchange;
  const int N1 = s.n1, N2 = s.n2;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  float2* bps = reinterpret_cast<float2*>(ex_shm4);  // [rows][N2]: this CTA's rows of A^H y
  float* tab = reinterpret_cast<float*>(bps + T::rows * N2);
  const int L = T::table_len(N2);
  const PolishScene* ps = reinterpret_cast<const PolishScene*>(A.p.pstate) + scene;
  {
    // A^H y rows, asynchronous copies in flight during the set-up and the
    // MAC loop: 16-byte chunks when N2 is even (every row then starts on a
    // 16-byte boundary), else one 8-byte element each
    const float2* src = A.p.bp + scene * s.n() + static_cast<long long>(r0) * N2;
    const int rows = min(T::rows, N1 - r0);
    if ((N2 & 1) == 0) {
      for (int c = threadIdx.x; c < rows * N2 / 2; c += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(bps + 2 * c)), "l"(src + 2 * c)
                     : "memory");
    } else {
      for (int c = threadIdx.x; c < rows * N2; c += blockDim.x)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(bps + c)), "l"(src + c) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // D2 tables: [parity][re, im, -im][L]; parity p holds D2[(e + p) mod N2] at
  // e.  Unrolled to the widest table, so that every thread's loads are in
  // flight together.
  constexpr int kTabIters = (T::table_len(T::n2_max) + T::threads - 1) / T::threads;
#pragma unroll
  for (int it = 0; it < kTabIters; ++it) {
    const int e = threadIdx.x + it * T::threads;
    if (e < L) {
      const int e0 = e % N2;
      const int e1 = e0 + 1 == N2 ? 0 : e0 + 1;
      const float2 v0 = __ldg(A.p.dir2 + e0), v1 = __ldg(A.p.dir2 + e1);
      tab[e] = v0.x;
      tab[L + e] = v0.y;
      tab[2 * L + e] = -v0.y;
      tab[3 * L + e] = v1.x;
      tab[4 * L + e] = v1.y;
      tab[5 * L + e] = -v1.y;
    }
  }
  for (int i = threadIdx.x; i < T::rows * 16; i += blockDim.x) (&excl[0][0])[i] = 0u;
  if (threadIdx.x < K) {
    const int idx = ps->active[threadIdx.x];
    const int a = idx / N2;
    atom_a[threadIdx.x] = a;
    atom_b[threadIdx.x] = idx - a * N2;
    atom_mu[threadIdx.x] = ps->best_mean[threadIdx.x];
  }
  __syncthreads();
  if (threadIdx.x < K) {
    const int ra = atom_a[threadIdx.x] - r0, b = atom_b[threadIdx.x];
    if (ra >= 0 && ra < T::rows) atomicOr(&excl[ra][b >> 5], 1u << (b & 31));
  }
  constexpr int kUIters = (kMaxPolish * T::rows + T::threads - 1) / T::threads;
#pragma unroll
  for (int it = 0; it < kUIters; ++it) {
    const int i = threadIdx.x + it * T::threads;
    const int k = i / T::rows, ri = i % T::rows;
    if (k < K) {
      float2 uv = make_float2(0.f, 0.f);
      if (r0 + ri < N1) {
        int dd = r0 + ri - atom_a[k];
        dd += dd < 0 ? N1 : 0;
        uv = cmul(atom_mu[k], __ldg(A.p.dir1 + dd));
      }
      u4[k][ri] = make_float4(uv.x, uv.x, uv.y, uv.y);
    }
  }
  __syncthreads();
  float2 re[RPT][T::pairs], im[RPT][T::pairs];
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int c = 0; c < T::pairs; ++c) {
      re[r][c] = make_float2(0.f, 0.f);
      im[r][c] = make_float2(0.f, 0.f);
    }
#pragma unroll 1
  for (int k = 0; k < K; ++k) {
    // pair (D2[e], D2[e+1]) at e = n2 - b + N2 >= 1; e's parity is the warp's
    const int e0 = 2 * tx - atom_b[k] + N2;
    const int odd = e0 & 1;
    const float* base = tab + odd * 3 * L + (e0 - odd);
    float2 dx[T::pairs], dy[T::pairs], ny[T::pairs];
#pragma unroll
    for (int c = 0; c < T::pairs; ++c) {
      dx[c] = *reinterpret_cast<const float2*>(base + 2 * TX * c);
      dy[c] = *reinterpret_cast<const float2*>(base + L + 2 * TX * c);
      ny[c] = *reinterpret_cast<const float2*>(base + 2 * L + 2 * TX * c);
    }
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const float4 uu = u4[k][ty * RPT + r];
      const float2 ux = make_float2(uu.x, uu.y), uy = make_float2(uu.z, uu.w);
#pragma unroll
      for (int c = 0; c < T::pairs; ++c) {
        re[r][c] = __ffma2_rn(ux, dx[c], re[r][c]);
        im[r][c] = __ffma2_rn(ux, dy[c], im[r][c]);
        re[r][c] = __ffma2_rn(uy, ny[c], re[r][c]);
        im[r][c] = __ffma2_rn(uy, dx[c], im[r][c]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  uint32_t key[T::kpt];
  uint32_t valid = 0u;
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int c = 0; c < T::pairs; ++c)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int i = (r * T::pairs + c) * 2 + j;
        const int lr = ty * RPT + r;
        const int n2 = 2 * tx + 2 * TX * c + j;
        key[i] = 0u;
        if (r0 + lr < N1 && n2 < N2) {
          valid |= 1u << i;
          const float2 bv = bps[lr * N2 + n2];
          const float2 acc = j ? make_float2(re[r][c].y, im[r][c].y) : make_float2(re[r][c].x, im[r][c].x);
          const float2 d = make_float2(bv.x - acc.x, bv.y - acc.y);
          const bool act = (excl[lr][n2 >> 5] >> (n2 & 31)) & 1u;
          key[i] = act ? 0u : float_key_t(abs_sq(d));
        }
      }
  const size_t off = (static_cast<size_t>(scene) * nbx + bx) * E;
  auto gidx = [&](int i) {
    const int r = i / (2 * T::pairs), c = (i / 2) % T::pairs, j = i & 1;
    return (r0 + ty * RPT + r) * N2 + 2 * tx + 2 * TX * c + j;
  };
  // residual scores of one CTA crowd into few top-byte bins (radix fallback)
  block_topk_pruned<T::kpt, true>(key, valid, gidx, E, S, cand_key + off, cand_idx + off);
}

template <typename T>
__global__ void __launch_bounds__(T::threads, 2)
exchange_kernel(PolishArgs A, uint32_t* cand_key, int* cand_idx) {
  dep_sync();
  exchange_body<T>(A, cand_key, cand_idx, blockIdx.y, blockIdx.x, gridDim.x);
}

using ExSmall = ExTile<8, 2, 32, 256, 64>;
using ExMid = ExTile<8, 2, 64, 256, 128>;
using ExWide = ExTile<8, 4, 64, 256, 256>;
using ExWidest = ExTile<4, 8, 64, 256, 512>;

// Final K-space outputs, fixed-budget diagnostics, effective DOF
// (solver.py:1989-2021, 2081-2092, 3408-3496, 2108-2126).
FBME_DEV void polish_finish_body(const PolishArgs& A, GramSums& gm, const FbmeOutputs& out, int scene) {
  extern __shared__ float2 dtab[];
  const int lane = threadIdx.x & 31;
  if (scene >= A.s.B) return;
  const BatchShape& s = A.s;
  const DevConfig& c = A.c;
  const int K = c.polish_size, P = c.polish_iters;
  const int R = c.repairs;
  const bool on = lane < K;
  const PolishScene* ps = reinterpret_cast<const PolishScene*>(A.p.pstate) + scene;
  const float fl = A.p.sc.floor_[scene];
  const float Mf = static_cast<float>(observed_samples(s, c));
  const long long N = s.n();
  float2* d1 = dtab;
  float2* d2 = dtab + s.n1;
  load_dirichlet(A, d1, d2);
  const int idx = on ? ps->active[lane] : 0;
  const float2 mu = on ? ps->best_mean[lane] : make_float2(0.f, 0.f);
  const float pv = on ? ps->best_pv[lane] : 0.f;
  const float dd = on ? ps->best_dd[lane] : 0.f;
  const float g = on ? ps->best_gamma[lane] : 1.0f;
  const float nu = ps->best_noise;
  // effective DOF with relevance projection
  float rel = on ? fminf(fmaxf(g * dd, 0.f), 1.f) : 0.f;
  const float raw = warp_sum(rel);
  const float max_dof = static_cast<float>(observed_samples(s, c) * (1.0 - 10.0 * kEpsP));
  const float sc = fminf(1.0f, max_dof / fmaxf(raw, kEpsP));
  const float dof = warp_sum(rel * sc);
  if (threadIdx.x == 0) {
    out.noise_variance[scene] = nu;
    out.effective_dof[scene] = dof;
    out.negative_log_evidence[scene] = static_cast<float>(ps->best_nle);
    for (int p = 0; p < P; ++p) out.evidence_trace[scene * (P + R) + p] = ps->trace[p];
    if (out.support_exchanges_accepted) out.support_exchanges_accepted[scene] = ps->exch_acc;
    // the support repairs append their evidence after the polish's
    for (int r = 0; r < R; ++r) out.evidence_trace[scene * (P + R) + P + r] = ps->trace[P + r];
    if (out.support_score_threshold && c.false_alarm > 0.f)
      out.support_score_threshold[scene] =
          static_cast<float>(log(static_cast<double>(N) / static_cast<double>(c.false_alarm)));
  }
  if (threadIdx.x < K && out.active_indices) out.active_indices[scene * K + lane] = idx;
  if (c.fixed_budget && out.fixed_budget_gamma_residual) {
    const float ag = fmaxf(g, kTinyP);
    const float gt = fminf(fmaxf(abs_sq(mu) + pv, fl), c.max_prec);
    const float gs = fmaxf(fmaxf(fabsf(ag), fabsf(gt)), kTinyP);
    const float gr = warp_max(on ? fabsf(ag - gt) / gs : 0.f);
    float dofd = on ? fminf(fmaxf(1.0f - pv / ag, 0.f), 1.f) : 0.f;
    dofd = warp_sum(dofd);
    const float2 cv = on ? A.p.bp[scene * N + idx] : make_float2(0.f, 0.f);
    const double er = residual_energy(A, gm, d1, d2, K, idx, mu, cv, A.p.sc.data_energy[scene]);
    float nt;
    if (c.fixed_noise > 0.f) {
      nt = nu;
    } else if (!c.noise_evidence) {
      nt = static_cast<float>((er + static_cast<double>(nu) * dofd + c.noise_rate) /
                              (static_cast<double>(Mf) + c.noise_shape));
    } else {
      nt = static_cast<float>((er + c.noise_rate) /
                              fmax(static_cast<double>(Mf) - dofd + c.noise_shape, kEpsP));
    }
    nt = fminf(fmaxf(nt, fl), c.max_prec);
    const float ns = fmaxf(fmaxf(fabsf(nu), fabsf(nt)), kTinyP);
    if (threadIdx.x == 0) {
      out.fixed_budget_gamma_residual[scene] = gr;
      out.fixed_budget_noise_residual[scene] = c.fixed_noise > 0.f ? 0.f : fabsf(nu - nt) / ns;
      bool fin = true, mono = true;
      for (int p = 0; p < P; ++p) fin &= isfinite(ps->trace[p]) != 0;
      for (int p = 1; p < P; ++p) mono &= ps->trace[p] <= ps->trace[p - 1];
      out.fixed_budget_monotone[scene] = fin && mono;
      out.fixed_budget_objective_decrease[scene] = fmaxf(ps->trace[0] - ps->trace[P - 1], 0.f);
    }
  }
}
__global__ void __launch_bounds__(kPolishThreads) polish_finish_kernel(PolishArgs A, FbmeOutputs out) {
  dep_sync();
  __shared__ GramSums gm;
  polish_finish_body(A, gm, out, blockIdx.x);
}

// ---------------------------------------------------------------------------
// Global certificate and support repairs (solver.py:3522-3588 inactive
// certificate, 3219-3317 active certificate, 4511-4628 repairs, 4851-4870
// and 5388-5460 final diagnostics).  A block per scene runs the K-dimensional
// algebra (evaluate(), as in the polish) between grid scans on many blocks,
// whose threads score a pair of atoms at a time.  For atom j, with
// g_i = a_j^H a_i from the Dirichlet tables,
//   q_j   = (A^H y)[j] - sum_i g_i mu_i             (nu a_j^H C^-1 y)
//   v     = L^-1 D^-1 conj(g)                       (forward substitution)
//   s_j   = M / nu - ||v||^2 / nu^2                 (a_j^H C^-1 a_j)
//   rho_j = |q_j / nu|^2 / s_j, and 0 on the active set,
// where L is the Cholesky factor of the equilibrated reduced system
// D^-1 (Gamma^-1 + A_S^H A_S / nu) D^-1: the reference obtains the same
// quantities from K adjoint transforms of the active columns and a
// K-right-hand-side triangular solve over the grid.
constexpr int kCertThreads = 256;

struct CertBest {
  float ratio, prec;
  int index;
};

FBME_DEV void cert_pick(CertBest& b, float ratio, float prec, int index) {
  if (ratio > b.ratio || (ratio == b.ratio && index < b.index)) b = CertBest{ratio, prec, index};
}

FBME_DEV CertBest cert_warp_best(CertBest b) {
  for (int off = 16; off > 0; off >>= 1) {
    const float r = __shfl_xor_sync(0xffffffffu, b.ratio, off);
    const float p = __shfl_xor_sync(0xffffffffu, b.prec, off);
    const int i = __shfl_xor_sync(0xffffffffu, b.index, off);
    cert_pick(b, r, p, i);
  }
  return b;
}

// The active set of one evaluation, staged for the grid scan.
struct CertModel {
  int a1[kMaxPolish], a2[kMaxPolish], idx[kMaxPolish];
  float2 mu[kMaxPolish];
  float inv_d[kMaxPolish], inv_l[kMaxPolish];
};

// Shared memory of a scan: the model's constants and factor, every value
// doubled (and where it is needed with both signs) as an operand of the
// paired FP32 instructions, and the Dirichlet table D2 split into re and im,
// unrolled past the wrap, at even and at odd offset (as the exchange's).
struct CertShared {
  float4 mu[kMaxPolish];    // mu.x, mu.x, mu.y, mu.y
  float4 scale[kMaxPolish]; // -mu.y, -mu.y, 1/d, 1/d
  float4 inv[kMaxPolish];   // -1/d, -1/d, 1/l, 1/l
  // row i's entries k < i in pairs (k, k + 1) of three float4s:
  // -Lx, -Lx, Ly, Ly | -Ly, -Ly, -Lx', -Lx' | Ly', Ly', -Ly', -Ly'
  float4 l[kMaxPolish * kMaxPolish / 4][3];
  int idx[kMaxPolish], a1[kMaxPolish], a2[kMaxPolish];
  CertBest red[kCertThreads / 32];
};
__host__ __device__ constexpr int cert_table_len(int n2) { return 2 * n2; }  // a pair ends at 2 n2 - 1 at most
static size_t cert_scan_smem(const BatchShape& s) {
  return s.n1 * sizeof(float2) + 4ull * cert_table_len(s.n2) * sizeof(float);
}

FBME_DEV float2 dup(float v) { return make_float2(v, v); }
FBME_DEV float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
FBME_DEV float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// Largest one-coordinate ratio over the atoms of the pairs [p0, p1) (pair p:
// columns 2c, 2c + 1 of row p / ppr, ppr pairs a row; first index on ties, as
// torch's max), with its atom precision s_j; the block's best, in every
// thread.  A thread carries its pair through the substitution in the paired
// FP32 instructions, each element with the rounding sequence of one atom
// alone (products and sums spelled out); the factor's entries are broadcast
// reads, three 16-byte ones for two entries and two atoms.  One block of
// eight warps with the whole register file an SM, its warps kept together by
// a barrier a pair: the unrolled substitution is longer than the instruction
// cache, and warps at different places of it wait for its refills (two blocks
// of four warps 2.24 ms, this block without the barrier 1.84 ms).  One atom at
// a time took 2.14 ms for two scans of 64 scenes of 256 x 256, this 1.78 ms,
// about a quarter of it in the hypotenuses.
template <bool MASKED>
FBME_DEV CertBest cert_scan(const PolishArgs& A, CertShared& S, int K, float nu, const float2* bp, const float2* d1,
                            const float* tab, long long p0, long long p1) {
  const BatchShape& s = A.s;
  const int n2 = s.n2, ppr = (n2 + 1) / 2, len = cert_table_len(n2);
  const float Mf = static_cast<float>(observed_samples(s, A.c));
  const float nu2 = nu * nu;
  CertBest b{-1.f, 1.f, 0x7fffffff};
  for (long long pb = p0; pb < p1; pb += kCertThreads) {
    __syncthreads();
    const long long p = min(pb + threadIdx.x, p1 - 1);
    const int j1 = static_cast<int>(p / ppr), j2 = 2 * static_cast<int>(p - static_cast<long long>(j1) * ppr);
    const int j = j1 * n2 + j2;
    const bool two = j2 + 1 < n2;
    const float2 b0 = bp[j], b1 = two ? bp[j + 1] : make_float2(0.f, 0.f);
    float2 qx = make_float2(-b0.x, -b1.x), qy = make_float2(-b0.y, -b1.y);  // minus q of the pair
    unsigned act = 0u;
    float2 vx[kMaxPolish], vy[kMaxPolish];
    float2 red2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kMaxPolish; ++i) {
      if (i < K) {
        const unsigned dj = static_cast<unsigned>(S.idx[i] - j);
        act |= dj < 2u ? 1u << dj : 0u;
        int i1 = j1 - S.a1[i], i2 = j2 - S.a2[i];
        if (i1 < 0) i1 += s.n1;
        float2 gx, gy;
        if constexpr (MASKED) {
          if (i2 < 0) i2 += n2;
          const float2* row = A.p.gram2d + static_cast<long long>(i1) * n2;
          const float2 g0 = __ldg(row + i2), g1 = __ldg(row + (i2 + 1 < n2 ? i2 + 1 : 0));
          gx = make_float2(g0.x, g1.x);
          gy = make_float2(g0.y, g1.y);
        } else {
          const int e = i2 + n2, odd = e & 1;  // e in [1, 2 n2)
          const float* base = tab + odd * 2 * len + (e - odd);
          const float2 yx = *reinterpret_cast<const float2*>(base);
          const float2 yy = *reinterpret_cast<const float2*>(base + len);
          const float2 x = d1[i1];
          gx = __ffma2_rn(dup(x.x), yx, __fmul2_rn(dup(-x.y), yy));
          gy = __ffma2_rn(dup(x.y), yx, __fmul2_rn(dup(x.x), yy));
        }
        const float4 cm = S.mu[i], cs = S.scale[i], ci = S.inv[i];
        qx = __fadd2_rn(qx, __ffma2_rn(gx, lo2(cm), __fmul2_rn(gy, lo2(cs))));
        qy = __fadd2_rn(qy, __ffma2_rn(gy, lo2(cm), __fmul2_rn(gx, hi2(cm))));
        float2 cx, cy;
        if (i == 0) {
          cx = __fmul2_rn(gx, hi2(cs));
          cy = __fmul2_rn(gy, lo2(ci));
        }
        // minus the terms L[i][k] v[k], k ascending; the first one is fused
        // with the scaling of conj(g)
#pragma unroll
        for (int k = 0; k < i; k += 2) {
          const float4* e = S.l[i * i / 4 + k / 2];
          const float4 e0 = e[0], e1 = e[1], e2 = e[2];
          const float2 tx = __ffma2_rn(lo2(e0), vx[k], __fmul2_rn(hi2(e0), vy[k]));
          const float2 ty = __ffma2_rn(lo2(e0), vy[k], __fmul2_rn(lo2(e1), vx[k]));
          cx = k == 0 ? __ffma2_rn(gx, hi2(cs), tx) : __fadd2_rn(cx, tx);
          cy = k == 0 ? __ffma2_rn(gy, lo2(ci), ty) : __fadd2_rn(cy, ty);
          if (k + 1 < i) {
            cx = __fadd2_rn(cx, __ffma2_rn(hi2(e1), vx[k + 1], __fmul2_rn(lo2(e2), vy[k + 1])));
            cy = __fadd2_rn(cy, __ffma2_rn(hi2(e1), vy[k + 1], __fmul2_rn(hi2(e2), vx[k + 1])));
          }
        }
        vx[i] = __fmul2_rn(cx, hi2(ci));
        vy[i] = __fmul2_rn(cy, hi2(ci));
        const float2 h = make_float2(hypotf(vx[i].x, vy[i].x), hypotf(vx[i].y, vy[i].y));
        red2 = __ffma2_rn(h, h, red2);
      }
    }
    auto pick = [&](float qxj, float qyj, float r2, bool active, int jj) {
      const float prec = fmaxf(Mf / nu - r2 / nu2, kTinyP);
      const float2 qn = make_float2(qxj / nu, qyj / nu);
      cert_pick(b, active ? 0.f : abs_sq(qn) / prec, prec, jj);
    };
    pick(qx.x, qy.x, red2.x, act & 1u, j);
    if (two) pick(qx.y, qy.y, red2.y, (act >> 1) & 1u, j + 1);
  }
  b = cert_warp_best(b);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) S.red[w] = b;
  __syncthreads();
  b = lane < kCertThreads / 32 ? S.red[lane] : CertBest{-1.f, 1.f, 0x7fffffff};
  return cert_warp_best(b);
}

// Inactive certificate of the best atom (solver.py:3568-3588).
struct CertState {
  float ratio, gain, optvar;
  int index;
};

FBME_DEV CertState cert_state(const CertBest& b) {
  const bool up = b.ratio > 1.0f;
  return CertState{b.ratio, up ? b.ratio - 1.0f - logf(fmaxf(b.ratio, kTinyP)) : 0.f,
                   up ? (b.ratio - 1.0f) / b.prec : 0.f, b.index};
}

// Lane k's exact one-coordinate terms (solver.py:3244-3290): the current
// deletion delta, the gain of the optimal variance and that variance.
struct ActiveTerms {
  float current, gain, optvar;
};

FBME_DEV ActiveTerms active_terms(float2 mean, float pv, float gamma) {
  const float g = fmaxf(gamma, kTinyP);
  const float2 q = make_float2(mean.x / g, mean.y / g);
  const float sc = fmaxf((g - pv) / (g * g), kTinyP);
  const float down = fminf(fmaxf(pv / g, kTinyP), 1.0f);
  const float loo = fmaxf(sc / down, kTinyP);
  const float ratio = abs_sq(q) / fmaxf(sc * down, kTinyP);
  ActiveTerms t;
  t.optvar = ratio > 1.0f ? (ratio - 1.0f) / loo : 0.f;
  t.current = -logf(down) - g * abs_sq(q) / down;
  const float opt = ratio > 1.0f ? logf(fmaxf(ratio, kTinyP)) - ratio + 1.0f : 0.f;
  t.gain = fmaxf(t.current - opt, 0.f);
  return t;
}

// Warp argmax of (value, lane), the first lane on ties.
FBME_DEV int warp_argmax(float v, float* best) {
  int pos = threadIdx.x & 31;
  for (int off = 16; off > 0; off >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, off);
    const int op = __shfl_xor_sync(0xffffffffu, pos, off);
    if (ov > v || (ov == v && op < pos)) {
      v = ov;
      pos = op;
    }
  }
  *best = v;
  return pos;
}

// Per-scene scratch of the certificate steps (caller workspace): the
// factor and staged active set of the model whose certificate the next
// scan computes, the pending repair, the current inactive certificate and
// the scan's per-block partial results.
struct CertScratch {
  float2 L[kMaxPolish][kMaxPolish];
  CertModel m;
  int nu_bits;  // the model's noise variance
  int pending;  // the scanned model is a repair proposal
  int p_idx[kMaxPolish];
  float p_gam[kMaxPolish];
  float2 p_mean[kMaxPolish];
  float p_pv[kMaxPolish], p_dd[kMaxPolish];
  double p_nle;
  CertState cur;
};

// Scan blocks per scene: enough CTAs to cover the SMs a few times, at least
// 1024 atoms per block, at most kCertMaxBlocks.  Within that range the
// count is raised (up to 4x) until the B * nblk CTAs fill their last wave of
// `resident` CTAs per SM to 97 %, or to the best fill seen: a last wave that
// is mostly empty leaves the scan's slowest blocks running alone.  The
// result does not depend on the count (first index on ties).
constexpr int kCertMaxBlocks = 256;
int cert_blocks(const BatchShape& s, int resident) {
  static const int sms = [] {
    int dev = 0, v = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  const long long most = std::min(std::max(1LL, (s.n() + 1023) / 1024), static_cast<long long>(kCertMaxBlocks));
  const long long lo = std::max(1LL, std::min((4LL * sms + s.B - 1) / s.B, most));
  const long long slots = static_cast<long long>(sms) * std::max(1, resident);
  long long best = lo;
  double best_fill = 0.0;
  for (long long n = lo; n <= std::min(most, 4 * lo); ++n) {
    const long long ctas = n * s.B;
    const double fill = static_cast<double>(ctas) / static_cast<double>(((ctas + slots - 1) / slots) * slots);
    if (fill > best_fill + 1e-9) {
      best_fill = fill;
      best = n;
    }
    if (fill >= 0.97) break;
  }
  return static_cast<int>(best);
}

size_t cert_scratch_bytes(const BatchShape& s) {
  return static_cast<size_t>(s.B) * (sizeof(CertScratch) + sizeof(CertBest) * kCertMaxBlocks);
}

FBME_DEV CertScratch* cert_scene(void* ws, int scene) {
  return reinterpret_cast<CertScratch*>(ws) + scene;
}
FBME_DEV CertBest* cert_parts(void* ws, int B, int scene) {
  return reinterpret_cast<CertBest*>(reinterpret_cast<CertScratch*>(ws) + B) + static_cast<long long>(scene) *
         kCertMaxBlocks;
}

// Evaluate the work set (idx, gam) on the block and stage its factor and
// active set for the scan.
FBME_DEV EvalOut cert_model(const PolishArgs& A, CertScratch* cs, PolishShared& S, const float2* d1,
                            const float2* d2, int idx, float gam, float nu, const float2* bp, float data_energy) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int K = A.c.polish_size;
  const bool on = lane < K;
  const EvalOut o = evaluate(A, S, d1, d2, K, idx, gam, nu, on ? bp[idx] : make_float2(0.f, 0.f), data_energy);
  if (on)
    for (int k = w; k < lane; k += kPolishWarps) cs->L[lane][k] = S.L[k][lane];
  if (on && w == 0) {
    cs->m.idx[lane] = idx;
    cs->m.a1[lane] = idx / A.s.n2;
    cs->m.a2[lane] = idx % A.s.n2;
    cs->m.mu[lane] = o.mean;
    cs->m.inv_d[lane] = 1.0f / o.dscale;
    cs->m.inv_l[lane] = 1.0f / S.L[lane][lane].x;
  }
  if (threadIdx.x == 0) cs->nu_bits = __float_as_int(nu);
  return o;
}

// The scan's result: the block partials merged (first index on ties).
FBME_DEV CertBest cert_merge(void* ws, int B, int scene, int nblk) {
  const int lane = threadIdx.x & 31;
  const CertBest* part = cert_parts(ws, B, scene);
  CertBest b{-1.f, 1.f, 0x7fffffff};
  for (int i = lane; i < nblk; i += 32) cert_pick(b, part[i].ratio, part[i].prec, part[i].index);
  return cert_warp_best(b);
}

// One certificate step of one scene (one block; warp 0 writes the state).  Step 0 stages the model
// the polish kept.  Step t in [1, R] merges the previous scan (the kept
// model's certificate at t = 1; otherwise repair t-1's certificate and its
// decision: kept when the inactive ratio that proposed it exceeds 1 and
// the exact evidence does not rise) and stages repair t: the best inactive
// atom replaces the active atom of largest deletion delta, with variance
// max(optimal, floor).  Step R + 1 merges the last scan and writes the
// final certificate (solver.py:4851-4870, 5388-5460).
__global__ void __launch_bounds__(kPolishThreads) cert_step_kernel(PolishArgs A, FbmeCertificate C, void* ws,
                                                                   int nblk, int t) {
  dep_sync();
  __shared__ PolishShared S;
  extern __shared__ float2 dtab[];
  const int scene = blockIdx.x;
  if (scene >= A.s.B) return;
  const BatchShape& s = A.s;
  const DevConfig& c = A.c;
  const int K = c.polish_size, P = c.polish_iters, R = c.repairs;
  const int lane = threadIdx.x & 31;
  const bool on = lane < K;
  PolishScene* ps = reinterpret_cast<PolishScene*>(A.p.pstate) + scene;
  CertScratch* cs = cert_scene(ws, scene);
  const long long N = s.n();
  const float2* bp = A.p.bp + scene * N;
  const float fl = A.p.sc.floor_[scene];
  const float data_energy = A.p.sc.data_energy[scene];
  const float nu = ps->best_noise;
  if (threadIdx.x == 0) S.status = 0;
  if (t > 0) {
    if (threadIdx.x < 32) {
      const CertState next = cert_state(cert_merge(ws, s.B, scene, nblk));
      bool keep = true;
      if (cs->pending) {  // decide the repair the scan certified
        const CertState prop = cs->cur;
        const double nle = cs->p_nle;
        keep = prop.ratio > 1.0f && isfinite(nle) && static_cast<float>(nle) <= static_cast<float>(ps->best_nle);
        __syncwarp();
        if (keep) {
          if (on) {
            ps->active[lane] = cs->p_idx[lane];
            ps->best_mean[lane] = cs->p_mean[lane];
            ps->best_pv[lane] = cs->p_pv[lane];
            ps->best_dd[lane] = cs->p_dd[lane];
            ps->best_gamma[lane] = cs->p_gam[lane];
          }
          if (lane == 0) {
            ps->best_nle = nle;
            ps->exch_acc += 1;
          }
        }
        __syncwarp();
        if (lane == 0) ps->trace[P + t - 2] = static_cast<float>(ps->best_nle);
      }
      __syncwarp();
      if (lane == 0 && keep) cs->cur = next;
    }
    __syncthreads();
  }
  if (t <= R) {
    float2* d1 = dtab;
    float2* d2 = dtab + s.n1;
    load_dirichlet(A, d1, d2);
    int idx = on ? ps->active[lane] : 0;
    float gam = on ? ps->best_gamma[lane] : 1.0f;
    if (t > 0) {
      const float2 mu = on ? ps->best_mean[lane] : make_float2(0.f, 0.f);
      const float pv = on ? ps->best_pv[lane] : 0.f;
      float dmax;
      const int pos = warp_argmax(on ? deletion_gain(mu, pv, gam) : -INFINITY, &dmax);
      const CertState cur = cs->cur;
      if (lane == pos) {
        idx = cur.index;
        gam = fmaxf(cur.optvar, fl);
      }
    }
    const EvalOut o = cert_model(A, cs, S, d1, d2, idx, gam, nu, bp, data_energy);
    if (threadIdx.x < K) {
      cs->p_idx[lane] = idx;
      cs->p_gam[lane] = gam;
      cs->p_mean[lane] = o.mean;
      cs->p_pv[lane] = o.pv;
      cs->p_dd[lane] = o.dd;
    }
    if (threadIdx.x == 0) {
      cs->p_nle = o.nle;
      cs->pending = t > 0;
    }
  } else {
    // final certificate of the kept model
    const float2 mu = on ? ps->best_mean[lane] : make_float2(0.f, 0.f);
    const float pv = on ? ps->best_pv[lane] : 0.f;
    const float g = on ? ps->best_gamma[lane] : 1.0f;
    const int idx = on ? ps->active[lane] : 0;
    const ActiveTerms at = active_terms(mu, pv, g);
    float max_gain, max_nondel, max_del;
    const int gp = warp_argmax(on ? at.gain : -INFINITY, &max_gain);
    warp_argmax(on ? (at.optvar > 0.f ? at.gain : 0.f) : -INFINITY, &max_nondel);
    warp_argmax(on ? at.current : -INFINITY, &max_del);
    const int best_idx = __shfl_sync(0xffffffffu, idx, gp);
    const float best_var = __shfl_sync(0xffffffffu, at.optvar, gp);
    if (threadIdx.x == 0) {
      const CertState cur = cs->cur;
      const float tol = C.coordinate_tolerance;
      const float pen = fmaxf(max_nondel, fmaxf(max_del, 0.f));
      C.inactive_max_evidence_ratio[scene] = cur.ratio;
      C.inactive_best_index[scene] = cur.index;
      C.inactive_evidence_gain[scene] = cur.gain;
      C.inactive_optimal_variance[scene] = cur.optvar;
      C.support_repairs_accepted[scene] = ps->exch_acc;
      C.active_max_evidence_gain[scene] = max_gain;
      C.active_best_index[scene] = best_idx;
      C.active_optimal_variance[scene] = best_var;
      C.active_max_deletion_gain[scene] = max_del;
      C.active_penalized_evidence_gain[scene] = pen;
      C.coordinate_stationary[scene] = cur.gain <= tol && max_gain <= tol;
      C.type2_map_coordinate_stationary[scene] = fmaxf(cur.gain, 0.f) <= tol && pen <= tol;
      if (C.familywise_ratio_threshold > 0.f)
        C.familywise_no_discovery[scene] = cur.ratio <= C.familywise_ratio_threshold;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && S.status) atomicOr(&A.p.status[scene], S.status);
}

// Block (bx, scene) scores the atom pairs [bx chunk, (bx + 1) chunk) against
// the staged model and writes its best to the scene's partials.
template <bool MASKED>
__global__ void __launch_bounds__(kCertThreads, 1) cert_scan_kernel(PolishArgs A, void* ws) {
  dep_sync();
  __shared__ CertShared S;
  extern __shared__ float2 dtab[];  // D1 (n1), then the four D2 tables
  const int scene = blockIdx.y;
  if (scene >= A.s.B) return;
  const BatchShape& s = A.s;
  const int K = A.c.polish_size, tid = threadIdx.x;
  const CertScratch* cs = cert_scene(ws, scene);
  float* tab = reinterpret_cast<float*>(dtab + s.n1);
  if constexpr (!MASKED) {
    const int len = cert_table_len(s.n2);
    for (int i = tid; i < s.n1; i += kCertThreads) dtab[i] = __ldg(A.p.dir1 + i);
    for (int e = tid; e < 2 * s.n2; e += kCertThreads) {
      const int e0 = e < s.n2 ? e : e - s.n2, e1 = e0 + 1 < s.n2 ? e0 + 1 : 0;
      const float2 v0 = __ldg(A.p.dir2 + e0), v1 = __ldg(A.p.dir2 + e1);
      tab[e] = v0.x;
      tab[len + e] = v0.y;
      tab[2 * len + e] = v1.x;
      tab[3 * len + e] = v1.y;
    }
  }
  for (int e = tid; e < kMaxPolish * (kMaxPolish / 2); e += kCertThreads) {
    const int i = e / (kMaxPolish / 2), k = 2 * (e % (kMaxPolish / 2));
    if (k < i && i < K) {
      const float2 l0 = cs->L[i][k], l1 = k + 1 < i ? cs->L[i][k + 1] : make_float2(0.f, 0.f);
      float4* d = S.l[i * i / 4 + k / 2];
      d[0] = make_float4(-l0.x, -l0.x, l0.y, l0.y);
      d[1] = make_float4(-l0.y, -l0.y, -l1.x, -l1.x);
      d[2] = make_float4(l1.y, l1.y, -l1.y, -l1.y);
    }
  }
  if (tid < K) {
    const float2 mu = cs->m.mu[tid];
    const float id = cs->m.inv_d[tid], il = cs->m.inv_l[tid];
    S.idx[tid] = cs->m.idx[tid];
    S.a1[tid] = cs->m.a1[tid];
    S.a2[tid] = cs->m.a2[tid];
    S.mu[tid] = make_float4(mu.x, mu.x, mu.y, mu.y);
    S.scale[tid] = make_float4(-mu.y, -mu.y, id, id);
    S.inv[tid] = make_float4(-id, -id, il, il);
  }
  __syncthreads();
  const float nu = __int_as_float(cs->nu_bits);
  const long long P = static_cast<long long>(s.n1) * ((s.n2 + 1) / 2);
  const long long chunk = (P + gridDim.x - 1) / gridDim.x;
  const long long p0 = blockIdx.x * chunk, p1 = min(P, p0 + chunk);
  const CertBest b = cert_scan<MASKED>(A, S, K, nu, A.p.bp + scene * s.n(), dtab, tab, p0, p1);
  if (tid == 0) cert_parts(ws, s.B, scene)[blockIdx.x] = b;
}

// N-space outputs in one pass: zero mean, floor variance and 1/floor
// precision off the active set, and the active entries.  Block b of a scene
// owns the contiguous pixel range [e0, e1): it fills the range, then its
// threads k < K write active atom k where it falls inside the range, so no
// other block touches those pixels and one launch replaces fill + scatter.
FBME_DEV void output_body(const PolishArgs& A, const FbmeOutputs& out, int scene, int bx, int nbx) {
  const BatchShape& s = A.s;
  const long long N = s.n();
  const int K = A.c.polish_size;
  const float fl = A.p.sc.floor_[scene];
  const float inv = 1.0f / fl;
  const long long chunk = (N + nbx - 1) / nbx;
  const long long e0 = bx * chunk, e1 = min(N, e0 + chunk);
  float2* x = reinterpret_cast<float2*>(out.x) + scene * N;
  float* pv = out.posterior_variance + scene * N;
  float* pr = out.precision + scene * N;
  uint8_t* mk = out.support_mask ? out.support_mask + scene * N : nullptr;
  for (long long e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
    x[e] = make_float2(0.f, 0.f);
    pv[e] = fl;
    pr[e] = inv;
    if (mk) mk[e] = 0;
  }
  __syncthreads();
  const int k = threadIdx.x;
  if (k >= K) return;
  const PolishScene* ps = reinterpret_cast<const PolishScene*>(A.p.pstate) + scene;
  const int idx = ps->active[k];
  const float2 mu = ps->best_mean[k];
  if (bx == 0 && out.active_values) reinterpret_cast<float2*>(out.active_values)[scene * K + k] = mu;
  if (idx < e0 || idx >= e1) return;
  const float apv = ps->best_pv[k];
  x[idx] = mu;
  pv[idx] = apv;
  pr[idx] = 1.0f / ps->best_gamma[k];
  if (mk && A.c.false_alarm > 0.f) {
    const float thr = static_cast<float>(log(static_cast<double>(N) / A.c.false_alarm));
    mk[idx] = (abs_sq(mu) / fmaxf(apv, kTinyP)) > thr;
  }
}
__global__ void __launch_bounds__(256) output_kernel(PolishArgs A, FbmeOutputs out) {
  dep_sync();
  output_body(A, out, blockIdx.y, blockIdx.x, gridDim.x);
}

void launch_topk_blocks(const uint32_t* keys, long long n, int k, int B, uint32_t* cand_key, int* cand_idx,
                        cudaStream_t st);

// The polish steps of several shape buckets (an uneven plan's), one launch
// each: bucket i is blockIdx.z = i with its own arguments; blocks past its
// scenes or blocks return, and every scene runs the single-bucket code.
struct PolishSet {
  int n;
  PolishArgs a[kBucketSetMax];
  FbmeOutputs out[kBucketSetMax];
  int slices[kBucketSetMax];      // top-k slices per scene
  int ex_blocks[kBucketSetMax];   // exchange row blocks per scene
  int out_blocks[kBucketSetMax];  // output blocks per scene
};
static_assert(sizeof(PolishSet) <= 32764, "kernel parameter limit");

FBME_DEV bool has_exchange(const DevConfig& c) { return c.exchange > 0 && c.polish_iters > 1; }

__global__ void __launch_bounds__(kPolishThreads) polish_set_kernel(const PolishSet set, int phase) {
  dep_sync();
  __shared__ PolishShared S;
  __shared__ TopkMergeShared T;
  const PolishArgs& A = set.a[blockIdx.z];
  if (phase == 1 && !has_exchange(A.c)) return;
  polish_body(A, S, T, phase, phase == 0 ? set.slices[blockIdx.z] : set.ex_blocks[blockIdx.z], blockIdx.x);
}

template <typename T>
__global__ void __launch_bounds__(T::threads, 2) exchange_set_kernel(const PolishSet S) {
  dep_sync();
  const PolishArgs& A = S.a[blockIdx.z];
  const int nbx = S.ex_blocks[blockIdx.z];
  if (static_cast<int>(blockIdx.x) >= nbx || static_cast<int>(blockIdx.y) >= A.s.B) return;
  exchange_body<T>(A, A.p.cand_key, A.p.cand_idx, blockIdx.y, blockIdx.x, nbx);
}

__global__ void __launch_bounds__(kPolishThreads) polish_finish_set_kernel(const PolishSet set) {
  dep_sync();
  __shared__ GramSums gm;
  polish_finish_body(set.a[blockIdx.z], gm, set.out[blockIdx.z], blockIdx.x);
}

__global__ void __launch_bounds__(256) output_set_kernel(const PolishSet S) {
  dep_sync();
  const int nbx = S.out_blocks[blockIdx.z];
  if (static_cast<int>(blockIdx.x) >= nbx || static_cast<int>(blockIdx.y) >= S.a[blockIdx.z].s.B) return;
  output_body(S.a[blockIdx.z], S.out[blockIdx.z], blockIdx.y, blockIdx.x, nbx);
}

static int exchange_rows(int n2) {
  return n2 <= 64 ? ExSmall::rows : n2 <= 128 ? ExMid::rows : n2 <= 256 ? ExWide::rows : ExWidest::rows;
}

int exchange_blocks(const BatchShape& s) {
  const int rows = exchange_rows(s.n2);
  return (s.n1 + rows - 1) / rows;
}

template <typename T>
static cudaError_t set_exchange_smem() {
  cudaError_t e = cudaFuncSetAttribute(exchange_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(T::smem_bytes(T::n2_max)));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(exchange_set_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(T::smem_bytes(T::n2_max)));
  return e;
}

// Dynamic shared memory of the kernels that hold the Dirichlet tables: plans
// run for N1 + N2 <= kDirichletMax, whose tables (32 KB) and the block's own
// 23 KB are more than the 48 KB a kernel may take without asking.  The
// certificate scan holds D1 and four forms of D2 (N2 <= 512).
constexpr int kDirichletMax = 4032;

template <typename K>
static cudaError_t set_smem(K kern, size_t bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

cudaError_t set_polish_attributes() {
  constexpr size_t tables = kDirichletMax * sizeof(float2);
  constexpr size_t scan = tables + 512 * (4 * 2 * sizeof(float) - sizeof(float2));
  cudaError_t e = set_smem(polish_kernel, tables);
  if (e == cudaSuccess) e = set_smem(polish_set_kernel, tables);
  if (e == cudaSuccess) e = set_smem(cert_step_kernel, tables);
  if (e == cudaSuccess) e = set_smem(cert_scan_kernel<false>, scan);
  if (e == cudaSuccess) e = set_exchange_smem<ExSmall>();
  if (e == cudaSuccess) e = set_exchange_smem<ExMid>();
  if (e == cudaSuccess) e = set_exchange_smem<ExWide>();
  if (e == cudaSuccess) e = set_exchange_smem<ExWidest>();
  return e;
}

// Residual exchange scoring under an observation mask (solver.py:4398-4412
// with the masked operator): score[n] = |A^H y[n] - sum_k mu_k G(n - a_k)|^2
// with the mask's 2-D Gram table G, written as order-preserving keys for a
// top-E selection; active atoms get key 0 (the reference's -inf).  One
// thread per grid point; the table lookups hit L2.
__global__ void __launch_bounds__(256) exchange_masked_kernel(PolishArgs A) {
  dep_sync();
  __shared__ int atom1[kMaxPolish], atom2[kMaxPolish], atom[kMaxPolish];
  __shared__ float2 amu[kMaxPolish];
  const int scene = blockIdx.y;
  const BatchShape& s = A.s;
  const int K = A.c.polish_size;
  const PolishScene* ps = reinterpret_cast<const PolishScene*>(A.p.pstate) + scene;
  if (threadIdx.x < K) {
    const int a = ps->active[threadIdx.x];
    atom[threadIdx.x] = a;
    atom1[threadIdx.x] = a / s.n2;
    atom2[threadIdx.x] = a % s.n2;
    amu[threadIdx.x] = ps->best_mean[threadIdx.x];
  }
  __syncthreads();
  const long long N = s.n();
  const float2* bp = A.p.bp + scene * N;
  uint32_t* keys = A.p.keys + scene * N;
  for (long long n = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; n < N;
       n += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int n1 = static_cast<int>(n / s.n2), n2 = static_cast<int>(n % s.n2);
    float2 r = bp[n];
    bool act = false;
    for (int k = 0; k < K; ++k) {
      act |= atom[k] == n;
      const float2 t = cmul(amu[k], gram_at(A, nullptr, nullptr, n1, n2, atom1[k], atom2[k]));
      r = make_float2(r.x - t.x, r.y - t.y);
    }
    keys[n] = act ? 0u : float_key_t(abs_sq(r));
  }
}

template <typename T>
static void launch_exchange(const PolishArgs& A, const PolishBuffers& p, cudaStream_t st) {
  const dim3 grid(exchange_blocks(A.s), A.s.B);
  launch_dep(exchange_kernel<T>, grid, T::threads, T::smem_bytes(A.s.n2), st, A, p.cand_key, p.cand_idx);
}

void polish_run(const BatchShape& s, const DevConfig& c, const PolishBuffers& p,
                const FbmeOutputs& out, cudaStream_t st, Profiler* prof, const FbmeCertificate* cert) {
  PolishArgs A{s, c, p};
  const int K = c.polish_size;
  // each launch timed on its own, so the profile counts launches
  FBME_TIMED(prof, FBME_GROUP_TOPK, launch_topk_blocks(p.keys, s.n(), K, s.B, p.cand_key, p.cand_idx, st));
  const size_t dsm = (s.n1 + s.n2) * sizeof(float2);
  FBME_TIMED(prof, FBME_GROUP_POLISH, (launch_dep(polish_kernel, s.B, kPolishThreads, dsm, st, A, 0, topk_slices(s.n()))));
  if (c.exchange > 0 && c.polish_iters > 1 && p.gram2d) {
    const long long nblk = (s.n() + 255) / 256;
    FBME_TIMED(prof, FBME_GROUP_EXCHANGE,
               (launch_dep(exchange_masked_kernel, dim3(static_cast<unsigned>(nblk < 1024 ? nblk : 1024), s.B), 256, 0, st, A)));
    FBME_TIMED(prof, FBME_GROUP_TOPK,
               launch_topk_blocks(p.keys, s.n(), c.exchange, s.B, p.cand_key, p.cand_idx, st));
    FBME_TIMED(prof, FBME_GROUP_POLISH,
               (launch_dep(polish_kernel, s.B, kPolishThreads, dsm, st, A, 1, topk_slices(s.n()))));
  } else if (c.exchange > 0 && c.polish_iters > 1) {
    const int nb = exchange_blocks(s);
    if (s.n2 <= 64)
      FBME_TIMED(prof, FBME_GROUP_EXCHANGE, (launch_exchange<ExSmall>(A, p, st)));
    else if (s.n2 <= 128)
      FBME_TIMED(prof, FBME_GROUP_EXCHANGE, (launch_exchange<ExMid>(A, p, st)));
    else if (s.n2 <= 256)
      FBME_TIMED(prof, FBME_GROUP_EXCHANGE, (launch_exchange<ExWide>(A, p, st)));
    else
      FBME_TIMED(prof, FBME_GROUP_EXCHANGE, (launch_exchange<ExWidest>(A, p, st)));
    FBME_TIMED(prof, FBME_GROUP_POLISH, (launch_dep(polish_kernel, s.B, kPolishThreads, dsm, st, A, 1, nb)));
  }
  if (cert) {  // model, scan, (decide + model, scan) per repair, final
    auto scan = p.gram2d ? cert_scan_kernel<true> : cert_scan_kernel<false>;
    const size_t csm = p.gram2d ? 0 : cert_scan_smem(s);
    int resident = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, scan, kCertThreads, csm) != cudaSuccess) resident = 1;
    const int nblk = cert_blocks(s, resident);
    for (int t = 0; t <= c.repairs + 1; ++t) {
      FBME_TIMED(prof, FBME_GROUP_CERTIFICATE,
                 (launch_dep(cert_step_kernel, s.B, kPolishThreads, dsm, st, A, *cert, cert->workspace, nblk, t)));
      if (t <= c.repairs)
        FBME_TIMED(prof, FBME_GROUP_CERTIFICATE,
                   (launch_dep(scan, dim3(nblk, s.B), kCertThreads, csm, st, A, cert->workspace)));
    }
  }
  FBME_TIMED(prof, FBME_GROUP_POLISH, (launch_dep(polish_finish_kernel, s.B, kPolishThreads, dsm, st, A, out)));
  const int fb = static_cast<int>((s.n() + 2047) / 2048);
  FBME_TIMED(prof, FBME_GROUP_OUTPUT, (launch_dep(output_kernel, dim3(fb < 64 ? fb : 64, s.B), 256, 0, st, A, out)));
}

// The polish of an uneven plan's buckets, one launch per step over all of
// them (at most kBucketSetMax per launch), in polish_run's order.  Buckets
// under an observation mask take polish_run.
static int exchange_class(int n2) { return n2 <= 64 ? 0 : n2 <= 128 ? 1 : n2 <= 256 ? 2 : 3; }

template <typename T>
static void launch_exchange_set(const PolishSet& S, int max_blocks, int max_b, int max_n2, cudaStream_t st) {
  launch_dep(exchange_set_kernel<T>, dim3(max_blocks, max_b, S.n), T::threads, T::smem_bytes(max_n2), st, S);
}

void polish_run_multi(const PolishBucket* b, int n, cudaStream_t st) {
  for (int c0 = 0; c0 < n; c0 += kBucketSetMax) {
    const int cnt = n - c0 < kBucketSetMax ? n - c0 : kBucketSetMax;
    std::vector<int> plain;  // set members (masked buckets run on their own)
    for (int i = 0; i < cnt; ++i) {
      const PolishBucket& k = b[c0 + i];
      if (k.p.gram2d) {
        polish_run(k.s, k.c, k.p, k.out, st);
        if (k.out.status && k.out.status != k.p.status)
          cudaMemcpyAsync(k.out.status, k.p.status, k.s.B * sizeof(int), cudaMemcpyDeviceToDevice, st);
      } else {
        plain.push_back(c0 + i);
      }
    }
    if (plain.empty()) continue;
    const int m = static_cast<int>(plain.size());
    auto* S = new PolishSet();  // ~31 KB: not on the stack
    TopkJobs tj{};
    S->n = m;
    tj.n = m;
    int max_b = 1, max_slices = 1, max_out = 1;
    size_t dsm = 0;
    for (int i = 0; i < m; ++i) {
      const PolishBucket& k = b[plain[i]];
      const int K = k.c.polish_size, sl = topk_slices(k.s.n());
      S->a[i] = PolishArgs{k.s, k.c, k.p};
      S->out[i] = k.out;
      S->slices[i] = sl;
      S->ex_blocks[i] = exchange_blocks(k.s);
      const int fb = static_cast<int>((k.s.n() + 2047) / 2048);
      S->out_blocks[i] = fb < 64 ? fb : 64;
      tj.j[i] = TopkJob{k.p.keys, k.s.n(), K, k.s.B, k.p.cand_key, k.p.cand_idx};
      max_b = std::max(max_b, k.s.B);
      max_slices = std::max(max_slices, sl);
      max_out = std::max(max_out, S->out_blocks[i]);
      dsm = std::max(dsm, static_cast<size_t>(k.s.n1 + k.s.n2) * sizeof(float2));
    }
    launch_topk_blocks_multi(tj, max_slices, max_b, st);
    launch_dep(polish_set_kernel, dim3(max_b, 1, m), kPolishThreads, dsm, st, *S, 0);
    // the exchange, one launch per row-tile class
    bool any = false;
    for (int cls = 0; cls < 4; ++cls) {
      auto* X = new PolishSet();
      int xb = 1, xbl = 1, xn2 = 1;
      X->n = 0;
      for (int i = 0; i < m; ++i) {
        const PolishArgs& A = S->a[i];
        if (!(A.c.exchange > 0 && A.c.polish_iters > 1) || exchange_class(A.s.n2) != cls) continue;
        X->a[X->n] = A;
        X->ex_blocks[X->n] = S->ex_blocks[i];
        xb = std::max(xb, A.s.B);
        xbl = std::max(xbl, S->ex_blocks[i]);
        xn2 = std::max(xn2, A.s.n2);
        ++X->n;
      }
      if (X->n > 0) {
        any = true;
        if (cls == 0) launch_exchange_set<ExSmall>(*X, xbl, xb, xn2, st);
        else if (cls == 1) launch_exchange_set<ExMid>(*X, xbl, xb, xn2, st);
        else if (cls == 2) launch_exchange_set<ExWide>(*X, xbl, xb, xn2, st);
        else launch_exchange_set<ExWidest>(*X, xbl, xb, xn2, st);
      }
      delete X;
    }
    if (any) launch_dep(polish_set_kernel, dim3(max_b, 1, m), kPolishThreads, dsm, st, *S, 1);
    launch_dep(polish_finish_set_kernel, dim3(max_b, 1, m), kPolishThreads, dsm, st, *S);
    launch_dep(output_set_kernel, dim3(max_out, max_b, m), 256, 0, st, *S);
    for (int i = 0; i < m; ++i) {
      const PolishBucket& k = b[plain[i]];
      if (k.out.status && k.out.status != k.p.status)
        cudaMemcpyAsync(k.out.status, k.p.status, k.s.B * sizeof(int), cudaMemcpyDeviceToDevice, st);
    }
    delete S;
  }
}

}  // namespace fbme

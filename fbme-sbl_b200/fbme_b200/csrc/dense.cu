// mode="dense": the exact posterior through the M x M data covariance
// (torch_sbl/solver.py:2962-2990 with 3025-3035; operators.py:282-297 and
// 418-442), per scene, in FP64 on the device:
//
//   lags      L(d) = sum_n gamma_n exp(-2 pi i d.n / N) for the sample lags
//             d in (-(M1-1)..M1-1) x (-(M2-1)..M2-1), separable (two passes)
//   Q         Q[i][j] = L(m_i - m_j) + noise delta_ij, plus the deterministic
//             loading of the CUDA Cholesky branch (m * eps64 * mean|diag|)
//   Q^-1      in place by blocked symmetric sweeps: 32-column panels, each
//             step one Hermitian rank-32 update of the whole lower triangle
//             that advances the Cholesky factor's trailing matrix, L^-1 and
//             L^-H L^-1 together (dense_sweep_kernel)
//   Q^-1 y, the lag sums of Q^-1 and the data diagonal
//             diag(A^H Q^-1 A) = Re N ifft2(lag sums); A^H Q^-1 y; the
//             residual energy from the identity y - A mean = (noise +
//             loading) Q^-1 y
//
// The reference's FP32 run loses the posterior variance gamma - gamma^2 dd to
// cancellation (its FP32 and FP64 runs differ by 50-230 times the norm on the
// C1 scenes); FP64 here keeps it, and matches the reference's FP64 run.
// Matrices are column-major ([j * M + i]) with the lower triangle in use.
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "stage.cuh"

namespace fbme {

namespace {

// The deterministic Cholesky loading m * eps * mean|diag| of the CUDA branch
// (solver.py:2907-2920) takes eps of the arithmetic's precision: FP64 here,
// as the reference's complex128 path does.
constexpr double kEps64 = 2.220446049250313e-16;
constexpr int kPanel = 32;   // panel width of the sweeps
constexpr int kDiagWarps = 8;
constexpr int kDiagCols = kPanel / kDiagWarps;
constexpr int kTile = 64;    // output tile of the update kernels

__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 warp_sum2(double2 v) {
  v.x = warp_sum(v.x);
  v.y = warp_sum(v.y);
  return v;
}

// exp(-2 pi i k / L), k < L, FP64
__global__ void dense_twiddle_kernel(double2* tw, int L) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= L) return;
  double s, c;
  sincospi(-2.0 * static_cast<double>(k) / static_cast<double>(L), &s, &c);
  tw[k] = make_double2(c, s);
}

// w^(sign e) for e = e0, e0 + step, e0 + 2 step, ... from the table of
// w = exp(-2 pi i / L): the exponent is kept reduced, one compare and
// subtract a term instead of a 64-bit remainder.
struct TwidStep {
  const double2* tw;
  int L, e, step;
  __device__ TwidStep(const double2* t, int len, long long e0, long long s)
      : tw(t), L(len), e(reduce(e0, len)), step(reduce(s, len)) {}
  static __device__ int reduce(long long v, int len) {
    const int r = static_cast<int>(v % len);
    return r < 0 ? r + len : r;
  }
  __device__ double2 next(int sign) {
    const double2 w = tw[e];
    e += step;
    if (e >= L) e -= L;
    return sign < 0 ? w : make_double2(w.x, -w.y);
  }
};

// One output of a separable pass on one warp: sum_k in(k) w^(sign (e0 +
// step k)), k < count, lanes over k (a thread per output left 16 blocks
// walking 64 terms each: 27 us a pass at 64 x 64, 6 us so).
template <typename F>
__device__ __forceinline__ double2 warp_dft(F in, int count, const double2* tw, int L, long long e0, long long step,
                                            int sign) {
  const int lane = threadIdx.x & 31;
  TwidStep t(tw, L, e0 + step * lane, 32 * step);
  double2 acc = make_double2(0.0, 0.0);
  for (int k = lane; k < count; k += 32) acc = zadd(acc, zmul(in(k), t.next(sign)));
  return warp_sum2(acc);
}
// Outputs t of a pass, one per warp.
#define FBME_WARP_OUTPUTS(total)                                                              \
  for (long long t = blockIdx.x * 8LL + (threadIdx.x >> 5); t < (total); t += gridDim.x * 8LL)

// Lag pass 1: T[b][n1][e2] = sum_n2 gamma[b][n1][n2] w2^(d2 n2), d2 = e2 - (M2 - 1)
__global__ void __launch_bounds__(256) dense_lag1_kernel(const float* gamma, int B, int n1, int n2, int m2,
                                                         const double2* tw2, double2* T) {
  const int W2 = 2 * m2 - 1;
  FBME_WARP_OUTPUTS(static_cast<long long>(B) * n1 * W2) {
    const int d2 = static_cast<int>(t % W2) - (m2 - 1);
    const float* g = gamma + t / W2 * n2;  // b * n1 + row
    const double2 v = warp_dft([&](int k) { return make_double2(g[k], 0.0); }, n2, tw2, n2, 0, d2, -1);
    if ((threadIdx.x & 31) == 0) T[t] = v;
  }
}

// Lag pass 2: lag[b][e1][e2] = sum_n1 w1^(d1 n1) T[b][n1][e2], d1 = e1 - (M1 - 1)
__global__ void __launch_bounds__(256) dense_lag2_kernel(const double2* T, int B, int n1, int m1, int m2,
                                                         const double2* tw1, double2* lag) {
  const int W1 = 2 * m1 - 1, W2 = 2 * m2 - 1;
  FBME_WARP_OUTPUTS(static_cast<long long>(B) * W1 * W2) {
    const int e2 = static_cast<int>(t % W2);
    const long long r = t / W2;
    const int d1 = static_cast<int>(r % W1) - (m1 - 1);
    const double2* tb = T + r / W1 * n1 * W2 + e2;
    const double2 v = warp_dft([&](int k) { return tb[static_cast<long long>(k) * W2]; }, n1, tw1, n1, 0, d1, -1);
    if ((threadIdx.x & 31) == 0) lag[t] = v;
  }
}

// Q (lower triangle, column-major) from the lags, noise and loading.
__global__ void dense_build_q_kernel(const double2* lag, int B, int m1, int m2, const float* noise, float jitter,
                                     double2* Q) {
  const int M = m1 * m2, W1 = 2 * m1 - 1, W2 = 2 * m2 - 1;
  const long long MM = static_cast<long long>(M) * M;
  const long long total = static_cast<long long>(B) * MM;
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int b = static_cast<int>(t / MM);
    const long long r = t - b * MM;
    const int j = static_cast<int>(r / M), i = static_cast<int>(r - static_cast<long long>(j) * M);
    if (i < j) continue;
    const int i1 = i / m2, i2 = i - (i / m2) * m2, j1 = j / m2, j2 = j - (j / m2) * m2;
    const double2* lb = lag + static_cast<long long>(b) * W1 * W2;
    double2 q = lb[(i1 - j1 + m1 - 1) * W2 + (i2 - j2 + m2 - 1)];
    if (i == j) {
      // every diagonal entry is L(0) + noise: the loading is m eps64 (L(0) + noise)
      const double dg = lb[(m1 - 1) * W2 + (m2 - 1)].x + noise[b];
      q = make_double2(dg + static_cast<double>(jitter) * kEps64 * fabs(dg), 0.0);
    }
    Q[t] = q;
  }
}


// ---------------------------------------------------------------------------
// Q^-1 by blocked symmetric sweeps, in place in the lower triangle of S
// ---------------------------------------------------------------------------
// With Q = L L^H and X = L^-1, before the sweep of panel [k, k + nb) entry
// (i, j), i >= j, of S holds
//     j >= k       the trailing matrix of the right-looking Cholesky,
//     j < k <= i   minus the sum that becomes X[i][j],
//     i < k        the sum over the swept rows r of conj(X[r][i]) X[r][j].
// Let Z = L11^-1 of the diagonal block and W (M x nb) the panel
//     W[r][c] = sum_c' s_r[c'] conj(Z[c][c']),   s_r = row r of the panel's
// columns of the Hermitian S (the identity's rows for r in the panel).  Then
// W[r] is row r of L below the panel and conj(column r of X) above and in
// it, and the whole sweep is D = W W^H: S -= D for the rows below the
// panel and S += D for the others, starting from zero in the panel's own
// rows (columns j <= k) and columns (rows i >= k).  After the last panel S is
// Q^-1.  Every sweep has the same work (M^2 / 2 entries, depth nb), which
// fills the GPU at M = 1024 (136 tiles), and takes one launch: each block
// forms the rows of W that its tile needs, and writes what becomes the next
// sweep's panel to a separate buffer, so that no block reads what another
// one writes; an extra block updates, factors and inverts the next diagonal
// block meanwhile.  What sets the time is that block's chain of 32 square
// roots.  Separate factor, inverse and product passes took five launches a
// panel, with 32-column triangular solves and a one-warp factorisation in
// series between them: 4.9 ms an EM iteration at M = 1024, 0.8 ms so.

// Factor and invert an nb x nb diagonal block on 256 threads: lane i owns
// row i, warp w columns w, w + 8, w + 16, w + 24 (r: its entries).  An
// entry is first the block's, then (once its column is posted) the sum that
// becomes the inverse's; the warp owning column q + 1 takes it first and
// arrives at its barrier without waiting, as its square root is the chain
// that sets the time.  Z (row-major, lower) goes to global memory.
struct DiagShared {
  double2 L[kPanel][kPanel + 1];  // by columns: L[q][i] is entry (i, q)
  double rl[kPanel];              // 1 / L[q][q]
};

__device__ __forceinline__ void diag_arrive(int q) {
  asm volatile("bar.arrive %0, %1;" ::"r"(1 + (q & 1)), "n"(32 * kDiagWarps) : "memory");
}
__device__ __forceinline__ void diag_sync(int q) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + (q & 1)), "n"(32 * kDiagWarps) : "memory");
}

__device__ __forceinline__ void diag_factor(DiagShared& S, double2 (&r)[kDiagCols], int nb, double2* Z, int* status) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int failed = 0;
  auto post = [&](int q, double2& v) {
    const double d = __shfl_sync(0xffffffffu, v.x, q);
    const double rq = rsqrt(d > 0.0 ? d : 2.2250738585072014e-308);
    S.L[q][lane] = lane > q ? make_double2(v.x * rq, v.y * rq) : make_double2(0.0, 0.0);
    S.rl[q] = rq;  // the same value from every lane
    __syncwarp();  // this warp reads the column without waiting at its barrier
    diag_arrive(q);
    v = make_double2(0.0, 0.0);
    failed |= d > 0.0 ? 0 : isfinite(d) ? FBME_STATUS_CHOLESKY : FBME_STATUS_NONFINITE;
  };
  auto sub_c = [](double2 v, double2 a, double2 b) {  // v - a conj(b)
    return make_double2(fma(-a.x, b.x, fma(-a.y, b.y, v.x)), fma(-a.y, b.x, fma(a.x, b.y, v.y)));
  };
  auto add_m = [](double2 v, double2 a, double2 b) {  // v + a b
    return make_double2(fma(a.x, b.x, fma(-a.y, b.y, v.x)), fma(a.x, b.y, fma(a.y, b.x, v.y)));
  };
  if (w == 0) post(0, r[0]);
#pragma unroll
  for (int uq = 0; uq < kDiagCols; ++uq) {
#pragma unroll 1
    for (int wq = 0; wq < kDiagWarps; ++wq) {
      const int q = kDiagWarps * uq + wq;
      if (q >= nb) break;
      if (w != wq) diag_sync(q);
      const double2 a = S.L[q][lane];
      const double rlq = S.rl[q];
      const int next = q + 1 < nb ? q + 1 : -1;
      if (wq + 1 < kDiagWarps) {
        if (w == wq + 1 && next > 0) {
          if (lane >= next) r[uq] = sub_c(r[uq], a, S.L[q][next]);
          post(next, r[uq]);
        }
      } else if (uq + 1 < kDiagCols) {
        if (w == 0 && next > 0) {
          if (lane >= next) r[uq + 1] = sub_c(r[uq + 1], a, S.L[q][next]);
          post(next, r[uq + 1]);
        }
      }
#pragma unroll
      for (int u = 0; u < kDiagCols; ++u) {
        const int j = w + kDiagWarps * u;
        const bool right = u > uq || (u == uq && w > wq);
        double2 v = r[u];
        if (u >= uq) {
          const double2 t = sub_c(r[u], a, S.L[q][j]);
          if (right && j != next && lane >= j) v = t;
        }
        if (u <= uq) {
          double2 xq = make_double2(__shfl_sync(0xffffffffu, r[u].x, q), __shfl_sync(0xffffffffu, r[u].y, q));
          xq = j == q ? make_double2(rlq, 0.0) : make_double2(-xq.x * rlq, -xq.y * rlq);
          const double2 t = add_m(r[u], a, xq);
          if (!right) {
            if (lane > q) v = t;
            if (lane == 0) Z[q * kPanel + j] = xq;
          }
        }
        r[u] = v;
      }
    }
  }
  if (failed && lane == 0 && status) atomicOr(status, failed);
}

// The first panel's diagonal block.
__global__ void __launch_bounds__(32 * kDiagWarps) dense_diag_kernel(const double2* Sm, double2* Z, int M, int* status) {
  __shared__ DiagShared S;
  const double2* A = Sm + static_cast<long long>(blockIdx.x) * M * M;
  const int nb = M < kPanel ? M : kPanel, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double2 r[kDiagCols];
#pragma unroll
  for (int u = 0; u < kDiagCols; ++u) {
    const int j = w + kDiagWarps * u;
    r[u] = (lane < nb && j < nb && lane >= j) ? A[static_cast<long long>(j) * M + lane] : make_double2(0.0, 0.0);
  }
  diag_factor(S, r, nb, Z + blockIdx.x * kPanel * kPanel, status ? status + blockIdx.x : nullptr);
}

// Shared memory of a sweep's block: the panel's rows of the tile's rows and
// columns, the conjugated Z, and the rows of W formed from them.
struct SweepShared {
  double2 src[2][kPanel][kTile];
  double2 W[2][kPanel][kTile];
  double2 z[kPanel][kPanel];
};
union SweepUnion {
  SweepShared s;
  struct {
    double2 src[kPanel][kPanel];
    double2 z[kPanel][kPanel];
    double2 W[kPanel][kPanel];
    DiagShared d;
  } g;
};

// The panel's rows r0 .. r0 + RB (RB = 32 or 64) into shared memory,
// asynchronous copies (the caller waits); the panel's own rows are the
// identity's.
template <int RB>
__device__ __forceinline__ void sweep_load(const double2* P, int M, int k, int nb, int r0, double2 (*src)[RB]) {
#pragma unroll
  for (int i = 0; i < kPanel * RB / 256; ++i) {
    const int e = threadIdx.x + 256 * i;
    const int c = e / RB, r = r0 + e % RB;
    double2* dst = &src[c][e % RB];
    if (!(r >= k && r < k + kPanel) && c < nb && r < M)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)),
                   "l"(P + static_cast<long long>(c) * M + r) : "memory");
    else
      *dst = make_double2(r - k == c ? 1.0 : 0.0, 0.0);
  }
}
__device__ __forceinline__ void sweep_wait() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
}

// Rows of W from the panel's: lane = row (and row + 32), warp w the columns
// w, w + 8, w + 16, w + 24.
template <int RB>
__device__ __forceinline__ void sweep_rows(const double2 (*src)[RB], const double2 (*z)[kPanel], double2 (*W)[RB]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int H = RB / 32;
  double2 acc[4][H];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int h = 0; h < H; ++h) acc[u][h] = make_double2(0.0, 0.0);
#pragma unroll
  for (int uc = 0; uc < 4; ++uc) {  // c' in [8 uc, 8 uc + 8): columns c < 8 uc have none
#pragma unroll 4
    for (int i = 0; i < 8; ++i) {
      const int cp = 8 * uc + i;
      double2 s[H];
#pragma unroll
      for (int h = 0; h < H; ++h) s[h] = src[cp][lane + 32 * h];
#pragma unroll
      for (int u = uc; u < 4; ++u) {  // z is zero above its diagonal
        const double2 f = z[w + 8 * u][cp];
#pragma unroll
        for (int h = 0; h < H; ++h) {
          acc[u][h].x = fma(s[h].x, f.x, fma(-s[h].y, f.y, acc[u][h].x));
          acc[u][h].y = fma(s[h].x, f.y, fma(s[h].y, f.x, acc[u][h].y));
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int h = 0; h < H; ++h) W[w + 8 * u][lane + 32 * h] = acc[u][h];
}

// Sweep k of scene blockIdx.y: block 0 the next diagonal block, the others
// one 64 x 64 tile of the lower triangle each; thread (ri, rj) of 16 x 16
// owns the rows i0 + ri + 16 a and columns j0 + rj + 16 b (a, b < 4), so that
// stores of consecutive threads are consecutive in a column.  P: this
// sweep's panel [c][r], Pn: the next one's, Z: this sweep's diagonal
// inverse, Zn: the next one's.  The last sweep stores both triangles.
__global__ void __launch_bounds__(256) dense_sweep_kernel(double2* Sm, const double2* Pm, double2* Pn, const double2* Zm,
                                                          double2* Zn, int M, int k, int* status) {
  extern __shared__ double2 sweep_shm[];
  SweepUnion& sh = *reinterpret_cast<SweepUnion*>(sweep_shm);
  const int scene = blockIdx.y;
  double2* S = Sm + static_cast<long long>(scene) * M * M;
  const double2* P = Pm + static_cast<long long>(scene) * kPanel * M;
  const double2* Z = Zm + scene * kPanel * kPanel;
  const int tid = threadIdx.x;
  const int k1 = k + kPanel < M ? k + kPanel : M, nb = k1 - k;
  auto load_z = [&](double2 (*z)[kPanel]) {
    for (int e = tid; e < kPanel * kPanel; e += 256) {
      const int c = e / kPanel, cp = e % kPanel;
      const double2 v = (c < nb && cp <= c) ? Z[e] : make_double2(0.0, 0.0);
      z[c][cp] = make_double2(v.x, -v.y);
    }
  };
  if (blockIdx.x == 0) {
    if (k1 >= M) return;
    const int nn = M - k1 < kPanel ? M - k1 : kPanel, lane = tid & 31, w = tid >> 5;
    double2 v[kDiagCols];  // the block's entries, loaded ahead of their update
#pragma unroll
    for (int u = 0; u < kDiagCols; ++u) {
      const int j = w + kDiagWarps * u;
      v[u] = (lane < nn && j < nn && lane >= j) ? S[static_cast<long long>(k1 + j) * M + k1 + lane]
                                                : make_double2(0.0, 0.0);
    }
    sweep_load<kPanel>(P, M, k, nb, k1, sh.g.src);
    load_z(sh.g.z);
    sweep_wait();
    sweep_rows<kPanel>(sh.g.src, sh.g.z, sh.g.W);
    __syncthreads();
#pragma unroll 8
    for (int c = 0; c < kPanel; ++c) {
      const double2 a = sh.g.W[c][lane];
#pragma unroll
      for (int u = 0; u < kDiagCols; ++u) {
        const double2 b = sh.g.W[c][w + kDiagWarps * u];
        v[u].x = fma(-a.x, b.x, fma(-a.y, b.y, v[u].x));
        v[u].y = fma(-a.y, b.x, fma(a.x, b.y, v[u].y));
      }
    }
    diag_factor(sh.g.d, v, nn, Zn + scene * kPanel * kPanel, status ? status + scene : nullptr);
    return;
  }
  const int t = blockIdx.x - 1;
  int ti = static_cast<int>((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
  while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
  while (ti * (ti + 1) / 2 > t) --ti;
  const int tj = t - ti * (ti + 1) / 2;
  const int i0 = ti * kTile, j0 = tj * kTile;
  const int ri = tid & 15, rj = tid >> 4;
  sweep_load<kTile>(P, M, k, nb, i0, sh.s.src[0]);
  if (ti != tj) sweep_load<kTile>(P, M, k, nb, j0, sh.s.src[1]);
  // the tile's entries, loaded ahead of the products; the panel's own rows
  // and columns start from zero
  double2 old[4][4];
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = i0 + ri + 16 * a, j = j0 + rj + 16 * b;
      const bool fresh = i >= k1 ? (j >= k && j < k1) : i >= k;
      old[a][b] = (i < M && i >= j && !fresh) ? S[static_cast<long long>(j) * M + i] : make_double2(0.0, 0.0);
    }
  load_z(sh.s.z);
  sweep_wait();
  sweep_rows<kTile>(sh.s.src[0], sh.s.z, sh.s.W[0]);
  if (ti != tj) sweep_rows<kTile>(sh.s.src[1], sh.s.z, sh.s.W[1]);
  __syncthreads();
  const double2(*Wi)[kTile] = sh.s.W[0];
  const double2(*Wj)[kTile] = ti != tj ? sh.s.W[1] : sh.s.W[0];
  double2 acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int d = 0; d < kPanel; ++d) {
    double2 av[4], bv[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) av[a] = Wi[d][ri + 16 * a];
#pragma unroll
    for (int b = 0; b < 4; ++b) bv[b] = Wj[d][rj + 16 * b];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {  // W_i conj(W_j)
        acc[a][b].x = fma(av[a].x, bv[b].x, fma(av[a].y, bv[b].y, acc[a][b].x));
        acc[a][b].y = fma(-av[a].x, bv[b].y, fma(av[a].y, bv[b].x, acc[a][b].y));
      }
  }
  double2* Pnext = Pn + static_cast<long long>(scene) * kPanel * M;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const int j = j0 + rj + 16 * b;
    if (j >= M) continue;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = i0 + ri + 16 * a;
      // the next diagonal block is block 0's, which reads it meanwhile
      if (i >= M || i < j || (j >= k1 && i < k1 + kPanel)) continue;
      double2* dst = S + static_cast<long long>(j) * M + i;
      const double2 o = old[a][b];
      const double2 v = i >= k1 ? make_double2(o.x - acc[a][b].x, o.y - acc[a][b].y) : zadd(o, acc[a][b]);
      // what the next sweep takes as its panel goes there alone
      if (j >= k1 && j < k1 + kPanel) Pnext[static_cast<long long>(j - k1) * M + i] = v;
      else if (i >= k1 && i < k1 + kPanel) Pnext[static_cast<long long>(i - k1) * M + j] = make_double2(v.x, -v.y);
      else *dst = v;
      if (k1 == M && i != j) S[static_cast<long long>(i) * M + j] = make_double2(v.x, -v.y);
    }
  }
}


// z = Q^-1 y (y complex64 [B][M]): one warp per row i, over column i of the
// Hermitian R (z_i = sum_j conj(R[j][i]) y_j), coalesced.
__global__ void __launch_bounds__(256) dense_qinv_y_kernel(const double2* R, const float2* y, int B, int M,
                                                            double2* z) {
  const int b = blockIdx.y;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= M) return;
  const double2* col = R + static_cast<long long>(b) * M * M + static_cast<long long>(i) * M;
  const float2* yb = y + static_cast<long long>(b) * M;
  double2 acc = make_double2(0.0, 0.0);
  for (int j = lane; j < M; j += 32) {
    const double2 r = col[j];
    const float2 v = yb[j];
    acc.x += r.x * v.x + r.y * v.y;  // conj(r) * v
    acc.y += r.x * v.y - r.y * v.x;
  }
  acc = warp_sum2(acc);
  if (lane == 0) z[static_cast<long long>(b) * M + i] = acc;
}

// Lag sums of Q^-1 (operators.py:427-435): S[e1][e2] = sum of R[i][j] over
// the sample pairs with m_i - m_j = (e1 - (M1-1), e2 - (M2-1)); one warp
// per lag, lanes over the pairs in a fixed order.
__global__ void __launch_bounds__(256) dense_lag_sum_kernel(const double2* R, int B, int m1, int m2,
                                                             double2* S) {
  const int M = m1 * m2, W1 = 2 * m1 - 1, W2 = 2 * m2 - 1;
  const long long total = static_cast<long long>(B) * W1 * W2;
  const long long t = blockIdx.x * 8LL + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= total) return;
  const int e2 = static_cast<int>(t % W2);
  const long long r = t / W2;
  const int e1 = static_cast<int>(r % W1), b = static_cast<int>(r / W1);
  const int d1 = e1 - (m1 - 1), d2 = e2 - (m2 - 1);
  const double2* Rb = R + static_cast<long long>(b) * M * M;
  const int a1lo = d1 > 0 ? d1 : 0, a1hi = d1 < 0 ? m1 + d1 : m1;
  const int a2lo = d2 > 0 ? d2 : 0, a2hi = d2 < 0 ? m2 + d2 : m2;
  const int w = a2hi - a2lo, cnt = (a1hi - a1lo) * w;
  const int shift = d1 * m2 + d2;  // j = i - shift
  double2 acc = make_double2(0.0, 0.0);
  for (int u = lane; u < cnt; u += 32) {
    const int a1 = a1lo + u / w, a2 = a2lo + u % w;
    const int i = a1 * m2 + a2;
    acc = zadd(acc, Rb[static_cast<long long>(i - shift) * M + i]);
  }
  acc = warp_sum2(acc);
  if (lane == 0) S[t] = acc;
}

// Inverse-sign separable transform of a W1 x W2 rectangle of frequencies
// (offsets o1, o2) to the N1 x N2 grid:
//   out[n1][n2] = sum_{e1,e2} S[e1][e2] exp(+2 pi i ((e1+o1) n1 / N1 + (e2+o2) n2 / N2))
// pass 1: U[b][e1][n2]; pass 2: out (complex, or its real part).
__global__ void __launch_bounds__(256) dense_inv1_kernel(const double2* S, int B, int W1, int W2, int o2, int n2,
                                                         const double2* tw2, double2* U) {
  FBME_WARP_OUTPUTS(static_cast<long long>(B) * W1 * n2) {
    const int k2 = static_cast<int>(t % n2);
    const double2* row = S + t / n2 * W2;  // b * W1 + e1
    const double2 v = warp_dft([&](int e) { return row[e]; }, W2, tw2, n2, static_cast<long long>(o2) * k2, k2, +1);
    if ((threadIdx.x & 31) == 0) U[t] = v;
  }
}
template <bool REAL>
__global__ void __launch_bounds__(256) dense_inv2_kernel(const double2* U, int B, int W1, int o1, int n1, int n2,
                                                         const double2* tw1, double2* out, double* out_re) {
  FBME_WARP_OUTPUTS(static_cast<long long>(B) * n1 * n2) {
    const int k2 = static_cast<int>(t % n2);
    const long long r = t / n2;
    const int k1 = static_cast<int>(r % n1);
    const double2* ub = U + r / n1 * W1 * n2 + k2;
    const double2 v = warp_dft([&](int e) { return ub[static_cast<long long>(e) * n2]; }, W1, tw1, n1,
                               static_cast<long long>(o1) * k1, k1, +1);
    if ((threadIdx.x & 31) == 0) {
      if (REAL)
        out_re[t] = v.x;
      else
        out[t] = v;
    }
  }
}

// Residual energy |y - A mean|^2 of the exact posterior: A Gamma A^H =
// Q - (noise + loading) I, so y - A Gamma A^H Q^-1 y = (noise + loading) z
// with z = Q^-1 y; FP64, into the energy slots of the scalar update
// (slot 2 of tile 0; its other warps' slots zero).
__global__ void __launch_bounds__(256) dense_energy_kernel(const double2* z, const double2* lag, const float* noise,
                                                          float jitter, int m1, int m2, double* part) {
  __shared__ double red[8];
  const int b = blockIdx.x, M = m1 * m2, W1 = 2 * m1 - 1, W2 = 2 * m2 - 1;
  double acc = 0.0;
  for (int i = threadIdx.x; i < M; i += blockDim.x) {
    const double2 v = z[static_cast<long long>(b) * M + i];
    acc += v.x * v.x + v.y * v.y;
  }
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double e = 0.0;
    for (int w = 0; w < 8; ++w) e += red[w];
    const double dg = lag[static_cast<long long>(b) * W1 * W2 + (m1 - 1) * W2 + (m2 - 1)].x + noise[b];
    const double load = static_cast<double>(noise[b]) + static_cast<double>(jitter) * kEps64 * fabs(dg);
    double* slot = part + static_cast<long long>(b) * kMaxTilesPerScene * kPartSlots + 2 * kPartWarps;
    slot[0] = load * load * e;
    for (int w = 1; w < kPartWarps; ++w) slot[w] = 0.0;
  }
}

// mean = gamma A^H Q^-1 y, posterior variance max(gamma - gamma^2 dd, 0),
// clipped relevance gamma dd (solver.py:3025-3029, 3156-3163); per-block
// relevance sums in partial slot 0, as cg_hutch_kernel's.
__global__ void __launch_bounds__(kEwThreads)
dense_finish_kernel(BatchShape s, const float* gamma, const double2* lift, const double* dd, float2* mean,
                    float* relc, float* pv_out, double* part) {
  __shared__ double red[32];
  const int b = blockIdx.y;
  const long long N = s.n();
  double acc = 0.0;
  for (long long n = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; n < N;
       n += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long e = b * N + n;
    const double g = gamma[e];
    const double2 l = lift[e];
    mean[e] = make_float2(static_cast<float>(g * l.x), static_cast<float>(g * l.y));
    const double d = dd[e];
    const float rc = static_cast<float>(fmin(fmax(g * d, 0.0), 1.0));
    relc[e] = rc;
    if (pv_out) pv_out[e] = static_cast<float>(fmax(g - g * g * d, 0.0));
    acc += rc;
  }
  write_block_partial(acc, red, part, b, blockIdx.x, 0 * kPartWarps);
}

// Blocks of eight warps, one warp an output.
int warp_grid(long long n) {
  const long long g = (n + 7) / 8;
  return static_cast<int>(g < 148 * 64 ? (g > 0 ? g : 1) : 148 * 64);
}
int grid_of(long long n) {
  const long long g = (n + 255) / 256;
  return static_cast<int>(g < 148 * 16 ? (g > 0 ? g : 1) : 148 * 16);
}

}  // namespace

// Workspace of the dense posterior: Q, swept in place to Q^-1, per scene (FP64
// complex M x M), the sweeps' panels and diagonal inverses (two each), lags, pass buffers, Q^-1 y, lift, data diagonal and
// the FP64 twiddle tables.
size_t dense_bytes(const BatchShape& s) {
  const size_t B = s.B, M = s.m(), N = s.n();
  const size_t W1 = 2 * s.m1 - 1, W2 = 2 * s.m2 - 1;
  auto up = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
  const size_t pass = std::max(std::max(static_cast<size_t>(s.n1) * W2, W1 * static_cast<size_t>(s.n2)),
                               static_cast<size_t>(s.m1) * s.n2);
  return up(B * M * M * sizeof(double2)) + 2 * up(B * kPanel * M * sizeof(double2)) +
         2 * up(B * kPanel * kPanel * sizeof(double2)) + 2 * up(B * W1 * W2 * sizeof(double2)) +
         up(B * pass * sizeof(double2)) + up(B * M * sizeof(double2)) + up(B * N * sizeof(double2)) +
         up(B * N * sizeof(double)) + up(s.n1 * sizeof(double2)) + up(s.n2 * sizeof(double2));
}

DenseBufs dense_bind(uint8_t* w, const BatchShape& s, cudaStream_t st) {
  const size_t B = s.B, M = s.m(), N = s.n();
  const size_t W1 = 2 * s.m1 - 1, W2 = 2 * s.m2 - 1;
  auto up = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
  const size_t pass = std::max(std::max(static_cast<size_t>(s.n1) * W2, W1 * static_cast<size_t>(s.n2)),
                               static_cast<size_t>(s.m1) * s.n2);
  DenseBufs d;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    uint8_t* p = w + o;
    o += up(bytes);
    return p;
  };
  d.Q = reinterpret_cast<double2*>(take(B * M * M * sizeof(double2)));
  for (int i = 0; i < 2; ++i) d.P[i] = reinterpret_cast<double2*>(take(B * kPanel * M * sizeof(double2)));
  for (int i = 0; i < 2; ++i) d.Z[i] = reinterpret_cast<double2*>(take(B * kPanel * kPanel * sizeof(double2)));
  d.lag = reinterpret_cast<double2*>(take(B * W1 * W2 * sizeof(double2)));
  d.lsum = reinterpret_cast<double2*>(take(B * W1 * W2 * sizeof(double2)));
  d.pass = reinterpret_cast<double2*>(take(B * pass * sizeof(double2)));
  d.z = reinterpret_cast<double2*>(take(B * M * sizeof(double2)));
  d.lift = reinterpret_cast<double2*>(take(B * N * sizeof(double2)));
  d.dd = reinterpret_cast<double*>(take(B * N * sizeof(double)));
  d.tw1 = reinterpret_cast<double2*>(take(s.n1 * sizeof(double2)));
  d.tw2 = reinterpret_cast<double2*>(take(s.n2 * sizeof(double2)));
  dense_twiddle_kernel<<<(s.n1 + 255) / 256, 256, 0, st>>>(d.tw1, s.n1);
  dense_twiddle_kernel<<<(s.n2 + 255) / 256, 256, 0, st>>>(d.tw2, s.n2);
  cudaFuncSetAttribute(dense_sweep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       static_cast<int>(sizeof(SweepUnion)));
  return d;
}

void dense_posterior(const BatchShape& s, const DenseBufs& d, const float* gamma, const float* noise,
                     const float2* y, float jitter, float2* mean, float* relc, float* pv_out, double* part, int nb,
                     int* status, cudaStream_t st) {
  const int B = s.B, M = static_cast<int>(s.m()), m1 = s.m1, m2 = s.m2, n1 = s.n1, n2 = s.n2;
  const int W1 = 2 * m1 - 1, W2 = 2 * m2 - 1;
  // lags of the prior and the data covariance
  dense_lag1_kernel<<<warp_grid(1LL * B * n1 * W2), 256, 0, st>>>(gamma, B, n1, n2, m2, d.tw2, d.pass);
  dense_lag2_kernel<<<warp_grid(1LL * B * W1 * W2), 256, 0, st>>>(d.pass, B, n1, m1, m2, d.tw1, d.lag);
  dense_build_q_kernel<<<grid_of(1LL * B * M * M), 256, 0, st>>>(d.lag, B, m1, m2, noise, jitter, d.Q);
  // Q^-1 in place; the first panel is Q's first columns
  const int T = (M + kTile - 1) / kTile;
  dense_diag_kernel<<<B, 32 * kDiagWarps, 0, st>>>(d.Q, d.Z[0], M, status);
  const size_t panel = sizeof(double2) * kPanel * M;
  cudaMemcpy2DAsync(d.P[0], panel, d.Q, sizeof(double2) * M * M, sizeof(double2) * std::min(kPanel, M) * M, B,
                    cudaMemcpyDeviceToDevice, st);
  for (int k = 0, i = 0; k < M; k += kPanel, i ^= 1)
    dense_sweep_kernel<<<dim3(1 + T * (T + 1) / 2, B), 256, sizeof(SweepUnion), st>>>(
        d.Q, d.P[i], d.P[i ^ 1], d.Z[i], d.Z[i ^ 1], M, k, status);
  dense_qinv_y_kernel<<<dim3((M + 7) / 8, B), 256, 0, st>>>(d.Q, y, B, M, d.z);
  dense_energy_kernel<<<B, 256, 0, st>>>(d.z, d.lag, noise, jitter, m1, m2, part);
  // data diagonal: Re N ifft2 of the lag sums
  dense_lag_sum_kernel<<<static_cast<int>((1LL * B * W1 * W2 + 7) / 8), 256, 0, st>>>(d.Q, B, m1, m2, d.lsum);
  dense_inv1_kernel<<<warp_grid(1LL * B * W1 * n2), 256, 0, st>>>(d.lsum, B, W1, W2, -(m2 - 1), n2, d.tw2, d.pass);
  dense_inv2_kernel<true><<<warp_grid(1LL * B * n1 * n2), 256, 0, st>>>(d.pass, B, W1, -(m1 - 1), n1, n2, d.tw1,
                                                                         nullptr, d.dd);
  // A^H Q^-1 y: the same transform of the M1 x M2 block
  dense_inv1_kernel<<<warp_grid(1LL * B * m1 * n2), 256, 0, st>>>(d.z, B, m1, m2, 0, n2, d.tw2, d.pass);
  dense_inv2_kernel<false><<<warp_grid(1LL * B * n1 * n2), 256, 0, st>>>(d.pass, B, m1, 0, n1, n2, d.tw1, d.lift,
                                                                          nullptr);
  dense_finish_kernel<<<dim3(nb, B), kEwThreads, 0, st>>>(s, gamma, d.lift, d.dd, mean, relc, pv_out, part);
}

}  // namespace fbme

// Hermitian eigensolver on the GPU in FP64: the Coulomb-matrix
// diagonalisation that feeds v^1/2 and the E basis (main_hvccfp0.f90:322-367,
// zhgv_d / zhgv_h in m_lapack.f90:64-104, 203-229).
//
// Parallel cyclic two-sided Jacobi: each step applies N/2 disjoint plane
// rotations chosen by a round-robin tournament ordering; a sweep is N-1
// steps.  A step is ONE kernel: the rotations of pairs k and l touch the
// 2 x 2 block (rows of k, columns of l) and nothing else, so each thread
// takes one block from A to the next A (two copies, as the angles of a step
// come from diagonal blocks that other blocks of threads are rotating) and
// further threads rotate the columns of V.  The complex rotation first
// removes the phase of a_pq, then applies the real Jacobi rotation with
// t = sgn(tau) / (|tau| + sqrt(1 + tau^2)).  Sweeps stop when the
// off-diagonal norm is below 1e-14 of the Frobenius norm.
//
// What bounds it: the chain of N-1 dependent steps a sweep, each a few
// microseconds of launch, L2 round trips and the angle's square roots.
// Programmatic dependent launch starts a step's blocks while the previous
// step ends.  n = 260: 3.9 us a step, 14.1 ms in all (12.8 us a step with
// three kernels, 46.3 ms).
// The generalised problem (-v) z = lambda O z is reduced with O^-1/2 built
// from a Jacobi solve of O.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>
#include "zgemm_f64.cuh"

namespace qsgw {

struct Rot {
  double c, s;        // real rotation
  double2 ph;         // e^{-i phi}, b = a_pq = |b| e^{i phi}
};

__device__ __forceinline__ void pair_of(int t, int k, int ne, int& p, int& q) {
  // round-robin: player ne-1 fixed, the others rotate
  if (k == 0) {
    p = ne - 1; q = t;
  } else {
    p = t + k; q = t - k;
    if (p >= ne - 1) p -= ne - 1;
    if (q < 0) q += ne - 1;
  }
  if (p > q) { const int x = p; p = q; q = x; }
}

// the rotation of pair (p, q), q < n.  No __restrict__ here and in the step kernel: A is written by the
// previous step, which may still run when this step's blocks start, so its loads must not be non-coherent.
__device__ __forceinline__ Rot rotation(const double2* A, long long lda, int p, int q) {
  Rot r{1.0, 0.0, make_double2(1.0, 0.0)};
  const double a = A[p + p * lda].x, d = A[q + q * lda].x;
  const double2 b = A[p + q * lda];
  const double ab2 = b.x * b.x + b.y * b.y;
  if (ab2 > 1e-300 && ab2 > 1e-36 * fabs(a * d)) {
    // t = sgn(tau) / (|tau| + sqrt(1 + tau^2)), tau = delta / |b|, multiplied through by |b|: two
    // independent square roots, one division and one reciprocal root stand between the loads and the rotation
    const double delta = 0.5 * (d - a);
    const double iab = rsqrt(ab2), ab = ab2 * iab;
    const double tt = copysign(ab / (fabs(delta) + sqrt(fma(delta, delta, ab2))), delta);
    r.c = rsqrt(fma(tt, tt, 1.0));
    r.s = tt * r.c;
    r.ph = make_double2(b.x * iab, -b.y * iab);
  }
  return r;
}

// columns (p, q) of one row: col_p' = c col_p - s e^{-i phi} col_q,  col_q' = s col_p + c e^{-i phi} col_q
__device__ __forceinline__ void rotate(double2& xp, double2& xq, const Rot& r, double2 ph) {
  const double2 a = xp, b = xq;
  const double2 eb = make_double2(ph.x * b.x - ph.y * b.y, ph.x * b.y + ph.y * b.x);
  xp = make_double2(r.c * a.x - r.s * eb.x, r.c * a.y - r.s * eb.y);
  xq = make_double2(r.s * a.x + r.c * eb.x, r.s * a.y + r.c * eb.y);
}

// One step t: B <- J^H A J and V <- V J.  Blocks x < nA take JT x JT pairs of A (thread = one 2 x 2 block),
// the others JT pairs x JVR rows of V.  An odd n pairs one index with the absent player ne - 1: it keeps
// its row and column.
constexpr int JT = 16, JVR = 64;
__global__ void __launch_bounds__(JT * JT) jacobi_step_kernel(const double2* A, double2* B, double2* V, int n, int ne, int t,
                                                              int nA, int ntile) {
  __shared__ Rot rk[JT], rl[JT];
  __shared__ int pl[JT][2];
  const int tid = threadIdx.x, npair = ne / 2;
  const bool isA = static_cast<int>(blockIdx.x) < nA;
  const int bi = isA ? blockIdx.x % ntile : (blockIdx.x - nA) / ntile;   // A: row pairs; V: row block
  const int bl = isA ? blockIdx.x / ntile : (blockIdx.x - nA) % ntile;   // column pairs
  // the previous step has to be complete before anything of it is read or overwritten
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // a block's elements are requested before the angles are formed
  const int ta = tid & (JT - 1), tb = tid / JT;
  int p0 = n, p1 = n, q0 = n, q1 = n;
  const double2 zero = make_double2(0.0, 0.0);
  double2 a00 = zero, a01 = zero, a10 = zero, a11 = zero;
  if (isA) {
    if (bi * JT + ta < npair) pair_of(t, bi * JT + ta, ne, p0, p1);
    if (bl * JT + tb < npair) pair_of(t, bl * JT + tb, ne, q0, q1);
    const double2 *c0 = A + static_cast<long long>(q0) * n, *c1 = A + static_cast<long long>(q1) * n;
    if (p0 < n && q0 < n) a00 = c0[p0];
    if (p0 < n && q1 < n) a01 = c1[p0];
    if (p1 < n && q0 < n) a10 = c0[p1];
    if (p1 < n && q1 < n) a11 = c1[p1];
  }
  if (tid < 2 * JT) {
    const bool col = tid < JT;
    const int k = (col ? bl : bi) * JT + ta;
    int p = n, q = n;
    Rot r{1.0, 0.0, make_double2(1.0, 0.0)};
    if ((col || isA) && k < npair) {
      pair_of(t, k, ne, p, q);
      if (q < n) r = rotation(A, n, p, q);
    }
    (col ? rl : rk)[ta] = r;
    if (col) { pl[ta][0] = p; pl[ta][1] = q; }
  }
  __syncthreads();
  if (isA) {
    const Rot r = rk[ta], c = rl[tb];
    if (c.s != 0.0) {
      rotate(a00, a01, c, c.ph);
      rotate(a10, a11, c, c.ph);
    }
    if (r.s != 0.0) {                                 // rows: the conjugate phase
      const double2 cph = make_double2(r.ph.x, -r.ph.y);
      rotate(a00, a10, r, cph);
      rotate(a01, a11, r, cph);
    }
    double2 *c0 = B + static_cast<long long>(q0) * n, *c1 = B + static_cast<long long>(q1) * n;
    if (p0 < n && q0 < n) c0[p0] = a00;
    if (p0 < n && q1 < n) c1[p0] = a01;
    if (p1 < n && q0 < n) c0[p1] = a10;
    if (p1 < n && q1 < n) c1[p1] = a11;
  } else {
    const int i = bi * JVR + (tid & (JVR - 1));
    if (i >= n) return;
#pragma unroll
    for (int u = 0; u < JT * JVR / (JT * JT); ++u) {
      const int l = tid / JVR + u * (JT * JT / JVR);
      const Rot c = rl[l];
      if (c.s == 0.0) continue;                       // also the pairs without a second index
      double2 *xp = V + i + static_cast<long long>(pl[l][0]) * n, *xq = V + i + static_cast<long long>(pl[l][1]) * n;
      double2 a = *xp, b = *xq;
      rotate(a, b, c, c.ph);
      *xp = a;
      *xq = b;
    }
  }
}

// off-diagonal and total squared norms -> out[0], out[1]
__global__ void offdiag_norm_kernel(const double2* __restrict__ A, long long lda, int n, double* out) {
  double off = 0.0, tot = 0.0;
  const long long nn = static_cast<long long>(n) * n;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < nn;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(e % n), j = static_cast<int>(e / n);
    const double2 v = A[i + j * lda];
    const double m = v.x * v.x + v.y * v.y;
    tot += m;
    if (i != j) off += m;
  }
  for (int o = 16; o; o >>= 1) {
    off += __shfl_xor_sync(0xffffffffu, off, o);
    tot += __shfl_xor_sync(0xffffffffu, tot, o);
  }
  if ((threadIdx.x & 31) == 0) { atomicAdd(out, off); atomicAdd(out + 1, tot); }
}

__global__ void set_identity_kernel(double2* V, long long ldv, int n) {
  const long long nn = static_cast<long long>(n) * n;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < nn;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(e % n), j = static_cast<int>(e / n);
    V[i + j * ldv] = make_double2(i == j ? 1.0 : 0.0, 0.0);
  }
}

__global__ void diag_kernel(const double2* A, long long lda, int n, double* d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) d[i] = A[i + i * lda].x;
}

// out(:, j) = V(:, perm[j]) * colscale[j]
__global__ void permute_cols_kernel(double2* __restrict__ out, long long ldo, const double2* __restrict__ V,
                                    long long ldv, int n, const int* __restrict__ perm) {
  const long long nn = static_cast<long long>(n) * n;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < nn;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(e % n), j = static_cast<int>(e / n);
    out[i + j * ldo] = V[i + static_cast<long long>(perm[j]) * ldv];
  }
}

// M(:, j) *= f[j]
__global__ void scale_cols_kernel(double2* M, long long ld, int n, const double* f) {
  const long long nn = static_cast<long long>(n) * n;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < nn;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(e % n), j = static_cast<int>(e / n);
    double2& v = M[i + j * ld];
    v.x *= f[j]; v.y *= f[j];
  }
}

static DevBuf g_jc_b, g_jc_norm, g_jc_d, g_jc_v, g_jc_w, g_jc_x, g_jc_perm;

static int grid_for(long long n) {
  return static_cast<int>(std::max<long long>(1, std::min<long long>((n + 255) / 256, 16LL * ctx().sm_count)));
}

// A (n x n Hermitian, kept): V (n x n) <- eigenvectors; d <- unsorted eigenvalues (host).
static int jacobi_solve(double2* A, long long lda, double2* V, int n, std::vector<double>& d, cudaStream_t s) {
  const int ne = n + (n & 1);
  const int npair = ne / 2;
  // the two copies the steps go back and forth between (ld n)
  int rc = g_jc_b.ensure(2 * static_cast<size_t>(n) * n * sizeof(double2));
  if (rc) return rc;
  rc = g_jc_norm.ensure(2 * sizeof(double));
  if (rc) return rc;
  rc = g_jc_d.ensure(n * sizeof(double));
  if (rc) return rc;
  double2* cur = g_jc_b.as<double2>();
  double2* nxt = cur + static_cast<size_t>(n) * n;
  const size_t row = static_cast<size_t>(n) * sizeof(double2);
  QSGW_CUDA(cudaMemcpy2DAsync(cur, row, A, lda * sizeof(double2), row, n, cudaMemcpyDeviceToDevice, s));
  const int ntile = (npair + JT - 1) / JT, nA = ntile * ntile, nV = ntile * ((n + JVR - 1) / JVR);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(nA + nV));
  cfg.blockDim = dim3(JT * JT);
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  set_identity_kernel<<<grid_for(static_cast<long long>(n) * n), 256, 0, s>>>(V, n, n);
  count_launch();
  bool converged = (n <= 1);
  for (int sweep = 0; sweep < 40 && !converged; ++sweep) {
    for (int t = 0; t < ne - 1; ++t) {
      QSGW_CUDA(cudaLaunchKernelEx(&cfg, jacobi_step_kernel, static_cast<const double2*>(cur), nxt, V, n, ne, t, nA,
                                   ntile));
      std::swap(cur, nxt);
    }
    count_launch(ne - 1);
    QSGW_LAUNCH_CHECK("jacobi sweep");
    QSGW_CUDA(cudaMemsetAsync(g_jc_norm.p, 0, 2 * sizeof(double), s));
    offdiag_norm_kernel<<<grid_for(static_cast<long long>(n) * n), 256, 0, s>>>(cur, n, n, g_jc_norm.as<double>());
    count_launch();
    double h[2] = {0.0, 0.0};
    QSGW_CUDA(cudaMemcpyAsync(h, g_jc_norm.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
    QSGW_CUDA(cudaStreamSynchronize(s));
    if (!std::isfinite(h[0]) || !std::isfinite(h[1])) {
      set_error("zhegv: non-finite matrix entries");
      return QSGW_ERR_NUMERIC;
    }
    converged = h[0] <= 1e-28 * h[1];
  }
  if (!converged) {
    set_error("zhegv: Jacobi sweeps did not converge");
    return QSGW_ERR_NUMERIC;
  }
  diag_kernel<<<(n + 127) / 128, 128, 0, s>>>(cur, n, n, g_jc_d.as<double>());
  count_launch();
  d.resize(n);
  QSGW_CUDA(cudaMemcpyAsync(d.data(), g_jc_d.p, n * sizeof(double), cudaMemcpyDeviceToHost, s));
  QSGW_CUDA(cudaStreamSynchronize(s));
  return QSGW_OK;
}

}  // namespace qsgw

using namespace qsgw;

extern "C" int qsgw_zhegv_d(double* v_d, const double* o_d, int n, int lda, double* vcoud) {
  int rc = require_init();
  if (rc) return rc;
  QSGW_ARG(v_d && vcoud && n >= 1 && lda >= n, "zhegv: n=%d lda=%d", n, lda);
  cudaStream_t s = ctx().stream;
  const long long nn = static_cast<long long>(n) * n;
  rc = g_jc_v.ensure(nn * sizeof(double2));
  if (rc) return rc;
  rc = g_jc_w.ensure(nn * sizeof(double2));
  if (rc) return rc;
  double2* V = g_jc_v.as<double2>();
  double2* W = g_jc_w.as<double2>();
  double2* A = reinterpret_cast<double2*>(v_d);
  double2* Oh = nullptr;                         // O^-1/2 when an overlap is given
  if (o_d) {
    rc = g_jc_x.ensure(2 * nn * sizeof(double2));
    if (rc) return rc;
    double2* X = g_jc_x.as<double2>();           // working copy of O, then O^-1/2
    double2* Y = X + nn;
    QSGW_CUDA(cudaMemcpy2DAsync(X, n * sizeof(double2), o_d, lda * sizeof(double2), n * sizeof(double2), n,
                                cudaMemcpyDeviceToDevice, s));
    std::vector<double> mu;
    rc = jacobi_solve(X, n, V, n, mu, s);
    if (rc) return rc;
    std::vector<double> f(n);
    for (int j = 0; j < n; ++j) {
      if (!(mu[j] > 0.0)) {
        set_error("zhegv: overlap matrix is not positive definite");
        return QSGW_ERR_NUMERIC;
      }
      f[j] = 1.0 / std::sqrt(mu[j]);
    }
    rc = g_jc_d.ensure(n * sizeof(double));
    if (rc) return rc;
    QSGW_CUDA(cudaMemcpyAsync(g_jc_d.p, f.data(), n * sizeof(double), cudaMemcpyHostToDevice, s));
    // Y = U diag(mu^-1/2), X = Y U^H = O^-1/2
    QSGW_CUDA(cudaMemcpyAsync(Y, V, nn * sizeof(double2), cudaMemcpyDeviceToDevice, s));
    scale_cols_kernel<<<grid_for(nn), 256, 0, s>>>(Y, n, n, g_jc_d.as<double>());
    count_launch();
    rc = zgemm_f64(0, 2, n, n, n, make_double2(1, 0), Y, n, 0, V, n, 0, make_double2(0, 0), X, n, 0, 1, s);
    if (rc) return rc;
    // A <- O^-1/2 v O^-1/2
    rc = zgemm_f64(0, 0, n, n, n, make_double2(1, 0), A, lda, 0, X, n, 0, make_double2(0, 0), W, n, 0, 1, s);
    if (rc) return rc;
    rc = zgemm_f64(0, 0, n, n, n, make_double2(1, 0), X, n, 0, W, n, 0, make_double2(0, 0), A, lda, 0, 1, s);
    if (rc) return rc;
    Oh = X;
  }
  std::vector<double> lam;
  rc = jacobi_solve(A, lda, V, n, lam, s);
  if (rc) return rc;
  // descending eigenvalues of v = ascending eigenvalues of -v (main_hvccfp0.f90:339, vcoud = -eb)
  std::vector<int> perm(n);
  std::iota(perm.begin(), perm.end(), 0);
  std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) { return lam[a] > lam[b]; });
  for (int j = 0; j < n; ++j) vcoud[j] = lam[perm[j]];
  rc = g_jc_perm.ensure(n * sizeof(int));
  if (rc) return rc;
  QSGW_CUDA(cudaMemcpyAsync(g_jc_perm.p, perm.data(), n * sizeof(int), cudaMemcpyHostToDevice, s));
  if (Oh) {
    // z = O^-1/2 y
    rc = zgemm_f64(0, 0, n, n, n, make_double2(1, 0), Oh, n, 0, V, n, 0, make_double2(0, 0), W, n, 0, 1, s);
    if (rc) return rc;
    permute_cols_kernel<<<grid_for(nn), 256, 0, s>>>(A, lda, W, n, n, g_jc_perm.as<int>());
  } else {
    permute_cols_kernel<<<grid_for(nn), 256, 0, s>>>(A, lda, V, n, n, g_jc_perm.as<int>());
  }
  count_launch();
  QSGW_LAUNCH_CHECK("permute_cols_kernel");
  QSGW_CUDA(cudaStreamSynchronize(s));
  return QSGW_OK;
}

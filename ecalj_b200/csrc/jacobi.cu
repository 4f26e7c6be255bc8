// Hermitian eigensolver on the GPU in FP64: the Coulomb-matrix
// diagonalisation that feeds v^1/2 and the E basis (main_hvccfp0.f90:322-367,
// zhgv_d / zhgv_h in m_lapack.f90:64-104, 203-229).
//
// Parallel cyclic block Jacobi.  The matrix is cut into blocks of 16 rows; a
// step pairs the blocks by a round-robin tournament (a sweep meets every
// pair of blocks once) and is two kernels: jacobi_solve_kernel runs the
// plane rotations of the 32 x 32 diagonal problem of each pair in shared
// memory and leaves its unitary U, jacobi_apply_kernel forms
// A <- U^H A U and V <- V U block by block.  A plane rotation first removes
// the phase of a_pq, then applies the real Jacobi rotation with
// t = sgn(tau) / (|tau| + sqrt(1 + tau^2)).  Sweeps stop when the
// off-diagonal norm is below 1e-14 of the Frobenius norm.
//
// What bounds it: chains of dependent steps, not arithmetic.  Rotations
// between global steps cost a launch and an L2 round trip each (3.9 us at
// n = 260, N-1 of them a sweep); inside a block's 32 x 32 problem a set of
// rotations is two barriers and the angle's square roots (0.9 us).  So a
// step rotates only the 256 pairs between its two blocks (16 sets), and the
// pairs inside the blocks once a sweep: the sweeps needed are those of all
// 31 sets in every step (15 against 16 at n = 260 with eigenvalues over five
// decades, 30 against 29 with four eigenvalues in all), their length half.
// The angles have a warp of their own, which forms the next set's while the
// others bring U up to date.  Programmatic dependent launch overlaps the
// launches.  n = 260: 23 us a step, 17 steps a sweep: 5.9 ms (10.0 with 31
// sets in every step, 14.1 with a global step per rotation set, 46.3 with
// three launches for each); updates by 128 threads a tile 6.2 ms.  Angles
// formed in FP32 (rotations normalised in FP64) did not converge at n = 160.
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

constexpr int JB = 16, JW = 2 * JB, JP = JW + 1;     // block width, pair width, shared-memory pitch
constexpr int JT = JB * JB + 32;                     // threads of the solve: the 2 x 2 blocks and a warp for the angles
constexpr int JA = 256, JV = JW * JB / JA;             // threads of an update, columns of its 2-row strips

// global index of slot i (0..31) of the block pair (P, Q): P's rows, then Q's; n for an absent one
__device__ __forceinline__ int slot_index(int i, int P, int Q, int n) {
  const int blk = i < JB ? P : Q, g = blk * JB + (i & (JB - 1));
  return g < n ? g : n;
}

// The plane rotations of step t for every block pair (P, Q): the 16 x 16 pairs between the blocks, in the
// first step of a sweep those inside the blocks as well, so that a sweep meets each pair once.  U[pair]
// (32 x 32, column-major) <- the unitary.  Absent slots are zero rows and columns: nothing rotates with
// them.  Thread = one 2 x 2 block of a rotation set, the ninth warp the set's angles; two copies of the
// problem, as a set's angles come from blocks other threads are rotating.  U takes a set's rotations while
// the next angles are formed.
// No __restrict__ on A: the previous kernel, which may still run when these blocks start, writes it.
__global__ void __launch_bounds__(JT) jacobi_solve_kernel(const double2* A, double2* U, int n, int ne, int t) {
  extern __shared__ double2 jac_smem[];
  double2* sa[2] = {jac_smem, jac_smem + JW * JP};
  double2* su = jac_smem + 2 * JW * JP;
  __shared__ Rot rot[JB];
  const int tid = threadIdx.x, kb = tid & (JB - 1), lb = (tid / JB) & (JB - 1);
  const bool work = tid < JB * JB, angle = tid >= JB * JB && tid < JB * JB + JB;
  int P, Q;
  pair_of(t, blockIdx.x, ne, P, Q);
  const bool all = t == 0;                              // pairs inside the blocks too
  const int nset = all ? JW - 1 : JB;
  auto pair = [&](int st, int k, int& p, int& q) {
    if (all) {
      pair_of(st, k, JW, p, q);
    } else {
      p = k;
      q = JB + ((k + st) & (JB - 1));
    }
  };
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (work) {
#pragma unroll
    for (int e = 0; e < JW * JW / (JB * JB); ++e) {
      const int i = tid & (JW - 1), j = tid / JW + e * (JB * JB / JW);
      const int gi = slot_index(i, P, Q, n), gj = slot_index(j, P, Q, n);
      sa[0][i + j * JP] = (gi < n && gj < n) ? A[gi + static_cast<long long>(gj) * n] : make_double2(0.0, 0.0);
      su[i + j * JP] = make_double2(i == j ? 1.0 : 0.0, 0.0);
    }
  }
  __syncthreads();
  Rot c{1.0, 0.0, make_double2(1.0, 0.0)};              // the columns' rotation, still to be applied to U
  int u0 = 0, u1 = 0;
  auto rotate_u = [&]() {                               // U's columns u0, u1: rows kb, kb + 16
    if (c.s != 0.0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double2 *xp = su + (kb + h * JB) + u0 * JP, *xq = su + (kb + h * JB) + u1 * JP;
        double2 x = *xp, y = *xq;
        rotate(x, y, c, c.ph);
        *xp = x;
        *xq = y;
      }
    }
  };
  for (int st = 0; st < nset; ++st) {
    const double2* cur = sa[st & 1];
    double2* nxt = sa[(st & 1) ^ 1];
    if (angle) {
      int p, q;
      pair(st, kb, p, q);
      rot[kb] = rotation(cur, JP, p, q);
    }
    int p0, p1, q0, q1;
    double2 a00, a01, a10, a11;
    if (work) {
      pair(st, kb, p0, p1);
      pair(st, lb, q0, q1);
      a00 = cur[p0 + q0 * JP], a01 = cur[p0 + q1 * JP], a10 = cur[p1 + q0 * JP], a11 = cur[p1 + q1 * JP];
      rotate_u();
    }
    __syncthreads();
    if (work) {
      const Rot r = rot[kb];
      c = rot[lb];
      u0 = q0, u1 = q1;
      rotate(a00, a01, c, c.ph);
      rotate(a10, a11, c, c.ph);
      const double2 cph = make_double2(r.ph.x, -r.ph.y);              // rows: the conjugate phase
      rotate(a00, a10, r, cph);
      rotate(a01, a11, r, cph);
      nxt[p0 + q0 * JP] = a00;
      nxt[p0 + q1 * JP] = a01;
      nxt[p1 + q0 * JP] = a10;
      nxt[p1 + q1 * JP] = a11;
    }
    __syncthreads();
  }
  if (!work) return;
  rotate_u();
  asm volatile("bar.sync 1, %0;" ::"n"(JB * JB) : "memory");          // the working warps
  double2* Up = U + static_cast<long long>(blockIdx.x) * JW * JW;
#pragma unroll
  for (int e = 0; e < JW * JW / (JB * JB); ++e) {
    const int i = tid & (JW - 1), j = tid / JW + e * (JB * JB / JW);
    Up[i + j * JW] = su[i + j * JP];
  }
}

// out(2 x JV per thread) = op(X) Y for 32 x 32 tiles in shared memory; CONJ: X^H
template <bool CONJ>
__device__ __forceinline__ void tile_product(double2 (&o)[2][JV], const double2* X, const double2* Y, int i0, int j0) {
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < JV; ++v) o[u][v] = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int k = 0; k < JW; ++k) {
    double2 x[2], y[JV];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      x[u] = CONJ ? X[k + (i0 + 16 * u) * JP] : X[i0 + 16 * u + k * JP];
      if (CONJ) x[u].y = -x[u].y;
    }
#pragma unroll
    for (int v = 0; v < JV; ++v) y[v] = Y[k + (j0 + v) * JP];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < JV; ++v) {
        o[u][v].x += x[u].x * y[v].x - x[u].y * y[v].y;
        o[u][v].y += x[u].x * y[v].y + x[u].y * y[v].x;
      }
  }
}

// A <- U^H A U (blocks x < npair^2: pair of rows k, pair of columns l, in place) and V <- V U (the others: 32
// rows of V, pair l)
__global__ void __launch_bounds__(JA) jacobi_apply_kernel(double2* A, double2* V, const double2* U, int n, int ne,
                                                           int t, int npair) {
  extern __shared__ double2 jac_smem[];
  double2 *sx = jac_smem, *sl = sx + JW * JP, *sk = sl + JW * JP;
  const int tid = threadIdx.x, i0 = tid & 15, j0 = (tid >> 4) * JV;
  const bool isA = static_cast<int>(blockIdx.x) < npair * npair;
  const int b = isA ? blockIdx.x : blockIdx.x - npair * npair;
  const int l = b % npair, k = b / npair;               // V: k = row block
  int P, Q, R, S;
  pair_of(t, l, ne, P, Q);
  pair_of(t, k, ne, R, S);                              // unused for V
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  double2* M = isA ? A : V;
#pragma unroll
  for (int e = 0; e < JW * JW / JA; ++e) {
    const int i = tid & (JW - 1), j = tid / JW + e * (JA / JW);
    const int gi = isA ? slot_index(i, R, S, n) : (k * JW + i < n ? k * JW + i : n), gj = slot_index(j, P, Q, n);
    sx[i + j * JP] = (gi < n && gj < n) ? M[gi + static_cast<long long>(gj) * n] : make_double2(0.0, 0.0);
    sl[i + j * JP] = U[static_cast<long long>(l) * JW * JW + i + j * JW];
    if (isA) sk[i + j * JP] = U[static_cast<long long>(k) * JW * JW + i + j * JW];
  }
  __syncthreads();
  double2 o[2][JV];
  tile_product<false>(o, sx, sl, i0, j0);
  if (isA) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < JV; ++v) sx[i0 + 16 * u + (j0 + v) * JP] = o[u][v];
    __syncthreads();
    tile_product<true>(o, sk, sx, i0, j0);
  }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < JV; ++v) {
      const int i = i0 + 16 * u;
      const int gi = isA ? slot_index(i, R, S, n) : (k * JW + i < n ? k * JW + i : n), gj = slot_index(j0 + v, P, Q, n);
      if (gi < n && gj < n) M[gi + static_cast<long long>(gj) * n] = o[u][v];
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

// the largest finite |Re|, |Im| of A as ordered bits (NaN and infinities are left to the norms)
__global__ void absmax_kernel(const double2* __restrict__ A, long long lda, int n, unsigned long long* mx) {
  double m = 0.0;
  const long long nn = static_cast<long long>(n) * n;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < nn;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const double2 v = A[e % n + e / n * lda];
    const double x = fmax(fabs(v.x), fabs(v.y));
    if (isfinite(x)) m = fmax(m, x);
  }
  for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(mx, static_cast<unsigned long long>(__double_as_longlong(m)));
}

// The power of two that brings a small matrix up to entries of order one: squares of its entries would underflow.  A
// large one stays: its squares overflow in the norm, which refuses it.
__device__ __forceinline__ int small_exponent(const unsigned long long* mx) {
  const double m = __longlong_as_double(static_cast<long long>(*mx));
  return m > 0.0 ? min(ilogb(m), 0) : 0;
}
__global__ void scaled_copy_kernel(double2* __restrict__ out, const double2* __restrict__ A, long long lda, int n,
                                   const unsigned long long* __restrict__ mx) {
  const int ex = -small_exponent(mx);
  const long long nn = static_cast<long long>(n) * n;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < nn;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const double2 v = A[e % n + e / n * lda];
    out[e] = make_double2(scalbn(v.x, ex), scalbn(v.y, ex));
  }
}

__global__ void diag_kernel(const double2* A, long long lda, int n, const unsigned long long* mx, double* d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) d[i] = scalbn(A[i + i * lda].x, small_exponent(mx));
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
  const int nb = (n + JB - 1) / JB;
  const int ne = nb + (nb & 1);                         // an odd block count pairs one block with an absent one
  const int npair = ne / 2, nrow = (n + JW - 1) / JW;
  const size_t nn = static_cast<size_t>(n) * n;
  // working copy of A (ld n, scaled), then the pairs' unitaries
  int rc = g_jc_b.ensure((nn + static_cast<size_t>(npair) * JW * JW) * sizeof(double2));
  if (rc) return rc;
  rc = g_jc_norm.ensure(2 * sizeof(double) + sizeof(unsigned long long));   // norms, largest entry
  if (rc) return rc;
  rc = g_jc_d.ensure(n * sizeof(double));
  if (rc) return rc;
  double2* cur = g_jc_b.as<double2>();
  double2* U = cur + nn;
  unsigned long long* mx = reinterpret_cast<unsigned long long*>(g_jc_norm.as<double>() + 2);
  QSGW_CUDA(cudaMemsetAsync(mx, 0, sizeof(*mx), s));
  absmax_kernel<<<grid_for(static_cast<long long>(nn)), 256, 0, s>>>(A, lda, n, mx);
  scaled_copy_kernel<<<grid_for(static_cast<long long>(nn)), 256, 0, s>>>(cur, A, lda, n, mx);
  count_launch(2);
  QSGW_LAUNCH_CHECK("scaled_copy_kernel");
  constexpr int SMEM = 3 * JW * JP * static_cast<int>(sizeof(double2));
  static uint64_t at_solve = 0, at_apply = 0;           // one bit per device
  if ((rc = smem_limit_once(reinterpret_cast<const void*>(jacobi_solve_kernel), SMEM, at_solve))) return rc;
  if ((rc = smem_limit_once(reinterpret_cast<const void*>(jacobi_apply_kernel), SMEM, at_apply))) return rc;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t solve{}, apply{};
  solve.gridDim = dim3(static_cast<unsigned>(npair));
  solve.blockDim = dim3(JT);
  apply.gridDim = dim3(static_cast<unsigned>(npair * npair + nrow * npair));
  apply.blockDim = dim3(JA);
  for (cudaLaunchConfig_t* c : {&solve, &apply}) {
    c->dynamicSmemBytes = SMEM;
    c->stream = s;
    c->attrs = &attr;
    c->numAttrs = 1;
  }
  set_identity_kernel<<<grid_for(static_cast<long long>(n) * n), 256, 0, s>>>(V, n, n);
  count_launch();
  bool converged = (n <= 1);
  // many equal eigenvalues are the slow case: 25, 32, 34, 38 and 40 sweeps at n = 64, 260, 400, 800 and 1500 with four
  // in all, 27, 37, 34, 42 and 44 with two
  for (int sweep = 0; sweep < 60 && !converged; ++sweep) {
    for (int t = 0; t < ne - 1; ++t) {
      QSGW_CUDA(cudaLaunchKernelEx(&solve, jacobi_solve_kernel, static_cast<const double2*>(cur), U, n, ne, t));
      QSGW_CUDA(cudaLaunchKernelEx(&apply, jacobi_apply_kernel, cur, V, static_cast<const double2*>(U), n, ne, t, npair));
    }
    count_launch(2 * (ne - 1));
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
  diag_kernel<<<(n + 127) / 128, 128, 0, s>>>(cur, n, n, mx, g_jc_d.as<double>());
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

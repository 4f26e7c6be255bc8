// Complex FP64 GEMM engine on the FP64 tensor pipe (mma.sync m16n8k8 f64,
// "DMMA"), shared by chi0 (x0gemm), W (basis changes, Gauss-Jordan updates)
// and Sigma_c.  One CTA computes a 64x64 complex tile with 8 warps (each
// 32x16 = 2x2 m16n8 fragments, re and im accumulators); operands stream
// through a 3-stage cp.async pipeline in shared memory laid out [k][row]
// with a pitch of 66 complex (conflict-free fragment loads).
//
// What bounds it: the FP64 tensor pipe (64 FMA a clock and SM, 16 cycles of
// it for one m16n8k8).  A warp cannot issue its DMMAs back to back, so the
// pipe needs several warps per SM sub-partition: two CTAs of 8 warps keep
// four there (128 registers a thread) where 4-warp CTAs of 32x32 a warp kept
// two and lost a third of the cycles to issue waits and barriers.  1536^3:
// 32 TFLOP/s (cuBLAS 35), DMMA pipe 85 % busy in the chi0 mode at 600 rows; the basis change of 24
// matrices of 600: 1.70 -> 1.46 ms; chi0 of 260 rows, 12 800 pairs and 12
// frequencies (with the tile rules below) 3.99 -> 2.10 ms.  At 128 registers
// the gathered modes spill easily: strides, conjugations and the tile's
// columns kept out of registers there are worth 10 %.
//
// Three problem modes share the main loop:
//   ZM_GEMM  C = alpha op(A) op(B) + beta C, batched, optional split-K.
//   ZM_CHI0  per (jpm, iw) bin: C += sum_pairs conj(z) * w * z^T with the K
//            dimension gathered from a pair -> zmel-column list and the
//            weight applied while the B fragment is loaded (x0gemm.f90:72-89
//            without materialising zw / wzw); optional Hermitian tiling.
//   ZM_SEG   C(:, col) = sum_seg sum_k op(A_seg)(:, k) * s_seg(col) * Z(k, col)
//            over a gathered column list: the whole imaginary-axis sum of
//            Sigma_c (m_sxcf_gemm.f90:463-493) and the pole bins
//            (:556-590) in one launch, weights applied per column in the
//            B-fragment load.
#pragma once
#include <type_traits>
#include "common.cuh"

namespace qsgw {

constexpr int ZG_BM = 64, ZG_BN = 64, ZG_BK = 16, ZG_STAGES = 3, ZG_THREADS = 256;
constexpr int ZG_NI = 2, ZG_NJ = 2;              // m16 and n8 fragments of a warp
constexpr int ZG_PA = ZG_BM + 2, ZG_PB = ZG_BN + 2;

enum ZMode { ZM_GEMM = 0, ZM_CHI0 = 1, ZM_SEG = 2 };

struct ZSeg {
  const double2* mat;      // A operand of this segment
  const double* scale;     // per-column scale: scale[col * scale_cs]
  int scale_cs;
  int pad;
};

struct ZParams {
  int M, N, K;             // rows, cols, K (GEMM); K per segment (SEG)
  // A element (m, k) at A[m*a_rs + k*a_ks], B element (k, n) at B[n*b_rs + k*b_ks]
  const double2* A; long long a_rs, a_ks, a_bs; int a_conj;
  const double2* B; long long b_rs, b_ks, b_bs; int b_conj;
  double2* C; long long ldc, c_bs;
  double2 alpha, beta;
  int beta_zero;           // do not read C
  int acc_c;               // alpha = +-1 (real), beta = 1: the accumulators start from alpha C
  int splitk, kch_per_split;
  int ntm, ntn;            // tile counts
  // CHI0
  const int* bin_cnt; const long long* bin_coff; const long long* bin_woff;
  const int* bin_slab; const int* colidx;       // colidx null: entry k of a bin is column k 
  const double* wts; int herm;
  // SEG
  const int* tile_group; const int* tile_cols; const int* group_seg_off;
  const int* group_nseg; const ZSeg* segs;
};

struct ZSmem {
  double2 a[ZG_STAGES][ZG_BK][ZG_PA];
  double2 b[ZG_STAGES][ZG_BK][ZG_PB];
  double sk[ZG_STAGES][ZG_BK];
  double sn[ZG_STAGES][ZG_BN];
  int col[ZG_BN];
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  int sz = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, bool valid) {
  unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  int sz = valid ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// D(16x8) += A(16x8) B(8x8), FP64.  Lane (g = lane / 4, t = lane % 4) holds A(g, t), A(g+8, t),
// A(g, t+4), A(g+8, t+4); B(t, g), B(t+4, g); D(g, 2t), D(g, 2t+1), D(g+8, 2t), D(g+8, 2t+1).
__device__ __forceinline__ void dmma16(double (&d)[4], const double (&a)[4], double b0, double b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

// Decode the t-th lower-triangle tile (tm >= tn).
__device__ __forceinline__ void tri_decode(int t, int& tm, int& tn) {
  int r = static_cast<int>((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
  while ((r + 1) * (r + 2) / 2 <= t) ++r;
  while (r * (r + 1) / 2 > t) --r;
  tm = r;
  tn = t - r * (r + 1) / 2;
}

template <int MODE, bool A_RC, bool B_RC>
__global__ void __launch_bounds__(ZG_THREADS, 2) zgemm_f64_kernel(const ZParams p) {
  // known in the two gathered modes: the contiguous operand direction and the conjugations
  constexpr bool GATHER = MODE != ZM_GEMM;
  const long long a_rs = GATHER && A_RC ? 1 : p.a_rs, a_ks = GATHER && !A_RC ? 1 : p.a_ks;
  const long long b_rs = GATHER && B_RC ? 1 : p.b_rs, b_ks = GATHER && !B_RC ? 1 : p.b_ks;
  const bool a_conj = MODE == ZM_GEMM ? p.a_conj != 0 : true, b_conj = MODE == ZM_GEMM ? p.b_conj != 0 : false;
  extern __shared__ __align__(16) unsigned char zg_smem_raw[];
  ZSmem& sm = *reinterpret_cast<ZSmem*>(zg_smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = warp >> 2, wn = warp & 3;       // the row halves on every SM sub-partition (warp mod 4)

  // ---- per-CTA problem setup ----
  int tm = 0, tn = 0, batch = 0, split = 0, nchunk = 0, ch0 = 0, ch1 = 0;
  const double2* Ab = p.A;
  const double2* Bb = p.B;
  double2* Cb = p.C;
  const int* kcol = nullptr;      // CHI0: pair -> column
  const double* kw = nullptr;     // CHI0: pair weights
  int Kbin = 0;
  int group = 0, nseg = 0, seg0 = 0;
  int Mrows = p.M;
  if (MODE == ZM_GEMM) {
    tm = blockIdx.x % p.ntm; tn = blockIdx.x / p.ntm;
    batch = blockIdx.y; split = blockIdx.z;
    Ab += batch * p.a_bs; Bb += batch * p.b_bs; Cb += batch * p.c_bs;
    nchunk = (p.K + ZG_BK - 1) / ZG_BK;
  } else if (MODE == ZM_CHI0) {
    if (p.herm) tri_decode(blockIdx.x, tm, tn);
    else { tm = blockIdx.x % p.ntm; tn = blockIdx.x / p.ntm; }
    const int bin = blockIdx.y; split = blockIdx.z;
    Kbin = p.bin_cnt[bin];
    kcol = p.colidx ? p.colidx + p.bin_coff[bin] : nullptr;
    kw = p.wts + p.bin_woff[bin];
    Cb += static_cast<long long>(p.bin_slab[bin]) * p.c_bs;
    nchunk = (Kbin + ZG_BK - 1) / ZG_BK;
  } else {
    tm = blockIdx.x; tn = blockIdx.y; split = blockIdx.z;
    group = p.tile_group[tn];
    nseg = p.group_nseg[group];
    seg0 = p.group_seg_off[group];
    nchunk = nseg * ((p.K + ZG_BK - 1) / ZG_BK);
  }
  // SEG: the chunks of a tile's segments are dealt evenly (the tiles' segment counts differ)
  const int kper = MODE == ZM_SEG ? (nchunk + p.splitk - 1) / p.splitk : p.kch_per_split;
  ch0 = split * kper;
  ch1 = min(nchunk, ch0 + kper);
  const int m0 = tm * ZG_BM, n0 = tn * ZG_BN;
  const int kch_seg = (p.K + ZG_BK - 1) / ZG_BK;

  // The thread's operand elements: row and k of the first, and the steps to its others (rows run fastest
  // over the threads when they are contiguous, else k).  Columns, segment and weight addresses live in
  // registers or come by cp.async: a plain load here would hold the warp, and with it the block's next
  // barrier, for a memory round trip per chunk.
  constexpr int EA = (ZG_BK * ZG_BM) / ZG_THREADS, EB = (ZG_BK * ZG_BN) / ZG_THREADS;
  constexpr int AR = A_RC ? 0 : ZG_THREADS / ZG_BK, AK = A_RC ? ZG_THREADS / ZG_BM : 0;
  constexpr int BR = B_RC ? 0 : ZG_THREADS / ZG_BK, BK = B_RC ? ZG_THREADS / ZG_BN : 0;
  const int ar0 = A_RC ? tid % ZG_BM : tid / ZG_BK, ak0 = A_RC ? tid / ZG_BM : tid % ZG_BK;
  const int br0 = B_RC ? tid % ZG_BN : tid / ZG_BK, bk0 = B_RC ? tid / ZG_BN : tid % ZG_BK;
  const int Klim = (MODE == ZM_CHI0) ? Kbin : p.K;
  // SEG: the tile's columns (-1: none) stay in shared memory, a register apiece spilled the main loop
  if (MODE == ZM_SEG) {
    if (tid < ZG_BN) sm.col[tid] = p.tile_cols[tn * ZG_BN + tid];
    __syncthreads();
  }
  int kidx[EA];                                  // CHI0: zmel columns of the next chunk's entries (A and B alike)
  auto fetch_cols = [&](int c) {
#pragma unroll
    for (int i = 0; i < EA; ++i) {
      const int k = c * ZG_BK + ak0 + i * AK;
      kidx[i] = (kcol && k < Kbin) ? __ldg(kcol + k) : k;
    }
  };
  if (MODE == ZM_CHI0) fetch_cols(ch0);
  int lseg = MODE == ZM_SEG ? ch0 / kch_seg : 0, lin = MODE == ZM_SEG ? ch0 - lseg * kch_seg : 0;
  const double2* segA = Ab;                      // SEG: the segment load_chunk is in, the thread's column scale
  const double* segW = p.wts;
  auto next_seg = [&]() {
    const ZSeg& sg = p.segs[seg0 + lseg];
    segA = sg.mat;
    if (tid < ZG_BN) segW = sg.scale + static_cast<long long>(max(sm.col[tid], 0)) * sg.scale_cs;
  };
  if (MODE == ZM_SEG && ch0 < ch1) next_seg();
  auto load_chunk = [&](int c, int st) {         // chunks in ascending order
    const int kbase = (MODE == ZM_SEG ? lin : c) * ZG_BK;
    const double2* pa = segA + (m0 + ar0) * a_rs;
    const double2* pb = Bb + (MODE == ZM_SEG ? 0 : (n0 + br0) * b_rs);
    if (MODE != ZM_CHI0) {
      pa += (kbase + ak0) * a_ks;
      pb += (kbase + bk0) * b_ks;
    }
#pragma unroll
    for (int i = 0; i < EA; ++i) {
      const bool ok = kbase + ak0 + i * AK < Klim && m0 + ar0 + i * AR < Mrows;
      const double2* src = MODE == ZM_CHI0 ? pa + kidx[i] * a_ks : pa + i * (AR * a_rs + AK * a_ks);
      cp_async16(&sm.a[st][ak0 + i * AK][ar0 + i * AR], ok ? src : p.A, ok);
    }
#pragma unroll
    for (int i = 0; i < EB; ++i) {
      bool ok = kbase + bk0 + i * BK < Klim;
      const double2* src;
      if (MODE == ZM_SEG) {
        const int col = sm.col[br0 + i * BR];
        ok = ok && col >= 0;
        src = pb + col * b_rs;
      } else {
        ok = ok && n0 + br0 + i * BR < p.N;
        src = MODE == ZM_CHI0 ? pb + kidx[i] * b_ks : pb + i * (BR * b_rs + BK * b_ks);
      }
      cp_async16(&sm.b[st][bk0 + i * BK][br0 + i * BR], ok ? src : p.B, ok);
    }
    if (MODE == ZM_CHI0) {
      if (tid < ZG_BK) cp_async8(&sm.sk[st][tid], kbase + tid < Kbin ? kw + kbase + tid : kw, kbase + tid < Kbin);
      fetch_cols(c + 1);
    }
    if (MODE == ZM_SEG) {
      if (tid < ZG_BN) cp_async8(&sm.sn[st][tid], segW, sm.col[tid] >= 0);
      if (++lin == kch_seg) {
        lin = 0;
        ++lseg;
        if (lseg < nseg) next_seg();
      }
    }
  };

  double accr[ZG_NI][ZG_NJ][4], acci[ZG_NI][ZG_NJ][4];       // [m16 block][n8 block][fragment element]
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < ZG_NJ; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) accr[i][j][e] = acci[i][j][e] = 0.0;

  // The warp's fragments that hold output: m16 blocks i < ni and n8 blocks j < nj.  A ragged edge tile, and
  // the upper half of a Hermitian diagonal tile, issue no DMMA for fragments nobody reads.
  int ncol_tile = p.N - n0;
  if (MODE == ZM_SEG) {                         // -1 columns fill the end of a tile
    const int v = (sm.col[lane] >= 0) + (sm.col[lane + 32] >= 0);
    ncol_tile = __reduce_add_sync(0xffffffffu, v);
  }
  const int ni = min(2, max(0, (Mrows - m0 - wm * 32 + 15) / 16));
  int nj = ni > 0 ? min(ZG_NJ, max(0, (ncol_tile - wn * (8 * ZG_NJ) + 7) / 8)) : 0;
  if (MODE == ZM_CHI0 && p.herm && tm == tn && wm * 32 + 31 < wn * (8 * ZG_NJ)) nj = 0;   // mirrored from the quadrant below

  const int nloc = ch1 - ch0;
#pragma unroll
  for (int s = 0; s < ZG_STAGES - 1; ++s) {
    if (s < nloc) load_chunk(ch0 + s, s);
    cp_async_commit();
  }
  if (MODE == ZM_GEMM && p.acc_c) {
    // C is read while the first operand chunks are in flight, not after the last product: the rank-32
    // updates of the inverses are two chunks long
#pragma unroll
    for (int i = 0; i < ZG_NI; ++i)
#pragma unroll
      for (int j = 0; j < ZG_NJ; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int row = m0 + wm * 32 + i * 16 + (e >> 1) * 8 + g;
          const int col = n0 + wn * (8 * ZG_NJ) + j * 8 + 2 * t + (e & 1);
          if (row < p.M && col < p.N) {
            const double2 o = Cb[row + col * p.ldc];
            accr[i][j][e] = p.alpha.x * o.x;
            acci[i][j][e] = p.alpha.x * o.y;
          }
        }
  }
  for (int c = 0; c < nloc; ++c) {
    cp_async_wait<ZG_STAGES - 2>();
    __syncthreads();
    const int st = c % ZG_STAGES;
    const int cg = ch0 + c;                       // K elements left from this chunk on: an empty half is skipped
    const int krem = MODE == ZM_CHI0 ? Kbin - cg * ZG_BK
                                     : p.K - (MODE == ZM_SEG ? cg % kch_seg : cg) * ZG_BK;
    auto mult = [&](auto full_tile) {
      constexpr bool FULL = decltype(full_tile)::value;
#pragma unroll
      for (int k8 = 0; k8 < ZG_BK / 8; ++k8) {
        if (k8 * 8 >= krem) break;
        const int ka = k8 * 8 + t, kb = ka + 4;       // the lane's two k of the step
        double ar[2][4], ai[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int r0 = wm * 32 + i * 16 + g;
          const double2 v[4] = {sm.a[st][ka][r0], sm.a[st][ka][r0 + 8], sm.a[st][kb][r0], sm.a[st][kb][r0 + 8]};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ar[i][e] = v[e].x;
            ai[i][e] = a_conj ? -v[e].y : v[e].y;
          }
        }
        double ska = 1.0, skb = 1.0;
        if (MODE == ZM_CHI0) { ska = sm.sk[st][ka]; skb = sm.sk[st][kb]; }
#pragma unroll
        for (int j = 0; j < ZG_NJ; ++j) {
          if (!FULL && j >= nj) break;
          const int nn = wn * (8 * ZG_NJ) + j * 8 + g;
          const double2 va = sm.b[st][ka][nn], vb = sm.b[st][kb][nn];
          double sa = ska, sb = skb;
          if (MODE == ZM_SEG) sa = sb = sm.sn[st][nn];
          const double bra = va.x * sa, brb = vb.x * sb;
          const double bia = (b_conj ? -va.y : va.y) * sa, bib = (b_conj ? -vb.y : vb.y) * sb;
          // the two products of an accumulator stand apart: issued back to back the second waits for the first
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (FULL || i < ni) {
              dmma16(accr[i][j], ar[i], bra, brb);
              dmma16(acci[i][j], ar[i], bia, bib);
            }
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (FULL || i < ni) {
              dmma16(accr[i][j], ai[i], -bia, -bib);
              dmma16(acci[i][j], ai[i], bra, brb);
            }
        }
      }
    };
    if (ni == ZG_NI && nj == ZG_NJ) mult(std::true_type());
    else if (nj > 0) mult(std::false_type());
    const int cn = c + ZG_STAGES - 1;
    if (cn < nloc) load_chunk(ch0 + cn, cn % ZG_STAGES);
    cp_async_commit();
  }
  cp_async_wait<0>();
  if (nloc <= 0 && (MODE == ZM_CHI0 || p.splitk > 1)) return;

  if (MODE == ZM_CHI0) {
    // The tile leaves through shared memory (the stage buffers are free): its columns, and with herm the
    // columns of its mirror image, as whole runs of 64 rows.  Bins of a few pairs are bound by this
    // read-modify-write; straight from the fragments the mirror wrote 16-byte pieces.
    double2 (*tile)[ZG_PA] = reinterpret_cast<double2 (*)[ZG_PA]>(zg_smem_raw);     // [column][row]
    static_assert(sizeof(double2) * ZG_BN * ZG_PA <= sizeof(ZSmem), "the tile fits the stage buffers");
    __syncthreads();
    if (nj > 0) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < ZG_NJ; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int rl = wm * 32 + i * 16 + (e >> 1) * 8 + g, cl = wn * (8 * ZG_NJ) + j * 8 + 2 * t + (e & 1);
            const double2 v = make_double2(accr[i][j][e], acci[i][j][e]);
            tile[cl][rl] = v;
            if (p.herm && tm == tn && wm == 1 && wn < 2) tile[rl][cl] = make_double2(v.x, -v.y);
          }
    }
    __syncthreads();
    auto store = [&](int r0, int c0, bool mirror) {
      const int r = tid % ZG_BM, row = r0 + r;
      if (row >= (mirror ? p.N : p.M)) return;
      const int cend = min(ZG_BN, (mirror ? p.M : p.N) - c0);
      constexpr int STEP = ZG_THREADS / ZG_BM, NCOL = ZG_BN / STEP, RUN = 8;   // a thread's columns, in runs
      for (int q0 = 0; q0 < NCOL; q0 += RUN) {
        double2 v[RUN], o[RUN];
#pragma unroll
        for (int q = 0; q < RUN; ++q) {                // a run's old values are requested together
          const int cl = tid / ZG_BM + (q0 + q) * STEP;
          o[q] = make_double2(0.0, 0.0);
          if (cl < cend && p.splitk == 1) o[q] = Cb[row + static_cast<long long>(c0 + cl) * p.ldc];
        }
#pragma unroll
        for (int q = 0; q < RUN; ++q) {
          const int cl = tid / ZG_BM + (q0 + q) * STEP;
          if (cl >= cend) continue;
          v[q] = mirror ? tile[r][cl] : tile[cl][r];
          if (mirror) v[q].y = -v[q].y;
          double2* dst = Cb + row + static_cast<long long>(c0 + cl) * p.ldc;
          if (p.splitk > 1) {
            atomicAdd(&dst->x, v[q].x); atomicAdd(&dst->y, v[q].y);
          } else {
            *dst = make_double2(o[q].x + v[q].x, o[q].y + v[q].y);
          }
        }
      }
    };
    store(m0, n0, false);
    if (p.herm && tm != tn) store(n0, m0, true);     // rcxq(col, row) += conj(acc(row, col))
    return;
  }

  // ---- epilogue ----
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
    const int row = m0 + wm * 32 + i * 16 + h * 8 + g;
#pragma unroll
    for (int j = 0; j < ZG_NJ; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cl = wn * (8 * ZG_NJ) + j * 8 + 2 * t + e;
        double vr = accr[i][j][2 * h + e], vi = acci[i][j][2 * h + e];
        if (MODE == ZM_GEMM) {
          const int col = n0 + cl;
          if (row >= p.M || col >= p.N) continue;
          double2* dst = Cb + row + col * p.ldc;
          const double r2 = p.alpha.x * vr - p.alpha.y * vi;
          const double i2 = p.alpha.x * vi + p.alpha.y * vr;
          if (p.splitk > 1) {
            atomicAdd(&dst->x, r2);
            atomicAdd(&dst->y, i2);
          } else if (p.beta_zero || p.acc_c) {
            *dst = make_double2(r2, i2);
          } else {
            const double2 o = *dst;
            *dst = make_double2(r2 + p.beta.x * o.x - p.beta.y * o.y,
                                i2 + p.beta.x * o.y + p.beta.y * o.x);
          }
        } else {
          const int col = sm.col[cl];
          if (row >= p.M || col < 0) continue;
          double2* dst = Cb + row + static_cast<long long>(col) * p.ldc;
          if (p.splitk > 1) { atomicAdd(&dst->x, vr); atomicAdd(&dst->y, vi); }
          else *dst = make_double2(vr, vi);
        }
      }
  }
}

// Host launch helpers (defined in zgemm_f64.cu).  op: 0 'N', 1 'T', 2 'C', 3 conjugated without transposing.
int zgemm_f64(int opa, int opb, int m, int n, int k, double2 alpha,
              const double2* A, long long lda, long long a_bs,
              const double2* B, long long ldb, long long b_bs, double2 beta,
              double2* C, long long ldc, long long c_bs, int nbatch, cudaStream_t s);
int zgemm_chi0_launch(ZParams p, int nbins, int herm, int splitk, cudaStream_t s);
// C(0:n, 0:n) += A^H B for complex A, B of K x n (column-major), n <= 64, any K (FP64 atomics)
int zgemm_hn_thin(int n, long long K, const double2* A, long long lda, const double2* B, long long ldb, double2* C,
                  long long ldc, cudaStream_t s);
// C (ldc x p.N, contiguous columns) is overwritten; mean_nseg: the tiles' mean segment count
int zgemm_seg_launch(ZParams p, int ncol_tiles, int mean_nseg, cudaStream_t s);
// K splits of a launch of `ctas` equal tiles of nch K chunks (one split when nch is short)
int zgemm_splitk(long long ctas, int nch);
// Batched inverses (wv.cu: Hermitian positive definite; zminv_piv.cu: general, partial pivoting).
int zminv_hpd_batched(double2* A, int n, long long lda, long long a_bs, int nbatch, cudaStream_t s);
// result (may be null): receives the inverses' scratch copy (ld n, stride n*n), A is then left undefined;
// without it the inverses are copied back into A.
int zminv_general_batched(double2* A, int n, long long lda, long long a_bs, int nbatch, cudaStream_t s,
                          const double2** result = nullptr);

}  // namespace qsgw

// chi0 rank-k accumulation.
//   qsgw_x0gemm / qsgw_x0gemm_d : drop-in for x0gemm (x0gemm.f90:2-97).
//   qsgw_chi0_lorentz_d          : every k and every iw in one launch, with
//                                  the Lorentzian pair weights built on the
//                                  GPU in FP64.
// The host builds the (jpm, iw) bin lists in the reference's icoun order
// (x0gemm.f90:37-64); the GPU never materialises zw / wzw: the pair gather
// and the weight are folded into the operand loads of the DMMA engine.
#include <algorithm>
#include <memory>
#include <cmath>
#include <vector>
#include "zgemm_f64.cuh"
#include "autotune.cuh"
#include "split_f16.cuh"
#include "ozaki_i8.cuh"
#include "hoststage.cuh"

namespace qsgw {

static DevBuf g_x0_idx, g_x0_w, g_x0_bins, g_x0_zm, g_x0_rc;

struct BinTables {
  std::vector<int> cnt, slab;
  std::vector<long long> off;
  int maxcnt = 0;
  void add(int c, long long o, int sl) {
    cnt.push_back(c);
    off.push_back(o);
    slab.push_back(sl);
    maxcnt = std::max(maxcnt, c);
  }
};

// Returns the number of chunks of the longest bin; the pair columns and weights are on the device already.
static int upload_bins(const BinTables& bt, ZParams& p, cudaStream_t s, int& rc) {
  const size_t nb = bt.cnt.size();
  const size_t bin_bytes = nb * (2 * sizeof(int) + sizeof(long long));
  rc = g_x0_bins.ensure(std::max<size_t>(bin_bytes, 64));
  if (rc) return 0;
  std::vector<unsigned char> hb(bin_bytes);
  memcpy(hb.data(), bt.off.data(), nb * sizeof(long long));
  memcpy(hb.data() + nb * sizeof(long long), bt.cnt.data(), nb * sizeof(int));
  memcpy(hb.data() + nb * (sizeof(long long) + sizeof(int)), bt.slab.data(), nb * sizeof(int));
  if ((rc = h2d(g_x0_bins.p, hb.data(), bin_bytes, s))) return 0;
  unsigned char* base = g_x0_bins.as<unsigned char>();
  p.bin_coff = reinterpret_cast<const long long*>(base);
  p.bin_woff = reinterpret_cast<const long long*>(base);
  p.bin_cnt = reinterpret_cast<const int*>(base + nb * sizeof(long long));
  p.bin_slab = reinterpret_cast<const int*>(base + nb * (sizeof(long long) + sizeof(int)));
  p.colidx = g_x0_idx.as<int>();
  p.wts = g_x0_w.as<double>();
  return (bt.maxcnt + ZG_BK - 1) / ZG_BK;
}

// In the int8 mode a bin of at most kFp64BinPairs pairs stays on the FP64 engine: it is the more accurate and, there,
// the faster one, as the int8 path's slicing passes and its CTAs' start and end cost more than the products.  Per call
// of 80 equal bins (FP64 / 3 slices, us): 300 rows, bins of 32 pairs 129 / 256, of 128 299 / 325, of 192 405 / 373; 600
// rows 318 / 664, 723 / 769, 1002 / 847; 1000 rows, of 128 1749 / 1693, of 192 2456 / 1810.
// The longer bins go to the int8 path together if they outweigh its fixed cost (scales, ranges, slicing launches:
// about 35 us), counted in pairs beyond kFp64BinPairs times 64 x 64 output tiles -- 160 rows, 24 bins of 256 pairs
// (18 000) 109 / 122, 80 of 256 (61 000) 307 / 308; 600 rows, 4 of 192 (14 000) 96 / 102, 24 of 192 (84 000) 334 / 300 --
// or if one of them is so long that the FP64 engine's chain over its chunks (0.17 us a pair) would.  95 bins of 10 and
// one of 8000 pairs at 300 and 600 rows: 255 and 508 us (all on FP64 2509 and 2704, all on int8 481 and 992).
constexpr int kFp64BinPairs = 128, kFp64LongestBin = 512;
constexpr long long kFp64PairTiles = 32768;

static int x0gemm_device(double2* rcxq, int npr, int ipr_col, int npr_col, int nwhis, int npm,
                         int ns1, int ns2, const double2* zmel, int nbb, int nm1, int nm2,
                         int nqtot, int icounkmink, int icounkmaxk, const int* itc, const int* itpc,
                         const int* jpmc, const int* iwini, const int* iwend, const int* icouini,
                         const double* whwc, int ncount) {
  cudaStream_t s = ctx().stream;
  const int nmz = nm2 - nm1 + 1;
  // ---- bin lists in icoun order (x0gemm.f90:37-64) ----
  const int nbins_all = nwhis * npm;
  std::vector<int> cnt(nbins_all, 0);
  for (int icoun = icounkmink; icoun <= icounkmaxk; ++icoun) {
    const int c = icoun - 1;
    const int jpm = jpmc[c], it = itc[c], itp = itpc[c];
    QSGW_ARG(jpm >= 1 && jpm <= npm, "x0gemm: jpmc(%d)=%d outside 1..npm", icoun, jpm);
    if (it < ns1 || it > ns2) continue;
    QSGW_ARG(it >= nm1 && it <= nm2, "x0gemm: itc(%d)=%d outside zmel bounds %d:%d", icoun, it, nm1, nm2);
    QSGW_ARG(itp >= 1 && itp <= nqtot, "x0gemm: itpc(%d)=%d outside 1..nqtot", icoun, itp);
    QSGW_ARG(iwini[c] >= 1 && iwend[c] <= nwhis, "x0gemm: bins %d..%d outside 1..nwhis", iwini[c], iwend[c]);
    QSGW_ARG(icouini[c] >= 1 && icouini[c] + (iwend[c] - iwini[c]) <= ncount,
             "x0gemm: icouini(%d)=%d outside whwc", icoun, icouini[c]);
    for (int iw = iwini[c]; iw <= iwend[c]; ++iw) cnt[(jpm - 1) * nwhis + (iw - 1)]++;
  }
  BinTables bt;
  std::vector<long long> start(nbins_all, 0);
  long long tot = 0;
  for (int jpm = 1; jpm <= npm; ++jpm)
    for (int iw = 1; iw <= nwhis; ++iw) {
      const int b = (jpm - 1) * nwhis + (iw - 1);
      start[b] = tot;
      if (cnt[b] > 0) bt.add(cnt[b], tot, iw * (3 - 2 * jpm) - (1 - npm) * nwhis);
      tot += cnt[b];
    }
  if (bt.cnt.empty()) return QSGW_OK;
  std::vector<int> colidx(tot);
  std::vector<double> wts(tot);
  std::vector<long long> fill(start);
  for (int icoun = icounkmink; icoun <= icounkmaxk; ++icoun) {
    const int c = icoun - 1;
    const int jpm = jpmc[c], it = itc[c], itp = itpc[c];
    if (it < ns1 || it > ns2) continue;
    const int col = (it - nm1) + nmz * (itp - 1);
    for (int iw = iwini[c]; iw <= iwend[c]; ++iw) {
      const int b = (jpm - 1) * nwhis + (iw - 1);
      colidx[fill[b]] = col;
      wts[fill[b]] = whwc[iw - iwini[c] + icouini[c] - 1];   // x0gemm.f90:62
      fill[b]++;
    }
  }
  int rc = g_x0_idx.ensure(tot * sizeof(int));
  if (rc) return rc;
  if ((rc = g_x0_w.ensure(tot * sizeof(double)))) return rc;
  if ((rc = h2d(g_x0_idx.p, colidx.data(), tot * sizeof(int), s))) return rc;
  if ((rc = h2d(g_x0_w.p, wts.data(), tot * sizeof(double), s))) return rc;
  const int herm = (ipr_col == 1 && npr_col == npr) ? 1 : 0;
  const int ntm = (npr + ZG_BM - 1) / ZG_BM, ntn = (npr_col + ZG_BN - 1) / ZG_BN;
  const long long ntiles = herm ? ntm * (ntm + 1LL) / 2 : static_cast<long long>(ntm) * ntn;
  if (ctx().prec_mode == QSGW_PREC_SPLIT_I8) {
    BinTables longer, rest;
    long long beyond = 0;
    int classes = 0;
    for (size_t i = 0; i < bt.cnt.size(); ++i) {
      if (bt.cnt[i] <= kFp64BinPairs) {
        rest.add(bt.cnt[i], bt.off[i], bt.slab[i]);
        continue;
      }
      longer.add(bt.cnt[i], bt.off[i], bt.slab[i]);
      beyond += bt.cnt[i] - kFp64BinPairs;
      for (long long e = bt.off[i]; e < bt.off[i] + bt.cnt[i]; ++e) classes |= (wts[e] < 0.0 ? 1 : 0) | (wts[e] > 0.0 ? 2 : 0);
    }
    if (beyond * ntiles >= kFp64PairTiles || longer.maxcnt > kFp64LongestBin) {
      // the pair columns and weights of a bin form one K range; rcxq accumulates (no tuning trials)
      OzChi0Bins ob;
      ob.ebeg = longer.off;
      ob.cnt = longer.cnt;
      ob.slab = longer.slab;
      const int ns = ctx().nslices > 0 ? ctx().nslices : 4;   // rcxq accumulates: no trials, the accurate count
      rc = chi0_split_i8(rcxq, npr, static_cast<long long>(npr) * npr_col, npr, npr_col, ipr_col - 1, herm != 0, zmel,
                         nbb, static_cast<long long>(nmz) * nqtot, g_x0_idx.as<int>(), g_x0_w.as<double>(), ob, classes,
                         ns, s, nullptr);
      if (rc || rest.cnt.empty()) return rc;
      bt = rest;
    }
  }
  ZParams p{};
  p.M = npr; p.N = npr_col;
  p.A = zmel; p.a_rs = 1; p.a_ks = nbb; p.a_conj = 1;               // zw^H   (:76, :88 opA=C)
  p.B = zmel + (ipr_col - 1); p.b_rs = 1; p.b_ks = nbb; p.b_conj = 0;  // wzw   (:84)
  p.C = rcxq; p.ldc = npr; p.c_bs = static_cast<long long>(npr) * npr_col;
  p.ntm = ntm; p.ntn = ntn;
  const int maxch = upload_bins(bt, p, s, rc);
  if (rc) return rc;
  const int nbins = static_cast<int>(bt.cnt.size());
  const int sk = zgemm_splitk(ntiles * nbins, maxch);
  p.kch_per_split = (maxch + sk - 1) / sk;
  rc = zgemm_chi0_launch(p, nbins, herm, sk, s);
  if (rc) return rc;
  return QSGW_OK;
}

static int x0gemm_check(int npr, int ipr_col, int npr_col, int nwhis, int npm, int nbb, int nm1,
                        int nm2, int nqtot, int icounkmink, int icounkmaxk, int ncount,
                        const void* rcxq, const void* zmel) {
  QSGW_ARG(npr >= 1 && npr_col >= 1 && ipr_col >= 1, "x0gemm: bad npr=%d npr_col=%d ipr_col=%d", npr, npr_col, ipr_col);
  QSGW_ARG(npr <= nbb && ipr_col - 1 + npr_col <= nbb, "x0gemm: product-basis range exceeds nbb=%d", nbb);
  QSGW_ARG(npm == 1 || npm == 2, "x0gemm: npm=%d", npm);
  QSGW_ARG(nwhis >= 1, "x0gemm: nwhis=%d", nwhis);
  QSGW_ARG(nm2 >= nm1 && nqtot >= 1, "x0gemm: zmel bounds %d:%d nqtot=%d", nm1, nm2, nqtot);
  QSGW_ARG(icounkmink >= 1 && icounkmaxk >= icounkmink - 1, "x0gemm: icoun range %d..%d", icounkmink, icounkmaxk);
  QSGW_ARG(ncount >= 0, "x0gemm: ncount=%d", ncount);
  QSGW_ARG(rcxq && zmel, "x0gemm: null array");
  QSGW_ARG((reinterpret_cast<uintptr_t>(rcxq) & 15) == 0 && (reinterpret_cast<uintptr_t>(zmel) & 15) == 0,
           "x0gemm: complex arrays must be 16-byte aligned");
  return QSGW_OK;
}

}  // namespace qsgw

using namespace qsgw;

extern "C" int qsgw_x0gemm_d(double* rcxq_d, int npr, int ipr_col, int npr_col, int nwhis, int npm,
                             int ns1, int ns2, const double* zmel_d, int nbb, int nm1, int nm2,
                             int nqtot, int icounkmink, int icounkmaxk, const int* itc,
                             const int* itpc, const int* jpmc, const int* iwini, const int* iwend,
                             const int* icouini, const double* whwc, int ncount) {
  int rc = require_init();
  if (rc) return rc;
  rc = x0gemm_check(npr, ipr_col, npr_col, nwhis, npm, nbb, nm1, nm2, nqtot, icounkmink, icounkmaxk,
                    ncount, rcxq_d, zmel_d);
  if (rc) return rc;
  if (icounkmaxk < icounkmink) return QSGW_OK;
  QSGW_ARG(itc && itpc && jpmc && iwini && iwend && icouini && whwc, "x0gemm: null index table");
  return x0gemm_device(reinterpret_cast<double2*>(rcxq_d), npr, ipr_col, npr_col, nwhis, npm, ns1,
                       ns2, reinterpret_cast<const double2*>(zmel_d), nbb, nm1, nm2, nqtot,
                       icounkmink, icounkmaxk, itc, itpc, jpmc, iwini, iwend, icouini, whwc, ncount);
}

extern "C" int qsgw_x0gemm(double* rcxq, int npr, int ipr_col, int npr_col, int nwhis, int npm,
                           int ns1, int ns2, const double* zmel, int nbb, int nm1, int nm2,
                           int nqtot, int icounkmink, int icounkmaxk, const int* itc,
                           const int* itpc, const int* jpmc, const int* iwini, const int* iwend,
                           const int* icouini, const double* whwc, int ncount) {
  int rc = require_init();
  if (rc) return rc;
  rc = x0gemm_check(npr, ipr_col, npr_col, nwhis, npm, nbb, nm1, nm2, nqtot, icounkmink, icounkmaxk,
                    ncount, rcxq, zmel);
  if (rc) return rc;
  if (icounkmaxk < icounkmink) return QSGW_OK;
  cudaStream_t s = ctx().stream;
  const size_t nslab = static_cast<size_t>(npm == 1 ? nwhis + 1 : 2 * nwhis + 1);
  const size_t rc_bytes = static_cast<size_t>(npr) * npr_col * nslab * 16;
  const size_t zm_bytes = static_cast<size_t>(nbb) * (nm2 - nm1 + 1) * nqtot * 16;
  rc = g_x0_rc.ensure(rc_bytes); if (rc) return rc;
  rc = g_x0_zm.ensure(zm_bytes); if (rc) return rc;
  QSGW_CUDA(cudaMemcpyAsync(g_x0_rc.p, rcxq, rc_bytes, cudaMemcpyHostToDevice, s));
  QSGW_CUDA(cudaMemcpyAsync(g_x0_zm.p, zmel, zm_bytes, cudaMemcpyHostToDevice, s));
  rc = qsgw_x0gemm_d(g_x0_rc.as<double>(), npr, ipr_col, npr_col, nwhis, npm, ns1, ns2,
                     g_x0_zm.as<double>(), nbb, nm1, nm2, nqtot, icounkmink, icounkmaxk, itc, itpc,
                     jpmc, iwini, iwend, icouini, whwc, ncount);
  if (rc) return rc;
  QSGW_CUDA(cudaMemcpyAsync(rcxq, g_x0_rc.p, rc_bytes, cudaMemcpyDeviceToHost, s));
  QSGW_CUDA(cudaStreamSynchronize(s));
  return QSGW_OK;
}

// ---------------------------------------------------------------------------
// All-k chi0 with Lorentzian weights built on the device.
namespace qsgw {

// A k-point's pairs: columns [col0, next col0) = (it - 1) + nocc (itp - 1), as zmel(:, it, itp); o0 and u0 are
// its first occupied and unoccupied energy.
struct KPairs {
  long long col0;
  int nocc, o0, u0, pad;
};
// the excitation energy of pair column pr
__device__ __forceinline__ double pair_energy(long long pr, const KPairs* __restrict__ kp, int nk,
                                              const double* __restrict__ eo, const double* __restrict__ eu) {
  int lo = 0, hi = nk - 1;                         // the last k with col0 <= pr (k-points without pairs share one)
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (kp[mid].col0 <= pr) lo = mid;
    else hi = mid - 1;
  }
  const KPairs k = kp[lo];
  const int c = static_cast<int>(pr - k.col0);
  return eu[k.u0 + c / k.nocc] - eo[k.o0 + c % k.nocc];
}

// One thread a pair, all frequencies: the pair's energies are found from the k table (pair index maps from the
// host were 8 bytes a pair of pageable copies, formed in a host loop).
__global__ void lorentz_weight_kernel(double* __restrict__ w, const KPairs* __restrict__ kp, int nk,
                                      const double* __restrict__ eo, const double* __restrict__ eu,
                                      const double* __restrict__ fi, long long npair, int niw, double inv_nk) {
  for (long long pr = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; pr < npair;
       pr += static_cast<long long>(gridDim.x) * blockDim.x) {
    const double de = pair_energy(pr, kp, nk, eo, eu);
    for (int iw = blockIdx.y; iw < niw; iw += gridDim.y) {
      const double om = fi[iw];
      w[iw * npair + pr] = -2.0 * de / (de * de + om * om) * inv_nk;   // chi0(iw) <= 0 (dpsion5.f90:218)
    }
  }
}

// Real frequency axis: f(w) = [1/(w - de + i eta) - 1/(w + de + i eta)] / nk, whose value at
// w = i nu is the imaginary-axis weight above.  Slot iw holds Re f, slot nw + iw holds Im f.
__global__ void lorentz_real_weight_kernel(double* __restrict__ w, const KPairs* __restrict__ kp, int nk,
                                           const double* __restrict__ eo, const double* __restrict__ eu,
                                           const double* __restrict__ fr, long long npair, int nw, double eta,
                                           double inv_nk) {
  for (long long pr = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; pr < npair;
       pr += static_cast<long long>(gridDim.x) * blockDim.x) {
    const double de = pair_energy(pr, kp, nk, eo, eu);
    for (int iw = blockIdx.y; iw < nw; iw += gridDim.y) {
      const double om = fr[iw];
      const double a = om - de, b = om + de, e2 = eta * eta;
      const double da = 1.0 / (a * a + e2), db = 1.0 / (b * b + e2);
      w[iw * npair + pr] = (a * da - b * db) * inv_nk;
      w[static_cast<long long>(nw + iw) * npair + pr] = (-eta * da + eta * db) * inv_nk;
    }
  }
}

static DevBuf g_lz_map, g_lz_e, g_lz_w, g_lz_bins;

// eta < 0: imaginary axis, nw slots of weights; eta >= 0: real axis, 2 nw slots (Re, Im).
// classes (out): bit 0 when a weight can be negative, bit 1 when one can be positive
int chi0_lorentz_weights(int niw, const double* freq_i, int nk, const int* nocc, const int* nun,
                         const double* eocc, const double* eunocc, long long& npair, double*& w_d,
                         cudaStream_t s, double eta = -1.0, int nk_norm = 0, int* classes = nullptr) {
  const double inv_nk = 1.0 / (nk_norm > 0 ? nk_norm : nk);   // 1/nk of the whole k mesh
  npair = 0;
  long long no_tot = 0, nu_tot = 0;
  for (int k = 0; k < nk; ++k) {
    QSGW_ARG(nocc[k] >= 0 && nun[k] >= 0, "chi0: negative band count at k=%d", k);
    npair += static_cast<long long>(nocc[k]) * nun[k];
    no_tot += nocc[k];
    nu_tot += nun[k];
  }
  std::vector<KPairs> kp(nk);
  long long c = 0, oo = 0, uo = 0;
  int cl = 0;
  for (int k = 0; k < nk; ++k) {
    kp[k] = KPairs{c, std::max(nocc[k], 1), static_cast<int>(oo), static_cast<int>(uo), 0};
    // imaginary axis: w = -2 de / (de^2 + w^2) / nk has the sign of -de, de between the extremes of this k
    if (classes && nocc[k] > 0 && nun[k] > 0) {
      double olo = INFINITY, ohi = -INFINITY, ulo = INFINITY, uhi = -INFINITY;
      for (int i = 0; i < nocc[k]; ++i) {              // fmin and fmax pass a NaN energy by, as its pairs have no sign
        olo = std::fmin(olo, eocc[oo + i]);
        ohi = std::fmax(ohi, eocc[oo + i]);
      }
      for (int i = 0; i < nun[k]; ++i) {
        ulo = std::fmin(ulo, eunocc[uo + i]);
        uhi = std::fmax(uhi, eunocc[uo + i]);
      }
      cl |= (uhi > olo ? 1 : 0) | (ulo < ohi ? 2 : 0);
    }
    c += static_cast<long long>(nocc[k]) * nun[k];
    oo += nocc[k];
    uo += nun[k];
  }
  if (classes) *classes = eta >= 0.0 ? 3 : cl;       // the real axis has both signs
  int rc = g_lz_map.ensure(nk * sizeof(KPairs));
  if (rc) return rc;
  rc = g_lz_e.ensure((no_tot + nu_tot + niw) * sizeof(double));
  if (rc) return rc;
  rc = g_lz_w.ensure(std::max<long long>(npair, 1) * niw * (eta >= 0.0 ? 2 : 1) * sizeof(double));
  if (rc) return rc;
  double* deo = g_lz_e.as<double>();
  double *deu = deo + no_tot, *dfi = deu + nu_tot;
  std::vector<double> tab(eocc, eocc + no_tot);
  tab.insert(tab.end(), eunocc, eunocc + nu_tot);
  tab.insert(tab.end(), freq_i, freq_i + niw);
  if ((rc = h2d(g_lz_map.p, kp.data(), nk * sizeof(KPairs), s))) return rc;
  if ((rc = h2d(deo, tab.data(), tab.size() * sizeof(double), s))) return rc;
  if (npair > 0) {
    const KPairs* dkp = g_lz_map.as<KPairs>();
    const unsigned gx = static_cast<unsigned>(std::min<long long>((npair + 255) / 256, 8LL * ctx().sm_count));
    // few pairs: the frequencies are spread over the grid as well
    const unsigned gy = static_cast<unsigned>(std::max<long long>(1, std::min<long long>(niw, 4LL * ctx().sm_count / gx)));
    if (eta < 0.0)
      lorentz_weight_kernel<<<dim3(gx, gy), 256, 0, s>>>(g_lz_w.as<double>(), dkp, nk, deo, deu, dfi, npair, niw, inv_nk);
    else
      lorentz_real_weight_kernel<<<dim3(gx, gy), 256, 0, s>>>(g_lz_w.as<double>(), dkp, nk, deo, deu, dfi, npair, niw,
                                                              eta, inv_nk);
    count_launch();
    QSGW_LAUNCH_CHECK("lorentz weight kernel");
  }
  w_d = g_lz_w.as<double>();
  return QSGW_OK;
}

// chi = Hre + i Him for the real axis (Hre, Him: the Re-weight and Im-weight slots)
__global__ void combine_re_im_kernel(double2* __restrict__ chi, const double2* __restrict__ hre,
                                     const double2* __restrict__ him, long long n) {
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < n;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const double2 a = hre[e], b = him[e];
    chi[e] = make_double2(a.x - b.y, a.y + b.x);
  }
}

static DevBuf g_lzr_h;
static DevBuf g_lz_ref, g_lz_try;       // chi0 of the slice-count trials

}  // namespace qsgw

static int chi0_run(double* chi0_d, int npr, int niw, const double* zcols_d, int ldz, long long npair,
                    const double* w_d, cudaStream_t s, bool accumulate = false, int classes = 3);

extern "C" int qsgw_chi0_lorentz_d(double* chi0_d, int npr, int niw, const double* freq_i, int nk,
                                   const int* nocc, const int* nun, const double* eocc,
                                   const double* eunocc, const double* zcols_d, int ldz) {
  int rc = require_init();
  if (rc) return rc;
  QSGW_ARG(chi0_d && zcols_d && freq_i && nocc && nun && eocc && eunocc, "chi0_lorentz: null pointer");
  QSGW_ARG(npr >= 1 && niw >= 1 && nk >= 1 && ldz >= npr, "chi0_lorentz: npr=%d niw=%d nk=%d ldz=%d", npr, niw, nk, ldz);
  QSGW_ARG((reinterpret_cast<uintptr_t>(chi0_d) & 15) == 0 && (reinterpret_cast<uintptr_t>(zcols_d) & 15) == 0,
           "chi0_lorentz: complex arrays must be 16-byte aligned");
  cudaStream_t s = ctx().stream;
  long long npair = 0;
  double* w_d = nullptr;
  int classes = 3;
  rc = chi0_lorentz_weights(niw, freq_i, nk, nocc, nun, eocc, eunocc, npair, w_d, s, -1.0, 0, &classes);
  if (rc) return rc;
  QSGW_ARG(npair < (1LL << 31), "chi0_lorentz: %lld pairs exceed the 32-bit column index", npair);
  return chi0_run(chi0_d, npr, niw, zcols_d, ldz, npair, w_d, s, false, classes);
}

// chi0 slots iw = conj(Z) diag(w[iw]) Z^T for precomputed weights w (nslot x npair), in the
// precision mode of the context; chi0_d is overwritten.
static int chi0_run(double* chi0_d, int npr, int niw, const double* zcols_d, int ldz, long long npair,
                    const double* w_d, cudaStream_t s, bool accumulate, int classes) {
  int rc = QSGW_OK;
  const size_t cbytes = static_cast<size_t>(npr) * npr * niw * 16;
  if (!accumulate) QSGW_CUDA(cudaMemsetAsync(chi0_d, 0, cbytes, s));
  if (npair == 0) return QSGW_OK;
  std::unique_ptr<TuneSuspend> hold(accumulate ? new TuneSuspend() : nullptr);   // trials would clear chi0
  if (ctx().prec_mode == QSGW_PREC_SPLIT_I8) {
    // one bin per frequency slot, every pair in every bin in column order (weights w[iw * npair + p])
    OzChi0Bins ob;
    for (int iw = 0; iw < niw; ++iw) {
      ob.ebeg.push_back(static_cast<long long>(iw) * npair);
      ob.cnt.push_back(static_cast<int>(npair));
      ob.slab.push_back(iw);
    }
    auto run_ns = [&](int ns, double2* out, const char* tune) {
      return chi0_split_i8(out, npr, static_cast<long long>(npr) * npr, npr, npr, 0, true,
                           reinterpret_cast<const double2*>(zcols_d), ldz, npair, nullptr, w_d, ob, classes, ns, s,
                           tune);
    };
    int ns = ctx().nslices;
    if (ns == 0) {
      // automatic slice count: the smallest whose chi0 stays within the relative target of the
      // 4-slice one (trials on scratch copies; accumulating calls take the choice already made)
      const long long nel = static_cast<long long>(npr) * npr * niw;
      bool have_ref = false;
      auto err = [&](int n, double* e) -> int {
        int r = g_lz_ref.ensure(nel * sizeof(double2));
        if (r) return r;
        r = g_lz_try.ensure(nel * sizeof(double2));
        if (r) return r;
        if (!have_ref) {
          QSGW_CUDA(cudaMemsetAsync(g_lz_ref.p, 0, nel * sizeof(double2), s));
          if ((r = run_ns(4, g_lz_ref.as<double2>(), nullptr))) return r;
          have_ref = true;
        }
        QSGW_CUDA(cudaMemsetAsync(g_lz_try.p, 0, nel * sizeof(double2), s));
        if ((r = run_ns(n, g_lz_try.as<double2>(), nullptr))) return r;
        return rel_diff_fro(g_lz_try.as<double2>(), g_lz_ref.as<double2>(), nel, s, e);
      };
      char key[160];
      std::snprintf(key, sizeof(key), "chi0_i8 slices npr=%d npair~2^%.3f niw=%d", npr,
                    std::round(8.0 * std::log2(static_cast<double>(npair))) / 8.0, niw);
      rc = tuned_slices(key, {2, 3}, 4, ctx().chi0_rel_tol, err, 3, &ns);
      if (rc) return rc;
    }
    return run_ns(ns, reinterpret_cast<double2*>(chi0_d), accumulate ? nullptr : "chi0_lorentz");
  }
  if (ctx().prec_mode == QSGW_PREC_SPLIT_F16) {
    return chi0_split_f16(reinterpret_cast<double2*>(chi0_d), npr, niw,
                          reinterpret_cast<const double2*>(zcols_d), ldz, npair, w_d, s);
  }
  // one bin per iw, all pairs in every bin, bin iw's weights at offset iw*npair
  std::vector<long long> off(2 * niw);
  std::vector<int> cs(2 * niw);
  for (int iw = 0; iw < niw; ++iw) {
    off[iw] = 0;                                  // no column list
    off[niw + iw] = static_cast<long long>(iw) * npair;   // weight offsets
    cs[iw] = static_cast<int>(npair);
    cs[niw + iw] = iw;                            // slab
  }
  rc = g_lz_bins.ensure(2 * niw * (sizeof(long long) + sizeof(int)));
  if (rc) return rc;
  unsigned char* base = g_lz_bins.as<unsigned char>();
  if ((rc = h2d(base, off.data(), 2 * niw * sizeof(long long), s))) return rc;
  if ((rc = h2d(base + 2 * niw * sizeof(long long), cs.data(), 2 * niw * sizeof(int), s))) return rc;
  ZParams p{};
  p.M = npr; p.N = npr;
  p.A = reinterpret_cast<const double2*>(zcols_d); p.a_rs = 1; p.a_ks = ldz; p.a_conj = 1;
  p.B = reinterpret_cast<const double2*>(zcols_d); p.b_rs = 1; p.b_ks = ldz; p.b_conj = 0;
  p.C = reinterpret_cast<double2*>(chi0_d); p.ldc = npr; p.c_bs = static_cast<long long>(npr) * npr;
  p.ntm = p.ntn = (npr + ZG_BM - 1) / ZG_BM;
  p.bin_coff = reinterpret_cast<const long long*>(base);
  p.bin_woff = reinterpret_cast<const long long*>(base) + niw;
  p.bin_cnt = reinterpret_cast<const int*>(base + 2 * niw * sizeof(long long));
  p.bin_slab = p.bin_cnt + niw;
  p.colidx = nullptr;                              // every bin holds every column in order
  p.wts = w_d;
  const int maxch = static_cast<int>((npair + ZG_BK - 1) / ZG_BK);
  const int ntiles = p.ntm * (p.ntm + 1) / 2;
  const int heur = zgemm_splitk(static_cast<long long>(ntiles) * niw, maxch);
  // split K: the autotuner times the heuristic and its neighbours (x1/2, x2, x4) on this shape
  auto run = [&](int sk, bool clear) -> int {      // trials clear chi0 (it was cleared above)
    ZParams q = p;
    q.kch_per_split = (maxch + sk - 1) / sk;
    if (clear) QSGW_CUDA(cudaMemsetAsync(chi0_d, 0, cbytes, s));
    return zgemm_chi0_launch(q, niw, 1, sk, s);
  };
  std::vector<int> cands;
  for (int c : {heur / 2, heur, heur * 2, heur * 4})
    if (c >= 1 && c <= maxch && (cands.empty() || cands.back() != c)) cands.push_back(c);
  char key[160];
  // pair counts within ~9% share a choice (they differ from q to q)
  std::snprintf(key, sizeof(key), "chi0_dmma npr=%d npair~2^%.3f niw=%d", npr,
                std::round(8.0 * std::log2(static_cast<double>(npair))) / 8.0, niw);
  int sk = heur;
  bool tried = false;
  rc = tuned_choice(key, cands, heur, [&](int c) { return run(c, true); }, s, &sk, &tried);
  if (rc) return rc;
  return run(sk, tried);
}

extern "C" int qsgw_chi0_lorentz_acc_d(double* chi0_d, int npr, int niw, const double* freq_i, int nk_total,
                                       int nkb, const int* nocc, const int* nun, const double* eocc,
                                       const double* eunocc, const double* zcols_d, int ldz) {
  int rc = require_init();
  if (rc) return rc;
  QSGW_ARG(chi0_d && zcols_d && freq_i && nocc && nun && eocc && eunocc, "chi0_lorentz_acc: null pointer");
  QSGW_ARG(npr >= 1 && niw >= 1 && nkb >= 1 && nk_total >= nkb && ldz >= npr,
           "chi0_lorentz_acc: npr=%d niw=%d nkb=%d nk_total=%d ldz=%d", npr, niw, nkb, nk_total, ldz);
  QSGW_ARG((reinterpret_cast<uintptr_t>(chi0_d) & 15) == 0 && (reinterpret_cast<uintptr_t>(zcols_d) & 15) == 0,
           "chi0_lorentz_acc: complex arrays must be 16-byte aligned");
  cudaStream_t s = ctx().stream;
  long long npair = 0;
  double* w_d = nullptr;
  int classes = 3;
  rc = chi0_lorentz_weights(niw, freq_i, nkb, nocc, nun, eocc, eunocc, npair, w_d, s, -1.0, nk_total, &classes);
  if (rc) return rc;
  QSGW_ARG(npair < (1LL << 31), "chi0_lorentz_acc: %lld pairs exceed the 32-bit column index", npair);
  return chi0_run(chi0_d, npr, niw, zcols_d, ldz, npair, w_d, s, true, classes);
}

extern "C" int qsgw_chi0_lorentz_real_d(double* chi0_d, int npr, int nw, const double* freq_r, double eta, int nk,
                                        const int* nocc, const int* nun, const double* eocc,
                                        const double* eunocc, const double* zcols_d, int ldz) {
  int rc = require_init();
  if (rc) return rc;
  QSGW_ARG(chi0_d && zcols_d && freq_r && nocc && nun && eocc && eunocc, "chi0_lorentz_real: null pointer");
  QSGW_ARG(npr >= 1 && nw >= 1 && nk >= 1 && ldz >= npr && eta >= 0.0,
           "chi0_lorentz_real: npr=%d nw=%d nk=%d ldz=%d eta=%g", npr, nw, nk, ldz, eta);
  QSGW_ARG((reinterpret_cast<uintptr_t>(chi0_d) & 15) == 0 && (reinterpret_cast<uintptr_t>(zcols_d) & 15) == 0,
           "chi0_lorentz_real: complex arrays must be 16-byte aligned");
  cudaStream_t s = ctx().stream;
  long long npair = 0;
  double* w_d = nullptr;
  rc = chi0_lorentz_weights(nw, freq_r, nk, nocc, nun, eocc, eunocc, npair, w_d, s, eta);
  if (rc) return rc;
  QSGW_ARG(npair < (1LL << 31), "chi0_lorentz_real: %lld pairs exceed the 32-bit column index", npair);
  const long long nn = static_cast<long long>(npr) * npr * nw;
  rc = g_lzr_h.ensure(static_cast<size_t>(2 * nn) * sizeof(double2));
  if (rc) return rc;
  double2* h = g_lzr_h.as<double2>();
  // both Hermitian parts in one run over 2 nw weight slots
  rc = chi0_run(reinterpret_cast<double*>(h), npr, 2 * nw, zcols_d, ldz, npair, w_d, s);
  if (rc) return rc;
  combine_re_im_kernel<<<static_cast<int>(std::min<long long>((nn + 255) / 256, 16LL * ctx().sm_count)), 256, 0,
                         s>>>(reinterpret_cast<double2*>(chi0_d), h, h + nn, nn);
  count_launch();
  QSGW_LAUNCH_CHECK("combine_re_im_kernel");
  return QSGW_OK;
}

static qsgw::DevBuf g_lzh_c;
static qsgw::HostRing g_lzh_ring(2);    // zcols of the host-pointer calls

extern "C" int qsgw_chi0_lorentz(double* chi0, int npr, int niw, const double* freq_i, int nk,
                                 const int* nocc, const int* nun, const double* eocc,
                                 const double* eunocc, const double* zcols, int ldz) {
  using namespace qsgw;
  int rc = require_init();
  if (rc) return rc;
  QSGW_ARG(chi0 && zcols && nocc && nun, "chi0_lorentz: null pointer");
  QSGW_ARG(npr >= 1 && niw >= 1 && nk >= 1 && ldz >= npr, "chi0_lorentz: npr=%d niw=%d nk=%d ldz=%d", npr, niw, nk, ldz);
  long long ncol = 0;
  for (int k = 0; k < nk; ++k) ncol += static_cast<long long>(nocc[k]) * nun[k];
  cudaStream_t s = ctx().stream;
  const size_t zb = static_cast<size_t>(ldz) * ncol * 16;
  const size_t cb = static_cast<size_t>(npr) * npr * niw * 16;
  HostSlot* sl = nullptr;
  cudaStream_t cs = nullptr;
  rc = g_lzh_ring.begin(&sl, &cs); if (rc) return rc;
  DevBuf& dz = sl->buf[0];
  rc = dz.ensure(zb); if (rc) return rc;
  rc = g_lzh_c.ensure(cb); if (rc) return rc;   // one output image, reused in stream order
  QSGW_CUDA(cudaMemcpyAsync(dz.p, zcols, zb, cudaMemcpyHostToDevice, cs));
  rc = g_lzh_ring.ready(*sl, cs);
  if (rc) return rc;
  rc = qsgw_chi0_lorentz_d(g_lzh_c.as<double>(), npr, niw, freq_i, nk, nocc, nun, eocc, eunocc,
                           dz.as<double>(), ldz);
  if (rc) return rc;
  QSGW_CUDA(cudaMemcpyAsync(chi0, g_lzh_c.p, cb, cudaMemcpyDeviceToHost, s));
  return g_lzh_ring.finish(*sl);
}

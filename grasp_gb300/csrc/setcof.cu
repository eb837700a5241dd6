// setcof.cu - SETCOF (rmcdhf90/setcof.f90) on the device: the coefficient
// lists of the direct (YPOT), exchange (XPOT) and one-body (DACON)
// potentials of an orbital, from the blocks' T/V lists and the mixing
// coefficients.
//
// The reference reads mcp.30/31/32+k from disk once per orbital and SCF
// iteration and, for each label that involves the orbital, adds its
// contributions' DSUBRS(IR, IC) COEFF (dsubrs.f90: the generalized weight of
// the CSF pair). Those label sums do not depend on the orbital except
// through the final 1/UCF(J), so here one pass computes them for every label
// of every block, together with the diagonal FCO/GCO sums of every pair of
// orbitals. DSUBRS depends on the position only, so it is formed once per EMT
// position (k_dsubrs_pos) and a contribution costs one FMA. The labels are
// decoded and their sums listed by orbital at the same time, so that a call
// for orbital J reads its own labels only; it forms the lists in the
// reference's order (FCO, GCO, the T list by block, the V^k lists by k and
// block), so they are the reference's entry for entry. (Forming every
// orbital's lists beforehand cost a caller who wants one of them the merging of
// all: 17.9 ms for five blocks over 23 subshells, now 2.7 and 0.44 a call.)
#include <algorithm>
#include <cstring>
#include <memory>
#include <unordered_map>
#include <utility>
#include <vector>

#include "gg_internal.cuh"

namespace gg {

// One list of one orbital: its labels and values. The labels of a later block
// (merge) that repeat one join its first entry.
struct SetcofList {
  std::vector<int32_t> lab;
  std::vector<double> val;
  std::unordered_map<int32_t, int> first;  // first entry of each label, filled when merging
  size_t merged = 0;                       // labels entered into `first` so far
  void put(int32_t l, double v, bool merge) {
    if (merge) {
      for (; merged < lab.size(); ++merged) first.emplace(lab[merged], (int)merged);
      const auto f = first.find(l);
      if (f != first.end()) {
        val[f->second] = val[f->second] + v;
        return;
      }
    }
    lab.push_back(l);
    val.push_back(v);
  }
};

// A label: half its sum, and its orbitals, a byte each (KEYORB = 215): a, b, c,
// d of R^k(ab;cd); a T label stays as it is
struct SetcofLabel {
  double v;
  uint32_t ix;
  uint8_t k;
  uint8_t places;  // bit f: the f-th orbital stands in no earlier place
  bool merge;      // not of the first block
};

// the sums of the last gg_setcof_prepare
struct SetcofState {
  int nw = 0;
  std::vector<int> nak, nkj;        // of the orbital set, 1-based
  std::vector<double> diag;         // k_diag_pairs' sums
  std::vector<SetcofLabel> labels;  // in SETCOF's order: the T lists by block, the V^k lists by k and block
  size_t nt = 0;                    // of them T labels
  // [ref0[j], ref0[j + 1]): the labels that name orbital j, in order, as 4 l +
  // the place that names it first (T: 0 or 1)
  std::vector<uint32_t> refs;
  std::vector<size_t> ref0;
};

namespace {

// the levels' coefficients by CSF: evr[r][k] = evec[k][r]
__global__ void k_by_csf(const double *__restrict__ evec, int ncf, int nev, double *__restrict__ evr) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)ncf * nev;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(e / nev), k = (int)(e % nev);
    evr[e] = evec[(size_t)k * ncf + r];
  }
}

// DSUBRS (rmcdhf90/dsubrs.f90:20-33) of every EMT position, doubled off the
// diagonal (setcof.f90:242-251): EOL, sum over the block's levels of EVEC(IR)
// EVEC(IC) WT(level); otherwise WT(IR) on the diagonal, 0 elsewhere. ev holds
// the levels' coefficients by CSF ([ncf][nev]). One warp per row IC, whose
// EVEC(IC) WT it holds in shared memory, 32 levels at a time; the diagonal's
// value also goes to diag. Bound: the FP64 pipe, one FMA per position and
// level. (Formed per contribution, three operations per level and about 2.4
// contributions per position, the label sums took 9.2 ms for 20,011 CSFs and
// 10 levels; now 97 us, and 118 us for the sums.)
// The positions [c0, c1) go to d (PART), or all of them.
constexpr int LS_WARPS = 4;
template <bool PART>
__global__ void __launch_bounds__(LS_WARPS * 32) k_dsubrs_pos(const int64_t *__restrict__ iendc,
                                                              const int32_t *__restrict__ irow, int64_t c0,
                                                              int64_t c1, int ncf, int eol, int nev,
                                                              const double *__restrict__ ev,
                                                              const double *__restrict__ wt, double *__restrict__ d,
                                                              double *__restrict__ diag) {
  __shared__ double sb[LS_WARPS][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x * LS_WARPS + w;
  if (r >= ncf) return;
  int64_t p0 = iendc[r], p1 = iendc[r + 1];
  if (PART) {
    p0 = max(p0, c0);
    p1 = min(p1, c1);
    if (p0 >= p1) return;
    d -= c0;
  }
  for (int k0 = 0; k0 < (eol ? nev : 1); k0 += 32) {
    const int nk = min(32, nev - k0);
    if (eol) {
      __syncwarp();
      if (lane < nk) sb[w][lane] = ev[(size_t)r * nev + k0 + lane] * wt[k0 + lane];
      __syncwarp();
    }
    for (int64_t p = p0 + lane; p < p1; p += 32) {
      const int c = irow[p] - 1;
      double v = 0.0;
      if (eol) {
        const double *a = ev + (size_t)c * nev + k0;
#pragma unroll 4
        for (int k = 0; k < nk; ++k) v = fma(__ldg(a + k), sb[w][k], v);
      } else if (c == r) {
        v = wt[r];
      }
      if (k0 > 0) v += c == r ? diag[r] : 0.5 * d[p];
      if (c == r) diag[r] = v;
      d[p] = c == r ? v : v + v;
    }
  }
}

// each label's sum of DSUBRS COEFF (setcof.f90:242-251 for the T list,
// :302-311 for the V lists), one block per label: its threads take every
// 256th contribution, eight gathers in flight, and a fixed tree adds them. Lists
// are uneven (a few labels hold tens of thousands of contributions), so the
// longest label sets the time: 193 us with 128 threads and four gathers. PART:
// only the contributions of the positions [c0, c1), added to out unless c0 = 0.
constexpr int LAB_THREADS = 256;
template <bool PART>
__global__ void __launch_bounds__(LAB_THREADS) k_label_sums(const int64_t *__restrict__ start,
                                                            const int32_t *__restrict__ loc,
                                                            const double *__restrict__ coeff,
                                                            const double *__restrict__ d, int64_t c0, int64_t c1,
                                                            double *__restrict__ out) {
  __shared__ double ws[LAB_THREADS / 32];
  const int64_t l = blockIdx.x, i0 = start[l], i1 = start[l + 1];
  double sum = 0.0;
#pragma unroll 8
  for (int64_t i = i0 + threadIdx.x; i < i1; i += LAB_THREADS) {
    if (!PART) {
      sum = fma(__ldg(d + loc[i] - 1), coeff[i], sum);
    } else {
      const int64_t p = loc[i] - 1 - c0;
      if (p >= 0 && p < c1 - c0) sum = fma(__ldg(d + p), coeff[i], sum);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = ws[0];
    for (int w = 1; w < LAB_THREADS / 32; ++w) v += ws[w];
    out[l] = PART && c0 ? out[l] + v : v;
  }
}

// one block's CSFs for the diagonal sums
struct DiagBlock {
  int ncf;
  const double *d;        // DSUBRS(IR, IR)
  const uint8_t *iq;      // [nconf][nw]
  const int32_t *conf;    // [ncf]
};

// The diagonal sums over blocks and CSFs of DSUBRS(IR, IR) times the
// occupation factors FCO (fco.f90) and GCO (gco.f90) are made of. They depend
// on K through a factor CLRX^2 only, so one block per pair a <= b of orbitals
// forms them all: a < b, sum d qa qb over all CSFs and over those where a or b
// is full; a = b, sum d qa (qa - 1) / 2 and sum d qa^2 over those where a is
// full. (One warp per (J, IB, K), adding 32 terms at a time on one lane, took
// 5.0 ms for 34 subshells and 20,011 CSFs; now 139 us.)
constexpr int DIAG_THREADS = 256;
__global__ void __launch_bounds__(DIAG_THREADS) k_diag_pairs(const int *__restrict__ full,
                                                             const DiagBlock *__restrict__ blocks, int nblocks,
                                                             int nw, double *__restrict__ out) {
  __shared__ double ws[2][DIAG_THREADS / 32];
  const int a = blockIdx.y, b = blockIdx.x;
  if (a > b) return;
  const int fa = full[a], fb = full[b];
  double s0 = 0.0, s1 = 0.0;
  for (int t = 0; t < nblocks; ++t) {
    const DiagBlock B = blocks[t];
#pragma unroll 4
    for (int r = threadIdx.x; r < B.ncf; r += DIAG_THREADS) {
      const uint8_t *q = B.iq + (size_t)B.conf[r] * nw;
      const int qa = q[a], qb = q[b];
      const double d = B.d[r];
      s0 = fma(d, (double)(a == b ? qa * (qa - 1) / 2 : qa * qb), s0);
      if (qa == fa || qb == fb) s1 = fma(d, (double)(qa * qb), s1);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  if ((threadIdx.x & 31) == 0) {
    ws[0][threadIdx.x >> 5] = s0;
    ws[1][threadIdx.x >> 5] = s1;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double v = ws[threadIdx.x][0];
    for (int i = 1; i < DIAG_THREADS / 32; ++i) v += ws[threadIdx.x][i];
    out[2 * ((size_t)a * nw + b) + threadIdx.x] = v;
  }
}

// positions of a block whose DSUBRS are held at a time; the fewest it is tried with
constexpr int64_t SETCOF_POS = 1 << 27, SETCOF_POS_MIN = 1 << 16;

template <class T> int upv(DBuf<T> &b, const std::vector<T> &h, cudaStream_t s) {
  GG_TRY(b.alloc(std::max<size_t>(1, h.size())));
  if (!h.empty()) GG_CUDA(cudaMemcpyAsync(b.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s));
  return GG_OK;
}

}  // namespace
}  // namespace gg

using namespace gg;

extern "C" {

int gg_setcof_prepare(gg_ctx *ctx, int nblocks, gg_hmat *const *h, const int *nev, const double *const *evec,
                      const double *const *wt, int eol) {
  if (!ctx || nblocks < 1 || !h || !wt || (eol && (!nev || !evec)))
    return fail(GG_ERR_ARG, "gg_setcof_prepare: bad arguments");
  GG_TRY(ensure_orbitals(ctx));
  GG_CUDA(cudaSetDevice(ctx->device));
  const Orbitals &o = ctx->orb;
  const int nw = o.nw;
  cudaStream_t s = ctx->stream;
  const int64_t test_pos = std::exchange(ctx->test_setcof_pos, 0);
  auto st = std::make_shared<SetcofState>();
  st->nw = nw;
  std::vector<std::vector<int32_t>> labs;  // per block: the labels of all its lists
  std::vector<std::vector<double>> sums;   // per block: each label's sum of DSUBRS COEFF (x2 off the diagonal)
  std::vector<DBuf<double>> devec(nblocks), dwt(nblocks), ddiag(nblocks);
  std::vector<DiagBlock> hb(nblocks);
  for (int b = 0; b < nblocks; ++b) {
    gg_hmat *m = h[b];
    if (!m || m->ctx->device != ctx->device) return fail(GG_ERR_ARG, "gg_setcof_prepare: bad block");
    Lists &L = *m->lists;
    if (!L.valid) return fail(GG_ERR_STATE, "gg_setcof_prepare: a block has no lists (gg_setham_upload)");
    if (m->host_prec >= 0) return fail(GG_ERR_ARG, "gg_setcof_prepare: a host-resident block has no lists");
    const int ncf = m->ncf, ne = eol ? nev[b] : 0;
    if (eol && (ne < 1 || !evec[b] || !wt[b])) return fail(GG_ERR_ARG, "gg_setcof_prepare: missing levels");
    if (!eol && !wt[b]) return fail(GG_ERR_ARG, "gg_setcof_prepare: missing CSF weights");
    if (eol) {
      DBuf<double> tmp;
      GG_TRY(tmp.alloc((size_t)ncf * ne));
      GG_TRY(devec[b].alloc((size_t)ncf * ne));
      GG_CUDA(cudaMemcpyAsync(tmp.p, evec[b], (size_t)ncf * ne * sizeof(double), cudaMemcpyHostToDevice, s));
      k_by_csf<<<std::max(1, std::min(4 * ctx->sms, (int)(((int64_t)ncf * ne + 255) / 256))), 256, 0, s>>>(
          tmp.p, ncf, ne, devec[b].p);
      ::gg::note_launch();
      GG_CUDA(cudaStreamSynchronize(s));  // tmp is freed here
      GG_TRY(dwt[b].alloc(ne));
      GG_CUDA(cudaMemcpyAsync(dwt[b].p, wt[b], ne * sizeof(double), cudaMemcpyHostToDevice, s));
    } else {
      GG_TRY(dwt[b].alloc(ncf));
      GG_CUDA(cudaMemcpyAsync(dwt[b].p, wt[b], ncf * sizeof(double), cudaMemcpyHostToDevice, s));
    }
    // DSUBRS by position, then every label's sum, SETCOF_POS positions (1 GB)
    // at a time, fewer where the device has no room for them: beside the lists
    // of a block that fills it, 8 bytes for every position need not fit. A
    // piece costs one more reading of LOC.
    DBuf<double> dpos, dsum;
    int64_t len = std::max<int64_t>(1, std::min<int64_t>(m->nnz, test_pos > 0 ? test_pos : SETCOF_POS));
    while (const int st_pos = dpos.alloc(len)) {
      if (st_pos != GG_ERR_NOMEM || len <= SETCOF_POS_MIN) return st_pos;
      len = (len + 1) / 2;
    }
    GG_TRY(ddiag[b].alloc(ncf));
    const bool part = len < m->nnz;
    for (int64_t c0 = 0; c0 < m->nnz; c0 += len) {
      const int64_t c1 = std::min(m->nnz, c0 + len);
      (part ? k_dsubrs_pos<true> : k_dsubrs_pos<false>)<<<(ncf + LS_WARPS - 1) / LS_WARPS, LS_WARPS * 32, 0, s>>>(
          m->dIendc.p, m->dIrow.p, c0, c1, ncf, eol ? 1 : 0, ne, devec[b].p, dwt[b].p, dpos.p, ddiag[b].p);
      ::gg::note_launch();
      GG_TRY(dsum.alloc(std::max<int64_t>(1, L.nlab)));
      if (L.nlab > 0) {
        (part ? k_label_sums<true> : k_label_sums<false>)<<<(unsigned)L.nlab, LAB_THREADS, 0, s>>>(
            L.dStart.p, L.dLoc.p, L.dCoeff.p, dpos.p, c0, c1, dsum.p);
        ::gg::note_launch();
      }
    }
    GG_CUDA(cudaGetLastError());
    labs.emplace_back(L.nlab);
    sums.emplace_back(L.nlab);
    if (L.nlab > 0) {
      GG_CUDA(cudaMemcpyAsync(labs.back().data(), L.dLab.p, L.nlab * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
      GG_CUDA(cudaMemcpyAsync(sums.back().data(), dsum.p, L.nlab * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    GG_CUDA(cudaStreamSynchronize(s));  // dpos and dsum are freed here
    hb[b] = DiagBlock{ncf, ddiag[b].p, L.dIq.p, L.dConf.p};
  }
  // the diagonal sums, by orbital pair
  std::vector<int> full(nw);
  for (int a = 0; a < nw; ++a) full[a] = o.nkj[a + 1] + 1;
  DBuf<int> dfull;
  DBuf<DiagBlock> dblocks;
  DBuf<double> dout;
  GG_TRY(upv(dfull, full, s));
  GG_TRY(upv(dblocks, hb, s));
  GG_TRY(dout.alloc((size_t)2 * nw * nw));
  k_diag_pairs<<<dim3(nw, nw), DIAG_THREADS, 0, s>>>(dfull.p, dblocks.p, nblocks, nw, dout.p);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  st->diag.resize((size_t)2 * nw * nw);
  GG_CUDA(cudaMemcpyAsync(st->diag.data(), dout.p, st->diag.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));
  st->nak = o.nak;
  st->nkj = o.nkj;
  // the labels in order, and how many name each orbital
  int64_t total = 0;
  int kmaxf = -1;
  for (int b = 0; b < nblocks; ++b) {
    total += h[b]->lists->nlab;
    kmaxf = std::max(kmaxf, h[b]->lists->kmaxf);
  }
  if (total > UINT32_MAX / 4) return fail(GG_ERR_RANGE, "gg_setcof_prepare: more than 2^30 - 1 labels");
  const int KEY = KEYORB;
  std::vector<SetcofLabel> &labels = st->labels;
  labels.reserve(total);
  std::vector<size_t> &ref0 = st->ref0;
  ref0.assign(258, 0);  // by byte; those that are no orbital of the set are not read
  auto named = [&](int a) { return a >= 1 && a <= nw; };
  // T labels (setcof.f90:188-285): DA of orbital a at b, of b at a
  for (int b = 0; b < nblocks; ++b) {
    const Lists &L = *h[b]->lists;
    for (int64_t l = L.list_lab0[0]; l < L.list_lab0[1]; ++l) {
      const int32_t lab = labs[b][l];
      const int x = lab % KEY, y = lab / KEY;
      const int places = (named(x) ? 1 : 0) | (y != x && named(y) ? 2 : 0);
      labels.push_back(SetcofLabel{0.5 * sums[b][l], (uint32_t)lab, 0, (uint8_t)places, b > 0});
      if (places & 1) ++ref0[x + 1];
      if (places & 2) ++ref0[y + 1];
    }
  }
  st->nt = labels.size();
  // V^k labels (:287-515)
  for (int k = 0; k <= kmaxf; ++k)
    for (int b = 0; b < nblocks; ++b) {
      const Lists &L = *h[b]->lists;
      if (k > L.kmaxf) continue;
      for (int64_t l = L.list_lab0[k + 1]; l < L.list_lab0[k + 2]; ++l) {
        if (labs[b][l] < 0) continue;
        uint32_t lab = (uint32_t)labs[b][l];  // unsigned: the divisions by KEY are multiplications
        uint32_t ix[4];
        ix[3] = lab % KEYORB;
        lab /= KEYORB;
        ix[1] = lab % KEYORB;
        lab /= KEYORB;
        ix[2] = lab % KEYORB;
        ix[0] = lab / KEYORB;  // at most 216: 2^31 / KEYORB^3
        const int places = 1 | (ix[1] != ix[0]) << 1 | (ix[2] != ix[0] && ix[2] != ix[1]) << 2 |
                           (ix[3] != ix[0] && ix[3] != ix[1] && ix[3] != ix[2]) << 3;
        labels.push_back(SetcofLabel{0.5 * sums[b][l], ix[0] | ix[1] << 8 | ix[2] << 16 | ix[3] << 24, (uint8_t)k,
                                     (uint8_t)places, b > 0});
        for (int f = 0; f < 4; ++f) ref0[ix[f] + 1] += places >> f & 1;
      }
    }
  for (int a = 1; a <= 257; ++a) ref0[a] += ref0[a - 1];
  std::vector<uint32_t> &refs = st->refs;
  refs.resize(ref0[257]);
  std::vector<size_t> at(ref0);
  for (size_t l = 0; l < labels.size(); ++l) {
    const SetcofLabel &L = labels[l];
    if (l < st->nt) {
      const int32_t lab = (int32_t)L.ix;
      if (L.places & 1) refs[at[lab % KEY]++] = (uint32_t)(4 * l);
      if (L.places & 2) refs[at[lab / KEY]++] = (uint32_t)(4 * l + 1);
      continue;
    }
    for (int f = 0; f < 4; ++f)
      if (L.places >> f & 1) refs[at[L.ix >> 8 * f & 255]++] = (uint32_t)(4 * l + f);
  }
  ctx->setcof = st;
  return GG_OK;
}

int gg_setcof(gg_ctx *ctx, int j, double ucfj, int cap, int *ny, int32_t *nya, double *ya, int *nx, int32_t *nxa,
              double *xa, int *nd, int32_t *nda, double *da) {
  if (!ctx || !ny || !nx || !nd || cap < 0 || (cap > 0 && (!nya || !ya || !nxa || !xa || !nda || !da)))
    return fail(GG_ERR_ARG, "gg_setcof: bad arguments");
  const auto st = std::static_pointer_cast<SetcofState>(ctx->setcof);
  if (!st) return fail(GG_ERR_STATE, "gg_setcof: call gg_setcof_prepare first");
  if (j < 1 || j > st->nw || ctx->orb.nw != st->nw) return fail(GG_ERR_ARG, "gg_setcof: orbital outside the orbital set");
  const int nw = st->nw, KEY = KEYORB;
  const std::vector<int> &nak = st->nak, &nkj = st->nkj;
  SetcofList ly, lx, ld;
  const uint32_t *ref = st->refs.data() + st->ref0[j], *end = st->refs.data() + st->ref0[j + 1];
  for (SetcofList *l : {&ly, &lx}) {
    l->lab.reserve(end - ref + 16 * nw);
    l->val.reserve(end - ref + 16 * nw);
  }
  for (int ib = 1; ib <= nw; ++ib) {
    const double *v = &st->diag[2 * ((size_t)(std::min(j, ib) - 1) * nw + (std::max(j, ib) - 1))];
    // Y from FCO (setcof.f90:73-105): NYA = K + IB KEY (KEY + 1)
    const int64_t l0 = (int64_t)ib * KEY * (KEY + 1);
    if (ib == j) {
      ly.put((int32_t)l0, 2.0 * v[0] / ucfj, false);
      for (int k = 2; k <= nkj[j] - 1; k += 2) {
        const double c = clrx_host(nak[j], k, nak[j]);
        ly.put((int32_t)(k + l0), -(c * c * v[1]) / ucfj, false);
      }
      continue;
    }
    ly.put((int32_t)l0, v[0] / ucfj, false);
    // X from GCO (:107-147): NXA = K + KEY J + IB KEY^2 (KEY + 1)
    const int64_t x0 = (int64_t)KEY * j + (int64_t)ib * KEY * KEY * (KEY + 1);
    const int kmin = (nak[j] * nak[ib] > 0) ? std::abs((nkj[j] - nkj[ib]) / 2) : std::abs((nkj[j] - nkj[ib]) / 2) + 1;
    for (int k = kmin; k <= (nkj[j] + nkj[ib]) / 2; k += 2) {
      const double c = clrx_host(nak[j], k, nak[ib]);
      lx.put((int32_t)(k + x0), -(c * c * v[1]) / ucfj, false);
    }
  }
  for (; ref != end; ++ref) {
    const size_t l = *ref >> 2;
    const int f = *ref & 3;
    const SetcofLabel &L = st->labels[l];
    const bool merge = L.merge;
    const double v = L.v;
    if (l < st->nt) {
      ld.put(f ? (int32_t)L.ix % KEY : (int32_t)L.ix / KEY, v / ucfj, merge);
      continue;
    }
    // the orbitals after J's first place, wrapped round: those that are J again
    // stand in later places
    const uint32_t r = f == 3 ? L.ix : L.ix >> 8 * (f + 1) | L.ix << 8 * (3 - f);
    const int o1 = r & 255, o2 = r >> 8 & 255, o3 = r >> 16 & 255, k = L.k;
    const int again = (o1 == j) + (o2 == j) + (o3 == j);
    if (again == 0) {
      lx.put(((o2 * KEY + o3) * KEY + o1) * KEY + k, v / ucfj, merge);
    } else if (again == 1) {
      if (o2 == j)
        ly.put((o3 * KEY + o1) * KEY + k, (v + v) / ucfj, merge);
      else
        lx.put(((o2 * KEY + o3) * KEY + o1) * KEY + k, (v + v) / ucfj, merge);
    } else if (again == 2) {
      const int other = o1 != j ? o1 : o2 != j ? o2 : o3;
      ly.put((other * KEY + j) * KEY + k, (v + v) / ucfj, merge);
      lx.put(((other * KEY + j) * KEY + j) * KEY + k, v / ucfj, merge);
    } else {
      ly.put((j * KEY + j) * KEY + k, 4.0 * v / ucfj, merge);
    }
  }
  *ny = (int)ly.lab.size();
  *nx = (int)lx.lab.size();
  *nd = (int)ld.lab.size();
  if (*ny > cap || *nx > cap || *nd > cap)
    return fail(GG_ERR_RANGE, "gg_setcof: a list is longer than cap (the counts are set)");
  auto give = [](const SetcofList &l, int32_t *lab, double *val) {
    std::copy(l.lab.begin(), l.lab.end(), lab);
    std::copy(l.val.begin(), l.val.end(), val);
  };
  give(ly, nya, ya);
  give(lx, nxa, xa);
  give(ld, nda, da);
  return GG_OK;
}

}  // extern "C"

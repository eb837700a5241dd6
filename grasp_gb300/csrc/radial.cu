// radial.cu - R^k table (GENINTRK/SLATER/YZK/QUAD) and one-body I(ab)
// (RINTI/DPBDT) on the GPU.
//
// Compiled with -fmad=false: every multiply and add below is rounded on its
// own, as in the reference's FP64 loops, so that the Y^k functions and the
// per-integral quadratures reproduce the reference's arithmetic step by
// step. The R^k contraction uses explicit fma() and QUAD's head term takes
// the grid's factors per point from a table, so neither is bit-exact.
//
// Layout in HBM (all FP64):
//   Y buffer   [nY][np]  Y^k_bd(r_i) at [f*np + i] (1-based i), zero beyond
//                        the integration limit MTP(b,d) of SLATER.
//   A buffer   [nP][KC]  w(i) * (P_a P_c + Q_a Q_c)(r_i) * RPOR(r_i) for
//                        every pair a <= c, zero outside 2 <= i <= min(MF).
//   VALTEIRK   [N_Rk]    written by the contraction epilogue in GENINTRK order.
#include <cuda_fp16.h>

#include <algorithm>
#include <map>
#include <tuple>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "gg_internal.cuh"

namespace gg {

namespace {

constexpr int KC_TILE = 16;  // the pair arrays' row length is a multiple of this

struct YDesc {
  int k, b, d;  // Y^k_{bd}
  int mtp;      // min(MF(b), MF(d)) (YZK's MTP)
  int mtpb;     // last point kept in the Y buffer (N when k == 0 and b == d)
  int cs;       // first function index with the same (k, b)
  int nd;       // number of functions with the same (k, b) = |D(b,k)|
};

struct RkTile {
  int r0, rn;  // first row ((a, c) pair of the k) and how many
  int f0, fn;  // first Y function and how many
};

struct QuadItem {  // one integral evaluated with the general QUAD
  int a, c, p, f, mtp;  // p: the pair's row of the pair arrays
  long long pos;
};

__device__ __forceinline__ double pf(const double *P, int ld, int i, int j) {
  return P[(size_t)(j - 1) * ld + (i - 1)];
}

// QUAD (lib9290/quad.f90:52-103) on a 1-based array TA with room for
// TA(MTP+3). Sequential, in the reference's order.
__device__ double quad_seq(double *TA, int mtp, const double *R, const double *RP, const QuadConst &q) {
  const int mtpm1 = mtp - 1;
  for (int i = 2; i <= mtpm1; ++i) {
    const double tai = TA[i];
    if (fabs(tai) <= 0.0) continue;
    const int ip1 = i + 1;
    const double taip1 = TA[ip1];
    const double quott = taip1 / tai;
    if (quott <= 0.0) continue;
    const double frip1 = taip1 / RP[ip1];
    double fri = tai / RP[i];
    const double ratio = frip1 / fri;
    const double rip1 = R[ip1], ri = R[i];
    const double sigma = log(ratio) / log(rip1 / ri);
    fri = ri * fri;
    double result = fri / (sigma + 1.0);
    TA[mtp + 1] = 0.0;
    TA[mtp + 2] = 0.0;
    TA[mtp + 3] = 0.0;
    result = result + q.C1 * tai;
    double s = 0.0;
    for (int j = ip1; j <= mtp; j += 4) s = s + (q.C2 * (TA[j] + TA[j + 2]) + q.C3 * TA[j + 1] + q.C4 * TA[j + 3]);
    result = result + s;
    if ((mtp - i) % 4 == 0) result = result - q.C1 * TA[mtp];
    return result;
  }
  return 0.0;
}

// dynamic shared memory of a launch without opting in: 48 KB less the 1 KB that
// a static array takes before it (the dynamic arrays of this file start on
// k_rk_tc's 1,024-byte alignment)
constexpr size_t SMEM_PLAIN = 47 * 1024;
__host__ __device__ constexpr int quad_panels(int np) { return np / 4 + 4; }

// QUAD's test of a head index (quad.f90:58-63), TA(i) != 0 and not TA(i+1)/TA(i)
// <= 0, without the division: ordinary numbers whose ratio does not underflow
// pass when their signs are equal. A ratio that is not a number passes, as in
// quad_seq.
__device__ __forceinline__ bool quad_head(double tai, double taip1) {
  const int h0 = __double2hiint(tai), h1 = __double2hiint(taip1);
  const int e0 = h0 >> 20 & 0x7ff, e1 = h1 >> 20 & 0x7ff;
  if (e0 > 0 && e0 < 0x7ff && e1 > 0 && e1 < 0x7ff && e1 - e0 > -1000) return (h0 ^ h1) >= 0;
  return !(fabs(tai) <= 0.0) && !(taip1 / tai <= 0.0);
}

// quad_seq by the lanes of a warp, the same value to the bit: the head index
// by ballot, the four-point panels (quad.f90:94-99) one per lane into `panel`
// (quad_panels(np) doubles), then lane 0 adds them in order, the only serial
// part. TA is zero beyond MTP; the result is lane 0's. (Sequential QUADs on
// one lane of each warp were most of RINTI: four of 148 panels of seven
// operations each, 168 us per I(ab) table whatever its size; this form 22 us
// for 16 subshells, 36 us for 43.)
__device__ double quad_warp(const double *TA, double *panel, int mtp, const double *R, const double *RP,
                            const QuadConst &q, int lane) {
  int h = 0;
  for (int i0 = 2; i0 <= mtp - 1 && h == 0; i0 += 32) {
    const int i = i0 + lane;
    bool hit = false;
    if (i <= mtp - 1) {
      const double tai = TA[i];
      if (!(fabs(tai) <= 0.0)) hit = !(TA[i + 1] / tai <= 0.0);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    if (bal) h = i0 + __ffs(bal) - 1;
  }
  if (h == 0) return 0.0;
  const int np = (mtp - h + 3) / 4;
  for (int t = lane; t < np; t += 32) {
    const int j = h + 1 + 4 * t;
    panel[t] = q.C2 * (TA[j] + TA[j + 2]) + q.C3 * TA[j + 1] + q.C4 * TA[j + 3];
  }
  __syncwarp();
  double result = 0.0;
  if (lane == 0) {
    const double tai = TA[h], frip1 = TA[h + 1] / RP[h + 1];
    double fri = tai / RP[h];
    const double ratio = frip1 / fri;
    const double sigma = log(ratio) / log(R[h + 1] / R[h]);
    fri = R[h] * fri;
    result = fri / (sigma + 1.0);
    result = result + q.C1 * tai;
    double s = 0.0;
#pragma unroll 8
    for (int t = 0; t < np; ++t) s = s + panel[t];
    result = result + s;
    if ((mtp - h) % 4 == 0) result = result - q.C1 * TA[mtp];
  }
  __syncwarp();
  return result;
}

// ---------------------------------------------------------------------------
// YZK part 1 (yzk.f90:105-126, 190-201): RHOP and the two TEMP arrays.
//   TZ(i) = r^k RHOP(i), TW(i) = RHOP(i) / r^(k+1) on 2 <= i <= MTP, else 0.
// ---------------------------------------------------------------------------
// In all kernels over functions, nfp (may be null) points to a number of
// functions on the device that replaces nf, the bound the launch was sized by.
__device__ __forceinline__ int nfuncs(int nf, const int *nfp) { return nfp ? min(nf, *nfp) : nf; }
__global__ void k_ytemp(const YDesc *__restrict__ yd, int nf, const int *__restrict__ nfp,
                        const double *__restrict__ PF, const double *__restrict__ QF, int ld,
                        const double *__restrict__ RP, const double *__restrict__ pw, int np,
                        double *__restrict__ TZ, double *__restrict__ TW) {
  nf = nfuncs(nf, nfp);
  for (int f = blockIdx.y; f < nf; f += gridDim.y) {
    const YDesc y = yd[f];
    const double *RTTK = pw + (size_t)(0 * (KLIMIT + 1) + y.k) * np;
    const double *RTTKM1 = pw + (size_t)(3 * (KLIMIT + 1) + y.k) * np;
    const double *RM = pw;  // row k = 0 of table 0
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
      double tz = 0.0, tw = 0.0;
      if (i >= 2 && i <= y.mtp) {
        const double rhop =
            RP[i] * (pf(PF, ld, i, y.b) * pf(PF, ld, i, y.d) + pf(QF, ld, i, y.b) * pf(QF, ld, i, y.d));
        if (y.k == 0) {
          tz = rhop;
          tw = rhop * RM[i];
        } else {
          tz = RTTK[i] * rhop;
          tw = rhop * RTTKM1[i];
        }
      }
      TZ[(size_t)f * np + i] = tz;
      TW[(size_t)f * np + i] = tw;
    }
  }
}

// ---------------------------------------------------------------------------
// YZK part 2 (yzk.f90:128-224): the four interleaved stride-4 Newton-Cotes
// recurrences for Z (forward) and W (backward). One thread per (function,
// residue class mod 4); the four threads of a function are adjacent lanes.
// ---------------------------------------------------------------------------
__global__ void k_ychain(const YDesc *__restrict__ yd, int nf, const int *__restrict__ nfp,
                         const double *__restrict__ TZ,
                         const double *__restrict__ TW, const double *__restrict__ R,
                         const double *__restrict__ pw, int np, QuadConst q, double *__restrict__ Y) {
  nf = nfuncs(nf, nfp);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int f = t >> 2, c = t & 3;
  const bool active = f < nf;
  YDesc y = active ? yd[f] : yd[0];
  const int K = y.k, MTP = y.mtp, MTPP3 = MTP + 3, N = q.n;
  const double *T = TZ + (size_t)(active ? f : 0) * np;
  const double *Tw = TW + (size_t)(active ? f : 0) * np;
  double *Yf = Y + (size_t)(active ? f : 0) * np;
  const int s = c + 2;  // chain start: 2, 3, 4, 5
  double z = 0.0;
  if (active) {
    if (s <= 4) {
      double sum = 0.0;
      for (int kk = 2; kk <= 5; ++kk) sum = sum + q.CNC5C[kk - 2][s - 2] * T[kk];
      z = sum;
    } else {  // ZK(5) = ZK(1) + RTMP(5), ZK(1) = 0
      const double rtmp = q.C1 * (T[1] + T[5]) + q.C2 * (T[2] + T[4]) + q.C3 * T[3];
      z = 0.0 + rtmp;
    }
    Yf[s] = z;
    for (int i = s + 4; i <= MTPP3; i += 4) {
      const double rtmp = q.C1 * (T[i - 4] + T[i]) + q.C2 * (T[i - 3] + T[i - 1]) + q.C3 * T[i - 2];
      z = z + rtmp;
      Yf[i] = z;
    }
  }
  // asymptotic value (yzk.f90:150-171)
  const int owner = (MTPP3 - 2) & 3;
  const double z_top = __shfl_sync(0xffffffffu, z, (threadIdx.x & ~3) + owner);
  if (!active) return;
  double zklim, dif = 0.0;
  if (K == 0) {
    zklim = (y.b == y.d) ? 1.0 : 0.0;
    const double d0 = z - zklim;  // this chain's value at its last point (in [MTP, MTP+3])
    if (fabs(d0) > q.accy) dif = d0;
  } else {
    zklim = z_top;
  }
  const double *RTTKM = pw + (size_t)(1 * (KLIMIT + 1) + K) * np;
  const double *RTTK1 = pw + (size_t)(2 * (KLIMIT + 1) + K) * np;
  // backward pass: W recurrence on i <= MTP, assembly of Y = Z + W on 2..N
  int top = s;
  while (top + 4 < np) top += 4;
  double wk_next = 0.0;
  for (int i = top; i >= s; i -= 4) {
    if (i > N) {
      Yf[i] = 0.0;
      continue;
    }
    double zf;
    if (K == 0) {
      if (i <= MTPP3)
        zf = (dif != 0.0) ? Yf[i] - dif : Yf[i];
      else
        zf = zklim;
    } else {
      zf = (i <= MTPP3) ? Yf[i] * RTTKM[i] : zklim * RTTKM[i];
    }
    double wkf = 0.0;
    if (i <= MTP) {
      const double wk = wk_next + q.C1 * (Tw[i] + Tw[i + 4]) + q.C2 * (Tw[i + 1] + Tw[i + 3]) + q.C3 * Tw[i + 2];
      wk_next = wk;
      wkf = (K == 0) ? wk * R[i] : wk * RTTK1[i];
    }
    double yv = zf + wkf;
    if (i > y.mtpb) yv = 0.0;
    Yf[i] = yv;
  }
}

// Pair arrays on 2 <= i <= min(MF(a), MF(c)): D = (P_a P_c + Q_a Q_c) RPOR and
// A = w D, w the closed Newton-Cotes weight pattern of QUAD started at i = 2:
// C1 at 2, then C2, C3, C2, C4 repeating.
__global__ void k_apairs(const int2 *__restrict__ pairs, int npairs, const double *__restrict__ PF,
                         const double *__restrict__ QF, int ld, const int *__restrict__ MF,
                         const double *__restrict__ RPOR, int KC, QuadConst q, double *__restrict__ A,
                         double *__restrict__ D) {
  pdl_wait();
  const int p = blockIdx.y;
  if (p >= npairs) return;
  const int a = pairs[p].x, c = pairs[p].y;
  const int m = min(MF[a], MF[c]);
  // the last row is followed by KC_TILE zeros: k_rk_dot reads up to G - 1
  // points past a row's last one
  const int end = p + 1 < npairs ? KC : KC + KC_TILE;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < end; i += gridDim.x * blockDim.x) {
    double v = 0.0, rho = 0.0;
    if (i >= 2 && i <= m) {
      rho = (pf(PF, ld, i, a) * pf(PF, ld, i, c) + pf(QF, ld, i, a) * pf(QF, ld, i, c)) * RPOR[i];
      const int ph = (i - 2) & 3;
      const double w = (i == 2) ? q.C1 : (ph == 1 || ph == 3) ? q.C2 : (ph == 2) ? q.C3 : q.C4;
      v = w * rho;
    }
    A[(size_t)p * KC + i] = v;
    D[(size_t)p * KC + i] = rho;
  }
}

// QUAD's power-law head term and end-panel correction (quad.f90:52-103) for
// integral (a, c; f) whose GEMM part (grid points 3.., the Newton-Cotes weights
// folded into A) is `sum`, stored at VALTEIRK position pos; an integral whose
// head index is not 2 goes to the general QUAD list. TA(i) = D(i) Y(i).
struct RkTabs {
  const double *D, *Y;
  const YDesc *yd;
  const int *MF;
  const double *HD;
  int KC, np;
};
__device__ __forceinline__ void rk_head_store(int a, int c, int p, int f, long long pos, double sum, const RkTabs &t,
                                              const QuadConst &q, double *__restrict__ val,
                                              QuadItem *__restrict__ fb, int *__restrict__ nfb) {
  const YDesc y = t.yd[f];
  int mtp = min(t.MF[a], t.MF[c]);
  if (!(y.k == 0 && y.b == y.d)) mtp = min(mtp, y.mtp);
  const double *D = t.D + (size_t)p * t.KC, *Y = t.Y + (size_t)f * t.np, *HD = t.HD;
  bool ok = mtp >= 3;
  double res = 0.0;
  if (ok) {
    const double tai = D[2] * Y[2], taip1 = D[3] * Y[3];
    const double r = taip1 / tai;
    ok = !(fabs(tai) <= 0.0) && (r > 0.0);
    if (ok) {
      // QUAD's head term with the grid's factors per point (HD): the ratio
      // (TA(3)/RP(3)) / (TA(2)/RP(2)), sigma = log(ratio) / log(R(3)/R(2)),
      // R(2) TA(2)/RP(2) / (sigma + 1); equal to quad.f90's to rounding
      const double sigma = log(r * HD[t.np + 2]) * HD[2];
      const double fri = tai * HD[2 * t.np + 2];
      res = fri / (sigma + 1.0) + sum;
      if ((mtp - 2) % 4 == 0) res = res - q.C1 * (D[mtp] * Y[mtp]);
    }
  }
  if (ok) {
    val[pos] = res;
  } else {
    const int slot = atomicAdd(nfb, 1);
    fb[slot] = QuadItem{a, c, p, f, mtp, pos};
  }
}

// ---------------------------------------------------------------------------
// R^k contraction in FP64: for each k, O[p, f] = sum_i A[p, i] Y[f, i] over its
// pairs p = (a, c) and the Y functions f = (b, d) with b >= a, then QUAD's head
// term and end-panel correction per entry, written at the GENINTRK position
// (k, a, b, c, d). A warp takes 32 functions, one per lane, x NR pairs, whose
// rows are read uniformly; each entry is one FMA chain over the points in
// order, up to the pairs' last point. Bound: the FP64 pipe on large sets, the
// chain's latency on small ones; NR is the largest of 8, 4, 2, 1 that still
// gives every SM four warps (fewer rows per warp read Y more often, more leave
// SMs idle). A block of 32 x 64 entries in shared memory left most rows of a
// tile empty (a (k, a) problem has 2 to 12 pairs) and most SMs idle: 371 us
// for 16 subshells, now 22 us; the chains are the same, so are the bits.
// ---------------------------------------------------------------------------
struct TcRow {  // one row of a k: its pair, problem and position data
  int p, a, c, ic, ncA, cs_a;
  long long base;
};
template <int NR>
__global__ void __launch_bounds__(128) k_rk_dot(const RkTile *__restrict__ tiles, int ntiles,
                                                const TcRow *__restrict__ rows, const double *__restrict__ A,
                                                RkTabs t, QuadConst q, double *__restrict__ val, long long nval,
                                                QuadItem *__restrict__ fb, int *__restrict__ nfb) {
  pdl_wait();
  const int w = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (w >= ntiles) return;
  const RkTile T = tiles[w];
  const double *ar[NR];
  int m = 0;
#pragma unroll
  for (int r = 0; r < NR; ++r) {  // rows past the tile repeat its last one
    const TcRow rw = rows[T.r0 + min(r, T.rn - 1)];
    ar[r] = A + (size_t)rw.p * t.KC;
    m = max(m, min(t.MF[rw.a], t.MF[rw.c]));
  }
  const int f = T.f0 + min(lane, T.fn - 1);
  const double *y = t.Y + (size_t)f * t.np;
  double acc[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) acc[r] = 0.0;
  // points 2 .. m in groups of G, the next group loaded before the current one
  // is added (a chain of loads and FMAs waits on L2 at every group otherwise).
  // A(m + 1) is zero (the row's end or point 0 of the next row); the last
  // group's loads reach up to G - 1 points past m, its sums stop at m
  constexpr int G = NR >= 8 ? 4 : NR == 4 ? 8 : 16;
  static_assert(G - 1 <= KC_TILE, "the loads past the last pair's points stay in k_apairs's zeros");
  static_assert(G - 1 <= GPAD, "the loads past the last function's points stay in its row");
  double2 cy[G / 2], ca[NR][G / 2];
  auto load = [&](int i, double2 *yv, double2(*av)[G / 2]) {
#pragma unroll
    for (int u = 0; u < G / 2; ++u) {
      yv[u] = __ldg(reinterpret_cast<const double2 *>(y + i) + u);
#pragma unroll
      for (int r = 0; r < NR; ++r) av[r][u] = __ldg(reinterpret_cast<const double2 *>(ar[r] + i) + u);
    }
  };
  auto add = [&](const double2 *yv, const double2(*av)[G / 2], int left) {
#pragma unroll
    for (int u = 0; u < G / 2; ++u)
      if (2 * u < left)
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          acc[r] = fma(av[r][u].x, yv[u].x, acc[r]);
          acc[r] = fma(av[r][u].y, yv[u].y, acc[r]);
        }
  };
  load(2, cy, ca);
  int i = 2;
  for (; i + G <= m; i += G) {
    double2 ny[G / 2], na[NR][G / 2];
    load(i + G, ny, na);
    add(cy, ca, G);
#pragma unroll
    for (int u = 0; u < G / 2; ++u) {
      cy[u] = ny[u];
#pragma unroll
      for (int r = 0; r < NR; ++r) ca[r][u] = na[r][u];
    }
  }
  add(cy, ca, m + 1 - i);
  if (lane >= T.fn) return;
  const YDesc yd = t.yd[f];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    if (r >= T.rn) continue;
    const TcRow rw = rows[T.r0 + r];
    if (f < rw.cs_a) continue;  // b < a: not a GENINTRK entry
    const long long pos =
        rw.base + (long long)rw.ncA * (yd.cs - rw.cs_a) + (long long)rw.ic * yd.nd + (long long)(f - yd.cs);
    if (pos < 0 || pos >= nval) {  // position outside the table: report, never write
      atomicExch(nfb + 1, 1);
      continue;
    }
    rk_head_store(rw.a, rw.c, rw.p, f, pos, acc[r], t, q, val, fb, nfb);
  }
}

// ---------------------------------------------------------------------------
// The same contraction on the tensor cores, split-precision (Ozaki): each row
// of A and of Y is scaled by a power of two 2^e (|row| < 2^(e-1)) and cut
// into OZ_S slices of 7 bits, x = 2^e sum_s q_s 2^(-7(s+1)), each q_s the
// nearest integer to the remainder, so |q_s| <= 64 (every step is exact in
// FP64). Products of slice pairs (s, t) with s + t < OZ_S are exact integer
// tensor products (|q_s q_t| <= 4096); pairs with the same q = s + t share one
// FP32 accumulator in tensor memory, where at most 10 pairs x 256 grid points
// x 4096 < 2^24 keeps every partial sum an exact integer between flushes. The sum over q is then
// sum_q acc_q 2^(eA + eY - 7(q + 2)). With OZ_S = 10 the result agrees with
// the FP64 contraction to a few 1e-13 relative on R^k data.
// ---------------------------------------------------------------------------
constexpr int OZ_S = 10;

// ---------------------------------------------------------------------------
// The Ozaki contraction on GB300's fifth-generation tensor cores (tcgen05).
//
// For each k the rows of all (k, a) problems (the (a, c) pairs with a <= c
// and TRIANGRK(l_a, k, l_c), in GENINTRK's order) and all Y functions of k
// form one GEMM, cut into tiles of TC_M = 128 functions (the MMA's M) x
// TC_N = 48 rows (N); tiles that hold no needed entry (b < a for all) are
// skipped. k_oz_tile writes the int8-range slices (|q| <= 64) as fp16, which
// holds them exactly, straight into per-tile blocks laid out as the MMA reads
// them from shared memory (no-swizzle K-major core matrices: 8 rows x 16 B,
// neighbours in K 128 B apart, in M/N 256 B apart), one block per 32 grid
// points: 80 KB of Y slices, 30 KB of A slices.
//
// k_rk_tc, one CTA per SM taking the tiles in turn, is warp-specialised. Warp
// 4 streams the tiles' blocks into two shared-memory stages with
// cp.async.bulk (completion counted in bytes on a per-stage "full" mbarrier)
// and issues, per K = 16 step, the 55 slice-pair MMAs
// tcgen05.mma.cta_group::1.kind::f16 into the FP32 tensor-memory accumulator
// of their group q = s + t (OZ_S x TC_N columns); a tcgen05.commit to the
// stage's "empty" mbarrier frees the stage. Every TC_FLUSH stages (256 grid
// points, while every group sum is still an exact integer below 2^24) and at
// a tile's end warps 0-3 read their 32 lanes of each group (tcgen05.ld) and
// fold group q, scaled by 2^(-7q), into double-float sums; the next MMA of
// each group overwrites. The raw sum 2^(eA+eY-14) (h + l) is stored at the
// entry's GENINTRK position while the next tile runs; k_rk_finish_all adds
// the head term. Every wait is bounded: on a timeout the CTA records it,
// waits (bounded) for what it issued, frees its tensor memory and writes
// nothing more.
// Bound: an MMA takes 44 cycles whatever N is (16 to 48), the read of its 128
// Y rows from shared memory, so a tile's 990 are 44,000 of its 75,000 cycles;
// the rest are two flushes (7,000 each) and the waits for copies, 110 KB a
// stage from L2 to every SM. 43 subshells, k <= 8 (194 tiles): 94 us; 175 us
// with rolled MMA loops (descriptors formed by one thread, 80 cycles per
// MMA), a CTA per tile and values scaled by scalbn one at a time after it.
// ---------------------------------------------------------------------------
constexpr int TC_M = 128, TC_N = 48, TC_KC = 32, TC_FLUSH = 8;
constexpr int TC_YBLK = OZ_S * 2 * (TC_M / 8) * 2 * 64;  // fp16 elements per Y block (80 KB)
constexpr int TC_ABLK = OZ_S * 2 * (TC_N / 8) * 2 * 64;  // fp16 elements per A block (30 KB)
constexpr size_t TC_SMEM = (size_t)2 * (TC_YBLK + TC_ABLK) * sizeof(__half) + 128;
constexpr uint32_t TC_TMEM_COLS = 512;  // >= OZ_S * TC_N, a power of two
constexpr int TC_SPIN = 1 << 24;
constexpr int TC_THREADS = 160;  // warps 0-3: accumulators; warp 4: copies and MMAs

struct TcTile {
  int k, fg, pg;  // k; global indices of the Y block column and the A block column
  int f0, fn;     // first Y function and how many are valid
  int r0, rn;     // first row (TcRow index) and how many are valid
  int c0, c1, s;  // grid chunks [c0, c1) of this split of the tile, split index
};

}  // namespace

// GENINTRK's orbital-set-dependent structure and its work buffers, kept on
// the context between calls (gg_genintrk rebuilds it when the orbitals' l, j
// or kmax change)
struct RkCache {
  std::vector<int> key;
  int nf = 0, npairs = 0;
  int nr = 8;  // rows of a tile of the FP64 contraction
  std::vector<YDesc> yd;
  std::vector<int> kend, yslot, aslot, fidx, pidx;
  std::vector<int2> pairs;
  std::vector<RkTile> tiles;
  std::vector<TcRow> tcrows;
  std::vector<TcTile> tct;
  DBuf<YDesc> dYd;
  DBuf<int2> dPairs;
  DBuf<RkTile> dTiles;
  DBuf<int> dYslot, dAslot, dFidx, dPidx, dNfb, dEA, dEY;
  DBuf<int32_t> dKst;
  DBuf<TcTile> dTct;
  // split-K form of tct (each tile's grid chunks over nsplit CTAs) for the
  // chunk count it was made for, and the partial sums it writes
  std::vector<TcTile> tcs;
  int tcs_nch = -1, tcs_split = 0;
  DBuf<TcTile> dTcs;
  DBuf<double> dParts;
  DBuf<TcRow> dTcr;
  DBuf<double> dY, dA, dD, scratch;
  DBuf<QuadItem> dFb;
  DBuf<__half> dYt, dAt;
};

void rk_cache_free(RkCache *c) { delete c; }

const std::vector<int> *rk_structure_key(const gg_ctx *ctx) {
  return (ctx->rk.cache && ctx->rk.valid) ? &ctx->rk.cache->key : nullptr;
}

namespace {

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: start address, leading (K) byte offset
// 128, stride (M/N) byte offset 256, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) |
         ((uint64_t)1 << 46);
}

__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity, int spin = TC_SPIN) {
  uint32_t done = 0;
  for (int it = 0; it < spin && !done; ++it)
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
  return done != 0;
}

// one lane of the converged warp, the same at every call
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.u32 %0, 1, 0, P;\n}" : "=r"(p));
  return p != 0;
}

// x 2^(35-e) = X1 + d exactly with X1 = rint(x 2^(35-e)), |d| <= 1/2 (|x| <
// 2^(e-1)), X2 = rint(d 2^35): x = (X1 + X2 2^-35) 2^(e-35) to 2^(e-71),
// |X1|, |X2| <= 2^34. A normal x on its mantissa in integers (GB300 issues
// FP64 slowly, and roundings to nearest even need none).
__device__ __forceinline__ void oz_parts(double x, int e, long long &X1, long long &X2) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)(bits >> 52) & 0x7ff;
  X1 = X2 = 0;
  if ((bits << 1) == 0) return;
  if (ex == 0 || ex == 0x7ff) {
    const double xs = scalbn(x, 35 - e), x1 = rint(xs);
    X1 = (long long)x1;
    X2 = (long long)rint((xs - x1) * 34359738368.0);  // 2^35
    return;
  }
  const unsigned long long m = (bits & 0xfffffffffffffull) | (1ull << 52);
  const int sh = 1040 + e - ex;  // |x| 2^(35 - e) = m 2^-sh < 2^34, so sh is 19 or more
  // v / 2^s to nearest even, 0 < s <= 53 (v < 2^53: beyond that it rounds to 0)
  auto div = [](unsigned long long v, int s) {
    const unsigned long long q = v >> s, r = v & ((1ull << s) - 1), h = 1ull << (s - 1);
    return q + (r > h || (r == h && (q & 1)));
  };
  const unsigned long long q = sh > 53 ? 0 : div(m, sh);
  const long long d = sh > 53 ? (long long)m : (long long)(m - (q << sh));  // in units of 2^-sh
  const unsigned long long a = d < 0 ? -d : d;
  const long long t = sh <= 35 ? (long long)(a << (35 - sh)) : sh - 35 > 53 ? 0 : (long long)div(a, sh - 35);
  const bool neg = (bits >> 63) != 0;
  X1 = neg ? -(long long)q : (long long)q;
  X2 = neg != (d < 0) ? -t : t;
}

// Slices of rows into their tile blocks: a CTA takes eight row slots (slot =
// tile block column g, row m < R; src_row[slot] < 0 pads with zeros). A row's
// exponent goes to exps[src_row] (the same row always gets the same value).
// A thread takes eight points of a row, a 16-byte unit of the block per
// slice; the eight rows' units make 128 bytes. Each of oz_parts' X1 and X2
// gives five balanced base-128 digits (|digit| <= 64).
// Bound: integer issue (43 subshells, k <= 8: 57 MB written, 35 us; a CTA per
// row 46 us, and with the parts and the row's largest value in FP64 and 2-byte
// stores 74 us).
constexpr int OZ_T = 256;
template <int R>
__global__ void __launch_bounds__(OZ_T) k_oz_tile(const double *__restrict__ M, int pitch, int K, int nch,
                                                  const int *__restrict__ src_row, int *__restrict__ exps,
                                                  __half *__restrict__ dst) {
  pdl_wait();
  constexpr int BLK = OZ_S * 2 * (R / 8) * 2 * 64;
  __shared__ int se[8];
  const int s0 = blockIdx.x * 8, g = s0 / R, m8 = s0 % R / 8;
  {
    const int lane = threadIdx.x & 31, row = src_row[s0 + (threadIdx.x >> 5)];
    const double *src = M + (size_t)max(row, 0) * pitch;
    unsigned long long mx = 0;  // the largest |x| but NaN, as its bits
    if (row >= 0)
      for (int i = lane; i < K; i += 32) {
        const unsigned long long v = (unsigned long long)__double_as_longlong(src[i]) & 0x7fffffffffffffffull;
        if (v > mx && v <= 0x7ff0000000000000ull) mx = v;
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) {
      const int e = mx ? ilogb(__longlong_as_double((long long)mx)) + 2 : 0;  // mx < 2^(e-1)
      se[threadIdx.x >> 5] = e;
      if (row >= 0) exps[row] = e;
    }
  }
  __syncthreads();
  const int m = threadIdx.x & 7, row = src_row[s0 + m], e = se[m];
  const double *src = M + (size_t)max(row, 0) * pitch;
  __half *base = dst + (size_t)g * nch * BLK + (size_t)m8 * 2 * 64 + m * 8;
  for (int u = threadIdx.x >> 3; u < nch * (TC_KC / 8); u += OZ_T / 8) {
    const int i0 = 8 * u;
    uint32_t out[OZ_S][4];  // the unit's digits + 1088 as fp16, two to a word
#pragma unroll
    for (int p = 0; p < 4; ++p) {
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const int i = i0 + 2 * p + w;
        long long X[2];
        oz_parts(row >= 0 && i < K ? src[i] : 0.0, e, X[0], X[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          long long v = X[h];
#pragma unroll
          for (int q = 4; q >= 0; --q) {
            const int r = q ? (int)(((v + 64) & 127) - 64) : (int)v;  // balanced remainder; at last |v| <= 64
            const uint32_t c = (uint32_t)(0x6400 + 64 + r);           // fp16 of 1088 + r
            out[h * 5 + q][p] = w ? out[h * 5 + q][p] | (c << 16) : c;
            v = (v - r) >> 7;
          }
        }
      }
    }
    const int c = u / (TC_KC / 8), j = (u / 2) % 2, k8 = u % 2;
    __half *blk = base + (size_t)c * BLK + k8 * 64;
    const __half2 off = __floats2half2_rn(1088.0f, 1088.0f);
#pragma unroll
    for (int q = 0; q < OZ_S; ++q) {
      uint4 o;
      uint32_t *ow = &o.x;
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        __half2 h = *reinterpret_cast<__half2 *>(&out[q][p]);
        h = __hsub2(h, off);
        ow[p] = *reinterpret_cast<uint32_t *>(&h);
      }
      *reinterpret_cast<uint4 *>(blk + (size_t)(q * 2 + j) * (R / 8) * 2 * 64) = o;
    }
  }
}

__global__ void __launch_bounds__(TC_THREADS, 1) k_rk_tc(const TcTile *__restrict__ tiles, int ntiles,
                                                         const TcRow *__restrict__ rows,
                                                         const __half *__restrict__ Yt,
                                                         const __half *__restrict__ At, int nch,
                                                         const int *__restrict__ eA, const int *__restrict__ eY,
                                                         const YDesc *__restrict__ yd, double *__restrict__ val,
                                                         long long nval, int *__restrict__ flags, int stall_tile) {
  pdl_wait();
  extern __shared__ __align__(1024) unsigned char tsm[];
  __half *Ysm = reinterpret_cast<__half *>(tsm);
  __half *Asm = Ysm + 2 * TC_YBLK;
  uint64_t *full = reinterpret_cast<uint64_t *>(Asm + 2 * TC_ABLK);
  uint64_t *empty = full + 2;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(empty + 2);
  int *okflag = reinterpret_cast<int *>(tslot + 1);
  __shared__ TcRow trow[TC_N];
  __shared__ int tex[TC_N];  // the rows' exponents
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tslot)),
                 "r"(TC_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int st = 0; st < 2; ++st) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&full[st])), "r"(1));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&empty[st])), "r"(1));
    }
    *okflag = 1;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);
  if (warp == 4) {
    // copies and MMAs (one elected lane issues; the warp stays converged).
    // The chunks of the CTA's tiles form one stream, chunk j in stage j & 1.
    // A tile named by stall_tile (a test of the bounded waits) withholds its
    // first copy and polls briefly: its first wait runs out with nothing in
    // flight.
    constexpr uint32_t YB = TC_YBLK * sizeof(__half), AB = TC_ABLK * sizeof(__half);
    int ct = blockIdx.x, cc = 0, cn = 0;  // the copy stream: tile, next chunk of it, its chunks
    const char *ysrc = nullptr, *asrc = nullptr;
    auto open = [&] {
      if (ct >= ntiles) return;
      const TcTile C = tiles[ct];
      cc = 0;
      cn = C.c1 - C.c0;
      ysrc = reinterpret_cast<const char *>(Yt) + ((size_t)C.fg * nch + C.c0) * YB;
      asrc = reinterpret_cast<const char *>(At) + ((size_t)C.pg * nch + C.c0) * AB;
    };
    int issued = -1;  // last chunk whose MMAs were committed
    int copied = -1;  // last chunk whose copy was issued
    auto copy = [&] {
      if (ct >= ntiles || ct == stall_tile) return;
      const int st = (copied + 1) & 1;
      if (elect_one()) {
        const uint32_t fb = smem_addr(&full[st]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(YB + AB) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_addr(Ysm + st * TC_YBLK)),
            "l"(ysrc + (size_t)cc * YB), "r"(YB), "r"(fb)
            : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_addr(Asm + st * TC_ABLK)),
            "l"(asrc + (size_t)cc * AB), "r"(AB), "r"(fb)
            : "memory");
      }
      __syncwarp();
      ++copied;
      if (++cc == cn) {
        ct += gridDim.x;
        open();
      }
    };
    bool ok = true;
    open();
    copy();
    int jg = 0;  // the stream's chunk
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      const int nloc = __shfl_sync(0xffffffffu, tiles[tile].c1 - tiles[tile].c0, 0);
      const int rn = __shfl_sync(0xffffffffu, tiles[tile].rn, 0);
      const int spin = tile == stall_tile ? (1 << 12) : TC_SPIN;
      // N: the tile's valid rows, rounded up to a multiple of 16
      const uint32_t idesc = (1u << 4) | ((uint32_t)((rn + 15) / 16 * 2) << 17) | ((uint32_t)(TC_M >> 4) << 24);
      for (int j = 0; j < nloc; ++j, ++jg) {
        const int st = jg & 1;
        if (ok) ok = __all_sync(0xffffffffu, tc_wait(smem_addr(&full[st]), (jg >> 1) & 1, spin));
        if (ok) {
          asm volatile("tcgen05.fence::after_thread_sync;");
          if (elect_one()) {
            const uint32_t yb = smem_addr(Ysm + st * TC_YBLK), ab = smem_addr(Asm + st * TC_ABLK);
            // unrolled, so that a descriptor is one addition: with the loops
            // rolled the issuing thread, not the tensor core, set the pace
#pragma unroll 1
            for (int ks = 0; ks < 2; ++ks) {
              // the first MMA of each group after a flush (slice 0 of A) overwrites
              const uint32_t cont = (j % TC_FLUSH == 0 && ks == 0) ? 0u : 1u;
              const uint64_t b0 = tc_desc(ab + (uint32_t)ks * ((TC_N / 8) * 2 * 64 * 2));
              const uint64_t a0 = tc_desc(yb + (uint32_t)ks * ((TC_M / 8) * 2 * 64 * 2));
#pragma unroll
              for (int sa = 0; sa < OZ_S; ++sa)
#pragma unroll
                for (int t = 0; t < OZ_S - sa; ++t)
                  asm volatile(
                      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(
                          tmem + (uint32_t)((sa + t) * TC_N)),
                      "l"(a0 + (uint64_t)(t * 2 * (TC_M / 8) * 2 * 64 * 2 / 16)),
                      "l"(b0 + (uint64_t)(sa * 2 * (TC_N / 8) * 2 * 64 * 2 / 16)), "r"(idesc), "r"(sa ? 1u : cont));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_addr(&empty[st]))
                         : "memory");
          }
          __syncwarp();
          issued = jg;
          // refill the other stage with the stream's next chunk once chunk jg - 1's MMAs are done
          if (copied == jg) {
            if (jg >= 1)
              ok = __all_sync(0xffffffffu, tc_wait(smem_addr(&empty[(jg - 1) & 1]), ((jg - 1) >> 1) & 1, spin));
            if (ok) copy();
          }
        }
        if ((j + 1) % TC_FLUSH == 0 || j == nloc - 1) {
          if (ok) ok = __all_sync(0xffffffffu, tc_wait(smem_addr(&empty[st]), (jg >> 1) & 1, spin));  // MMAs done
          if (!ok && lane == 0) *okflag = 0;
          asm volatile("tcgen05.fence::before_thread_sync;");
          __syncthreads();  // A: the accumulators are ready (or the flag says no)
          __syncthreads();  // B: warps 0-3 have read them
          asm volatile("tcgen05.fence::after_thread_sync;");
        }
      }
    }
    if (!ok) {
      // timed out: before the tensor memory is freed and the CTA leaves,
      // wait (bounded) for the last copy issued to land in shared memory and
      // for the last committed MMAs to finish; 2 records a failed drain
      bool drained = true;
      if (copied >= 0) drained = tc_wait(smem_addr(&full[copied & 1]), (copied >> 1) & 1);
      if (issued >= 0) drained = tc_wait(smem_addr(&empty[issued & 1]), (issued >> 1) & 1) && drained;
      if (lane == 0) atomicMax(flags + 1, drained ? 1 : 2);
    }
  } else {
    // warps 0-3: lane quadrant `warp` of each group accumulator; a tile's
    // values are stored while warp 4 works on the next tile
    const int m = warp * 32 + lane;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      const TcTile T = tiles[tile];
      const int nflush = (T.c1 - T.c0 + TC_FLUSH - 1) / TC_FLUSH;
      const bool valid = m < T.fn;
      const int f = valid ? T.f0 + m : T.f0;
      const YDesc y = yd[f];
      const int ey = eY[f] - 14;
      asm volatile("bar.sync 1, 128;" ::: "memory");  // the previous tile's rows are no longer read
      if (tid < TC_N) {
        trow[tid] = (tid < T.rn) ? rows[T.r0 + tid] : TcRow{-1, 0, 0, 0, 0, 0};
        tex[tid] = (tid < T.rn) ? eA[trow[tid].p] : 0;
      }
      float ah[TC_N], al[TC_N];
#pragma unroll
      for (int n = 0; n < TC_N; ++n) ah[n] = al[n] = 0.f;
      for (int fl = 0; fl < nflush; ++fl) {
        __syncthreads();  // A
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (*okflag) {
#pragma unroll 1
          for (int qg = 0; qg < OZ_S; ++qg) {
            const float scale = __int_as_float((127 - 7 * qg) << 23);  // 2^(-7 qg)
            uint32_t r[TC_N];
#pragma unroll
            for (int h = 0; h < TC_N / 16; ++h) {
              uint32_t *v = r + 16 * h;
              const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(qg * TC_N + h * 16);
              asm volatile(
                  "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                  "[%16];"
                  : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                    "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                    "=r"(v[15])
                  : "r"(taddr));
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
            for (int n = 0; n < TC_N; ++n) asm volatile("" : "+r"(r[n]));  // read only after the wait
#pragma unroll
            for (int n = 0; n < TC_N; ++n) {
              // (ah, al) += v: TwoSum into the high part, the error into al
              const float v = __uint_as_float(r[n]) * scale;
              const float sv = ah[n] + v;
              const float bb = sv - ah[n];
              const float e = (ah[n] - (sv - bb)) + (v - bb);
              ah[n] = sv;
              al[n] = al[n] + e;
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();  // B
      }
      if (!*okflag) continue;
      // split s of the contraction: its partial sum (val + s nval), scaled in
      // the exponent field where the result is a normal number
      double *out = val + (long long)T.s * nval;
      bool outside = false, scaled = true;
#pragma unroll
      for (int n = 0; n < TC_N; ++n) {
        const TcRow rw = trow[n];
        const long long pos =
            rw.base + (long long)rw.ncA * (y.cs - rw.cs_a) + (long long)rw.ic * y.nd + (long long)(f - y.cs);
        const bool need = valid && n < T.rn && f >= rw.cs_a;  // not padding, nor b < a
        const bool in = pos >= 0 && pos < nval;
        const int e = tex[n] + ey;
        const double v = (double)ah[n] + (double)al[n];
        const int hi = __double2hiint(v), ex = (hi >> 20) & 0x7ff;
        const bool zero = ((hi & 0x7fffffff) | __double2loint(v)) == 0;
        const bool fast = (ex > 0 && ex + e > 0 && ex + e < 2047) || zero;
        outside |= need && !in;
        scaled &= !need || fast;
        if (need && in) out[pos] = zero ? v : __hiloint2double(hi + (e << 20), __double2loint(v));
      }
      if (!scaled) {
#pragma unroll 1
        for (int n = 0; n < T.rn; ++n) {
          const TcRow rw = trow[n];
          const long long pos =
              rw.base + (long long)rw.ncA * (y.cs - rw.cs_a) + (long long)rw.ic * y.nd + (long long)(f - y.cs);
          double v = 0.0;
#pragma unroll
          for (int u = 0; u < TC_N; ++u)
            if (u == n) v = (double)ah[u] + (double)al[u];
          if (f >= rw.cs_a && pos >= 0 && pos < nval) out[pos] = scalbn(v, tex[n] + ey);
        }
      }
      if (outside) atomicExch(flags, 1);  // position outside the table
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS));
}

// QUAD head term for every table entry, one thread per entry: (a, b, c, d)
// from INDTEIRK, k from KSTART, the pair from pidx[a KEY + c] and the Y
// function from fidx[(k KEY + b) KEY + d]; the entry's GEMM part is the sum, in
// split order, of parts[s n + i] for s < nsplit (parts == val when the
// contraction was not split).
__global__ void k_rk_finish_all(const int32_t *__restrict__ ind, long long n, const int32_t *__restrict__ kstart,
                                int kloop, int KEY, const int *__restrict__ fidx, const int *__restrict__ pidx,
                                RkTabs tb, QuadConst q, double *__restrict__ val, QuadItem *__restrict__ fb,
                                int *__restrict__ nfb, const double *__restrict__ parts, int nsplit) {
  pdl_wait();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    int p = ind[i];
    const int d = p % KEY;
    p /= KEY;
    const int c = p % KEY;
    p /= KEY;
    const int b = p % KEY, a = p / KEY;
    int k = 0;
    while (k < kloop && (long long)kstart[k + 1] - 1 <= i) ++k;
    const int f = fidx[((size_t)k * KEY + b) * KEY + d], pr = pidx[(size_t)a * KEY + c];
    if (f < 0 || pr < 0) {
      atomicExch(nfb + 1, 1);
      continue;
    }
    double gemm = parts[i];
    for (int t = 1; t < nsplit; ++t) gemm += parts[(long long)t * n + i];
    rk_head_store(a, c, pr, f, i, gemm, tb, q, val, fb, nfb);
  }
}

// General per-integral QUAD (SLATER): TA(i) = ((P_a P_c + Q_a Q_c) RPOR) Y_f(i),
// one warp per integral, sequential reference-order sum on lane 0. TA lies in
// shared memory, or in `work` (np doubles per warp) on a grid too long for it.
__global__ void k_quad_items(const QuadItem *__restrict__ items, int nitems,
                             const double *__restrict__ Y, int np, const double *__restrict__ PF,
                             const double *__restrict__ QF, int ld, const double *__restrict__ R,
                             const double *__restrict__ RP, const double *__restrict__ RPOR, QuadConst q,
                             double *work, double *__restrict__ out) {
  extern __shared__ double sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  double *TA = work ? work + ((size_t)blockIdx.x * wpb + warp) * np : sm + (size_t)warp * np;
  for (int it = blockIdx.x * wpb + warp; it < nitems; it += gridDim.x * wpb) {
    const QuadItem w = items[it];
    const double *Yf = Y + (size_t)w.f * np;
    for (int i = lane; i < np; i += 32) {
      double v = 0.0;
      if (i >= 2 && i <= w.mtp)
        v = ((pf(PF, ld, i, w.a) * pf(PF, ld, i, w.c) + pf(QF, ld, i, w.a) * pf(QF, ld, i, w.c)) * RPOR[i]) * Yf[i];
      TA[i] = v;
    }
    __syncwarp();
    if (lane == 0) out[w.pos] = quad_seq(TA, w.mtp, R, RP, q);
    __syncwarp();
  }
}

// The same QUAD for the table's items, one warp per integral with the work
// spread over the lanes: the head index (first i in [2, MTP-1] that passes
// quad_head) by ballot, the 4-point panel sums
// (quad.f90:94-99) split over the lanes and combined by a fixed butterfly,
// so the result is deterministic. Only the order of the panel sum differs
// from quad_seq (a few ulps of the sum of |terms|). TA(i) = D(i) Y(i) from the
// pair array; formed from the orbitals at every use the 43-orbital table's
// items took 103 us, so 55 us.
__global__ void k_quad_table(const QuadItem *__restrict__ items, const int *__restrict__ nitems_p, int nitems_max,
                             RkTabs tb, QuadConst q, double *__restrict__ out) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  const int nitems = min(*nitems_p, nitems_max);
  const double *HD = tb.HD;
  const int np = tb.np;
  // One item per warp for the head index and the sum; the block's items then
  // get their head terms (a logarithm and divisions: serial FP64 work that
  // would otherwise occupy a warp per item) from the lanes of warp 0, one
  // item each
  __shared__ int sh_head[32];
  __shared__ double sh_s[32];
  for (int base = blockIdx.x * wpb; base < nitems; base += gridDim.x * wpb) {
    const int it = base + (threadIdx.x >> 5);
    if (it < nitems) {
      const QuadItem w = items[it];
      const double *D = tb.D + (size_t)w.p * tb.KC, *Y = tb.Y + (size_t)w.f * np;
      int head = -1;
      for (int i0 = 2; i0 <= w.mtp - 1 && head < 0; i0 += 32) {
        const int i = i0 + lane;
        bool hit = false;
        if (i <= w.mtp - 1) {
          hit = quad_head(D[i] * Y[i], D[i + 1] * Y[i + 1]);
        }
        const unsigned bal = __ballot_sync(0xffffffffu, hit);
        if (bal) head = i0 + __ffs(bal) - 1;
      }
      double sp = 0.0;
      auto ta = [&](int j) { return j <= w.mtp ? D[j] * Y[j] : 0.0; };
      if (head >= 0)
        for (int j = head + 1 + 4 * lane; j <= w.mtp; j += 128)
          sp += q.C2 * (ta(j) + ta(j + 2)) + q.C3 * ta(j + 1) + q.C4 * ta(j + 3);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sp += __shfl_xor_sync(0xffffffffu, sp, o);
      if (lane == 0) {
        sh_head[threadIdx.x >> 5] = head;
        sh_s[threadIdx.x >> 5] = sp;
      }
    }
    __syncthreads();
    if (threadIdx.x < wpb && base + (int)threadIdx.x < nitems) {
      const QuadItem w = items[base + threadIdx.x];
      const double *D = tb.D + (size_t)w.p * tb.KC, *Y = tb.Y + (size_t)w.f * np;
      const int i = sh_head[threadIdx.x];
      double result = 0.0;
      if (i >= 0) {
        // quad.f90:61-103 with the grid's factors per point (HD)
        const double tai = D[i] * Y[i], taip1 = D[i + 1] * Y[i + 1];
        const double sigma = log((taip1 / tai) * HD[np + i]) * HD[i];
        result = (tai * HD[2 * np + i]) / (sigma + 1.0);
        result = result + q.C1 * tai;
        result = result + sh_s[threadIdx.x];
        if ((w.mtp - i) % 4 == 0) result = result - q.C1 * (D[w.mtp] * Y[w.mtp]);
      }
      out[w.pos] = result;
    }
    __syncthreads();
  }
}

// YPOT / XPOT (rmcdhf90/ypot.f90:35-49, xpot.f90:31-54): sum_t COEFF TB (YPOT),
// sum_t CTB QF and sum_t CTB PF with CTB = COEFF TB (XPOT), cut into chunks of
// terms. A block takes 64 grid points of one chunk, its four rows of threads a
// quarter of the terms each; the rows' sums meet in shared memory and the
// chunk's are stored for k_pot_final, which adds them in list order. An XPOT
// chunk is ordered by the orbital the terms multiply, so that a run of terms
// of one orbital sums COEFF TB and multiplies by QF and PF once. Bound: the
// FP64 pipe, one operation per term and point and two per run (6,600 terms of
// 34 subshells: 26 us per orbital, 34 with three operations per term; one
// thread per point adding the terms in list order left the pipe to one
// dependent addition per term: 233 us).
constexpr int POT_CHUNK = 256;  // terms staged in shared memory at a time
struct PotChunk {
  const int *key, *iorb;  // iorb null: YPOT
  const double *coef;
  size_t out;             // where its n sums (YPOT) or 2 n (XPOT) go
  int nt;
};
__global__ void __launch_bounds__(256) k_pot_part(const PotChunk *__restrict__ ch, const int *__restrict__ tab,
                                                  const double *__restrict__ Y, int np,
                                                  const double *__restrict__ PF, const double *__restrict__ QF,
                                                  int ld, int n, double *__restrict__ part) {
  pdl_wait();
  __shared__ int sf[POT_CHUNK], so[POT_CHUNK];
  __shared__ int4 sk[POT_CHUNK / 4];
  __shared__ double sc[POT_CHUNK], red[2][4][64];
  const PotChunk g = ch[blockIdx.y];
  const int tid = threadIdx.x, tx = tid & 63, ty = tid >> 6;
  const int i = 1 + blockIdx.x * 64 + tx;
  const bool x = g.iorb != nullptr, in = i <= n;
  double a0 = 0.0, a1 = 0.0;
  for (int t0 = 0; t0 < g.nt; t0 += POT_CHUNK) {
    const int nt = min(POT_CHUNK, g.nt - t0);
    __syncthreads();
    const int io = x && tid < nt ? g.iorb[t0 + tid] : 1, k = io * POT_CHUNK + tid;
    int pos = tid;
    if (x) {  // the term's place: how many have a lower orbital, or the same and stand before it
      reinterpret_cast<int *>(sk)[tid] = tid < nt ? k : INT_MAX;
      __syncthreads();
      pos = 0;
#pragma unroll 16
      for (int u = 0; u < POT_CHUNK / 4; ++u) {
        const int4 v = sk[u];
        pos += (v.x < k) + (v.y < k) + (v.z < k) + (v.w < k);
      }
    }
    if (tid < nt) {
      sf[pos] = max(tab[g.key[t0 + tid]] - 1, 0);  // 0: a label the parser refused
      so[pos] = io;
      sc[pos] = g.coef[t0 + tid];
    }
    __syncthreads();
    const int tb = nt * ty / 4, te = nt * (ty + 1) / 4;
    if (!in || tb == te) continue;
    int o = so[tb];
    double run = 0.0, qv = x ? pf(QF, ld, i, o) : 1.0, pv = x ? pf(PF, ld, i, o) : 0.0;
    for (int t = tb; t < te; t += 8) {
      double yv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) yv[u] = t + u < te ? __ldg(Y + (size_t)sf[t + u] * np + i) : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (t + u >= te) break;
        if (so[t + u] != o) {  // the next run
          a0 = fma(run, qv, a0);
          a1 = fma(run, pv, a1);
          run = 0.0;
          o = so[t + u];
          qv = pf(QF, ld, i, o);
          pv = pf(PF, ld, i, o);
        }
        run = fma(sc[t + u], yv[u], run);
      }
    }
    a0 = fma(run, qv, a0);
    a1 = fma(run, pv, a1);
  }
  red[0][ty][tx] = a0;
  red[1][ty][tx] = a1;
  __syncthreads();
  if (ty < (x ? 2 : 1) && in)
    part[g.out + (size_t)ty * n + i - 1] = (red[ty][0][tx] + red[ty][1][tx]) + (red[ty][2][tx] + red[ty][3][tx]);
}

// The lists' labels decoded on the device, one thread per term (the
// first ny YPOT labels, then XPOT labels): the term's (K, a, b) key into a dense table
// over K <= KLIMIT and the orbital pairs; the orbital it multiplies (XPOT) and
// COEFF (XPOT: XA/C, as the reference forms it). The first term of a key
// takes the next function number (info[0]), writes its YZK descriptor and
// leaves the number + 1 in the table. The numbers depend on the order in
// which the threads run, no value does: every term finds its function by its
// key. (Marking the keys and numbering them by one block in table order took
// 16 us of a 34-subshell COFPOT call.) A label outside the orbital set or
// with K above KLIMIT sets info[1].
__global__ void k_parse_terms(int64_t ny, int64_t nt, const int32_t *__restrict__ lab, const double *__restrict__ co,
                              int nw, double c, const int *__restrict__ MF, int n, int *__restrict__ tab,
                              YDesc *__restrict__ yd, int *__restrict__ key, int *__restrict__ iorb,
                              double *__restrict__ coef, int *__restrict__ info) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nt; e += (int64_t)gridDim.x * blockDim.x) {
    const int32_t l0 = lab[e];
    const int mode = e < ny ? 0 : 1;
    int64_t l = l0;
    const int k = (int)(l % KEYORB);
    l /= KEYORB;
    const int a = (int)(l % KEYORB);
    l /= KEYORB;
    const int64_t b = mode == 0 ? l : l % KEYORB;
    const int64_t io = mode == 0 ? 1 : l / KEYORB;
    if (l0 < 0 || k > KLIMIT || a < 1 || a > nw || b < 1 || b > nw || io < 1 || io > nw) {
      atomicOr(info + 1, 1);
      key[e] = 0;
      iorb[e] = 1;
      coef[e] = 0.0;
      continue;
    }
    const int kk = (k * nw + (a - 1)) * nw + (int)(b - 1);
    if (atomicCAS(tab + kk, 0, -1) == 0) {
      const int f = atomicAdd(info, 1);
      yd[f] = YDesc{k, a, (int)b, min(MF[a], MF[b]), n, 0, 1};
      tab[kk] = f + 1;
    }
    key[e] = kk;
    iorb[e] = (int)io;
    coef[e] = mode == 0 ? co[e] : co[e] / c;
  }
}

// DPBDT (lib9290/dpbdt.f90:39-99): 13-point derivative of orbital J at grid
// index i (1-based): the end rows from the 13 x 13 table, the interior by the
// antisymmetric 12-neighbour formula.
__device__ __forceinline__ void dpbdt_point(const double *PF, const double *QF, int ld, int J, const QuadConst &q,
                                            int i, double &hp, double &hq) {
  const int N = q.n;
  hp = 0.0;
  hq = 0.0;
  if (i <= 6) {
    for (int k = 1; k <= 13; ++k) hp = hp + q.A13[i - 1][k - 1] * pf(PF, ld, k, J);
    for (int k = 1; k <= 13; ++k) hq = hq + q.A13[i - 1][k - 1] * pf(QF, ld, k, J);
  } else if (i <= N - 6) {
    const double A1 = q.A13[6][0], A2 = q.A13[6][1], A3 = q.A13[6][2], A4 = q.A13[6][3], A5 = q.A13[6][4],
                 A6 = q.A13[6][5];
    hp = A1 * (pf(PF, ld, i - 6, J) - pf(PF, ld, i + 6, J)) + A2 * (pf(PF, ld, i - 5, J) - pf(PF, ld, i + 5, J)) +
         A3 * (pf(PF, ld, i - 4, J) - pf(PF, ld, i + 4, J)) + A4 * (pf(PF, ld, i - 3, J) - pf(PF, ld, i + 3, J)) +
         A5 * (pf(PF, ld, i - 2, J) - pf(PF, ld, i + 2, J)) + A6 * (pf(PF, ld, i - 1, J) - pf(PF, ld, i + 1, J));
    hq = A1 * (pf(QF, ld, i - 6, J) - pf(QF, ld, i + 6, J)) + A2 * (pf(QF, ld, i - 5, J) - pf(QF, ld, i + 5, J)) +
         A3 * (pf(QF, ld, i - 4, J) - pf(QF, ld, i + 4, J)) + A4 * (pf(QF, ld, i - 3, J) - pf(QF, ld, i + 3, J)) +
         A5 * (pf(QF, ld, i - 2, J) - pf(QF, ld, i + 2, J)) + A6 * (pf(QF, ld, i - 1, J) - pf(QF, ld, i + 1, J));
  } else {
    const int irow = i - N + 13;
    for (int k = 1; k <= 13; ++k) hp = hp + q.A13[irow - 1][k - 1] * pf(PF, ld, N - 13 + k, J);
    for (int k = 1; k <= 13; ++k) hq = hq + q.A13[irow - 1][k - 1] * pf(QF, ld, N - 13 + k, J);
  }
}

// One orbital's potentials at each grid point from its lists' chunk sums:
//   YP = ZZ - sum, XP = sum CTB QF, XQ = -sum CTB PF (the chunks in list order);
// LAGCON (rmcdhf90/lagcon.f90:46-55): per multiplier in list order,
//   XP = XP + WARI QF(I,M), XQ = XQ - WARI PF(I,M), WARI = WA R(I), I <= MF(M);
//   lag[t] = M and lag_w[t] = ECV WB of the multipliers the host kept (those of
//   pairs with this orbital, |WA| >= EPS);
// DACON (rmcdhf90/dacon.f90:25-46): per entry of the list in order, with TA,
//   TB = DPBDT(IORB) at the point, for I = 2..MF(IORB):
//   XP(I) += COEFF (TA RPORII + FK PFI - (2C R(I) + ZBCI) QFI),
//   XQ(I) += COEFF (TB RPORII - FK QFI + ZBCI PFI),
//   RPORII = 1/(H RPOR(I)), ZBCI = ZZ(I)/C, FK = kappa(IORB).
struct PotFinal {
  double *out;  // YP, XP, XQ: n each
  size_t yc, xc;  // the lists' chunk sums
  int nyc, nxc;
  const int *lag, *da;
  const double *lag_w, *da_w;
  int nlag, nda;
};
// A block takes 32 points, its PF_ROWS rows of threads every PF_ROWS-th chunk,
// multiplier and DACON entry; the rows' sums are added in row order.
constexpr int PF_ROWS = 8;
__global__ void __launch_bounds__(32 * PF_ROWS) k_pot_final(const PotFinal *__restrict__ jobs,
                                                            const double *__restrict__ part, int n,
                                                            const int *__restrict__ NAK, const int *__restrict__ MF,
                                                            const double *__restrict__ R,
                                                            const double *__restrict__ RPOR,
                                                            const double *__restrict__ ZZ,
                                                            const double *__restrict__ PF,
                                                            const double *__restrict__ QF, int ld, QuadConst q) {
  pdl_wait();
  __shared__ double red[3][PF_ROWS][32];
  const PotFinal g = jobs[blockIdx.y];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int i = 1 + blockIdx.x * 32 + tx;
  double y = 0.0, p = 0.0, m = 0.0;
  if (i <= n) {
    const double *yc = part + g.yc + i - 1, *xc = part + g.xc + i - 1;
    for (int c = ty; c < g.nyc; c += PF_ROWS) y += __ldg(yc + (size_t)c * n);
#pragma unroll 4
    for (int c = ty; c < g.nxc; c += PF_ROWS) {
      p += __ldg(xc + (size_t)2 * c * n);
      m -= __ldg(xc + (size_t)(2 * c + 1) * n);
    }
    for (int t = ty; t < g.nlag; t += PF_ROWS) {
      const int M = g.lag[t];
      if (i > MF[M]) continue;
      const double wari = g.lag_w[t] * R[i];
      p = p + wari * pf(QF, ld, i, M);
      m = m - wari * pf(PF, ld, i, M);
    }
    if (ty < g.nda && i >= 2) {
      const double twoc = q.c + q.c, rporii = 1.0 / (q.h * RPOR[i]), zbci = ZZ[i] / q.c;
      for (int t = ty; t < g.nda; t += PF_ROWS) {
        const int io = g.da[t];
        if (i > MF[io]) continue;
        double ta, tb;
        dpbdt_point(PF, QF, ld, io, q, i, ta, tb);
        const double coeff = g.da_w[t], fk = (double)NAK[io];
        const double pfi = pf(PF, ld, i, io), qfi = pf(QF, ld, i, io);
        p = p + coeff * (ta * rporii + fk * pfi - (twoc * R[i] + zbci) * qfi);
        m = m + coeff * (tb * rporii - fk * qfi + zbci * pfi);
      }
    }
  }
  red[0][ty][tx] = y;
  red[1][ty][tx] = p;
  red[2][ty][tx] = m;
  __syncthreads();
  if (ty < 3 && i <= n) {
    double v = red[ty][0][tx];
#pragma unroll
    for (int r = 1; r < PF_ROWS; ++r) v += red[ty][r][tx];
    g.out[(size_t)ty * n + i - 1] = ty == 0 ? ZZ[i] - v : v;
  }
}

// SETLAG's quadrature (rmcdhf90/setlag.f90:177-219), one block per pair
// {J, M, case, MTP}: TA(I), I = 2..MTP, from the two orbitals' potentials
// (pot + 3 n slot: YP, XP, XQ, 0-based), then QUAD by one warp. case 0: M
// fixed; 1: J fixed; 2: occupations more than 10 % apart; 3: otherwise.
// QUAD's panels lie in shared memory while they fit what every launch
// has (SH; N <= 24,024), else behind the pair's TA.
template <bool SH>
__global__ void k_setlag_quad(const int4 *__restrict__ pj, const int2 *__restrict__ slots,
                              const double *__restrict__ pot, int n, const double *__restrict__ PF,
                              const double *__restrict__ QF, int ld, const double *__restrict__ R,
                              const double *__restrict__ RP, const double *__restrict__ RPOR, QuadConst q, int np,
                              double *__restrict__ TAall, double *__restrict__ result) {
  extern __shared__ double sm[];
  const int4 w = pj[blockIdx.x];
  const int J = w.x, M = w.y, cs = w.z, mtp = w.w;
  const double *ypj = pot + (size_t)3 * n * slots[blockIdx.x].x, *xpj = ypj + n, *xqj = xpj + n;
  const double *ypm = pot + (size_t)3 * n * slots[blockIdx.x].y, *xpm = ypm + n, *xqm = xpm + n;
  const size_t rec = SH ? (size_t)np : (size_t)np + quad_panels(np);
  double *TA = TAall + (size_t)blockIdx.x * rec, *panel = SH ? sm : TA + np;
  const double C = q.c;
  for (int i = threadIdx.x; i < np; i += blockDim.x) {
    double v = 0.0;
    if (i >= 2 && i <= mtp) {
      const double pj_ = pf(PF, ld, i, J), qj = pf(QF, ld, i, J), pm = pf(PF, ld, i, M), qm = pf(QF, ld, i, M);
      if (cs == 0)
        v = RPOR[i] * ((pm * xqj[i - 1] - qm * xpj[i - 1]) * C + (pm * pj_ + qm * qj) * ypj[i - 1]);
      else if (cs == 1)
        v = RPOR[i] * ((pj_ * xqm[i - 1] - qj * xpm[i - 1]) * C + (pj_ * pm + qj * qm) * ypm[i - 1]);
      else if (cs == 2)
        v = RPOR[i] * ((pm * xqj[i - 1] - qm * xpj[i - 1] - pj_ * xqm[i - 1] + qj * xpm[i - 1]) * C +
                       (ypj[i - 1] - ypm[i - 1]) * (pm * pj_ + qm * qj));
      else
        v = RPOR[i] * ((pm * xqj[i - 1] - qm * xpj[i - 1] + pj_ * xqm[i - 1] - qj * xpm[i - 1]) * C +
                       (ypj[i - 1] + ypm[i - 1]) * (pm * pj_ + qm * qj));
    }
    TA[i] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const double v = quad_warp(TA, panel, mtp, R, RP, q, threadIdx.x);
    if (threadIdx.x == 0) result[blockIdx.x] = v;
  }
}

// ECV from the pair's quadrature and RINTI (setlag.f90:184, 194, 205, 218)
__global__ void k_setlag_final(int np_, const int4 *__restrict__ pj, const double2 *__restrict__ ucf,
                               const double *__restrict__ result, const double *__restrict__ rijm,
                               double *__restrict__ ecv) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= np_) return;
  const double uj = ucf[t].x, um = ucf[t].y;
  switch (pj[t].z) {
    case 0: ecv[t] = (result[t] - rijm[t]) * uj; break;
    case 1: ecv[t] = (result[t] - rijm[t]) * um; break;
    case 2: ecv[t] = result[t] / (1.0 / uj - 1.0 / um); break;
    default: ecv[t] = (result[t] - 2.0 * rijm[t]) / (1.0 / uj + 1.0 / um); break;
  }
}

// RINTI (lib9290/rinti.f90:53-100) for a list of (J, K, place) entries: one block of
// four warps each, the four integrands formed by all threads, one QUAD per warp.
// The integrands and panels lie in shared memory while they fit what
// every launch has (SH; N <= 1,174: GRASP's 590 points take 25 KB), else in
// `work`, rinti_work(np) doubles per block: the same operations
// and bits (I(ab) of 8 subshells: 53 us at 1,174 points, 54 us at 1,175).
constexpr int RINTI_WARPS = 4;
__host__ __device__ constexpr size_t rinti_work(int np) { return (size_t)RINTI_WARPS * (np + quad_panels(np)); }
template <bool SH>
__global__ void __launch_bounds__(32 * RINTI_WARPS) k_rinti(const int4 *__restrict__ jk, int npairs, int mode,
                                                           const double *__restrict__ PF,
                                                           const double *__restrict__ QF, int ld,
                                                           const int *__restrict__ MF, const int *__restrict__ NAK,
                                                           const double *__restrict__ R,
                                                           const double *__restrict__ RP,
                                                           const double *__restrict__ RPOR,
                                                           const double *__restrict__ ZZ, int np, QuadConst q,
                                                           double *work, double *__restrict__ out) {
  extern __shared__ double sm[];
  __shared__ double piece[RINTI_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *TA = SH ? sm : work + blockIdx.x * rinti_work(np);
  double *panel = TA + (size_t)RINTI_WARPS * np + (size_t)warp * quad_panels(np);
  for (int it = blockIdx.x; it < npairs; it += gridDim.x) {
    const int J = jk[it].x, K = jk[it].y;
    const int mtp = max(MF[J], MF[K]);
    const double C = q.c;
    for (int i = threadIdx.x; i < np; i += blockDim.x) {
      double t1 = 0.0, t2 = 0.0, t3 = 0.0, t4 = 0.0;
      if (i >= 2 && i <= mtp) {
        const double pj = pf(PF, ld, i, J), qj = pf(QF, ld, i, J), pk = pf(PF, ld, i, K), qk = pf(QF, ld, i, K);
        double dp = 0.0, dq = 0.0;
        if (i <= q.n) dpbdt_point(PF, QF, ld, K, q, i, dp, dq);
        t1 = qj * dp - pj * dq;
        t2 = RP[i] * qj * qk;
        t3 = RPOR[i] * (pj * qk + qj * pk);
        if (mode == 0) t4 = RPOR[i] * ZZ[i] * (pj * pk + qj * qk);
      }
      TA[i] = t1;
      TA[np + i] = t2;
      TA[2 * np + i] = t3;
      TA[3 * np + i] = t4;
    }
    __syncthreads();
    double v = 0.0;
    if (warp < 3 || mode == 0) v = quad_warp(TA + (size_t)warp * np, panel, mtp, R, RP, q, lane);
    if (lane == 0) {
      if (warp == 0) v = C * v / q.h;
      if (warp == 1) v = -2.0 * C * C * v;
      if (warp == 2) v = v * C * (double)NAK[K];
      if (warp == 3 && mode == 0) v = -v;
      piece[warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) out[jk[it].z] = piece[0] + piece[1] + piece[2] + piece[3];
  }
}

__global__ void k_fill(double *p, size_t n, double v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

bool triangrk(int la, int k, int lb) {  // rci90/triangrk.f90:27-37
  if ((k + la + lb) % 2 != 0) return false;
  if (std::abs(la - lb) > k) return false;
  if (la + lb < k) return false;
  return true;
}

// The same YZK part 2 in three passes for many functions. Each step of
// k_ychain's recurrences adds an increment that does not depend on the
// chain, so the increments are formed by all SMs (k_yincr), the chains run
// only the dependent additions (k_ychain_sum), and Y = Z r^-k + W r^(k+1)
// is assembled per point (k_yassemble). The operations and their order are
// k_ychain's: the functions come out identical.
//   RZ(i) = C1 (T(i-4) + T(i)) + C2 (T(i-3) + T(i-1)) + C3 T(i-2), i >= 5,
//     added to Z as one term (Z = Z + RTMP);
//   RW(i) = the three terms C1 (TW(i) + TW(i+4)), C2 (TW(i+1) + TW(i+3)),
//     C3 TW(i+2), 2 <= i <= MTP, added to W one after the other
//     (WK = ((WK + t1) + t2) + t3, k_ychain's left-to-right sum).
// The chains read RZ up to MTP + 3 and RW up to MTP only.
__global__ void k_yincr(const YDesc *__restrict__ yd, int nf, const int *__restrict__ nfp,
                        const double *__restrict__ TZ, const double *__restrict__ TW, int np, QuadConst q,
                        double *__restrict__ RZ, double *__restrict__ RW) {
  pdl_wait();
  nf = nfuncs(nf, nfp);
  for (int f = blockIdx.y; f < nf; f += gridDim.y) {
    const int MTP = yd[f].mtp;
    const double *T = TZ + (size_t)f * np, *Tw = TW + (size_t)f * np;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= MTP + 3; i += gridDim.x * blockDim.x) {
      double rz = 0.0, w1 = 0.0, w2 = 0.0, w3 = 0.0;
      if (i >= 5) rz = q.C1 * (T[i - 4] + T[i]) + q.C2 * (T[i - 3] + T[i - 1]) + q.C3 * T[i - 2];
      if (i >= 2 && i <= MTP) {
        w1 = q.C1 * (Tw[i] + Tw[i + 4]);
        w2 = q.C2 * (Tw[i + 1] + Tw[i + 3]);
        w3 = q.C3 * Tw[i + 2];
      }
      RZ[(size_t)f * np + i] = rz;
      double *rw = RW + ((size_t)f * np + i) * 3;
      rw[0] = w1;
      rw[1] = w2;
      rw[2] = w3;
    }
  }
}

// acc = acc + P(o_j, 0) + ... + P(o_j, NT-1) (left to right), O(o_j) = acc
// for j = 0 .. cnt-1 in order, o_j = start + step j, P holding NT terms per
// point; the loads of group g + 1 are issued before the additions of group g
template <int NT, int A>
__device__ __forceinline__ double ychain_run(double acc, const double *__restrict__ P, double *__restrict__ O,
                                             int start, int step, int cnt) {
  double cur[A][NT], nxt[A][NT];
#pragma unroll
  for (int u = 0; u < A; ++u)
#pragma unroll
    for (int v = 0; v < NT; ++v) cur[u][v] = (u < cnt) ? P[(size_t)(start + step * u) * NT + v] : 0.0;
  int j = 0;
  for (; j + A <= cnt; j += A) {
    const int j1 = j + A;
#pragma unroll
    for (int u = 0; u < A; ++u)
#pragma unroll
      for (int v = 0; v < NT; ++v) nxt[u][v] = (j1 + u < cnt) ? P[(size_t)(start + step * (j1 + u)) * NT + v] : 0.0;
#pragma unroll
    for (int u = 0; u < A; ++u) {
#pragma unroll
      for (int v = 0; v < NT; ++v) acc = acc + cur[u][v];
      O[start + step * (j + u)] = acc;
    }
#pragma unroll
    for (int u = 0; u < A; ++u)
#pragma unroll
      for (int v = 0; v < NT; ++v) cur[u][v] = nxt[u][v];
  }
#pragma unroll
  for (int u = 0; u < A; ++u)
    if (j + u < cnt) {
#pragma unroll
      for (int v = 0; v < NT; ++v) acc = acc + cur[u][v];
      O[start + step * (j + u)] = acc;
    }
  return acc;
}
// the chains' additions (Z: 16 points loaded ahead, W: 8): blockIdx.y = 0
// writes Z into Y, each chain's K = 0 correction DIF and the function's
// asymptotic value ZKLIM, blockIdx.y = 1 writes W into W
__global__ void k_ychain_sum(const YDesc *__restrict__ yd, int nf, const int *__restrict__ nfp,
                             const double *__restrict__ TZ, const double *__restrict__ RZ,
                             const double *__restrict__ RW, int np, QuadConst q, double *__restrict__ Y,
                             double *__restrict__ W, double *__restrict__ dif_out, double *__restrict__ zk_out) {
  pdl_wait();
  nf = nfuncs(nf, nfp);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int f = t >> 2, c = t & 3;
  const bool active = f < nf;
  const YDesc y = active ? yd[f] : yd[0];
  const int K = y.k, MTP = y.mtp, MTPP3 = MTP + 3, N = q.n;
  const size_t base = (size_t)(active ? f : 0) * np;
  const int s = c + 2;  // chain start: 2, 3, 4, 5
  if (blockIdx.y == 1) {
    // W from the top of this chain's points with i <= min(N, MTP) down to s
    const int lim = min(N, MTP);
    if (!active || lim < s) return;
    const int cnt = (lim - s) / 4 + 1;  // the points s + 4 (cnt - 1), ..., s + 4, s
    ychain_run<3, 8>(0.0, RW + 3 * base, W + base, s + 4 * (cnt - 1), -4, cnt);
    return;
  }
  const double *T = TZ + base, *Rz = RZ + base;
  double *Yf = Y + base;
  double z = 0.0;
  if (active) {
    if (s <= 4) {
      double sum = 0.0;
      for (int kk = 2; kk <= 5; ++kk) sum = sum + q.CNC5C[kk - 2][s - 2] * T[kk];
      z = sum;
    } else {  // ZK(5) = ZK(1) + RTMP(5), ZK(1) = 0
      z = 0.0 + Rz[5];
    }
    Yf[s] = z;
    // the points s + 4, s + 8, ... <= MTP + 3
    const int cnt = (MTPP3 >= s + 4) ? (MTPP3 - s - 4) / 4 + 1 : 0;
    z = ychain_run<1, 16>(z, Rz, Yf, s + 4, 4, cnt);
  }
  const int owner = (MTPP3 - 2) & 3;
  const double z_top = __shfl_sync(0xffffffffu, z, (threadIdx.x & ~3) + owner);
  if (!active) return;
  double zklim, dif = 0.0;
  if (K == 0) {
    zklim = (y.b == y.d) ? 1.0 : 0.0;
    const double d0 = z - zklim;
    if (fabs(d0) > q.accy) dif = d0;
  } else {
    zklim = z_top;
  }
  dif_out[(size_t)f * 4 + c] = dif;
  if (c == 0) zk_out[f] = zklim;
}

__global__ void k_yassemble(const YDesc *__restrict__ yd, int nf, const int *__restrict__ nfp,
                            const double *__restrict__ R, const double *__restrict__ pw, int np, QuadConst q,
                            const double *__restrict__ dif, const double *__restrict__ zk,
                            const double *__restrict__ W, double *__restrict__ Y) {
  pdl_wait();
  nf = nfuncs(nf, nfp);
  for (int f = blockIdx.y; f < nf; f += gridDim.y) {
    const YDesc y = yd[f];
    const int K = y.k, MTP = y.mtp, MTPP3 = MTP + 3, N = q.n;
    const double zklim = zk[f];
    const double *RTTKM = pw + (size_t)(1 * (KLIMIT + 1) + K) * np;
    const double *RTTK1 = pw + (size_t)(2 * (KLIMIT + 1) + K) * np;
    const double *Wf = W + (size_t)f * np;
    double *Yf = Y + (size_t)f * np;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
      double yv = 0.0;
      if (i >= 2 && i <= N) {
        double zf;
        if (K == 0) {
          if (i <= MTPP3) {
            const double d = dif[(size_t)f * 4 + ((i - 2) & 3)];
            zf = (d != 0.0) ? Yf[i] - d : Yf[i];
          } else {
            zf = zklim;
          }
        } else {
          zf = (i <= MTPP3) ? Yf[i] * RTTKM[i] : zklim * RTTKM[i];
        }
        double wkf = 0.0;
        if (i <= MTP) {
          const double wk = Wf[i];
          wkf = (K == 0) ? wk * R[i] : wk * RTTK1[i];
        }
        yv = zf + wkf;
        if (i > y.mtpb) yv = 0.0;
      }
      Yf[i] = yv;
    }
  }
}

// build_y takes the three-pass form from this many functions on
constexpr int YSPLIT_MIN = 32;

// Builds Y functions for the descriptor list on the device: TZ/TW scratch
// then the chains. Y must hold nf * np doubles. nfp (may be null): the number
// of functions on the device, at most nf.
int build_y(gg_ctx *ctx, const YDesc *d_yd, int nf, double *dY, DBuf<double> &scratch, const int *nfp = nullptr) {
  Grid &g = ctx->grid;
  Orbitals &o = ctx->orb;
  const int np = g.np;
  const bool split = nf >= YSPLIT_MIN;
  GG_TRY(scratch.alloc(split ? (size_t)6 * nf * np + (size_t)5 * nf : (size_t)2 * nf * np));
  double *TZ = scratch.p, *TW = scratch.p + (size_t)nf * np;
  dim3 grid1((np + 127) / 128, std::min(nf, nfp ? 4 * ctx->sms : 65535));
  k_ytemp<<<grid1, 128, 0, ctx->stream>>>(d_yd, nf, nfp, o.dPF.p, o.dQF.p, o.ld, g.dRP.p, g.dPow.p, np, TZ, TW);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  const int nthr = nf * 4;
  if (!split) {
    GG_CUDA(cudaMemsetAsync(dY, 0, (size_t)nf * np * sizeof(double), ctx->stream));
    k_ychain<<<(nthr + 127) / 128, 128, 0, ctx->stream>>>(d_yd, nf, nfp, TZ, TW, g.dR.p, g.dPow.p, np, g.q, dY);
    ::gg::note_launch();
  } else {
    // RZ: one term per point; RW: three terms per point; DIF per chain; ZKLIM
    double *RZ = TW + (size_t)nf * np, *RW = RZ + (size_t)nf * np, *dif = RW + (size_t)3 * nf * np;
    double *zk = dif + 4 * nf;
    GG_CUDA(launch_pdl(k_yincr, grid1, 128, 0, ctx->stream, d_yd, nf, nfp, TZ, TW, np, g.q, RZ, RW));
    // W goes where TW was: k_yincr was its last reader
    GG_CUDA(launch_pdl(k_ychain_sum, dim3((nthr + 63) / 64, 2), 64, 0, ctx->stream, d_yd, nf, nfp, TZ, RZ, RW, np, g.q,
                       dY, TW, dif, zk));
    GG_CUDA(launch_pdl(k_yassemble, grid1, 128, 0, ctx->stream, d_yd, nf, nfp, g.dR.p, g.dPow.p, np, g.q, dif, zk, TW,
                       dY));
    ::gg::note_launch();
    ::gg::note_launch();
    ::gg::note_launch();
  }
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

// The Y functions of a potential call, a block per function from densities to
// Y with everything in between in shared memory: warp 0 runs the Z chains,
// warp 1 the W chains, each lane a run of up to YF_P points with its four
// chains' sums in registers; a scan over the lanes joins the runs. The sums
// are regrouped (YZK adds along a chain point by point), so R^k, whose values
// MANEIG's vectors follow to the last bit, keeps the passes above. Bound: the
// FP64 pipe, 20 instructions per 32 points. (COFPOT of 34 subshells: the four
// kernels above took 63 us per orbital, 15 us of it W's chain of 3 x 148
// dependent additions; this one 26.)
constexpr int YF_P = 20;       // points of a lane's run at most, a multiple of 4
constexpr int YF_MAXN = 2560;  // longer grids don't fit 48 KB of shared memory
__host__ __device__ __forceinline__ int yf_at(int i) { return i + (i >> 4); }  // spreads the lanes' runs over the banks
constexpr int YF_SLACK = YF_P + 8;  // zeros above MTP that the windows read
__global__ void __launch_bounds__(64) k_yfun(const YDesc *__restrict__ yd, int nf, const int *__restrict__ nfp,
                                             const double *__restrict__ PF, const double *__restrict__ QF, int ld,
                                             const double *__restrict__ R, const double *__restrict__ RP,
                                             const double *__restrict__ pw, int np, QuadConst q,
                                             double *__restrict__ Y) {
  pdl_wait();
  extern __shared__ double ysh[];
  __shared__ double zfin[4];  // the Z chains' last values
  double *TZ = ysh, *TW = ysh + yf_at(np + YF_SLACK);
  const int tid = threadIdx.x, lane = tid & 31, N = q.n;
  nf = nfuncs(nf, nfp);
  for (int f = blockIdx.x; f < nf; f += gridDim.x) {
    const YDesc y = yd[f];
    const int K = y.k, MTP = y.mtp, top = MTP + 3;
    {
      const double *TK = K ? pw + (size_t)K * np : nullptr;
      const double *TM = K ? pw + (size_t)(3 * (KLIMIT + 1) + K) * np : pw;
      for (int i = tid; i < MTP + YF_SLACK; i += 64) {
        double tz = 0.0, tw = 0.0;
        if (i >= 2 && i <= MTP) {
          const double rhop =
              RP[i] * (pf(PF, ld, i, y.b) * pf(PF, ld, i, y.d) + pf(QF, ld, i, y.b) * pf(QF, ld, i, y.d));
          tz = K ? TK[i] * rhop : rhop;
          tw = rhop * TM[i];
        }
        TZ[yf_at(i)] = tz;
        TW[yf_at(i)] = tw;
      }
    }
    __syncthreads();
    // runs of P points, 32 P to a pass; point i is on chain (i - 2) & 3, and a
    // run starts on chain 0
    const int P = min(YF_P, (top - 1 + 127) / 128 * 4), npass = (top - 1 + 32 * P - 1) / (32 * P);
    double v[YF_P], acc[4], ex[4], h1 = 0.0, h2 = 0.0, h3 = 0.0, h4 = 0.0;  // h: the neighbouring pass's temps
    double carry[4] = {0.0, 0.0, 0.0, 0.0};
    if (tid < 32) {
      // Z(2), Z(3), Z(4) from the five-point start formulas
      double st = 0.0;
      for (int kk = 2; kk <= 5; ++kk) st = fma(q.CNC5C[kk - 2][min(lane, 2)], TZ[yf_at(kk)], st);
      const double st0 = __shfl_sync(0xffffffffu, st, 0), st1 = __shfl_sync(0xffffffffu, st, 1),
                   st2 = __shfl_sync(0xffffffffu, st, 2);
      for (int p = 0; p < npass; ++p) {
        const int b = 2 + p * 32 * P, i0 = b + lane * P;
        const bool in = i0 <= top;
        double t1 = h1, t2 = h2, t3 = h3, t4 = h4;  // T(i - 1) ... T(i - 4)
        if (lane && in) {
          t1 = TZ[yf_at(i0 - 1)];
          t2 = TZ[yf_at(i0 - 2)];
          t3 = TZ[yf_at(i0 - 3)];
          t4 = TZ[yf_at(i0 - 4)];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = lane ? 0.0 : carry[c];
#pragma unroll
        for (int j = 0; j < YF_P; ++j) {
          if (j >= P) break;
          const int i = i0 + j;
          if (i <= top) {
            const double t0 = TZ[yf_at(i)];
            acc[j & 3] = fma(q.C3, t2, fma(q.C2, t3 + t1, fma(q.C1, t4 + t0, acc[j & 3])));
            t4 = t3;
            t3 = t2;
            t2 = t1;
            t1 = t0;
          }
          if (j < 3 && i < 5) acc[j] = j == 0 ? st0 : j == 1 ? st1 : st2;
          v[j] = acc[j & 3];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          double s = acc[c];
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const double u = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += u;
          }
          ex[c] = __shfl_up_sync(0xffffffffu, s, 1);
          if (lane == 0) ex[c] = 0.0;
          carry[c] = __shfl_sync(0xffffffffu, s, 31);
        }
        const int e = b + 32 * P;  // the next pass's first point
        if (e <= top) {
          h1 = TZ[yf_at(e - 1)];
          h2 = TZ[yf_at(e - 2)];
          h3 = TZ[yf_at(e - 3)];
          h4 = TZ[yf_at(e - 4)];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < YF_P; ++j) {
          if (j >= P) break;
          if (i0 + j <= top) TZ[yf_at(i0 + j)] = v[j] + ex[j & 3];
        }
        __syncwarp();
      }
      if (lane < 4) zfin[lane] = lane == 0 ? carry[0] : lane == 1 ? carry[1] : lane == 2 ? carry[2] : carry[3];
    } else {
      const int lim = min(N, MTP);
      for (int p = npass - 1; p >= 0; --p) {
        const int b = 2 + p * 32 * P, i0 = b + lane * P;
        const bool in = i0 <= lim;
        double t1 = h1, t2 = h2, t3 = h3, t4 = h4;  // TW(i + 1) ... TW(i + 4)
        if (lane < 31 || p == npass - 1) {
          t1 = in ? TW[yf_at(i0 + P)] : 0.0;
          t2 = in ? TW[yf_at(i0 + P + 1)] : 0.0;
          t3 = in ? TW[yf_at(i0 + P + 2)] : 0.0;
          t4 = in ? TW[yf_at(i0 + P + 3)] : 0.0;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = lane < 31 ? 0.0 : carry[c];
#pragma unroll
        for (int j = YF_P - 1; j >= 0; --j) {
          if (j >= P) continue;
          const int i = i0 + j;
          if (in) {
            const double t0 = TW[yf_at(i)];
            if (i <= lim) acc[j & 3] = fma(q.C3, t2, fma(q.C2, t1 + t3, fma(q.C1, t0 + t4, acc[j & 3])));
            t4 = t3;
            t3 = t2;
            t2 = t1;
            t1 = t0;
          }
          v[j] = acc[j & 3];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          double s = acc[c];
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const double u = __shfl_down_sync(0xffffffffu, s, o);
            if (lane + o < 32) s += u;
          }
          ex[c] = __shfl_down_sync(0xffffffffu, s, 1);
          if (lane == 31) ex[c] = 0.0;
          carry[c] = __shfl_sync(0xffffffffu, s, 0);
        }
        h1 = TW[yf_at(b)];
        h2 = TW[yf_at(b + 1)];
        h3 = TW[yf_at(b + 2)];
        h4 = TW[yf_at(b + 3)];
        __syncwarp();
#pragma unroll
        for (int j = 0; j < YF_P; ++j) {
          if (j >= P) break;
          if (i0 + j <= lim) TW[yf_at(i0 + j)] = v[j] + ex[j & 3];
        }
        __syncwarp();
      }
    }
    __syncthreads();
    // Y = Z r^-k + W r^(k+1); above MTP + 3 Z keeps its asymptotic value
    // (yzk.f90:150-171), k = 0: the chains are shifted to end on it
    const double *RTTKM = pw + (size_t)(1 * (KLIMIT + 1) + K) * np;
    const double *RTTK1 = pw + (size_t)(2 * (KLIMIT + 1) + K) * np;
    const double zklim = K ? zfin[(top - 2) & 3] : (y.b == y.d ? 1.0 : 0.0);
    double dif = 0.0;  // this thread's points are all on one chain: 64 is a multiple of 4
    if (K == 0) {
      const double d0 = zfin[(tid - 2) & 3] - zklim;
      if (fabs(d0) > q.accy) dif = d0;
    }
    double *Yf = Y + (size_t)f * np;
    for (int i = tid; i < np; i += 64) {
      double yv = 0.0;
      if (i >= 2 && i <= N && i <= y.mtpb) {
        if (K == 0) {
          yv = i <= top ? TZ[yf_at(i)] - dif : zklim;
          if (i <= MTP) yv = fma(TW[yf_at(i)], R[i], yv);
        } else {
          yv = (i <= top ? TZ[yf_at(i)] : zklim) * RTTKM[i];
          if (i <= MTP) yv = fma(TW[yf_at(i)], RTTK1[i], yv);
        }
      }
      Yf[i] = yv;
    }
    __syncthreads();
  }
}

// The Y functions of a potential call: nfp (on the device) of them, at most nf
int build_y_pot(gg_ctx *ctx, const YDesc *d_yd, int nf, double *dY, DBuf<double> &scratch, const int *nfp) {
  Grid &g = ctx->grid;
  Orbitals &o = ctx->orb;
  if (g.q.n > YF_MAXN) return build_y(ctx, d_yd, nf, dY, scratch, nfp);
  const size_t smem = 2 * sizeof(double) * yf_at(g.np + YF_SLACK);
  GG_CUDA(launch_pdl(k_yfun, std::min(nf, 32 * ctx->sms), 64, smem, ctx->stream, d_yd, nf, nfp, o.dPF.p, o.dQF.p, o.ld,
                     g.dR.p, g.dRP.p, g.dPow.p, g.np, g.q, dY));
  ::gg::note_launch();
  return GG_OK;
}

template <class T> int upload(DBuf<T> &b, const std::vector<T> &h, cudaStream_t s) {
  GG_TRY(b.alloc(h.size()));
  if (!h.empty()) GG_CUDA(cudaMemcpyAsync(b.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s));
  return GG_OK;
}

}  // namespace

}  // namespace gg

using namespace gg;

extern "C" {

// The part of GENINTRK that depends only on the orbitals' l and j and on
// kmax: Y functions, pairs, INDTEIRK and KSTART, the contraction tiles of
// both forms, and their device copies. Built once per orbital set.
static int rk_build_structure(gg_ctx *ctx, int kloop, RkCache &C) {
  Grid &g = ctx->grid;
  Orbitals &o = ctx->orb;
  RkTable &rk = ctx->rk;
  const int NW = o.nw, KEY = NW + 1;
  // Y functions, ordered (k, b, d): D(b,k) = {d >= b : TRIANGRK(l_b, k, l_d)}
  std::vector<YDesc> &yd = C.yd;
  yd.clear();
  std::vector<std::vector<int>> cs(kloop + 1, std::vector<int>(NW + 2, -1)), nd(kloop + 1, std::vector<int>(NW + 2, 0));
  std::vector<int> &kend = C.kend;
  kend.assign(kloop + 1, 0);
  for (int k = 0; k <= kloop; ++k) {
    for (int b = 1; b <= NW; ++b) {
      cs[k][b] = (int)yd.size();
      for (int d = b; d <= NW; ++d)
        if (triangrk(o.nkl[b], k, o.nkl[d])) {
          YDesc y;
          y.k = k;
          y.b = b;
          y.d = d;
          y.mtp = std::min(o.mf[b], o.mf[d]);
          y.mtpb = (k == 0 && b == d) ? g.n : y.mtp;
          y.cs = cs[k][b];
          y.nd = 0;
          yd.push_back(y);
        }
      nd[k][b] = (int)yd.size() - cs[k][b];
      for (int f = cs[k][b]; f < (int)yd.size(); ++f) yd[f].nd = nd[k][b];
    }
    kend[k] = (int)yd.size();
  }
  // pair list for the A rows (a <= c), k-independent
  std::vector<int2> &pairs = C.pairs;
  pairs.clear();
  std::vector<int> pidx((size_t)(NW + 1) * (NW + 1), -1);
  for (int a = 1; a <= NW; ++a)
    for (int c = a; c <= NW; ++c) {
      pidx[(size_t)a * (NW + 1) + c] = (int)pairs.size();
      pairs.push_back(make_int2(a, c));
    }
  // INDTEIRK and KSTART in GENINTRK order (rci90/genintrk.f90:64-86) and the
  // contraction problems (k, a); each problem's entries are contiguous.
  rk.kstart.assign(kloop + 2, 0);
  rk.hInd.clear();
  std::vector<RkTile> &tiles = C.tiles;
  std::vector<TcRow> &tcrows = C.tcrows;
  tiles.clear();
  tcrows.clear();
  std::vector<int> tcr0(kloop + 2, 0);  // first tcrows entry of each k
  int64_t N = 0;
  rk.kstart[0] = 1;
  for (int k = 0; k <= kloop; ++k) {
    tcr0[k] = (int)tcrows.size();
    for (int a = 1; a <= NW; ++a) {
      const int ncA = nd[k][a];
      if (ncA == 0) continue;
      const int c0 = cs[k][a];
      const long long base = N;
      // integer index list in reference order
      for (int b = a; b <= NW; ++b)
        for (int ic = 0; ic < ncA; ++ic) {
          const int c = yd[cs[k][a] + ic].d;
          for (int id = 0; id < nd[k][b]; ++id) {
            const int d = yd[cs[k][b] + id].d;
            rk.hInd.push_back(((a * KEY + b) * KEY + c) * KEY + d);
          }
        }
      N = (int64_t)rk.hInd.size();
      // the contraction's rows (all problems of one k, in order)
      for (int ic = 0; ic < ncA; ++ic) {
        const int c = yd[cs[k][a] + ic].d;
        tcrows.push_back(TcRow{pidx[(size_t)a * (NW + 1) + c], a, c, ic, ncA, c0, base});
      }
    }
    rk.kstart[k + 1] = (int32_t)(N + 1);
  }
  tcr0[kloop + 1] = (int)tcrows.size();
  // the FP64 form's tiles; the rows are ordered by a, so a tile's first row
  // has its smallest cs_a
  for (C.nr = 8;; C.nr /= 2) {
    tiles.clear();
    for (int k = 0; k <= kloop; ++k)
      for (int r = tcr0[k]; r < tcr0[k + 1]; r += C.nr)
        for (int f = tcrows[r].cs_a; f < kend[k]; f += 32)
          tiles.push_back(RkTile{r, std::min(C.nr, tcr0[k + 1] - r), f, std::min(32, kend[k] - f)});
    if (C.nr == 1 || (int)tiles.size() >= 4 * ctx->sms) break;
  }
  if (N > INT32_MAX) return fail(GG_ERR_RANGE, "genintrk: table too large");
  rk.n = N;
  C.nf = (int)yd.size();
  C.npairs = (int)pairs.size();
  const int nf = C.nf;
  {
  std::vector<int> fg0(kloop + 1), pg0(kloop + 1), kbeg(kloop + 1);
  std::vector<int> &yslot = C.yslot, &aslot = C.aslot;
  std::vector<TcTile> &tct = C.tct;
  yslot.clear();
  aslot.clear();
  tct.clear();
  C.tcs_nch = -1;  // the split-K list follows tct
  for (int k = 0; k <= kloop; ++k) {
    kbeg[k] = (k == 0) ? 0 : kend[k - 1];
    const int F = kend[k] - kbeg[k], Rk = tcr0[k + 1] - tcr0[k];
    const int nft = (F + TC_M - 1) / TC_M, npt = (Rk + TC_N - 1) / TC_N;
    fg0[k] = (int)(yslot.size() / TC_M);
    pg0[k] = (int)(aslot.size() / TC_N);
    for (int ft = 0; ft < nft; ++ft)
      for (int m = 0; m < TC_M; ++m) {
        const int f = kbeg[k] + ft * TC_M + m;
        yslot.push_back(f < kend[k] ? f : -1);
      }
    for (int pt = 0; pt < npt; ++pt)
      for (int n = 0; n < TC_N; ++n) {
        const int r = tcr0[k] + pt * TC_N + n;
        aslot.push_back(r < tcr0[k + 1] ? tcrows[r].p : -1);
      }
    for (int pt = 0; pt < npt; ++pt)
      for (int ft = 0; ft < nft; ++ft) {
        TcTile t;
        t.k = k;
        t.fg = fg0[k] + ft;
        t.pg = pg0[k] + pt;
        t.f0 = kbeg[k] + ft * TC_M;
        t.fn = std::min(TC_M, F - ft * TC_M);
        t.r0 = tcr0[k] + pt * TC_N;
        t.rn = std::min(TC_N, Rk - pt * TC_N);
        // rows are ordered by a, so the first row has the smallest cs_a:
        // no needed entry when every function of the tile is below it
        if (t.f0 + t.fn - 1 < tcrows[t.r0].cs_a) continue;
        tct.push_back(t);
      }
  }
    std::vector<int> &fidx = C.fidx;
    fidx.assign((size_t)(kloop + 1) * KEY * KEY, -1);
    for (int f = 0; f < nf; ++f) fidx[((size_t)yd[f].k * KEY + yd[f].b) * KEY + yd[f].d] = f;
  }
  GG_TRY(upload(C.dPairs, pairs, ctx->stream));
  GG_TRY(upload(C.dTiles, tiles, ctx->stream));
  GG_TRY(upload(C.dTct, C.tct, ctx->stream));
  GG_TRY(upload(C.dTcr, tcrows, ctx->stream));
  GG_TRY(upload(C.dYslot, C.yslot, ctx->stream));
  GG_TRY(upload(C.dAslot, C.aslot, ctx->stream));
  GG_TRY(upload(C.dFidx, C.fidx, ctx->stream));
  GG_TRY(upload(C.dPidx, pidx, ctx->stream));
  GG_TRY(upload(C.dKst, rk.kstart, ctx->stream));
  GG_TRY(rk.dInd.alloc(std::max<int64_t>(N, 1)));
  if (N > 0)
    GG_CUDA(cudaMemcpyAsync(rk.dInd.p, rk.hInd.data(), N * sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream));
  GG_CUDA(cudaStreamSynchronize(ctx->stream));
  return GG_OK;
}

int gg_genintrk(gg_ctx *ctx, int kmax, int precision, int64_t *n_out, int *j2max_out) {
  GG_TRY(ensure_orbitals(ctx));
  if (precision != GG_FP64 && precision != GG_SPLIT) return fail(GG_ERR_ARG, "gg_genintrk: unknown precision");
  GG_CUDA(cudaSetDevice(ctx->device));
  Grid &g = ctx->grid;
  Orbitals &o = ctx->orb;
  RkTable &rk = ctx->rk;
  const int NW = o.nw, KEY = NW + 1;
  int j2max = o.nkj[1];
  for (int i = 2; i <= NW; ++i) j2max = std::max(j2max, o.nkj[i]);
  if (j2max > KLIMIT) return fail(GG_ERR_ARG, "genintrk: KMAX too small");
  const int kloop = kmax < 0 ? j2max : kmax;
  if (kloop > KLIMIT) return fail(GG_ERR_ARG, "genintrk: k beyond KLIMIT = 20");
  GG_TRY(timer_start(ctx));
  // the index structure is rebuilt only when the orbital set's l, j or kmax change
  std::vector<int> key{NW, kloop};
  for (int i = 1; i <= NW; ++i) {
    key.push_back(o.nkl[i]);
    key.push_back(o.nkj[i]);
  }
  if (!rk.cache) rk.cache = new RkCache();
  RkCache &C = *rk.cache;
  if (C.key != key) {
    C.key.clear();  // not valid until built
    rk.valid = false;
    GG_TRY(rk_build_structure(ctx, kloop, C));
    C.key = key;
  }
  const int64_t N = rk.n;
  rk.valid = false;  // until this call's table is complete
  rk.kloop = kloop;
  rk.j2max = j2max;
  // per call: each Y function's MTP from the current orbital extents
  for (YDesc &y : C.yd) {
    y.mtp = std::min(o.mf[y.b], o.mf[y.d]);
    y.mtpb = (y.k == 0 && y.b == y.d) ? g.n : y.mtp;
  }
  GG_TRY(upload(C.dYd, C.yd, ctx->stream));
  const int nf = C.nf, npairs = C.npairs;
  const int np = g.np;
  const int KC = ((g.n + 1 + KC_TILE - 1) / KC_TILE) * KC_TILE;
  if (KC > np) return fail(GG_ERR_ARG, "genintrk: grid padding too small");
  const std::vector<RkTile> &tiles = C.tiles;
  GG_TRY(rk.dVal.alloc(std::max<int64_t>(N, 1)));
  GG_TRY(C.dY.alloc((size_t)std::max(nf, 1) * np));
  if (nf > 0) GG_TRY(build_y(ctx, C.dYd.p, nf, C.dY.p, C.scratch));
  GG_TRY(C.dA.alloc((size_t)std::max(npairs, 1) * KC + KC_TILE));
  GG_TRY(C.dD.alloc((size_t)std::max(npairs, 1) * KC + KC_TILE));
  if (npairs > 0) {
    dim3 gr((KC + 127) / 128, npairs);
    GG_CUDA(launch_pdl(k_apairs, gr, 128, 0, ctx->stream, C.dPairs.p, npairs, o.dPF.p, o.dQF.p, o.ld, o.dMF.p,
                       g.dRPOR.p, KC, g.q, C.dA.p, C.dD.p));
    ::gg::note_launch();
    GG_CUDA(cudaGetLastError());
  }
  const RkTabs tabs{C.dD.p, C.dY.p, C.dYd.p, o.dMF.p, g.dHead.p, KC, np};
  GG_TRY(C.dFb.alloc(std::max<int64_t>(N, 1)));
  GG_TRY(C.dNfb.alloc(3));  // [0] fallback count, [1] position error flag, [2] tensor-core wait timed out
  GG_CUDA(cudaMemsetAsync(C.dNfb.p, 0, 3 * sizeof(int), ctx->stream));
  if (!tiles.empty() && precision == GG_SPLIT) {
    // tensor-core contraction on Ozaki slices of A and Y
    const int KP = (KC + 31) / 32 * 32;
    GG_TRY(C.dEA.alloc(npairs + 1));
    GG_TRY(C.dEY.alloc(nf + 1));
    {
      // tcgen05: the slices written into the tile blocks, the raw GEMM parts
      // at their positions, then the head terms
      const int nch = KP / TC_KC;
      GG_TRY(C.dYt.alloc(std::max<size_t>(1, C.yslot.size() / TC_M * nch * TC_YBLK)));
      GG_TRY(C.dAt.alloc(std::max<size_t>(1, C.aslot.size() / TC_N * nch * TC_ABLK)));
      if (!C.yslot.empty()) {
        GG_CUDA(launch_pdl(k_oz_tile<TC_M>, (unsigned)C.yslot.size() / 8, OZ_T, 0, ctx->stream, C.dY.p, np, KC, nch,
                           C.dYslot.p, C.dEY.p, C.dYt.p));
        ::gg::note_launch();
      }
      if (!C.aslot.empty()) {
        GG_CUDA(launch_pdl(k_oz_tile<TC_N>, (unsigned)C.aslot.size() / 8, OZ_T, 0, ctx->stream, C.dA.p, KC, KC, nch,
                           C.dAslot.p, C.dEA.p, C.dAt.p));
        ::gg::note_launch();
      }
      // (on every call: the attribute is the current device's)
      GG_CUDA(cudaFuncSetAttribute(k_rk_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
      // split-K: one CTA per SM holds a tile (shared memory), so with
      // fewer tiles than SMs each tile's grid chunks are cut into nsplit
      // ranges of at least TC_FLUSH chunks, whose partial sums
      // k_rk_finish_all adds in order
      int nsplit = 1;
      if (!C.tct.empty()) {
        const int want = (ctx->sms + (int)C.tct.size() - 1) / (int)C.tct.size();
        nsplit = std::max(1, std::min(want, nch / TC_FLUSH));
      }
      if (C.tcs_nch != nch || C.tcs_split != nsplit) {
        C.tcs.clear();
        for (const TcTile &t : C.tct)
          for (int sp = 0; sp < nsplit; ++sp) {
            TcTile u = t;
            u.c0 = (int)((long long)nch * sp / nsplit);
            u.c1 = (int)((long long)nch * (sp + 1) / nsplit);
            u.s = sp;
            C.tcs.push_back(u);
          }
        GG_TRY(upload(C.dTcs, C.tcs, ctx->stream));
        C.tcs_nch = nch;
        C.tcs_split = nsplit;
      }
      double *parts = rk.dVal.p;
      if (nsplit > 1) {
        GG_TRY(C.dParts.alloc((size_t)nsplit * std::max<int64_t>(N, 1)));
        parts = C.dParts.p;
      }
      if (!C.tcs.empty()) {
        GG_CUDA(launch_pdl(k_rk_tc, (unsigned)std::min<size_t>(C.tcs.size(), ctx->sms), TC_THREADS, TC_SMEM,
                           ctx->stream, C.dTcs.p, (int)C.tcs.size(), C.dTcr.p, C.dYt.p, C.dAt.p, nch, C.dEA.p,
                           C.dEY.p, C.dYd.p, parts, (long long)N, C.dNfb.p + 1, ctx->test_stall_tile));
        ctx->test_stall_tile = -1;  // one call only
        ::gg::note_launch();
      }
      ctx->stats[25] = nsplit;
      GG_CUDA(cudaGetLastError());
      const unsigned fb_blocks = (unsigned)std::min<long long>((N + 255) / 256, 8LL * ctx->sms);
      GG_CUDA(launch_pdl(k_rk_finish_all, std::max(1u, fb_blocks), 256, 0, ctx->stream, rk.dInd.p, (long long)N,
                         C.dKst.p, kloop, KEY, C.dFidx.p, C.dPidx.p, tabs, g.q, rk.dVal.p, C.dFb.p, C.dNfb.p, parts,
                         nsplit));
      ::gg::note_launch();
    }
    GG_CUDA(cudaGetLastError());
  } else if (!tiles.empty()) {
    auto dot = C.nr == 8 ? k_rk_dot<8> : C.nr == 4 ? k_rk_dot<4> : C.nr == 2 ? k_rk_dot<2> : k_rk_dot<1>;
    GG_CUDA(launch_pdl(dot, (unsigned)((tiles.size() + 3) / 4), 128, 0, ctx->stream, C.dTiles.p, (int)tiles.size(),
                       C.dTcr.p, C.dA.p, tabs, g.q, rk.dVal.p, (long long)N, C.dFb.p, C.dNfb.p));
    ::gg::note_launch();
    GG_CUDA(cudaGetLastError());
  }
  if (!tiles.empty()) {
    // the items' number stays on the device: the blocks take it from there
    const int wpb = 16;  // warps per block: an item each, their head terms by warp 0
    const int blocks = (int)std::min<int64_t>((N + wpb - 1) / wpb, 4LL * ctx->sms);
    GG_CUDA(launch_pdl(k_quad_table, std::max(1, blocks), 32 * wpb, 0, ctx->stream, C.dFb.p, C.dNfb.p, (int)N, tabs,
                       g.q, rk.dVal.p));
    ::gg::note_launch();
    GG_CUDA(cudaGetLastError());
  }
  int hfb[3] = {0, 0, 0};
  GG_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
  GG_CUDA(cudaMemcpyAsync(hfb, C.dNfb.p, 3 * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  GG_CUDA(cudaStreamSynchronize(ctx->stream));
  double ms = 0;
  GG_TRY(timer_read(ctx, &ms));
  ctx->stats[0] = ms;
  if (hfb[1]) return fail(GG_ERR_STATE, "genintrk: contraction produced a table position out of range");
  if (hfb[2] == 1)
    return fail(GG_ERR_TIMEOUT, "genintrk: a tensor-core tile timed out waiting for its copies or MMAs (drained; "
                                "the table is not valid)");
  if (hfb[2] > 1)
    return fail(GG_ERR_TIMEOUT, "genintrk: a tensor-core tile timed out and its copies or MMAs did not drain");
  ctx->stats[20] = hfb[0];
  rk.valid = true;
  if (n_out) *n_out = N;
  if (j2max_out) *j2max_out = j2max;
  return GG_OK;
}

int gg_get_rk_table(gg_ctx *ctx, int32_t *indteirk, double *valteirk, int32_t *kstart) {
  if (!ctx || !ctx->rk.valid) return fail(GG_ERR_STATE, "gg_get_rk_table: no table (call gg_genintrk)");
  GG_CUDA(cudaSetDevice(ctx->device));
  const RkTable &rk = ctx->rk;
  if (indteirk && rk.n) std::memcpy(indteirk, rk.hInd.data(), rk.n * sizeof(int32_t));
  if (valteirk && rk.n) {
    GG_CUDA(cudaMemcpyAsync(valteirk, rk.dVal.p, rk.n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    GG_CUDA(cudaStreamSynchronize(ctx->stream));
  }
  if (kstart) std::memcpy(kstart, rk.kstart.data(), rk.kstart.size() * sizeof(int32_t));
  return GG_OK;
}

int gg_rkintc(gg_ctx *ctx, int ia, int ib, int ic, int id, int k, double *tegral) {
  if (!ctx || !ctx->rk.valid) return fail(GG_ERR_STATE, "gg_rkintc: no table");
  const RkTable &rk = ctx->rk;
  const int nw = ctx->orb.nw, KEY = nw + 1;
  if (k < 0 || k > rk.kloop || ia < 1 || ib < 1 || ic < 1 || id < 1 || ia > nw || ib > nw || ic > nw || id > nw)
    return fail(GG_ERR_ARG, "gg_rkintc: index out of range");
  // canonical order (rci90/rkintc.f90:45-62)
  if (ia > ic) std::swap(ia, ic);
  if (ib > id) std::swap(ib, id);
  if (ia > ib) {
    std::swap(ia, ib);
    std::swap(ic, id);
  }
  const int32_t index = ((ia * KEY + ib) * KEY + ic) * KEY + id;
  int64_t jl = rk.kstart[k], ju = rk.kstart[k + 1] - 1;
  if (ju < jl || index < rk.hInd[jl - 1] || index > rk.hInd[ju - 1])
    return fail(GG_ERR_NOTFOUND, "Something wrong in rkintc");
  while (ju - jl > 1) {
    const int64_t jm = (ju + jl) / 2;
    if (rk.hInd[jm - 1] > index)
      ju = jm;
    else
      jl = jm;
  }
  int64_t loc;
  if (index == rk.hInd[ju - 1])
    loc = ju;
  else if (index == rk.hInd[jl - 1])
    loc = jl;
  else
    return fail(GG_ERR_NOTFOUND, "Rkintc Integral not found");
  GG_CUDA(cudaSetDevice(ctx->device));
  GG_CUDA(cudaMemcpyAsync(tegral, rk.dVal.p + (loc - 1), sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  GG_CUDA(cudaStreamSynchronize(ctx->stream));
  return GG_OK;
}

int gg_slater(gg_ctx *ctx, int ia, int ib, int ic, int id, int k, double *out) {
  GG_TRY(ensure_orbitals(ctx));
  Orbitals &o = ctx->orb;
  Grid &g = ctx->grid;
  const int nw = o.nw;
  if (!out || k < 0 || k > KLIMIT || ia < 1 || ib < 1 || ic < 1 || id < 1 || ia > nw || ib > nw || ic > nw ||
      id > nw)
    return fail(GG_ERR_ARG, "gg_slater: bad arguments");
  GG_CUDA(cudaSetDevice(ctx->device));
  YDesc y;
  y.k = k;
  y.b = ib;
  y.d = id;
  y.mtp = std::min(o.mf[ib], o.mf[id]);
  y.mtpb = (k == 0 && ib == id) ? g.n : y.mtp;
  y.cs = 0;
  y.nd = 1;
  // SLATER's integration limit (slater.f90:56-60)
  QuadItem it{};
  it.a = ia;
  it.c = ic;
  it.f = 0;
  it.mtp = (k == 0 && ib == id) ? std::min(o.mf[ia], o.mf[ic]) : std::min(std::min(y.mtp, o.mf[ia]), o.mf[ic]);
  it.pos = 0;
  std::vector<YDesc> hy{y};
  std::vector<QuadItem> hi{it};
  DBuf<YDesc> dy;
  DBuf<QuadItem> di;
  DBuf<double> dY, scratch, dout;
  GG_TRY(upload(dy, hy, ctx->stream));
  GG_TRY(upload(di, hi, ctx->stream));
  GG_TRY(dY.alloc(g.np));
  GG_TRY(dout.alloc(1));
  GG_TRY(build_y(ctx, dy.p, 1, dY.p, scratch));
  // (the long grid's TA goes where build_y had its TEMP arrays)
  const size_t smem = g.np * sizeof(double);
  const bool sh = smem <= SMEM_PLAIN;
  k_quad_items<<<1, 32, sh ? smem : 0, ctx->stream>>>(di.p, 1, dY.p, g.np, o.dPF.p, o.dQF.p, o.ld, g.dR.p, g.dRP.p,
                                                      g.dRPOR.p, g.q, sh ? nullptr : scratch.p, dout.p);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaMemcpyAsync(out, dout.p, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  GG_CUDA(cudaStreamSynchronize(ctx->stream));
  return GG_OK;
}

}  // extern "C"


extern "C" {
static int run_rinti(gg_ctx *ctx, const std::vector<int2> &jk, int mode, double *dOut, const std::vector<int> *outidx);
}

// YPOT / XPOT on the device: the list's distinct Y^k_ab (every grid point,
// YZK's TB), then k_pot_part and k_pot_final. A list as the caller passed it: YPOT labels
// NYA = (IOY2 KEY + IOY1) KEY + K, XPOT labels NXA = ((IORB KEY + IOY2) KEY +
// IOY1) KEY + K, and their coefficients.
struct RawList {
  const int32_t *lab = nullptr;
  const double *co = nullptr;
  int n = 0;
};

static int raw_list(int ncof, const int32_t *lab, const double *co, RawList &r) {
  if (ncof < 0 || (ncof > 0 && (!lab || !co))) return fail(GG_ERR_ARG, "potential: bad coefficient list");
  r = RawList{lab, co, ncof};
  return GG_OK;
}

// One orbital's potentials on the device: YP, XP, XQ (N each, 0-based) at
// out, out + n, out + 2 n.
struct PotJob {
  RawList y, x;
  std::vector<int> nda;
  std::vector<double> da;
  std::vector<int> lag_m;      // LAGCON: the pairs' other orbitals
  std::vector<double> lag_wa;  // and their weights ECV WB
};

// What a potential call keeps on the context for the next: a pinned staging
// buffer and the device buffers (a COFPOT call for each orbital of an SCF cycle
// then allocates nothing), until gg_release_memory or a call whose buffers pass
// POT_KEEP bytes.
struct PotWork {
  void *stage = nullptr;
  size_t stage_bytes = 0;
  DBuf<char> up;  // the staged block on the device
  DBuf<int> term;
  DBuf<double> coef, Y, scratch, pot, part;
  DBuf<YDesc> yd;
  ~PotWork() { cudaFreeHost(stage); }
  size_t bytes() const {
    return stage_bytes + up.n + term.n * sizeof(int) + yd.n * sizeof(YDesc) +
           (coef.n + Y.n + scratch.n + pot.n + part.n) * sizeof(double);
  }
};
constexpr size_t POT_KEEP = (size_t)512 << 20, POT_BOUND = (size_t)256 << 20;

// a call's use of the context's PotWork: no other call nor gg_release_memory
// touches it meanwhile
struct PotUse {
  gg_ctx *ctx;
  std::lock_guard<std::mutex> lock;
  explicit PotUse(gg_ctx *c) : ctx(c), lock(c->pot_mu) {
    if (!ctx->pot_work) ctx->pot_work = std::make_shared<PotWork>();
  }
  ~PotUse() {
    if (work().bytes() > POT_KEEP) ctx->pot_work.reset();
  }
  PotWork &work() const { return *std::static_pointer_cast<PotWork>(ctx->pot_work); }
};

// the jobs' YPOT, XPOT, then LAGCON and DACON, into W.pot (3 n per job): all
// Y functions of all lists built once. Everything the host prepares (lists,
// chunk and job records) travels in one copy and the call waits once, at the
// end; the launches over functions are sized by a bound and read the number
// of functions on the device. out (may be null): where the potentials go on
// the host.
static int run_potentials(gg_ctx *ctx, PotWork &W, const std::vector<PotJob> &jobs, double *out = nullptr) {
  Orbitals &o = ctx->orb;
  Grid &g = ctx->grid;
  cudaStream_t s = ctx->stream;
  const int n = g.n, nw = o.nw;
  // every job's YPOT list, then every job's XPOT list, as the caller passed
  // them; the chunks of every list; the DACON and LAGCON lists; the job records
  std::vector<size_t> oy(jobs.size()), ox(jobs.size());
  size_t T = 0, nd = 0, nl = 0;
  for (size_t j = 0; j < jobs.size(); ++j) oy[j] = T, T += (size_t)jobs[j].y.n;
  const size_t TY = T;
  for (size_t j = 0; j < jobs.size(); ++j) ox[j] = T, T += (size_t)jobs[j].x.n;
  const int len = (int)(POT_CHUNK * (T / ((size_t)POT_CHUNK * 16384) + 1));
  size_t nch = 0;
  for (const PotJob &J : jobs) {
    nch += (size_t)(J.y.n + len - 1) / len + (size_t)(J.x.n + len - 1) / len;
    nd += J.nda.size();
    nl += J.lag_m.size();
  }
  size_t need = 0;
  auto place = [&](size_t bytes) {
    const size_t at = need;
    need += (bytes + 15) / 16 * 16;
    return at;
  };
  const size_t alab = place(T * sizeof(int32_t)), aco = place(T * sizeof(double)), ach = place(nch * sizeof(PotChunk)),
               afin = place(jobs.size() * sizeof(PotFinal)), aint = place((nd + nl) * sizeof(int)),
               adbl = place((nd + nl) * sizeof(double));
  const size_t ares = place(((out ? (size_t)3 * n * jobs.size() : 0) + 1) * sizeof(double));
  if (need > W.stage_bytes) {
    cudaFreeHost(W.stage);
    W.stage = nullptr;
    W.stage_bytes = 0;
    GG_CUDA(cudaHostAlloc(&W.stage, need + need / 4, cudaHostAllocDefault));
    note_alloc();
    W.stage_bytes = need + need / 4;
  }
  char *stage = static_cast<char *>(W.stage);
  const size_t tsize = (size_t)(KLIMIT + 1) * nw * nw, T1 = std::max<size_t>(T, 1);
  int nfb = (int)std::max<size_t>(1, std::min(T, tsize));  // at least as many as there are functions
  GG_TRY(W.up.alloc(ares));
  GG_TRY(W.term.alloc(2 * T1));
  GG_TRY(W.coef.alloc(T1));
  GG_TRY(W.yd.alloc(nfb));
  // the potentials, the parser's two counts and its table: one read-back and one clearing
  const size_t npot = (size_t)3 * n * jobs.size();
  GG_TRY(W.pot.alloc(npot + 1 + (tsize + 1) / 2));
  int *info = reinterpret_cast<int *>(W.pot.p + npot), *tab = info + 2;
  int *dkey = W.term.p, *diorb = dkey + T1;
  int32_t *hlab = reinterpret_cast<int32_t *>(stage + alab);
  double *hco = reinterpret_cast<double *>(stage + aco);
  PotChunk *hc = reinterpret_cast<PotChunk *>(stage + ach);
  PotFinal *hf = reinterpret_cast<PotFinal *>(stage + afin);
  int *hi = reinterpret_cast<int *>(stage + aint);
  double *hd = reinterpret_cast<double *>(stage + adbl);
  const int *di = reinterpret_cast<const int *>(W.up.p + aint);
  const double *dd = reinterpret_cast<const double *>(W.up.p + adbl);
  size_t po = 0, ic = 0, il = 0;  // partial sums (in doubles), chunks, one-body and multiplier entries
  for (size_t j = 0; j < jobs.size(); ++j) {
    const PotJob &J = jobs[j];
    const RawList *L[2] = {&J.y, &J.x};
    const size_t at[2] = {oy[j], ox[j]};
    size_t start[2];
    for (int m = 0; m < 2; ++m) {
      start[m] = po;
      if (L[m]->n > 0) {
        std::memcpy(hlab + at[m], L[m]->lab, (size_t)L[m]->n * sizeof(int32_t));
        std::memcpy(hco + at[m], L[m]->co, (size_t)L[m]->n * sizeof(double));
      }
      for (int t0 = 0; t0 < L[m]->n; t0 += len) {
        hc[ic++] = PotChunk{dkey + at[m] + t0, m ? diorb + at[m] + t0 : nullptr, W.coef.p + at[m] + t0, po,
                            std::min(len, L[m]->n - t0)};
        po += (size_t)(m ? 2 : 1) * n;
      }
    }
    const size_t i0 = il;
    for (size_t t = 0; t < J.lag_m.size(); ++t) hi[il] = J.lag_m[t], hd[il++] = J.lag_wa[t];
    const size_t i1 = il;
    for (size_t t = 0; t < J.nda.size(); ++t) hi[il] = J.nda[t], hd[il++] = J.da[t];
    hf[j] = PotFinal{W.pot.p + (size_t)3 * n * j, start[0], start[1], (J.y.n + len - 1) / len, (J.x.n + len - 1) / len,
                     di + i0, di + i1, dd + i0, dd + i1, (int)J.lag_m.size(), (int)J.nda.size()};
  }
  GG_TRY(W.part.alloc(std::max<size_t>(1, po)));
  if (ares > 0) GG_CUDA(cudaMemcpyAsync(W.up.p, stage, ares, cudaMemcpyHostToDevice, s));
  GG_CUDA(cudaMemsetAsync(info, 0, (2 + tsize) * sizeof(int), s));
  const int32_t *dlab = reinterpret_cast<const int32_t *>(W.up.p + alab);
  const double *dco = reinterpret_cast<const double *>(W.up.p + aco);
  const unsigned pgrid = (unsigned)std::max<size_t>(1, std::min<size_t>((T + 255) / 256, (size_t)8 * ctx->sms));
  if (T > 0) {
    k_parse_terms<<<pgrid, 256, 0, s>>>((int64_t)TY, (int64_t)T, dlab, dco, nw, g.c, o.dMF.p, n, tab, W.yd.p, dkey,
                                        diorb, W.coef.p, info);
    ::gg::note_launch();
  }
  if ((size_t)7 * nfb * g.np * sizeof(double) > POT_BOUND) {
    // too much to reserve for a bound: wait for the number. (7 arrays: Y and
    // the six of the long grids' build; k_yfun's grids need Y only and could
    // reserve seven times as many functions.)
    int cnt = 0;
    GG_CUDA(cudaMemcpyAsync(&cnt, info, sizeof(int), cudaMemcpyDeviceToHost, s));
    GG_CUDA(cudaStreamSynchronize(s));
    nfb = std::max(1, cnt);
  }
  GG_TRY(W.Y.alloc((size_t)nfb * g.np));
  if (T > 0) GG_TRY(build_y_pot(ctx, W.yd.p, nfb, W.Y.p, W.scratch, info));
  // one launch for all chunks, one for every job's point values
  if (nch > 0) {
    GG_CUDA(launch_pdl(k_pot_part, dim3((n + 63) / 64, (unsigned)nch), 256, 0, s,
                       reinterpret_cast<const PotChunk *>(W.up.p + ach), tab, W.Y.p, g.np, o.dPF.p, o.dQF.p, o.ld, n,
                       W.part.p));
    ::gg::note_launch();
  }
  if (!jobs.empty()) {
    GG_CUDA(launch_pdl(k_pot_final, dim3((n + 31) / 32, (unsigned)jobs.size()), 32 * PF_ROWS, 0, s,
                       reinterpret_cast<const PotFinal *>(W.up.p + afin), W.part.p, n, o.dNAK.p, o.dMF.p, g.dR.p,
                       g.dRPOR.p, g.dZZ.p, o.dPF.p, o.dQF.p, o.ld, g.q));
    ::gg::note_launch();
  }
  GG_CUDA(cudaGetLastError());
  // with out: the potentials and the counts behind them
  double *hres = reinterpret_cast<double *>(stage + ares);
  const size_t skip = out ? 0 : npot;
  int *hinfo = reinterpret_cast<int *>(hres + npot - skip);
  GG_CUDA(cudaMemcpyAsync(hres, W.pot.p + skip, (npot - skip + 1) * sizeof(double), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));
  const bool bad = hinfo[1] != 0;
  if (out && !bad) std::memcpy(out, hres, npot * sizeof(double));
  if (bad) return fail(GG_ERR_ARG, "potential: label outside the orbital set or K above 20");
  return GG_OK;
}

static int potential(gg_ctx *ctx, int mode, int ncof, const int32_t *lab, const double *co, double *out0,
                     double *out1) {
  GG_TRY(ensure_orbitals(ctx));
  if (!out0 || (mode == 1 && !out1)) return fail(GG_ERR_ARG, "gg_ypot/gg_xpot: bad arguments");
  GG_CUDA(cudaSetDevice(ctx->device));
  std::vector<PotJob> jobs(1);
  GG_TRY(raw_list(ncof, lab, co, mode == 0 ? jobs[0].y : jobs[0].x));
  const int n = ctx->grid.n;
  std::vector<double> h((size_t)3 * n);
  PotUse use(ctx);
  GG_TRY(run_potentials(ctx, use.work(), jobs, h.data()));
  if (mode == 0) {
    std::copy(h.begin(), h.begin() + n, out0);
  } else {
    std::copy(h.begin() + n, h.begin() + 2 * n, out0);
    std::copy(h.begin() + 2 * n, h.end(), out1);
  }
  return GG_OK;
}

// one orbital's SETCOF lists as a job (DACON's list checked here)
static int cof_job(gg_ctx *ctx, const gg_cof *c, PotJob &J) {
  if (!c) return fail(GG_ERR_ARG, "potential: missing coefficient lists");
  GG_TRY(raw_list(c->ny, c->nya, c->ya, J.y));
  GG_TRY(raw_list(c->nx, c->nxa, c->xa, J.x));
  if (c->nd < 0 || (c->nd > 0 && (!c->nda || !c->da))) return fail(GG_ERR_ARG, "potential: bad DACON list");
  J.nda.assign(c->nda, c->nda + std::max(0, c->nd));
  J.da.assign(c->da, c->da + std::max(0, c->nd));
  for (int io : J.nda)
    if (io < 1 || io > ctx->orb.nw) return fail(GG_ERR_ARG, "potential: DACON orbital outside the orbital set");
  return GG_OK;
}

extern "C" {

int gg_ypot(gg_ctx *ctx, int ncof, const int32_t *nya, const double *ya, double *yp) {
  if (!ctx) return fail(GG_ERR_ARG, "gg_ypot: no context");
  return potential(ctx, 0, ncof, nya, ya, yp, nullptr);
}

int gg_xpot(gg_ctx *ctx, int ncof, const int32_t *nxa, const double *xa, double *xp, double *xq) {
  if (!ctx) return fail(GG_ERR_ARG, "gg_xpot: no context");
  return potential(ctx, 1, ncof, nxa, xa, xp, xq);
}

int gg_cofpot(gg_ctx *ctx, int j, double ucfj, const gg_cof *cof, int nec, const int32_t *iecc, const double *ecv,
              double accy, double *yp, double *xp, double *xq) {
  if (!ctx || !cof || !yp || !xp || !xq || nec < 0 || (nec > 0 && (!iecc || !ecv)))
    return fail(GG_ERR_ARG, "gg_cofpot: bad arguments");
  GG_TRY(ensure_orbitals(ctx));
  const int nw = ctx->orb.nw;
  if (j < 1 || j > nw) return fail(GG_ERR_ARG, "gg_cofpot: orbital outside the orbital set");
  GG_CUDA(cudaSetDevice(ctx->device));
  std::vector<PotJob> jobs(1);
  GG_TRY(cof_job(ctx, cof, jobs[0]));
  // LAGCON's host part (lagcon.f90:32-45): the pairs with J and their weights
  if (nec > 0) {
    const double eps = (accy > 0 ? accy : std::pow(ctx->grid.h, 6)) * 0.01;
    const double wb = 1.0 / (ucfj * ctx->grid.c) / 1.0;
    for (int k = 0; k < nec; ++k) {
      const int l1 = iecc[k] / KEYORB, l2 = iecc[k] - KEYORB * l1;
      int m;
      if (j == l1)
        m = l2;
      else if (j == l2)
        m = l1;
      else
        continue;
      if (m < 1 || m > nw) return fail(GG_ERR_ARG, "gg_cofpot: multiplier pair outside the orbital set");
      const double wa = ecv[k] * wb;
      if (std::fabs(wa) < eps) continue;
      jobs[0].lag_m.push_back(m);
      jobs[0].lag_wa.push_back(wa);
    }
  }
  const int n = ctx->grid.n;
  std::vector<double> h((size_t)3 * n);  // one read-back of YP, XP, XQ
  PotUse use(ctx);
  GG_TRY(run_potentials(ctx, use.work(), jobs, h.data()));
  std::copy(h.begin(), h.begin() + n, yp);
  std::copy(h.begin() + n, h.begin() + 2 * n, xp);
  std::copy(h.begin() + 2 * n, h.end(), xq);
  return GG_OK;
}

int gg_setlag(gg_ctx *ctx, int nec, const int32_t *iecc, const double *ucf, const int *lfix, const gg_cof *cof,
              double *ecv) {
  if (!ctx || nec < 0 || (nec > 0 && (!iecc || !ucf || !lfix || !cof || !ecv)))
    return fail(GG_ERR_ARG, "gg_setlag: bad arguments");
  if (nec == 0) return GG_OK;
  GG_TRY(ensure_orbitals(ctx));
  const Orbitals &o = ctx->orb;
  Grid &g = ctx->grid;
  const int nw = o.nw;
  GG_CUDA(cudaSetDevice(ctx->device));
  // the pairs (setlag.f90:146-149: M = IECC / KEY, J = IECC - KEY M), one
  // potential job per orbital named in a pair
  std::vector<int> slot(nw + 1, -1), orbs;
  std::vector<int4> pj(nec);
  std::vector<int2> ps(nec);
  std::vector<double2> uc(nec);
  std::vector<int2> rjk;
  std::vector<int> ridx;
  for (int k = 0; k < nec; ++k) {
    const int M = iecc[k] / KEYORB, J = iecc[k] - KEYORB * M;
    if (J < 1 || J > nw || M < 1 || M > nw) return fail(GG_ERR_ARG, "gg_setlag: pair outside the orbital set");
    if (o.nak[J] != o.nak[M]) return fail(GG_ERR_KAPPA, "gg_setlag: pair with different kappa (RINTI)");
    for (int x : {J, M})
      if (slot[x] < 0) {
        slot[x] = (int)orbs.size();
        orbs.push_back(x);
      }
    const double uj = ucf[J - 1], um = ucf[M - 1];
    int cs;
    if (lfix[M - 1]) {
      cs = 0;
    } else if (lfix[J - 1]) {
      cs = 1;
    } else {
      const double qdif = std::fabs((uj - um) / std::max(uj, um));
      cs = (qdif > 1.0e-01) ? 2 : 3;
    }
    pj[k] = make_int4(J, M, cs, std::max(o.mf[J], o.mf[M]));
    ps[k] = make_int2(slot[J], slot[M]);
    uc[k] = make_double2(uj, um);
    if (cs != 2) {  // RINTI(M, J, 1), or RINTI(J, M, 1) when J is fixed
      rjk.push_back(cs == 1 ? make_int2(J, M) : make_int2(M, J));
      ridx.push_back(k);
    }
  }
  std::vector<PotJob> jobs(orbs.size());
  for (size_t i = 0; i < orbs.size(); ++i) GG_TRY(cof_job(ctx, &cof[orbs[i] - 1], jobs[i]));
  PotUse use(ctx);
  GG_TRY(run_potentials(ctx, use.work(), jobs));
  const DBuf<double> &pot = use.work().pot;
  cudaStream_t s = ctx->stream;
  DBuf<int4> dpj;
  DBuf<int2> dps;
  DBuf<double2> duc;
  DBuf<double> dTA, dres, drij, decv;
  GG_TRY(upload(dpj, pj, s));
  GG_TRY(upload(dps, ps, s));
  GG_TRY(upload(duc, uc, s));
  const size_t psm = quad_panels(g.np) * sizeof(double);
  const bool sh = psm <= SMEM_PLAIN;
  GG_TRY(dTA.alloc((size_t)nec * (g.np + (sh ? 0 : quad_panels(g.np)))));
  GG_TRY(dres.alloc(nec));
  GG_TRY(drij.alloc(nec));
  GG_TRY(decv.alloc(nec));
  GG_CUDA(cudaMemsetAsync(drij.p, 0, nec * sizeof(double), s));
  (sh ? k_setlag_quad<true> : k_setlag_quad<false>)<<<nec, 128, sh ? psm : 0, s>>>(
      dpj.p, dps.p, pot.p, g.n, o.dPF.p, o.dQF.p, o.ld, g.dR.p, g.dRP.p, g.dRPOR.p, g.q, g.np, dTA.p, dres.p);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  if (!rjk.empty()) GG_TRY(run_rinti(ctx, rjk, 1, drij.p, &ridx));
  k_setlag_final<<<(nec + 127) / 128, 128, 0, s>>>(nec, dpj.p, duc.p, dres.p, drij.p, decv.p);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaMemcpyAsync(ecv, decv.p, nec * sizeof(double), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));
  return GG_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// gg_slater_noalloc: SLATER without any device allocation.
//
// Some callers cannot allocate device memory when they need one integral: a
// host code that has handed the whole device to a memory pool or to the
// Hamiltonian and Davidson basis of a large block (where a cudaMalloc would
// fail or fragment the pool), or code whose error handling cannot recover
// from an allocation failure in the middle of a loop (the Fortran callers
// STOP). For them this entry point evaluates R^k(ab;cd) exactly like
// gg_slater, but its working arrays (the two TEMP arrays and Y^k of YZK, the
// integral's descriptors and its result) live in one file-scope device array
// of fixed size, reserved when the library is loaded and held by every GPU
// that loads it until the process exits.
//
// Limit: the grid must satisfy N + 26 <= NOALLOC_NP (N <= 2022 points; GRASP
// uses 590). The first call on a device looks up the array's device address
// (cudaGetSymbolAddress) with that device current; make that first call
// before any stream capture. All calls share the array and it keeps the last
// call's contents (Y^k is cleared at the start of each call): calls that can
// overlap on the GPU -- several host threads, or several contexts on one
// device -- race on it and must be serialised by the caller.
// ---------------------------------------------------------------------------
namespace gg {
namespace {
constexpr int NOALLOC_NP = 2048;              // doubles per working array
constexpr int NOALLOC_DESC = 64;              // doubles reserved for descriptors and the result
static __device__ __align__(256) double g_noalloc_scratch[3 * NOALLOC_NP + NOALLOC_DESC];

struct NoallocAddr {
  std::mutex mu;
  double *ptr[64] = {};
};
NoallocAddr &noalloc_addr() {
  static NoallocAddr a;
  return a;
}
}  // namespace
}  // namespace gg

extern "C" int gg_slater_noalloc(gg_ctx *ctx, int ia, int ib, int ic, int id, int k, double *out) {
  GG_TRY(ensure_orbitals(ctx));
  Orbitals &o = ctx->orb;
  Grid &g = ctx->grid;
  const int nw = o.nw;
  if (!out || k < 0 || k > KLIMIT || ia < 1 || ib < 1 || ic < 1 || id < 1 || ia > nw || ib > nw || ic > nw ||
      id > nw)
    return fail(GG_ERR_ARG, "gg_slater_noalloc: bad arguments");
  if (g.np > NOALLOC_NP)
    return fail(GG_ERR_ARG, "gg_slater_noalloc: grid of " + std::to_string(g.n) +
                                " points exceeds the fixed scratch (at most " + std::to_string(NOALLOC_NP - GPAD - 10) +
                                " points); use gg_slater");
  if (ctx->device < 0 || ctx->device >= 64) return fail(GG_ERR_ARG, "gg_slater_noalloc: device index above 63");
  GG_CUDA(cudaSetDevice(ctx->device));
  double *base = nullptr;
  {
    NoallocAddr &A = noalloc_addr();
    std::lock_guard<std::mutex> lock(A.mu);
    if (!A.ptr[ctx->device]) {
      void *p = nullptr;
      GG_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
      A.ptr[ctx->device] = static_cast<double *>(p);
    }
    base = A.ptr[ctx->device];
  }
  double *TZ = base, *TW = base + NOALLOC_NP, *Y = base + 2 * NOALLOC_NP;
  double *tail = base + 3 * NOALLOC_NP;  // 256-byte aligned: 3 * 2048 doubles = 192 * 256 bytes
  YDesc *dyd = reinterpret_cast<YDesc *>(tail);
  QuadItem *ditem = reinterpret_cast<QuadItem *>(tail + 8);
  double *dout = tail + 16;
  YDesc y;
  y.k = k;
  y.b = ib;
  y.d = id;
  y.mtp = std::min(o.mf[ib], o.mf[id]);
  y.mtpb = (k == 0 && ib == id) ? g.n : y.mtp;
  y.cs = 0;
  y.nd = 1;
  QuadItem it{};
  it.a = ia;
  it.c = ic;
  it.f = 0;
  it.mtp = (k == 0 && ib == id) ? std::min(o.mf[ia], o.mf[ic]) : std::min(std::min(y.mtp, o.mf[ia]), o.mf[ic]);
  it.pos = 0;
  const int np = g.np;
  GG_CUDA(cudaMemcpyAsync(dyd, &y, sizeof(YDesc), cudaMemcpyHostToDevice, ctx->stream));
  GG_CUDA(cudaMemcpyAsync(ditem, &it, sizeof(QuadItem), cudaMemcpyHostToDevice, ctx->stream));
  dim3 grid1((np + 127) / 128, 1);
  k_ytemp<<<grid1, 128, 0, ctx->stream>>>(dyd, 1, nullptr, o.dPF.p, o.dQF.p, o.ld, g.dRP.p, g.dPow.p, np, TZ, TW);
  ::gg::note_launch();
  GG_CUDA(cudaMemsetAsync(Y, 0, (size_t)np * sizeof(double), ctx->stream));
  k_ychain<<<1, 128, 0, ctx->stream>>>(dyd, 1, nullptr, TZ, TW, g.dR.p, g.dPow.p, np, g.q, Y);
  ::gg::note_launch();
  k_quad_items<<<1, 32, np * sizeof(double), ctx->stream>>>(ditem, 1, Y, np, o.dPF.p, o.dQF.p, o.ld, g.dR.p,
                                                            g.dRP.p, g.dRPOR.p, g.q, nullptr, dout);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  GG_CUDA(cudaMemcpyAsync(out, dout, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  GG_CUDA(cudaStreamSynchronize(ctx->stream));
  return GG_OK;
}

extern "C" {

static int run_rinti(gg_ctx *ctx, const std::vector<int2> &jk, int mode, double *dOut, const std::vector<int> *outidx) {
  Orbitals &o = ctx->orb;
  Grid &g = ctx->grid;
  std::vector<int4> h(jk.size());
  for (size_t i = 0; i < jk.size(); ++i) h[i] = make_int4(jk[i].x, jk[i].y, outidx ? (*outidx)[i] : (int)i, 0);
  DBuf<int4> djk;  // freed in stream order
  GG_TRY(upload(djk, h, ctx->stream));
  const size_t smem = rinti_work(g.np) * sizeof(double);
  const bool sh = smem <= SMEM_PLAIN;
  // with its arrays in global memory a block per SM is enough, and 0.6 GB at N = 100,000
  const int blocks = std::max(1, std::min((int)jk.size(), sh ? 2048 : ctx->sms));
  DBuf<double> work;
  if (!sh) GG_TRY(work.alloc(blocks * rinti_work(g.np)));
  (sh ? k_rinti<true> : k_rinti<false>)<<<blocks, 32 * RINTI_WARPS, sh ? smem : 0, ctx->stream>>>(
      djk.p, (int)jk.size(), mode, o.dPF.p, o.dQF.p, o.ld, o.dMF.p, o.dNAK.p, g.dR.p, g.dRP.p, g.dRPOR.p, g.dZZ.p,
      g.np, g.q, work.p, dOut);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

int gg_rinti(gg_ctx *ctx, int j, int k, int mode, double *out) {
  GG_TRY(ensure_orbitals(ctx));
  const Orbitals &o = ctx->orb;
  if (!out || j < 1 || k < 1 || j > o.nw || k > o.nw) return fail(GG_ERR_ARG, "gg_rinti: bad arguments");
  if (o.nak[j] != o.nak[k]) return fail(GG_ERR_KAPPA, "RINTI: Attempt to calculate I(a,b) with kappa(a) != kappa(b)");
  GG_CUDA(cudaSetDevice(ctx->device));
  DBuf<double> d;
  GG_TRY(d.alloc(1));
  GG_TRY(run_rinti(ctx, {make_int2(j, k)}, mode, d.p, nullptr));
  GG_CUDA(cudaMemcpy(out, d.p, sizeof(double), cudaMemcpyDeviceToHost));
  return GG_OK;
}

int gg_iabint_table(gg_ctx *ctx, double *iab) {
  GG_TRY(ensure_orbitals(ctx));
  GG_CUDA(cudaSetDevice(ctx->device));
  const Orbitals &o = ctx->orb;
  const int nw = o.nw;
  GG_TRY(timer_start(ctx));
  GG_TRY(ctx->dIab.alloc((size_t)nw * nw));
  k_fill<<<64, 256, 0, ctx->stream>>>(ctx->dIab.p, (size_t)nw * nw, nan("")); ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  std::vector<int2> jk;
  std::vector<int> idx;
  for (int a = 1; a <= nw; ++a)
    for (int b = 1; b <= nw; ++b)
      if (o.nak[a] == o.nak[b]) {
        jk.push_back(make_int2(a, b));
        idx.push_back((a - 1) * nw + (b - 1));
      }
  if (!jk.empty()) GG_TRY(run_rinti(ctx, jk, 0, ctx->dIab.p, &idx));
  GG_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
  if (iab)
    GG_CUDA(cudaMemcpyAsync(iab, ctx->dIab.p, (size_t)nw * nw * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  GG_CUDA(cudaStreamSynchronize(ctx->stream));
  double ms = 0;
  GG_TRY(timer_read(ctx, &ms));
  ctx->stats[1] = ms;
  ctx->iab_valid = true;
  return GG_OK;
}

}  // extern "C"

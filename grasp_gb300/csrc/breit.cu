// breit.cu - the transverse-photon (Breit) radial integrals of rci on the GPU:
// GENINTBREIT1/2's tables (rci90/genintbreit1.f90, genintbreit2.f90) and
// BRINTF (rci90/brintf.f90) for any list of integrals (what BRINT3-6 compute
// on demand).
//
// BRINTF(type, a, b, c, d, k) combines up to four RKINT (rkint.f90) or two
// SKINT (skint.f90) terms; each term is one QUAD (quad.f90) of a product
// with one or two ZKF functions (zkf.f90: Z_k of a radial product, the
// stride-4 Newton-Cotes chain), the frequency-dependent terms weighted by
// spherical Bessel factors (bessel.f90). On the device:
//
//  The tables are dot products of pair densities with one vector per (pair,
//  k): run_table and the k_br_* kernels. A list (gg_brintf), and the entries
//  of a table that the contraction cannot take, go term by term:
//
//  0. k_plan_items: the integrals' terms; one pass counts them, the host scans
//     the counts, a second pass writes them.
//  1. k_bessel: every Bessel function the integrals need, (pair, order) with
//     W = WFACT |E(a) - E(b)| / C, one block each: the series where it
//     converges in four terms, the asymptotic form from the first point where
//     it does not (JCHAN), as bessel.f90:104-201.
//  2. k_breit_jobs: one thread per QUAD term. The thread runs the ZKF chain
//     (or two) point by point and feeds each TA(i) straight into a streaming
//     QUAD (head search, power-law head term, stride-4 group sums, end
//     correction), so no ZK or TA array is stored: a term costs one pass
//     over its points. The arithmetic is the reference's, operation by
//     operation (compiled without FMA contraction), so the values are the
//     oracle's to the rounding of log, sin and cos.
//  3. k_breit_combine: each integral from its terms, BRRA's and SKINT's
//     combinations (brra.f90:36-118, skint.f90:70-83).
//
// BRINTF is evaluated as a function of its arguments: the reference keeps
// the last Bessel functions in four slots (bess_C KEEP) and skips a BESSEL
// call whose slot already holds the function; slot 1 holds pair (a, b),
// slot 2 pair (c, d). Where the reference skips the call for two equal
// orbitals (zero frequency, brintf.f90:47-48) its slot keeps earlier
// content; here that slot is the zero-frequency function (zero).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <vector>

#include "gg_internal.cuh"

namespace gg {
namespace {

constexpr int KLIM = 20;  // the power tables' rows (YZK's KLIMIT)

__device__ __forceinline__ double pfv(const double *P, int ld, int i, int j) {
  return P[(size_t)(j - 1) * ld + (i - 1)];
}

// libgcc's __powidf2 algorithm (gfortran's REAL**INTEGER)
__device__ __forceinline__ double powi_d(double x, int m) {
  unsigned n = m < 0 ? -(unsigned)m : (unsigned)m;
  double y = (n % 2) ? x : 1.0;
  while (n >>= 1) {
    x = x * x;
    if (n % 2) y = y * x;
  }
  return m < 0 ? 1.0 / y : y;
}

struct BessDesc {
  double w;  // W (> EPSI^2)
  int nn;    // order
};

// BESSEL (rci90/bessel.f90:96-201) for one (pair, order): BJ, BN at points
// 1..N ([f][np]). Series at each point while every earlier point converged
// in four terms; from the first that does not (JCHAN), the asymptotic form.
__global__ void __launch_bounds__(128) k_bessel(const BessDesc *__restrict__ bd, const double *__restrict__ R, int n,
                                                int np, double epsi, double *__restrict__ BJ,
                                                double *__restrict__ BN) {
  __shared__ int jchan_s;
  const BessDesc d = bd[blockIdx.x];
  double *J = BJ + (size_t)blockIdx.x * np, *N = BN + (size_t)blockIdx.x * np;
  const int nn = d.nn;
  const double W = d.w;
  if (threadIdx.x == 0) jchan_s = n + 1;
  __syncthreads();
  for (int j = 2 + threadIdx.x; j <= n; j += blockDim.x) {
    const double WA = -0.5 * ((R[j] * W) * (R[j] * W));
    double X1 = 1.0, X2 = 1.0, S1 = 0.0, S2 = 0.0;
    bool done = false;
    for (int i = 1; i <= 4; ++i) {
      X1 = X1 * WA / (double)(i * (2 * (nn + i) + 1));
      X2 = X2 * WA / (double)(i * (2 * (i - nn) - 1));
      S1 = S1 + X1;
      S2 = S2 + X2;
      if (fabs(X1) >= fabs(S1) * epsi || fabs(X2) >= fabs(S2) * epsi) continue;
      done = true;
      break;
    }
    J[j] = S1;
    N[j] = S2;
    if (!done) atomicMin(&jchan_s, j);
  }
  if (threadIdx.x == 0) {
    J[1] = 0.0;
    N[1] = 0.0;
  }
  __syncthreads();
  const int jchan = jchan_s;
  if (jchan > n) return;
  double DFNM = 1.0, DFN = 1.0;
  if (nn != 0) {
    for (int i = 3; i <= 2 * nn - 1; i += 2) DFNM = DFNM * (double)i;
    DFN = DFNM * (double)(2 * nn + 1);
  }
  DFNM = 1.0 / DFNM;
  const int irem = nn % 4;
  const double SSN = (irem == 1 || irem == 2) ? -1.0 : 1.0;
  const double SCN = (irem == 2 || irem == 3) ? -1.0 : 1.0;
  const bool swap = (irem == 1 || irem == 3);
  for (int j = jchan + threadIdx.x; j <= n; j += blockDim.x) {
    const double WA = W * R[j];
    double SN, CN;
    if (!swap) {
      SN = SSN * sin(WA);
      CN = SCN * cos(WA);
    } else {
      SN = SSN * cos(WA);
      CN = SCN * sin(WA);
    }
    const double OBWA = 1.0 / WA;
    double B = OBWA;
    double S1 = B * SN, S2 = B * CN;
    for (int i = 1; i <= nn; ++i) {
      const double SKEEP = SN;
      SN = CN;
      CN = -SKEEP;
      B = B * OBWA * (double)((nn + i) * (nn - i + 1)) / (double)(2 * i);
      S1 = S1 + B * SN;
      S2 = S2 + B * CN;
    }
    J[j] = S1 * DFN / powi_d(WA, nn) - 1.0;
    N[j] = S2 * powi_d(WA, nn + 1) * DFNM - 1.0;
  }
}

// One QUAD term. form 0: RKINT (one chain of order k from src (1 + BJ);
// TA = part (1 + BN) ZK RPOR); 1: SKINT at zero frequency (chains k - 1 and
// k + 1 of src; TA = part RPOR (ZK+ - ZK-)); 2: SKINT's first term (chains
// k - 1 of src and of (-src) BJ; TA = ((1 + BN) ZK2 - ZK1 BN) part / R^2
// RPOR); 3: SKINT's second term (chain k + 1 of src (1 + BJ); TA = part
// (1 + BN) ZK R RP). src and part are P_x Q_y (+ P_y Q_x with the aug flag);
// a Bessel index of -1 is the zero function.
struct BrJob {
  unsigned char form, sx, sy, px, py, flags;  // flags: 1 src aug, 2 part aug
  signed char k, pad;
  int bj, bn;
};

struct ChainState {
  double z0, z1, z2, z3;      // ZK(II-4 .. II-1)
  double t0, t1, t2, t3;      // TEMP(II-4 .. II-1)
};

// streaming QUAD (lib9290/quad.f90:52-103) over TA(2..mtp) fed in order
struct QuadStream {
  int mtp, head, cnt;
  double prev, result, s, g0, g1, g2, last;
  __device__ void init(int m) {
    mtp = m;
    head = 0;
    cnt = 0;
    prev = 0.0;
    result = 0.0;
    s = 0.0;
    last = 0.0;
  }
  __device__ __forceinline__ void group(double g3, const QuadConst &q) {
    s = s + (q.C2 * (g0 + g2) + q.C3 * g1 + q.C4 * g3);
  }
  __device__ __forceinline__ void push(int i, double ta, const double *R, const double *RP, const QuadConst &q) {
    last = ta;
    if (head) {
      switch (cnt) {
        case 0: g0 = ta; break;
        case 1: g1 = ta; break;
        case 2: g2 = ta; break;
        default: group(ta, q); break;
      }
      cnt = (cnt + 1) & 3;
      return;
    }
    // head search at i - 1 (2 <= i - 1 <= mtp - 1)
    const int h = i - 1;
    if (h >= 2 && fabs(prev) > 0.0) {
      const double tai = prev, taip1 = ta;
      const double quott = taip1 / tai;
      if (quott > 0.0) {
        const double frip1 = taip1 / RP[h + 1];
        double fri = tai / RP[h];
        const double ratio = frip1 / fri;
        const double sigma = log(ratio) / log(R[h + 1] / R[h]);
        fri = R[h] * fri;
        result = fri / (sigma + 1.0);
        result = result + q.C1 * tai;
        head = h;
        g0 = ta;  // the first group starts at h + 1
        cnt = 1;
        return;
      }
    }
    prev = ta;
  }
  __device__ __forceinline__ double finish(const QuadConst &q) {
    if (!head) return 0.0;
    if (cnt == 1) {
      g1 = 0.0;
      g2 = 0.0;
      group(0.0, q);
    } else if (cnt == 2) {
      g2 = 0.0;
      group(0.0, q);
    } else if (cnt == 3) {
      group(0.0, q);
    }
    double r = result + s;
    if ((mtp - head) % 4 == 0) r = r - q.C1 * last;
    return r;
  }
};

__device__ __forceinline__ double prod(const double *PF, const double *QF, int ld, int i, int x, int y, bool aug) {
  double v = pfv(PF, ld, i, x) * pfv(QF, ld, i, y);
  if (aug) v = v + pfv(PF, ld, i, y) * pfv(QF, ld, i, x);
  return v;
}

// the grid, orbitals and Bessel tables a term reads
struct TermTabs {
  const double *PF, *QF;
  int ld;
  const int *MF;
  const double *R, *RP, *RPOR, *Pow;
  int np;
  const double *BJ, *BN;
};

__device__ double breit_term(const BrJob &jb, const TermTabs &tt, const QuadConst &q) {
  const double *PF = tt.PF, *QF = tt.QF, *R = tt.R, *RP = tt.RP, *RPOR = tt.RPOR, *Pow = tt.Pow;
  const double *BJt = tt.BJ, *BNt = tt.BN;
  const int *MF = tt.MF;
  const int ld = tt.ld, np = tt.np;
  const int form = jb.form, K = jb.k;
  const bool saug = jb.flags & 1, paug = jb.flags & 2;
  const int mtpz = min(MF[jb.sx], MF[jb.sy]);
  const int mtpq = min(mtpz, min(MF[jb.px], MF[jb.py]));
  const double *BJ = jb.bj >= 0 ? BJt + (size_t)jb.bj * np : nullptr;
  const double *BN = jb.bn >= 0 ? BNt + (size_t)jb.bn * np : nullptr;
  // chain orders: form 0: k; 1: k - 1 (a) and k + 1 (b); 2: k - 1, k - 1; 3: k + 1
  const int ka = (form == 0) ? K : (form == 3 ? K + 1 : K - 1);
  const int kb = (form == 1) ? K + 1 : K - 1;
  const bool two = (form == 1 || form == 2);
  // RTTK rows: k > 0 the R**k row, k = -1 the 1/R row (R**-1), k = 0 unused
  const double *rta = ka > 0 ? Pow + (size_t)ka * np : (ka < 0 ? Pow : nullptr);
  const double *rtb = kb > 0 ? Pow + (size_t)kb * np : (kb < 0 ? Pow : nullptr);
  // TEMP(i) of chain a and b, 0 beyond MTPZ (zkf.f90:48-57)
  auto temps = [&](int i, double &ta_, double &tb_) {
    if (i > mtpz) {
      ta_ = 0.0;
      tb_ = 0.0;
      return;
    }
    const double src = prod(PF, QF, ld, i, jb.sx, jb.sy, saug);
    const double bj = BJ ? BJ[i] : 0.0;
    double inA, inB = 0.0;
    if (form == 0 || form == 3) {
      inA = src * (1.0 + bj);
    } else if (form == 1) {
      inA = src;
      inB = src;
    } else {
      inA = src;
      inB = -src * bj;
    }
    const double rhoA = RP[i] * inA;
    ta_ = (ka == 0) ? rhoA : rta[i] * rhoA;
    if (two) {
      const double rhoB = RP[i] * inB;
      tb_ = (kb == 0) ? rhoB : rtb[i] * rhoB;
    } else {
      tb_ = 0.0;
    }
  };
  // ZK(2..4) from TEMP(2..5) (zkf.f90:58-64)
  double T[4][2];
  for (int i = 0; i < 4; ++i) temps(i + 2, T[i][0], T[i][1]);
  ChainState A, B;
  A.z0 = 0.0;
  B.z0 = 0.0;
  double za[3], zb[3];
  for (int ii = 2; ii <= 4; ++ii) {
    double sa = 0.0, sb = 0.0;
    for (int kk = 2; kk <= 5; ++kk) {
      sa = sa + q.CNC5C[kk - 2][ii - 2] * T[kk - 2][0];
      sb = sb + q.CNC5C[kk - 2][ii - 2] * T[kk - 2][1];
    }
    za[ii - 2] = sa;
    zb[ii - 2] = sb;
  }
  A.z1 = za[0]; A.z2 = za[1]; A.z3 = za[2];
  B.z1 = zb[0]; B.z2 = zb[1]; B.z3 = zb[2];
  A.t0 = 0.0; A.t1 = T[0][0]; A.t2 = T[1][0]; A.t3 = T[2][0];
  B.t0 = 0.0; B.t1 = T[0][1]; B.t2 = T[1][1]; B.t3 = T[2][1];
  double nextA = T[3][0], nextB = T[3][1];  // TEMP(5)
  QuadStream Q;
  Q.init(mtpq);
  for (int i = 2; i <= mtpq; ++i) {
    double zA, zB;
    if (i <= 4) {
      zA = za[i - 2];
      zB = zb[i - 2];
    } else {
      // ZK(II) = ZK(II-4) + C1 (TEMP(II-4) + TEMP(II)) + C2 (TEMP(II-3) +
      // TEMP(II-1)) + C3 TEMP(II-2) (zkf.f90:65-68)
      double tA, tB;
      if (i == 5) {
        tA = nextA;
        tB = nextB;
      } else {
        temps(i, tA, tB);
      }
      zA = A.z0 + q.C1 * (A.t0 + tA) + q.C2 * (A.t1 + A.t3) + q.C3 * A.t2;
      A.z0 = A.z1; A.z1 = A.z2; A.z2 = A.z3; A.z3 = zA;
      A.t0 = A.t1; A.t1 = A.t2; A.t2 = A.t3; A.t3 = tA;
      if (two) {
        zB = B.z0 + q.C1 * (B.t0 + tB) + q.C2 * (B.t1 + B.t3) + q.C3 * B.t2;
        B.z0 = B.z1; B.z1 = B.z2; B.z2 = B.z3; B.z3 = zB;
        B.t0 = B.t1; B.t1 = B.t2; B.t2 = B.t3; B.t3 = tB;
      } else {
        zB = 0.0;
      }
    }
    // ZK(i) / RTTK(i) for k != 0 (zkf.f90:70-74)
    const double ZA = (ka == 0) ? zA : zA / rta[i];
    const double ZB = two ? ((kb == 0) ? zB : zB / rtb[i]) : 0.0;
    const double part = prod(PF, QF, ld, i, jb.px, jb.py, paug);
    const double bn = BN ? BN[i] : 0.0;
    double ta;
    if (form == 0)
      ta = part * (1.0 + bn) * ZA * RPOR[i];
    else if (form == 1)
      ta = part * RPOR[i] * (ZB - ZA);
    else if (form == 2)
      ta = ((1.0 + bn) * ZB - ZA * bn) * part / powi_d(R[i], 2) * RPOR[i];
    else
      ta = part * (1.0 + bn) * ZA * R[i] * RP[i];
    Q.push(i, ta, R, RP, q);
  }
  return Q.finish(q);
}

__global__ void __launch_bounds__(128) k_breit_jobs(const BrJob *__restrict__ jobs, int64_t njobs, TermTabs tt,
                                                    QuadConst q, double *__restrict__ out) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= njobs) return;
  const BrJob jb = jobs[t];
  out[t] = breit_term(jb, tt, q);
}

// One integral: its first term, the combination (code) and SKINT's data.
// code: 0 2 q0; 1 q0 + q1; 2 (((q0 + q1) + q2) + q3) / 2; 3 S(1);
// 4 (S(1) + S(2)) / 2. S(w) = (WK / W)^2 qa - qb W W / ((2K+3)(2K-1)) at a
// frequency, WK qa / 2 at zero frequency (|W| < 1e-10).
struct BrInt {
  int q0;
  short code, k;
  double w1, w2;
};

__device__ __forceinline__ double skint_comb(const double *v, int &at, double W, int K) {
  const double WK = (double)(K + K + 1);
  if (fabs(W) < 1.0e-10) return WK * v[at++] * 0.5;
  double sk = powi_d(WK / W, 2) * v[at++];
  sk = sk - v[at++] * W * W / (double)((2 * K + 3) * (2 * K - 1));
  return sk;
}

__global__ void k_breit_combine(const BrInt *__restrict__ ints, int64_t n, const double *__restrict__ v,
                                double *__restrict__ out) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const BrInt b = ints[t];
  int at = b.q0;
  double r;
  switch (b.code) {
    case 0: r = 2.0 * v[at]; break;
    case 1: r = v[at] + v[at + 1]; break;
    case 2: r = (v[at] + v[at + 1] + v[at + 2] + v[at + 3]) * 0.5; break;
    case 3: r = skint_comb(v, at, b.w1, b.k); break;
    default: {
      const double s1 = skint_comb(v, at, b.w1, b.k);
      const double s2 = skint_comb(v, at, b.w2, b.k);
      r = (s1 + s2) * 0.5;
    }
  }
  out[t] = r;
}

// ---------------------------------------------------------------------------
// the terms of each integral (brintf.f90:34-69, brra.f90:36-118), planned on
// the device: one thread per integral (or per (k, a, b) row of a table)
// counts its terms, the counts are scanned, the same thread writes them.
// ---------------------------------------------------------------------------
struct PlanTabs {
  const double *W;   // [a][b]: W = WFACT |E(a) - E(b)| / C
  const int *bid;    // [order + 1][min(a,b)][max(a,b)]: Bessel function, -1 zero
  int nw;
};

__device__ __forceinline__ int bes_id(const PlanTabs &T, int x, int y, int nn) {
  const int lo = min(x, y), hi = max(x, y);
  return T.bid[((size_t)(nn + 1) * T.nw + (lo - 1)) * T.nw + (hi - 1)];
}

// BRINTF(type, a, b, c, d, k): RAC = P_a Q_b, RBD = P_c Q_d; Bessel slot 1
// pair (a, b), slot 2 pair (c, d). Returns the number of terms; with bi and
// jb set, writes the integral's record (first term q0) and its terms.
__device__ int plan_one(int type, int a, int b, int c, int d, int K, const PlanTabs &T, int q0, BrInt *bi,
                        BrJob *jb) {
  auto w = [&](int x, int y) { return T.W[(size_t)(x - 1) * T.nw + (y - 1)]; };
  int n = 0;
  auto job = [&](int form, int sx, int sy, bool saug, int px, int py, bool paug, int bj, int bn) {
    if (jb) {
      BrJob j;
      j.form = (unsigned char)form;
      j.sx = (unsigned char)sx;
      j.sy = (unsigned char)sy;
      j.px = (unsigned char)px;
      j.py = (unsigned char)py;
      j.flags = (unsigned char)((saug ? 1 : 0) | (paug ? 2 : 0));
      j.k = (signed char)K;
      j.pad = 0;
      j.bj = bj;
      j.bn = bn;
      jb[n] = j;
    }
    ++n;
  };
  auto R = [&](bool rac, int iw, bool augac, bool augbd) {
    const int f = iw == 0 ? -1 : (iw == 1 ? bes_id(T, a, b, K) : bes_id(T, c, d, K));
    if (rac)
      job(0, a, b, augac, c, d, augbd, f, f);
    else
      job(0, c, d, augbd, a, b, augac, f, f);
  };
  auto S = [&](int iw) {
    const int x = iw == 1 ? a : c, y = iw == 1 ? b : d;
    if (fabs(w(x, y)) < 1.0e-10) {
      job(1, a, b, false, c, d, false, -1, -1);
    } else {
      const int f1 = bes_id(T, x, y, K - 1), f2 = bes_id(T, x, y, K + 1);
      job(2, a, b, false, c, d, false, f1, f2);
      job(3, c, d, false, a, b, false, f2, f1);
    }
  };
  int code;
  switch (type) {
    case 1:
      if (a == c && b == d) {
        code = 0;
        R(true, 1, false, false);
      } else if (a == d && b == c) {
        code = 1;
        R(true, 1, false, false);
        R(false, 1, false, false);
      } else {
        code = 2;
        R(true, 1, false, false);
        R(true, 2, false, false);
        R(false, 1, false, false);
        R(false, 2, false, false);
      }
      break;
    case 2:
      if ((a == c && b == d) || (a == d && b == c)) {
        code = 3;
        S(1);
      } else {
        code = 4;
        S(1);
        S(2);
      }
      break;
    case 3:
      code = 2;
      if (a == b) {
        R(true, 0, false, true);
        R(false, 0, false, true);
        R(true, 2, false, true);
        R(false, 2, false, true);
      } else {
        R(true, 1, true, false);
        R(false, 1, true, false);
        R(true, 0, true, false);
        R(false, 0, true, false);
      }
      break;
    case 4:
      code = 1;
      R(true, 0, false, false);
      R(false, 0, false, false);
      break;
    case 5:
      if (a == d && b == c) {
        code = 1;
        R(true, 1, false, false);
        R(false, 1, false, false);
      } else {
        code = 0;
        R(true, 1, false, false);
      }
      break;
    default:
      code = 3;
      S(1);
      break;
  }
  if (bi) {
    BrInt r;
    r.q0 = q0;
    r.code = (short)code;
    r.k = (short)K;
    r.w1 = w(a, b);
    r.w2 = w(c, d);
    *bi = r;
  }
  return n;
}

// a list of integrals (items[6 t ..] = type, a, b, c, d, k)
__global__ void k_plan_items(const int32_t *__restrict__ items, int n, PlanTabs T, int pass, int *__restrict__ cnt_j,
                             const int64_t *__restrict__ off_j, BrInt *__restrict__ ints, BrJob *__restrict__ jobs) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int32_t *it = items + 6 * (size_t)t;
  if (pass)
    plan_one(it[0], it[1], it[2], it[3], it[4], it[5], T, (int)off_j[t], ints + t, jobs + off_j[t]);
  else
    cnt_j[t] = plan_one(it[0], it[1], it[2], it[3], it[4], it[5], T, 0, nullptr, nullptr);
}

// ---------------------------------------------------------------------------
// The tables by contraction. For one k, a term is linear in its source pair's
// density and in its partner pair's: with pair s the source and pair p the
// part, TA(i) = rho_p(i) q(i) Z(i), Z the stride-4 chain of e(j) rho_s(j),
//   sum_i w_i TA(i) = rho_p . F_s   (the frequency is s's: F_s = q Z[e rho_s])
//                   = rho_s . U_p   (the frequency is p's: U_p = e A[w q rho_p],
//                                    A the transposed chain, run backwards),
// so every integral of a table is a dot product of a pair density with one
// vector per (pair, k), where the term list ran a chain per term: 131 ms of
// FP64 pipe for the 1.16 M type-1 integrals of 34 subshells, against 1.8 ms
// for all the kernels below (same table), 5.1 ms against 0.40 ms for the 26 K
// type-2 integrals of 16. Bound: the FP64 pipe in k_br_gemm (1.34 ms).
//
// QUAD's weights w depend on the head index h (its first point with a
// positive ratio TA(h+1)/TA(h)) and on the last point mtpq = min(MTP_s,
// MTP_p). h is a property of the source (its chain's signs at points 2..5),
// found once per (pair, k) by k_br_heads; mtpq depends on the column's MTP.
// The columns (the pairs whose density is dotted) of one k are therefore
// grouped by (MTP, h) into buckets, a warp takes 32 rows of one bucket's
// columns (up to BR_NC), and U is U^(M0) plus a term per residue class:
//   U^(m)(j) = e(j) (c^(M0)(j) + K(j mod 4)),  j <= J0,
// with M0 the smallest MTP of all pairs, J0 <= M0 - 4, and K the class sums
// of w q rho over (M0, mtpq] (added, so nothing cancels); the points J0 < j
// <= m have their vectors per bucket (k_br_tail). An entry whose terms do not
// have the head index assumed for their bucket is evaluated term by term
// (breit_term), as are the lists of gg_brintf.
// The sums are FMA chains over the points and the 1/r^k factors multiply by
// the power table's reciprocals; the values agree with the term by term form
// to a few ulps of the largest partial sum.
// ---------------------------------------------------------------------------
constexpr int BR_NC = 8;      // columns of one warp's tile
constexpr int BR_MIN_MF = 16; // shortest orbital the contraction takes

struct BrRow {  // one (k, pair) row, padded rows have a = 0
  short a, b, K;
  int mtp;
  int fa, fb;        // Bessel functions: type 1 order k; type 2 orders k - 1, k + 1
  double w;          // the pair's frequency
  long long off;     // position of the row's first integral
  int lo, P, pad;    // the k's first row, pairs and padded rows
  unsigned char mask, h[3];  // TRIANGBREIT mask; heads by operator (k_br_heads)
};

struct BrEnt {  // up to BR_NC columns of one bucket
  int lo, P, pad, m, h, set, nc, col[BR_NC];
  long long xt, kv, g;  // offsets: tail vectors, class terms, output block
};

struct BrBucket {
  int lo, P, pad, m, h, set;
  long long xt, kv;
};

// the arrays [point][pitch] over all rows: densities, operators (e, q) of the
// chains (0, 1: the terms with RPOR weights, 2: SKINT's second form), forward
// vectors F, class sums S of q rho up to M0 and the base vectors by set and head
struct BrArr {
  double *rho, *e[3], *q[3], *F[2], *S[3], *base[2][3];
  int pitch, maxm, m0, j0, type;
};

__device__ __forceinline__ double br_pat(const QuadConst &q, int ph) {
  ph &= 3;
  return (ph & 1) ? q.C2 : (ph == 2) ? q.C3 : q.C4;
}

// QUAD's weight of point i for head h and last point mq
__device__ __forceinline__ double br_w(const QuadConst &q, int i, int h, int mq) {
  if (i < h) return 0.0;
  if (i == h) return q.C1;
  const double w = br_pat(q, i - h);
  return (i == mq && ((mq - h) & 3) == 0) ? w - q.C1 : w;
}

// densities by pair [nw * nw][np] (P_a Q_b on 2..MTP) for the columns
__global__ void k_br_rho(int nw, const double *__restrict__ PF, const double *__restrict__ QF, int ld,
                         const int *__restrict__ MF, int np, double *__restrict__ rho) {
  const int a = blockIdx.y + 1, b = blockIdx.x + 1;
  const int m = min(MF[a], MF[b]);
  double *r = rho + ((size_t)(a - 1) * nw + (b - 1)) * np;
  for (int i = threadIdx.x; i < np; i += blockDim.x)
    r[i] = (i >= 2 && i <= m) ? pfv(PF, ld, i, a) * pfv(QF, ld, i, b) : 0.0;
}

// the head index each pair's chain gives as a source, from the signs of its
// first values: operator 0 (type 1: Z_k; type 2 at a frequency: the leading
// r^2 order of SKINT's first term), 1 (SKINT at zero frequency), 2 (SKINT's
// second term, Z_{k+1}); 2 where none of 2..4 qualifies (the entry's own
// check then sends it to the term by term form)
__global__ void k_br_heads(BrRow *__restrict__ rows, int nrows, int type, const double *__restrict__ rho, int nw,
                           int np, const double *__restrict__ R, const double *__restrict__ RP,
                           const double *__restrict__ Pow, QuadConst q, unsigned char *__restrict__ out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrows) return;
  const BrRow b = rows[r];
  unsigned char h[3] = {2, 2, 2};
  if (b.a) {
    const double *p = rho + ((size_t)(b.a - 1) * nw + (b.b - 1)) * np;
    auto pw = [&](int k, int i) { return k > 0 ? Pow[(size_t)k * np + i] : k < 0 ? Pow[i] : 1.0; };
    // Z(2..5) of order k over src(i)
    auto chain = [&](int k, int extra, double *z) {
      double t[4];
      for (int i = 2; i <= 5; ++i) {
        t[i - 2] = RP[i] * pw(k, i) * p[i];
        if (extra) t[i - 2] = t[i - 2] * (R[i] * R[i]);
      }
      for (int s = 0; s < 3; ++s) {
        z[s] = 0.0;
        for (int c = 0; c < 4; ++c) z[s] = z[s] + q.CNC5C[c][s] * t[c];
      }
      z[3] = q.C1 * t[3] + q.C2 * (t[0] + t[2]) + q.C3 * t[1];
    };
    auto head = [&](const double *z) {
      for (int i = 0; i < 3; ++i)
        if (z[i] != 0.0 && ((z[i] > 0.0 && z[i + 1] > 0.0) || (z[i] < 0.0 && z[i + 1] < 0.0)))
          return (unsigned char)(i + 2);
      return (unsigned char)2;
    };
    double za[4], zb[4], d[4];
    if (type == 1) {
      chain(b.K, 0, za);
      h[0] = head(za);
    } else {
      chain(b.K - 1, 0, za);
      chain(b.K - 1, 1, zb);
      for (int i = 0; i < 4; ++i) d[i] = zb[i] - (R[i + 2] * R[i + 2]) * za[i];
      h[0] = head(d);
      chain(b.K + 1, 0, zb);
      h[2] = head(zb);
      for (int i = 0; i < 4; ++i) d[i] = zb[i] / pw(b.K + 1, i + 2) - za[i] / pw(b.K - 1, i + 2);
      h[1] = head(d);
    }
  }
  for (int t = 0; t < 3; ++t) {
    rows[r].h[t] = h[t];
    out[(size_t)3 * r + t] = h[t];
  }
}

// densities and operators per (row, point)
__global__ void k_br_elem(const BrRow *__restrict__ rows, BrArr A, const double *__restrict__ rhop, int nw, int np,
                          const double *__restrict__ R, const double *__restrict__ RP,
                          const double *__restrict__ RPOR, const double *__restrict__ Pow,
                          const double *__restrict__ BJ, const double *__restrict__ BN) {
  const int r = blockIdx.x * 32 + threadIdx.x;
  const BrRow b = rows[r];
  for (int i = blockIdx.y * blockDim.y + threadIdx.y; i <= A.maxm; i += gridDim.y * blockDim.y) {
    const size_t at = (size_t)i * A.pitch + r;
    double rho = 0.0, e0 = 0.0, e1 = 0.0, e2 = 0.0, q0 = 0.0, q1 = 0.0, q2 = 0.0;
    if (b.a && i >= 2) {
      rho = rhop[((size_t)(b.a - 1) * nw + (b.b - 1)) * np + i];
      const int K = b.K;
      // r^k and 1 / r^k, k = -1 .. KLIM
      auto up = [&](int k) { return k > 0 ? Pow[(size_t)k * np + i] : k < 0 ? Pow[i] : 1.0; };
      auto dn = [&](int k) { return k > 0 ? Pow[(size_t)(KLIM + 1 + k) * np + i] : k < 0 ? R[i] : 1.0; };
      if (A.type == 1) {
        const double bj = b.fa >= 0 ? BJ[(size_t)b.fa * np + i] : 0.0, bn = b.fa >= 0 ? BN[(size_t)b.fa * np + i] : 0.0;
        e0 = RP[i] * up(K) * (1.0 + bj);
        q0 = (1.0 + bn) * RPOR[i] * dn(K);
      } else {
        const double ra = RP[i] * up(K - 1), rb = RP[i] * up(K + 1), da = dn(K - 1), db = dn(K + 1);
        const double WK = (double)(K + K + 1);
        if (fabs(b.w) < 1.0e-10) {
          // WK / 2 part RPOR (Z_{k+1} - Z_{k-1})
          e0 = rb;
          q0 = 0.5 * WK * RPOR[i] * db;
          e1 = ra;
          q1 = -0.5 * WK * RPOR[i] * da;
        } else {
          const double j1 = b.fa >= 0 ? BJ[(size_t)b.fa * np + i] : 0.0, n1 = b.fa >= 0 ? BN[(size_t)b.fa * np + i] : 0.0;
          const double j2 = b.fb >= 0 ? BJ[(size_t)b.fb * np + i] : 0.0, n2 = b.fb >= 0 ? BN[(size_t)b.fb * np + i] : 0.0;
          const double wr = WK / b.w, al = wr * wr * RPOR[i] / (R[i] * R[i]) * da;
          e0 = -ra * j1;
          q0 = al * (1.0 + n2);
          e1 = ra;
          q1 = -al * n2;
          e2 = rb * (1.0 + j2);
          q2 = -(b.w * b.w / (double)((2 * K + 3) * (2 * K - 1))) * (1.0 + n1) * R[i] * RP[i] * db;
        }
      }
    }
    A.rho[at] = rho;
    A.e[0][at] = e0;
    A.q[0][at] = q0;
    if (A.type == 2) {
      A.e[1][at] = e1;
      A.q[1][at] = q1;
      A.e[2][at] = e2;
      A.q[2][at] = q2;
    }
  }
}

// the forward vectors F = sum_chains q Z[e rho] (task 0: operator 0 (+ 1),
// task 1: operator 2) and the backward class sums S(i) = sum q rho over i, i +
// 4, .. <= M0 (tasks 2..: chain t - 2). A block takes 32 rows; a warp one
// residue class and one of BR_SEG runs of its points: it adds its run, the
// runs' sums are added through shared memory, and the second pass shifts it.
// One thread per (row, class) walking all points took 257 us for 16 subshells
// (three dependent loads and an addition per step, few warps), this 24 us.
constexpr int BR_SEG = 8;
__global__ void __launch_bounds__(32 * BR_SEG) k_br_chains(const BrRow *__restrict__ rows, BrArr A, QuadConst q) {
  __shared__ double tot[BR_SEG][32];
  const int lane = threadIdx.x, cls = blockIdx.z, seg = threadIdx.y;
  const int r = blockIdx.x * 32 + lane;
  const int nfwd = A.type == 1 ? 1 : 2;
  const int task = blockIdx.y, s = cls + 2;
  const size_t p = A.pitch;
  const double *rho = A.rho + r;
  const bool fwd = task < nfwd;
  const int end = fwd ? A.maxm : A.m0;
  const int steps = (end - s) / 4 + 1, run = (steps + BR_SEG - 1) / BR_SEG;
  const int c0 = fwd ? (task == 0 ? 0 : 2) : task - nfwd, nch = (task == 0 && A.type == 2) ? 2 : 1;
  const int mt = fwd ? rows[r].mtp : A.m0;
  for (int c = c0; c < c0 + nch; ++c) {
    const double *e = A.e[c] + r, *qq = A.q[c] + r;
    double *out = fwd ? A.F[task] + r : A.S[c] + r;
    // the second chain's own sums wait in a base plane, written later
    double *part = c > c0 ? A.base[0][0] + r : out;
    double v = 0.0;
    if (fwd) {
      auto t = [&](int j) { return __ldg(e + j * p) * __ldg(rho + j * p); };
      for (int u = seg * run; u < min(steps, (seg + 1) * run); ++u) {
        const int i = s + 4 * u;
        if (i <= mt) {
          if (i <= 4) {
            for (int k = 2; k <= 5; ++k) v = fma(q.CNC5C[k - 2][i - 2], t(k), v);
          } else {
            v = v + fma(q.C1, t(i - 4) + t(i), fma(q.C2, t(i - 3) + t(i - 1), q.C3 * t(i - 2)));
          }
        }
        part[i * p] = v;
      }
    } else {
      for (int u = min(steps, (seg + 1) * run) - 1; u >= seg * run; --u) {
        const int i = s + 4 * u;
        v = fma(__ldg(qq + i * p), __ldg(rho + i * p), v);
        part[i * p] = v;
      }
    }
    tot[seg][lane] = v;
    __syncthreads();
    double off = 0.0;
    if (fwd)
      for (int g = 0; g < seg; ++g) off = off + tot[g][lane];
    else
      for (int g = BR_SEG - 1; g > seg; --g) off = off + tot[g][lane];
    for (int u = seg * run; u < min(steps, (seg + 1) * run); ++u) {
      const int i = s + 4 * u;
      const double z = part[i * p] + off;
      if (!fwd)
        out[i * p] = z;
      else
        out[i * p] = i <= mt ? fma(__ldg(qq + i * p), z, c > c0 ? out[i * p] : 0.0) : 0.0;
    }
    __syncthreads();
  }
}

// adjoint chains of a set: type 1: 0; type 2 set 0 (source's frequency first
// pair): 2; set 1: 0 and 1
__device__ __forceinline__ int br_adj(int type, int set, int &first) {
  first = (type == 2 && set == 0) ? 2 : 0;
  return (type == 2 && set == 1) ? 2 : 1;
}
// operator whose head a row's forward vector has, -1: no forward vector
__device__ __forceinline__ int br_fwd(int type, int set, const BrRow &b) {
  const bool zero = type == 2 && fabs(b.w) < 1.0e-10;
  if (type == 1) return 0;
  if (set == 0) return zero ? 1 : 0;
  return zero ? -1 : 2;
}

// the transposed chain's weights times QUAD's: a point j >= 6 takes
// sum_t w[(j - h) & 3][t] S(j + t)
struct BrFold {
  double w[4][5];
};

// base vectors: the transposed chains cut at M0, by assumed head of the
// column, plus the weighted forward vector; points 2..J0
__global__ void k_br_base(const BrRow *__restrict__ rows, BrArr A, QuadConst q, BrFold fold) {
  const int r = blockIdx.x * 32 + threadIdx.x, set = blockIdx.z;
  const BrRow b = rows[r];
  const size_t p = A.pitch;
  int c0;
  const int nch = br_adj(A.type, set, c0);
  const int fo = b.a ? br_fwd(A.type, set, b) : -1;
  for (int j = 2 + blockIdx.y * blockDim.y + threadIdx.y; j <= A.j0; j += gridDim.y * blockDim.y) {
    const double f = fo < 0 ? 0.0 : br_w(q, j, b.h[fo], 0) * __ldg(A.F[set] + j * p + r);
    double x[3] = {f, f, f};
    for (int c = c0; c < c0 + nch; ++c) {
      const double *S = A.S[c] + r;
      const double e = __ldg(A.e[c] + j * p + r);
      if (j >= 6) {
        double sv[5];
#pragma unroll
        for (int t = 0; t < 5; ++t) sv[t] = __ldg(S + (j + t) * p);
#pragma unroll
        for (int h = 2; h <= 4; ++h) {
          const double *w = fold.w[(j - h) & 3];
          double v = w[0] * sv[0];
#pragma unroll
          for (int t = 1; t < 5; ++t) v = fma(w[t], sv[t], v);
          x[h - 2] = fma(e, v, x[h - 2]);
        }
      } else {
        for (int h = 2; h <= 4; ++h) {
          auto sw = [&](int i) {  // suffix sum of the class of i with QUAD's weights
            if (i > h) return br_pat(q, i - h) * S[i * p];
            if (i == h) return q.C4 * S[i * p] - q.C1 * (A.q[c][i * p + r] * A.rho[i * p + r]);
            return br_pat(q, i + 4 - h) * S[(i + 4) * p];
          };
          double v = 0.0;
          for (int i = 2; i <= 4; ++i) v = fma(q.CNC5C[j - 2][i - 2], sw(i), v);
          for (int i = 5; i <= j + 4; ++i) {
            const int dlt = i - j;
            v = fma((dlt == 0 || dlt == 4) ? q.C1 : dlt == 2 ? q.C3 : q.C2, sw(i), v);
          }
          x[h - 2] = fma(e, v, x[h - 2]);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < 3; ++h) A.base[set][h][j * p + r] = x[h];
  }
}

// a bucket's own part: the vectors of the points J0 < j <= m and the class
// terms K of the points up to J0 (8 per chain: j = 2..5, then j mod 4). One
// thread per (row, bucket), the transposed chain run backwards in registers
__global__ void k_br_tail(const BrBucket *__restrict__ bk, const BrRow *__restrict__ rows, BrArr A, QuadConst q,
                          double *__restrict__ xt, double *__restrict__ kv) {
  const BrBucket B = bk[blockIdx.x];
  const int l = blockIdx.y * blockDim.x + threadIdx.x;
  if (l >= B.pad) return;
  const int r = B.lo + l;
  const BrRow b = rows[r];
  const size_t p = A.pitch;
  const int m = B.m, h = B.h, mq = b.a ? min(m, (int)b.mtp) : 0;
  int c0;
  const int nch = br_adj(A.type, B.set, c0);
  const int fo = b.a ? br_fwd(A.type, B.set, b) : -1;
  const int tl = (m - A.j0 + 1) & ~1;
  double *X = xt + B.xt + l;
  double *Kv = kv + B.kv + l;
  if (tl > m - A.j0) X[(size_t)(tl - 1) * B.pad] = 0.0;
  // S(j), S(j+1), S(j+2), S(j+3) of each chain
  double s0[2] = {0.0, 0.0}, s1[2] = {0.0, 0.0}, s2[2] = {0.0, 0.0}, s3[2] = {0.0, 0.0};
#pragma unroll 4
  for (int j = m; j > A.j0; --j) {
    double x = 0.0;
    if (j <= mq) {
      const double rho = __ldg(A.rho + j * p + r), w = br_w(q, j, h, mq) * rho;
      for (int c = 0; c < nch; ++c) {
        const double o = s3[c], n = fma(w, __ldg(A.q[c0 + c] + j * p + r), o);
        const double v = fma(q.C1, n + o, fma(q.C2, s0[c] + s2[c], q.C3 * s1[c]));
        s3[c] = s2[c];
        s2[c] = s1[c];
        s1[c] = s0[c];
        s0[c] = n;
        x = fma(__ldg(A.e[c0 + c] + j * p + r), v, x);
      }
      if (fo >= 0) x = fma(br_w(q, j, b.h[fo], mq), __ldg(A.F[B.set] + j * p + r), x);
    }
    X[(size_t)(j - A.j0 - 1) * B.pad] = x;
    if (j == A.m0 + 1 || (m == A.m0 && j == m)) {
      // class sums of the points beyond M0: D[i & 3]
      for (int c = 0; c < nch; ++c) {
        double D[4] = {0.0, 0.0, 0.0, 0.0};
        if (m > A.m0) {
          D[j & 3] = s0[c];
          D[(j + 1) & 3] = s1[c];
          D[(j + 2) & 3] = s2[c];
          D[(j + 3) & 3] = s3[c];
        }
        // QUAD's last point is M0 itself, which the base weights as an inner one
        if (mq == A.m0 && ((mq - h) & 3) == 0) D[mq & 3] = -q.C1 * (A.q[c0 + c][mq * p + r] * A.rho[mq * p + r]);
        for (int t = 2; t <= 5; ++t) {
          double v = 0.0;
          for (int i = 2; i <= 4; ++i) v = fma(q.CNC5C[t - 2][i - 2], D[i & 3], v);
          for (int i = 5; i <= t + 4; ++i) {
            const int dlt = i - t;
            v = fma((dlt == 0 || dlt == 4) ? q.C1 : dlt == 2 ? q.C3 : q.C2, D[i & 3], v);
          }
          Kv[(size_t)(8 * c + t - 2) * B.pad] = v;
        }
        for (int t = 0; t < 4; ++t)
          Kv[(size_t)(8 * c + 4 + t) * B.pad] =
              2.0 * q.C1 * D[t] + q.C2 * (D[(t + 1) & 3] + D[(t + 3) & 3]) + q.C3 * D[(t + 2) & 3];
      }
    }
  }
}

// QUAD's head term from TA(h), TA(h+1); *ok is cleared where h is not QUAD's
// head index (the test at h fails, or one before it passes)
__device__ __forceinline__ double br_head(const double *ta, int h, const double *HD, int np, bool *ok) {
  bool good = true;
  double res = 0.0;
#pragma unroll
  for (int i = 2; i <= 4; ++i) {
    const double t0 = ta[i - 2], t1 = ta[i - 1];
    if (i < h) {
      if ((t0 > 0.0 && t1 > 0.0) || (t0 < 0.0 && t1 < 0.0) || t0 != t0 || t1 != t1) good = false;
    } else if (i == h) {
      const double t = t1 / t0;
      if (fabs(t0) > 0.0 && t > 0.0) {
        const double sigma = log(t * HD[np + h]) * HD[h];
        res = (t0 * HD[2 * np + h]) / (sigma + 1.0);
      } else {
        good = false;
      }
    }
  }
  if (!good) *ok = false;
  return res;
}

// One block: 32 rows x NC columns of one bucket, the points shared out among
// its four warps (a set of few pairs has too few warps otherwise: 239 us with
// a warp per tile, 76 us so, 16 subshells). Per point the row's vector value
// is formed (base + e K, or the tail's) and multiplied into NC accumulators:
// 1 + NC (2 + NC with two chains) FP64 instructions, the columns' densities
// read uniformly. The warps' sums meet in shared memory; each warp then adds
// the head contributions of its columns.
template <int NC, int NCH>
__device__ __forceinline__ void br_gemm(const BrEnt &E, int lane, int warp, double (*red)[BR_NC][32],
                                        const BrRow *__restrict__ rows, const BrArr &A, int c0,
                                        const double *__restrict__ rhop, int nw, int np,
                                        const double *__restrict__ xt, const double *__restrict__ kv,
                                        const double *__restrict__ HD, const QuadConst &q, double *__restrict__ G) {
  const int l = blockIdx.y * 32 + lane, r = E.lo + l;
  const size_t p = A.pitch;
  const double *e0 = A.e[c0] + r, *e1 = A.e[c0 + NCH - 1] + r;
  const double *rc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const BrRow cr = rows[E.lo + E.col[c]];
    rc[c] = rhop + ((size_t)(cr.a - 1) * nw + (cr.b - 1)) * np;
  }
  {
    const double *B = A.base[E.set][E.h - 2] + r;
    const double *Kv = kv + E.kv + l;
    double K[NCH][4], acc[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = 0.0;
    auto add2 = [&](int j, double xa, double xb) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double2 v = __ldg(reinterpret_cast<const double2 *>(rc[c] + j));
        acc[c] = fma(xa, v.x, acc[c]);
        acc[c] = fma(xb, v.y, acc[c]);
      }
    };
    auto step = [&](int j) {  // points j .. j + 3 with the class terms K[..][0..3]
      double x[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const size_t o = (size_t)(j + t) * p;
        x[t] = fma(__ldg(e0 + o), K[0][t], __ldg(B + o));
        if (NCH == 2) x[t] = fma(__ldg(e1 + o), K[NCH - 1][t], x[t]);
      }
      add2(j, x[0], x[1]);
      add2(j + 2, x[2], x[3]);
    };
    if (warp == 0) {
#pragma unroll
      for (int c = 0; c < NCH; ++c)
#pragma unroll
        for (int t = 0; t < 4; ++t) K[c][t] = Kv[(size_t)(8 * c + t) * E.pad];
      step(2);
    }
#pragma unroll
    for (int c = 0; c < NCH; ++c)
#pragma unroll
      for (int t = 0; t < 4; ++t) K[c][t] = Kv[(size_t)(8 * c + 4 + ((6 + t) & 3)) * E.pad];
#pragma unroll 4
    for (int j = 6 + 4 * warp; j < A.j0; j += 16) step(j);
    const double *X = xt + E.xt + l;
    const int tl = (E.m - A.j0 + 1) & ~1;
#pragma unroll 4
    for (int t = 2 * warp; t < tl; t += 8)
      add2(A.j0 + 1 + t, __ldg(X + (size_t)t * E.pad), __ldg(X + (size_t)(t + 1) * E.pad));
#pragma unroll
    for (int c = 0; c < NC; ++c) red[warp][c][lane] = acc[c];
  }
  __syncthreads();
  if (l >= E.P) return;
  const BrRow b = rows[r];
  const int fo = br_fwd(A.type, E.set, b);
  const bool adj = A.type == 1 || E.set == 1 || fo == 0;  // set 0 at zero frequency has no second term
  for (int c = warp; c < NC; c += 4) {
    double v = (red[0][c][lane] + red[1][c][lane]) + (red[2][c][lane] + red[3][c][lane]), s[4], ta[4];
    bool ok = true;
    const BrRow cr = rows[E.lo + E.col[c]];
    const double *rs = rhop + ((size_t)(cr.a - 1) * nw + (cr.b - 1)) * np;
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] = rs[i + 2];
    if (fo >= 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) ta[i] = __ldg(A.F[E.set] + (i + 2) * p + r) * s[i];
      v += br_head(ta, b.h[fo], HD, np, &ok);
    }
    if (adj) {
#pragma unroll
      for (int i = 0; i < 4; ++i) ta[i] = 0.0;
#pragma unroll
      for (int u = 0; u < NCH; ++u) {
        const double *ee = u ? e1 : e0;
        double t[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = __ldg(ee + (i + 2) * p) * s[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i > E.h - 1) continue;  // TA(h + 1) is the last one read
          double z;
          if (i < 3)
            z = fma(q.CNC5C[3][i], t[3], fma(q.CNC5C[2][i], t[2], fma(q.CNC5C[1][i], t[1], q.CNC5C[0][i] * t[0])));
          else
            z = fma(q.C3, t[1], fma(q.C2, t[0] + t[2], q.C1 * t[3]));
          ta[i] = fma(__ldg(A.q[c0 + u] + (i + 2) * p + r) * __ldg(A.rho + (i + 2) * p + r), z, ta[i]);
        }
      }
      v += br_head(ta, E.h, HD, np, &ok);
    }
    G[E.g + (size_t)E.col[c] * E.pad + l] = ok ? v : __longlong_as_double(0x7ff8000000000000ll);
  }
}

template <int NCH>
__global__ void __launch_bounds__(128) k_br_gemm(const BrEnt *__restrict__ ents, const BrRow *__restrict__ rows,
                                                 BrArr A, int c0, const double *__restrict__ rhop, int nw, int np,
                                                 const double *__restrict__ xt, const double *__restrict__ kv,
                                                 const double *__restrict__ HD, QuadConst q, double *__restrict__ G) {
  __shared__ double red[4][BR_NC][32];
  __shared__ BrEnt E;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) E = ents[blockIdx.x];
  __syncthreads();
  if ((int)blockIdx.y * 32 >= E.pad) return;
  switch (E.nc) {
#define BR_CASE(N) \
  case N: br_gemm<N, NCH>(E, lane, warp, red, rows, A, c0, rhop, nw, np, xt, kv, HD, q, G); break;
    BR_CASE(1) BR_CASE(2) BR_CASE(3) BR_CASE(4) BR_CASE(5) BR_CASE(6) BR_CASE(7) BR_CASE(8)
#undef BR_CASE
  }
}

// the integrals: row (k, a, b) x column (c, d), half the sum of the two
// orders, at the row's position plus the column's rank among those the row's
// mask admits; a value that is not a number (an entry marked by k_br_gemm, or
// inputs that are not finite) goes to the term by term list
struct BrRedo {
  long long pos;
  int row, col;
};
__global__ void k_br_table(const BrRow *__restrict__ rows, const int *__restrict__ rank, const double *__restrict__ G1,
                           const double *__restrict__ G2, const long long *__restrict__ g0, int KEY,
                           int32_t *__restrict__ ind, double *__restrict__ val, BrRedo *__restrict__ redo,
                           int *__restrict__ nredo) {
  const int r = blockIdx.x;
  const BrRow b = rows[r];
  if (!b.a) return;
  const int l = r - b.lo;
  const long long g = g0[b.K];
  const int *rk = rank + (size_t)8 * b.lo + (size_t)b.mask * b.pad;
  for (int s = threadIdx.x; s < b.P; s += blockDim.x) {
    const BrRow c = rows[b.lo + s];
    if (!(b.mask & c.mask)) continue;
    const double v = G1 ? 0.5 * (G1[g + (size_t)s * b.pad + l] + G2[g + (size_t)l * b.pad + s])
                        : __longlong_as_double(0x7ff8000000000000ll);
    const long long pos = b.off + rk[s];
    ind[pos] = ((b.a * KEY + b.b) * KEY + c.a) * KEY + c.b;
    val[pos] = v;
    if (v != v) redo[atomicAdd(nredo, 1)] = BrRedo{pos, r, b.lo + s};
  }
}

// an entry of the table term by term: one thread per (entry, term), 2^tsh terms
// to an entry (4, or 2 in a type 2 table without a frequency, whose warps would
// be half empty: 15.4 ms for 120,818 entries, 8.4 so), then the
// combination. A launch takes up to BR_REDO entries of the list: enough threads
// for many waves, 4 n and a thread's index stay ints whatever the table's size
// (up to 2^31 - 1 integrals), and the terms' values take 17 MB instead of 32
// bytes for every entry of the list.
constexpr int BR_REDO = 1 << 19;
static_assert(4LL * BR_REDO + 128 <= INT32_MAX, "k_br_redo's thread index is an int");
__global__ void __launch_bounds__(128) k_br_redo(int type, int tsh, const BrRedo *__restrict__ redo, int n,
                                                 const BrRow *__restrict__ rows, PlanTabs T, TermTabs tt, QuadConst q,
                                                 double *__restrict__ v, BrInt *__restrict__ ints) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t >> tsh, u = t & ((1 << tsh) - 1);
  if (i >= n) return;
  const BrRedo e = redo[i];
  const BrRow a = rows[e.row], c = rows[e.col];
  BrJob jb[4];
  BrInt bi;
  const int k = plan_one(type, a.a, a.b, c.a, c.b, a.K, T, i << tsh, &bi, jb);
  if (u == 0) ints[i] = bi;
  if (u < k) v[t] = breit_term(jb[u], tt, q);
}

__global__ void k_br_redo_store(const BrRedo *__restrict__ redo, int n, const double *__restrict__ v,
                                double *__restrict__ val) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) val[redo[t].pos] = v[t];
}

template <class T> int upload_vec(DBuf<T> &b, const std::vector<T> &h, cudaStream_t s) {
  GG_TRY(b.alloc(std::max<size_t>(1, h.size())));
  if (!h.empty()) GG_CUDA(cudaMemcpyAsync(b.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s));
  return GG_OK;
}

// the host side of a plan: the frequencies, the Bessel functions the
// integrals read (pair, order) with their ids, on the device
struct Plan {
  gg_ctx *ctx = nullptr;
  int nw = 0;
  double wfact = 0, epsi = 0;
  std::vector<double> e, W;
  std::vector<int> bid;  // [order + 1][lo][hi]
  std::vector<BessDesc> bess;
  DBuf<double> dW;
  DBuf<int> dbid;
  int norders() const { return KLIM + 3; }
  int &slot(int x, int y, int nn) {
    const int lo = std::min(x, y), hi = std::max(x, y);
    return bid[((size_t)(nn + 1) * nw + (lo - 1)) * nw + (hi - 1)];
  }
  void need(int x, int y, int nn) {
    int &s = slot(x, y, nn);
    if (s != -2) return;
    const double w = W[(size_t)(x - 1) * nw + (y - 1)];
    if (w < epsi * epsi) {
      s = -1;
    } else {
      s = (int)bess.size();
      bess.push_back(BessDesc{w, nn});
    }
  }
  int upload(cudaStream_t s) {
    for (int &v : bid)
      if (v == -2) v = -1;
    GG_TRY(upload_vec(dW, W, s));
    GG_TRY(upload_vec(dbid, bid, s));
    return GG_OK;
  }
  int id(int x, int y, int nn) const {
    const int lo = std::min(x, y), hi = std::max(x, y);
    return bid[((size_t)(nn + 1) * nw + (lo - 1)) * nw + (hi - 1)];
  }
  PlanTabs tabs() const { return PlanTabs{dW.p, dbid.p, nw}; }
};

int make_plan(gg_ctx *ctx, double wfact, const double *e, double accy, Plan &P) {
  GG_TRY(ensure_orbitals(ctx));
  const Orbitals &o = ctx->orb;
  if (!e) return fail(GG_ERR_ARG, "Breit integrals: orbital energies required");
  if (o.nw > 214) return fail(GG_ERR_ARG, "Breit integrals: more than 214 orbitals");
  P.ctx = ctx;
  P.nw = o.nw;
  P.wfact = wfact;
  P.epsi = std::sqrt(0.1 * (accy > 0 ? accy : std::pow(ctx->grid.h, 6)));
  P.e.assign(e, e + o.nw);
  P.W.assign((size_t)o.nw * o.nw, 0.0);
  for (int x = 1; x <= o.nw; ++x)
    for (int y = 1; y <= o.nw; ++y)
      P.W[(size_t)(x - 1) * o.nw + (y - 1)] = wfact * std::fabs(e[x - 1] - e[y - 1]) / ctx->grid.c;
  P.bid.assign((size_t)P.norders() * o.nw * o.nw, -2);
  return GG_OK;
}

// the Bessel functions, the terms and the combinations; values into out
// (host, ni integrals); *kernel_ms: device time of these kernels
int run_terms(gg_ctx *ctx, const Plan &P, const BrJob *djobs, int64_t nj, const BrInt *dints, int64_t ni,
              double *out, double *kernel_ms = nullptr) {
  const Grid &g = ctx->grid;
  const Orbitals &o = ctx->orb;
  cudaStream_t s = ctx->stream;
  const int nb = (int)P.bess.size();
  DBuf<BessDesc> dbd;
  DBuf<double> dBJ, dBN, dv, dout;
  GG_TRY(upload_vec(dbd, P.bess, s));
  GG_TRY(dBJ.alloc((size_t)std::max(1, nb) * g.np));
  GG_TRY(dBN.alloc((size_t)std::max(1, nb) * g.np));
  GG_TRY(dv.alloc(std::max<int64_t>(1, nj)));
  GG_TRY(dout.alloc(std::max<int64_t>(1, ni)));
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (kernel_ms) {
    GG_CUDA(cudaEventCreate(&e0));
    GG_CUDA(cudaEventCreate(&e1));
    GG_CUDA(cudaEventRecord(e0, s));
  }
  if (nb > 0) {
    k_bessel<<<nb, 128, 0, s>>>(dbd.p, g.dR.p, g.n, g.np, P.epsi, dBJ.p, dBN.p);
    ::gg::note_launch();
  }
  if (nj > 0) {
    const TermTabs tt{o.dPF.p, o.dQF.p, o.ld, o.dMF.p, g.dR.p, g.dRP.p, g.dRPOR.p, g.dPow.p, g.np, dBJ.p, dBN.p};
    k_breit_jobs<<<(unsigned)((nj + 127) / 128), 128, 0, s>>>(djobs, nj, tt, g.q, dv.p);
    ::gg::note_launch();
  }
  if (ni > 0) {
    k_breit_combine<<<(unsigned)((ni + 255) / 256), 256, 0, s>>>(dints, ni, dv.p, dout.p);
    ::gg::note_launch();
  }
  GG_CUDA(cudaGetLastError());
  if (kernel_ms) GG_CUDA(cudaEventRecord(e1, s));
  if (ni > 0) GG_CUDA(cudaMemcpyAsync(out, dout.p, ni * sizeof(double), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));
  if (kernel_ms) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    *kernel_ms = ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }
  return GG_OK;
}

// the tables' contraction: rows, operators, buckets and the dense products
int run_table(gg_ctx *ctx, int type, const Plan &P, int j2max, const std::vector<unsigned char> &mask, BreitTable &T,
              double *plan_ms, double *kernel_ms) {
  const Grid &g = ctx->grid;
  const Orbitals &o = ctx->orb;
  cudaStream_t s = ctx->stream;
  const int nw = o.nw, KEY = nw + 1, np = g.np;
  const size_t msz = (size_t)(nw + 1) * (nw + 1);
  const auto th0 = std::chrono::steady_clock::now();
  *plan_ms = *kernel_ms = 0.0;
  // rows: the admitted pairs of each k in (a, b) order, padded to whole warps
  std::vector<BrRow> rows;
  std::vector<int> lo(j2max + 2, 0), cnt(j2max + 1, 0);
  std::vector<long long> g0(j2max + 1, 0);
  std::vector<int> rank;
  long long ni = 0, nj = 0, gsz = 0;
  T.kstart.assign(j2max + 2, 1);
  int maxm = 0, m0 = INT32_MAX;
  for (int x = 1; x <= nw; ++x) {
    maxm = std::max(maxm, o.mf[x]);
    m0 = std::min(m0, o.mf[x]);
  }
  for (int K = 0; K <= j2max; ++K) {
    const unsigned char *mk = mask.data() + (size_t)K * msz;
    lo[K] = (int)rows.size();
    for (int a = 1; a <= nw; ++a)
      for (int b = 1; b <= nw; ++b)
        if (mk[a * (nw + 1) + b]) {
          BrRow r{};
          r.a = (short)a;
          r.b = (short)b;
          r.K = (short)K;
          r.mtp = std::min(o.mf[a], o.mf[b]);
          r.fa = P.id(a, b, type == 1 ? K : K - 1);
          r.fb = type == 1 ? -1 : P.id(a, b, K + 1);
          r.w = P.W[(size_t)(a - 1) * nw + (b - 1)];
          r.mask = mk[a * (nw + 1) + b];
          rows.push_back(r);
        }
    const int np_ = cnt[K] = (int)rows.size() - lo[K];
    while (rows.size() % 32) rows.push_back(BrRow{});
    const int pad = (int)rows.size() - lo[K];
    g0[K] = gsz;
    gsz += (long long)pad * pad;
    // positions: rank of a column among those a row's mask admits
    rank.resize((size_t)8 * rows.size(), 0);
    int n[8] = {}, nz[8] = {};  // admitted columns by row mask; those at a frequency
    for (int c = 0; c < np_; ++c) {
      const BrRow &r = rows[lo[K] + c];
      for (int m = 1; m < 8; ++m) {
        rank[(size_t)8 * lo[K] + (size_t)m * pad + c] = n[m];
        if (m & r.mask) {
          ++n[m];
          nz[m] += std::fabs(r.w) >= 1.0e-10;
        }
      }
    }
    for (int c = lo[K]; c < (int)rows.size(); ++c) {
      BrRow &r = rows[c];
      r.lo = lo[K];
      r.P = np_;
      r.pad = pad;
      r.off = ni;
      if (!r.a) continue;
      ni += n[r.mask];
      // the terms of the row's integrals (plan_one), which bound the table
      const int own = type == 1 ? 2 : std::fabs(r.w) >= 1.0e-10 ? 2 : 1;
      nj += type == 1 ? 4LL * n[r.mask] : (long long)own * n[r.mask] + n[r.mask] + nz[r.mask];
      nj -= type == 1 ? (r.a == r.b ? 3 : 5) : (r.a == r.b ? own : 2 * own);
    }
    T.kstart[K + 1] = (int32_t)(ni + 1);
  }
  if (ni > INT32_MAX || nj > INT32_MAX) return fail(GG_ERR_RANGE, "gg_genintbreit: table too large");
  T.n = ni;
  const int R = (int)rows.size();
  if (ni == 0) return GG_OK;
  // the contraction takes orbitals that reach past the chains' start and end
  // on the grid; any other set is evaluated term by term
  const bool plain = m0 >= BR_MIN_MF && maxm <= g.n;
  bool moving = false;  // some pair is at a frequency
  for (const BrRow &r : rows) moving |= r.a && std::fabs(r.w) >= 1.0e-10;

  // the operators, forward vectors and class sums need no buckets: they run
  // while the host builds these from the heads
  const int nch = type == 1 ? 1 : 3, nset = type == 1 ? 1 : 2;
  const size_t plane = plain ? (size_t)(maxm + 1) * R : 0;
  const int j0 = 5 + 4 * ((m0 - 9) / 4);
  DBuf<BrRow> drows;
  DBuf<double> drho, darr, dBJ, dBN, dG;
  DBuf<BessDesc> dbd;
  DBuf<unsigned char> dheads;
  DBuf<int> drank, dnredo;
  DBuf<long long> dg0;
  GG_TRY(upload_vec(drows, rows, s));
  GG_TRY(upload_vec(drank, rank, s));
  GG_TRY(upload_vec(dg0, g0, s));
  GG_TRY(upload_vec(dbd, P.bess, s));
  const int nb = (int)P.bess.size();
  GG_TRY(drho.alloc((size_t)nw * nw * np));
  GG_TRY(darr.alloc(plane * (size_t)(1 + 3 * nch + nset * 4)));
  GG_TRY(dBJ.alloc((size_t)std::max(1, nb) * np));
  GG_TRY(dBN.alloc((size_t)std::max(1, nb) * np));
  GG_TRY(dheads.alloc((size_t)3 * R));
  GG_TRY(dG.alloc(plain ? (size_t)gsz * nset : 0));
  GG_TRY(T.dInd.alloc(ni));
  GG_TRY(T.dVal.alloc(ni));
  GG_TRY(dnredo.alloc(1));
  BrArr A{};
  {
    double *p = darr.p;
    auto take = [&] {
      double *r = p;
      p += plane;
      return r;
    };
    A.rho = take();
    for (int c = 0; c < nch; ++c) {
      A.e[c] = take();
      A.q[c] = take();
      A.S[c] = take();
    }
    for (int t = 0; t < nset; ++t) {
      A.F[t] = take();
      for (int h = 0; h < 3; ++h) A.base[t][h] = take();
    }
    A.pitch = R;
    A.maxm = maxm;
    A.m0 = m0;
    A.j0 = j0;
    A.type = type;
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  GG_CUDA(cudaEventCreate(&e0));
  GG_CUDA(cudaEventCreate(&e1));
  struct Ev {
    cudaEvent_t a, b;
    ~Ev() {
      cudaEventDestroy(a);
      cudaEventDestroy(b);
    }
  } ev{e0, e1};
  GG_CUDA(cudaEventRecord(e0, s));
  GG_CUDA(cudaMemsetAsync(dnredo.p, 0, sizeof(int), s));
  k_br_rho<<<dim3(nw, nw), 128, 0, s>>>(nw, o.dPF.p, o.dQF.p, o.ld, o.dMF.p, np, drho.p);
  ::gg::note_launch();
  k_br_heads<<<(R + 127) / 128, 128, 0, s>>>(drows.p, R, type, drho.p, nw, np, g.dR.p, g.dRP.p, g.dPow.p, g.q,
                                            dheads.p);
  ::gg::note_launch();
  std::vector<unsigned char> heads((size_t)3 * R);
  GG_CUDA(cudaMemcpyAsync(heads.data(), dheads.p, heads.size(), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));  // the densities and heads, a few us of kernels
  if (nb > 0) {
    k_bessel<<<nb, 128, 0, s>>>(dbd.p, g.dR.p, std::min(maxm, g.n), np, P.epsi, dBJ.p, dBN.p);
    ::gg::note_launch();
  }
  DBuf<BrBucket> dbk;
  DBuf<BrEnt> dents;
  DBuf<double> dxt, dkv;
  if (plain) {
    k_br_elem<<<dim3(R / 32, (maxm + 32) / 32), dim3(32, 8), 0, s>>>(drows.p, A, drho.p, nw, np, g.dR.p, g.dRP.p,
                                                                    g.dRPOR.p, g.dPow.p, dBJ.p, dBN.p);
    ::gg::note_launch();
    k_br_chains<<<dim3(R / 32, nset + nch, 4), dim3(32, BR_SEG), 0, s>>>(drows.p, A, g.q);
    ::gg::note_launch();
    BrFold fold;
    for (int f = 0; f < 4; ++f) {
      const double pat[4] = {g.q.C4, g.q.C2, g.q.C3, g.q.C2}, inc[5] = {g.q.C1, g.q.C2, g.q.C3, g.q.C2, g.q.C1};
      for (int t = 0; t < 5; ++t) fold.w[f][t] = inc[t] * pat[(f + t) & 3];
    }
    k_br_base<<<dim3(R / 32, (j0 + 31) / 32, nset), dim3(32, 8), 0, s>>>(drows.p, A, g.q, fold);
    ::gg::note_launch();

    // buckets: the columns of each (set, k) by (MTP, head as a source)
    std::vector<BrBucket> bk;
    std::vector<BrEnt> ents;
    std::vector<int> cols;
    long long xt = 0, kv = 0;
    int maxpad = 0, split = 0;  // ents[0, split): set 0
    for (int set = 0; set < nset; ++set) {
      const int op = type == 1 ? 0 : set == 0 ? 2 : moving ? 0 : 1;
      const int ac = (type == 2 && set == 1) ? 2 : 1;
      for (int K = 0; K <= j2max; ++K) {
        const int n = cnt[K], pad = (K < j2max ? lo[K + 1] : R) - lo[K];
        if (n == 0) continue;
        maxpad = std::max(maxpad, pad);
        cols.resize(n);
        for (int c = 0; c < n; ++c) cols[c] = c;
        auto key = [&](int c) { return (int)rows[lo[K] + c].mtp * 8 + heads[(size_t)3 * (lo[K] + c) + op]; };
        std::stable_sort(cols.begin(), cols.end(), [&](int x, int y) { return key(x) > key(y); });
        for (int c = 0; c < n;) {
          int e = c;
          while (e < n && key(cols[e]) == key(cols[c])) ++e;
          const int m = rows[lo[K] + cols[c]].mtp, h = heads[(size_t)3 * (lo[K] + cols[c]) + op];
          bk.push_back(BrBucket{lo[K], n, pad, m, h, set, xt, kv});
          const int tiles = (e - c + BR_NC - 1) / BR_NC;
          for (int t = 0; t < tiles; ++t) {  // columns shared out evenly
            BrEnt E{};
            E.lo = lo[K];
            E.P = n;
            E.pad = pad;
            E.m = m;
            E.h = h;
            E.set = set;
            const int b0 = c + (e - c) * t / tiles, b1 = c + (e - c) * (t + 1) / tiles;
            E.nc = b1 - b0;
            for (int u = 0; u < E.nc; ++u) E.col[u] = cols[b0 + u];
            E.xt = xt;
            E.kv = kv;
            E.g = g0[K] + (long long)set * gsz;
            ents.push_back(E);
          }
          xt += (long long)((m - j0 + 1) & ~1) * pad;
          kv += 8LL * ac * pad;
          c = e;
        }
      }
      if (set == 0) split = (int)ents.size();
    }
    GG_TRY(upload_vec(dbk, bk, s));
    GG_TRY(upload_vec(dents, ents, s));
    GG_TRY(dxt.alloc((size_t)xt));
    GG_TRY(dkv.alloc((size_t)kv));
    const int yt = (maxpad + 127) / 128;
    k_br_tail<<<dim3((unsigned)bk.size(), yt), 128, 0, s>>>(dbk.p, drows.p, A, g.q, dxt.p, dkv.p);
    ::gg::note_launch();
    k_br_gemm<1><<<dim3((unsigned)split, maxpad / 32), 128, 0, s>>>(dents.p, drows.p, A, type == 1 ? 0 : 2, drho.p, nw, np, dxt.p,
                                                          dkv.p, g.dHead.p, g.q, dG.p);
    ::gg::note_launch();
    if (nset == 2) {
      k_br_gemm<2><<<dim3((unsigned)(ents.size() - split), maxpad / 32), 128, 0, s>>>(dents.p + split, drows.p, A, 0, drho.p, nw,
                                                                            np, dxt.p, dkv.p, g.dHead.p, g.q, dG.p);
      ::gg::note_launch();
    }
  }
  DBuf<BrRedo> dredo;
  GG_TRY(dredo.alloc(ni));
  k_br_table<<<R, 128, 0, s>>>(drows.p, drank.p, plain ? dG.p : nullptr, dG.p + (nset == 2 ? gsz : 0), dg0.p, KEY, T.dInd.p,
                               T.dVal.p, dredo.p, dnredo.p);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  *plan_ms = 1e3 * std::chrono::duration<double>(std::chrono::steady_clock::now() - th0).count();
  int nredo = 0;
  GG_CUDA(cudaMemcpyAsync(&nredo, dnredo.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));
  if (nredo > 0) {
    // k_bessel ran to the longest orbital, which covers every term
    DBuf<double> dv, dout;
    DBuf<BrInt> dints;
    const int piece = std::min(nredo, BR_REDO), tsh = type == 1 || moving ? 2 : 1;
    GG_TRY(dv.alloc((size_t)4 * piece));
    GG_TRY(dout.alloc(piece));
    GG_TRY(dints.alloc(piece));
    const TermTabs tt{o.dPF.p, o.dQF.p, o.ld, o.dMF.p, g.dR.p, g.dRP.p, g.dRPOR.p, g.dPow.p, np, dBJ.p, dBN.p};
    for (int done = 0; done < nredo;) {
      const int n = std::min(piece, nredo - done);
      const BrRedo *part = dredo.p + done;
      k_br_redo<<<((n << tsh) + 127) / 128, 128, 0, s>>>(type, tsh, part, n, drows.p, P.tabs(), tt, g.q, dv.p, dints.p);
      ::gg::note_launch();
      k_breit_combine<<<(n + 255) / 256, 256, 0, s>>>(dints.p, n, dv.p, dout.p);
      ::gg::note_launch();
      k_br_redo_store<<<(n + 255) / 256, 256, 0, s>>>(part, n, dout.p, T.dVal.p);
      ::gg::note_launch();
      GG_CUDA(cudaGetLastError());
      done += n;
    }
  }
  GG_CUDA(cudaEventRecord(e1, s));
  GG_CUDA(cudaStreamSynchronize(s));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  *kernel_ms = ms;
  return GG_OK;
}

// exclusive scan of counts into int64 offsets; returns the total
int64_t scan(const std::vector<int> &cnt, std::vector<int64_t> &off) {
  off.resize(cnt.size());
  int64_t t = 0;
  for (size_t i = 0; i < cnt.size(); ++i) {
    off[i] = t;
    t += cnt[i];
  }
  return t;
}

}  // namespace
}  // namespace gg

using namespace gg;

extern "C" {

int gg_genintbreit(gg_ctx *ctx, int type, double wfact, const double *e, double accy, int64_t *nb_out,
                   int *j2max_out) {
  if (!ctx || (type != 1 && type != 2)) return fail(GG_ERR_ARG, "gg_genintbreit: type 1 or 2");
  GG_CUDA(cudaSetDevice(ctx->device));
  Plan P;
  GG_TRY(make_plan(ctx, wfact, e, accy, P));
  GG_TRY(timer_start(ctx));
  const Orbitals &o = ctx->orb;
  const int nw = o.nw;
  int j2max = o.nkj[1];
  for (int i = 2; i <= nw; ++i) j2max = std::max(j2max, o.nkj[i]);
  if (j2max + 1 > KLIM) return fail(GG_ERR_ARG, "gg_genintbreit: 2j above 19");
  BreitTable &T = ctx->breit[type - 1];
  T.valid = false;
  T.on_host = false;
  T.j2max = j2max;
  cudaStream_t s = ctx->stream;
  // TRIANGBREIT1 (rci90/triangbreit1.f90:27-46) and TRIANGBREIT2
  // (triangbreit2.f90:27-42) factor into one condition per pair: type 1
  // admits (a, b, c, d) when some L in K-1..K+1 admits both pairs, type 2
  // when both pairs are admitted at L = K. mask[k][pair] holds those bits
  // (per L); the Bessel functions the admitted integrals read are those of
  // the pairs with a mask bit, at order k (type 1) or k -+ 1 (type 2).
  const size_t msz = (size_t)(nw + 1) * (nw + 1);
  std::vector<unsigned char> mask((size_t)(j2max + 1) * msz, 0);
  for (int K = 0; K <= j2max; ++K)
    for (int a = 1; a <= nw; ++a)
      for (int b = 1; b <= nw; ++b) {
        unsigned char m = 0;
        const int la = o.nkl[a], lb = o.nkl[b], ja = o.nkj[a], jb = o.nkj[b];
        if (type == 1) {
          for (int t = 0; t < 3; ++t) {
            const int L = K - 1 + t;
            if ((K + la + lb) % 2 == 1 && std::abs(ja - jb) <= 2 * L && std::abs(ja + jb) >= 2 * L) m |= 1 << t;
          }
          if (m) P.need(a, b, K);
        } else if ((K + la + lb) % 2 == 0 && std::abs(ja - jb) <= 2 * K && std::abs(ja + jb) >= 2 * K) {
          m = 1;
          P.need(a, b, K - 1);
          P.need(a, b, K + 1);
        }
        mask[(size_t)K * msz + (size_t)a * (nw + 1) + b] = m;
      }
  GG_TRY(P.upload(s));
  GG_TRY(run_table(ctx, type, P, j2max, mask, T, &ctx->stats[32], &ctx->stats[33]));
  T.valid = true;
  double ms = 0;
  GG_TRY(timer_stop(ctx, &ms));
  ctx->stats[31] = ms;
  if (nb_out) *nb_out = T.n;
  if (j2max_out) *j2max_out = j2max;
  return GG_OK;
}

int gg_get_breit_table(gg_ctx *ctx, int type, int32_t *indtp, double *valtp, int32_t *kstart) {
  if (!ctx || (type != 1 && type != 2)) return fail(GG_ERR_ARG, "gg_get_breit_table: type 1 or 2");
  const BreitTable &T = ctx->breit[type - 1];
  if (!T.valid) return fail(GG_ERR_STATE, "gg_get_breit_table: no table of this type (call gg_genintbreit)");
  // straight into the caller's arrays (a host copy of the table in between
  // cost a quarter of the 34-subshell table's time)
  GG_CUDA(cudaSetDevice(ctx->device));
  if (indtp && T.n) GG_CUDA(cudaMemcpyAsync(indtp, T.dInd.p, T.n * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
  if (valtp && T.n) GG_CUDA(cudaMemcpyAsync(valtp, T.dVal.p, T.n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  GG_CUDA(cudaStreamSynchronize(ctx->stream));
  if (kstart) std::copy(T.kstart.begin(), T.kstart.end(), kstart);
  return GG_OK;
}

// BRINT1 / BRINT2 (rci90/brint1.f90:30-66): binary search in the k range
int gg_brint(gg_ctx *ctx, int type, int ia, int ib, int ic, int id, int k, double *tegral) {
  if (!ctx || (type != 1 && type != 2) || !tegral) return fail(GG_ERR_ARG, "gg_brint: bad arguments");
  BreitTable &T = ctx->breit[type - 1];
  if (!T.valid) return fail(GG_ERR_STATE, "gg_brint: no table of this type (call gg_genintbreit)");
  const int nw = ctx->orb.nw, KEY = nw + 1;
  if (k < 0 || k > T.j2max || ia < 1 || ib < 1 || ic < 1 || id < 1 || ia > nw || ib > nw || ic > nw || id > nw)
    return fail(GG_ERR_NOTFOUND, "gg_brint: integral not in the table");
  if (!T.on_host.load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> lock(T.host_mu);
    if (!T.on_host.load(std::memory_order_relaxed)) {
      GG_CUDA(cudaSetDevice(ctx->device));
      T.hInd.resize(T.n);
      T.hVal.resize(T.n);
      if (T.n) {
        GG_CUDA(cudaMemcpyAsync(T.hInd.data(), T.dInd.p, T.n * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
        GG_CUDA(cudaMemcpyAsync(T.hVal.data(), T.dVal.p, T.n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        GG_CUDA(cudaStreamSynchronize(ctx->stream));
      }
      T.on_host.store(true, std::memory_order_release);
    }
  }
  const int32_t index = ((ia * KEY + ib) * KEY + ic) * KEY + id;
  const int32_t *b = T.hInd.data() + (T.kstart[k] - 1), *e = T.hInd.data() + (T.kstart[k + 1] - 1);
  const int32_t *p = std::lower_bound(b, e, index);
  if (p == e || *p != index) return fail(GG_ERR_NOTFOUND, "gg_brint: integral not in the table");
  *tegral = T.hVal[p - T.hInd.data()];
  return GG_OK;
}

int gg_brintf(gg_ctx *ctx, int n, const int32_t *items, double wfact, const double *e, double accy, double *out) {
  if (!ctx || n < 0 || (n > 0 && (!items || !out))) return fail(GG_ERR_ARG, "gg_brintf: bad arguments");
  if (n == 0) return GG_OK;
  GG_CUDA(cudaSetDevice(ctx->device));
  Plan P;
  GG_TRY(make_plan(ctx, wfact, e, accy, P));
  const int nw = ctx->orb.nw;
  // the Bessel functions the integrals read (brintf.f90:34-69)
  for (int t = 0; t < n; ++t) {
    const int32_t *it = items + 6 * (size_t)t;
    if (it[0] < 1 || it[0] > 6) return fail(GG_ERR_ARG, "gg_brintf: type outside 1..6");
    for (int j = 1; j <= 4; ++j)
      if (it[j] < 1 || it[j] > nw) return fail(GG_ERR_ARG, "gg_brintf: orbital outside the orbital set");
    const int K = it[5];
    if (K < 0 || K + 1 > KLIM) return fail(GG_ERR_ARG, "gg_brintf: k outside 0..19");
    switch (it[0]) {
      case 1: case 3: P.need(it[1], it[2], K); P.need(it[3], it[4], K); break;
      case 5: P.need(it[1], it[2], K); break;
      case 2: P.need(it[3], it[4], K - 1); P.need(it[3], it[4], K + 1);  // fall through
      case 6: P.need(it[1], it[2], K - 1); P.need(it[1], it[2], K + 1); break;
      default: break;
    }
  }
  cudaStream_t s = ctx->stream;
  GG_TRY(P.upload(s));
  DBuf<int32_t> ditems;
  DBuf<int> dcj;
  GG_TRY(ditems.alloc((size_t)6 * n));
  GG_CUDA(cudaMemcpyAsync(ditems.p, items, (size_t)6 * n * sizeof(int32_t), cudaMemcpyHostToDevice, s));
  GG_TRY(dcj.alloc(n));
  k_plan_items<<<(n + 127) / 128, 128, 0, s>>>(ditems.p, n, P.tabs(), 0, dcj.p, nullptr, nullptr, nullptr);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  std::vector<int> cj(n);
  GG_CUDA(cudaMemcpyAsync(cj.data(), dcj.p, n * sizeof(int), cudaMemcpyDeviceToHost, s));
  GG_CUDA(cudaStreamSynchronize(s));
  std::vector<int64_t> oj;
  const int64_t nj = scan(cj, oj);
  DBuf<int64_t> doj;
  DBuf<BrInt> dints;
  DBuf<BrJob> djobs;
  GG_TRY(upload_vec(doj, oj, s));
  GG_TRY(dints.alloc(n));
  GG_TRY(djobs.alloc(std::max<int64_t>(1, nj)));
  k_plan_items<<<(n + 127) / 128, 128, 0, s>>>(ditems.p, n, P.tabs(), 1, nullptr, doj.p, dints.p, djobs.p);
  ::gg::note_launch();
  GG_CUDA(cudaGetLastError());
  return run_terms(ctx, P, djobs.p, nj, dints.p, n, out);
}

}  // extern "C"

// bpx_fit_single.cuh -- the LM driver of the first fit (PVM_single, PVM_single_c), included by bpx_fit.cu.
//
// What bounds the fits is the latency of dependent FP64 instructions (the CUDA exp, sin and atan among
// them), so this form of lm_run spends fewer of them per LM trial and keeps more warps resident:
//   * about every second trial fails, and the normal equations at an accepted point need the fibre
//     signals its cost evaluation formed: the cost leaves them in the warp's shared memory (lcache, K
//     values per measurement) and the Jacobian reads them back;
//   * the isotropic signal depends on the b-value alone, and protocols hold few distinct ones: it is
//     formed once per distinct b-value and trial (BTable), one lane each, not once per measurement;
//   * sines, cosines and arctangents of the parameters are formed one per lane, not all in every lane;
//   * parameters live one per lane and the point's constants in shared memory, which leaves registers
//     for kFitStartMinBlocks blocks per SM.  Shared memory, K values per measurement and warp, leaves room
//     for them up to 333 measurements of three fibres, for four blocks up to 454 and for three at 512, where
//     the register form had four; model 1 fits of 4000 voxels of 512 measurements take 22.8 ms all the same
//     (55.0 in the register form with a counter per block), of 288 measurements 11.9 (36.2).
// Every value is formed by the operations, in the order, of the register form (bpx_fit.cu), and the fits
// are equal bit for bit.  The first fit of 12800 whole-brain voxels took 32.4 ms in the register form.
// PVM_multi keeps that form: with two and three fibres its normal equations are so ill-conditioned that
// the last bits of log1p, which the compiler contracts differently under another register pressure,
// change a third of the voxels' fits in FP32.
#pragma once

namespace bpx {

constexpr int kMaxK = BPX_MAX_FIBRES;
// distinct b-values the isotropic table holds; with more (or a b-matrix per voxel) the isotropic
// signal is formed per measurement
constexpr int kMaxB = 32;

// The distinct b-values of the launch's protocol (one copy per block); n = 0: no table.
struct BTable {
  float b[kMaxB];
  int n;
};

// the constants of one parameter vector
struct PointConst {
  Real fs[kMaxK], vx[kMaxK], vy[kMaxK], vz[kMaxK], sth[kMaxK], cth[kMaxK], sph[kMaxK], cph[kMaxK], dfx[kMaxK];
  Real deriv[kMaxK][kMaxK];
  Real wiso, d, S0, f0v, dfx0, sgn1, p1;
};

// Staging of [J | r] rows for the tensor cores: kRowsW measurements at a time, column-major with a
// stride of kRowsLd doubles (the stores and the fragment loads are both bank-conflict free); N takes
// its place when the last rows are in (row stride kNormLd).
constexpr int kRowsW = 16;
constexpr int kRowsLd = 20;
constexpr int kRowsDoubles = 16 * kRowsLd;
static_assert(16 * kNormLd <= kRowsDoubles, "N must fit the staging area");

// one warp's shared memory; lcache follows it: the fibre signals [K][M], left by the cost for the
// normal equations at the same point
struct WarpMem {
  Real st[kRowsDoubles];
  Real iso[kMaxB];
  Real x[16];  // the parameter vector the constants are formed from
  PointConst q;
};

__host__ __device__ constexpr size_t single_warp_bytes(int K, int M) {
  return sizeof(WarpMem) + (size_t)K * M * sizeof(Real);
}
// the block's b-value table and the measurements' entries in it, before the warps' areas
__host__ __device__ constexpr size_t single_block_bytes(int M) { return (sizeof(BTable) + (size_t)M + 15) / 16 * 16; }

// one warp's fit of a voxel
struct SingleFit {
  Meas ms;
  const BTable* bt;
  const unsigned char* bidx;  // measurement -> entry of bt
  WarpMem* w;
  Real* lcache;
  int lane;
};

// The distinct b-values of the protocol and each measurement's entry (none with a b-matrix per voxel,
// or with more than kMaxB of them).  The order of the entries does not matter.
__device__ void build_btable(const FitArgs& a, BTable& t, unsigned char* bidx) {
  if (threadIdx.x == 0) t.n = 0;
  __syncthreads();
  if (!a.gradnonlin) {
    for (int m = threadIdx.x; m < a.ndir; m += blockDim.x) {
      const float b = a.bvals[m];
      int first = 0;
      while (first < m && a.bvals[first] != b) ++first;
      if (first == m) {
        const int e = atomicAdd(&t.n, 1);
        if (e < kMaxB) t.b[e] = b;
      }
    }
  }
  __syncthreads();
  const int n = t.n;
  __syncthreads();
  if (n > kMaxB) {
    if (threadIdx.x == 0) t.n = 0;
  } else if (n > 0) {
    for (int m = threadIdx.x; m < a.ndir; m += blockDim.x) {
      const float b = a.bvals[m];
      int e = 0;
      while (e < n - 1 && t.b[e] != b) ++e;
      bidx[m] = (unsigned char)e;
    }
  }
  __syncthreads();
}

// Constants of the parameter vector held one entry per lane (xi: lane i holds parameter i).
template <int KIND, int K, bool F0>
__device__ __forceinline__ void point_constants(Real xi, WarpMem& w, int lane) {
  constexpr int P = LmShape<KIND, K, F0>::P, O = LmShape<KIND, K, F0>::O;
  PointConst& q = w.q;
  const int o = lane - O, k = o / 3, c = o % 3;
  const bool fibre = o >= 0 && o < 3 * K;
  const bool frac = (fibre && c == 0) || (F0 && lane == P - 1);
  Real sn = 0.0, s2 = 0.0;
  __syncwarp();  // the previous point's constants are no longer read
  if (lane < P) w.x[lane] = xi;
  if (fibre && c != 0) {
    Real cs;
    sincos(xi, &sn, &cs);
    if (c == 1) {
      q.sth[k] = sn;
      q.cth[k] = cs;
    } else {
      q.sph[k] = sn;
      q.cph[k] = cs;
    }
  }
  if (frac) {
    if (KIND == kSingleC) {
      sn = sin(xi);
      s2 = sin(2.0 * xi);
    } else {
      const Real f = x2fd(xi);
      const Real df = kTwoPiGpuD * sgnd(xi) / (1.0 + xi * xi);
      if (fibre) {
        q.fs[k] = f;
        q.dfx[k] = df;
      } else {
        q.f0v = f;
        q.dfx0 = df;
      }
    }
  }
  __syncwarp();
  if (lane < K) {
    q.vx[lane] = q.sth[lane] * q.cph[lane];
    q.vy[lane] = q.sth[lane] * q.sph[lane];
    q.vz[lane] = q.cth[lane];
  }
  if (KIND == kSingleC) {
    // fractions f_k = sin^2(beta_k) (1 - sum of the earlier ones) and d f_j / d beta_k
    // (fractions_deriv_PVM_single_c, CUDA/PVM_single_c.cu:104-139); every lane forms all of them
    Real sb[K], s2b[K], fs[K], deriv[K][K], sumf = 0.0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      sb[j] = __shfl_sync(0xffffffffu, sn, O + 3 * j);
      s2b[j] = __shfl_sync(0xffffffffu, s2, O + 3 * j);
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
      Real pf = 1.0;
#pragma unroll
      for (int n = 0; n < j; ++n) pf -= fs[n];
      fs[j] = sb[j] * sb[j] * pf;
      sumf += fs[j];
    }
#pragma unroll
    for (int m = 0; m < K; ++m) {
#pragma unroll
      for (int j = 0; j < K; ++j) {
        if (j == m) {
          Real fsum = 1.0;
#pragma unroll
          for (int n = 0; n < j; ++n) fsum -= fs[n];
          deriv[j][m] = s2b[m] * fsum;
        } else if (j > m) {
          Real fsum = 0.0;
#pragma unroll
          for (int n = 0; n < j; ++n) fsum += deriv[n][m];
          deriv[j][m] = -(sb[j] * sb[j]) * fsum;
        } else {
          deriv[j][m] = 0.0;
        }
      }
    }
    Real f0v = 0.0, dfx0 = 0.0;
    if (F0) {
      const Real s0 = __shfl_sync(0xffffffffu, sn, P - 1), s20 = __shfl_sync(0xffffffffu, s2, P - 1);
      const Real pfs = 1.0 - sumf;
      f0v = s0 * s0 * pfs;
      dfx0 = s20 * pfs;
    }
    if (lane == 0) {
#pragma unroll
      for (int j = 0; j < K; ++j) {
        q.fs[j] = fs[j];
#pragma unroll
        for (int m = 0; m < K; ++m) q.deriv[j][m] = deriv[j][m];
      }
      q.f0v = f0v;
      q.dfx0 = dfx0;
      q.wiso = 1.0 - sumf - f0v;
      q.p1 = w.x[1];
      q.S0 = w.x[0];
      q.d = w.x[1] * w.x[1];
    }
  } else if (lane == 0) {
    Real sumf = 0.0;
#pragma unroll
    for (int j = 0; j < K; ++j) sumf += q.fs[j];
    if (!F0) {
      q.f0v = 0.0;
      q.dfx0 = 0.0;
    }
    q.wiso = 1.0 - sumf - (F0 ? q.f0v : 0.0);
    const Real p1 = w.x[1];
    q.p1 = p1;
    q.sgn1 = pm1d(p1);
    q.d = fabs(p1);
    q.S0 = w.x[0];
  }
  __syncwarp();
}

// Sum of squared residuals at the point of point_constants(); leaves the isotropic table and lcache for
// the normal equations.
template <int KIND, int K, bool F0>
__device__ double single_cost(const SingleFit& c) {
  const PointConst& q = c.w->q;
  const Meas& ms = c.ms;
  const int nb = c.bt->n;
  if (c.lane < nb) {
    const Real b = c.bt->b[c.lane];
    c.w->iso[c.lane] = exp(-b * q.d);
  }
  __syncwarp();
  double acc = 0.0;
  for (int m = c.lane; m < ms.M; m += 32) {
    const Real gx = ms.gx[m], gy = ms.gy[m], gz = ms.gz[m], b = ms.b[m];
    const Real iso = nb ? c.w->iso[c.bidx[m]] : exp(-b * q.d);
    Real sig = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const Real dp = gx * q.vx[k] + gy * q.vy[k] + gz * q.vz[k];
      const Real d = q.d;
      const Real an = exp(-b * d * dp * dp);
      c.lcache[k * ms.M + m] = an;
      sig += q.fs[k] * an;
    }
    const Real wiso = q.wiso;
    const Real full = q.S0 * ((q.f0v + wiso * iso) + sig);
    const Real e = full - (Real)ms.y[m];
    acc += e * e;
  }
  return group_sum<32>(acc);
}

// Predicted signal of one measurement with its Jacobian row J, from what single_cost() left for the point.
template <int KIND, int K, bool F0>
__device__ __forceinline__ Real single_jacobian(const SingleFit& c, int m, Real (&J)[LmShape<KIND, K, F0>::P]) {
  constexpr int P = LmShape<KIND, K, F0>::P, O = LmShape<KIND, K, F0>::O;
  const PointConst& q = c.w->q;
  const Meas& ms = c.ms;
  const Real gx = ms.gx[m], gy = ms.gy[m], gz = ms.gz[m], b = ms.b[m];
  const Real iso = c.bt->n ? c.w->iso[c.bidx[m]] : exp(-b * q.d);
  const Real wiso = q.wiso, d = q.d;
  Real sig = 0.0, an[K], dp[K];
#pragma unroll
  for (int i = 0; i < P; ++i) J[i] = 0.0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    dp[k] = gx * q.vx[k] + gy * q.vy[k] + gz * q.vz[k];
    an[k] = c.lcache[k * ms.M + m];
    sig += q.fs[k] * an[k];
  }
  if (KIND == kSingle) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      J[1] += q.sgn1 * q.S0 * q.fs[k] * (-b * dp[k] * dp[k] * an[k]);
      J[O + 3 * k] = q.S0 * (an[k] - iso) * q.dfx[k];
    }
    J[1] += q.sgn1 * q.S0 * wiso * (-b * iso);
  } else {
    const Real lam = q.p1;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      J[1] += q.S0 * q.fs[k] * (-2.0 * b * lam * dp[k] * dp[k] * an[k]);
      Real s = 0.0;
#pragma unroll
      for (int j = 0; j < K; ++j) s += q.S0 * (an[j] - iso) * q.deriv[j][k];
      J[O + 3 * k] = s;
    }
    J[1] += q.S0 * wiso * (-2.0 * b * lam * iso);
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const Real dp1 = q.cth[k] * (gx * q.cph[k] + gy * q.sph[k]) - gz * q.sth[k];
    const Real dp2 = q.sth[k] * (-gx * q.sph[k] + gy * q.cph[k]);
    const Real cc = q.S0 * q.fs[k] * (-2.0 * b * d * dp[k] * an[k]);
    J[O + 3 * k + 1] = cc * dp1;
    J[O + 3 * k + 2] = cc * dp2;
  }
  if (F0) J[P - 1] = q.S0 * (1.0 - iso) * q.dfx0;
  const Real full = q.S0 * ((q.f0v + wiso * iso) + sig);
  J[0] = full / q.S0;  // S0 is the parameter itself in both forms
  return full;
}

// Gauss-Newton normal equations at the point single_cost() evaluated last, as normal_eqs leaves them.
template <int KIND, int K, bool F0>
__device__ void single_normal_eqs(const SingleFit& c) {
  constexpr int P = LmShape<KIND, K, F0>::P;
  constexpr bool kWide = P + 1 > 8;
  constexpr int kCols = kWide ? 16 : 8;
  Real* st = c.w->st;
  const int lane = c.lane;
  double n00[2] = {0.0, 0.0}, n01[2] = {0.0, 0.0}, n11[2] = {0.0, 0.0};
  const int fr = lane >> 2, fk = lane & 3;  // fragment row (parameter) and k (measurement) of this lane
  __syncwarp();  // the previous N is no longer read
  for (int i = (P + 1) * kRowsLd + lane; i < kCols * kRowsLd; i += 32) st[i] = 0.0;
  for (int m0 = 0; m0 < c.ms.M; m0 += 32) {
    const int m = m0 + lane;
    Real J[P], diff = 0.0;
    if (m < c.ms.M) {
      const Real sig = single_jacobian<KIND, K, F0>(c, m, J);
      diff = sig - (Real)c.ms.y[m];
    } else {
#pragma unroll
      for (int i = 0; i < P; ++i) J[i] = 0.0;
    }
#pragma unroll
    for (int h = 0; h < 32 / kRowsW; ++h) {
      __syncwarp();  // the previous rows' fragment loads are done
      if (lane / kRowsW == h) {
#pragma unroll
        for (int i = 0; i < P; ++i) st[i * kRowsLd + lane % kRowsW] = J[i];
        st[P * kRowsLd + lane % kRowsW] = diff;
      }
      __syncwarp();
#pragma unroll
      for (int k0 = 0; k0 < kRowsW; k0 += 4) {
        const double lo = st[fr * kRowsLd + k0 + fk];
        dmma_8x8x4(n00, lo, lo);
        if (kWide) {
          const double hi = st[(8 + fr) * kRowsLd + k0 + fk];
          dmma_8x8x4(n01, lo, hi);
          dmma_8x8x4(n11, hi, hi);
        }
      }
    }
  }
  __syncwarp();
  const int c0 = 2 * fk;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    st[fr * kNormLd + c0 + i] = n00[i];
    if (kWide) {
      st[fr * kNormLd + 8 + c0 + i] = n01[i];
      st[(8 + c0 + i) * kNormLd + fr] = n01[i];
      st[(8 + fr) * kNormLd + 8 + c0 + i] = n11[i];
    }
  }
  __syncwarp();
}

// lm_run with lane i holding parameter i; p returns the whole vector in every lane.
template <int KIND, int K, bool F0>
__device__ bool single_lm_run(const SingleFit& c, Real (&p)[LmShape<KIND, K, F0>::P]) {
  static_assert(KIND == kSingle || KIND == kSingleC, "PVM_multi runs in lm_run");
  constexpr int P = LmShape<KIND, K, F0>::P;
  const int lane = c.lane;
  double lambda = 0.1;
  const double cftol = 1.0e-8, ltol = 1.0e20;
  Real pi = 0.0;
#pragma unroll
  for (int i = 0; i < P; ++i)
    if (lane == i) pi = p[i];
  point_constants<KIND, K, F0>(pi, *c.w, lane);
  double pcf = single_cost<KIND, K, F0>(c);
  int niter = 0;
  bool success = true, stopped = false;
  const Real* st = c.w->st;
  const int row = lane < P ? lane : 0;
  while (!(success && niter++ >= 200)) {
    if (success) single_normal_eqs<KIND, K, F0>(c);
    double A[P];
#pragma unroll
    for (int j = 0; j < P; ++j) A[j] = 2.0 * st[row * kNormLd + j] + ((lane == j) ? lambda : 0.0);
    const double grow = 2.0 * st[row * kNormLd + P];
    double x[P];
    warp_solve<P>(A, grow, x, lane);
    Real xi = 0.0;
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (lane == i) xi = x[i];
    const Real step = pi - xi;
    point_constants<KIND, K, F0>(step, *c.w, lane);
    const double ncf = single_cost<KIND, K, F0>(c);
    bool end = false;
    if ((success = (ncf < pcf))) {
      pi = step;
      lambda /= 10.0;
      if (2.0 * fabs(pcf - ncf) <= cftol * (fabs(pcf) + fabs(ncf) + 2.0e-16)) end = true;
      pcf = ncf;
    } else {
      lambda *= 10.0;
      if (lambda > ltol) end = true;
    }
    if (end) {
      stopped = true;
      break;
    }
  }
#pragma unroll
  for (int i = 0; i < P; ++i) p[i] = __shfl_sync(0xffffffffu, pi, i);
  return stopped;
}

}  // namespace bpx

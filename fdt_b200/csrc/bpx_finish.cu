// bpx_finish.cu -- sample finishing on the GPU.
//
// Replaces record_finish_voxels + Samples::record / finish_voxel / save
// (CUDA/xfibres_gpu.cu:659-738, CUDA/samples.cu:134-347), which the reference runs on the host
// after copying every record back: per voxel the sample means, the principal eigenvector of
// each fibre's mean dyadic tensor, and the fibres re-ordered by decreasing sum of f over samples
// into the th/ph/f sample arrays.
//
// Layout: a block takes 32 voxels, its eight warps every eighth sample of them, so each row of a
// sample is one 128-byte line and 64K voxels (or 500) put eight times as many loads in flight as one
// thread per voxel walking all samples would; that serial walk, not HBM, bounded the first form (65536
// voxels x 50 samples, 3 fibres: 439 us for finishing and 246 us for the post-processing maps).  The
// warps' FP64 partial sums are added in warp order, so a run reproduces.
#include <cstdint>

#include "bpx_device.cuh"
#include "bpx_internal.h"

namespace bpx {

// principal eigenvector of a symmetric 3x3 (cyclic Jacobi, FP64), largest |component| positive;
// returns the largest eigenvalue.  A rotation is a chain of long FP64 operations and few threads run it, so
// it is bound by their latency: the tangent takes one square root and one division, the cosine one
// reciprocal square root, and the sweeps end when the off-diagonal elements are below FP64 rounding of
// the matrix (1e-16.5 of its norm) instead of at underflow.
__device__ double principal_vector(double (&A)[3][3], double (&out)[3]) {
  double V[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
  const double tol = 1e-33 * (A[0][0] * A[0][0] + A[1][1] * A[1][1] + A[2][2] * A[2][2] +
                              2.0 * (A[0][1] * A[0][1] + A[0][2] * A[0][2] + A[1][2] * A[1][2]));
  for (int sweep = 0; sweep < 50; ++sweep) {
    const double off = A[0][1] * A[0][1] + A[0][2] * A[0][2] + A[1][2] * A[1][2];
    if (off <= tol) break;
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
      for (int q = p + 1; q < 3; ++q) {
        const double apq = A[p][q];
        if (apq * apq <= 0.1 * tol) continue;
        const double b = A[q][q] - A[p][p], e = 2.0 * apq;
        const double m = fabs(e) / (fabs(b) + sqrt(b * b + e * e));
        const double t = (b == 0.0 || (b > 0.0) == (e > 0.0)) ? m : -m;
        const double c = rsqrt(t * t + 1.0), s = t * c;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double akp = A[k][p], akq = A[k][q];
          A[k][p] = c * akp - s * akq;
          A[k][q] = s * akp + c * akq;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double apk = A[p][k], aqk = A[q][k];
          A[p][k] = c * apk - s * aqk;
          A[q][k] = s * apk + c * aqk;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double vkp = V[k][p], vkq = V[k][q];
          V[k][p] = c * vkp - s * vkq;
          V[k][q] = s * vkp + c * vkq;
        }
      }
  }
  int best = 0;
  if (A[1][1] > A[best][best]) best = 1;
  if (A[2][2] > A[best][best]) best = 2;
  double col[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) col[r] = (best == 0) ? V[r][0] : (best == 1 ? V[r][1] : V[r][2]);
  int big = 0;
  if (fabs(col[1]) > fabs(col[big])) big = 1;
  if (fabs(col[2]) > fabs(col[big])) big = 2;
  const double sg = col[big] < 0 ? -1.0 : 1.0;
#pragma unroll
  for (int r = 0; r < 3; ++r) out[r] = sg * col[r];
  return A[best][best];
}

constexpr int kVox = 32, kGroups = 8;  // voxels and sample groups (warps) of a block

// Sums over the block's sample groups of Q quantities per voxel: fin[q][voxel] on return (synchronised).
template <int Q>
__device__ __forceinline__ void sum_groups(const double (&val)[Q], double (*fin)[kVox]) {
  __shared__ double buf[kGroups][kGroups][kVox];
  const int x = threadIdx.x, g = threadIdx.y;
#pragma unroll
  for (int q0 = 0; q0 < Q; q0 += kGroups) {
#pragma unroll
    for (int q = 0; q < kGroups; ++q)
      if (q0 + q < Q) buf[g][q][x] = val[q0 + q];
    __syncthreads();
    if (q0 + g < Q) {  // group g adds up quantity q0 + g
      double t = buf[0][g][x];
#pragma unroll
      for (int j = 1; j < kGroups; ++j) t += buf[j][g][x];
      fin[q0 + g][x] = t;
    }
    __syncthreads();
  }
}

// unit vector of the angles, as the reference forms it: FP32 sines and cosines, FP64 products
__device__ __forceinline__ void direction(float th, float ph, double (&x)[3]) {
  float st, ct, sp, cp;
  sincosf(th, &st, &ct);
  sincosf(ph, &sp, &cp);
  x[0] = (double)st * cp;
  x[1] = (double)st * sp;
  x[2] = (double)ct;
}

// adds x x^T to the upper triangle t = {xx, xy, xz, yy, yz, zz}
__device__ __forceinline__ void add_dyad(double* t, const double (&x)[3]) {
  t[0] += x[0] * x[0];
  t[1] += x[0] * x[1];
  t[2] += x[0] * x[2];
  t[3] += x[1] * x[1];
  t[4] += x[1] * x[2];
  t[5] += x[2] * x[2];
}

__device__ __forceinline__ void full_tensor(double (*t)[kVox], int x, double scale, double (&A)[3][3]) {
  A[0][0] = t[0][x] * scale;
  A[0][1] = A[1][0] = t[1][x] * scale;
  A[0][2] = A[2][0] = t[2][x] * scale;
  A[1][1] = t[3][x] * scale;
  A[1][2] = A[2][1] = t[4][x] * scale;
  A[2][2] = t[5][x] * scale;
}

template <int K>
__global__ void __launch_bounds__(kVox * kGroups, 3) finish_kernel(FinishArgs a) {
  constexpr int Q = 6 + 6 * K;
  __shared__ double sumf[K][kVox], fin[Q][kVox];
  const int x = threadIdx.x, g = threadIdx.y;
  const int ns = a.nsamples, nvox = a.nvox;
  const int v = blockIdx.x * kVox + x;
  const bool in = v < nvox;
  const size_t row = (size_t)ns * nvox;
  const float* rec = a.records + (in ? v : 0);
  // the fibre order first, from the sums of f over the samples (the f rows, a fifth of the
  // records): sort (sum f, index) ascending and read it backwards (CUDA/samples.cu:299-330)
  {
    double sf[K];
#pragma unroll
    for (int k = 0; k < K; ++k) sf[k] = 0;
    if (in)
      for (int s = g; s < ns; s += kGroups)
#pragma unroll
        for (int k = 0; k < K; ++k) sf[k] += __ldg(rec + (8 + 3 * k) * row + (size_t)s * nvox);
    sum_groups<K>(sf, sumf);
  }
  int slot[K];  // output position of fibre k: the number of fibres that come before it
#pragma unroll
  for (int i = 0; i < K; ++i) {
    int rank = 0;
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (j != i && (sumf[j][x] > sumf[i][x] || (sumf[j][x] == sumf[i][x] && j > i))) ++rank;
    slot[i] = rank;
  }
  // one pass over the records: sums, dyadic tensors, and every sample copied to its sorted slot
  // (each output row is written once, a whole line at a time)
  const bpx_outputs& out = a.out;
  double val[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) val[q] = 0;
  if (in) {
    for (int s = g; s < ns; s += kGroups) {
      const size_t o = (size_t)s * nvox;
#pragma unroll
      for (int r = 0; r < 6; ++r) val[r] += __ldg(rec + r * row + o);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const float th = __ldg(rec + (6 + 3 * k) * row + o), ph = __ldg(rec + (7 + 3 * k) * row + o);
        const size_t oo = ((size_t)slot[k] * ns + s) * nvox + v;
        if (out.th) out.th[oo] = th;
        if (out.ph) out.ph[oo] = ph;
        if (out.f) out.f[oo] = __ldg(rec + (8 + 3 * k) * row + o);
        double d[3];
        direction(th, ph, d);
        add_dyad(val + 6 + 6 * k, d);
      }
    }
  }
  sum_groups<Q>(val, fin);
  if (!in) return;
  const double inv = 1.0 / ns;
  if (g < K) {  // warp g: the mean and dyad of output position g
    // the fibre that comes there: sums that are NaN compare with none, so positions can then hold two
    // fibres (the later one counts) or none (fibre 0)
    int src = 0;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (slot[k] == g) src = k;
    if (out.mean_f) out.mean_f[(size_t)g * nvox + v] = (float)(sumf[src][x] * inv);
    if (out.dyads) {
      double A[3][3], pv[3];
      full_tensor(fin + 6 + 6 * src, x, 1.0, A);
      principal_vector(A, pv);
#pragma unroll
      for (int r = 0; r < 3; ++r) out.dyads[((size_t)g * 3 + r) * nvox + v] = (float)pv[r];
    }
  } else if (g == kGroups - 1) {
    float* mean[6] = {out.mean_d, out.mean_f0, out.mean_tau, out.mean_dstd, out.mean_R, out.mean_S0};
#pragma unroll
    for (int r = 0; r < 6; ++r)
      if (mean[r]) mean[r][v] = (float)(fin[r][x] * inv);
  }
}

// bedpostx_postproc_gpu.sh arithmetic (CUDA/bedpostx_postproc_gpu.sh:20-49) on the finished
// outputs, in the layout of finish_kernel: fslmaths -Tmean of merged_th/ph, the dispersion of each fibre's
// mean dyadic tensor (make_dyadic_vectors.cc:60-92: 1 - max |eigenvalue|), maskdyads
// (dyads{k} where mean_f{k} >= thr, fslmaths -thr -bin -mul), the _modf{k} scaling by
// mean_f{k}/mean_f1 (fslmaths -div gives 0 where the divisor is 0) and mean_fsumsamples.
template <int K>
__global__ void __launch_bounds__(kVox * kGroups, 3) postproc_kernel(PostArgs a) {
  constexpr int Q = 8 * K;  // per fibre: sum th, sum ph, the tensor's upper triangle
  __shared__ double fin[Q][kVox];
  const int x = threadIdx.x, g = threadIdx.y;
  const int ns = a.nsamples, nvox = a.nvox;
  const int v = blockIdx.x * kVox + x;
  const bool in = v < nvox;
  const bpx_postproc& p = a.post;
  double val[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) val[q] = 0;
  if (in) {
    for (int s = g; s < ns; s += kGroups) {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const size_t o = ((size_t)k * ns + s) * nvox + v;
        const float th = __ldg(a.th + o), ph = __ldg(a.ph + o);
        val[8 * k] += th;
        val[8 * k + 1] += ph;
        double d[3];
        direction(th, ph, d);
        add_dyad(val + 8 * k + 2, d);
      }
    }
  }
  sum_groups<Q>(val, fin);
  if (!in) return;
  if (g < K) {
    const size_t o = (size_t)g * nvox + v;
    if (p.mean_th) p.mean_th[o] = (float)(fin[8 * g][x] / ns);
    if (p.mean_ph) p.mean_ph[o] = (float)(fin[8 * g + 1][x] / ns);
    if (p.dispersion) {
      double A[3][3], pv[3];
      full_tensor(fin + 8 * g + 2, x, 1.0 / ns, A);
      const double lmax = principal_vector(A, pv);  // the tensor is positive semi-definite
      p.dispersion[o] = (float)(1.0 - fabs(lmax));
    }
  } else if (g == kGroups - 1) {
    float mf[K];
    double fsum = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      mf[k] = a.mean_f[(size_t)k * nvox + v];
      fsum += mf[k];
    }
    if (p.mean_fsum) p.mean_fsum[v] = (float)fsum;
#pragma unroll
    for (int k = 1; k < K; ++k) {
      const bool keep = mf[k] >= a.thr && mf[k] != 0.f;
      const float ratio = mf[0] != 0.f ? mf[k] / mf[0] : 0.f;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const size_t o = ((size_t)k * 3 + r) * nvox + v;
        const float dt = keep ? a.dyads[o] : 0.f;
        if (p.dyads_thr) p.dyads_thr[o] = dt;
        if (p.dyads_modf) p.dyads_modf[o] = dt * ratio;
      }
    }
  }
}

cudaError_t launch_postproc(const PostArgs& a, cudaStream_t s) {
  if (a.nvox == 0) return cudaSuccess;
  const dim3 threads(kVox, kGroups);
  const int grid = (a.nvox - 1) / kVox + 1;
  switch (a.nfib) {
    case 1: postproc_kernel<1><<<grid, threads, 0, s>>>(a); break;
    case 2: postproc_kernel<2><<<grid, threads, 0, s>>>(a); break;
    case 3: postproc_kernel<3><<<grid, threads, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_finish(const FinishArgs& a, cudaStream_t s) {
  if (a.nvox == 0) return cudaSuccess;
  const dim3 threads(kVox, kGroups);
  const int grid = (a.nvox - 1) / kVox + 1;
  switch (a.nfib) {
    case 1: finish_kernel<1><<<grid, threads, 0, s>>>(a); break;
    case 2: finish_kernel<2><<<grid, threads, 0, s>>>(a); break;
    case 3: finish_kernel<3><<<grid, threads, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace bpx

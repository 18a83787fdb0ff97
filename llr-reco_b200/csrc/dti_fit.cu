// DTI scalar maps downstream of the recon (diffusion_models.rs:21-129, calc_scalars):
// per voxel, s0 = mean |b0|, rhs_q = ln(clamp(|s_q| / max(s0, FLT_MIN), FLT_MIN, 1)), the
// 6-parameter tensor d = argmin ||A d - rhs|| with the design matrix of build_design_matrix
// (columns -b gx^2, -b gy^2, -b gz^2, -2b gx gy, -2b gx gz, -2b gy gz), the eigenvalues of the
// 3 x 3 tensor (e1 >= e2 >= e3), and MD = mean, RD = (e2 + e3) / 2,
// FA = sqrt(3/2) sqrt(sum (e_i - MD)^2) / sqrt(sum e_i^2) (NaN for a zero tensor, as there).
//
// Two voxels per thread: the least-squares solve is the same pseudo-inverse for every voxel
// (A has full column rank for six or more non-coplanar directions), formed once on the host in
// FP64 from the normal equations and applied from shared memory; the symmetric 3 x 3 eigen
// problem is a few cyclic Jacobi sweeps in registers.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

#include "llr_common.cuh"
#include "llr_internal.h"

namespace llr {

namespace {

constexpr int kDtiOut = 7;   // b0av, e1, e2, e3, md, rd, fa

__device__ __forceinline__ void jacobi_rot(float& app, float& aqq, float& apq, float& arp, float& arq) {
  // zero apq; arp / arq: the third row's entries against p and q.  The tangent is the smaller root of
  // t^2 + t (aqq - app) / apq - 1 = 0 with one square root and one division; entries are scaled to at most
  // 1, so the squares neither overflow nor lose an apq that matters.
  if (fabsf(apq) <= 1e-18f) return;
  const float d = aqq - app, a2 = 2.f * apq;
  const float t = __fdividef(d >= 0.f ? a2 : -a2, fabsf(d) + sqrtf(fmaf(d, d, a2 * a2)));
  const float c = rsqrtf(fmaf(t, t, 1.f)), s = t * c;
  app -= t * apq;
  aqq += t * apq;
  apq = 0.f;
  const float rp = arp, rq = arq;
  arp = c * rp - s * rq;
  arq = s * rp + c * rq;
}

// eigenvalues of the symmetric [[a, d, e], [d, b, f], [e, f, c]], descending.  The matrix is scaled by a
// power of two (exact) so that its largest entry lies in [1, 2).
__device__ void sym3_eigenvalues(float a, float b, float c, float d, float e, float f, float* out) {
  const float mx = fmaxf(fmaxf(fmaxf(fabsf(a), fabsf(b)), fabsf(c)), fmaxf(fmaxf(fabsf(d), fabsf(e)), fabsf(f)));
  const int ex = min(max((__float_as_int(mx) >> 23) & 0xff, 1), 253);
  const float up = __int_as_float((254 - ex) << 23), dn = __int_as_float(ex << 23);
  a *= up; b *= up; c *= up; d *= up; e *= up; f *= up;
  for (int sweep = 0; sweep < 8; ++sweep) {
    // off-diagonal entries this far below the diagonal move no eigenvalue by half an ulp
    if (fabsf(d) + fabsf(e) + fabsf(f) <= 1e-9f * (fabsf(a) + fabsf(b) + fabsf(c))) break;
    jacobi_rot(a, b, d, e, f);   // (0,1); third index 2: (a02, a12) = (e, f)
    jacobi_rot(a, c, e, d, f);   // (0,2); third index 1: (a01, a21) = (d, f)
    jacobi_rot(b, c, f, d, e);   // (1,2); third index 0: (a10, a20) = (d, e)
  }
  float l[3] = {a, b, c};
  if (l[0] < l[1]) { float t = l[0]; l[0] = l[1]; l[1] = t; }
  if (l[1] < l[2]) { float t = l[1]; l[1] = l[2]; l[2] = t; }
  if (l[0] < l[1]) { float t = l[0]; l[0] = l[1]; l[1] = t; }
  out[0] = l[0] * dn; out[1] = l[1] * dn; out[2] = l[2] * dn;
}

// ln x of a positive normal x: x = 2^k m with m in [sqrt 1/2, sqrt 2), f = m - 1, and
// ln(1 + f) = f - f^2 / 2 + f^3 P(f), P the least-maximum-error degree-7 fit of the series' tail over
// that range (relative error 6e-9 before rounding, Lawson's iteratively weighted least squares).
// Measured against FP64 over (e^-8, 1): relative error at most 1e-7.
__device__ __forceinline__ float ln_normal(float x) {
  const int ix = __float_as_int(x) - 0x3f3504f3;
  const float k = (float)(ix >> 23);
  const float f = __int_as_float((ix & 0x7fffff) + 0x3f3504f3) - 1.f;
  float p = -0.07634474337100983f;
  p = fmaf(p, f, 0.12761567533016205f);
  p = fmaf(p, f, -0.13160187005996704f);
  p = fmaf(p, f, 0.14201758801937103f);
  p = fmaf(p, f, -0.16623356938362122f);
  p = fmaf(p, f, 0.20001226663589478f);
  p = fmaf(p, f, -0.2500081956386566f);
  p = fmaf(p, f, 0.3333333134651184f);
  const float q = fmaf(p, f, -0.5f);
  return fmaf(k, 0.69314718056f, fmaf(f * f, q, f));
}

// Right-hand sides 2 ln(clamp(|z_q| / s0, FLT_MIN, 1)) of QB samples of two voxels (z[voxel][sample]) into
// the tensor sums dt (the factor 2 is taken out of the weights; w: eight floats per sample, six used).  The
// common form is ln(|z|^2 / s0^2): one multiplication by the voxel's 1 / s0^2 in place of a square root
// and a division per sample.  Where a square could leave the range of normal numbers (s0 outside
// [1e-15, 1e15], |z| below 1e-15 s0) or z is not a number, the batch forms the ratios themselves.
template <int QB>
__device__ __forceinline__ void add_samples(const float2 (&z)[2][QB], const float* w, const float* s0c,
                                            const float* inv2, const float* lo2, float (&dt)[2][6]) {
  float r[2][QB];
  bool fast = true;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int u = 0; u < QB; ++u) {
      r[h][u] = z[h][u].x * z[h][u].x + z[h][u].y * z[h][u].y;
      fast = fast && r[h][u] >= lo2[h];
    }
  unsigned zero = 0;   // samples that are zero, where nothing else is out of range
  if (!fast) {
    fast = true;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        if (r[h][u] == 0.f) zero |= 1u << (h * QB + u);
        else fast = fast && r[h][u] >= lo2[h];
      }
  }
  if (fast) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int u = 0; u < QB; ++u) r[h][u] = ln_normal(fminf(r[h][u] * inv2[h], 1.f));
    if (zero) {
      const float ln_tiny = 2.f * logf(FLT_MIN);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < QB; ++u)
          if (zero >> (h * QB + u) & 1) r[h][u] = ln_tiny;
    }
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll 1
      for (int u = 0; u < QB; ++u) r[h][u] = 2.f * logf(fminf(fmaxf(sqrtf(r[h][u]) / s0c[h], FLT_MIN), 1.f));
  }
#pragma unroll
  for (int u = 0; u < QB; ++u) {
    const float4 pa = *reinterpret_cast<const float4*>(w + 8 * u);
    const float2 pb = *reinterpret_cast<const float2*>(w + 8 * u + 4);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      dt[h][0] = fmaf(pa.x, r[h][u], dt[h][0]);
      dt[h][1] = fmaf(pa.y, r[h][u], dt[h][1]);
      dt[h][2] = fmaf(pa.z, r[h][u], dt[h][2]);
      dt[h][3] = fmaf(pa.w, r[h][u], dt[h][3]);
      dt[h][4] = fmaf(pb.x, r[h][u], dt[h][4]);
      dt[h][5] = fmaf(pb.y, r[h][u], dt[h][5]);
    }
  }
}

// Bound: HBM, 8 (nq + nb0) + 28 bytes per voxel (1.83 GB at 192 x 192 x 96 x (54 + 7): 280 us at the measured
// copy rate); the instruction issue of the logarithms comes next.  Eight samples of two voxels are in flight
// per thread before the first logarithm, and a row of the weights (two shared loads) serves both voxels.
// Calls at that size: 625 us with a square root, a division and a logf per sample, one load at a time and
// IEEE rotations; 485 us with ln_normal and the one-division rotations; 433 us with one range check per
// batch instead of per sample; 404 us at four CTAs per SM (64 registers) instead of three.  Half of the volume masked
// to zero, in turn on one box: 844 us (8^3 patches of zeros: 1440) with the ratios formed one by one, 402 us (450) with the
// zeros kept as a mask over the batch, whose logarithms are set afterwards; without zeros 393 us either way.  Adding the zeros'
// six terms apart, before the others, took 430 us (593), and 403 us without zeros.
__global__ void __launch_bounds__(256, 4) dti_fit_kernel(const float2* __restrict__ dwi, const float2* __restrict__ b0,
                                                      long long V, int nq, int nb0, const float* __restrict__ pinv,
                                                      float* __restrict__ out) {
  constexpr int QB = 8;               // samples in flight per voxel
  extern __shared__ __align__(16) float s_pinv[];   // [nq][8], six used
  for (int i = threadIdx.x; i < 8 * nq; i += blockDim.x) s_pinv[i] = pinv[i];
  __syncthreads();
  const long long step = (long long)gridDim.x * blockDim.x * 2;
  for (long long vb = blockIdx.x * (long long)blockDim.x * 2 + threadIdx.x; vb < V; vb += step) {
    // the thread's two voxels are a CTA width apart; a missing second one repeats the first
    const long long v[2] = {vb, vb + blockDim.x < V ? vb + blockDim.x : vb};
    float s0[2] = {0.f, 0.f};
    for (int k = 0; k < nb0; ++k) {
      float2 z[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) z[h] = b0[v[h] + V * k];
#pragma unroll
      for (int h = 0; h < 2; ++h) s0[h] += sqrtf(z[h].x * z[h].x + z[h].y * z[h].y);
    }
    float s0c[2], inv2[2], lo2[2], dt[2][6];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      s0[h] = nb0 > 0 ? s0[h] / (float)nb0 : 0.f;
      s0c[h] = fmaxf(s0[h], FLT_MIN);
      const bool in_range = s0c[h] >= 1e-15f && s0c[h] <= 1e15f;
      inv2[h] = in_range ? 1.f / (s0c[h] * s0c[h]) : 0.f;
      lo2[h] = in_range ? fmaxf(1e-30f * (s0c[h] * s0c[h]), FLT_MIN) : NAN;   // no sample compares with it, infinite ones included
#pragma unroll
      for (int j = 0; j < 6; ++j) dt[h][j] = 0.f;
    }
    const float2* p0 = dwi + v[0];
    const float2* p1 = dwi + v[1];
    int q = 0;
    for (; q + QB <= nq; q += QB) {
      float2 z[2][QB];
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        z[0][u] = __ldcs(p0);
        z[1][u] = __ldcs(p1);
        p0 += V;
        p1 += V;
      }
      add_samples<QB>(z, s_pinv + 8 * q, s0c, inv2, lo2, dt);
    }
    for (; q < nq; ++q) {
      const float2 z[2][1] = {{__ldcs(p0)}, {__ldcs(p1)}};
      p0 += V;
      p1 += V;
      add_samples<1>(z, s_pinv + 8 * q, s0c, inv2, lo2, dt);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 1 && vb + blockDim.x >= V) break;
      float l[3];
      sym3_eigenvalues(dt[h][0], dt[h][1], dt[h][2], dt[h][3], dt[h][4], dt[h][5], l);
      const float md = (l[0] + l[1] + l[2]) / 3.f;
      const float rd = 0.5f * (l[1] + l[2]);
      const float num = sqrtf((l[0] - md) * (l[0] - md) + (l[1] - md) * (l[1] - md) + (l[2] - md) * (l[2] - md));
      const float den = sqrtf(l[0] * l[0] + l[1] * l[1] + l[2] * l[2]);
      const float fa = 1.22474487139158904910f * num / den;
      float* o = out + v[h];
      o[0] = s0[h];
      o[V] = l[0];
      o[2 * V] = l[1];
      o[3 * V] = l[2];
      o[4 * V] = md;
      o[5 * V] = rd;
      o[6 * V] = fa;
    }
  }
}

// (A^T A)^{-1} A^T in FP64 (Gauss-Jordan with partial pivoting on the 6 x 6 normal matrix)
int design_pinv(const float* b, const float* g, int nq, std::vector<float>& pinv) {
  std::vector<double> A((size_t)nq * 6);
  for (int q = 0; q < nq; ++q) {
    const double bb = b[q], gx = g[3 * q], gy = g[3 * q + 1], gz = g[3 * q + 2];
    const double row[6] = {-bb * gx * gx, -bb * gy * gy, -bb * gz * gz, -2 * bb * gx * gy, -2 * bb * gx * gz,
                           -2 * bb * gy * gz};
    for (int j = 0; j < 6; ++j) A[(size_t)q * 6 + j] = row[j];
  }
  double M[6][12];
  for (int i = 0; i < 6; ++i)
    for (int j = 0; j < 6; ++j) {
      double s = 0.0;
      for (int q = 0; q < nq; ++q) s += A[(size_t)q * 6 + i] * A[(size_t)q * 6 + j];
      M[i][j] = s;
      M[i][6 + j] = i == j ? 1.0 : 0.0;
    }
  double scale = 0.0;
  for (int i = 0; i < 6; ++i) scale = std::max(scale, std::fabs(M[i][i]));
  for (int c = 0; c < 6; ++c) {
    int p = c;
    for (int r = c + 1; r < 6; ++r)
      if (std::fabs(M[r][c]) > std::fabs(M[p][c])) p = r;
    if (!(std::fabs(M[p][c]) > 1e-12 * scale))
      return set_error(LLR_ERR_INVALID, "DTI design matrix is rank deficient (need 6 independent directions)");
    if (p != c)
      for (int j = 0; j < 12; ++j) std::swap(M[p][j], M[c][j]);
    const double inv = 1.0 / M[c][c];
    for (int j = 0; j < 12; ++j) M[c][j] *= inv;
    for (int r = 0; r < 6; ++r)
      if (r != c) {
        const double f = M[r][c];
        for (int j = 0; j < 12; ++j) M[r][j] -= f * M[c][j];
      }
  }
  pinv.assign((size_t)8 * nq, 0.f);   // one sample's six weights per 32-byte row, halved
  for (int j = 0; j < 6; ++j)
    for (int q = 0; q < nq; ++q) {
      double s = 0.0;
      for (int i = 0; i < 6; ++i) s += M[j][6 + i] * A[(size_t)q * 6 + i];
      pinv[(size_t)q * 8 + j] = 0.5f * (float)s;
    }
  return LLR_OK;
}

}  // namespace

}  // namespace llr

using namespace llr;

extern "C" {

int llr_dti_fit_dev(const llr_cf32* d_dwi, int32_t nq, const llr_cf32* d_b0, int32_t nb0, int64_t n_vox,
                    const float* b_vals, const float* b_vecs, float* d_out, void* stream) {
  if (!d_dwi || !b_vals || !b_vecs || !d_out || nq < 6 || nb0 < 0 || (nb0 > 0 && !d_b0) || n_vox < 0)
    return set_error(LLR_ERR_INVALID, "bad DTI fit arguments (need >= 6 diffusion volumes)");
  if (n_vox == 0) return LLR_OK;
  std::vector<float> pinv;
  LLR_TRY(design_pinv(b_vals, b_vecs, nq, pinv));
  cudaStream_t s = (cudaStream_t)stream;
  float* d_pinv = nullptr;
  LLR_CUDA_TRY(scratch_alloc((void**)&d_pinv, sizeof(float) * pinv.size(), s));
  cudaError_t e = cudaMemcpyAsync(d_pinv, pinv.data(), sizeof(float) * pinv.size(), cudaMemcpyHostToDevice, s);
  const size_t smem = sizeof(float) * 8 * (size_t)nq;
  if (e == cudaSuccess && smem > 48 * 1024)
    e = allow_smem(dti_fit_kernel);
  if (e == cudaSuccess) {
    const long long blocks = std::min<long long>((n_vox + 511) / 512, 148LL * 32);
    note_launch();
    dti_fit_kernel<<<(unsigned)blocks, 256, smem, s>>>(
        (const float2*)d_dwi, (const float2*)d_b0, n_vox, nq, nb0, d_pinv, d_out);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);   // the host pinv copy must outlive the transfer
  cudaFreeAsync(d_pinv, s);
  if (e != cudaSuccess) return cuda_error(e, "dti_fit_kernel", __FILE__, __LINE__);
  return LLR_OK;
}

int llr_dti_fit(const llr_cf32* dwi, int32_t nq, const llr_cf32* b0, int32_t nb0, int64_t n_vox, const float* b_vals,
                const float* b_vecs, float* out) {
  if (!dwi || !out || (nb0 > 0 && !b0) || n_vox < 0) return set_error(LLR_ERR_INVALID, "null pointer");
  float2 *d_dwi = nullptr, *d_b0 = nullptr;
  float* d_out = nullptr;
  int st = LLR_OK;
  auto fail = [&](int code) {
    cudaFree(d_dwi);
    cudaFree(d_b0);
    cudaFree(d_out);
    return code;
  };
  cudaError_t e = device_alloc((void**)&d_dwi, sizeof(float2) * (size_t)n_vox * nq);
  if (e == cudaSuccess && nb0 > 0) e = device_alloc((void**)&d_b0, sizeof(float2) * (size_t)n_vox * nb0);
  if (e == cudaSuccess) e = device_alloc((void**)&d_out, sizeof(float) * (size_t)n_vox * kDtiOut);
  if (e == cudaSuccess) e = cudaMemcpy(d_dwi, dwi, sizeof(float2) * (size_t)n_vox * nq, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && nb0 > 0)
    e = cudaMemcpy(d_b0, b0, sizeof(float2) * (size_t)n_vox * nb0, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return fail(cuda_error(e, "DTI fit buffers", __FILE__, __LINE__));
  st = llr_dti_fit_dev((const llr_cf32*)d_dwi, nq, (const llr_cf32*)d_b0, nb0, n_vox, b_vals, b_vecs, d_out, nullptr);
  if (st != LLR_OK) return fail(st);
  e = cudaMemcpy(out, d_out, sizeof(float) * (size_t)n_vox * kDtiOut, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return fail(cuda_error(e, "cudaMemcpy", __FILE__, __LINE__));
  return fail(LLR_OK);
}

}  // extern "C"

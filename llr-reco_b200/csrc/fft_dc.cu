// Fused hybrid-space data consistency: forward 2-D DFT over (y, z), hard DC on the sampled
// lines, inverse 2-D DFT, for one (x, volume) plane at a time with the plane held in shared
// memory.  One HBM read and one write of the iterate per iteration, against two of each per
// cuFFT pass plus the DC pass (signal_model.rs:34-79 with the x-transform cancelled, see the
// hybrid-space identity; hard_project lib.rs:392-406 on the sampled lines).
//
// Each axis of length N = N1 * N2 is a four-step transform in place: N2 register DFTs of
// length N1 (stride N2) with twiddles W_N^{n2 k1}, then N1 register DFTs of length N2; the
// spectrum is left in the permuted order p = N2 (k mod N1) + k / N1, which the DC indexes
// directly and the inverse (the same steps mirrored) consumes.  Register DFTs have lengths 1 to 16
// (fft_codelets.cuh); a length whose factors do not fit that (a prime above 16, say) goes to cuFFT.
// Forward and inverse are unnormalised like cuFFT's; the residual sum |F x - yhat|^2 is
// accumulated in FP64 per CTA (fixed plane order) for the deterministic finalize kernel.
#include <cmath>
#include <cstdio>
#include <vector>
#include <algorithm>

#include "llr_common.cuh"
#include "llr_internal.h"
#include "llr_prox_common.cuh"
#include "fft_codelets.cuh"

namespace llr {

namespace {

__host__ __device__ inline size_t align16b(size_t x) { return (x + 15) & ~size_t(15); }

// Twiddle-table layout in shared memory (float2 entries): W_ny^j, then W_nz^j.
struct FftTab {
  int off_y, off_z, total;
};

__host__ __device__ inline FftTab fft_tab(int ny, int nz) { return FftTab{0, ny, ny + nz}; }

// One pass over every transform of an axis: B transforms (batch stride bs), each of length
// N = N1 N2 with element stride es.  STEP 0: DFTs of length R = N1 over n1 (stride N2), then
// twiddles; STEP 1: DFTs of length R = N2 over contiguous positions.  Forward order: 0 then 1;
// inverse: 1 then 0 (twiddles before the DFT).
template <int R, int DIR, int STEP>
__device__ __forceinline__ void axis_pass(float2* s, FastDiv dB, int bs, int es, int N1, int N2, const float2* wN) {
  const int J = STEP == 0 ? N2 : N1;   // transforms of length R per batch entry
  const int tasks = (int)dB.d * J;
  const int st = STEP == 0 ? N2 * es : es;
  for (int t = threadIdx.x; t < tasks; t += blockDim.x) {
    const int j = (int)dB.div(t), b = t - j * (int)dB.d;
    float2* base = s + b * bs + (STEP == 0 ? j * es : N2 * j * es);
    float2 v[R];
    if (STEP == 0) {   // j = n2; elements at N2 n1 + n2
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = base[i * st];
      // twiddle W_N^{n2 k1}, n2 k1 < N (before the inverse DFT, after the forward one)
      if (DIR < 0) {
#pragma unroll
        for (int i = 1; i < R; ++i) v[i] = twmul<DIR>(v[i], wN[j * i]);
      }
      Dft<R, DIR>::run(v, nullptr);
      if (DIR > 0) {
#pragma unroll
        for (int i = 1; i < R; ++i) v[i] = twmul<DIR>(v[i], wN[j * i]);
      }
#pragma unroll
      for (int i = 0; i < R; ++i) base[i * st] = v[i];
    } else {           // j = k1; elements at N2 k1 + n2
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = base[i * st];
      Dft<R, DIR>::run(v, nullptr);
#pragma unroll
      for (int i = 0; i < R; ++i) base[i * st] = v[i];
    }
  }
}

template <int DIR, int STEP>
__device__ __forceinline__ void axis_dispatch(float2* s, FastDiv dB, int bs, int es, int N1, int N2, const float2* wN) {
  with_radix(STEP == 0 ? N1 : N2, [&](auto rc) {
    axis_pass<decltype(rc)::value, DIR, STEP>(s, dB, bs, es, N1, N2, wN);
  });
}

__device__ __forceinline__ int perm_pos(int k, int N1, int N2) { return N2 * (k % N1) + k / N1; }

struct FftDcArgs {
  float2* u;                 // planar iterate: plane (ix, q) at ny * nz * (ix + nx * q)
  const float2* yhat;        // per volume q: nx x L_q, x-major (line index fastest)
  const int* pos;            // sampled (ky + ny kz) per line
  const long long* off;      // line offsets per volume (nq + 1)
  const float2* twiddle;     // FftTab entries
  double* partials;          // one FP64 residual per CTA
  int nx, ny, nz, nq;
  int y1, y2, z1, z2;        // ny = y1 y2, nz = z1 z2
  int pitch;                 // odd row pitch of the shared plane
  FastDiv dny, dnz;
  float unc_scale;           // run-time sizes, != 0: elements outside the block grid of zsrc are multiplied by
                             // this as they are loaded (the prox leaves them raw)
  const int* zero_ra;        // optional: per-block kept counts of this iteration's prox; blocks
                             // with 0 were left unwritten and are zero-filled on load
  BlockSource zsrc;          // block grid and shift of that prox (when zero_ra is set)
};

constexpr int kZeroFlagMax = 4096;   // blocks per (x) block slab covered by the zero-fill table

// Passes of one axis with every size a compile-time constant (hot plane shapes).
template <int DIR, int STEP, int B, int BS, int ES, int N1, int N2, int NT>
__device__ __forceinline__ void axis_pass_fixed(float2* s, const float2* wN) {
  constexpr int R = STEP == 0 ? N1 : N2;
  constexpr int J = STEP == 0 ? N2 : N1;
  constexpr int TASKS = B * J;
#pragma unroll 1
  for (int t = threadIdx.x; t < TASKS; t += NT) {
    const int b = t % B, j = t / B;
    float2* base = s + b * BS + (STEP == 0 ? j : N2 * j) * ES;
    float2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = base[(STEP == 0 ? N2 * i : i) * ES];
    if (STEP == 0 && DIR < 0) {
#pragma unroll
      for (int i = 1; i < R; ++i) v[i] = twmul<DIR>(v[i], wN[j * i]);
    }
    Dft<R, DIR>::run(v, nullptr);
    if (STEP == 0 && DIR > 0) {
#pragma unroll
      for (int i = 1; i < R; ++i) v[i] = twmul<DIR>(v[i], wN[j * i]);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) base[(STEP == 0 ? N2 * i : i) * ES] = v[i];
  }
}

// First forward / last inverse pass of the z axis (step 0: DFTs of length Z1 at stride Z2 down z)
// on the plane in HBM (element (y, z) at g[y + ny z], lanes along y: 256-byte warp accesses) and
// the shared plane (row pitch PP) on the other side: the forward pass loads its elements straight
// into registers, zero-filling those of zero blocks (zero(y, z)), and stores the twiddled result
// in shared memory; the inverse pass reads shared memory and stores its result to HBM.
template <int DIR, int NY, int PP, int Z1, int Z2, int NT, class ZeroFn>
__device__ __forceinline__ void z_pass_hbm(float2* s, float2* g, const float2* wN, ZeroFn zero) {
  constexpr int TASKS = NY * Z2;
#pragma unroll 1
  for (int t = threadIdx.x; t < TASKS; t += NT) {
    const int y = t % NY, j = t / NY;
    float2* sb = s + y + PP * j;
    float2* gb = g + y + NY * j;
    float2 v[Z1];
    if (DIR > 0) {
#pragma unroll
      for (int i = 0; i < Z1; ++i) v[i] = zero(y, Z2 * i + j) ? make_float2(0.f, 0.f) : gb[NY * Z2 * i];
      Dft<Z1, DIR>::run(v, nullptr);
#pragma unroll
      for (int i = 1; i < Z1; ++i) v[i] = twmul<DIR>(v[i], wN[j * i]);
#pragma unroll
      for (int i = 0; i < Z1; ++i) sb[PP * Z2 * i] = v[i];
    } else {
#pragma unroll
      for (int i = 0; i < Z1; ++i) v[i] = sb[PP * Z2 * i];
#pragma unroll
      for (int i = 1; i < Z1; ++i) v[i] = twmul<DIR>(v[i], wN[j * i]);
      Dft<Z1, DIR>::run(v, nullptr);
#pragma unroll
      for (int i = 0; i < Z1; ++i) gb[NY * Z2 * i] = v[i];
    }
  }
}

// Plane geometry with run-time sizes (any shape radix_split accepts).
struct GeoRt {
  static constexpr bool kHbmPasses = false;
  int ny, nz, y1, y2, z1, z2, P;
  FastDiv dny, dnz;
  __device__ void forward(float2* s, const float2* tw, const FftTab& T) const {
    axis_dispatch<1, 0>(s, dnz, P, 1, y1, y2, tw + T.off_y);
    __syncthreads();
    axis_dispatch<1, 1>(s, dnz, P, 1, y1, y2, tw + T.off_y);
    __syncthreads();
    axis_dispatch<1, 0>(s, dny, 1, P, z1, z2, tw + T.off_z);
    __syncthreads();
    axis_dispatch<1, 1>(s, dny, 1, P, z1, z2, tw + T.off_z);
  }
  __device__ void inverse(float2* s, const float2* tw, const FftTab& T) const {
    axis_dispatch<-1, 1>(s, dny, 1, P, z1, z2, tw + T.off_z);
    __syncthreads();
    axis_dispatch<-1, 0>(s, dny, 1, P, z1, z2, tw + T.off_z);
    __syncthreads();
    axis_dispatch<-1, 1>(s, dnz, P, 1, y1, y2, tw + T.off_y);
    __syncthreads();
    axis_dispatch<-1, 0>(s, dnz, P, 1, y1, y2, tw + T.off_y);
  }
};

// Plane geometry with compile-time sizes: ny = Y1 Y2, nz = Z1 Z2, NT threads.  The forward
// transform runs the z axis first and the inverse the z axis last, so that the z axis's step-0
// pass reads (forward) and writes (inverse) the plane in HBM directly; the y-axis passes and the
// z axis's step 1 run in shared memory.  Each axis leaves its spectrum in the same permuted order
// whichever axis runs first.
template <int Y1, int Y2, int Z1, int Z2, int NT>
struct GeoFixed {
  static constexpr bool kHbmPasses = true;
  static constexpr int NY = Y1 * Y2, NZ = Z1 * Z2, PP = NY | 1;
  int ny = NY, nz = NZ, y1 = Y1, y2 = Y2, z1 = Z1, z2 = Z2, P = PP;
  template <class ZeroFn>
  __device__ void forward_hbm(float2* s, float2* g, const float2* tw, const FftTab& T, ZeroFn zero) const {
    z_pass_hbm<1, NY, PP, Z1, Z2, NT>(s, g, tw + T.off_z, zero);
    __syncthreads();
    axis_pass_fixed<1, 1, NY, 1, PP, Z1, Z2, NT>(s, tw + T.off_z);
    __syncthreads();
    axis_pass_fixed<1, 0, NZ, PP, 1, Y1, Y2, NT>(s, tw + T.off_y);
    __syncthreads();
    axis_pass_fixed<1, 1, NZ, PP, 1, Y1, Y2, NT>(s, tw + T.off_y);
  }
  __device__ void inverse_hbm(float2* s, float2* g, const float2* tw, const FftTab& T) const {
    axis_pass_fixed<-1, 1, NZ, PP, 1, Y1, Y2, NT>(s, tw + T.off_y);
    __syncthreads();
    axis_pass_fixed<-1, 0, NZ, PP, 1, Y1, Y2, NT>(s, tw + T.off_y);
    __syncthreads();
    axis_pass_fixed<-1, 1, NY, 1, PP, Z1, Z2, NT>(s, tw + T.off_z);
    __syncthreads();
    z_pass_hbm<-1, NY, PP, Z1, Z2, NT>(s, g, tw + T.off_z, [](int, int) { return false; });
  }
};

template <class Geo>
__device__ __forceinline__ void fft_dc_body(const FftDcArgs& a, const Geo& geo) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int ny = geo.ny, nz = geo.nz, P = geo.P;
  const FftTab T = fft_tab(ny, nz);
  float2* tw = reinterpret_cast<float2*>(smem);
  double* red = reinterpret_cast<double*>(smem + align16b(sizeof(float2) * T.total));
  float2* s = reinterpret_cast<float2*>(smem + align16b(sizeof(float2) * T.total) + 32 * sizeof(double));
  // zero-fill tables: block column of every y, block row of every z (-1: no block), the shift,
  // and one flag per block of the current x slab
  int* zgy = reinterpret_cast<int*>(s + (size_t)P * nz);
  int* zgz = zgy + ny;
  int* zsh = zgz + nz;
  unsigned char* zfl = reinterpret_cast<unsigned char*>(smem + align16b(sizeof(float2) * T.total) +
                                                        32 * sizeof(double) + sizeof(float2) * (size_t)P * nz +
                                                        align16b(sizeof(int) * (size_t)(ny + nz + 4)));
  const bool zf = a.zero_ra != nullptr;
  const bool unc = !Geo::kHbmPasses && a.unc_scale != 0.f;
  const int tid = threadIdx.x;
  for (int i = tid; i < T.total; i += blockDim.x) tw[i] = a.twiddle[i];
  if (zf || unc) {
    if (tid == 0) block_shift(a.zsrc, zsh);
    __syncthreads();
    const BlockSource& zs = a.zsrc;
    for (int y = tid; y < ny; y += blockDim.x) {
      int r = (y - zsh[1]) % ny;
      if (r < 0) r += ny;
      zgy[y] = r < zs.gy * zs.by ? r / zs.by : -1;
    }
    for (int z = tid; z < nz; z += blockDim.x) {
      int r = (z - zsh[2]) % nz;
      if (r < 0) r += nz;
      zgz[z] = r < zs.gz * zs.bz ? r / zs.bz : -1;
    }
  }
  // element (y, z) of the current plane lies in a block whose prox output was left unwritten
  // (the block column of the thread's y is cached: with a thread count that is a multiple of ny,
  // y never changes along a thread's elements)
  int zy = -1, zby = -1;
  auto zero_at = [&](int y, int z) {
    if (!zf) return false;
    if (y != zy) { zy = y; zby = zgy[y]; }
    const int bz = zgz[z];
    return zby >= 0 && bz >= 0 && zfl[zby + a.zsrc.gy * bz] != 0;
  };
  const long long nyz = (long long)ny * nz;
  const long long planes = (long long)a.nx * a.nq;
  double err = 0.0;
  for (long long pl = blockIdx.x; pl < planes; pl += gridDim.x) {
    const int q = (int)(pl / a.nx), ix = (int)(pl - (long long)q * a.nx);
    float2* g = a.u + pl * nyz;
    __syncthreads();   // previous plane stored, twiddles visible
    int gxi = 0;
    if (zf || unc) {
      const BlockSource& zs = a.zsrc;
      int r = (ix - zsh[0]) % a.nx;
      if (r < 0) r += a.nx;
      gxi = r < zs.gx * zs.bx ? r / zs.bx : -1;
    }
    if (zf) {          // flags of the blocks of this plane's x slab
      const int nslab = a.zsrc.gy * a.zsrc.gz;
      for (int t = tid; t < nslab; t += blockDim.x)
        zfl[t] = gxi >= 0 && a.zero_ra[t + (long long)nslab * gxi] == 0;
      __syncthreads();
    }
    if constexpr (Geo::kHbmPasses) {
      // forward: z axis (its first pass loads the plane from HBM), then y axis
      geo.forward_hbm(s, g, tw, T, zero_at);
    } else {
      // asynchronous 8-byte copies: every element in flight at once, no register staging; elements of
      // blocks left unwritten become zero, those outside the block grid are scaled
      for (int e = tid; e < ny * nz; e += blockDim.x) {
        const int z = (int)geo.dny.div(e), y = e - z * ny;
        float2* d = s + z * P + y;
        if (zf || unc) {
          const int by = zgy[y], bz = zgz[z];
          if (by < 0 || bz < 0 || gxi < 0) {
            if (unc) {
              *d = cscale(g[e], a.unc_scale);
              continue;
            }
          } else if (zf && zfl[by + a.zsrc.gy * bz]) {
            *d = make_float2(0.f, 0.f);
            continue;
          }
        }
        const unsigned dst = (unsigned)__cvta_generic_to_shared(d);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(g + e) : "memory");
      }
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      // forward: y axis (rows, element stride 1, batch stride P), then z axis (columns)
      geo.forward(s, tw, T);
    }
    __syncthreads();
    // hard DC on the sampled lines of this plane
    {
      const long long o0 = a.off[q], L = a.off[q + 1] - o0;
      const float2* yq = a.yhat + o0 * a.nx + (long long)ix * L;
      const int* pq = a.pos + o0;
      for (long long l = tid; l < L; l += blockDim.x) {
        const int p = pq[l];
        const int ky = p % ny, kz = p / ny;
        const int at = perm_pos(kz, geo.z1, geo.z2) * P + perm_pos(ky, geo.y1, geo.y2);
        const float2 yv = yq[l];
        const float2 uv = s[at];
        const double dx = (double)uv.x - (double)yv.x, dy2 = (double)uv.y - (double)yv.y;
        err += dx * dx + dy2 * dy2;
        s[at] = yv;
      }
    }
    __syncthreads();
    if constexpr (Geo::kHbmPasses) {
      // inverse: y axis, then z axis (its last pass stores the plane to HBM)
      geo.inverse_hbm(s, g, tw, T);
    } else {
      // inverse: z axis then y axis, each mirrored (step 1 then step 0)
      geo.inverse(s, tw, T);
      __syncthreads();
      for (int e = tid; e < ny * nz; e += blockDim.x) {
        const int z = (int)geo.dny.div(e);
        g[e] = s[z * P + e - z * ny];
      }
    }
  }
  // deterministic CTA reduction of the residual
  for (int o = 16; o > 0; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
  __syncthreads();
  if ((tid & 31) == 0) red[tid >> 5] = err;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    a.partials[blockIdx.x] = t;
  }
}

// Run-time sizes.  Every instance keeps 24 warps per SM at 85 registers; small planes run them as several
// small CTAs, whose barriers hold back fewer warps (75 x 52 planes, 90 x 33 of them: 264 us with one CTA
// of 512 threads per SM, 169 us now).
template <int NT, int PER_SM>
__global__ void __launch_bounds__(NT, PER_SM) fft_dc_kernel(FftDcArgs a) {
  GeoRt geo;
  geo.ny = a.ny; geo.nz = a.nz; geo.y1 = a.y1; geo.y2 = a.y2; geo.z1 = a.z1; geo.z2 = a.z2; geo.P = a.pitch;
  geo.dny = a.dny; geo.dnz = a.dnz;
  fft_dc_body(a, geo);
}

template <int Y1, int Y2, int Z1, int Z2, int NT>
__global__ void __launch_bounds__(NT, 1) fft_dc_fixed_kernel(FftDcArgs a) {
  fft_dc_body(a, GeoFixed<Y1, Y2, Z1, Z2, NT>());
}

size_t fft_dc_smem(int ny, int nz, int pitch) {
  const FftTab T = fft_tab(ny, nz);
  return align16b(sizeof(float2) * T.total) + 32 * sizeof(double) + sizeof(float2) * (size_t)pitch * nz +
         align16b(sizeof(int) * (size_t)(ny + nz + 4)) + kZeroFlagMax;
}

}  // namespace

bool fft_dc_supported(int ny, int nz) {
  int a, b, c, d;
  if (!radix_split(ny, a, b) || !radix_split(nz, c, d)) return false;
  return fft_dc_smem(ny, nz, ny | 1) <= 227 * 1024;
}

// FP64 twiddle table for fft_dc_kernel (FftTab layout), uploaded once per context.
std::vector<float2> fft_dc_twiddles(int ny, int nz) {
  const FftTab T = fft_tab(ny, nz);
  std::vector<float2> h((size_t)T.total);
  auto fill = [&](int off, int N) {
    for (int j = 0; j < N; ++j) {
      const double ang = -2.0 * M_PI * (double)j / (double)N;
      h[(size_t)off + j] = make_float2((float)std::cos(ang), (float)std::sin(ang));
    }
  };
  fill(T.off_y, ny);
  fill(T.off_z, nz);
  return h;
}

namespace {

// Compile-time instances for the hot plane shapes; every other factorable shape uses the
// run-time kernel.  The pass loops stride by the thread count, so any count is correct.
struct FftKernelChoice {
  void (*kern)(FftDcArgs);
  int nt, y1, y2, z1, z2;
};

FftKernelChoice choose_fft(int ny, int nz) {
  FftKernelChoice c;
  // 192 x 96 fills a CTA's shared memory (one CTA per SM): 24 warps (the pass loops take the
  // 1152-task first pass in two rounds); the smaller planes run several CTAs per SM.
  if (ny == 192 && nz == 96) c = {fft_dc_fixed_kernel<16, 12, 12, 8, 768>, 768, 16, 12, 12, 8};
  else if (ny == 96 && nz == 48) c = {fft_dc_fixed_kernel<12, 8, 8, 6, 192>, 192, 12, 8, 8, 6};
  else if (ny == 64 && nz == 64) c = {fft_dc_fixed_kernel<8, 8, 8, 8, 256>, 256, 8, 8, 8, 8};
  else {
    // CTAs per SM that the plane's shared memory allows
    const size_t per = (228 * 1024) / (fft_dc_smem(ny, nz, ny | 1) + 1024);
    if (per >= 6) c = {fft_dc_kernel<128, 6>, 128};
    else if (per >= 3) c = {fft_dc_kernel<256, 3>, 256};
    else if (per == 2) c = {fft_dc_kernel<384, 2>, 384};
    else c = {fft_dc_kernel<768, 1>, 768};
    radix_split(ny, c.y1, c.y2);
    radix_split(nz, c.z1, c.z2);
  }
  return c;
}

}  // namespace

// Whether the plane's kernel scales the elements outside the block grid itself.
bool fft_dc_scales_uncovered(int ny, int nz) {
  return !((ny == 192 && nz == 96) || (ny == 96 && nz == 48) || (ny == 64 && nz == 64));
}

int fft_dc_grid(int ny, int nz) {
  int dev = 0, nsm = 0, smem_sm = 0, regs_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev) != cudaSuccess) return 0;
  const FftKernelChoice c = choose_fft(ny, nz);
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, c.kern) != cudaSuccess) return 0;
  const int by_smem = smem_sm / (int)(fft_dc_smem(ny, nz, ny | 1) + 1024);
  const int regs_warp = ((fa.numRegs * 32 + 255) / 256) * 256;
  const int by_regs = regs_sm / std::max(1, regs_warp * (c.nt / 32));
  const int per = std::max(1, std::min(6, std::min(by_smem, by_regs)));
  return nsm * per;
}

// Planes of a few hundred samples leave a CTA more barriers than work; with several of them per CTA, cuFFT's batched kernels
// and the DC pass are faster.  Forward, DC and inverse, fused / cuFFT: 12000 planes of 5 x 5 79 / 37 us, 11 x 13
// 113 / 58, 16 x 16 105 / 73, 25 x 20 137 / 107, 25 x 25 154 / 145 us; 7680 of 35 x 30 139 / 161.  With up to two planes
// per CTA the launches count: 1920 planes of 16 x 16 34 / 35 us, 640 of 11 x 13 27 / 31.
bool fft_dc_preferred(int ny, int nz, long long planes) {
  return (long long)ny * nz >= 768 || planes <= 2ll * fft_dc_grid(ny, nz);
}

int launch_fft_dc(float2* u, const float2* yhat, const int* pos, const long long* off, const float2* twiddle,
                  const Geom& g, double* partials, int grid, const int* zero_ra, const BlockSource* zsrc,
                  float unc_scale, cudaStream_t s) {
  FftDcArgs a;
  a.zero_ra = nullptr;
  a.zsrc = BlockSource{};
  a.unc_scale = 0.f;
  if (unc_scale != 0.f && zsrc) {
    a.unc_scale = unc_scale;
    a.zsrc = *zsrc;
  }
  a.dny = FastDiv(g.ny);
  a.dnz = FastDiv(g.nz);
  if (zero_ra && zsrc && zsrc->kind == 1 && (long long)zsrc->gy * zsrc->gz <= kZeroFlagMax) {
    a.zero_ra = zero_ra;
    a.zsrc = *zsrc;
  }
  a.u = u; a.yhat = yhat; a.pos = pos; a.off = off; a.twiddle = twiddle; a.partials = partials;
  a.nx = g.nx; a.ny = g.ny; a.nz = g.nz; a.nq = g.nq;
  if (!fft_dc_supported(g.ny, g.nz))
    return set_error(LLR_ERR_UNSUPPORTED, "fused FFT: %d x %d plane is not supported", g.ny, g.nz);
  const FftKernelChoice c = choose_fft(g.ny, g.nz);
  a.y1 = c.y1; a.y2 = c.y2; a.z1 = c.z1; a.z2 = c.z2;
  a.pitch = g.ny | 1;
  const size_t smem = fft_dc_smem(g.ny, g.nz, a.pitch);
  LLR_CUDA_TRY(allow_smem(c.kern));
  LLR_CUDA_TRY(cudaFuncSetAttribute(c.kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  if (grid < 1) return set_error(LLR_ERR_INVALID, "fused FFT: empty grid");
  note_launch();
  c.kern<<<grid, c.nt, smem, s>>>(a);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

}  // namespace llr

// Hybrid-space data consistency for (y, z) planes that do not fit shared memory (signal_model.rs:34-79 with
// the x-transform cancelled, hard_project lib.rs:392-406): a column pass over z, a row pass over y that
// holds the data consistency, a column pass back.
//
//   columns forward   u(y, z) -> along z
//   rows              along y, replace the sampled (ky, kz), residual in FP64, back along y
//   columns inverse
//
// Every pass reads and writes the iterate once, with the line in registers and shared memory between (a
// line of length n = n1 n2 is two register DFTs and one exchange); natural order in HBM throughout.
// cuFFT's four kernels plus the scattered DC pass moved 64 + 8 bytes per element and rewrote single 8-byte
// samples; here it is 48.  At 128 x 256 x 256 x 61, rank 7, per iteration: expand 0.97 + cuFFT 2 x 2.53 + DC
// 1.45 ms before, coefficient columns 0.21 + expanding rows 2.33 + columns 1.65 ms now.
//
// Every plane whose extents factor comes here: data consistency with both transforms, 64 x 16 planes, cuFFT / here:
// 256 x 256 1.15 / 0.75 ms, 240 x 240 1.47 / 0.80, 224 x 224 1.44 / 0.68, 192 x 192 0.75 / 0.51, 176 x 176 0.63 / 0.49, 169 x 196
// 0.66 / 0.54, 130 x 256 0.68 / 0.58, 117 x 256 0.62 / 0.55; one plane of 256 x 256 32.5 / 31.4 us.  Length 256 alone
// has its sizes at compile time (the usual matrix size beyond shared memory): 11 ns per 1000 samples, other
// lengths 13 to 14.
//
// With a temporal subspace whose volumes share their phase, X = C S^H and the transforms commute: the forward
// transform runs on the srank coefficient volumes, and the row pass expands each k-space row of every
// volume from the srank transformed rows in shared memory before it applies the data consistency.  The
// expanded image and its forward passes are never stored.
#include <cmath>
#include <type_traits>
#include <vector>

#include "llr_internal.h"
#include "fft_codelets.cuh"

namespace llr {

namespace {

constexpr int kColThreads = 256;
constexpr int kRowThreads = 128;
constexpr int kColLanes = 32;

// f for the compile-time radix when FIX > 0, else for the run-time one
template <int FIX, class F>
__device__ __forceinline__ void radix_or(int R, F f) {
  if constexpr (FIX > 0) f(Radix<FIX>{});
  else with_radix(R, f);
}

struct ColArgs {
  const float2* src;
  float2* dst;
  const float2* tw;      // W_n^j
  long long planes;
  int nc;                // contiguous extent (lines per plane)
  int n, n1, n2;         // line length
  PhaseTab ph;           // forward: phase of volume 0 and scale applied on load (ph_on)
  Geom g;
  int ph_on;
  float scale;
};

// Bound: HBM, 16 bytes per element.  A CTA takes 32 adjacent lines (256-byte warp accesses); the first register
// DFT loads from HBM, the second stores to it.
template <int DIR, int N1, int N2>
__global__ void __launch_bounds__(kColThreads, 3) fft_cols_kernel(ColArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  float2* s = tw + a.n;                       // [n][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i = threadIdx.x; i < a.n; i += blockDim.x) tw[i] = a.tw[i];
  const int n1 = N1 ? N1 : a.n1, n2 = N2 ? N2 : a.n2;
  const long long per = (a.nc + kColLanes - 1) / kColLanes, total = a.planes * per;
  for (long long w = blockIdx.x; w < total; w += gridDim.x) {
    const long long p = w / per;
    const int y = (int)(w - p * per) * kColLanes + lane;
    const bool ok = y < a.nc;
    const int yc = min(y, a.nc - 1);
    const float2* src = a.src + p * a.nc * (long long)a.n + yc;
    float2* dst = a.dst + p * a.nc * (long long)a.n + y;
    float2 py = make_float2(1.f, 0.f);
    if (DIR > 0 && a.ph_on) {
      py = cscale(a.ph.y ? a.ph.y[yc] : py, a.scale);
      if (a.ph.x) py = cmul(py, a.ph.x[p % a.g.nx]);
    }
    __syncthreads();                          // the previous tile has left s; tw is in place
    radix_or<N1>(n1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int j = warp; j < n2; j += nw) {
        float2 v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = src[(long long)(n2 * i + j) * a.nc];
        if (DIR > 0 && a.ph_on) {
#pragma unroll
          for (int i = 0; i < R; ++i) v[i] = cmul(v[i], a.ph.z ? cmul(py, a.ph.z[n2 * i + j]) : py);
        }
        Dft<R, DIR>::run(v, nullptr);
#pragma unroll
        for (int i = 0; i < R; ++i)
          s[(i * n2 + j) * kColLanes + lane] = i == 0 ? v[0] : twmul<DIR>(v[i], tw[j * i]);
      }
    });
    __syncthreads();
    radix_or<N2>(n2, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int k1 = warp; k1 < n1; k1 += nw) {
        float2 v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = s[(k1 * n2 + i) * kColLanes + lane];
        Dft<R, DIR>::run(v, nullptr);
        if (ok) {
#pragma unroll
          for (int i = 0; i < R; ++i) dst[(long long)(k1 + n1 * i) * a.nc] = v[i];
        }
      }
    });
  }
}

struct RowArgs {
  float2* u;             // planar iterate
  const float2* coef;    // kExpand: srank volumes, transformed along z
  const float2* S;       // kExpand: nq x srank column-major
  int srank;
  const float2* tw;      // W_ny^j
  const int* rowptr;     // first sampled line of every (volume, kz) within its volume, nz + 1 per volume
  const int* pos;        // sampled ky + ny kz per line
  const float2* yhat;
  const long long* off;  // line offsets per volume
  double* partials;
  int nx, ny, nz, nq, n1, n2;
};

enum RowMode { kDc, kFill, kExpand };

// Row pass.  kDc / kFill: a CTA takes rt consecutive rows.  kExpand: a CTA takes one (ix, kz), transforms its
// srank coefficient rows along y into shared memory, and produces the row of every volume, rt at a time.
// A row's spectrum sits in shared memory in the order the register DFTs leave it (ky = k1 + n1 k2 at
// k1 pitch + k2) while its sampled lines alone are visited for the data consistency: testing every
// sample in registers cost 80 instructions per element (1.88 ms for kFill at 128 x 256 x 256 x 61, now
// 1.32), the lists a few.  kExpand holds the coefficients of two ky in registers for all volumes of a batch.
// Bound: HBM, 16 bytes per element (kFill, kExpand 8: the row is only written), then instruction issue: the
// sizes N1 x N2 given at compile time make the addresses immediates, and CTAs of 128 threads wait less
// at the barriers between the steps than CTAs of 256 (2.77 -> 2.36 ms).  kExpand 4.02 -> 2.36 ms there.
template <int MODE, int N1, int N2>
__global__ void __launch_bounds__(kRowThreads, 6) fft_rows_kernel(RowArgs a, int rt_) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[kRowThreads / 32];
  const int n1 = N1 ? N1 : a.n1, n2 = N2 ? N2 : a.n2, ny = n1 * n2;
  const int rt = N1 ? kRowThreads / (N1 > N2 ? N1 : N2) : rt_;
  const int pitch = n2 | 1, rp = n1 * pitch;
  float2* tw = reinterpret_cast<float2*>(smem);
  float2* s = tw + ny;
  float4* Ss = reinterpret_cast<float4*>(s + (((size_t)rt * rp + ny) & 1 ? (size_t)rt * rp + 1 : (size_t)rt * rp));
  float2* cs = reinterpret_cast<float2*>(Ss + (MODE == kExpand ? a.nq * a.srank : 0));   // kExpand: [srank][ny]
  const int tid = threadIdx.x;
  for (int i = tid; i < ny; i += kRowThreads) tw[i] = a.tw[i];
  if (MODE == kExpand)   // c conj(S) = c.x (S.x, -S.y) + c.y (S.y, S.x)
    for (int i = tid; i < a.nq * a.srank; i += kRowThreads) {
      const int q = i / a.srank, k = i - q * a.srank;
      const float2 sv = a.S[q + (long long)a.nq * k];
      Ss[i] = make_float4(sv.x, -sv.y, sv.y, sv.x);
    }
  double err = 0.0;
  const long long rows = (long long)a.nx * a.nz * a.nq;
  const long long items = MODE == kExpand ? (long long)a.nx * a.nz : (rows + rt - 1) / rt;
  const int tpr = max(1, kRowThreads / rt);     // threads per row in the data consistency
  // first register DFT of `rn` rows at src (row stride rs), into s
  auto forward_step0 = [&](const float2* src, long long rs, int rn) {
    radix_or<N1>(n1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int t = tid; t < rn * n2; t += kRowThreads) {
        const int r = t / n2, j = t - r * n2;
        const float2* g = src + r * rs + j;
        float2* sr = s + r * rp + j;
        float2 v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = g[n2 * i];
        Dft<R, 1>::run(v, nullptr);
#pragma unroll
        for (int i = 0; i < R; ++i) sr[i * pitch] = i == 0 ? v[0] : twmul<1>(v[i], tw[j * i]);
      }
    });
  };
  // second register DFT of `rn` rows in place (DIR < 0: the first one of the inverse, with its twiddles)
  auto inner_step = [&](auto dir, int rn) {
    constexpr int DIR = decltype(dir)::value;
    radix_or<N2>(n2, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int t = tid; t < rn * n1; t += kRowThreads) {
        const int r = t / n1, k1 = t - r * n1;
        float2* sr = s + r * rp + k1 * pitch;
        float2 v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = sr[i];
        Dft<R, DIR>::run(v, nullptr);
#pragma unroll
        for (int i = 0; i < R; ++i) sr[i] = DIR < 0 ? twmul<-1>(v[i], tw[k1 * i]) : v[i];
      }
    });
  };
  for (long long it = blockIdx.x; it < items; it += gridDim.x) {
    __syncthreads();
    if (MODE == kExpand) {
      // the item's coefficient rows, forward along y, rt at a time
      const long long rs = (long long)a.nx * a.nz * ny;
      for (int k0 = 0; k0 < a.srank; k0 += rt) {
        const int kn = min(rt, a.srank - k0);
        forward_step0(a.coef + ((long long)k0 * a.nx * a.nz + it) * ny, rs, kn);
        __syncthreads();
        inner_step(std::integral_constant<int, 1>{}, kn);
        __syncthreads();
        for (int t = tid; t < kn * ny; t += kRowThreads) {
          const int r = t / ny, ky = t - r * ny;
          cs[(k0 + r) * ny + ky] = s[r * rp + (ky % n1) * pitch + ky / n1];
        }
        __syncthreads();
      }
    }
    const int batches = MODE == kExpand ? (a.nq + rt - 1) / rt : 1;
    for (int bt = 0; bt < batches; ++bt) {
      const int rn = MODE == kExpand ? min(rt, a.nq - bt * rt) : (int)min((long long)rt, rows - it * rt);
      // first row of this batch (row r follows at stride rs): volume, x plane and kz
      const long long row0 = MODE == kExpand ? (long long)bt * rt * a.nx * a.nz + it : it * rt;
      const long long rs = (MODE == kExpand ? (long long)a.nx * a.nz : 1LL) * ny;
      const long long xq0 = row0 / a.nz;
      const int kz0 = (int)(row0 - xq0 * a.nz), q0 = (int)(xq0 / a.nx), ix0 = (int)(xq0 - (long long)q0 * a.nx);
      if (MODE == kDc) {
        forward_step0(a.u + row0 * ny, rs, rn);
        __syncthreads();
        inner_step(std::integral_constant<int, 1>{}, rn);
      } else if (MODE == kFill) {
        for (int t = tid; t < rn * rp; t += kRowThreads) s[t] = make_float2(0.f, 0.f);
      } else {
        // two ky (a half row apart) of four volumes per thread
        const int half = (ny + 1) / 2;
        for (int t = tid; t < half * ((rn + 3) / 4); t += kRowThreads) {
          const int r0 = t / half * 4, k1st = t % half;
          const bool two = k1st + half < ny;
          const int k2nd = two ? k1st + half : k1st;
          float2* d0 = s + r0 * rp + (k1st % n1) * pitch + k1st / n1;
          float2* d1 = s + r0 * rp + (k2nd % n1) * pitch + k2nd / n1;
          float2 v0[4], v1[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) v0[e] = v1[e] = make_float2(0.f, 0.f);
          const float4* S0 = Ss + (size_t)(bt * rt + r0) * a.srank;
          int so[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) so[e] = min(e, rn - 1 - r0) * a.srank;
          for (int k = 0; k < a.srank; ++k) {
            const float2 c0 = cs[k * ny + k1st], c1 = cs[k * ny + k2nd];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float4 sv = S0[so[e] + k];
              cfma2(v0[e], c0, make_float2(sv.x, sv.y), make_float2(sv.z, sv.w));
              cfma2(v1[e], c1, make_float2(sv.x, sv.y), make_float2(sv.z, sv.w));
            }
          }
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (r0 + e < rn) {
              d0[e * rp] = v0[e];
              if (two) d1[e * rp] = v1[e];
            }
        }
      }
      __syncthreads();
      // hard data consistency on the sampled lines of each row
      for (int t = tid; t < rn * tpr; t += kRowThreads) {
        const int r = t / tpr, sub = t - r * tpr;
        int kz = kz0, ix = ix0, q = q0;
        if (MODE == kExpand) {
          q += r;
        } else {
          const int dz = (kz0 + r) / a.nz, dx = (ix0 + dz) / a.nx;
          kz += r - dz * a.nz;
          ix += dz - dx * a.nx;
          q += dx;
        }
        const int* rw = a.rowptr + (long long)q * (a.nz + 1) + kz;
        const int lo = rw[0], hi = rw[1];
        const long long o0 = a.off[q], L = a.off[q + 1] - o0;
        const float2* yq = a.yhat + o0 * a.nx + (long long)ix * L;
        const int* pq = a.pos + o0;
        for (int l = lo + sub; l < hi; l += tpr) {
          const int ky = pq[l] - ny * kz;
          const float2 yv = yq[l];
          float2* at = s + r * rp + (ky % n1) * pitch + ky / n1;
          if (MODE != kFill) {
            const float2 uv = *at;
            const double dx = (double)uv.x - (double)yv.x, dy = (double)uv.y - (double)yv.y;
            err += dx * dx + dy * dy;
          }
          *at = yv;
        }
      }
      __syncthreads();
      inner_step(std::integral_constant<int, -1>{}, rn);
      __syncthreads();
      radix_or<N1>(n1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        for (int t = tid; t < rn * n2; t += kRowThreads) {
          const int r = t / n2, j = t - r * n2;
          float2* dst = a.u + row0 * ny + r * rs + j;
          const float2* sr = s + r * rp + j;
          float2 v[R];
#pragma unroll
          for (int i = 0; i < R; ++i) v[i] = sr[i * pitch];
          Dft<R, -1>::run(v, nullptr);
#pragma unroll
          for (int i = 0; i < R; ++i) dst[n2 * i] = v[i];
        }
      });
      if (MODE == kExpand) __syncthreads();
    }
  }
  if (MODE == kFill) return;
  // deterministic CTA reduction of the residual
  for (int o = 16; o > 0; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
  if ((tid & 31) == 0) red[tid >> 5] = err;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < kRowThreads / 32; ++w) t += red[w];
    a.partials[blockIdx.x] = t;
  }
}

size_t col_smem(int n) { return sizeof(float2) * ((size_t)n + (size_t)n * kColLanes); }

// rows per batch: as many as fill the threads in the wider of the two register passes
int rows_per_batch(int n1, int n2) { return std::max(1, kRowThreads / std::max(n1, n2)); }

size_t row_smem(int n1, int n2, int nq, int srank) {
  return sizeof(float2) * ((size_t)n1 * n2 + (size_t)rows_per_batch(n1, n2) * n1 * (n2 | 1) + 2 +
                           (size_t)srank * n1 * n2 + 2 * (size_t)srank * nq);
}

template <class K>
int resident_grid(K kern, int threads, size_t sm, long long items, int* grid) {
  int dev = 0, nsm = 0, occ = 0;
  LLR_CUDA_TRY(cudaGetDevice(&dev));
  LLR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  LLR_CUDA_TRY(allow_smem(kern));
  LLR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, sm));
  if (occ < 1) return set_error(LLR_ERR_UNSUPPORTED, "row / column FFT kernel needs %zu B of shared memory", sm);
  *grid = (int)std::max<long long>(1, std::min<long long>(items, (long long)nsm * occ));
  return LLR_OK;
}

}  // namespace

bool fft_rows_supported(int ny, int nz) {
  int a, b;
  return radix_split(ny, a, b) && radix_split(nz, a, b);
}

// The expanding row pass keeps srank rows, S and the exchange buffer in shared memory.  More than 64 volumes are
// refused by launch_subspace_expand, whatever the plane.
bool fft_rows_expand_supported(int ny, int nq, int srank) {
  int a, b;
  return nq <= 64 && radix_split(ny, a, b) && row_smem(a, b, nq, srank) <= 200 * 1024;
}

// W_ny^j then W_nz^j, FP64-computed.
std::vector<float2> fft_rows_twiddles(int ny, int nz) {
  std::vector<float2> h((size_t)ny + nz);
  for (int i = 0; i < ny + nz; ++i) {
    const int N = i < ny ? ny : nz, j = i < ny ? i : i - ny;
    const double ang = -2.0 * M_PI * (double)j / (double)N;
    h[i] = make_float2((float)std::cos(ang), (float)std::sin(ang));
  }
  return h;
}

// First line of every (volume, kz) within its volume, from the sorted line positions of every volume.
std::vector<int> fft_rows_ptr(const std::vector<int>& pos, const std::vector<long long>& off, int ny, int nz) {
  const int nq = (int)off.size() - 1;
  std::vector<int> p((size_t)nq * (nz + 1));
  for (int q = 0; q < nq; ++q) {
    long long l = off[q];
    for (int kz = 0; kz <= nz; ++kz) {
      while (l < off[q + 1] && pos[l] < ny * kz) ++l;
      p[(size_t)q * (nz + 1) + kz] = (int)(l - off[q]);
    }
  }
  return p;
}

// Column transforms along z of `planes` planes, in place or src -> dst; with ph, the load applies the phase of
// volume 0 and `scale`.
int launch_fft_cols(const float2* src, float2* dst, const float2* tw_z, const Geom& g, long long planes, int dir,
                    const PhaseTab* ph, float scale, cudaStream_t s) {
  ColArgs a = {};
  a.src = src; a.dst = dst; a.tw = tw_z; a.planes = planes; a.nc = g.ny; a.n = g.nz; a.g = g; a.scale = scale;
  if (!radix_split(g.nz, a.n1, a.n2)) return set_error(LLR_ERR_UNSUPPORTED, "column FFT of length %d", g.nz);
  if (ph) { a.ph = *ph; a.ph_on = 1; }
  void (*kern)(ColArgs) = dir > 0 ? fft_cols_kernel<1, 0, 0> : fft_cols_kernel<-1, 0, 0>;
  if (a.n1 == 16 && a.n2 == 16) kern = dir > 0 ? fft_cols_kernel<1, 16, 16> : fft_cols_kernel<-1, 16, 16>;
  int grid = 0;
  LLR_TRY(resident_grid(kern, kColThreads, col_smem(g.nz), planes * ((g.ny + kColLanes - 1) / kColLanes), &grid));
  note_launch();
  kern<<<grid, kColThreads, col_smem(g.nz), s>>>(a);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

// Row pass (mode 0: data consistency, 1: zero-filled start, 2: expand from coef); *np receives the number of
// residual partials (at most 148 x 8).
int launch_fft_rows(int mode, float2* u, const float2* coef, const float2* S, int srank, const float2* tw_y,
                    const int* rowptr, const int* pos, const float2* yhat, const long long* off, const Geom& g,
                    double* partials, int* np, cudaStream_t s) {
  RowArgs a = {};
  a.u = u; a.coef = coef; a.S = S; a.srank = mode == 2 ? srank : 0; a.tw = tw_y; a.rowptr = rowptr;
  a.pos = pos; a.yhat = yhat; a.off = off; a.partials = partials;
  a.nx = g.nx; a.ny = g.ny; a.nz = g.nz; a.nq = g.nq;
  if (!radix_split(g.ny, a.n1, a.n2)) return set_error(LLR_ERR_UNSUPPORTED, "row FFT of length %d", g.ny);
  const int rt = rows_per_batch(a.n1, a.n2);
  const size_t sm = row_smem(a.n1, a.n2, g.nq, a.srank);
  const long long rows = (long long)g.nx * g.nz * g.nq;
  void (*kern)(RowArgs, int) = mode == 2   ? fft_rows_kernel<kExpand, 0, 0>
                               : mode == 1 ? fft_rows_kernel<kFill, 0, 0>
                                           : fft_rows_kernel<kDc, 0, 0>;
  if (a.n1 == 16 && a.n2 == 16)
    kern = mode == 2 ? fft_rows_kernel<kExpand, 16, 16> : mode == 1 ? fft_rows_kernel<kFill, 16, 16> : fft_rows_kernel<kDc, 16, 16>;
  int grid = 0;
  LLR_TRY(resident_grid(kern, kRowThreads, sm, mode == 2 ? (long long)g.nx * g.nz : (rows + rt - 1) / rt, &grid));
  grid = std::min(grid, 148 * 8);
  if (np) *np = grid;
  note_launch();
  kern<<<grid, kRowThreads, sm, s>>>(a, rt);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

}  // namespace llr

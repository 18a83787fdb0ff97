// Fused locally-low-rank proximal step.
//
// One CTA owns one Casorati matrix at a time (persistent grid):
//   gather (periodic wrap, scale + phase on load)  -> shared memory C (m x n)
//   Gram G = C^H C on FP32 FMA                      -> shared memory
//   cyclic parallel Jacobi (round-robin pairs)      -> eigenpairs of G
//   singular-value map g(sigma) (hard rank / soft threshold)
//   W = V diag(g) V^H ;  C' = C W                   -> scatter (phase on store)
// This replaces, per block, lift_data_set (block.rs:147-164), cusolver gesvda
// (cusolver.rs:20-151), rhsCdgmmBatched (kernels.cu:11-67), the CGEMM (U S) V^H
// (low_rank.rs:55) and un_lift_data_set (block.rs:166-184): since U_r S_r V_r^H = C V_r V_r^H,
// every prox is C -> C W with W Hermitian n x n.
#include <cstdio>
#include <algorithm>

#include "llr_prox_common.cuh"

namespace llr {

namespace {

struct SmemLayout {
  int ldc;        // leading dimension of C in shared memory (odd)
  int np;         // padded n for Gram tiles
  int ksplit;     // Gram K-split factor
  size_t off_rot, off_pair, off_ev, off_g, off_act, off_A, off_V, off_scr, off_C, total;
};



template <int NPMAX, int TG>
SmemLayout make_layout(int m, int n) {
  SmemLayout L;
  L.ldc = (m & 1) ? m : m + 1;
  int nt = (n + TG - 1) / TG;
  L.np = nt * TG;
  int tiles = nt * nt;
  L.ksplit = std::max(1, kLlrThreads / tiles);
  size_t off = 256;  // misc
  L.off_rot = off; off = align16(off + sizeof(float4) * (NPMAX / 2));
  L.off_pair = off; off = align16(off + sizeof(int2) * (NPMAX / 2));
  L.off_ev = off; off = align16(off + sizeof(float) * NPMAX);
  L.off_g = off; off = align16(off + sizeof(float) * NPMAX);
  L.off_act = off; off = align16(off + sizeof(int) * NPMAX);
  L.off_A = off; off = align16(off + sizeof(float2) * NPMAX * (NPMAX + 1));
  L.off_V = off; off = align16(off + sizeof(float2) * NPMAX * (NPMAX + 1));
  L.off_scr = off;
  if (L.ksplit > 1) off = align16(off + sizeof(float2) * (size_t)L.ksplit * L.np * L.np);
  L.off_C = off; off = align16(off + sizeof(float2) * (size_t)n * L.ldc);
  L.total = off;
  return L;
}

template <int NPMAX, int TG>
__global__ void __launch_bounds__(kLlrThreads) llr_prox_jacobi_kernel(BlockSource src, ProxOp op, SmemLayout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  Misc* misc = reinterpret_cast<Misc*>(smem);
  float4* rot = reinterpret_cast<float4*>(smem + L.off_rot);
  int2* pairs = reinterpret_cast<int2*>(smem + L.off_pair);
  float* ev = reinterpret_cast<float*>(smem + L.off_ev);
  float* g = reinterpret_cast<float*>(smem + L.off_g);
  int* act = reinterpret_cast<int*>(smem + L.off_act);
  float2* A = reinterpret_cast<float2*>(smem + L.off_A);
  float2* V = reinterpret_cast<float2*>(smem + L.off_V);
  float2* scr = reinterpret_cast<float2*>(smem + L.off_scr);
  float2* Cs = reinterpret_cast<float2*>(smem + L.off_C);
  constexpr int lda = NPMAX + 1;
  const int m = op.m, n = op.n;

  if (threadIdx.x == 0) block_shift(src, misc->shift);
  __syncthreads();
  int sh[3] = {misc->shift[0], misc->shift[1], misc->shift[2]};
  const long long count = src.blk_list ? (long long)*src.blk_count : src.nblocks;

  for (long long i = blockIdx.x; i < count; i += gridDim.x) {
    const long long blk = src.blk_list ? (long long)src.blk_list[i] : i;
    gather_block(src, blk, sh, m, n, Cs, L.ldc);
    __syncthreads();
    gram<NPMAX, TG>(Cs, L.ldc, m, n, A, scr, L.ksplit);
    jacobi<NPMAX>(A, V, n, rot, pairs, misc, 16);
    if (op.block_stat) {
      if (threadIdx.x == 0) {
        float mx = 0.f;
        for (int k = 0; k < n; ++k) mx = fmaxf(mx, A[k * lda + k].x);
        op.block_stat[blk] = mx;
      }
      __syncthreads();
      continue;
    }
    singular_map(A, lda, n, op.mode, op.rank, op.lambda, ev, g, act, misc);
    if (op.blk_nuc && op.mode != LLR_PROX_HARD_RANK && threadIdx.x == 0)
      op.blk_nuc[blk] = nuclear_from_eigs(ev, n, op.lambda);
    const int na = misc->n_active;
    if (!(na == n && op.mode == LLR_PROX_HARD_RANK)) {
      form_W(A, V, lda, n, g, act, na);
      apply_W<NPMAX, TG>(Cs, L.ldc, m, n, A);
    }
    scatter_block(src, blk, sh, m, n, Cs, L.ldc);
    __syncthreads();
  }
}

template <int NPMAX, int TG>
int launch_jacobi_instance(const BlockSource& src, const ProxOp& op, cudaStream_t stream) {
  SmemLayout L = make_layout<NPMAX, TG>(op.m, op.n);
  if (L.total > 227 * 1024)
    return set_error(LLR_ERR_UNSUPPORTED, "Casorati %dx%d needs %zu B of shared memory (max 232448)", op.m, op.n,
                     L.total);
  auto kern = llr_prox_jacobi_kernel<NPMAX, TG>;
  LLR_CUDA_TRY(allow_smem(kern));
    LLR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  int dev = 0, nsm = 0, occ = 0;
  LLR_CUDA_TRY(cudaGetDevice(&dev));
  LLR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  LLR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kLlrThreads, L.total));
  if (occ < 1) return set_error(LLR_ERR_UNSUPPORTED, "prox kernel cannot be resident (smem %zu B)", L.total);
  long long grid = std::min<long long>(src.nblocks, (long long)nsm * occ);
  if (grid < 1) return LLR_OK;
  note_launch();
  kern<<<(unsigned)grid, kLlrThreads, L.total, stream>>>(src, op, L);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

}  // namespace

bool llr_prox_jacobi_supported(int m, int n) {
  if (m < 1 || n < 1 || n > 64) return false;
  size_t t;
  if (n <= 16) t = make_layout<16, 2>(m, n).total;
  else if (n <= 32) t = make_layout<32, 2>(m, n).total;
  else t = make_layout<64, 4>(m, n).total;
  return t <= 227 * 1024;
}

// Jacobi-path prox over all blocks of `src` (or over src.blk_list when set).
int launch_llr_prox_jacobi(const BlockSource& src, const ProxOp& op, cudaStream_t stream) {
  if (op.n < 1 || op.m < 1) return set_error(LLR_ERR_INVALID, "empty Casorati matrix %dx%d", op.m, op.n);
  if (src.nblocks == 0) return LLR_OK;
  if (op.n <= 16) return launch_jacobi_instance<16, 2>(src, op, stream);
  if (op.n <= 32) return launch_jacobi_instance<32, 2>(src, op, stream);
  if (op.n <= 64) return launch_jacobi_instance<64, 4>(src, op, stream);
  return set_error(LLR_ERR_UNSUPPORTED, "Casorati column count %d > 64 is not supported", op.n);
}



// =======================================================================================
// Subspace-constrained prox: X <- LR(X S) S^H per block (lib.rs:281-289).  The projected
// matrix Z = X S (m x srank) is formed while gathering (each voxel's nq-vector times S),
// so the full m x nq Casorati never needs to be staged; Z' = Z W (srank x srank Jacobi);
// the store streams X' = Z' S^H back volume by volume.
// =======================================================================================
namespace {

constexpr int kSubMax = 16;   // max subspace rank

template <int NPMAX, int KM>
__global__ void __launch_bounds__(kLlrThreads) llr_subspace_kernel(BlockSource src, SubspaceOp op, SmemLayout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  Misc* misc = reinterpret_cast<Misc*>(smem);
  float4* rot = reinterpret_cast<float4*>(smem + L.off_rot);
  int2* pairs = reinterpret_cast<int2*>(smem + L.off_pair);
  float* ev = reinterpret_cast<float*>(smem + L.off_ev);
  float* g = reinterpret_cast<float*>(smem + L.off_g);
  int* act = reinterpret_cast<int*>(smem + L.off_act);
  float2* A = reinterpret_cast<float2*>(smem + L.off_A);
  float2* V = reinterpret_cast<float2*>(smem + L.off_V);
  float2* scr = reinterpret_cast<float2*>(smem + L.off_scr);
  float2* Z = reinterpret_cast<float2*>(smem + L.off_C);           // srank x ldc
  float2* Ss = Z + (size_t)op.srank * L.ldc;                        // nq x srank
  constexpr int lda = NPMAX + 1;
  const int m = op.m, nq = op.nq, sr = op.srank;
  // S is nq x srank column-major; keep it row-major (q, k) in shared memory.
  for (int i = threadIdx.x; i < nq * sr; i += blockDim.x) {
    const int q = i / sr, k = i - q * sr;
    Ss[i] = op.S[q + (long long)nq * k];
  }
  if (threadIdx.x == 0) block_shift(src, misc->shift);
  __syncthreads();
  int sh[3] = {misc->shift[0], misc->shift[1], misc->shift[2]};

  for (long long blk = blockIdx.x; blk < src.nblocks; blk += gridDim.x) {
    // Z[r, k] = sum_q X[r, q] S[q, k]
    for (int r = threadIdx.x; r < m; r += blockDim.x) {
      float2 z[KM];
#pragma unroll
      for (int k = 0; k < KM; ++k) z[k] = make_float2(0.f, 0.f);
      int ix = 0, iy = 0, iz = 0;
      if (src.kind == 1) block_row_coord(src, blk, sh, r, ix, iy, iz);
      for (int q = 0; q < nq; ++q) {
        float2 v;
        if (src.kind == 0) {
          v = src.data[blk * (long long)m * nq + (long long)q * m + r];
        } else {
          v = src.data[planar_index(src.g, ix, iy, iz, q)];
          v = cscale(cmul_bc(v, phase_at(src.ph, src.g, q, ix, iy, iz)), src.load_scale);
        }
#pragma unroll
        for (int k = 0; k < KM; ++k)
          if (k < sr) cfma(z[k], v, Ss[q * sr + k]);
      }
#pragma unroll
      for (int k = 0; k < KM; ++k)
        if (k < sr) Z[k * L.ldc + r] = z[k];
    }
    __syncthreads();
    gram<NPMAX, 2>(Z, L.ldc, m, sr, A, scr, L.ksplit);
    if (threadIdx.x < 32) jacobi_warp<NPMAX>(A, V, sr, rot, pairs, misc, 16);
    __syncthreads();
    singular_map(A, lda, sr, op.mode, op.rank, op.lambda, ev, g, act, misc);
    form_W(A, V, lda, sr, g, act, misc->n_active);
    apply_W<NPMAX, 2>(Z, L.ldc, m, sr, A);
    // X'[r, q] = sum_k Z'[r, k] conj(S[q, k])
    for (int r = threadIdx.x; r < m; r += blockDim.x) {
      float2 z[KM];
#pragma unroll
      for (int k = 0; k < KM; ++k) z[k] = (k < sr) ? Z[k * L.ldc + r] : make_float2(0.f, 0.f);
      int ix = 0, iy = 0, iz = 0;
      if (src.kind == 1) block_row_coord(src, blk, sh, r, ix, iy, iz);
      for (int q = 0; q < nq; ++q) {
        float2 v = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < KM; ++k)
          if (k < sr) cfma_cb(v, z[k], Ss[q * sr + k]);
        if (src.kind == 0) {
          src.data[blk * (long long)m * nq + (long long)q * m + r] = v;
        } else {
          v = cscale(v, src.store_scale);
          if (src.store_phase) v = cmul(v, phase_at(src.ph, src.g, q, ix, iy, iz));
          src.data[planar_index(src.g, ix, iy, iz, q)] = v;
        }
      }
    }
    __syncthreads();
  }
}

// Coefficient path (wavelet shrink in the coefficient domain), two kernels.
//
// The first forms Z = X S for every voxel, as srank planar coefficient volumes in image space: a stream over
// the iterate that needs no block structure.  Bound: HBM, 8 nq + 8 srank bytes per voxel (4.6 GB at
// 128 x 256 x 256 x 61, rank 7: 0.70 ms at the measured copy rate).  Four volumes of two voxels are in flight
// per thread, a row of S (shared memory, broadcast) serves both voxels, and a phase shared by every
// volume is taken out of the sum.  The second kernel makes the blocks low rank in place on those volumes
// (7 / 61 of the data).  One kernel doing both per block waited on its 7 x 7 eigenproblem with the
// gather's loads idle: 3.52 ms, now 0.89 ms + 0.58 ms.
template <int KM, bool UNI>   // UNI: every volume has the same phase
__global__ void __launch_bounds__(256, KM <= 8 && UNI ? 3 : KM <= 8 ? 2 : 1) subspace_project_kernel(const float2* __restrict__ x, float2* __restrict__ z,
                                                               const float2* __restrict__ S, int srank, Geom g,
                                                               PhaseTab ph, float scale) {
  constexpr int QB = 4;
  extern __shared__ __align__(16) float4 Sq[];   // [nq][KM] (S, i S), zero beyond srank
  for (int i = threadIdx.x; i < g.nq * KM; i += 256) {
    const int q = i / KM, k = i - q * KM;
    const float2 c = k < srank ? S[q + (long long)g.nq * k] : make_float2(0.f, 0.f);
    Sq[i] = make_float4(c.x, c.y, -c.y, c.x);
  }
  __syncthreads();
  for (long long v0 = blockIdx.x * 512LL + threadIdx.x; v0 < g.V; v0 += gridDim.x * 512LL) {
    const bool two = v0 + 256 < g.V;              // a missing second voxel repeats the first
    const long long v[2] = {v0, two ? v0 + 256 : v0};
    int ix[2], iy[2], iz[2];
    float2 acc[2][KM];
    auto coords = [&](int h) {
      const long long r = v[h] / g.ny;
      iy[h] = (int)(v[h] - r * g.ny);
      ix[h] = (int)(r / g.nz);
      iz[h] = (int)(r - (long long)ix[h] * g.nz);
    };
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!UNI) coords(h);
#pragma unroll
      for (int k = 0; k < KM; ++k) acc[h][k] = make_float2(0.f, 0.f);
    }
    auto add = [&](int q, float2 xv, int h) {
      if (!UNI) xv = cscale(cmul_bc(xv, phase_at(ph, g, q, ix[h], iy[h], iz[h])), scale);
#pragma unroll
      for (int k = 0; k < KM; ++k) {
        const float4 c = Sq[q * KM + k];
        cfma2(acc[h][k], xv, make_float2(c.x, c.y), make_float2(c.z, c.w));
      }
    };
    const float2* xa = x + v[0];
    const float2* xb = x + v[1];
    int q = 0;
    for (; q + QB <= g.nq; q += QB) {
      float2 a[QB], b[QB];
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        a[u] = __ldcs(xa);
        b[u] = __ldcs(xb);
        xa += g.V;
        xb += g.V;
      }
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        add(q + u, a[u], 0);
        add(q + u, b[u], 1);
      }
    }
    for (; q < g.nq; ++q) {
      add(q, __ldcs(xa), 0);
      add(q, __ldcs(xb), 1);
      xa += g.V;
      xb += g.V;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 1 && !two) break;
      float2 p0 = make_float2(1.f, 0.f);
      if (UNI) {
        coords(h);
        p0 = cscale(phase_at(ph, g, 0, ix[h], iy[h], iz[h]), scale);
      }
#pragma unroll
      for (int k = 0; k < KM; ++k)
        if (k < srank) z[v[h] + g.V * k] = UNI ? cmul_bc(acc[h][k], p0) : acc[h][k];
    }
  }
}

// Low rank of every block of the coefficient volumes, in place, rank at most 8: one warp per block.  Bound:
// latency (the eigenproblem is a chain of rotations); a warp's chain of gather, Gram sums in
// registers, rotations and apply needs no CTA barrier, and 24 of them run per SM.  The second read of
// the block comes from L2.  One CTA per block, 256 threads waiting on one warp's rotations, took 2.47 ms
// at 128 x 256 x 256 in 8^3 blocks of rank 7, now 0.58 ms.
constexpr int kCoefK = 8, kCoefWarps = 4;

struct CoefWarp {
  float2 A[kCoefK * (kCoefK + 1)], V[kCoefK * (kCoefK + 1)];
  float4 W[kCoefK * kCoefK];   // (W, i W)
  float4 rot[kCoefK / 2];
  int2 pairs[kCoefK / 2];
  float ev[kCoefK], g[kCoefK];
  Misc misc;
};

__global__ void __launch_bounds__(32 * kCoefWarps, 5) llr_coef_warp_kernel(BlockSource src, SubspaceOp op) {
  constexpr int K = kCoefK, lda = K + 1;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, m = op.m, sr = op.srank;
  CoefWarp* C = reinterpret_cast<CoefWarp*>(smem) + (threadIdx.x >> 5);
  unsigned short* rowt = reinterpret_cast<unsigned short*>(smem + sizeof(CoefWarp) * kCoefWarps);   // [m][4]: rx ry rz
  for (int r = threadIdx.x; r < m; r += blockDim.x) {
    rowt[4 * r] = (unsigned short)(r / (src.by * src.bz));
    rowt[4 * r + 1] = (unsigned short)(r % src.by);
    rowt[4 * r + 2] = (unsigned short)((r / src.by) % src.bz);
  }
  __syncthreads();
  int sh[3];
  block_shift(src, sh);
  const Geom& g = src.g;
  const long long nwarps = (long long)gridDim.x * kCoefWarps;
  for (long long blk = blockIdx.x * (long long)kCoefWarps + (threadIdx.x >> 5); blk < src.nblocks; blk += nwarps) {
    const int gyi = (int)(blk % src.gy);
    const long long t = blk / src.gy;
    const int gzi = (int)(t % src.gz), gxi = (int)(t / src.gz);
    const int cx = (gxi * src.bx + sh[0]) % g.nx, cy = (gyi * src.by + sh[1]) % g.ny, cz = (gzi * src.bz + sh[2]) % g.nz;
    auto row = [&](int r) {
      const ushort4 q = *reinterpret_cast<const ushort4*>(rowt + 4 * r);
      int ix = cx + q.x, iy = cy + q.y, iz = cz + q.z;
      if (ix >= g.nx) ix -= g.nx;
      if (iy >= g.ny) iy -= g.ny;
      if (iz >= g.nz) iz -= g.nz;
      return op.coef_out + planar_index(g, ix, iy, iz, 0);
    };
    // Gram sums: the diagonal (real), then the pairs i > j
    float s[K * K];
#pragma unroll
    for (int e = 0; e < K * K; ++e) s[e] = 0.f;
#pragma unroll 2
    for (int r = lane; r < m; r += 32) {
      const float2* c = row(r);
      float2 z[K];
#pragma unroll
      for (int k = 0; k < K; ++k) z[k] = k < sr ? c[g.V * k] : make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < K; ++i) {
        s[i] = fmaf(z[i].x, z[i].x, fmaf(z[i].y, z[i].y, s[i]));
#pragma unroll
        for (int j = 0; j < i; ++j) {   // conj(z_i) z_j
          float2 a = make_float2(s[K + i * (i - 1) + 2 * j], s[K + i * (i - 1) + 2 * j + 1]);
          cfma_ca(a, z[i], z[j]);
          s[K + i * (i - 1) + 2 * j] = a.x;
          s[K + i * (i - 1) + 2 * j + 1] = a.y;
        }
      }
    }
    // recursive halving over the warp: lane l ends with the sums of elements 2 l and 2 l + 1
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < 2 * o; ++i) {
        const float send = up ? s[i] : s[i + 2 * o], keep = up ? s[i + 2 * o] : s[i];
        s[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    if (lane < K / 2) {
      C->A[(2 * lane) * lda + 2 * lane] = make_float2(s[0], 0.f);
      C->A[(2 * lane + 1) * lda + 2 * lane + 1] = make_float2(s[1], 0.f);
    } else {
      const int p = lane - K / 2;       // pair index i (i - 1) / 2 + j
      int i = 1;
      while (i * (i + 1) / 2 <= p) ++i;
      const int j = p - i * (i - 1) / 2;
      C->A[i * lda + j] = make_float2(s[0], s[1]);
      C->A[j * lda + i] = make_float2(s[0], -s[1]);
    }
    __syncwarp();
    jacobi_warp<K>(C->A, C->V, sr, C->rot, C->pairs, &C->misc, 16);
    __syncwarp();
    if (lane < sr) C->ev[lane] = C->A[lane * lda + lane].x;
    __syncwarp();
    if (lane < sr) {
      const float e = C->ev[lane];
      float gv;
      if (op.mode == LLR_PROX_HARD_RANK) {
        int pos = 0;
        for (int j = 0; j < sr; ++j) pos += (C->ev[j] > e) || (C->ev[j] == e && j < lane);
        gv = pos < op.rank ? 1.f : 0.f;
      } else {
        const float sv = sqrtf(fmaxf(e, 0.f));
        gv = sv > op.lambda ? 1.f - op.lambda / sv : 0.f;
      }
      C->g[lane] = gv;
    }
    __syncwarp();
    for (int e = lane; e < K * K; e += 32) {   // W = V diag(g) V^H
      const int i = e / K, j = e - i * K;
      float2 w = make_float2(0.f, 0.f);
      if (i < sr && j < sr)
        for (int k = 0; k < sr; ++k) {
          const float2 p = cmul_bc(C->V[i * lda + k], C->V[j * lda + k]);
          w.x = fmaf(C->g[k], p.x, w.x);
          w.y = fmaf(C->g[k], p.y, w.y);
        }
      C->W[e] = make_float4(w.x, w.y, -w.y, w.x);
    }
    __syncwarp();
#pragma unroll 2
    for (int r = lane; r < m; r += 32) {   // z <- z W
      float2* c = const_cast<float2*>(row(r));
      float2 z[K];
#pragma unroll
      for (int k = 0; k < K; ++k) z[k] = k < sr ? c[g.V * k] : make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < K; ++j) {
        if (j < sr) {
          float2 a = make_float2(0.f, 0.f);
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const float4 w = C->W[k * K + j];
            cfma2(a, z[k], make_float2(w.x, w.y), make_float2(w.z, w.w));
          }
          c[g.V * j] = a;
        }
      }
    }
    __syncwarp();
  }
}

int launch_coef_warp(const BlockSource& src, const SubspaceOp& op, cudaStream_t stream) {
  const size_t sm = sizeof(CoefWarp) * kCoefWarps + sizeof(unsigned short) * 4 * (size_t)op.m;
  LLR_CUDA_TRY(allow_smem(llr_coef_warp_kernel));
  int occ = 0;
  LLR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, llr_coef_warp_kernel, 32 * kCoefWarps, sm));
  if (occ < 1) return set_error(LLR_ERR_UNSUPPORTED, "coefficient kernel cannot be resident (smem %zu B)", sm);
  const long long want = (src.nblocks + kCoefWarps - 1) / kCoefWarps;
  note_launch();
  llr_coef_warp_kernel<<<(unsigned)std::min<long long>(want, 148LL * occ), 32 * kCoefWarps, sm, stream>>>(src, op);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

// The same for ranks 9 to 16, whose Gram sums do not fit a lane's registers: one CTA per block, the small
// eigenproblem by one warp.
template <int NPMAX>
__global__ void __launch_bounds__(kLlrThreads) llr_coef_low_rank_kernel(BlockSource src, SubspaceOp op, SmemLayout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  Misc* misc = reinterpret_cast<Misc*>(smem);
  float4* rot = reinterpret_cast<float4*>(smem + L.off_rot);
  int2* pairs = reinterpret_cast<int2*>(smem + L.off_pair);
  float* ev = reinterpret_cast<float*>(smem + L.off_ev);
  float* g = reinterpret_cast<float*>(smem + L.off_g);
  int* act = reinterpret_cast<int*>(smem + L.off_act);
  float2* A = reinterpret_cast<float2*>(smem + L.off_A);
  float2* V = reinterpret_cast<float2*>(smem + L.off_V);
  float2* scr = reinterpret_cast<float2*>(smem + L.off_scr);
  float2* Z = reinterpret_cast<float2*>(smem + L.off_C);
  const int m = op.m, sr = op.srank;
  if (threadIdx.x == 0) block_shift(src, misc->shift);
  __syncthreads();
  int sh[3] = {misc->shift[0], misc->shift[1], misc->shift[2]};
  for (long long blk = blockIdx.x; blk < src.nblocks; blk += gridDim.x) {
    for (int r = threadIdx.x; r < m; r += blockDim.x) {
      int ix = 0, iy = 0, iz = 0;
      block_row_coord(src, blk, sh, r, ix, iy, iz);
      const float2* c = op.coef_out + planar_index(src.g, ix, iy, iz, 0);
#pragma unroll 8
      for (int k = 0; k < sr; ++k) Z[k * L.ldc + r] = c[src.g.V * k];
    }
    __syncthreads();
    gram<NPMAX, 2>(Z, L.ldc, m, sr, A, scr, L.ksplit);
    if (threadIdx.x < 32) jacobi_warp<NPMAX>(A, V, sr, rot, pairs, misc, 16);
    __syncthreads();
    singular_map(A, NPMAX + 1, sr, op.mode, op.rank, op.lambda, ev, g, act, misc);
    form_W(A, V, NPMAX + 1, sr, g, act, misc->n_active);
    apply_W<NPMAX, 2>(Z, L.ldc, m, sr, A);
    for (int r = threadIdx.x; r < m; r += blockDim.x) {
      int ix = 0, iy = 0, iz = 0;
      block_row_coord(src, blk, sh, r, ix, iy, iz);
      float2* c = op.coef_out + planar_index(src.g, ix, iy, iz, 0);
      for (int k = 0; k < sr; ++k) c[src.g.V * k] = Z[k * L.ldc + r];
    }
    __syncthreads();
  }
}

template <int KM>
int launch_subspace_project(const BlockSource& src, const SubspaceOp& op, cudaStream_t stream) {
  const size_t sm = sizeof(float4) * (size_t)op.nq * KM;
  auto kern = src.ph_uniform ? subspace_project_kernel<KM, true> : subspace_project_kernel<KM, false>;
  if (sm > 48 * 1024) LLR_CUDA_TRY(allow_smem(kern));
  int occ = 0;
  LLR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 256, sm));
  if (occ < 1) return set_error(LLR_ERR_UNSUPPORTED, "subspace projection needs %zu B smem", sm);
  const long long blocks = std::min<long long>((src.g.V + 511) / 512, 148LL * occ * 4);
  note_launch();
  kern<<<(unsigned)blocks, 256, sm, stream>>>(src.data, op.coef_out, op.S, op.srank, src.g, src.ph, src.load_scale);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

template <int KM>
__global__ void __launch_bounds__(256) subspace_expand_kernel(const float2* __restrict__ coef, float2* __restrict__ x,
                                                              const float2* __restrict__ S, int srank, Geom g,
                                                              PhaseTab ph, int store_phase, int ph_uniform,
                                                              float scale) {
  __shared__ float2 Ss[64 * kSubMax];
  for (int i = threadIdx.x; i < g.nq * srank; i += blockDim.x) Ss[i] = S[i];   // column-major (q, k)
  __syncthreads();
  for (long long v = blockIdx.x * 256LL + threadIdx.x; v < g.V; v += (long long)gridDim.x * 256) {
    float2 c[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) c[k] = k < srank ? coef[v + g.V * k] : make_float2(0.f, 0.f);
    const int iy = (int)(v % g.ny);
    const long long r = v / g.ny;
    const int iz = (int)(r % g.nz), ix = (int)(r / g.nz);
    // the stored value's factor: scale times the phase (computed once when every volume shares it)
    const float2 f0 = cscale(store_phase ? phase_at(ph, g, 0, ix, iy, iz) : make_float2(1.f, 0.f), scale);
#pragma unroll 4
    for (int q = 0; q < g.nq; ++q) {
      float2 a = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < KM; ++k)
        if (k < srank) cfma_cb(a, c[k], Ss[q + g.nq * k]);
      const float2 f = (ph_uniform || !store_phase) ? f0 : cscale(phase_at(ph, g, q, ix, iy, iz), scale);
      x[v + g.V * q] = cmul(a, f);
    }
  }
}

}  // namespace

int launch_llr_prox_subspace(const BlockSource& src, const SubspaceOp& op, cudaStream_t stream) {
  if (op.srank < 1 || op.srank > kSubMax)
    return set_error(LLR_ERR_UNSUPPORTED, "subspace rank %d outside [1, %d]", op.srank, kSubMax);
  if (src.nblocks == 0) return LLR_OK;
  SmemLayout L = make_layout<16, 2>(op.m, op.srank);
  L.total = align16(L.total + sizeof(float2) * (size_t)op.nq * op.srank);
  if (L.total > 227 * 1024) return set_error(LLR_ERR_UNSUPPORTED, "subspace prox needs %zu B smem", L.total);
  if (op.coef_out && src.kind != 1) return set_error(LLR_ERR_INVALID, "coefficient output needs volume blocks");
  if (op.coef_out) {   // accumulators sized to the rank (two voxels per thread)
    if (op.srank <= 4) LLR_TRY(launch_subspace_project<4>(src, op, stream));
    else if (op.srank <= 6) LLR_TRY(launch_subspace_project<6>(src, op, stream));
    else if (op.srank == 7) LLR_TRY(launch_subspace_project<7>(src, op, stream));
    else if (op.srank == 8) LLR_TRY(launch_subspace_project<8>(src, op, stream));
    else if (op.srank <= 12) LLR_TRY(launch_subspace_project<12>(src, op, stream));
    else LLR_TRY(launch_subspace_project<16>(src, op, stream));
    // a row table of more than 8000 rows would leave the warps of the rank-8 kernel too few
    if (op.srank <= kCoefK && op.m <= 8000) return launch_coef_warp(src, op, stream);
  }
  // per-thread coefficient registers sized to the rank class (fewer registers, more CTAs per SM)
  auto kern = op.coef_out ? llr_coef_low_rank_kernel<16>
                          : (op.srank <= 8 ? llr_subspace_kernel<16, 8> : llr_subspace_kernel<16, 16>);
  LLR_CUDA_TRY(allow_smem(kern));
    LLR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  int dev = 0, nsm = 0, occ = 0;
  LLR_CUDA_TRY(cudaGetDevice(&dev));
  LLR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  LLR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kLlrThreads, L.total));
  if (occ < 1) return set_error(LLR_ERR_UNSUPPORTED, "subspace kernel cannot be resident");
  long long grid = std::min<long long>(src.nblocks, (long long)nsm * occ);
  note_launch();
  kern<<<(unsigned)grid, kLlrThreads, L.total, stream>>>(src, op, L);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

// =======================================================================================
// Reference-layout lift / un-lift (block.rs:147-184): row r of block i in block
// col-major order (x fastest), volume q is column q.
// =======================================================================================
namespace {

// Bound: HBM, one read and one write of every element.  A CTA takes up to kLiftRows consecutive rows of the matrices, of one
// block or of many, and a slice of the volumes: the rows' voxel and matrix offsets are computed once into shared
// memory (all the index divisions there are), then the elements go by volume after volume, eight in flight per thread.
// With three 64-bit divisions per element the kernel was issue-bound: 315 us for 4096 blocks of 216 x 61 on
// 96 x 96 x 48 x 61 (0.43 GB moved), about 100 us this way (lift, rank truncation and un-lift 1617 -> 1213 us).
// A CTA per block in place of one per row chunk took, both ways, 1.80 ms for 2^3 blocks of one 128^3 volume and 23.9 ms for a
// single 256 x 256 x 64 block of three: 53 and 119 us this way.  One address per element is kept for the second half of a
// batch, so four CTAs fit an SM (both addresses took 80 registers, three CTAs); over 36 shapes of blocks of one to 32^3
// voxels and 1 to 61 volumes nothing is slower than with a CTA per block, 4^3 to 8^3 blocks 1.0 to 1.7 times as fast.
constexpr int kLiftRows = 1024;   // most rows per chunk (16 KB of offsets)

// QFAST: volumes run fastest over a slice's elements, else rows.  U: unsigned where every row and block index fits.
template <int DIR, bool QFAST, class U>
__global__ void __launch_bounds__(256, 4) lift_kernel(float2* __restrict__ vol, float2* __restrict__ mat, int nx, int ny,
                                                   int nz, int nq, int bx, int by, int bz, int gx, int gy, int sx,
                                                   int sy, int sz, long long start, long long n, int qper, int rc) {
  __shared__ long long off[kLiftRows], moff[kLiftRows];
  constexpr int LB = 8;
  const U m = (U)bx * by * bz;
  const long long V = (long long)nx * ny * nz, total = (long long)m * n;
  const int q0 = blockIdx.y * qper, q1 = min(nq, q0 + qper);
  for (long long r0 = (long long)blockIdx.x * rc; r0 < total; r0 += (long long)gridDim.x * rc) {
    const int rows = (int)min((long long)rc, total - r0);
    __syncthreads();
    for (int i = threadIdx.x; i < rows; i += 256) {
      const U g = (U)(r0 + i), c = g / m, r = g - c * m;
      const U blk = (U)start + c, t = blk / (U)gx, t2 = r / (U)bx;
      const int gxi = (int)(blk - t * gx), gzi = (int)(t / (U)gy), gyi = (int)(t - (U)gzi * gy);
      const int rx = (int)(r - t2 * bx), rz = (int)(t2 / (U)by), ry = (int)(t2 - (U)rz * by);
      const int ix = (gxi * bx + sx + rx) % nx, iy = (gyi * by + sy + ry) % ny, iz = (gzi * bz + sz + rz) % nz;
      off[i] = (long long)ix + (long long)nx * ((long long)iy + (long long)ny * iz);
      moff[i] = (long long)c * m * nq + r;
    }
    __syncthreads();
    // the slice's elements, stepped without divisions
    const int nf = QFAST ? q1 - q0 : rows, ns = QFAST ? rows : q1 - q0;
    const int ds = 256 / nf, df = 256 - ds * nf;
    int f = (int)threadIdx.x % nf, sl = (int)threadIdx.x / nf;
    while (sl < ns) {
      float2 v[LB];
      long long to[LB];
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        to[u] = -1;
        if (sl < ns) {
          const int r = QFAST ? sl : f, q = q0 + (QFAST ? f : sl);
          const long long va = off[r] + V * q, ma = moff[r] + (long long)m * q;
          v[u] = DIR == 0 ? vol[va] : mat[ma];
          to[u] = DIR == 0 ? ma : va;
        }
        f += df;
        sl += ds;
        if (f >= nf) { f -= nf; ++sl; }
      }
#pragma unroll
      for (int u = 0; u < LB; ++u)
        if (to[u] >= 0) (DIR == 0 ? mat : vol)[to[u]] = v[u];
    }
  }
}

}  // namespace

int launch_lift(const float2* vol, float2* mat, const int* vs, int nq, const int* bs, const int* sh, long long start,
                long long n, int dir, cudaStream_t s) {
  int g[3];
  for (int a = 0; a < 3; ++a) g[a] = vs[a] / bs[a];
  const long long tot = (long long)bs[0] * bs[1] * bs[2] * nq * n;
  if (tot == 0) return LLR_OK;
  if (tot < 0) return set_error(LLR_ERR_INVALID, "negative block count");
  // Rows per chunk: 512, with few volumes 1024, so that a thread has loads in flight; shorter chunks where the split of the
  // volumes below would leave a chunk's offsets fewer than eight volumes to serve (55 x 119 x 17 x 25 in 5 x 6 x 8 blocks, both
  // ways: 53 us with 512 rows and two volumes, 33 with 128 and seven).  The volumes are split for eight CTAs per SM where the
  // chunks alone do not give them: one wave; for sixteen above 64 MB, where a second wave evens out the end (96 x 96 x 48 x 61
  // in 6^3 blocks 229 us, 238 with eight; 48 x 48 x 24 x 20 in 8^3 blocks 25 us, 33 with sixteen).
  const long long rows = (long long)bs[0] * bs[1] * bs[2] * n;
  const long long ctas = 148 * (rows * nq > 8000000 ? 16 : 8);
  int rc = nq < 4 ? kLiftRows : 512, qper;
  long long chunks;
  for (;; rc /= 2) {
    chunks = (rows + rc - 1) / rc;
    const long long want = chunks < ctas ? std::min<long long>(nq, (ctas + chunks - 1) / chunks) : 1;
    qper = (int)((nq + want - 1) / want);
    if (rc <= 128 || qper >= std::min(nq, 8)) break;
  }
  dim3 grid((unsigned)std::min<long long>(chunks, 1ll << 30), (unsigned)((nq + qper - 1) / qper));
  const bool narrow = rows < (1ll << 31) && start >= 0 && start + n < (1ll << 31);
  // where a matrix has only one to three rows, a column's stores are single elements: 96^3 x 61 in 1^3 blocks took
  // 846 us with rows fastest, 309 with volumes fastest
  const bool qfast = (long long)bs[0] * bs[1] * bs[2] < 4;
  using u64 = unsigned long long;
  auto kern = dir == 1 ? (narrow ? lift_kernel<1, false, unsigned> : lift_kernel<1, false, u64>)
              : qfast  ? (narrow ? lift_kernel<0, true, unsigned> : lift_kernel<0, true, u64>)
                       : (narrow ? lift_kernel<0, false, unsigned> : lift_kernel<0, false, u64>);
  note_launch();
  kern<<<grid, 256, 0, s>>>(const_cast<float2*>(vol), mat, vs[0], vs[1], vs[2], nq, bs[0], bs[1], bs[2], g[0], g[1], sh[0],
                            sh[1], sh[2], start, n, qper, rc);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

// =======================================================================================
// rhsCdgmmBatched (kernels.cu:11-67) and a batched complex GEMM with the semantics of
// cublas_cgemm_strided_batched_device (cublas.rs:12-105).
int launch_subspace_expand(const float2* coef, float2* x, const float2* S, int srank, const Geom& g, PhaseTab ph,
                           int store_phase, int ph_uniform, float scale, cudaStream_t s) {
  if (srank < 1 || srank > kSubMax || g.nq > 64) return set_error(LLR_ERR_UNSUPPORTED, "subspace expand shape");
  const long long blocks = std::min<long long>((g.V + 255) / 256, 148LL * 16);
  note_launch();
  if (srank <= 8)
    subspace_expand_kernel<8><<<(unsigned)blocks, 256, 0, s>>>(coef, x, S, srank, g, ph, store_phase, ph_uniform, scale);
  else
    subspace_expand_kernel<16><<<(unsigned)blocks, 256, 0, s>>>(coef, x, S, srank, g, ph, store_phase, ph_uniform,
                                                                scale);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

// =======================================================================================
namespace {

__global__ void rhs_cdgmm_kernel(int m, int n, int batch, float2* a, const float* d) {
  const long long tot = (long long)m * n * batch;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
    const long long col = i / m;  // j + n * b
    a[i] = cscale(a[i], d[col]);
  }
}

// C[i, j] = alpha * sum_l op(A)[i, l] op(B)[l, j] + beta * C[i, j], 16x16 output tiles.
__global__ void cgemm_kernel(int m, int k, int n, int broadcast_a, float2 alpha, float2 beta, int ta, int tb,
                             const float2* __restrict__ A, const float2* __restrict__ B, float2* __restrict__ C) {
  __shared__ float2 As[16][17];
  __shared__ float2 Bs[16][17];
  const int b = blockIdx.z;
  const float2* Ab = A + (broadcast_a ? 0 : (long long)b * m * k);
  const float2* Bb = B + (long long)b * k * n;
  float2* Cb = C + (long long)b * m * n;
  const int i = blockIdx.x * 16 + threadIdx.x;
  const int j = blockIdx.y * 16 + threadIdx.y;
  float2 acc = make_float2(0.f, 0.f);
  for (int l0 = 0; l0 < k; l0 += 16) {
    {  // A tile: rows blockIdx.x*16 + tx, cols l0 + ty
      const int ii = blockIdx.x * 16 + threadIdx.x, ll = l0 + threadIdx.y;
      float2 v = make_float2(0.f, 0.f);
      if (ii < m && ll < k) v = ta ? cconj(Ab[ll + (long long)k * ii]) : Ab[ii + (long long)m * ll];
      As[threadIdx.x][threadIdx.y] = v;
    }
    {  // B tile: rows l0 + tx, cols blockIdx.y*16 + ty
      const int ll = l0 + threadIdx.x, jj = blockIdx.y * 16 + threadIdx.y;
      float2 v = make_float2(0.f, 0.f);
      if (ll < k && jj < n) v = tb ? cconj(Bb[jj + (long long)n * ll]) : Bb[ll + (long long)k * jj];
      Bs[threadIdx.x][threadIdx.y] = v;
    }
    __syncthreads();
#pragma unroll
    for (int l = 0; l < 16; ++l) cfma(acc, As[threadIdx.x][l], Bs[l][threadIdx.y]);
    __syncthreads();
  }
  if (i < m && j < n) {
    float2 c = Cb[i + (long long)m * j];
    float2 out = cmul(alpha, acc);
    if (beta.x != 0.f || beta.y != 0.f) out = cadd(out, cmul(beta, c));
    Cb[i + (long long)m * j] = out;
  }
}

}  // namespace

namespace {
// out (n x m per batch) = conj(in (m x n per batch))^T, column-major (dti_subspace.rs:211-221).
__global__ void conj_transpose_kernel(const float2* __restrict__ in, float2* __restrict__ out, int m, int n) {
  __shared__ float2 tile[32][33];
  const long long off = (long long)blockIdx.z * m * n;
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int i = i0 + threadIdx.x, j = j0 + k;
    if (i < m && j < n) tile[k][threadIdx.x] = in[off + i + (long long)m * j];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int j = j0 + threadIdx.x, i = i0 + k;
    if (i < m && j < n) out[off + j + (long long)n * i] = cconj(tile[threadIdx.x][k]);
  }
}
}  // namespace

int launch_conj_transpose(const float2* in, float2* out, int m, int n, int batch, cudaStream_t s) {
  if ((long long)m * n * batch == 0) return LLR_OK;
  dim3 grid((m + 31) / 32, (n + 31) / 32, batch);
  note_launch();
  conj_transpose_kernel<<<grid, dim3(32, 8), 0, s>>>(in, out, m, n);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

int launch_rhs_cdgmm(int m, int n, int batch, float2* a, const float* d, cudaStream_t s) {
  const long long tot = (long long)m * n * batch;
  if (tot == 0) return LLR_OK;
  long long blocks = std::min<long long>((tot + 255) / 256, 148LL * 32);
  note_launch();
  rhs_cdgmm_kernel<<<(unsigned)blocks, 256, 0, s>>>(m, n, batch, a, d);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

int launch_cgemm(int m, int k, int n, int batch, int broadcast_a, float2 alpha, float2 beta, int ta, int tb,
                 const float2* A, const float2* B, float2* C, cudaStream_t s) {
  if (m == 0 || n == 0 || batch == 0) return LLR_OK;
  dim3 grid((m + 15) / 16, (n + 15) / 16, batch);
  dim3 block(16, 16);
  note_launch();
  cgemm_kernel<<<grid, block, 0, s>>>(m, k, n, broadcast_a, alpha, beta, ta, tb, A, B, C);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

}  // namespace llr

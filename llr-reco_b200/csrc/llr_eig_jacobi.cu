// Eigen stage of the split LLR prox path for 64 < n <= 128 columns: one CTA per Casorati block.
//
// The decisions and the rotations of the wide Jacobi kernel (llr_prox_trd.cu): ||G||_F or the trace bound of
// Wolkowicz and Styan (1980) proves a block zero; otherwise cyclic parallel Jacobi in round-robin order.  The packed
// Gram matrix (tensor-core Gram kernel) is replaced by the kept eigenvectors (n x kFacCols, q-major) and gains, the
// kept count goes to op.blk_ra.  Blocks that are not finite, or not converged after kJacobiLogSweeps sweeps, go to the wide
// kernel through the fallback list; so do blocks that keep more than kFacCols components, with W = V diag(g) V^H
// in place of their Gram matrix, so that only the product C W is left there.  Up to kColBatch columns are formed like
// the few of a factor; for more the rotations are undone on diag(g), which costs about what the sweeps did, whatever the
// count.  1024 blocks of 512 x 106 keeping 12 / all: 41 ms with everything done twice, 29 / 30 ms in the wide
// kernel alone, 16 / 20 ms this way; 16 blocks keeping all 6.3, 4.7 and 3.9 ms.
//
// Against that kernel, which updates the full matrix and the full eigenvector matrix in every step:
//   * only the upper triangle is kept and updated (half the 2 x 2 blocks of a step);
//   * eigenvectors are not accumulated: every step's rotations go to a log in global memory (L2), and the few
//     kept columns are formed afterwards as J_1 J_2 ... J_N e_k by running the log backwards, one warp
//     per column -- the same matrix product, associated from the right, at 1 / n of the work;
//   * 49 KB of shared memory at n = 106 (packed) instead of 212, so four CTAs of 256 threads per SM: one CTA's
//     rotation angles (a serial chain on n / 2 threads) and barriers overlap the others' updates.
// Bound: instruction issue of the updates (68 % of the slots; index arithmetic of the half storage as much as the
// rotations), then the two barriers per step.  4096 blocks of 512 x 106, 1857 of them through the sweeps:
// 67.6 ms in the wide kernel (Gram and apply included), 14.5 ms here with two CTAs of 512 threads per SM, 12.9 ms
// with four of 256.
// A Householder path in its place took 2.5 ms.  A rotation's c^2 + s^2 = 1 + O(eps) makes the Jacobi kernels' singular
// values and vectors short by a few 1e-6 (residuals 5e-5), so its results differ from these by that much, towards
// 64 bits; it is not built.
#include <algorithm>
#include <type_traits>

#include "llr_prox_common.cuh"

namespace llr {

namespace {

constexpr int kJacThreads = 256;
constexpr int kJacHalf = kProxMaxN / 2;
constexpr int kColBatch = kJacThreads / 32 * 4;   // kept columns formed one by one; above, W is
constexpr int kJacTasks = (kJacHalf * (kJacHalf + 1) / 2 + kJacThreads - 1) / kJacThreads;   // 2 x 2 blocks per thread

struct JacSmem {
  float4 rot[kJacHalf];          // c, s, e of every pair
  int2 pairs[kJacHalf];          // p < q
  float ev[kProxMaxN], g[kProxMaxN];
  int act[kProxMaxN];
  float red[2][kJacThreads / 32];
  int flag[2];
  int n_active;
  int next;
};

__device__ __forceinline__ int2 jac_pair(int k, int step, int M) {
  int p, q;
  if (k == 0) { p = step; q = M; }
  else {   // modulo M
    p = step + k; if (p >= M) p -= M;
    q = step - k; if (q < 0) q += M;
  }
  return p < q ? make_int2(p, q) : make_int2(q, p);
}

__global__ void __launch_bounds__(kJacThreads, 4) llr_eig_jacobi_kernel(ProxOp op, long long nblocks) {
  extern __shared__ __align__(16) unsigned char smem[];
  JacSmem* W = reinterpret_cast<JacSmem*>(smem);
  // upper triangle packed by rows: (i, j), i <= j, at row(i) + j
  float2* A = reinterpret_cast<float2*>(smem + align16(sizeof(JacSmem)));
  const int n = op.n, n2 = (n + 1) & ~1, half = n2 >> 1, M = n2 - 1;
  auto row = [&](int i) { return (i * (2 * n2 - 1 - i)) >> 1; };
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool soft = op.mode != LLR_PROX_HARD_RANK;
  const float thr = op.lambda * op.lambda;
  float* log = op.rot_log + (long long)blockIdx.x * jacobi_log_stride(n);   // (t, e) per pair and step
  int* counter = op.blk_ra + nblocks;   // dynamic block queue, zeroed before the launch
  // the thread's 2 x 2 blocks (k1 <= k2), the same in every step
  int task[kJacTasks];
#pragma unroll
  for (int u = 0; u < kJacTasks; ++u) {
    const int b = tid + u * kJacThreads;
    int k2 = (int)((sqrtf(8.f * b + 1.f) - 1.f) * 0.5f);
    while ((k2 + 1) * (k2 + 2) / 2 <= b) ++k2;
    while (k2 * (k2 + 1) / 2 > b) --k2;
    task[u] = k2 < half ? (b - k2 * (k2 + 1) / 2) | (k2 << 8) : -1;
  }
  int slot = 0;
  auto block_total = [&](float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    float* r = W->red[slot];
    slot ^= 1;
    if (lane == 0) r[warp] = v;
    __syncthreads();
    float s = 0.f;
    for (int w = 0; w < kJacThreads / 32; ++w) s += r[w];
    return s;
  };
  for (;;) {
    if (tid == 0) W->next = atomicAdd(counter, 1);
    __syncthreads();
    const long long blk = W->next;
    if (blk >= nblocks) break;
    float2* G = op.gram + blk * op.gram_stride;
    // upper triangle from the packed lower one
    float s_all = 0.f, s_diag = 0.f, tr = 0.f;
    if (n2 != n)
      for (int i = tid; i < n2; i += kJacThreads) A[row(i) + n] = make_float2(0.f, 0.f);
    for (int i = warp; i < n; i += kJacThreads / 32)
      for (int j = lane; j <= i; j += 32) {
        const float2 v = G[i * (i + 1) / 2 + j];
        A[row(j) + i] = make_float2(v.x, -v.y);
        s_all += cabs2(v);
        if (j == i) { s_diag += v.x * v.x; tr += v.x; }
      }
    const float fro2 = block_total(2.f * s_all - s_diag);
    const float trace = block_total(tr);
    const double mu = (double)trace / n;
    const double ub = mu + sqrt(fmax((double)fro2 / n - mu * mu, 0.0)) * sqrt((double)(n - 1));
    int ra = 0;
    bool done = true;
    if (soft ? op.lambda <= 0.f : op.rank >= n) ra = -2;    // every component kept: identity
    else if (!isfinite(fro2)) ra = -1;   // no angle compares with it: the wide kernel multiplies C by W and lets NaN through
    else if (soft && (fro2 <= thr * thr || ub <= (double)thr)) ra = 0;
    else done = false;
    // one step's rotations on the packed matrix: A <- J^H A J, or undone A <- J A J^H
    auto update = [&](auto undo) {
#pragma unroll
      for (int u = 0; u < kJacTasks; ++u) {
        if (task[u] < 0) continue;
        const int k1 = task[u] & 255, k2 = task[u] >> 8;
        const float4 R1 = W->rot[k1], R2 = W->rot[k2];
        const bool id1 = R1.y == 0.f, id2 = R2.y == 0.f;
        if (id1 && id2) continue;
        const int2 P1 = W->pairs[k1], P2 = W->pairs[k2];
        // element (i, j) lives at (min, max), conjugated below the diagonal
        auto at = [&](int i, int j) { return row(min(i, j)) + max(i, j); };
        const int i11 = at(P1.x, P2.x), i12 = at(P1.x, P2.y), i21 = at(P1.y, P2.x), i22 = at(P1.y, P2.y);
        const float2 f11 = make_float2(1.f, P1.x <= P2.x ? 1.f : -1.f), f12 = make_float2(1.f, P1.x <= P2.y ? 1.f : -1.f);
        const float2 f21 = make_float2(1.f, P1.y <= P2.x ? 1.f : -1.f), f22 = make_float2(1.f, P1.y <= P2.y ? 1.f : -1.f);
        float2 a11 = __fmul2_rn(A[i11], f11), a12 = __fmul2_rn(A[i12], f12);
        float2 a21 = __fmul2_rn(A[i21], f21), a22 = __fmul2_rn(A[i22], f22);
        // (x, y) <- (c x - s e y, s x + c e y), undone (c x + s y, e (c y - s x)); ex = (e.x, e.x), ey = (-e.y, e.y)
        auto turn = [](float2& x, float2& y, float2 cc, float2 ss, float2 ms, float2 ex, float2 ey) {
          if constexpr (decltype(undo)::value) {
            const float2 d = __ffma2_rn(ms, x, __fmul2_rn(cc, y));
            x = __ffma2_rn(ss, y, __fmul2_rn(cc, x));
            y = __ffma2_rn(make_float2(d.y, d.x), ey, __fmul2_rn(d, ex));
          } else {
            const float2 ty = __ffma2_rn(make_float2(y.y, y.x), ey, __fmul2_rn(y, ex));
            const float2 nx = __ffma2_rn(ms, ty, __fmul2_rn(cc, x));
            y = __ffma2_rn(ss, x, __fmul2_rn(cc, ty));
            x = nx;
          }
        };
        const float sg = decltype(undo)::value ? -1.f : 1.f;
        if (!id2) {  // columns: [x_p, x_q] J2 (undone: J2^H),  J2 = [[c, s], [-s e2*, c e2*]]
          const float2 cc = make_float2(R2.x, R2.x), ss = make_float2(R2.y, R2.y), ms = make_float2(-R2.y, -R2.y);
          const float2 ex = make_float2(R2.z, R2.z), ey = make_float2(sg * R2.w, -sg * R2.w);
          turn(a11, a12, cc, ss, ms, ex, ey);
          turn(a21, a22, cc, ss, ms, ex, ey);
        }
        if (!id1) {  // rows: J1^H [row_p; row_q] (undone: J1),  J1^H = [[c, -s e1], [s, c e1]]
          const float2 cc = make_float2(R1.x, R1.x), ss = make_float2(R1.y, R1.y), ms = make_float2(-R1.y, -R1.y);
          const float2 ex = make_float2(R1.z, R1.z), ey = make_float2(-sg * R1.w, sg * R1.w);
          turn(a11, a21, cc, ss, ms, ex, ey);
          turn(a12, a22, cc, ss, ms, ex, ey);
        }
        if (k1 == k2) {
          A[i11] = make_float2(a11.x, 0.f);
          A[i12] = decltype(undo)::value ? a12 : make_float2(0.f, 0.f);
          A[i22] = make_float2(a22.x, 0.f);
        } else {
          A[i11] = __fmul2_rn(a11, f11);
          A[i12] = __fmul2_rn(a12, f12);
          A[i21] = __fmul2_rn(a21, f21);
          A[i22] = __fmul2_rn(a22, f22);
        }
      }
    };
    if (!done) {
      // Scale the matrix by a power of two (exact) so that its norm lies in [1, 2): entries that matter can
      // be squared.  The angle's quotients may be off in the last bits (its tangent only has to annihilate to
      // rounding); c, s and the unit phase e, which set how orthogonal the rotation is, are formed as in the
      // wide kernel.
      const float nrm = sqrtf(fro2);
      const int ex2 = min(max((__float_as_int(nrm) >> 23) & 0xff, 1), 253);
      const float up = __int_as_float((254 - ex2) << 23), down = __int_as_float(ex2 << 23);
      const float normF = nrm * up, rthr = 2.4e-7f * normF;
      for (int i = warp; i < n; i += kJacThreads / 32)
        for (int j = i + lane; j < n; j += 32) {
          const float2 v = A[row(i) + j];
          A[row(i) + j] = make_float2(v.x * up, v.y * up);
        }
      if (tid == 0) W->flag[0] = W->flag[1] = 0;
      __syncthreads();
      int steps = 0;
      bool converged = !(normF > 0.f);
      for (int sweep = 0; sweep < kJacobiLogSweeps && !converged; ++sweep) {
        const int fs = sweep & 1;
        for (int step = 0; step < M; ++step, ++steps) {
          if (tid < half) {
            const int2 pq = jac_pair(tid, step, M);
            const int p = pq.x, q = pq.y;
            float c = 1.f, s = 0.f, ex = 1.f, ey = 0.f, t = 0.f;
            if (q < n) {
              const float app = A[row(p) + p].x, aqq = A[row(q) + q].x;
              const float2 apq = A[row(p) + q];
              const float r = sqrtf(apq.x * apq.x + apq.y * apq.y);
              if (r > rthr) {
                // t = sign(tau) / (|tau| + sqrt(1 + tau^2)), tau = (aqq - app) / (2 r)
                const float d = aqq - app, r2 = 2.f * r;
                t = __fdividef(d >= 0.f ? r2 : -r2, fabsf(d) + __fsqrt_rn(fmaf(d, d, r2 * r2)));
                c = rsqrtf(1.f + t * t);
                s = t * c;
                ex = apq.x / r; ey = apq.y / r;
                W->flag[fs] = 1;
              }
            }
            W->rot[tid] = make_float4(c, s, ex, ey);
            W->pairs[tid] = pq;
            float* lg = log + 3 * (steps * half + tid);
            lg[0] = t;
            lg[1] = ex;
            lg[2] = ey;
          }
          __syncthreads();
          if (step == 0 && tid == 0) W->flag[fs ^ 1] = 0;
          update(std::false_type{});
          __syncthreads();
        }
        converged = W->flag[fs] == 0;
      }
      // eigenvalues, gains and the kept list, as singular_map() orders them
      if (tid < n) W->ev[tid] = A[row(tid) + tid].x * down;
      __syncthreads();
      if (tid < n) {
        const float e = W->ev[tid];
        float gv;
        if (!soft) {
          int pos = 0;
          for (int j = 0; j < n; ++j) pos += (W->ev[j] > e) || (W->ev[j] == e && j < tid);
          gv = pos < op.rank ? 1.f : 0.f;
        } else {
          const float sv = sqrtf(fmaxf(e, 0.f));
          gv = sv > op.lambda ? 1.f - op.lambda / sv : 0.f;
        }
        W->g[tid] = gv;
      }
      __syncthreads();
      if (tid == 0) {
        int c = 0;
        for (int j = 0; j < n; ++j)
          if (W->g[j] != 0.f) W->act[c++] = j;
        W->n_active = c;
        if (op.blk_nuc && soft) op.blk_nuc[blk] = nuclear_from_eigs(W->ev, n, op.lambda);
      }
      __syncthreads();
      ra = W->n_active;
      if (!converged) ra = -1;
      // columns act[c0] .. act[c0 + CB - 1] of J_1 ... J_steps, each n2 entries from v on (the matrix is spent); past
      // the last kept one zeros
      auto columns = [&](auto cb, float2* v, int c0) {
        constexpr int CB = decltype(cb)::value;
#pragma unroll
        for (int c = 0; c < CB; ++c) {
          const int col = c0 + c < ra ? W->act[c0 + c] : -1;
          for (int i = lane; i < n2; i += 32) v[c * n2 + i] = make_float2(i == col ? 1.f : 0.f, 0.f);
        }
        __syncwarp();
        constexpr int PF = 4;        // log entries in flight per lane and pair set
        const int ka = lane, kb = lane + 32;
        auto fetch = [&](int st, int k) {
          const float* lg = log + 3 * (st * half + k);
          return st >= 0 && k < half ? make_float3(__ldcg(lg), __ldcg(lg + 1), __ldcg(lg + 2)) : make_float3(0.f, 1.f, 0.f);
        };
        float3 ra4[PF], rb4[PF];
#pragma unroll
        for (int u = 0; u < PF; ++u) {
          ra4[u] = fetch(steps - 1 - u, ka);
          rb4[u] = fetch(steps - 1 - u, kb);
        }
        auto rotate = [&](float3 r3, int k, int step) {
          if (r3.x == 0.f) return;   // identity (also lanes past the last pair)
          const float cs = rsqrtf(1.f + r3.x * r3.x);
          const float4 r = make_float4(cs, r3.x * cs, r3.y, r3.z);
          const int2 pq = jac_pair(k, step, M);
          const float2 ec = make_float2(r.z, -r.w);
          float2 vp[CB], vq[CB];
#pragma unroll
          for (int c = 0; c < CB; ++c) { vp[c] = v[c * n2 + pq.x]; vq[c] = v[c * n2 + pq.y]; }
#pragma unroll
          for (int c = 0; c < CB; ++c) {
            const float2 d = make_float2(r.x * vq[c].x - r.y * vp[c].x, r.x * vq[c].y - r.y * vp[c].y);
            v[c * n2 + pq.x] = make_float2(r.x * vp[c].x + r.y * vq[c].x, r.x * vp[c].y + r.y * vq[c].y);
            v[c * n2 + pq.y] = cmul(ec, d);
          }
        };
        int step = M - 1;
        for (int st0 = steps - 1; st0 >= 0; st0 -= PF) {
#pragma unroll
          for (int u = 0; u < PF; ++u) {
            const int st = st0 - u;
            const float3 a = ra4[u], b = rb4[u];
            ra4[u] = fetch(st - PF, ka);
            rb4[u] = fetch(st - PF, kb);
            if (st >= 0) {
              rotate(a, ka, step);
              rotate(b, kb, step);
              __syncwarp();
              step = step == 0 ? M - 1 : step - 1;
            }
          }
        }
      };
      if (ra > kColBatch) {
        // W = J_1 ... J_steps diag(g) J_steps^H ... J_1^H: the rotations undone on the gains
        for (int i = warp; i < n2; i += kJacThreads / 32)
          for (int j = i + lane; j < n2; j += 32) A[row(i) + j] = make_float2(i == j && i < n ? W->g[i] : 0.f, 0.f);
        int step = M - 1;
        float t = 0.f, ex = 1.f, ey = 0.f;
        auto fetch = [&](int st) {
          if (tid >= half || st < 0) return;
          const float* lg = log + 3 * (st * half + tid);
          t = __ldcg(lg); ex = __ldcg(lg + 1); ey = __ldcg(lg + 2);
        };
        fetch(steps - 1);
        for (int st = steps - 1; st >= 0; --st) {
          if (tid < half) {
            const float c = rsqrtf(1.f + t * t);
            W->rot[tid] = make_float4(c, t * c, ex, ey);
            W->pairs[tid] = jac_pair(tid, step, M);
          }
          fetch(st - 1);
          __syncthreads();
          update(std::true_type{});
          __syncthreads();
          step = step == 0 ? M - 1 : step - 1;
        }
        for (int i = warp; i < n; i += kJacThreads / 32)
          for (int j = lane; j <= i; j += 32) {
            const float2 w = A[row(j) + i];
            G[i * (i + 1) / 2 + j] = make_float2(w.x, -w.y);
          }
        ra = kBlkW;
      } else if (ra > kFacCols) {
        // W = V diag(g) V^H from the columns themselves, four per warp
        if (4 * warp < ra) columns(std::integral_constant<int, 4>{}, A + 4 * warp * n2, 4 * warp);
        __syncthreads();
        for (int i = warp; i < n; i += kJacThreads / 32)
          for (int j = lane; j <= i; j += 32) {
            float2 w = make_float2(0.f, 0.f);
            for (int c = 0; c < ra; ++c) {
              const float2 p = cmul_bc(A[c * n2 + i], A[c * n2 + j]);
              const float gc = W->g[W->act[c]];
              w.x = fmaf(gc, p.x, w.x);
              w.y = fmaf(gc, p.y, w.y);
            }
            G[i * (i + 1) / 2 + j] = w;
          }
        ra = kBlkW;
      } else if (ra > 0 && warp < ra) {
        float2* v = A + warp * n2;
        columns(std::integral_constant<int, 1>{}, v, warp);
        for (int i = lane; i < n; i += 32) G[i * kFacCols + warp] = v[i];
        if (lane == 0) G[n * kFacCols + warp] = make_float2(W->g[W->act[warp]], 0.f);
      }
    }
    if (tid == 0) {
      op.blk_ra[blk] = ra;
      if (ra == -1 || ra == kBlkW) op.fb_list[atomicAdd(op.fb_count, 1)] = (int)blk;
    }
    __syncthreads();
  }
}

size_t jac_smem(int n) {
  const int n2 = (n + 1) & ~1;
  // the packed matrix, or the columns that follow it (fewer from n2 = 64 on)
  return align16(sizeof(JacSmem)) + sizeof(float2) * std::max<size_t>((size_t)n2 * (n2 + 1) / 2, (size_t)kColBatch * n2);
}

}  // namespace

int jacobi_ctas(int n) {
  return wide_jacobi_ctas() * (int)std::max<size_t>(1, std::min<size_t>(kJacobiPerSm, 228 * 1024 / (jac_smem(n) + 1024)));
}

int launch_llr_eig_jacobi(const ProxOp& op, long long nblocks, cudaStream_t stream) {
  if (!op.gram || !op.blk_ra || !op.fb_list || !op.fb_count || !op.rot_log || op.rot_ctas < 1)
    return set_error(LLR_ERR_INVALID, "eigen kernel needs the Gram scratch, block codes, fallback list and log");
  if (op.n > kProxMaxN || op.gram_stride < prox_gram_stride(op.n)) return set_error(LLR_ERR_INVALID, "bad Gram scratch");
  if (nblocks == 0) return LLR_OK;
  auto kern = llr_eig_jacobi_kernel;
  const size_t smem = jac_smem(op.n);
  LLR_CUDA_TRY(allow_smem(kern));
  LLR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  LLR_CUDA_TRY(cudaMemsetAsync(op.blk_ra + nblocks, 0, sizeof(int), stream));
  note_launch();
  kern<<<(unsigned)std::min<long long>(nblocks, op.rot_ctas), kJacThreads, smem, stream>>>(op, nblocks);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

}  // namespace llr

// Eigen stage of the split LLR prox path for 48 < n <= 64 columns: a CTA of two warps per Casorati block.
//
// The same decisions, method and outputs as the one-warp kernel for n <= 48 (llr_eig_warp.cu: Frobenius bound,
// diagonal test, Cholesky certificate, Householder tridiagonalisation, Sturm counts, multisection, twisted
// factorisation, back-transformation; factors and gains in place of the packed Gram matrix, kept count in
// op.blk_ra, blocks it cannot finish on the fallback list).
//
// Bound: shared-memory accesses and latency of the Householder steps.  A block's matrix and vectors (20.5 KB at
// n = 61) allow ten blocks per SM; two warps per block are twenty per SM where one warp per block left ten,
// with a third of the issue slots and half of the shared-memory bandwidth used.  A thread owns one row of
// the trailing matrix, so the steps walk the columns with the vector entries broadcast, stored twice per
// component (two packed FMAs per complex MAC).  Which warp takes which rows alternates from CTA to CTA, since
// the rows that die first leave a warp idle.  4096 blocks of 61 columns, rank 6: 719 us with one warp per block,
// 627 us here (4096 blocks of 33 columns: 140 and 165 us, hence the line at 48).  Keeping
// the rows in registers (two warps, columns unrolled) took 1227 us: 255 registers or spills.
#include <algorithm>

#include "llr_prox_common.cuh"

namespace llr {

namespace {

constexpr int kTeam = 64;            // threads per block, at least n
constexpr float kTeamMargin = 0.1f;  // eigenvalues this far below lambda^2 are kept for the refined gains

__host__ __device__ inline int tri(int i) { return (i * (i + 1)) / 2; }

struct TeamEig {
  union {
    struct {
      float4 ud[kTeam];              // (u.x, u.x, u.y, u.y): Householder vector / Cholesky column
      float4 wd[kTeam];              // the same for p - K u
    };
    float um[kFacCols * kTeam];      // eigenvector stage: D+ / U- of each lane's factorisation
  };
  float Y[kFacCols * kTeam];         // eigenvectors of T', column a at Y[a * kTeam]
  float2 e[kTeam];                   // complex sub-diagonal of T, then the unitary diagonal delta
  float d[kTeam], ae[kTeam], tau[kTeam];
  float lam[kFacCols];
  float red[2][2];
  float gl, gu, tnorm, pivmin;
  int next, flag;
};

struct Team {
  TeamEig* W;
  float2* A;                         // packed lower triangle; later Householder vectors
  int n, tid, lane, warp, row;       // row: the thread's row of the trailing matrix
  int slot;                          // alternating reduction slots

  __device__ __forceinline__ float sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    float* r = W->red[slot];
    slot ^= 1;
    if (lane == 0) r[warp] = v;
    __syncthreads();
    return r[0] + r[1];
  }
  __device__ __forceinline__ float maxv(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    float* r = W->red[slot];
    slot ^= 1;
    if (lane == 0) r[warp] = v;
    __syncthreads();
    return fmaxf(r[0], r[1]);
  }
};

__device__ __forceinline__ float4 dup2(float2 v) { return make_float4(v.x, v.x, v.y, v.y); }
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

// True when thr I - G is positive definite (unpivoted Cholesky).  Overwrites A.
__device__ bool team_below(Team& t, float thr) {
  float2* A = t.A;
  TeamEig* W = t.W;
  const int n = t.n, P = tri(n), w0 = t.row & ~31;
  for (int i = t.tid; i < P; i += kTeam) A[i] = make_float2(-A[i].x, -A[i].y);
  __syncthreads();
  if (t.tid < n) A[tri(t.tid) + t.tid].x += thr;
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    const float dk = A[tri(k) + k].x;
    if (!(dk > 0.f)) return false;   // the same value in every thread
    const float s = 1.f / sqrtf(dk);
    const int o = k + 1, L = n - o;
    if (L == 0) break;
    const int i = min(t.row, L - 1);
    const float2 l = cscale(A[tri(o + i) + k], s);
    if (t.row < L) W->ud[t.row] = dup2(l);
    __syncthreads();
    if (w0 < L) {
      // A[i][j] -= l_i conj(l_j): l conj(m) = l m.x + (l.y, -l.x) m.y
      const float2 nl = make_float2(-l.x, -l.y), nls = make_float2(-l.y, l.x);
      float2* a = A + tri(o + i) + o;
#pragma unroll 4
      for (int j = 0; j < w0; ++j) {
        const float4 m = W->ud[j];
        const float2 v = ffma2(nls, hi2(m), ffma2(nl, lo2(m), a[j]));
        if (t.row < L) a[j] = v;
      }
      const int je = min(w0 + 32, L);
      for (int j = w0; j < je; ++j)
        if (j <= t.row && t.row < L) {
          const float4 m = W->ud[j];
          a[j] = ffma2(nls, hi2(m), ffma2(nl, lo2(m), a[j]));
        }
    }
    __syncthreads();
  }
  return true;
}

// Householder reduction of the packed Hermitian A to tridiagonal T (H = I - tau u u^H); column k keeps u_k below
// the diagonal for the back-transformation.
__device__ void team_tridiag(Team& t) {
  float2* A = t.A;
  TeamEig* W = t.W;
  const int n = t.n, w0 = t.row & ~31;
  for (int k = 0; k + 2 < n; ++k) {
    const int o = k + 1, L = n - o;
    const bool own = t.row < L;
    const int i = min(t.row, L - 1);
    float2 x = A[tri(o + i) + k];
    if (!own) x = make_float2(0.f, 0.f);
    const float2 x0 = A[tri(o) + k];
    const float s2 = t.sum(cabs2(x));
    const float xn = sqrtf(s2), aa = sqrtf(cabs2(x0));
    const float phx = aa > 0.f ? x0.x / aa : 1.f, phy = aa > 0.f ? x0.y / aa : 0.f;
    const float2 u0 = make_float2(x0.x + phx * xn, x0.y + phy * xn);
    const float un2 = s2 - aa * aa + cabs2(u0);
    const float tk = (xn > 0.f && un2 > 0.f) ? 2.f / un2 : 0.f;
    if (t.row == 0) {
      W->tau[k] = tk;
      W->e[k] = make_float2(-phx * xn, -phy * xn);
      A[tri(o) + k] = u0;
      x = u0;
    }
    if (tk == 0.f) {   // the same value in every thread: no reflection at this step
      __syncthreads();
      continue;
    }
    W->ud[t.row] = dup2(x);
    __syncthreads();
    // p = tau A22 u: columns left of the warp's rows from the row itself, columns right of them
    // from the rows below (conjugated), the 32 in between by comparison
    float2 p = make_float2(0.f, 0.f);
    if (w0 < L) {
      float2 c1 = p, c2 = p, c3 = p, c4 = p;
      const float2* a = A + tri(o + i) + o;
#pragma unroll 8
      for (int j = 0; j < w0; ++j) {
        const float4 u = W->ud[j];
        const float2 v = a[j];
        c1 = ffma2(v, lo2(u), c1);
        c2 = ffma2(v, hi2(u), c2);
      }
      const int je = min(w0 + 32, L);
      const float2* b = A + tri(o + w0) + o + i;   // A[o + j][o + i]
      int step = o + w0 + 1;
#pragma unroll 4
      for (int j = w0; j < je; ++j) {
        const float4 u = W->ud[j];
        const bool low = j <= i;
        float2 v = *(low ? a + j : b);
        if (!low) v.y = -v.y;
        c1 = ffma2(v, lo2(u), c1);
        c2 = ffma2(v, hi2(u), c2);
        b += step++;
      }
#pragma unroll 8
      for (int j = je; j < L; ++j) {
        const float4 u = W->ud[j];
        const float2 v = *b;
        c3 = ffma2(v, lo2(u), c3);
        c4 = ffma2(v, hi2(u), c4);
        b += step++;
      }
      p = make_float2((c1.x - c2.y) + (c3.x + c4.y), (c1.y + c2.x) + (c4.x - c3.y));
      p = own ? cscale(p, tk) : make_float2(0.f, 0.f);
    }
    const float dp = t.sum(x.x * p.x + x.y * p.y);
    const float K = 0.5f * tk * dp;
    const float2 w = csub(p, cscale(x, K));
    W->wd[t.row] = dup2(w);
    __syncthreads();
    // A22 -= u w^H + w u^H on the lower triangle
    if (w0 < L) {
      const float2 nu = make_float2(-x.x, -x.y), nus = make_float2(-x.y, x.x);
      const float2 nw = make_float2(-w.x, -w.y), nws = make_float2(-w.y, w.x);
      float2* a = A + tri(o + i) + o;
#pragma unroll 4
      for (int j = 0; j < w0; ++j) {
        const float4 wj = W->wd[j], uj = W->ud[j];
        float2 v = ffma2(nus, hi2(wj), ffma2(nu, lo2(wj), a[j]));
        v = ffma2(nws, hi2(uj), ffma2(nw, lo2(uj), v));
        if (own) a[j] = v;
      }
      const int je = min(w0 + 32, L);
#pragma unroll 2
      for (int j = w0; j < je; ++j) {
        const float4 wj = W->wd[j], uj = W->ud[j];
        const bool on = own && j <= t.row;
        float2 v = a[on ? j : 0];
        v = ffma2(nus, hi2(wj), ffma2(nu, lo2(wj), v));
        v = ffma2(nws, hi2(uj), ffma2(nw, lo2(uj), v));
        if (on) a[j] = v;
      }
    }
    __syncthreads();
  }
  if (t.tid < n) W->d[t.tid] = A[tri(t.tid) + t.tid].x;
  if (t.tid == 0) {
    if (n >= 2) W->e[n - 2] = A[tri(n - 1) + n - 2];
    for (int k = max(0, n - 2); k < n; ++k) W->tau[k] = 0.f;
  }
  __syncthreads();
}

__device__ __forceinline__ int team_sturm(const float* d, const float* ae, int n, float x, float pivmin) {
  float q = d[0] - x;
  if (fabsf(q) <= pivmin) q = -pivmin;
  int c = q < 0.f;
  for (int i = 1; i < n; ++i) {
    const float a = ae[i - 1];
    q = d[i] - x - a * a * __frcp_rn(q);
    if (fabsf(q) <= pivmin) q = -pivmin;
    c += q < 0.f;
  }
  return c;
}

// Real form T' = D^H T D (D a prefix product of unit phases, left in W->e), |e| and the Gershgorin
// bounds.  Warp 0, two columns per lane.
__device__ void team_setup(Team& t) {
  TeamEig* W = t.W;
  const int n = t.n, lane = t.lane;
  if (t.warp == 0) {
    float2 ph[2];
    float e2m = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = 2 * lane + h;
      ph[h] = make_float2(1.f, 0.f);
      if (k + 1 < n) {
        const float2 ek = W->e[k];
        const float a = sqrtf(cabs2(ek));
        W->ae[k] = a;
        e2m = fmaxf(e2m, a * a);
        if (a > 0.f) ph[h] = make_float2(ek.x / a, ek.y / a);
      } else if (k < n) {
        W->ae[k] = 0.f;
      }
    }
    float2 pr = cmul(ph[0], ph[1]);
    for (int o = 1; o < 32; o <<= 1) {
      const float ox = __shfl_up_sync(0xffffffffu, pr.x, o), oy = __shfl_up_sync(0xffffffffu, pr.y, o);
      if (lane >= o) pr = cmul(make_float2(ox, oy), pr);
    }
    float ex = __shfl_up_sync(0xffffffffu, pr.x, 1), ey = __shfl_up_sync(0xffffffffu, pr.y, 1);
    if (lane == 0) { ex = 1.f; ey = 0.f; }
    __syncwarp();
    float2 run = make_float2(ex, ey);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = 2 * lane + h;
      if (k < n) W->e[k] = run;
      run = cmul(run, ph[h]);
    }
    __syncwarp();
    float gl = 3.0e38f, gu = -3.0e38f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = 2 * lane + h;
      if (k < n) {
        const float r = (k > 0 ? W->ae[k - 1] : 0.f) + (k + 1 < n ? W->ae[k] : 0.f);
        gl = fminf(gl, W->d[k] - r);
        gu = fmaxf(gu, W->d[k] + r);
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      gl = fminf(gl, __shfl_xor_sync(0xffffffffu, gl, o));
      gu = fmaxf(gu, __shfl_xor_sync(0xffffffffu, gu, o));
      e2m = fmaxf(e2m, __shfl_xor_sync(0xffffffffu, e2m, o));
    }
    if (lane == 0) {
      const float tn = fmaxf(fabsf(gl), fabsf(gu)), pad = 4.f * 1.1920929e-7f * tn * n + 1e-30f;
      W->tnorm = tn;
      W->gl = gl - pad;
      W->gu = gu + pad;
      W->pivmin = 1.1754944e-38f * fmaxf(1.f, e2m);
    }
  }
  __syncthreads();
}

// Eigenvalues j0 .. j0 + count - 1 (ascending, count <= kFacCols) by multisection: 32, 16 or 8 lanes per
// eigenvalue for up to two, four and eight of them; a group splits its interval that many ways plus one per round.
__device__ void team_eigenvalues(Team& t, int j0, int count) {
  TeamEig* W = t.W;
  const int G = count <= 2 ? 32 : (count <= 4 ? 16 : 8);
  const int gl = t.lane & (G - 1), group = t.tid / G;
  const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << G) - 1u);
  const float inv = 1.f / (float)(G + 1);
  const bool act = group < count;
  const int j = j0 + (act ? group : 0);
  float lo = W->gl, hi = W->gu;
  const float pivmin = W->pivmin;
  for (int round = 0; round < 40; ++round) {
    const bool conv = !act || (hi - lo) <= 2.4e-7f * fmaxf(fabsf(lo), fabsf(hi)) + pivmin;
    if (__all_sync(0xffffffffu, conv)) break;
    const float x = lo + (hi - lo) * (float)(gl + 1) * inv;
    const bool le = act ? (team_sturm(W->d, W->ae, t.n, x, pivmin) <= j) : true;
    const unsigned bal = __ballot_sync(0xffffffffu, le);
    const int nt = __popc((bal >> (t.lane & ~(G - 1) & 31)) & gmask);
    const float nlo = nt > 0 ? lo + (hi - lo) * (float)nt * inv : lo;
    const float nhi = nt < G ? lo + (hi - lo) * (float)(nt + 1) * inv : hi;
    lo = nlo;
    hi = nhi;
  }
  if (act && gl == 0) W->lam[group] = 0.5f * (lo + hi);
  __syncthreads();
}

// Eigenvectors of T' for the ra kept eigenvalues (warp 0): lane a solves its twisted factorisation, then the warp
// orthonormalises them and checks ||T' y - lam y||.  Returns false when a vector fails.
__device__ bool team_vectors(Team& t, int ra) {
  TeamEig* W = t.W;
  const int n = t.n, lane = t.lane;
  if (t.warp == 0) {
    const float eps = 1.1920929e-7f, tnorm = fmaxf(W->tnorm, 1e-30f);
    const float tiny = eps * tnorm;
    if (lane == 0) {
      const float sep = 10.f * eps * tnorm;
      for (int a = 1; a < ra; ++a)
        if (W->lam[a] - W->lam[a - 1] < sep) W->lam[a] = W->lam[a - 1] + sep;
    }
    __syncwarp();
    if (lane < ra) {
      float* y = W->Y + lane * kTeam;
      float* Um = W->um + lane * kTeam;
      const float lam = W->lam[lane];
      float dp = W->d[0] - lam;
#pragma unroll 4
      for (int i = 0; i + 1 < n; ++i) {
        if (fabsf(dp) < tiny) dp = copysignf(tiny, dp);
        Um[i] = dp;   // D+_i, replaced by U-_i on the way back
        const float l = W->ae[i] * __frcp_rn(dp);
        y[i] = l;
        dp = W->d[i + 1] - lam - l * W->ae[i];
      }
      if (fabsf(dp) < tiny) dp = copysignf(tiny, dp);
      float dm = W->d[n - 1] - lam;
      float best = fabsf(dp);
      int r = n - 1;
#pragma unroll 4
      for (int i = n - 2; i >= 0; --i) {
        if (fabsf(dm) < tiny) dm = copysignf(tiny, dm);
        const float um = W->ae[i] * __frcp_rn(dm);
        const float dpi = Um[i];
        Um[i] = um;
        dm = W->d[i] - lam - um * W->ae[i];
        const float gamma = dpi + dm - (W->d[i] - lam);
        if (fabsf(gamma) < best) { best = fabsf(gamma); r = i; }
      }
      float zz = 1.f;
      for (int i = r - 1; i >= 0; --i) { zz = -y[i] * zz; y[i] = zz; }
      y[r] = 1.f;
      zz = 1.f;
      for (int i = r; i + 1 < n; ++i) { zz = -Um[i] * zz; y[i + 1] = zz; }
      float mx = 0.f;
      for (int i = 0; i < n; ++i) mx = fmaxf(mx, fabsf(y[i]));
      const float sc = (mx > 0.f && mx < 3.0e38f) ? 1.f / mx : 0.f;
      for (int i = 0; i < n; ++i) y[i] *= sc;
    }
    __syncwarp();
    auto wsum = [](float v) {
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      return v;
    };
    const float tol = 2e-5f * tnorm;
    bool bad = false;
    for (int a = 0; a < ra; ++a) {
      float* y = W->Y + a * kTeam;
      float v[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) v[h] = lane + 32 * h < n ? y[lane + 32 * h] : 0.f;
      for (int c = 0; c < a; ++c) {
        const float* zc = W->Y + c * kTeam;
        float z[2], s = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          z[h] = lane + 32 * h < n ? zc[lane + 32 * h] : 0.f;
          s += v[h] * z[h];
        }
        s = wsum(s);
#pragma unroll
        for (int h = 0; h < 2; ++h) v[h] -= s * z[h];
      }
      const float nn = wsum(v[0] * v[0] + v[1] * v[1]);
      const float inv = nn > 0.f ? rsqrtf(nn) : 0.f;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (lane + 32 * h < n) y[lane + 32 * h] = v[h] * inv;
      __syncwarp();
      const float lam = W->lam[a];
      float r2 = 0.f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;
        if (i < n) {
          float rr = (W->d[i] - lam) * y[i];
          if (i > 0) rr += W->ae[i - 1] * y[i - 1];
          if (i + 1 < n) rr += W->ae[i] * y[i + 1];
          r2 += rr * rr;
        }
      }
      r2 = wsum(r2);
      if (!(nn > 0.f) || !(sqrtf(r2) <= tol)) bad = true;
      __syncwarp();
    }
    if (lane == 0) W->flag = bad ? 1 : 0;
  }
  __syncthreads();
  return W->flag == 0;
}

// V = Q D Y, Q = H_0 H_1 ... H_{n-3}: 32, 16 or 8 lanes per kept vector, rows g, g + Gv, ... in registers.
//  Written q-major to fac[q * kFacCols + a].
__device__ void team_backtransform(Team& t, int ra, float2* fac) {
  constexpr int kPer = kTeam / 8;
  TeamEig* W = t.W;
  const float2* A = t.A;
  const int n = t.n;
  const int Gv = ra <= 2 ? 32 : (ra <= 4 ? 16 : 8);
  const int a = t.tid / Gv, g = t.tid - a * Gv;
  const bool act = a < ra;
  const float2 z = make_float2(0.f, 0.f);
  float2 v[kPer];
#pragma unroll
  for (int h = 0; h < kPer; ++h) {
    const int i = g + Gv * h;
    v[h] = (act && i < n) ? cscale(W->e[i], W->Y[a * kTeam + i]) : z;
  }
  if (32 * t.warp < ra * Gv)
    for (int k = n - 3; k >= 0; --k) {
      const float tk = W->tau[k];
      if (tk == 0.f) continue;
      float2 s = z, uu[kPer];
#pragma unroll
      for (int h = 0; h < kPer; ++h) {
        const int i = g + Gv * h;
        uu[h] = (i > k && i < n) ? A[tri(i) + k] : z;
        s = cadd(s, cmulc(uu[h], v[h]));
      }
      for (int o = Gv >> 1; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
      }
      s = cscale(s, tk);
#pragma unroll
      for (int h = 0; h < kPer; ++h) v[h] = csub(v[h], cmul(uu[h], s));
    }
#pragma unroll
  for (int h = 0; h < kPer; ++h) {
    const int i = g + Gv * h;
    if (act && i < n) fac[i * kFacCols + a] = v[h];
  }
}

__global__ void __launch_bounds__(kTeam, 10) llr_eig_team_kernel(ProxOp op, long long nblocks) {
  extern __shared__ __align__(16) unsigned char smem[];
  Team t;
  t.W = reinterpret_cast<TeamEig*>(smem);
  t.A = reinterpret_cast<float2*>(smem + sizeof(TeamEig));
  t.n = op.n;
  t.tid = threadIdx.x;
  t.lane = t.tid & 31;
  t.warp = t.tid >> 5;
  t.row = 32 * ((t.warp + blockIdx.x) & 1) + t.lane;
  t.slot = 0;
  TeamEig* W = t.W;
  const int n = op.n, P = tri(n);
  const bool soft = op.mode != LLR_PROX_HARD_RANK;
  const float thr = op.lambda * op.lambda;
  const float thr_lo = thr * (1.f - kTeamMargin);
  int* counter = op.blk_ra + nblocks;   // dynamic block queue, zeroed before the launch
  for (;;) {
    if (t.tid == 0) W->next = atomicAdd(counter, 1);
    __syncthreads();
    const long long blk = W->next;
    if (blk >= nblocks) break;
    float2* G = op.gram + blk * op.gram_stride;
    float s_all = 0.f;
    for (int i = t.tid; i < P; i += kTeam) {
      const float2 v = G[i];
      t.A[i] = v;
      s_all += cabs2(v);
    }
    __syncthreads();
    float dg = t.tid < n ? t.A[tri(t.tid) + t.tid].x : 0.f;
    const float fro2 = t.sum(2.f * s_all - dg * dg);   // ||G||_F^2 from the lower triangle
    const float dmax = t.maxv(dg);
    int ra;
    if ((!soft && op.rank >= n) || (soft && !(op.lambda > 0.f))) {
      ra = -2;                                            // identity: leave the block as is
    } else if (soft && fro2 <= thr_lo * thr_lo) {
      ra = 0;                                             // lambda_max <= ||G||_F, clear of the margin
    } else {
      bool eig = !soft || dmax > thr_lo;                  // lambda_max >= max_i G_ii
      if (!eig) {
        eig = !team_below(t, thr_lo);
        if (eig) {                                        // the test overwrote A: reload
          __syncthreads();
          for (int i = t.tid; i < P; i += kTeam) t.A[i] = G[i];
          __syncthreads();
        }
      }
      if (!eig) {
        ra = 0;
      } else {
        team_tridiag(t);
        team_setup(t);
        int nb, nb_lo;
        if (!soft) {
          nb = nb_lo = n - op.rank;
        } else {                                          // every thread runs the counts: same answer
          nb = team_sturm(W->d, W->ae, n, thr, W->pivmin);
          nb_lo = team_sturm(W->d, W->ae, n, thr_lo, W->pivmin);
        }
        ra = n - nb > kFacCols ? -1 : min(n - nb_lo, kFacCols);   // kept in FP32, plus the near-threshold ones
        if (ra > 0) {
          team_eigenvalues(t, n - ra, ra);
          if (!team_vectors(t, ra)) {
            ra = -1;
          } else {
            team_backtransform(t, ra, G);
            if (t.tid < ra) {
              float gv = 1.f;
              if (soft) {
                const float sv = sqrtf(fmaxf(W->lam[t.tid], 0.f));
                gv = sv > op.lambda ? 1.f - op.lambda / sv : 0.f;
              }
              G[n * kFacCols + t.tid] = make_float2(gv, 0.f);
            }
          }
        }
      }
    }
    if (t.tid == 0) {
      op.blk_ra[blk] = ra;
      if (ra == -1) op.fb_list[atomicAdd(op.fb_count, 1)] = (int)blk;
    }
    __syncthreads();
  }
}

}  // namespace

int launch_llr_eig_team(const ProxOp& op, long long nblocks, cudaStream_t stream) {
  if (!op.gram || !op.blk_ra || !op.fb_list || !op.fb_count)
    return set_error(LLR_ERR_INVALID, "eigen kernel needs the Gram scratch, block codes and fallback list");
  if (op.n > kTeam || op.gram_stride < prox_gram_stride(op.n)) return set_error(LLR_ERR_INVALID, "bad Gram scratch");
  if (nblocks == 0) return LLR_OK;
  const size_t smem = sizeof(TeamEig) + sizeof(float2) * (size_t)tri(op.n);
  auto kern = llr_eig_team_kernel;
  LLR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  LLR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  int dev = 0, nsm = 0, occ = 0;
  LLR_CUDA_TRY(cudaGetDevice(&dev));
  LLR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  LLR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kTeam, smem));
  if (occ < 1) return set_error(LLR_ERR_UNSUPPORTED, "eigen kernel cannot be resident (smem %zu B)", smem);
  LLR_CUDA_TRY(cudaMemsetAsync(op.blk_ra + nblocks, 0, sizeof(int), stream));
  note_launch();
  kern<<<(unsigned)std::min<long long>(nblocks, (long long)nsm * occ), kTeam, smem, stream>>>(op, nblocks);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

}  // namespace llr

// Gram matrices of the LLR blocks on the 5th-generation tensor cores (tcgen05).
//
// For a Casorati block C (m x n complex) let D = [Re C | Im C] (m x 2n real).  Then
// P = D^T D (2n x 2n) gives G = C^H C as
//   Re G[i][j] = P[i][j] + P[n+i][n+j],   Im G[i][j] = P[i][n+j] - P[n+i][j].
// P is one 128 x 128 UMMA accumulator in tensor memory (2n <= 128), K = the m voxel rows.
// Both operands are the same shared-memory tile of D in the K-major layout with the 128-byte
// swizzle (one 128-byte row of 32 TF32 per column of D and chunk), so A = B and the MMA
// computes D^T D directly.
// Precision: 3xTF32 -- x = hi + lo with hi = tf32(x), and P accumulates hi*hi + hi*lo + lo*hi
// in FP32, which keeps FP32-level accuracy (the lo*lo term is below FP32 rounding).
// Wider matrices (64 < n <= 128, NPMAX = 128): Re C and Im C are two operand tiles of 128 columns, and the
// accumulator pair R = Re^T Re + Im^T Im, Q = Re^T Im (256 TMEM columns) gives Re G = R and
// Im G[i][j] = Q[i][j] - Q[j][i].  One CTA of 16 warps per SM (the two chunk buffers take 128 KB).
// Tensor memory truncates its sums, which over a block's 512 rows left G 6.2e-6 short where FP32 FMAs are off by 4.6e-7
// (norm of the error, 106 columns).  So each operand buffer has its own pair, a step's 32 rows start from zero, the
// products with a low part come first, and the pair is added to FP32 sums in registers when its buffer comes
// round again: 1.6e-7, whatever the number of rows.  It costs registers: one step of loads is in flight instead
// of two, and 4096 contiguous blocks of 512 x 106 take 1.26 ms instead of 0.85 (512 blocks of a volume: 272 us
// instead of 188; a 128^3 x 106 reconstruction at stride 4: 3 to 5 % of its iteration).
// Narrow matrices: up to 32, 16 and 8 columns the 128 tile rows hold S = 2, 4 and 8 row chunks side by side
// (2n <= 128 / S columns of D each), so a step covers 32 S rows; the S diagonal blocks of the accumulator
// are the chunks' own sums (the blocks off the diagonal are never read) and the epilogue adds them.
// With one chunk per step a step of 16 columns had two loads per thread in flight and took 2 us of latency.
// Rows stream in steps of S 32-row chunks, double-buffered, with the loads of the chunk two positions
// ahead (possibly of the CTA's next block) in flight: while the tensor core consumes one step's chunks
// the 8 warps gather, phase-correct and split the next ones.  One elected thread issues the
// MMAs and commits them to an mbarrier; every wait is bounded and reports a timeout through
// op.err instead of hanging.
// Tile rows beyond 2n hold whatever was there: row i and column j of the accumulator depend on tile rows i and j
// alone, and only those below 2n are read.
// Bound at 61 columns: the gather (48-byte runs of 6^3 blocks; 154 us of 290 remain without it) on top of the split's
// instruction issue and the shared memory that MMAs and stores share; MMA count hardly matters (one of three
// products less: 284 us).  32-bit block coordinates, the source's kind and phases as template arguments, one
// barrier per step, no re-zeroing: 192 x 192 x 96 x 61, 6^3 blocks 1244 -> 1181 us, 2048 contiguous blocks of
// 216 x 61 105 -> 90 us.  Chunks side by side: 512 blocks of 512 x 17
// 65.2 -> 44.3 us, 32 blocks of 512 x 9 29.9 -> 20.4 us.
#include <cstdio>
#include <algorithm>

#include "llr_prox_common.cuh"
#include "llr_umma.cuh"

namespace llr {

namespace {

constexpr int kKC = 32;                    // rows (K) per staged chunk
constexpr int kQT = 8;                     // volumes per warp per chunk (warps x kQT >= n)
constexpr int tc_warps(int npmax) { return npmax / kQT; }
constexpr int kOpBytes = 128 * kKC * 4;    // one operand plane (hi or lo) of one chunk
// Row table of one block: planar offset of every row and either the row's phase (uniform
// over the volumes) or its coordinates (per-volume phase).  The kernel keeps kRowBufs tables:
// the one of the block being converted and those of the blocks whose chunks are prefetched.
union TcRowAux {
  float2 ph;
  int2 c;              // x, y | z << 16
};

struct TcLayout {
  size_t off_hdr, off_row, off_aux, off_op, total;
  int op_bytes;        // bytes of the operand / P-staging region
  int nbuf;            // row tables: 2 (3 when a block is a single step)
};

struct TcHdr {
  unsigned long long mbar[3];   // chunk buffer 0, chunk buffer 1, block done
  unsigned int tmem;            // tensor-memory base address
  int shift[3];
  int fail;
  int pad;
};

// Instruction descriptor: TF32 x TF32 -> F32, both K-major, M = 128, N = 128.
constexpr uint32_t kIdesc = umma_idesc_tf32(128, 128);

// S: row chunks side by side in the tile; PH: 0 contiguous matrices, 1 planar volumes with one phase per row,
// 2 with a phase per row and volume.
template <int NPMAX, int S, int PH>
__global__ void __launch_bounds__(32 * tc_warps(NPMAX), NPMAX == 64 ? 3 : 1)
    llr_gram_tc_kernel(BlockSource src, ProxOp op, TcLayout L) {
  constexpr bool WIDE = NPMAX > 64;
  constexpr int kTcWarps = tc_warps(NPMAX), kTcThreads = 32 * kTcWarps;
  constexpr int kPlanes = WIDE ? 2 : 1;            // operand tiles per precision part (Re, Im)
  constexpr int kT = kQT / S;                      // volumes per warp
  static_assert(!WIDE || S == 1, "two operand tiles leave no room for chunks side by side");
  constexpr uint32_t kTmemCols = WIDE ? 512u : 128u;   // WIDE: one accumulator pair per operand buffer
  extern __shared__ __align__(1024) unsigned char smem[];
  TcHdr* hdr = reinterpret_cast<TcHdr*>(smem + L.off_hdr);
  int* row_off = reinterpret_cast<int*>(smem + L.off_row);        // [nbuf][m]
  TcRowAux* row_aux = reinterpret_cast<TcRowAux*>(smem + L.off_aux);   // [nbuf][m]
  unsigned char* ops = smem + L.off_op;   // [buf][hi, lo] planes; reused as P staging
  const int m = op.m, n = op.n, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long qstride = PH != 0 ? src.g.V : (long long)m;
  const int nsteps = (m + kKC * S - 1) / (kKC * S);
  const int nbuf = L.nbuf, la = nbuf - 1;   // row-table lookahead in blocks

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&hdr->tmem)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int b = 0; b < 3; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&hdr->mbar[b])));
    asm volatile("fence.mbarrier_init.release.cluster;");
    block_shift(src, hdr->shift);
    hdr->fail = 0;
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = hdr->tmem;
  const int sh[3] = {hdr->shift[0], hdr->shift[1], hdr->shift[2]};
  uint32_t phase[3] = {0u, 0u, 0u};
  bool used[2] = {false, false};
  bool failed = false;

  // Lane layout of the gather: lane = row of the chunk, warp w = volumes w, w + kTcWarps, ...: every
  // request reads 32 consecutive rows of one volume (the block's runs along y of one DRAM
  // page); requests that mix volumes, one short run each, reach a fraction of the HBM rate.
  // In shared memory the 32 lanes write one 128-byte swizzled row (all banks).
  // Chunks form one stream over the CTA's blocks; two register sets alternate, and after a
  // set is converted it is refilled with the chunk two positions ahead, so two chunks of
  // loads are in flight while the tensor core and the epilogue run.  WIDE, short of registers: one set, one step
  // ahead.
  float2 preA[kQT], preB[kQT];
  auto build_rows = [&](long long b, int buf) {
    if (PH == 0) return;
    int* ro = row_off + (size_t)buf * m;
    TcRowAux* ra = row_aux + (size_t)buf * m;
    for (int r = tid; r < m; r += kTcThreads) {
      int ix, iy, iz;
      block_row_coord(src, b, sh, r, ix, iy, iz);
      ro[r] = (int)planar_index(src.g, ix, iy, iz, 0);
      TcRowAux a;
      if (PH == 1) a.ph = phase_at(src.ph, src.g, 0, ix, iy, iz);
      else a.c = make_int2(ix, iy | (iz << 16));
      ra[r] = a;
    }
  };
  // rows past the block's end repeat its last row here and count as zero in the conversion
  auto load_step = [&](float2 (&pre)[kQT], int c, long long b, int buf) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int r = min((c * S + s) * kKC + lane, m - 1);
      const float2* p = src.data + (PH == 0 ? b * (long long)m * n + r : (long long)row_off[buf * m + r]) + warp * qstride;
#pragma unroll
      for (int t = 0; t < kT; ++t) {
        if (warp + kTcWarps * t < n) pre[s * kT + t] = *p;      // warp-uniform
        p += kTcWarps * qstride;
      }
    }
  };
  // the step `ahead` positions after (block iteration j, step c); false past the CTA's blocks
  auto locate = [&](long long blk, int j, int c, int ahead, long long& b2, int& j2, int& c2) {
    c2 = c + ahead;
    j2 = j;
    b2 = blk;
    while (c2 >= nsteps) { c2 -= nsteps; ++j2; b2 += gridDim.x; }
    return b2 < src.nblocks;
  };
  // one step: wait for its operand buffer, convert `pre` into it, refill `pre` two steps
  // ahead, hand the buffer to the tensor core
  int gpar = 0;
  // operand offsets of this thread's elements: row q = warp + kTcWarps t (and n + q, or the Im tile's
  // row q), column lane; adding 8 to a row leaves its swizzle phase and moves it one 1 KB atom on, so
  // op_offset(q + 8 t, lane) = op_offset(q, lane) + 1024 t, and chunk s starts 128 / S rows on
  static_assert(kTcWarps % 8 == 0 && (128 / S) % 8 == 0, "the step per t assumes rows a multiple of 8 apart");
  constexpr int kStepT = 1024 * (kTcWarps / 8), kStepS = 1024 * (128 / S / 8);
  const int oq0 = op_offset(warp, lane), oi0 = WIDE ? kOpBytes + oq0 : op_offset(n + warp, lane);
  // WIDE: this thread's row of the block's sums, R columns 32 g .. + 31 then Q columns 32 g .. + 31 (g = warp / 4); a step's
  // accumulators are added here in FP32
  float sums[WIDE ? 64 : 1];
  auto take = [&](int b) {
    if constexpr (WIDE) {
      if (32 * (warp >> 2) >= n) return;   // warp-uniform
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        uint32_t r[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(tmem + ((uint32_t)(32 * (warp & 3)) << 16) +
                  (uint32_t)(256 * b + 128 * (h >> 1) + 32 * (warp >> 2) + 16 * (h & 1))));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int k = 0; k < 16; ++k) sums[16 * h + k] += __uint_as_float(r[k]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
    }
  };
  auto step = [&](float2 (&pre)[kQT], long long blk, int j, int c) {
    const int b = gpar;
    if (used[b] && !failed) {  // the MMAs that read this buffer two steps ago must be done
      failed = !mbar_wait(smem_u32(&hdr->mbar[b]), phase[b]);
      phase[b] ^= 1u;
      if constexpr (WIDE)
        if (__all_sync(0xffffffffu, !failed)) take(b);
    }
    unsigned char* hi = ops + (size_t)b * 2 * kPlanes * kOpBytes;
    unsigned char* lo = hi + kPlanes * kOpBytes;
    const TcRowAux* ra = row_aux + (j % nbuf) * m;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int r = (c * S + s) * kKC + lane;
      const bool in = r < m;
      const TcRowAux aux = PH == 0 ? TcRowAux{} : ra[min(r, m - 1)];
      const float rowsc = in ? src.load_scale : 0.f;
#pragma unroll
      for (int t = 0; t < kT; ++t) {
        const int q = warp + kTcWarps * t;
        if (q >= n) break;                              // warp-uniform
        float2 x = pre[s * kT + t];
        if (PH == 0) x = in ? x : make_float2(0.f, 0.f);
        if (PH == 1) x = cscale(cmul_bc(x, aux.ph), rowsc);
        if (PH == 2) x = cscale(cmul_bc(x, phase_at(src.ph, src.g, q, aux.c.x, aux.c.y & 0xffff, aux.c.y >> 16)), rowsc);
        const uint32_t a = tf32_rna(x.x), bb = tf32_rna(x.y);
        const int oq = oq0 + kStepT * t + kStepS * s, oi = oi0 + kStepT * t + kStepS * s;
        *reinterpret_cast<uint32_t*>(hi + oq) = a;
        *reinterpret_cast<uint32_t*>(hi + oi) = bb;
        *reinterpret_cast<uint32_t*>(lo + oq) = __float_as_uint(x.x - __uint_as_float(a));
        *reinterpret_cast<uint32_t*>(lo + oi) = __float_as_uint(x.y - __uint_as_float(bb));
      }
    }
    {
      long long b2;
      int j2, c2;
      if (locate(blk, j, c, WIDE ? 1 : 2, b2, j2, c2)) load_step(pre, c2, b2, j2 % nbuf);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (warp == 0) {   // the whole warp, one lane issuing
      const uint32_t leader = elect_one();
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint64_t d0 = umma_desc_sw128(smem_u32(hi));
      const uint32_t h0 = (uint32_t)d0, dw = (uint32_t)(d0 >> 32);
      constexpr uint32_t kLo = kPlanes * kOpBytes / 16, kIm = kOpBytes / 16;   // descriptors count 16 bytes
      if constexpr (WIDE) {   // the products with a low part first: the small sums lose nothing to truncation
        const uint32_t d = tmem + 256u * (uint32_t)b;
#pragma unroll
        for (int s = 0; s < kKC / 8; ++s) {
          const uint32_t dh = h0 + 2 * s, dl = dh + kLo, ih = dh + kIm, il = dl + kIm;
          umma_tf32_by(leader, d, dh, dl, dw, kIdesc, s > 0 ? 1u : 0u);
          umma_tf32_by(leader, d, dl, dh, dw, kIdesc, 1u);
          umma_tf32_by(leader, d, ih, il, dw, kIdesc, 1u);
          umma_tf32_by(leader, d, il, ih, dw, kIdesc, 1u);
          umma_tf32_by(leader, d + 128, dh, il, dw, kIdesc, s > 0 ? 1u : 0u);
          umma_tf32_by(leader, d + 128, dl, ih, dw, kIdesc, 1u);
        }
#pragma unroll
        for (int s = 0; s < kKC / 8; ++s) {
          const uint32_t dh = h0 + 2 * s, ih = dh + kIm;
          umma_tf32_by(leader, d, dh, dh, dw, kIdesc, 1u);
          umma_tf32_by(leader, d, ih, ih, dw, kIdesc, 1u);
          umma_tf32_by(leader, d + 128, dh, ih, dw, kIdesc, 1u);
        }
      } else {
#pragma unroll
        for (int s = 0; s < kKC / 8; ++s) {
          const uint32_t dh = h0 + 2 * s, dl = dh + kLo;
          const uint32_t acc = (c > 0 || s > 0) ? 1u : 0u;
          umma_tf32_by(leader, tmem, dh, dh, dw, kIdesc, acc);
          umma_tf32_by(leader, tmem, dh, dl, dw, kIdesc, 1u);
          umma_tf32_by(leader, tmem, dl, dh, dw, kIdesc, 1u);
        }
      }
      umma_commit_by(leader, smem_u32(&hdr->mbar[b]));
      if (c == nsteps - 1) umma_commit_by(leader, smem_u32(&hdr->mbar[2]));
    }
    used[b] = true;
    gpar ^= 1;
  };

  long long blk = blockIdx.x;
  if (blk < src.nblocks) {
    for (int jj = 0; jj <= la; ++jj)
      if (blk + (long long)jj * gridDim.x < src.nblocks) build_rows(blk + (long long)jj * gridDim.x, jj % nbuf);
    __syncthreads();
    long long b2;
    int j2, c2;
    if (locate(blk, 0, 0, 0, b2, j2, c2)) load_step(preA, c2, b2, j2 % nbuf);
    if (!WIDE && locate(blk, 0, 0, 1, b2, j2, c2)) load_step(preB, c2, b2, j2 % nbuf);
  }

  for (int j = 0; blk < src.nblocks && !failed; blk += gridDim.x, ++j) {
    if (j > 0) {   // (the barrier also ends the reads of the staged accumulator) the table of the block `la` ahead goes into the buffer the previous block freed
      const long long bl = blk + (long long)la * gridDim.x;
      if (bl < src.nblocks) build_rows(bl, (j + la) % nbuf);
      __syncthreads();
    }
    if constexpr (WIDE) {
      gpar = 0;   // both buffers are free: a block's partial sums are added in the same order wherever it comes
#pragma unroll
      for (int k = 0; k < 64; ++k) sums[k] = 0.f;
    }
    for (int c = 0; c < nsteps; ++c) {
      if (gpar == 0) step(preA, blk, j, c);
      else if (WIDE) step(preA, blk, j, c);
      else step(preB, blk, j, c);
    }
    // all MMAs of this block complete -> read P and stage it in the (now idle) operand area
    if (!failed) failed = !mbar_wait(smem_u32(&hdr->mbar[2]), phase[2]);
    phase[2] ^= 1u;
    // the done barrier implies every step barrier's MMAs finished too; consume them, the older step's first
    auto consume = [&](int bb) {
      if (!used[bb]) return;
      if (!failed) failed = !mbar_wait(smem_u32(&hdr->mbar[bb]), phase[bb]);
      phase[bb] ^= 1u;
      used[bb] = false;
      if constexpr (WIDE)
        if (__all_sync(0xffffffffu, !failed)) take(bb);
    };
    if (WIDE && (nsteps & 1)) {
      consume(1);
      consume(0);
    } else {
      consume(0);
      consume(1);
    }
    failed = __syncthreads_or(failed);
    if (failed) break;
    asm volatile("tcgen05.fence::after_thread_sync;");
    float* Ps = reinterpret_cast<float*>(ops);
    // narrow: P (2n x 2n, its S diagonal blocks 128 / S rows apart), odd pitch; wide: R then Q (n x n each, odd pitch)
    constexpr int W = 128 / S;
    const int cols = WIDE ? n : 2 * n, ldp = cols | 1;
    // warp w reads TMEM lanes 32 (w mod 4) .. + 31 (its quadrant); the warps sharing a quadrant
    // split the 32-column chunks
    const int quad = warp & 3;
    const int a = 32 * quad + lane;          // accumulator row held by this thread
    if constexpr (WIDE) {
      const int cc = 32 * (warp >> 2);
      if (a < n && cc < n) {
#pragma unroll
        for (int k = 0; k < 64; ++k) {
          const int col = cc + (k & 31);
          if (col < n) Ps[(k < 32 ? (size_t)0 : (size_t)n * ldp) + a * ldp + col] = sums[k];
        }
      }
    } else
    for (int c2 = 32 * (warp >> 2); c2 < (int)kTmemCols; c2 += 32 * (kTcWarps / 4)) {
      // column within P's diagonal block; the tests are warp-uniform (S = 8: two blocks per 32 columns)
      if (S > 1 && (S == 8 ? c2 != 32 * quad : c2 / W != 32 * quad / W)) continue;
      const int cc = S == 8 ? -(lane & 16) : c2 & (W - 1);
      if (S < 8 && cc >= cols) continue;
      uint32_t r[32];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
          "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
            "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
            "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
            "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
          : "r"(tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)c2));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if ((a & (W - 1)) < cols) {
#pragma unroll
        for (int jj = 0; jj < 32; ++jj)
          if (cc + jj < cols && (S < 8 || cc + jj >= 0)) Ps[a * ldp + cc + jj] = __uint_as_float(r[jj]);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    // packed lower triangle by row pairs (i, n - 1 - i): n + 1 elements per pair, so a warp's
    // lanes stay busy; two elements per lane in flight
    float2* G = op.gram + blk * op.gram_stride;
    for (int i = warp; i < (n + 1) / 2; i += kTcThreads / 32) {
      const int i2 = n - 1 - i, len = i2 == i ? i + 1 : n + 1;
      for (int s0 = lane; s0 < len; s0 += 64) {
        float re[2], im[2];
        int row[2], col[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int s = min(s0 + 32 * u, len - 1);
          row[u] = s <= i ? i : i2;
          col[u] = s <= i ? s : s - i - 1;
          if (WIDE) {
            const float* Q = Ps + (size_t)n * ldp;
            re[u] = Ps[row[u] * ldp + col[u]];
            im[u] = Q[row[u] * ldp + col[u]] - Q[col[u] * ldp + row[u]];
          } else {
            re[u] = im[u] = 0.f;
#pragma unroll
            for (int k = 0; k < S; ++k) {
              const float* P = Ps + k * W * ldp;
              re[u] += P[row[u] * ldp + col[u]] + P[(n + row[u]) * ldp + n + col[u]];
              im[u] += P[row[u] * ldp + n + col[u]] - P[(n + row[u]) * ldp + col[u]];
            }
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (s0 + 32 * u < len) G[row[u] * (row[u] + 1) / 2 + col[u]] = make_float2(re[u], im[u]);
      }
    }
  }

  if (failed && tid == 0 && op.err) atomicExch(op.err, 1);
  // nothing may still write the accumulator when it is released: a commit covers the MMAs of its own thread
  if (warp == 0) umma_commit_by(elect_one(), smem_u32(&hdr->mbar[2]));
  mbar_wait(smem_u32(&hdr->mbar[2]), phase[2]);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

template <int NPMAX>
TcLayout make_tc_layout(int m, int n, int S) {
  TcLayout L;
  size_t off = 0;
  L.off_hdr = off; off = align16(off + sizeof(TcHdr));
  L.nbuf = m <= kKC * S ? 3 : 2;
  L.off_row = off; off = align16(off + sizeof(int) * (size_t)m * L.nbuf);
  L.off_aux = off; off = align16(off + sizeof(TcRowAux) * (size_t)m * L.nbuf);
  off = (off + 1023) & ~size_t(1023);
  L.off_op = off;
  const size_t stage = NPMAX > 64 ? 2 * (size_t)n * (n | 1) : (size_t)(128 - 128 / S + 2 * n) * (2 * n + 1);
  const size_t opb = std::max<size_t>((NPMAX > 64 ? 8 : 4) * (size_t)kOpBytes, sizeof(float) * stage);
  L.op_bytes = (int)opb;
  off += opb;
  L.total = off;
  return L;
}

// Chunks side by side change the order of the FP32 sums.  A soft threshold is a continuous map and carries that as
// is; a rank cut may fall between two nearly equal singular values, where the last bits of the Gram matrix
// turn the kept subspace (one in a few thousand blocks by 1e-3), so hard rank keeps one chunk per step.
int chunks_side_by_side(int n, bool soft) { return !soft ? 1 : n <= 8 ? 8 : n <= 16 ? 4 : n <= 32 ? 2 : 1; }

}  // namespace

bool llr_gram_tc_supported(int m, int n) {
  if (n < 1 || n > 128 || m < 1) return false;
  return (n <= 64 ? make_tc_layout<64>(m, n, 1) : make_tc_layout<128>(m, n, 1)).total <= 227 * 1024;
}

namespace {

template <int NPMAX, int S, int PH>
int launch_gram_instance(const BlockSource& src, const ProxOp& op, cudaStream_t stream) {
  constexpr int kTcThreads = 32 * tc_warps(NPMAX);
  TcLayout L = make_tc_layout<NPMAX>(op.m, op.n, S);
  if (L.total > 227 * 1024) return set_error(LLR_ERR_UNSUPPORTED, "tensor-core Gram needs %zu B smem", L.total);
  auto kern = llr_gram_tc_kernel<NPMAX, S, PH>;
  LLR_CUDA_TRY(allow_smem(kern));
  LLR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  int dev = 0, nsm = 0, smem_sm = 0, regs_sm = 0;
  LLR_CUDA_TRY(cudaGetDevice(&dev));
  LLR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  LLR_CUDA_TRY(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  LLR_CUDA_TRY(cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev));
  cudaFuncAttributes fa{};
  LLR_CUDA_TRY(cudaFuncGetAttributes(&fa, kern));
  // Residency from the kernel's own resources. The occupancy query reports one CTA per SM for
  // this kernel although three fit, so the count is derived here: shared memory (the driver
  // reserves 1 KB per CTA), registers (allocated per warp in units of 256) and TMEM (128 or all of
  // the SM's 512 columns per CTA). The kernel strides over blocks, so a grid larger than
  // what is resident is still correct, only slower.
  const int regs_warp = ((fa.numRegs * 32 + 255) / 256) * 256;
  const int by_regs = regs_warp > 0 ? regs_sm / (regs_warp * (kTcThreads / 32)) : 4;
  const int by_smem = smem_sm / (int)(L.total + fa.sharedSizeBytes + 1024);
  int occ = std::min(std::min(by_regs, by_smem), NPMAX > 64 ? 1 : 4);
  if (occ < 1) return set_error(LLR_ERR_UNSUPPORTED, "tensor-core Gram kernel cannot be resident");
  const long long grid = std::min<long long>(src.nblocks, (long long)nsm * occ);
  if (grid < 1) return LLR_OK;
  note_launch();
  kern<<<(unsigned)grid, kTcThreads, L.total, stream>>>(src, op, L);
  LLR_CUDA_TRY(cudaGetLastError());
  return LLR_OK;
}

template <int NPMAX, int S>
int launch_gram_source(const BlockSource& src, const ProxOp& op, cudaStream_t stream) {
  if (src.kind != 1) return launch_gram_instance<NPMAX, S, 0>(src, op, stream);
  return src.ph_uniform ? launch_gram_instance<NPMAX, S, 1>(src, op, stream)
                        : launch_gram_instance<NPMAX, S, 2>(src, op, stream);
}

}  // namespace

int launch_llr_gram_tc(const BlockSource& src, const ProxOp& op, cudaStream_t stream) {
  if (op.n > 128) return set_error(LLR_ERR_UNSUPPORTED, "tensor-core Gram needs n <= 128 (n = %d)", op.n);
  if (op.n > 64) return launch_gram_source<128, 1>(src, op, stream);
  switch (chunks_side_by_side(op.n, op.mode != LLR_PROX_HARD_RANK)) {
    case 8: return launch_gram_source<64, 8>(src, op, stream);
    case 4: return launch_gram_source<64, 4>(src, op, stream);
    case 2: return launch_gram_source<64, 2>(src, op, stream);
    default: return launch_gram_source<64, 1>(src, op, stream);
  }
}

}  // namespace llr

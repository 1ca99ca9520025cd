// band_lu_patch.cu -- many patches' FP32 linear solves in two launches.
//
// The batched FP32 form solves K Δu = -r for every patch of a batch with one
// CTA (or a small cluster) per patch: `patch_factor_kernel` factors each patch's
// FP32 band and `patch_refine_kernel` runs the FP32 substitutions and FP64
// iterative refinement x += K^-1 (r - A0 x) until the last correction is at most
// tol |x| -- the role of `K_gl \ r_gl` (FiniteElement.jl:38).  A single patch's
// LU is a chain of dependent panels; across a batch the chains are independent,
// so one CTA per patch keeps every SM busy without any inter-CTA
// synchronisation (the multi-CTA persistent kernel spends most of its SM time
// waiting on the chain, which pays only for one patch alone).
//
// The factors are kept in block form.  Per panel (columns [j0, j1), w <= 32 wide,
// whole node blocks) with A11 its diagonal block,
//   Ai = A11^-1,  Y = Ai A12,  A22 -= A21 Y;
// stored are Ai (job.inv), Y in place of A12 and the raw A21.  The
// substitutions are then z = Ai b1, b2 -= A21 z forward and x1 = z - Y x2
// backward: no triangle is ever solved, one 32 x 32 product per panel instead of
// three (L11^-1, U11^-1 and their product), and Y serves the trailing update and
// the back substitution alike.  Ai comes from one in-place Gauss-Jordan sweep
// by a warp with the pivot of column k searched among the rows of k's node block
// not yet used, the same pivots as a node-block pivoted LU; the refinement
// absorbs the explicit inverse's rounding.

#include <cuda_runtime.h>

#include <cstdint>

#include "band_lu_common.cuh"
#include "tcgen05.cuh"

namespace mafem {

// lambdas with register arrays: always inlined, so that the arrays stay in registers
#define MAFEM_INLINE __attribute__((always_inline))

constexpr int kPT = 512;   // threads per CTA of the factorisation (16 warps)
constexpr int kRT = 512;   // threads per CTA of the refinement (16 warps)
constexpr int kNCH = 256;  // trailing columns per chunk at most (the MMA's N <= 256)
constexpr int kMT = 128;   // rows of A22 per tensor-core tile (the MMA's M)
constexpr int kIS = 36;    // shared-memory row stride of the 32 x 32 inverse (16-byte rows)
// Y (the MMA's B operand, K-major core matrices): element (k, c) of a chunk at
// float (k / 4) * kYQuad + 4 c + k % 4, hi and lo parts in two such arrays; the
// k-quads are 16 bytes more than their size apart, so that a warp's 32 rows of
// one column fall into 32 banks
constexpr int kYQuad = 4 * kNCH + 4;
constexpr uint32_t kYPlane = 4u * kYQuad;               // bytes between k-quads (the LBO of B)
constexpr uint32_t kYBytes = 8u * kYPlane;              // one of Yh / Yl
constexpr uint32_t kATile = 8u * kMT * 16u;             // one of A21h / A21l per M tile: 16 KB
constexpr uint32_t kChunkBytes = 2 * kYBytes + 4 * kATile;  // Yh, Yl and two (A21h, A21l) tile buffers: 128 KB
static_assert(kYBytes % 128 == 0, "the TMA tile buffers follow Y on a 128-byte boundary");
constexpr uint32_t kTmemCols = 2 * kNCH;                // two FP32 accumulators of 128 x 256
// A factorisation CTA asks for more than half of an SM's shared memory, so no
// two of them share an SM and its Tensor Memory (each allocates all 512 columns).
constexpr size_t kFactorSmem = kChunkBytes + sizeof(float) * (kBlkW * kIS + 16 * 4 * kBlkW);
static_assert(kFactorSmem > 116 * 1024, "one factorisation CTA per SM");

size_t patch_factor_smem() { return kFactorSmem; }
// Rows of the split-A21 buffer per part (hi, lo) and rank: the most rows below
// a panel's diagonal block (kl), rounded up to whole M tiles.
int patch_a21_rows(int kl) { return (kl + kMT - 1) / kMT * kMT; }
size_t patch_a21_elems(int rows) { return (size_t)8 * 4 * 2 * rows * 4; }  // k-quads, ranks, parts, rows, k % 4

// x = hi + lo with hi, lo TF32 (round to nearest): the 3xTF32 split
__device__ __forceinline__ void split_tf32(float x, float& hi, float& lo) {
  unsigned h, l;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
  const float r = x - __uint_as_float(h);
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(r));
  hi = __uint_as_float(h);
  lo = __uint_as_float(l);
}

__device__ __forceinline__ void stamp(long long* tr, int slot) {
  if (tr && threadIdx.x == 0) {
    unsigned long long v;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v));
    tr[slot] = (long long)v;
  }
}

// all threads of every CTA of the cluster; orders each CTA's prior memory
// accesses (global included) before the others' later ones
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Bounded wait on an mbarrier phase: after kMbarPolls polls the wait gives up
// and records 1 in *err (the patch's wait-ran-out word); once that word is
// set every later wait gives up within 64 polls, so the kernel runs to its end
// quickly, and the host reports the failure.
constexpr int kMbarPolls = 1 << 20;
__device__ __forceinline__ void mbar_wait_bounded(uint64_t* bar, uint32_t& ph, int* err) {
  for (int it = 0; !mbar_try_wait(bar, ph); ++it)  // (the word is in global memory: a look at it delays the next poll)
    if (it > kMbarPolls || ((it & 63) == 63 && *(volatile int*)err)) {
      atomicExch(err, 1);
      break;
    }
  ph ^= 1u;
}

// Two FP32 FMAs in one instruction, each rounded as fmaf: (a, b) as 64-bit pairs.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rc, ra, rb, rc;\n\tmov.b64 {%0, %1}, rc;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// Inverse of the w x w block (row `lane` in S, zero beyond w) by one warp: a
// Gauss-Jordan sweep in place.  Step k exchanges column k for the pivot row p_k,
// picked by size (to 17 bits) among the rows of k's node block -- they end at row
// bend of position k -- not yet used; rows are never moved.  A row's scaling by
// -1/pivot at its own step is kept apart (sc), since the later steps' multipliers
// -S[k]/pivot do not see it: the step is 31 shuffles and 31 FMAs for every row
// alike.  Afterwards sc S of row p_k is row k of the inverse, its entry k'
// standing for the block's row p_k', and goes to Ai[row][column] (stride kIS)
// and, transposed, to inv.  The columns rotate through the registers, so that the
// pivot column is always S[0] and the step is one small loop body (unrolled over
// k it is 70 KB of code, which one warp fetches at 0.5 us a step): 6.4 us for a
// panel of 32 with the block's load, against 10.5 us for an eight-warp LU.
// Returns the first step (1-based) that found no usable pivot, 0 if none.
__device__ __forceinline__ int warp_inverse(float (&S)[32], int w, int bend, int* sp, float* Ai, float* inv) {
  const int lane = threadIdx.x & 31;
  unsigned mine = lane < w ? 1u : 0u;  // this row can still be a pivot
  int pos = lane, bad = 0;
  float sc = 1.0f;
  if (lane >= w) sp[lane] = lane;
  int bk = __shfl_sync(kFull, bend, 0);
#pragma unroll 1
  for (int k = 0; k < w; ++k) {
    const unsigned key = (mine && lane < bk) ? ((pkey(S[0]) & ~63u) | (63u - lane)) : 0u;
    bk = __shfl_sync(kFull, bend, (k + 1) & 31);
    const unsigned mx = __reduce_max_sync(kFull, key);  // the candidates are never empty
    const int p = 63 - (int)(mx & 63u);
    if (mx < 64u && bad == 0) bad = k + 1;
    const float d = __shfl_sync(kFull, S[0], p);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    r = fmaf(r, fmaf(-d, r, 1.0f), r);  // one Newton step on the hardware's approximation
    const bool own = lane == p;
    const float m = own ? 0.0f : -(S[0] * r);
    if (own) {
      pos = k;
      sc = -r;
      mine = 0u;
      sp[k] = p;
    }
#pragma unroll
    for (int c = 1; c < 32; ++c) S[c - 1] = fmaf(m, __shfl_sync(kFull, S[c], p), S[c]);
    S[31] = own ? -1.0f : -m;
  }
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 32; ++c) {  // S[c] holds column (c + w) mod 32
    const int col = sp[(c + w) & 31];
    const float v = sc * S[c];
    Ai[pos * kIS + col] = v;
    if (inv) inv[col * kBlkW + pos] = v;
  }
  return bad;
}

// trace (J.trace, optional): per panel 6 globaltimer stamps -- [0] start,
// [1] diagonal block inverted, [2] A21 split too, [3] Y of the first chunk,
// [4] its trailing update, [5] panel done
//
// Per panel: warp 0 inverts the diagonal block while the other warps split A21
// into TF32 hi / lo parts (it needs nothing from the inverse) and every warp has
// its first A12 columns in flight; then, per chunk of up to 256 trailing columns,
// Y = Ai A12 (a lane per row, four columns at a time, Ai's row in registers) and
// A22 -= A21 Y.
//
// NR > 1: a patch on a cluster of NR CTAs.  Every rank inverts the diagonal block
// and splits A21 for itself (into its own part of the split buffer) and updates
// the trailing chunks rank, rank + NR, ...: what a rank needs of the others'
// work is the band itself, so a panel has one cluster barrier, at its end.  All
// ranks run the same panel loop, so every barrier is reached by all threads of
// all CTAs.  Band reads go to L2 (ld.global.cg): a column moves between the
// ranks' chunks as the panels advance.
//
// The trailing update runs on the fifth-generation tensor cores: per 128-row
// tile of A22, 3 x 4 tcgen05.mma of kind::tf32 (the 3xTF32 split
// a b ~ al bh + ah bl + ah bh over K = 32 in steps of 8) accumulate A21 Y in
// Tensor Memory; the A21 tiles come by TMA (a 3-D tensor map over the patch's
// split-A21 buffer, written once per panel) into two shared-memory buffers, so
// the copy of tile t + 2 and the MMAs of tile t + 1 run while all 16 warps read
// tile t's accumulators back (tcgen05.ld) and write A22 - A21 Y to the band.  What
// bounds it is the band's round trip through L2: a warp has the next 16 columns'
// loads in flight while it subtracts the current ones.
// Measured on a GB300 against an LU with staged panels and per-rank hand-overs
// (three small triangular products per panel, 64-bit indexing in every access; it
// was bound by its instructions, 316 k per panel of 24 x 24 ALEVB): 16 x 16 ALEVB
// on four CTAs 3.3 -> 1.15 ms, 24 x 24 on one 12.5 -> 7.5 ms, 32 x 32 on one 31.4
// -> 20.3 ms, 48 x 48 on four 50.6 -> 27.0 ms.
template <int NR>
__global__ void __launch_bounds__(kPT, 1) patch_factor_kernel(const PatchJob* __restrict__ jobs,
                                                             const int* __restrict__ order) {
  const int rank = (int)(blockIdx.x % NR);
  const PatchJob& J = jobs[order[blockIdx.x / NR]];
  const BandLayout L = J.L;
  float* __restrict__ ab = J.band;
  extern __shared__ __align__(1024) unsigned char smem_fac[];
  float* Yh = reinterpret_cast<float*>(smem_fac);
  float* Yl = reinterpret_cast<float*>(smem_fac + kYBytes);
  unsigned char* Abuf = smem_fac + 2 * kYBytes;                       // [2][A21h tile | A21l tile]
  float* Ai = reinterpret_cast<float*>(smem_fac + kChunkBytes);       // [32][kIS]
  float* sA = Ai + kBlkW * kIS;                                       // [16 warps][4][32]: four columns of A12
  __shared__ int sp[32];
  __shared__ __align__(8) uint64_t bar_tma[2], bar_mma[2];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t ldm = L.ldb - 1;  // A(i, j + 1) - A(i, j) in the band array
  const int nrp = J.a21_rows;     // rows per part of the split-A21 buffer
  const int npan = J.npan, kuf = J.kuf;
  const int* __restrict__ ps = J.ps;
  float* a21 = J.a21 + (size_t)rank * 2 * nrp * 4;  // this rank's rows of every k-quad plane
  const size_t plane = (size_t)4 * 2 * nrp;         // float4 per k-quad plane (four ranks)
  int* err = J.info + 1;

  if (tid == 0) {
    mbar_init(&bar_tma[0], 1);
    mbar_init(&bar_tma[1], 1);
    mbar_init(&bar_mma[0], 1);
    mbar_init(&bar_mma[1], 1);
    mbar_init_fence();
  }
  if (warp == 0) {
    tc::tmem_alloc(&s_tmem, kTmemCols);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = s_tmem;
  uint32_t ph_tma[2] = {0u, 0u}, ph_mma[2] = {0u, 0u};  // phases (thread 0 uses ph_tma)
  float* sAw = sA + warp * 4 * kBlkW;

  int j1n = ps[1];
  for (int p = 0; p < npan; ++p) {
    const int64_t j0 = p ? (int64_t)ps[p] : 0, j1 = j1n;
    const int w = (int)(j1 - j0);
    j1n = p + 1 < npan ? ps[p + 2] : 0;
    const int R = (int)min64b(L.n - j0, (int64_t)w + L.kl);
    const int C = (int)(min64b(L.n, j1 + kuf) - j1);
    const int nr = R - w;
    const int ntile = (nr + kMT - 1) / kMT;
    // trailing columns [j1, j1 + C) in chunks of nch <= kNCH, balanced over the ranks
    const int cpr = (C + NR * kNCH - 1) / (NR * kNCH);  // chunks per rank
    const int nch = C > 0 ? ((C + NR * cpr - 1) / (NR * cpr) + 15) & ~15 : kNCH;
    long long* tr = J.trace ? J.trace + (size_t)p * 6 : nullptr;
    stamp(tr, 0);

    // this warp's columns of A12 in chunk cb: 4 (warp + 16 g) .. + 3, g < 4; a lane per row
    float a12[4][4];
    auto load_a12 = [&](int cb) {
      const int nc = min(nch, C - cb);
      const float* src = ab + bix(L, j0 + lane, j1 + cb);
#pragma unroll
      for (int g = 0; g < 4; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = 4 * (warp + 16 * g) + e;
          a12[g][e] = (c < nc && lane < w) ? __ldcg(src + (int64_t)c * ldm) : 0.0f;
        }
    };

    // 1. the diagonal block's inverse; A21 split
    if (warp == 0) {
      float S[32];
      const float* src = ab + bix(L, j0 + lane, j0);
#pragma unroll
      for (int c = 0; c < 32; ++c) S[c] = (lane < w && c < w) ? __ldcg(src + (int64_t)c * ldm) : 0.0f;
      const int bend = lane < w ? (int)(J.blk_end[j0 + lane] - j0) : 0;
      const int bad =
          warp_inverse(S, w, bend, sp, Ai, rank == 0 ? J.inv + (size_t)p * kBlkW * kBlkW : nullptr);
      if (rank == 0 && lane == 0 && bad) atomicCAS(J.info, 0, (int)(j0 + bad));
      load_a12(rank * nch);
    } else {
      load_a12(rank * nch);
      // A21 (rows w .. R-1 of the panel) split into TF32 hi / lo parts, written to
      // the rank's part of the split-A21 buffer as 8 k-quad planes [k/4][row][k%4]
      // (hi rows 0 .. nrp-1, lo rows nrp .. 2 nrp-1), rows past the panel and
      // columns k >= w zero
      for (int task = warp - 1; task < ntile * (kMT / 4); task += kPT / 32 - 1) {  // a k-quad of 32 rows
        const int kq = task & 7, r = (task >> 3) * 32 + lane;
        const float* src = ab + bix(L, j0 + w + min(r, nr - 1), j0 + 4 * kq);
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = 4 * kq + e < w ? __ldcg(src + e * ldm) : 0.0f;
        float4 h, l;
        const bool in = r < nr;
        split_tf32(in ? v[0] : 0.0f, h.x, l.x);
        split_tf32(in ? v[1] : 0.0f, h.y, l.y);
        split_tf32(in ? v[2] : 0.0f, h.z, l.z);
        split_tf32(in ? v[3] : 0.0f, h.w, l.w);
        float4* pl = reinterpret_cast<float4*>(a21) + kq * plane;
        pl[r] = h;
        pl[nrp + r] = l;
      }
      fence_proxy_async_global();  // read by TMA
    }
    stamp(tr, 1);
    __syncthreads();
    stamp(tr, 2);

    bool first = true;
    for (int cb = rank * nch; cb < C; cb += NR * nch) {
      const int nc = min(nch, C - cb);
      const int ncp = (nc + 15) & ~15;  // the MMA's N
      auto tma_tile = [&](int t) {      // thread 0: tile t's A21h and A21l into buffer t & 1
        const int b = t & 1, row = rank * 2 * nrp + t * kMT;
        mbar_arrive_expect_tx(&bar_tma[b], 2 * kATile);
        tc::tma_load_3d(Abuf + b * 2 * kATile, &J.a21_map, 0, row, 0, &bar_tma[b]);
        tc::tma_load_3d(Abuf + b * 2 * kATile + kATile, &J.a21_map, 0, nrp + row, 0, &bar_tma[b]);
      };
      if (tid == 0 && ntile > 0) {
        tma_tile(0);
        if (ntile > 1) tma_tile(1);
      }
      // Y = Ai A12, split into TF32 parts for the MMA and written over A12
      if (!first) load_a12(cb);
      {
        float ar[32];  // row `lane` of Ai
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float4 q = reinterpret_cast<const float4*>(Ai + lane * kIS)[k];
          ar[4 * k] = q.x, ar[4 * k + 1] = q.y, ar[4 * k + 2] = q.z, ar[4 * k + 3] = q.w;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int c = 4 * (warp + 16 * g);
          if (c < ncp) {  // warp-uniform
#pragma unroll
            for (int e = 0; e < 4; ++e) sAw[e * kBlkW + lane] = a12[g][e];
            __syncwarp();
            float y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float2 s0 = make_float2(0.0f, 0.0f), s1 = s0;
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const float4 q = reinterpret_cast<const float4*>(sAw + e * kBlkW)[k];
                s0 = fma2(make_float2(ar[4 * k], ar[4 * k + 1]), make_float2(q.x, q.y), s0);
                s1 = fma2(make_float2(ar[4 * k + 2], ar[4 * k + 3]), make_float2(q.z, q.w), s1);
              }
              y[e] = (s0.x + s0.y) + (s1.x + s1.y);
            }
            __syncwarp();
            float* dst = ab + bix(L, j0 + lane, j1 + cb + c);
            const int o = (lane >> 2) * kYQuad + 4 * c + (lane & 3);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float v = (lane < w && c + e < nc) ? y[e] : 0.0f;  // rows k >= w of Y: zero
              float yh, yl;
              split_tf32(v, yh, yl);
              Yh[o + 4 * e] = yh;
              Yl[o + 4 * e] = yl;
              if (lane < w && c + e < nc) dst[(int64_t)e * ldm] = y[e];
            }
          }
        }
      }
      fence_proxy_async_smem();  // Yh / Yl are read by the tensor cores
      __syncthreads();
      if (first) stamp(tr, 3);

      // A22 -= A21 Y, 128 rows at a time
      const uint32_t idesc = tc::idesc_tf32(kMT, ncp);
      const uint32_t yh = tc::saddr(Yh), yl = tc::saddr(Yl), a0 = tc::saddr(Abuf);
      const int ksteps = (w + 7) >> 3;
      auto mma_tile = [&](int t) {  // thread 0: tile t's products into accumulator t & 1
        const int b = t & 1;
        mbar_wait_bounded(&bar_tma[b], ph_tma[b], err);
        tc::fence_after();
        const uint32_t ah = a0 + b * 2 * kATile, al = ah + kATile, d = tmem + b * kNCH;
        for (int s = 0; s < ksteps; ++s) {  // k = 8 s .. 8 s + 7: k-quads 2 s and 2 s + 1
          const uint64_t dah = tc::smem_desc(ah + 2 * s * (kMT * 16), kMT * 16, 128);
          const uint64_t dal = tc::smem_desc(al + 2 * s * (kMT * 16), kMT * 16, 128);
          const uint64_t dbh = tc::smem_desc(yh + 2 * s * kYPlane, kYPlane, 128);
          const uint64_t dbl = tc::smem_desc(yl + 2 * s * kYPlane, kYPlane, 128);
          tc::mma_tf32(d, dal, dbh, idesc, s > 0 ? 1u : 0u);
          tc::mma_tf32(d, dah, dbl, idesc, 1u);
          tc::mma_tf32(d, dah, dbh, idesc, 1u);
        }
        tc::commit(&bar_mma[b]);
      };
      if (tid == 0 && ntile > 0) mma_tile(0);
      // epilogue roles: warp w reads lanes 32 (w % 4) .. + 31 (its rows) of
      // column group w / 4 (a quarter of the chunk, in multiples of 8 columns),
      // 16 columns at a time
      const int q = warp & 3, grp = warp >> 2;
      const int cpg = ((ncp >> 2) + 7) & ~7;
      const int cs = min(ncp, grp * cpg), ce = min(ncp, cs + cpg), lim = min(ce, nc);
      // the steps of this warp: tile t, columns c .. c + 15 of its group; the next
      // step's loads are issued after the current one's use (two steps ahead: +3 %
      // time, three: +10 %)
      auto next = [&](int& t, int& c) MAFEM_INLINE {
        c += 16;
        if (c >= lim) {
          c = cs;
          ++t;
        }
      };
      auto load_a22 = [&](float (&v)[16], int t, int c) MAFEM_INLINE {
        if (t >= ntile) return;  // warp-uniform
        const float* pa = ab + bix(L, j0 + min(w + t * kMT + 32 * q + lane, R - 1), j1 + cb + c);
        if (c + 16 <= lim) {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            v[k] = __ldcg(pa);
            pa += ldm;
          }
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            v[k] = c + k < lim ? __ldcg(pa) : 0.0f;
            pa += ldm;
          }
        }
      };
      auto tile_begin = [&](int t) MAFEM_INLINE {
        const int b = t & 1;
        mbar_wait_bounded(&bar_mma[b], ph_mma[b], err);  // tile t's products are in Tensor Memory
        if (tid == 0) {
          if (t + 2 < ntile) tma_tile(t + 2);  // buffer b is free: tile t's MMAs have completed
          if (t + 1 < ntile) mma_tile(t + 1);  // into the other accumulator, read back at t - 1
        }
        tc::fence_after();
      };
      auto tile_end = [&]() MAFEM_INLINE {
        tc::fence_before();
        __syncthreads();  // the accumulator is read before the MMAs of tile t + 2 overwrite it
      };
      if (cs < lim) {
        float va[16];
        int t = 0, c = cs;
        load_a22(va, t, c);
        while (t < ntile) {
          if (c == cs) tile_begin(t);
          const int row = w + t * kMT + 32 * q + lane;  // panel row of this thread
          const uint32_t dt = tmem + ((uint32_t)(32 * q) << 16) + (t & 1) * kNCH;
          float d0[8], d1[8];
          tc::ld8(dt + c, d0);
          if (c + 8 < ce) tc::ld8(dt + c + 8, d1);
          tc::wait_ld();
          if (row < R) {
            float* pa = ab + bix(L, j0 + row, j1 + cb + c);  // A(j0 + row, j1 + cb + c), + ldm: the next column
            if (c + 16 <= lim) {
#pragma unroll
              for (int k = 0; k < 16; ++k) {
                *pa = va[k] - (k < 8 ? d0[k] : d1[k - 8]);
                pa += ldm;
              }
            } else {
#pragma unroll
              for (int k = 0; k < 16; ++k) {
                if (c + k < lim) *pa = va[k] - (k < 8 ? d0[k] : d1[k - 8]);
                pa += ldm;
              }
            }
          }
          const bool last = c + 16 >= lim;
          next(t, c);
          load_a22(va, t, c);
          if (last) tile_end();
        }
      } else {  // no columns for this warp: the tiles' barriers only
        for (int t = 0; t < ntile; ++t) {
          tile_begin(t);
          tile_end();
        }
      }
      if (first) stamp(tr, 4);
      first = false;
    }
    if (NR > 1) cluster_sync();
    else __syncthreads();
    stamp(tr, 5);
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (warp == 0) tc::tmem_dealloc(tmem, kTmemCols);
}

// ---------------------------------------------------------------------------
// Solve + refinement, one CTA per patch.  The FP32 working vector lives in
// shared memory; x and the FP64 residual in global memory.

__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  for (int q = 0; q < kRT / 32; ++q) s += red[q];  // same order in every thread
  return s;
}

// 16-byte global -> shared copy, L2 only (16-byte aligned addresses)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}

constexpr int kTraceSweeps = 32;  // sweeps the refinement trace records
constexpr int kRing = 4;          // panels whose critical blocks are staged ahead
constexpr int kRowT = kRT - 32;   // rows (columns) the update warps hold per register set
struct RefineSmem {
  float ring[kRing][2][kBlkW * kBlkW];  // forward: A21's rows of the next panel, the next panel's Ai; backward: Y's columns
  float zb[2][kBlkW];                   // z of the current panel, by parity
  float bb[kBlkW];
  alignas(16) float part[2][kRT / 32][kBlkW];  // backward: the update warps' sums, by parity
  double red[kRT / 32];
};
static size_t refine_smem_base(int npan) { return sizeof(RefineSmem) + sizeof(int) * ((size_t)npan + 1); }
bool patch_vector_fits(int64_t n, int npan, int dyn) {
  return refine_smem_base(npan) + sizeof(float) * (size_t)n <= (size_t)dyn;
}
size_t patch_refine_smem(int64_t n, int npan, int dyn) {
  return refine_smem_base(npan) + (patch_vector_fits(n, npan, dyn) ? sizeof(float) * (size_t)n : 0);
}

__device__ __forceinline__ long long gtime() {
  unsigned long long v;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v));
  return (long long)v;
}

// sum_k m[k * 32 + lane] x[k]: a 32 x 32 block (column-major) times a vector, both in shared memory
__device__ __forceinline__ float block_times(const float* m, const float* x) {
  const int lane = threadIdx.x & 31;
  float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float4 q = reinterpret_cast<const float4*>(x)[k];
    s[0] = fmaf(m[(4 * k) * 32 + lane], q.x, s[0]);
    s[1] = fmaf(m[(4 * k + 1) * 32 + lane], q.y, s[1]);
    s[2] = fmaf(m[(4 * k + 2) * 32 + lane], q.z, s[2]);
    s[3] = fmaf(m[(4 * k + 3) * 32 + lane], q.w, s[3]);
  }
  return (s[0] + s[1]) + (s[2] + s[3]);
}

// v <- K^-1 v with the block factors.  Warp 0 runs the chain: per panel of the
// forward pass it finishes the next panel's rows (b1 = v - A21 z there), forms
// z = Ai b1 and publishes it; the other 15 warps subtract A21 z from the rows
// below (32 rows a warp), one step behind.  Backward: x1 = z - Y x2, the chain
// with the columns of the panel solved last, the others with the columns beyond
// (a run of columns per warp), one panel ahead of it.  One barrier per panel.  The
// blocks of the chain come through a ring of cp.async copies kRing - 1 panels
// ahead; the update warps hold their rows (columns) in registers, loaded ahead:
// with RPT = 1 two panels ahead (bands up to 480 rows below the next panel), with
// RPT = 2 two sets, one panel ahead; wider bands read the rest on the spot.  Bound:
// the chain's two 32 x 32 products and the barrier, and the update warps'
// instructions, one load per 32 entries.
// Measured on a GB300, one forward and backward pass, against whole-CTA steps with
// three small products and three barriers per panel: 16 x 16 ALEVB (70 panels) 666
// -> 150 us, 32 x 32 3.13 -> 1.07 ms, 48 x 48 (RPT = 2) 10.7 -> 3.06 ms; 116 us,
// 0.83 and 2.37 ms in a kernel without the residual, whose registers had made this
// pass spill.
// prof (trace mode, optional): [0] forward, [1] backward time of warp 0 in ns.
__device__ __forceinline__ void solve_barrier() { bar_sync_n(1, kRT); }
// dot product of 32 register values with 32 values in shared memory (16-byte aligned)
__device__ __forceinline__ float dot32(const float (&x)[32], const float* z) {
  float2 s0 = make_float2(0.0f, 0.0f), s1 = s0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float4 q = reinterpret_cast<const float4*>(z)[k];
    s0 = fma2(make_float2(x[4 * k], x[4 * k + 1]), make_float2(q.x, q.y), s0);
    s1 = fma2(make_float2(x[4 * k + 2], x[4 * k + 3]), make_float2(q.z, q.w), s1);
  }
  return (s0.x + s0.y) + (s1.x + s1.y);
}
template <int RPT>
__device__ __forceinline__ void patch_solve_pass(const PatchJob& J, float* v, const int* ps, RefineSmem& S,
                                                 long long* prof) {
  constexpr int NB = 3 - RPT;          // panels in flight in registers
  constexpr int kUW = kRT / 32 - 1;    // update warps
  const float* __restrict__ ab = J.band;
  const float* __restrict__ invs = J.inv;
  const int ldm = (int)J.L.ldb - 1, n = (int)J.L.n, off = (int)J.L.off;
  const int lane = threadIdx.x & 31, cw = (int)(threadIdx.x >> 5) - 1;
  const int npan = J.npan, kuf = J.kuf, kl = J.L.kl;
  auto at = [&](int i, int j) MAFEM_INLINE { return ab + ((int64_t)j * ldm + off + i); };  // A(i, j)

  if (cw < 0) {  // ---- warp 0: the chain
    const long long t0 = prof ? gtime() : 0;
    {
      const int w = ps[1];
      const float b = lane < w ? v[lane] : 0.0f;
      float z = 0.0f;
#pragma unroll
      for (int k = 0; k < 32; ++k) z = fmaf(__ldcg(invs + k * 32 + lane), __shfl_sync(kFull, b, k), z);
      S.zb[0][lane] = lane < w ? z : 0.0f;
      if (lane < w) v[lane] = z;
    }
    int j1 = ps[1];
#pragma unroll 1
    for (int p = 0; p + 1 < npan; ++p) {
      const int j2 = ps[p + 2], wn = j2 - j1;
      solve_barrier();  // ring slot p; the updates by panel p - 1
      const float b = (lane < wn ? v[j1 + lane] : 0.0f) - block_times(S.ring[p % kRing][0], S.zb[p & 1]);
      S.bb[lane] = lane < wn ? b : 0.0f;
      __syncwarp();
      const float z = block_times(S.ring[p % kRing][1], S.bb);
      S.zb[(p + 1) & 1][lane] = lane < wn ? z : 0.0f;
      if (lane < wn) v[j1 + lane] = z;
      __syncwarp();
      j1 = j2;
    }
    solve_barrier();
    const long long t1 = prof ? gtime() : 0;
    solve_barrier();  // the last panel's sums
#pragma unroll 1
    for (int p = npan - 1; p >= 0; --p) {
      const int j0 = ps[p], w = ps[p + 1] - j0;
      float s = p + 1 < npan ? block_times(S.ring[p % kRing][0], S.bb) : 0.0f;
      float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int k = 0; k < kUW; ++k) a[k & 3] += S.part[p & 1][k][lane];
      const float x = (lane < w ? v[j0 + lane] : 0.0f) - (s + ((a[0] + a[1]) + (a[2] + a[3])));
      __syncwarp();  // bb is read before it is overwritten
      S.bb[lane] = lane < w ? x : 0.0f;
      if (lane < w) v[j0 + lane] = x;
      solve_barrier();
    }
    if (prof && lane == 0) {
      prof[0] += t1 - t0;
      prof[1] += gtime() - t1;
    }
    return;
  }

  // ---- the update warps
  float t[2][32];
  // ring slot p: A21 of panel p in panel p + 1's rows (a warp per column), Ai of panel p + 1
  auto stage_fwd = [&](int p) MAFEM_INLINE {
    if (p + 1 < npan) {
      const int j0 = ps[p], j1 = ps[p + 1], w = j1 - j0, lim = min(ps[p + 2] - j1, kl);
      float* T = S.ring[p % kRing][0];
      for (int c = cw; c < kBlkW; c += kUW) {  // (columns c >= w meet zeros of z: they must be finite)
        if (lane < lim && c < w) cp_async(T + c * 32 + lane, at(j1 + lane, j0 + c));
        else T[c * 32 + lane] = 0.0f;
      }
      if (cw < 8)
        cp_async16(S.ring[p % kRing][1] + 128 * cw + 4 * lane, invs + (size_t)(p + 1) * kBlkW * kBlkW + 128 * cw + 4 * lane);
    }
    cp_async_commit();
  };
  // this warp's 32 rows of panel p's A21 below panel p + 1: set q starts at row0 + 32 (cw + 15 q)
  auto row0 = [&](int p) MAFEM_INLINE { return (p + 1 < npan ? ps[p + 2] : n) + 32 * cw; };
  auto load_rows = [&](int p, float (&x)[32], int q) MAFEM_INLINE {
    if (p >= npan) return;
    const int j0 = ps[p], w = ps[p + 1] - j0, rend = min(n, ps[p + 1] + kl), i0 = row0(p) + 32 * kUW * q;
    if (i0 >= rend) return;  // warp-uniform
    const float* a = at(min(i0 + lane, rend - 1), j0);
    if (w == 32) {
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        x[k] = __ldcg(a);
        a += ldm;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        x[k] = k < w ? __ldcg(a) : 0.0f;
        a += ldm;
      }
    }
  };
  auto use_rows = [&](int p, const float (&x)[32], int q) MAFEM_INLINE {
    const int rend = min(n, ps[p + 1] + kl), i0 = row0(p) + 32 * kUW * q;
    if (i0 >= rend) return;
    const float s = dot32(x, S.zb[p & 1]);
    if (i0 + lane < rend) v[i0 + lane] -= s;
  };
  auto far_rows = [&](int p) MAFEM_INLINE {  // rows beyond the registers' reach
    const int j0 = ps[p], w = ps[p + 1] - j0, rend = min(n, ps[p + 1] + kl);
    for (int i = row0(p) + 32 * kUW * RPT + lane; i < rend; i += 32 * kUW) {
      const float* a = at(i, j0);
      float s = 0.0f;
#pragma unroll 8
      for (int k = 0; k < w; ++k) s = fmaf(__ldcg(a + (int64_t)k * ldm), S.zb[p & 1][k], s);
      v[i] -= s;
    }
  };
  for (int p = 0; p < kRing - 1; ++p) stage_fwd(p);
  load_rows(0, t[0], 0);
  if constexpr (RPT == 1) load_rows(1, t[1], 0);
  else load_rows(0, t[1], 1);
  auto fwd_step = [&](int p, float (&x0)[32], float (&x1)[32]) MAFEM_INLINE {
    cp_async_wait_group<kRing - 2>();  // ring slot p (this thread's part)
    solve_barrier();                   // z of panel p; the updates by panel p - 1
    stage_fwd(p + kRing - 1);
    use_rows(p, x0, 0);
    load_rows(p + NB, x0, 0);
    if constexpr (RPT == 2) {
      use_rows(p, x1, 1);
      load_rows(p + NB, x1, 1);
      far_rows(p);
    }
  };
#pragma unroll 1
  for (int p = 0; p < npan; p += NB) {
    fwd_step(p, t[0], t[1]);
    if (NB == 2 && p + 1 < npan) fwd_step(p + 1, t[1], t[0]);
  }
  cp_async_wait_group<0>();
  // backward.  Ring slot p: Y of panel p in panel p + 1's columns
  auto stage_bwd = [&](int p) MAFEM_INLINE {
    if (p >= 0 && p + 1 < npan) {
      const int j0 = ps[p], j1 = ps[p + 1], w = j1 - j0, lim = min(ps[p + 2] - j1, kuf);
      float* T = S.ring[p % kRing][0];
      for (int c = cw; c < kBlkW; c += kUW) {
        if (lane < w && c < lim) cp_async(T + c * 32 + lane, at(j0 + lane, j1 + c));
        else T[c * 32 + lane] = 0.0f;
      }
    }
    cp_async_commit();
  };
  // this warp's run of columns of panel p's Y beyond panel p + 1: `len` columns from first
  struct Run {
    int first, len;
  };
  auto run_of = [&](int p) MAFEM_INLINE {
    const int c0 = p + 1 < npan ? ps[p + 2] : n, end = min(n, ps[p + 1] + kuf);
    const int len = max(0, (end - c0 + kUW - 1) / kUW), first = c0 + cw * len;
    return Run{first, max(0, min(len, end - first))};
  };
  auto load_cols = [&](int p, float (&x)[32], int q) MAFEM_INLINE {
    if (p < 0) return;
    const Run r = run_of(p);
    const int j0 = ps[p], w = ps[p + 1] - j0;
    const float* a = at(j0 + min(lane, w - 1), r.first + 32 * q);
#pragma unroll
    for (int m0 = 0; m0 < 32; m0 += 8) {
      if (32 * q + m0 >= r.len) break;  // warp-uniform
#pragma unroll
      for (int m = m0; m < m0 + 8; ++m) {
        x[m] = 32 * q + m < r.len ? __ldcg(a) : 0.0f;
        a += ldm;
      }
    }
  };
  auto use_cols = [&](int p, const float (&x)[32], int q) MAFEM_INLINE {
    const Run r = run_of(p);
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const float* vx = v + r.first + 32 * q;
#pragma unroll
    for (int m0 = 0; m0 < 32; m0 += 8) {
      if (32 * q + m0 >= r.len) break;
#pragma unroll
      for (int m = m0; m < m0 + 8; ++m) s[m & 3] = fmaf(x[m], 32 * q + m < r.len ? vx[m] : 0.0f, s[m & 3]);
    }
    return (s[0] + s[1]) + (s[2] + s[3]);
  };
  auto far_cols = [&](int p) MAFEM_INLINE {
    const Run r = run_of(p);
    const int j0 = ps[p], w = ps[p + 1] - j0;
    const float* a = at(j0 + min(lane, w - 1), r.first);
    float s = 0.0f;
#pragma unroll 8
    for (int m = 32 * RPT; m < r.len; ++m) s = fmaf(__ldcg(a + (int64_t)m * ldm), v[r.first + m], s);
    return s;
  };
  for (int k = 0; k < kRing - 1; ++k) stage_bwd(npan - 1 - k);
  load_cols(npan - 1, t[0], 0);
  if constexpr (RPT == 1) load_cols(npan - 2, t[1], 0);
  else load_cols(npan - 1, t[1], 1);
  // step p: the sums of panel p's far columns while warp 0 solves panel p + 1
  auto bwd_step = [&](int p, float (&x0)[32], float (&x1)[32]) MAFEM_INLINE {
    float s = use_cols(p, x0, 0);
    if constexpr (RPT == 2) s += use_cols(p, x1, 1) + far_cols(p);
    S.part[p & 1][cw][lane] = s;
    load_cols(p - NB, x0, 0);
    if constexpr (RPT == 2) load_cols(p - NB, x1, 1);
    cp_async_wait_group<kRing - 2>();  // ring slot p
    solve_barrier();
    stage_bwd(p - (kRing - 1));
  };
#pragma unroll 1
  for (int p = npan - 1; p >= 0; p -= NB) {
    bwd_step(p, t[0], t[1]);
    if (NB == 2 && p - 1 >= 0) bwd_step(p - 1, t[1], t[0]);
  }
  solve_barrier();  // x of panel 0
  cp_async_wait_group<0>();
}

// One column run [j0, j1) of a warp's double-float row sums (see patch_residual).
__device__ __forceinline__ void residual_run(const float* a, int64_t ldm, const float2* xs, int64_t j0, int64_t j1,
                                             float& sh, float& sl) {
  constexpr int kB = 16;  // columns whose loads, of A0 and of x, are in flight together
  for (int64_t j = j0; j < j1; j += kB) {
    const int cnt = (int)min64b(kB, j1 - j);  // warp-uniform
    float av[kB];
    const float* p = a + j * ldm;
#pragma unroll
    for (int m = 0; m < kB; ++m) {
      av[m] = m < cnt ? p[0] : 0.0f;
      p += ldm;
    }
#pragma unroll
    for (int m = 0; m < kB; ++m) {
      if (m >= cnt) break;
      const float2 xv = xs[j + m];
      // explicit roundings: a contraction of p into t would break TwoSum
      const float p = __fmul_rn(av[m], xv.x);
      const float e = fmaf(av[m], xv.y, fmaf(av[m], xv.x, -p));
      const float t = __fadd_rn(sh, p);
      const float z = __fsub_rn(t, sh);
      sl = __fadd_rn(sl, __fadd_rn(__fadd_rn(__fsub_rn(sh, __fsub_rn(t, z)), __fsub_rn(p, z)), e));
      sh = t;
    }
  }
}

// res = rhs - A0 x (A0: the unfactored FP32 band); returns |res|.  The
// products are formed on the FP32 pipe in double-float arithmetic: x = xh + xl
// (two floats, split once per sweep), a xh = p + e exactly (FMA), and the row
// sum kept as an unevaluated float pair (Knuth's TwoSum for the high part);
// the pair's error (~2^-44 of the row's term magnitudes) is far below the
// refinement tolerance, at a sixth of the cost of FP64 FMAs on this GPU.
// A warp takes 32 rows and walks, in increasing order, only the columns their
// control points couple to: an unknown of control point (s1, s2) couples only
// to the unknowns of points (s1 +- 2, s2 +- 2) (biquadratic elements).  The
// rows' points run from (s1a, s2a) to (s1b, s2b) in lexicographic order, so
// grid row g is coupled to points [s1a - 2, W) through the points of grid row
// s2a (if |g - s2a| <= 2), to [0, s1b + 2] through those of grid row s2b (if
// |g - s2b| <= 2), and to the whole grid row through any grid row between
// them: at most two runs per grid row.  The columns skipped hold stored
// zeros, whose products leave the pair unchanged: the sums equal a walk of
// the whole band window.
// The 32-row blocks w0, w0 + nw, ... of a warp; the squares of the k-th one's entries go to ss[k mod NS].
template <int NS>
__device__ __forceinline__ void residual_rows(const PatchJob& J, const float2* xs, int w0, int nw, double (&ss)[NS]) {
  const BandLayout L = J.L;
  const int lane = threadIdx.x & 31;
  const int64_t ldm = L.ldb - 1;
#pragma unroll
  for (int u = 0; u < NS; ++u) ss[u] = 0.0;
  int k = 0;
  // With nb >= 32 every (i, j) of the band window [rb - ku, rb + 32 + kl) lies
  // inside the band's storage, where the entries outside the band are stored
  // zeros, so A0(i, j) = a[j * ldm + lane] with a at row rb of column 0 needs
  // no guard but i < n; the runs are clipped to that window.
  for (int64_t rb = (int64_t)w0 * 32; rb < L.n; rb += (int64_t)nw * 32, ++k) {
    const int64_t i = rb + lane;
    const bool live = i < L.n;
    const int64_t jlo = rb - L.ku > 0 ? rb - L.ku : 0;
    const int64_t jhi = min64b(L.n, rb + 32 + L.kl);
    const float* a = J.band0 + L.off + (live ? i : rb);  // + j * ldm: A0(i, j)
    float sh = 0.0f, sl = 0.0f;
    if (J.node_first) {
      const int W = J.num1np, H = J.num2np;
      const int na = J.unk_node[rb], nb = J.unk_node[min64b(rb + 31, L.n - 1)];
      const int s1a = na % W, s2a = na / W, s1b = nb % W, s2b = nb / W;
      for (int g = max(s2a - 2, 0); g <= min(s2b + 2, H - 1); ++g) {
        // the runs [c0, c1] (and [d0, d1] after it) of grid row g, in points
        int c0 = 0, c1 = -1, d0 = 0, d1 = -1;
        const bool fa = abs(g - s2a) <= 2, fb = abs(g - s2b) <= 2;
        const bool fm = s2b - s2a >= 2 && g >= s2a - 1 && g <= s2b + 1;  // a grid row strictly between
        if (s2a == s2b) {
          c0 = max(s1a - 2, 0);
          c1 = min(s1b + 2, W - 1);
        } else if (fm || (fa && fb && s1b + 3 >= s1a - 2)) {
          c1 = W - 1;
        } else {
          if (fb) c1 = min(s1b + 2, W - 1);  // [0, s1b + 2] comes first
          if (fa) {
            d0 = max(s1a - 2, 0);
            d1 = W - 1;
          }
        }
        for (int r = 0; r < 2; ++r) {
          const int e0 = r ? d0 : c0, e1 = r ? d1 : c1;
          if (e1 < e0) continue;
          const int64_t j0 = max((int64_t)J.node_first[g * W + e0], jlo);
          const int64_t j1 = min64b((int64_t)J.node_first[g * W + e1 + 1], jhi);
          if (j0 < j1) residual_run(a, ldm, xs, j0, j1, sh, sl);
        }
      }
    } else {
      residual_run(a, ldm, xs, jlo, jhi, sh, sl);
    }
    if (live) {
      const double r = J.rhs[i] - ((double)sh + (double)sl);
      J.res[i] = r;
#pragma unroll
      for (int u = 0; u < NS; ++u)
        if (NS == 1 || k % NS == u) ss[u] = fma(r, r, ss[u]);
    }
  }
}
// The residual after a sweep on kResC CTAs per patch: partial sums of its squares to J.rs + 8.
constexpr int kResC = 8, kResT = 256;
__global__ void __launch_bounds__(kResT) patch_residual_kernel(const PatchJob* __restrict__ jobs,
                                                              const int* __restrict__ order) {
  const PatchJob& J = jobs[order[blockIdx.x / kResC]];
  const int c = blockIdx.x % kResC;
  if (J.rs[4] != 0.0) return;  // this patch's refinement has ended
  __shared__ double red[kResT / 32];
  double ss[1];
  residual_rows(J, J.xs, c * (kResT / 32) + (threadIdx.x >> 5), kResC * kResT / 32, ss);
  for (int o = 16; o > 0; o >>= 1) ss[0] += __shfl_xor_sync(kFull, ss[0], o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss[0];
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < kResT / 32; ++q) t += red[q];
    J.rs[8 + c] = t;
  }
}
// The same by one CTA of kRT threads, its norm summed in the same order: a patch's sweeps give the same bits
// in either kernel, whichever group of a round it is in.  A warp holds the sums of the kNS warps there whose
// blocks it takes.  red: kResC * kResT / 32 doubles of shared memory.
__device__ double patch_residual(const PatchJob& J, const float2* xs, double* red) {
  constexpr int kW = kResT / 32;  // warps of a CTA of patch_residual_kernel
  constexpr int kNS = kResC * kW / (kRT / 32);
  static_assert(kNS * (kRT / 32) == kResC * kW, "whole shares");
  double ss[kNS];
  residual_rows(J, xs, threadIdx.x >> 5, kRT / 32, ss);
#pragma unroll
  for (int u = 0; u < kNS; ++u) {
    for (int o = 16; o > 0; o >>= 1) ss[u] += __shfl_xor_sync(kFull, ss[u], o);
    if ((threadIdx.x & 31) == 0) red[(threadIdx.x >> 5) + u * (kRT / 32)] = ss[u];
  }
  __syncthreads();
  double s = 0.0;
  for (int c = 0; c < kResC; ++c) {
    double t = 0.0;
    for (int q = 0; q < kW; ++q) t += red[c * kW + q];
    s += t;
  }
  return sqrt(s);
}


// The refinement.  The first kSplit sweeps are launches of their own (MONO = false),
// each followed by patch_residual_kernel, which has several CTAs per patch where a
// sweep can have but one; this kernel with MONO = true then ends the patches that
// need more.  Measured on a GB300, the residual of one patch and the whole
// refinement (two sweeps; three at 48 x 48), against sweeps and residuals in one
// CTA: 16 x 16 ALEVB 157 -> 51 and 485 -> 342 us, 32 x 32 706 -> 171 us and 2.96 ->
// 1.96 ms, 48 x 48 1740 -> 383 us and 8.8 -> 5.4 ms.  What a sweep hands on stands in J.rs: [0] |r0|, [1] the last
// correction's norm, [2] and [3] the norms of the current one and of x, [4] nonzero
// once the patch is done, [8 ..] the residual's partial sums.
// GV: patches whose working vector of n floats does not fit the shared memory beside
// the rest (from 47 k unknowns: 110 x 110 LAG) keep it in global memory, in L1 and L2.
// The arithmetic is that of the other forms.
constexpr int kSplit = 3;
template <int RPT, bool MONO, bool GV = false>
__global__ void __launch_bounds__(kRT, 1) patch_refine_kernel(const PatchJob* __restrict__ jobs,
                                                             const int* __restrict__ order, int k0, int max_sweeps,
                                                             double tol) {
  const PatchJob& J = jobs[order[blockIdx.x]];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RefineSmem& S = *reinterpret_cast<RefineSmem*>(smem_raw);
  int* ps = reinterpret_cast<int*>(smem_raw + sizeof(RefineSmem));  // [npan + 1]
  float* vs = reinterpret_cast<float*>(ps + J.npan + 1);            // [n]
  float* v = GV && J.vg ? J.vg : vs;
  double* red = S.red;
  const int tid = threadIdx.x;
  const int64_t n = J.L.n;
  int* stat = J.stat;  // [0] status, [1] sweeps
  float2* xs = J.xs;   // x split into two floats
  auto end = [&](int status, int sweeps) MAFEM_INLINE {  // by every thread, none of which reads J.rs[4] again
    if (tid == 0) {
      stat[0] = status;
      stat[1] = sweeps;
      J.rs[4] = 1.0;
    }
  };
  double r0, rn, prev_dn;
  if (k0 == 0) {
    if (J.info[1] != 0 || J.info[0] != 0) {  // a bounded wait ran out, or a node block had no usable pivot
      end(J.info[1] != 0 ? MAFEM_ERR_CUDA : MAFEM_ZERO_PIVOT, 0);
      return;
    }
    double ss = 0.0;
    for (int64_t i = tid; i < n; i += kRT) {
      const double r = J.rhs[i];
      J.res[i] = r;
      J.x[i] = 0.0;
      ss = fma(r, r, ss);
    }
    r0 = rn = sqrt(block_sum(ss, red));
    prev_dn = INFINITY;
    if (tid == 0) {
      J.rs[0] = r0;
      J.rs[4] = 0.0;
    }
    if (!(r0 > 0.0)) {
      end(MAFEM_OK, 0);
      return;
    }
  } else if (J.rs[4] != 0.0) {
    return;
  }
  for (int k = J.npan - tid; k >= 0; k -= kRT) ps[k] = J.ps[k];
  // trace: per sweep 4 stamps after J.trace's 6 per panel -- [0] sweep start,
  // [1] substitutions done, [2] x updated and norms formed, [3] residual done
  long long* tr = J.trace ? J.trace + (size_t)J.npan * 6 : nullptr;
  // After sweep k (counted from 0) and its residual rn: a residual at FP64 level
  // (<= min(tol, 1e-10) |r0|) ends the solve: on large, stiff tangents the relative
  // correction has a rounding floor (about 1e-9 on the 64 x 64 patch) that a tight
  // tol would never reach.  So does the end of the contraction: at the rounding
  // floor (the correction a small part of x) the solution is as accurate as the
  // factors allow, and is accepted.
  auto after_residual = [&](int k, double dn, double xn) -> bool {
    if (tr && tid == 0 && k < kTraceSweeps) {  // trace: the residual after each sweep, relative to |r0|
      stamp(tr + 4 * k, 3);
      tr[4 * kTraceSweeps + 16 + k] = __double_as_longlong(rn / r0);
    }
    if (!isfinite(rn)) {
      end(MAFEM_NAN_DETECTED, k + 1);
    } else if (rn <= fmin(tol, 1e-10) * r0) {
      end(MAFEM_OK, k + 1);
    } else if (k >= 3 && dn > 0.5 * prev_dn) {
      end(dn <= 1e-8 * xn ? MAFEM_OK : MAFEM_REFINE_STALLED, k + 1);
    } else {
      return true;
    }
    return false;
  };
  if (k0 > 0) {
    r0 = J.rs[0];
    prev_dn = J.rs[1];
    const double dn = J.rs[2], xn = J.rs[3];
    double ss = 0.0;
    for (int q = 0; q < kResC; ++q) ss += J.rs[8 + q];
    rn = sqrt(ss);
    __syncthreads();  // J.rs is read
    if (!after_residual(k0 - 1, dn, xn)) return;
    prev_dn = dn;
  }
  for (int k = k0;; ++k) {
    if (k >= max_sweeps) {
      end(MAFEM_REFINE_STALLED, k);
      return;
    }
    long long* trk = tr && k < kTraceSweeps ? tr + 4 * k : nullptr;
    stamp(trk, 0);
    const double sc = 1.0 / rn;
    for (int64_t i = tid; i < n; i += kRT) v[i] = (float)(J.res[i] * sc);
    __syncthreads();
    patch_solve_pass<RPT>(J, v, ps, S, tr && k == 0 ? tr + 4 * kTraceSweeps : nullptr);
    stamp(trk, 1);
    double dd = 0.0, xx = 0.0;
    for (int64_t i = tid; i < n; i += kRT) {
      const double d = rn * (double)v[i];
      const double x = fma(rn, (double)v[i], J.x[i]);
      J.x[i] = x;
      const float xh = (float)x;
      xs[i] = make_float2(xh, (float)(x - (double)xh));
      dd = fma(d, d, dd);
      xx = fma(x, x, xx);
    }
    const double dn = sqrt(block_sum(dd, red));
    const double xn = sqrt(block_sum(xx, red));
    stamp(trk, 2);
    if (!isfinite(dn) || !isfinite(xn)) {
      end(MAFEM_NAN_DETECTED, k + 1);
      return;
    }
    // Stop when the error left in x is small against x.  After sweep k that
    // error is about the next correction, rho |d_k| with rho = |d_k| / |d_k-1|
    // the sweeps' contraction: stop once rho |d_k| <= tol |x| while the sweeps
    // contract (rho <= 1/2), or once |d_k| <= tol |x| itself.  A bound on the
    // forward error of x whatever the conditioning, where a residual test would
    // accept a large error in x on an ill-conditioned tangent; the residual
    // after the final sweep is never needed.
    const double rho = dn / prev_dn;  // 0 after the first sweep (prev_dn infinite)
    if (dn <= tol * xn || (k >= 1 && rho <= 0.5 && rho * dn <= tol * xn)) {
      end(MAFEM_OK, k + 1);
      return;
    }
    if constexpr (!MONO) {
      if (tid == 0) {
        J.rs[1] = prev_dn;
        J.rs[2] = dn;
        J.rs[3] = xn;
      }
      return;
    } else {
      // block_sum orders the x / xs writes before it; the update warps' sums are not in use
      rn = patch_residual(J, xs, reinterpret_cast<double*>(S.part));
      if (!after_residual(k, dn, xn)) return;
      prev_dn = dn;
    }
  }
}

// The split-A21 buffer as a 3-D tensor (k % 4, row, k / 4) of FP32 with strides
// 16 bytes (rows) and 8 a21_rows x 16 bytes (k-quad planes); one 4 x 128 x 8 box
// is one M tile in the MMA's K-major core-matrix layout (k-quad planes 2 KB
// apart, rows 16 bytes apart).
bool patch_a21_map(PatchJob& J) {
  using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static EncodeFn encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return false;
    encode = reinterpret_cast<EncodeFn>(fn);
  }
  const cuuint64_t rows = (cuuint64_t)4 * 2 * J.a21_rows;  // four ranks x (hi, lo)
  const cuuint64_t dims[3] = {4, rows, 8};
  const cuuint64_t strides[2] = {16, rows * 16};
  const cuuint32_t box[3] = {4, (cuuint32_t)kMT, 8};
  const cuuint32_t estr[3] = {1, 1, 1};
  return encode(&J.a21_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, J.a21, dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int patch_solve_setup() {
  int dev = 0, cap = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
  const int dyn = patch_dyn_smem(cap);
  if (cudaFuncSetAttribute(patch_factor_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess ||
      cudaFuncSetAttribute(patch_factor_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess ||
      cudaFuncSetAttribute(patch_factor_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess ||
      cudaFuncSetAttribute(patch_refine_kernel<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess ||
      cudaFuncSetAttribute(patch_refine_kernel<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess ||
      cudaFuncSetAttribute(patch_refine_kernel<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess ||
      cudaFuncSetAttribute(patch_refine_kernel<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess)
    return 0;
  return dyn;
}
bool patch_vector_setup(int dyn) {
  return cudaFuncSetAttribute(patch_refine_kernel<2, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) ==
             cudaSuccess &&
         cudaFuncSetAttribute(patch_refine_kernel<2, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) ==
             cudaSuccess;
}

int patch_cluster_ctas(int kuf) { return kuf > 2 * kNCH ? 4 : kuf > kNCH ? 2 : 1; }

static cudaError_t launch_factor(const PatchJob* d_jobs, const int* d_order, int njobs, int nr, size_t smem,
                                 cudaStream_t st) {
  if (njobs <= 0) return cudaSuccess;
  if (nr == 1) {
    patch_factor_kernel<1><<<njobs, kPT, smem, st>>>(d_jobs, d_order);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nr * njobs));
  cfg.blockDim = dim3(kPT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)nr;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return nr == 4 ? cudaLaunchKernelEx(&cfg, patch_factor_kernel<4>, d_jobs, d_order)
                 : cudaLaunchKernelEx(&cfg, patch_factor_kernel<2>, d_jobs, d_order);
}

// A band is wide for the refinement (two register sets per thread) with more rows or
// columns beyond a panel than one set of the update warps holds.
int patch_form(const PatchJob& J) { return J.vg ? 2 : J.L.kl > kRowT || J.kuf > kRowT ? 1 : 0; }
static cudaError_t launch_refine(const PatchJob* d_jobs, const int* d_order, int njobs, int form, size_t smem,
                                 int max_sweeps, double tol, cudaStream_t st, bool apart = true) {
  auto sweeps = [&](auto kern, int k0) { kern<<<njobs, kRT, smem, st>>>(d_jobs, d_order, k0, max_sweeps, tol); };
  const int split = apart ? std::min(kSplit, max_sweeps) : 0;
  for (int k = 0; k < split; ++k) {
    if (form == 2) sweeps(patch_refine_kernel<2, false, true>, k);
    else if (form == 1) sweeps(patch_refine_kernel<2, false>, k);
    else sweeps(patch_refine_kernel<1, false>, k);
    patch_residual_kernel<<<njobs * kResC, kResT, 0, st>>>(d_jobs, d_order);
  }
  if (form == 2) sweeps(patch_refine_kernel<2, true, true>, split);
  else if (form == 1) sweeps(patch_refine_kernel<2, true>, split);
  else sweeps(patch_refine_kernel<1, true>, split);
  return cudaGetLastError();
}

cudaError_t patch_solve_stage(const PatchJob* d_jobs, const int* d_order, int njobs, int nr, size_t smem_factor,
                              size_t smem_refine, int form, int max_sweeps, double tol, cudaStream_t st) {
  if (njobs <= 0) return cudaSuccess;
  if (smem_factor) {
    const cudaError_t e = launch_factor(d_jobs, d_order, njobs, nr, smem_factor, st);
    if (e != cudaSuccess) return e;
  }
  if (smem_refine) return launch_refine(d_jobs, d_order, njobs, form, smem_refine, max_sweeps, tol, st);
  return cudaGetLastError();
}

// ---- autotuning: the factorisation's time per cluster size -------------------------
// A synthetic band of the job's shape: entries of the band uniform in [-1, 1)
// (a hash of i and j), the diagonal kl + ku + 2 (diagonally dominant, so every
// node block keeps its own pivots), the pivoting fill rows zero.  The
// factorisation's time does not depend on the values.
__global__ void patch_fill_synthetic_kernel(const PatchJob* __restrict__ jobs, const int* __restrict__ order) {
  const PatchJob& J = jobs[order[0]];
  const BandLayout L = J.L;
  const int64_t total = L.ldb * L.n;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = idx / L.ldb, i = j + (idx - j * L.ldb) - L.off;
    float v = 0.0f;
    if (i >= 0 && i < L.n && i - j <= L.kl && j - i <= L.ku) {
      uint32_t h = (uint32_t)i * 73856093u ^ (uint32_t)j * 19349663u;
      h ^= h >> 13;
      h *= 0x5bd1e995u;
      h ^= h >> 15;
      v = i == j ? (float)(L.kl + L.ku + 2) : (float)(h & 0xffffu) * (1.0f / 32768.0f) - 1.0f;
    }
    J.band[idx] = v;
  }
}

cudaError_t patch_time_factor(const PatchJob* d_jobs, const int* d_order1, int nr, size_t smem, cudaStream_t st,
                              float* ms) {
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaError_t e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  for (int rep = 0; rep < 2 && e == cudaSuccess; ++rep) {  // the second run is timed
    patch_fill_synthetic_kernel<<<1024, 256, 0, st>>>(d_jobs, d_order1);
    e = cudaEventRecord(e0, st);
    if (e == cudaSuccess) e = launch_factor(d_jobs, d_order1, 1, nr, smem, st);
    if (e == cudaSuccess) e = cudaEventRecord(e1, st);
    if (e == cudaSuccess) e = cudaEventSynchronize(e1);
  }
  if (e == cudaSuccess) e = cudaEventElapsedTime(ms, e0, e1);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  return e;
}

int patch_solve_launches(const PatchGroups& G, int njobs, int max_sweeps) {
  const int groups = (G.n4 > 0) + (G.n2 > 0) + (njobs - G.n4 - G.n2 > 0);
  // the factor launches, and the refinement of each stream (launch_refine)
  return groups + 1 + 2 * std::min(kSplit, max_sweeps) + (groups > 1 ? 1 : 0);
}

cudaError_t patch_solve(const PatchJob* d_jobs, const int* d_order, const PatchGroups& G, int njobs,
                        size_t smem_factor, size_t smem_refine, int max_sweeps, double tol, cudaStream_t st,
                        cudaStream_t st2, cudaEvent_t ev_fork, cudaEvent_t ev_join) {
  if (njobs <= 0) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  // the groups in launch order: four-CTA clusters, two-CTA clusters, single
  // CTAs; the first non-empty group on st, the others one after the other on
  // st2 beside it (their chains are the shorter ones).  Each stream refines its
  // own patches as soon as their factors are done, so the refinement of one
  // group overlaps the factorisations of the other.  The first group's sweeps and
  // residuals are launches apart (it ends the round); beside it one kernel will do.
  const int cnt[3] = {G.n4, G.n2, njobs - G.n4 - G.n2}, nrs[3] = {4, 2, 1};
  int first = 0;
  while (first < 3 && cnt[first] == 0) ++first;
  const bool fork = cnt[first] < njobs;
  if (fork) {
    e = cudaEventRecord(ev_fork, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st2, ev_fork, 0);
  }
  int off = 0;
  for (int g = 0; g < 3 && e == cudaSuccess; ++g) {
    if (cnt[g] == 0) continue;
    e = launch_factor(d_jobs, d_order + off, cnt[g], nrs[g], smem_factor, g == first ? st : st2);
    off += cnt[g];
    if (g == first && e == cudaSuccess)
      e = launch_refine(d_jobs, d_order, cnt[g], G.form[g], smem_refine, max_sweeps, tol, st);
  }
  if (fork && e == cudaSuccess) {
    int form = 0;
    for (int g = first + 1; g < 3; ++g) form = std::max(form, G.form[g]);
    e = launch_refine(d_jobs, d_order + cnt[first], njobs - cnt[first], form, smem_refine, max_sweeps, tol, st2, false);
  }
  if (fork && e == cudaSuccess) e = cudaEventRecord(ev_join, st2);
  if (fork && e == cudaSuccess) e = cudaStreamWaitEvent(st, ev_join, 0);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

}  // namespace mafem

// band_lu_blk.cu -- banded LU with pivoting restricted to each node's dof block.
//
// The tangent is ordered node-major (Mesh.jl:276-284), so the unknowns of one
// control point are consecutive: a "pivot block" of at most ndf rows.  Here the
// pivot of column j is searched only among the rows of j's block that are not
// yet eliminated, instead of among all kl rows below the diagonal as LAPACK's
// gbtrf does.  On the membrane tangents this is as accurate as full partial
// pivoting (growth ~1e2, backward error ~1e-15, forward error at the
// conditioning floor) and it changes the work and the critical path on a GPU:
//   * panels are runs of whole blocks, so interchanges never leave a panel and
//     U fills only to kuf = ku + ndfp columns (ndfp = largest block - 1)
//     instead of kl + ku: half the FP64 work of the trailing updates;
//   * the pivot search is one warp reduction over <= 8 rows;
//   * rows below a panel never take part in its pivot steps, so their
//     multipliers L21 = A21 U11^-1 are never formed: the trailing update and
//     the forward substitution apply L21 u = A21 (U11^-1 u) with the raw A21;
//   * the solved columns Y = A11^-1 A12 are kept in place of U12 = U11 Y: the
//     forward substitution then leaves z = A11^-1 b1, the back substitution is
//     x1 = z - Y x2, and no triangle is solved on its chain of panels.
// A zero or non-finite pivot sets `info`; the caller then falls back to the
// full partial-pivoting factorisation (band_lu.cu).
//
// After panel p (columns [j0, j1), w = j1 - j0 <= 32) the band holds, in the
// panel's columns, L11 (unit, strict lower) and U11 in rows [j0, j1) and the
// untouched A21 in rows [j1, j0 + R), R = w + kl, and Y in rows [j0, j1) of the
// columns right of it; rdiag[j] = 1 / U(j, j);
// perm_all[p * kBlkW + i] = the panel row moved to position i.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "band_lu_common.cuh"

namespace mafem {


// ---------------------------------------------------------------------------
// Panel factorisation kernel: one CTA, the body in blk_panel_factor.
template <class T>
__global__ void __launch_bounds__(32 * kPanelWarps) blk_panel_kernel(T* __restrict__ ab, BandLayout L, int64_t j0, int w,
                                                                     const int* __restrict__ blk_end,
                                                                     int* __restrict__ perm, T* __restrict__ rdiag,
                                                                     int* __restrict__ info) {
  __shared__ T s_l[2][32];
  __shared__ int s_p[2];
  blk_panel_factor<T, false>(ab + bix(L, j0, j0), 1, L.ldb - 1, (int)j0, w, (int)j0 + 1, 1, blk_end + j0, perm,
                             rdiag + j0, info, s_l, s_p);
}

// ---------------------------------------------------------------------------
// Trailing update of a panel: four columns per CTA, each column run by a pair
// of warps (warps q and q + 4 share a sub-partition's FP64 pipe, so one warp's
// issue stalls overlap the other's work).  Per column segment
// s = A(j0 .. j0+R-1, c), rows [0, w) permuted:
//   u = L11^-1 s[0:w],   y = U11^-1 u   (kept as Y),   s[w:R] -= A21 y.
// Warp q stages the column and runs the two triangular solves, then releases
// warp q + 4 (named barrier 1 + q); the two split the 32-row chunks of the
// A21 y update (NCH chunks each per pass).  Before warp q overwrites the
// column buffer for its next column it waits until warp q + 4 is done with
// the previous one (named barrier 5 + q).  The panel columns (L11\U11 and
// A21) are staged in shared memory once per CTA.
template <class T, int NCH>
__global__ void __launch_bounds__(256) blk_apply_kernel(T* __restrict__ ab, BandLayout L, int64_t j0, int w,
                                                        const int* __restrict__ perm, const T* __restrict__ rdiag,
                                                        T* __restrict__ rhs, int64_t c0, int ncol) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int R = (int)min64b(L.n - j0, (int64_t)w + L.kl);
  T* Lp = reinterpret_cast<T*>(smem_raw);  // [w][R] + 64 NCH padding (chunk reads past R)
  T* S = Lp + (size_t)w * R + 64 * NCH;    // [4][R]
  T* Y = S + (size_t)4 * R;                // [4][32]
  T* rd = Y + 128;                         // [32]
  int* sp = reinterpret_cast<int*>(rd + 32);  // [32]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int slot = warp & 3, half = warp >> 2;
  const int ntot = ncol + (rhs ? 1 : 0);
  if ((int)blockIdx.x * 4 >= ntot) return;
  for (int c = 0; c < w; ++c) {
    const T* src = ab + bix(L, j0, j0 + c);  // A(j0 + r, j0 + c) = src[r]
    for (int r = tid; r < R; r += 256) cp_async(Lp + (size_t)c * R + r, src + r);
  }
  if (tid < w) {
    rd[tid] = rdiag[j0 + tid];
    sp[tid] = perm[tid];
  }
  cp_async_wait_all();
  __syncthreads();
  T* s = S + (size_t)slot * R;
  T* yw = Y + slot * 32;
  for (int cc = blockIdx.x * 4 + slot; cc < ntot; cc += gridDim.x * 4) {
    const bool is_rhs = cc == ncol;
    const bool more = cc + (int)gridDim.x * 4 < ntot;
    T* dst = is_rhs ? rhs + j0 : ab + bix(L, j0, c0 + cc);  // row j0 + r of the column = dst[r]
    if (half == 0) {
      if (cc != (int)blockIdx.x * 4 + slot) bar_sync_n(5 + slot, 64);  // partner done with the previous column
      for (int r = lane; r < R; r += 32) cp_async(s + r, dst + (r < w ? sp[r] : r));
      cp_async_wait_all();
      __syncwarp();
      T x = lane < w ? s[lane] : T(0);
      for (int k = 0; k < w; ++k) {
        const T xk = __shfl_sync(kFull, x, k);
        if (lane > k && lane < w) x -= Lp[k * R + lane] * xk;
      }
      T v = x;
      for (int k = w - 1; k >= 0; --k) {
        T yk = lane == k ? v * rd[k] : T(0);
        yk = __shfl_sync(kFull, yk, k);
        if (lane == k) v = yk;
        if (lane < k) v -= Lp[k * R + lane] * yk;
      }
      if (lane < w) dst[lane] = v;  // Y
      yw[lane] = v;
      bar_arrive_n(1 + slot, 64);
    } else {
      bar_sync_n(1 + slot, 64);
    }
    for (int base = w; base < R; base += 64 * NCH) {
      const int hb = base + half * 32 * NCH;  // this warp's first row
      T acc[NCH];
#pragma unroll
      for (int j = 0; j < NCH; ++j) acc[j] = s[min(hb + 32 * j + lane, R - 1)];
      for (int k = 0; k < w; ++k) {
        const T yk = yw[k];
        const T* lk = Lp + (size_t)k * R + hb + lane;
#pragma unroll
        for (int j = 0; j < NCH; ++j)
          if (hb + 32 * j < R) acc[j] = fma(-lk[32 * j], yk, acc[j]);  // warp-uniform guard
      }
#pragma unroll
      for (int j = 0; j < NCH; ++j) {
        const int r = hb + 32 * j + lane;
        if (r < R) dst[r] = acc[j];
      }
    }
    if (half == 1 && more) bar_arrive_n(5 + slot, 64);
  }
}

// ---------------------------------------------------------------------------
// Critical-path variant for the next panel's columns: one CTA per column.
// Warp 0 runs the triangular solves; the four warps share the A21 y update,
// NR rows per thread, reading A21 straight from the band (L2-resident).
template <class T, int NR>
__global__ void __launch_bounds__(128) blk_apply_col_kernel(T* __restrict__ ab, BandLayout L, int64_t j0, int w,
                                                            const int* __restrict__ perm,
                                                            const T* __restrict__ rdiag, int64_t c0) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int R = (int)min64b(L.n - j0, (int64_t)w + L.kl);
  const int64_t c = c0 + blockIdx.x;
  T* s = reinterpret_cast<T*>(smem_raw);  // [R]
  __shared__ T T11[32][33];               // L11 below, U11 on and above the diagonal (transposed: [col][row])
  __shared__ T y[32];
  __shared__ T rd[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < w) rd[tid] = rdiag[j0 + tid];
  for (int r = tid; r < R; r += 128) s[r] = ab[bix(L, j0 + (r < w ? perm[r] : r), c)];
  for (int k = tid; k < w * w; k += 128) {
    const int cc = k / w, i = k - cc * w;
    T11[cc][i] = ab[bix(L, j0 + i, j0 + cc)];
  }
  __syncthreads();
  if (warp == 0) {
    T x = lane < w ? s[lane] : T(0);
    for (int k = 0; k < w; ++k) {
      const T xk = __shfl_sync(kFull, x, k);
      if (lane > k && lane < w) x -= T11[k][lane] * xk;
    }
    T v = x;
    for (int k = w - 1; k >= 0; --k) {
      T yk = lane == k ? v * rd[k] : T(0);
      yk = __shfl_sync(kFull, yk, k);
      if (lane == k) v = yk;
      if (lane < k) v -= T11[k][lane] * yk;
    }
    if (lane < w) s[lane] = v;
    y[lane] = lane < w ? v : T(0);
  }
  __syncthreads();
  for (int base = w; base < R; base += 128 * NR) {
    T acc[NR];
    int ri[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      ri[i] = min(base + 128 * i + tid, R - 1);
      acc[i] = s[ri[i]];
    }
    const int wrow = base + warp * 32;
    const T* col0 = ab + bix(L, j0, j0);  // A(j0 + r, j0 + k) = col0[k * (ldb - 1) + r]
    for (int k0 = 0; k0 < w; k0 += 8) {
      T a[8][NR];  // eight columns of A21 in flight per thread
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const T* col = col0 + (int64_t)min(k0 + kk, w - 1) * (L.ldb - 1);
#pragma unroll
        for (int i = 0; i < NR; ++i) a[kk][i] = (wrow + 128 * i < R) ? col[ri[i]] : T(0);
      }
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        if (k0 + kk < w) {
          const T yk = y[k0 + kk];
#pragma unroll
          for (int i = 0; i < NR; ++i)
            if (wrow + 128 * i < R) acc[i] = fma(-a[kk][i], yk, acc[i]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int r = base + 128 * i + tid;
      if (r < R) ab[bix(L, j0 + r, c)] = acc[i];
    }
  }
  for (int r = tid; r < w; r += 128) ab[bix(L, j0 + r, c)] = s[r];
}

// A launch covers panels [p0, p1) of one chain, or of two chains side by side (CTAs
// below `split` the first): the columns right of panel p1 - 1 (backward) or the panels
// before p0 (forward) belong to an earlier launch.
struct BlkSpan {
  BlkChain c;
  int p0, p1;
};

// ---------------------------------------------------------------------------
// Substitutions by one CTA, over the spans of the cooperative ones (below) in the same
// order, where a cooperative launch is not possible.  Forward: z(p) = A11^-1 (b(p) -
// the panels before it), pulled, so that either kernel can go on after the other.
template <class T>
__global__ void __launch_bounds__(1024) blk_forward_kernel(const T* __restrict__ ab, int kl, BlkSpan S,
                                                           const int* __restrict__ perm_all,
                                                           const T* __restrict__ rdiag_all, double* bv,
                                                           const int* __restrict__ gate) {
  __shared__ double part[32][33], Ls[32][33], xs[32];
  if (gate && *gate) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int64_t si = S.c.si, sj = S.c.sj;
  const T* __restrict__ A = ab + S.c.org;  // element (i, j) at A[i si + j sj]
  double* b = bv + S.c.vorg;               // element i at b[i si]
  for (int p = S.p0; p < S.p1; ++p) {
    const int j0 = S.c.ps[p], w = S.c.ps[p + 1] - j0;
    for (int k = tid; k < w * w; k += blockDim.x) {
      const int c = k / w, i = k - c * w;
      Ls[c][i] = (double)A[(j0 + i) * si + (j0 + c) * sj];
    }
    double acc = 0.0;
    const int r = j0 + lane;
    if (lane < w) {
      int c = max(0, r - kl) + warp;  // the row's first stored column
      for (; c + 7 * nw < j0; c += 8 * nw) {
        double a[8], z[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          a[q] = (double)A[r * si + (c + q * nw) * sj];
          z[q] = b[(c + q * nw) * si];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) acc = fma(a[q], z[q], acc);
      }
      for (; c < j0; c += nw) acc = fma((double)A[r * si + c * sj], b[c * si], acc);
    }
    part[warp][lane] = acc;
    __syncthreads();
    if (warp == 0) {
      double sum = 0.0;
      for (int k = 0; k < nw; ++k) sum += part[k][lane];
      xs[lane] = lane < w ? b[r * si] - sum : 0.0;
      __syncwarp();
      double x = lane < w ? xs[perm_all[(size_t)(S.c.pbase + p) * kBlkW + lane]] : 0.0;
      for (int k = 0; k < w; ++k) {
        const double xk = __shfl_sync(kFull, x, k);
        if (lane > k && lane < w) x -= Ls[k][lane] * xk;
      }
      const double rd = lane < w ? (double)rdiag_all[S.c.rbase + r] : 0.0;
      for (int k = w - 1; k >= 0; --k) {
        const double yk = __shfl_sync(kFull, x * rd, k);
        if (lane == k) x = yk;
        if (lane < k) x -= Ls[k][lane] * yk;
      }
      if (lane < w) b[r * si] = x;
    }
    __syncthreads();
  }
}

// Back substitution x1 = z - Y x2, panels in reverse; Y has kuf super-diagonals.
template <class T>
__global__ void __launch_bounds__(1024) blk_backward_kernel(const T* __restrict__ ab, int kuf, BlkSpan S, double* yv,
                                                            const int* __restrict__ gate) {
  __shared__ double part[32][33];
  if (gate && *gate) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int64_t si = S.c.si, sj = S.c.sj;
  double* y = yv + S.c.vorg;
  for (int p = S.p1 - 1; p >= S.p0; --p) {
    const int j0 = S.c.ps[p], j1 = S.c.ps[p + 1], w = j1 - j0, jend = min(S.c.n, j1 + kuf);
    const T* __restrict__ row = ab + S.c.org + (j0 + lane) * si;  // A(j0 + lane, c) at row[c sj]
    double acc = 0.0;
    if (lane < w) {
      int c = j1 + warp;
      for (; c + 7 * nw < jend; c += 8 * nw) {
        double u[8], xv[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          u[q] = (double)row[(c + q * nw) * sj];
          xv[q] = y[(c + q * nw) * si];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) acc = fma(u[q], xv[q], acc);
      }
      for (; c < jend; c += nw) acc = fma((double)row[c * sj], y[c * si], acc);
    }
    part[warp][lane] = acc;
    __syncthreads();
    if (warp == 0) {
      double sum = 0.0;
      for (int k = 0; k < nw; ++k) sum += part[k][lane];
      if (lane < w) y[(j0 + lane) * si] -= sum;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Two 32 x 32 matrices per panel for the cooperative forward substitution, element
// (i, k) at k * 32 + i, zero outside the panel's rows and columns.  One warp per panel
// (four per CTA), lane c forming column c of both.
// FP32 factors: Ai = U11^-1 L11^-1 P, and W = Ai A(p, p - 1), the panel's rows of the
// panel before it, so that of z(p) = Ai (b - sum over q < p of A(p, q) z(q)) everything
// but W z(p - 1) can be formed before z(p - 1) is there.  Formed and applied in FP64,
// their rounding, of the size of A11's condition, stays far below the factors' own.
// FP64 factors: L11^-1 P and U11^-1, each applied by itself: on tangents whose diagonal
// blocks are ill-conditioned (strips of the ALE motions) Ai and W left backward errors
// of up to 2e-4 (median 2e-15, nine in ten below 3e-11) where the triangles' inverses
// stay at the level of the triangles' solves, 2e-16.
template <class T>
constexpr bool kTriangles = sizeof(T) == 8;
template <class T>
__global__ void __launch_bounds__(128) blk_inverses_kernel(const T* __restrict__ ab, BlkChain c0, BlkChain c1, int split,
                                                           int kl,
                                                           const int* __restrict__ perm_all,
                                                           const T* __restrict__ rdiag_all, double* __restrict__ inv) {
  __shared__ double S[4][32][33];  // per warp: S[k][i] = A(j0 + i, j0 + k) of its panel, then Ai
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool second = (int)blockIdx.x >= split;
  const BlkChain& c = second ? c1 : c0;
  const int p = ((int)blockIdx.x - (second ? split : 0)) * 4 + warp;
  if (p >= c.npan) return;  // warp-uniform; only warp-level synchronisation below
  const int j0 = c.ps[p], w = c.ps[p + 1] - j0;
  const T* blk = ab + c.org + j0 * c.si + j0 * c.sj;
  const T* rdiag = rdiag_all + c.rbase;
  for (int k = 0; k < 32; ++k) S[warp][k][lane] = (k < w && lane < w) ? (double)blk[lane * c.si + k * c.sj] : 0.0;
  const double rd = lane < w ? (double)rdiag[j0 + lane] : 0.0;
  const int pr = lane < w ? perm_all[(size_t)(c.pbase + p) * kBlkW + lane] : -1;
  __syncwarp();
  double* Ai = inv + (size_t)(c.pbase + p) * 2 * kBlkW * kBlkW;
  double* W = Ai + kBlkW * kBlkW;
  // column `lane`: L11 y = P e_lane forward, U11 x = y (triangles: e_lane) backward
  double x[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) x[i] = __shfl_sync(kFull, pr, i) == lane ? 1.0 : 0.0;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const double xk = x[k];
#pragma unroll
    for (int i = k + 1; i < 32; ++i) x[i] = fma(-S[warp][k][i], xk, x[i]);
  }
  if constexpr (kTriangles<T>) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      Ai[lane * 32 + i] = (lane < w && i < w) ? x[i] : 0.0;
      x[i] = i == lane ? 1.0 : 0.0;
    }
  }
#pragma unroll
  for (int k = 31; k >= 0; --k) {
    const double xk = x[k] * __shfl_sync(kFull, rd, k);
    x[k] = xk;
#pragma unroll
    for (int i = 0; i < k; ++i) x[i] = fma(-S[warp][k][i], xk, x[i]);
  }
  if constexpr (kTriangles<T>) {
#pragma unroll
    for (int i = 0; i < 32; ++i) W[lane * 32 + i] = (lane < w && i < w) ? x[i] : 0.0;
    return;
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const double v = (lane < w && i < w) ? x[i] : 0.0;
    Ai[lane * 32 + i] = v;
    S[warp][lane][i] = v;
  }
  __syncwarp();
  const int q0 = p > 0 ? c.ps[p - 1] : j0;  // column q0 + lane of the panel before
  const T* col = ab + c.org + j0 * c.si + (q0 + lane) * c.sj;
#pragma unroll
  for (int i = 0; i < 32; ++i) x[i] = 0.0;
  for (int m = 0; m < w; ++m) {
    const double am = q0 + lane < j0 && j0 + m - (q0 + lane) <= kl ? (double)col[m * c.si] : 0.0;
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = fma(S[warp][m][i], am, x[i]);
  }
#pragma unroll
  for (int i = 0; i < 32; ++i) W[lane * 32 + i] = x[i];
}

// ---------------------------------------------------------------------------
// Substitutions on many SMs: one cooperative launch, panel by panel over its CTAs
// of four warps (one per sub-partition).  A panel's solution is handed on as
// 16-byte words of a value and a tag, written and read whole: whoever needs it polls
// the words themselves, so a panel's step on the chain is one store, one load, eight
// multiply-adds per lane and two shuffles -- no fence, no flag, no barrier.  (With a
// flag per panel, a fence before it and a barrier after it: 2.9 us per panel back,
// about 8 us forward.)  A lane holds one of its warp's 8 rows and every fourth
// column; the matrix entries of the next panel are loaded before the poll.  Tags are
// the launch's epoch, so they never need clearing.  Waits are bounded: after wt.limit
// polls (kSpinLimit by default) the kernel sets *err and every CTA returns (no GPU
// hang; the host reports the error).  wt.withhold = k >= 0 (failure-detection tests
// only): the back substitution's panel npan - 1 - k is never published, so the CTAs
// that need it run out of polls.
__device__ __forceinline__ void publish(SolveWord* p, double v, long long tag) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ double peek(const SolveWord* p, long long& tag) {
  long long v;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(v), "=l"(tag)
               : "l"(p)
               : "memory");
  return __longlong_as_double(v);
}
// This lane's entries cg, cg + 4, ... < nc of a panel's words X, once all of the warp's
// carry the tag (tag 0: from an earlier launch, at once).  false, for the whole warp,
// when the polls ran out or another warp has set *err.
__device__ __forceinline__ bool fetch(const SolveWord* X, int cg, int nc, long long tag, bool far, double (&y)[8], int* err,
                                      int limit) {
  const int lim = limit > 0 ? limit : kSpinLimit;
  for (int it = 0;; ++it) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      long long t = tag;
      y[i] = cg + 4 * i < nc ? peek(X + cg + 4 * i, t) : 0.0;
      ok &= t == tag;
    }
    if (tag == 0 || __all_sync(kFull, ok)) return true;
    if (it > lim || ((it & 31) == 31 && __any_sync(kFull, *(volatile int*)err != 0))) {
      if ((threadIdx.x & 31) == 0) atomicCAS(err, 0, 1);
      return false;
    }
    __nanosleep(far ? 200 : 20);
  }
}

constexpr int kSolveThreads = 128;

// Back substitution x1 = z - Y x2.
template <class T>
__global__ void __launch_bounds__(kSolveThreads)
    blk_backward_coop_kernel(const T* __restrict__ ab, int kuf, BlkSpan s0, BlkSpan s1, int split, double* yv,
                             SolveWord* xch, long long epoch, int* err, WaitTest wt, const int* gate) {
  if (gate && *gate) return;  // every CTA reads the same word: all return (refinement already stopped)
  const int lane = threadIdx.x & 31, row = 8 * (threadIdx.x >> 5) + (lane & 7), cg = lane >> 3;
  const bool second = (int)blockIdx.x >= split;
  const BlkSpan& S = second ? s1 : s0;
  const int me = (int)blockIdx.x - (second ? split : 0), G = second ? (int)gridDim.x - split : split;
  const int* __restrict__ ps = S.c.ps;
  const int64_t si = S.c.si, sj = S.c.sj;
  double* y = yv + S.c.vorg;  // element i at y[i si]
  SolveWord* X = xch + (size_t)S.c.pbase * kBlkW;
  for (int q = S.p1 - 1 - me; q >= S.p0; q -= G) {
    const int j0 = ps[q], j1 = ps[q + 1];
    const int w = j1 - j0;
    const int jend = min(S.c.n, j1 + kuf);
    const int r = j0 + min(row, w - 1);
    const T* arow = ab + S.c.org + r * si;
    const double z = y[r * si];
    double acc[2] = {0.0, 0.0};
    for (int c0 = max(j1, ps[S.p1]) + cg; c0 < jend; c0 += 32) {  // columns solved before this launch
      T av[8];
      double xv[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = c0 + 4 * i;
        av[i] = c < jend ? arow[c * sj] : T(0);
        xv[i] = c < jend ? y[c * si] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i & 1] = fma((double)av[i], xv[i], acc[i & 1]);
    }
    int p = q;  // last panel of the launch with columns in [j1, jend)
    while (p + 1 < S.p1 && ps[p + 1] < jend) ++p;
    T an[8];
    auto load = [&](int pp) {
      const int cb = ps[pp], ce = min(ps[pp + 1], jend);
#pragma unroll
      for (int i = 0; i < 8; ++i) an[i] = cb + cg + 4 * i < ce ? arow[(cb + cg + 4 * i) * sj] : T(0);
    };
    if (p > q) load(p);
    for (; p > q; --p) {
      double av[8], xv[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) av[i] = (double)an[i];
      if (p - 1 > q) load(p - 1);
      if (!fetch(X + (size_t)p * kBlkW, cg, min(ps[p + 1], jend) - ps[p], epoch, p > q + 2, xv, err, wt.limit)) return;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i & 1] = fma(av[i], xv[i], acc[i & 1]);
    }
    double s = acc[0] + acc[1];
    s += __shfl_xor_sync(kFull, s, 8);
    s += __shfl_xor_sync(kFull, s, 16);
    if (cg == 0 && row < w) {
      const double x = z - s;
      if (second || S.c.npan - 1 - q != wt.withhold) publish(X + (size_t)q * kBlkW + row, x, epoch);
      y[r * si] = x;
    }
  }
}

// Forward substitution z(p) = A11^-1 (b(p) - sum over q < p of A(p, q) z(q)), each panel's
// contributions pulled from the panels before it; FP32 factors: the last of them by W,
// FP64 factors: L11^-1 P and U11^-1 after it (blk_inverses_kernel).
template <class T>
__global__ void __launch_bounds__(kSolveThreads)
    blk_forward_coop_kernel(const T* __restrict__ ab, int kl, BlkSpan s0, BlkSpan s1, int split,
                            const double* __restrict__ inv_all, double* bv, SolveWord* xch, long long epoch, int* err,
                            WaitTest wt, const int* gate) {
  __shared__ double xs[2][32];
  [[maybe_unused]] __shared__ double ys[32];
  if (gate && *gate) return;
  const int lane = threadIdx.x & 31, row = 8 * (threadIdx.x >> 5) + (lane & 7), cg = lane >> 3;
  const bool second = (int)blockIdx.x >= split;
  const BlkSpan& S = second ? s1 : s0;
  const int me = (int)blockIdx.x - (second ? split : 0), G = second ? (int)gridDim.x - split : split;
  const int* __restrict__ ps = S.c.ps;
  const int64_t si = S.c.si, sj = S.c.sj;
  double* b = bv + S.c.vorg;  // element i at b[i si]
  SolveWord* X = xch + (size_t)S.c.pbase * kBlkW;
  int par = 0;
  bool ok = true;
  for (int p = S.p0 + me; p < S.p1; p += G, par ^= 1) {
    const int j0 = ps[p];
    const int w = ps[p + 1] - j0;
    const int r = j0 + min(row, w - 1);
    const T* arow = ab + S.c.org + r * si;
    const double br = row < w ? b[r * si] : 0.0;
    const double* Ip = inv_all + (size_t)(S.c.pbase + p) * 2 * kBlkW * kBlkW;
    double Ai[8], W[8];  // (FP64 factors: L11^-1 P, U11^-1)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      Ai[i] = Ip[(cg + 4 * i) * 32 + row];
      W[i] = Ip[kBlkW * kBlkW + (cg + 4 * i) * 32 + row];
    }
    int q = p;  // earliest panel whose rows reach j0
    while (q > 0 && ps[q] + kl > j0) --q;
    double acc[2] = {0.0, 0.0};
    T an[8];
    auto load = [&](int qq) {
      const int cb = ps[qq], ce = ps[qq + 1];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = cb + cg + 4 * i;
        an[i] = c < ce && r - c <= kl ? arow[c * sj] : T(0);  // inside that panel's band rows
      }
    };
    const int qe = kTriangles<T> ? p : p - 1;
    if (q < qe) load(q);
    for (; ok && q < qe; ++q) {
      double av[8], zv[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) av[i] = (double)an[i];
      if (q + 1 < qe) load(q + 1);
      ok = fetch(X + (size_t)q * kBlkW, cg, ps[q + 1] - ps[q], q >= S.p0 ? epoch : 0, q < p - 3, zv, err, wt.limit);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i & 1] = fma(av[i], zv[i], acc[i & 1]);
    }
    double s = acc[0] + acc[1];
    s += __shfl_xor_sync(kFull, s, 8);
    s += __shfl_xor_sync(kFull, s, 16);
    if (cg == 0) xs[par][row] = br - (row < w ? s : 0.0);
    if (!__syncthreads_and(ok)) return;
    double u[2] = {0.0, 0.0};
#pragma unroll
    for (int i = 0; i < 8; ++i) u[i & 1] = fma(Ai[i], xs[par][cg + 4 * i], u[i & 1]);
    if constexpr (kTriangles<T>) {
      double y = u[0] + u[1];
      y += __shfl_xor_sync(kFull, y, 8);
      y += __shfl_xor_sync(kFull, y, 16);
      if (cg == 0) ys[row] = y;
      __syncthreads();  // (ys is written again after the next panel's first barrier)
      u[0] = u[1] = 0.0;
#pragma unroll
      for (int i = 0; i < 8; ++i) u[i & 1] = fma(W[i], ys[cg + 4 * i], u[i & 1]);
    } else if (p > 0) {
      double zv[8];
      ok = fetch(X + (size_t)(p - 1) * kBlkW, cg, j0 - ps[p - 1], p - 1 >= S.p0 ? epoch : 0, false, zv, err, wt.limit);
#pragma unroll
      for (int i = 0; i < 8; ++i) u[i & 1] = fma(-W[i], zv[i], u[i & 1]);
    }
    double z = u[0] + u[1];
    z += __shfl_xor_sync(kFull, z, 8);
    z += __shfl_xor_sync(kFull, z, 16);
    if (cg == 0 && row < w && ok) {
      publish(X + (size_t)p * kBlkW + row, z, epoch);
      b[r * si] = z;
    }
  }
}
// The backward chain's contributions to the rows [lo, mid) above it, before the
// forward chain goes on through them: b[i] -= sum_j A(i, j) z(j) over the columns
// j >= mid that reach row i (physical numbering; z stands in b).  A warp per row.
template <class T>
__global__ void __launch_bounds__(256) blk_forward_mid_kernel(const T* __restrict__ ab, BandLayout L, int mid, int lo,
                                                              double* __restrict__ b, const int* __restrict__ gate) {
  if (gate && *gate) return;
  const int i = lo + blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= mid) return;
  const int jend = (int)min64b(L.n, (int64_t)i + L.ku + 1);
  double s = 0.0;
  for (int j = mid + lane; j < jend; j += 32) s += (double)ab[bix(L, i, j)] * b[j];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
  if (lane == 0) b[i] -= s;
}

// ---------------------------------------------------------------------------
// host side
constexpr int kApplyNR = 9;     // 32-row chunks per warp per pass of the bulk update (two warps per column)
constexpr int kColNR = 6;       // rows per thread per pass of the critical-path update

template <class T>
static size_t blk_apply_smem(const BandLayout& L, int w) {
  const size_t R = (size_t)w + L.kl;
  return ((size_t)w * R + 64 * kApplyNR) * sizeof(T) + 4 * R * sizeof(T) + 128 * sizeof(T) + 32 * sizeof(T) +
         32 * sizeof(int);  // Lp (+ padding) S Y rd sp
}

bool blk_plan(const std::vector<int>& blk_end, int wmax, int ku, BlkPlan& out) {
  const int n = (int)blk_end.size();
  out.ps.clear();
  out.ndfp = 0;
  out.wmax = 0;
  int j0 = 0;
  out.ps.push_back(0);
  while (j0 < n) {
    int j1 = j0;
    while (j1 < n && blk_end[j1] - j0 <= wmax) {
      out.ndfp = std::max(out.ndfp, blk_end[j1] - j1 - 1);
      j1 = blk_end[j1];
    }
    if (j1 == j0) return false;  // a block wider than wmax
    out.wmax = std::max(out.wmax, j1 - j0);
    out.ps.push_back(j1);
    j0 = j1;
  }
  out.kuf = ku + out.ndfp;
  return true;
}

// The backward chain takes the unknowns [mid, n), whole pivot blocks, so many that
// 2 kuf unknowns are left between the chains when the forward chain has done as
// many: until then a panel of the forward chain (it reaches kuf unknowns beyond
// itself) and one of the backward chain (it reaches down to mid - kuf) never touch
// the same entries.  pm: the forward chain's panel at which they meet; the panels
// before it reach no further than mid - kuf.  Panel pm's own block ends there too:
// the forward chain's factorising CTA does not wait at the meeting and may factorise
// panel pm before it, once the panels before pm have updated its columns.  (In a band
// with kuf < 32 a panel can be wider than its reach, so that this asks for more.)
// The chain of dependent panels is then n / 2 + kuf unknowns long instead of n; bands
// shorter than 10/3 kuf keep the one chain (LAG 8 x 8 at 3.6 kuf, six panels instead
// of eight and a meeting of all CTAs: 0.24 -> 0.19 ms; below, the meeting costs what
// the shorter chain saves).
bool blk_two_plan(const std::vector<int>& blk_end, const BandLayout& L, BlkPlan& out, std::vector<int>& ps0,
                  std::vector<int>& ps1, std::vector<int>& blk_end1) {
  const int n = (int)blk_end.size(), kuf = out.kuf, kl = L.kl;
  // the backward chain's fill takes rows up to kuf + kBlkW below the diagonal of a
  // band column; those beyond ldb are the first rows of the next one, unused there
  if (kl != L.ku || L.ldb <= 2 * ((int64_t)kuf + kBlkW) || 3 * (int64_t)n < 10 * (int64_t)kuf) return false;
  const int want = (n - 2 * kuf) / 2;  // unknowns of the backward chain
  int mid = n;
  std::vector<int> first(n);  // first unknown of each unknown's block
  for (int q = 0; q < n; ++q) first[q] = q > 0 && blk_end[q - 1] > q ? first[q - 1] : q;
  while (mid > 0 && n - first[mid - 1] <= want) mid = first[mid - 1];
  if (n - mid < 2 * kBlkW || mid < 2 * kBlkW) return false;
  BlkPlan a, b;
  std::vector<int> e0(blk_end.begin(), blk_end.begin() + mid);
  blk_end1.resize(n - mid);
  for (int j = 0; j < n - mid; ++j) blk_end1[j] = n - first[n - 1 - j];  // reversed: the block ends where it began
  if (!blk_plan(e0, out.wmax, kl, a) || !blk_plan(blk_end1, out.wmax, kl, b)) return false;
  ps0 = a.ps;
  ps1 = b.ps;
  out.mid = mid;
  out.pm = 0;
  while (out.pm < a.npan() && ps0[out.pm + 1] + kuf <= mid - kuf) ++out.pm;
  while (out.pm > 0 && ps0[out.pm + 1] > mid - kuf) --out.pm;
  return out.pm > 0;  // their panels are no wider than out.wmax
}

template <class T>
int blk_panel_width(const BandLayout& L, int cap) {
  for (int w : {32, 24, 16, 8}) {
    if (w > L.nb) continue;
    if (blk_apply_smem<T>(L, w) <= (size_t)cap && ((size_t)w + L.kl) * sizeof(double) + 10 * 1024 <= (size_t)cap)
      return w;
  }
  return 0;
}

template <class T>
int blk_lu_setup(const BandLayout& L) {
  int dev = 0, cap = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
  const int wmax = blk_panel_width<T>(L, cap);
  if (!wmax) return 0;
  if (cudaFuncSetAttribute(blk_apply_kernel<T, kApplyNR>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap) !=
          cudaSuccess ||
      cudaFuncSetAttribute(blk_apply_col_kernel<T, kColNR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           cap - 10 * 1024) != cudaSuccess)
    return 0;
  return wmax;
}

// Factor with node-block pivoting (and forward-substitute rhs when given).
// Lookahead on two streams: st2 updates the next panel's columns (one CTA
// each) and factors that panel while st carries the bulk of the update.
// With prof != nullptr it runs serially on st, recording prof[3p..3p+2].
template <class T>
int blk_lu_factor(T* ab, const BandLayout& L, const BlkPlan& B, int* perm_all, T* rdiag, int* info, T* rhs,
                  cudaStream_t st, cudaStream_t st2, cudaEvent_t* ev_pool, cudaEvent_t* prof) {
  const int npan = B.npan();
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int launches = 0;
  auto w_of = [&](int p) { return B.ps[p + 1] - B.ps[p]; };
  auto ncol_of = [&](int p) -> int {
    const int64_t j1 = B.ps[p + 1];
    return (int)(min64b(L.n, j1 + B.kuf) - j1);
  };
  auto panel = [&](int p, cudaStream_t s) {
    blk_panel_kernel<T><<<1, 32 * kPanelWarps, 0, s>>>(ab, L, B.ps[p], w_of(p), B.d_blk_end, perm_all + (size_t)p * kBlkW, rdiag,
                                          info);
    ++launches;
  };
  // columns [cb, ce) of the trailing block of panel p (relative to its end)
  auto apply = [&](int p, int cb, int ce, bool with_rhs, cudaStream_t s, bool narrow) {
    const int ncol = ce - cb;
    const int ntot = ncol + (with_rhs ? 1 : 0);
    if (ntot <= 0) return;
    const int64_t j0 = B.ps[p], c0 = B.ps[p + 1] + cb;
    const int w = w_of(p);
    const int* pm = perm_all + (size_t)p * kBlkW;
    if (narrow) {
      const size_t sm = ((size_t)w + L.kl) * sizeof(T);
      blk_apply_col_kernel<T, kColNR><<<ncol, 128, sm, s>>>(ab, L, j0, w, pm, rdiag, c0);
    } else {
      const int blocks = (int)min64b(sms, (ntot + 3) / 4);
      blk_apply_kernel<T, kApplyNR><<<blocks, 256, blk_apply_smem<T>(L, w), s>>>(
          ab, L, j0, w, pm, rdiag, with_rhs ? rhs : nullptr, c0, ncol);
    }
    ++launches;
  };
  if (prof || !st2) {
    for (int p = 0; p < npan; ++p) {
      if (prof) cudaEventRecord(prof[3 * p], st);
      panel(p, st);
      if (prof) cudaEventRecord(prof[3 * p + 1], st);
      apply(p, 0, ncol_of(p), rhs != nullptr, st, false);
      if (prof) cudaEventRecord(prof[3 * p + 2], st);
    }
    return launches;
  }
  cudaEvent_t* ev_panel = ev_pool;
  cudaEvent_t* ev_rest = ev_pool + npan;
  cudaEvent_t ev_start = ev_pool[2 * npan], ev_join = ev_pool[2 * npan + 1];
  cudaEventRecord(ev_start, st);
  cudaStreamWaitEvent(st2, ev_start, 0);
  panel(0, st2);
  cudaEventRecord(ev_panel[0], st2);
  for (int p = 0; p < npan; ++p) {
    const int nc = ncol_of(p);
    const int split = (p + 1 < npan) ? std::min(nc, w_of(p + 1)) : 0;
    cudaStreamWaitEvent(st, ev_panel[p], 0);
    apply(p, split, nc, rhs != nullptr, st, false);
    cudaEventRecord(ev_rest[p], st);
    if (p + 1 < npan) {
      if (p > 0) cudaStreamWaitEvent(st2, ev_rest[p - 1], 0);
      apply(p, 0, split, false, st2, true);
      panel(p + 1, st2);
      cudaEventRecord(ev_panel[p + 1], st2);
    }
  }
  cudaEventRecord(ev_join, st2);
  cudaStreamWaitEvent(st, ev_join, 0);
  return launches;
}

template <class T>
int blk_inverses(const T* ab, const BandLayout& L, const BlkPlan& B, bool two, const int* perm_all, const T* rdiag,
                 double* inv, cudaStream_t st) {
  const BlkChain &c0 = two ? B.two[0] : B.one, &c1 = B.two[1];
  const int b0 = (c0.npan + 3) / 4, b1 = two ? (c1.npan + 3) / 4 : 0;
  blk_inverses_kernel<T><<<b0 + b1, 128, 0, st>>>(ab, c0, c1, b0, L.kl, perm_all, rdiag, inv);
  return 1;
}
// One cooperative launch over spans a and (optionally) b, its CTAs shared out by their
// panels.  Where it is refused (then *coop = false) or *coop is false already: one(a),
// one(b), single-CTA launches.  Returns the launches.
template <class F, class G>
static int coop_spans(F&& launch, G&& one, const BlkSpan& a, const BlkSpan* b, int grid, bool* coop) {
  const int na = a.p1 - a.p0, nb = b ? b->p1 - b->p0 : 0;
  if (na + nb <= 0) return 0;
  if (*coop && nb > 0 && grid < 2)  // one after the other
    return coop_spans(launch, one, a, nullptr, grid, coop) + coop_spans(launch, one, *b, nullptr, grid, coop);
  if (*coop) {
    const int ga = std::min(na, nb > 0 ? grid / 2 : grid), gb = std::min(nb, grid - ga);
    if (launch(a, b ? *b : a, ga, ga + gb) == cudaSuccess) return 1;
    cudaGetLastError();
    *coop = false;
  }
  one(a);
  if (nb > 0) one(*b);
  return nb > 0 ? 2 : 1;
}
template <class T>
int blk_backward(const T* ab, const BlkPlan& B, bool two, double* y, SolveWord* xch, int64_t& epoch, int* err,
                 int& grid, cudaStream_t st, WaitTest wt, const int* gate) {
  int kuf = B.kuf, through = 0;
  bool coop = grid > 0;
  auto launch = [&](BlkSpan a, BlkSpan b, int split, int ctas) {
    if (wt.refuse >= 0 && through++ >= wt.refuse) return cudaErrorCooperativeLaunchTooLarge;
    ++epoch;
    void* args[] = {(void*)&ab,    (void*)&kuf, (void*)&a,  (void*)&b,   (void*)&split, (void*)&y, (void*)&xch,
                    (void*)&epoch, (void*)&err, (void*)&wt, (void*)&gate};
    return cudaLaunchCooperativeKernel((const void*)blk_backward_coop_kernel<T>, dim3(ctas), dim3(kSolveThreads), args, 0,
                                       st);
  };
  auto one = [&](const BlkSpan& s) { blk_backward_kernel<T><<<1, 1024, 0, st>>>(ab, kuf, s, y, gate); };
  int nl;
  if (!two) {
    nl = coop_spans(launch, one, BlkSpan{B.one, 0, B.one.npan}, nullptr, grid, &coop);
  } else {
    // the unknowns between the chains, then both chains side by side
    nl = coop_spans(launch, one, BlkSpan{B.two[0], B.pm, B.two[0].npan}, nullptr, grid, &coop);
    const BlkSpan b1{B.two[1], 0, B.two[1].npan};
    nl += coop_spans(launch, one, BlkSpan{B.two[0], 0, B.pm}, &b1, grid, &coop);
  }
  if (!coop) grid = 0;
  return nl;
}
template <class T>
int blk_forward(const T* ab, const BandLayout& L, const BlkPlan& B, bool two, const int* perm_all, const T* rdiag,
                const double* inv, double* b, SolveWord* xch, int64_t& epoch, int* err, int& grid, cudaStream_t st,
                WaitTest wt, const int* gate) {
  int kl = L.kl, through = 0;
  bool coop = grid > 0;
  auto launch = [&](BlkSpan s0, BlkSpan s1, int split, int ctas) {
    if (wt.refuse >= 0 && through++ >= wt.refuse) return cudaErrorCooperativeLaunchTooLarge;
    ++epoch;
    void* args[] = {(void*)&ab, (void*)&kl,  (void*)&s0,    (void*)&s1,  (void*)&split, (void*)&inv,
                    (void*)&b,  (void*)&xch, (void*)&epoch, (void*)&err, (void*)&wt,    (void*)&gate};
    return cudaLaunchCooperativeKernel((const void*)blk_forward_coop_kernel<T>, dim3(ctas), dim3(kSolveThreads), args, 0,
                                       st);
  };
  auto one = [&](const BlkSpan& s) { blk_forward_kernel<T><<<1, 1024, 0, st>>>(ab, kl, s, perm_all, rdiag, b, gate); };
  int nl;
  if (!two) {
    nl = coop_spans(launch, one, BlkSpan{B.one, 0, B.one.npan}, nullptr, grid, &coop);
  } else {
    const BlkSpan s1{B.two[1], 0, B.two[1].npan};
    nl = coop_spans(launch, one, BlkSpan{B.two[0], 0, B.pm}, &s1, grid, &coop);
    const int lo = std::max(0, B.mid - L.kl);
    blk_forward_mid_kernel<T><<<(B.mid - lo + 7) / 8, 256, 0, st>>>(ab, L, B.mid, lo, b, gate);
    nl += 1 + coop_spans(launch, one, BlkSpan{B.two[0], B.pm, B.two[0].npan}, nullptr, grid, &coop);
  }
  if (!coop) grid = 0;
  return nl;
}
// CTAs of the cooperative back substitution that can be resident at once
template <class T>
int blk_backward_grid() {
  int dev = 0, sms = 0, back = 0, forw = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&back, blk_backward_coop_kernel<T>, kSolveThreads, 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&forw, blk_forward_coop_kernel<T>, kSolveThreads, 0);
  return std::max(0, sms * std::min(std::min(back, forw), 1));
}

template int blk_panel_width<double>(const BandLayout&, int);
template int blk_panel_width<float>(const BandLayout&, int);
template int blk_lu_setup<double>(const BandLayout&);
template int blk_lu_setup<float>(const BandLayout&);
template int blk_lu_factor<double>(double*, const BandLayout&, const BlkPlan&, int*, double*, int*, double*,
                                   cudaStream_t, cudaStream_t, cudaEvent_t*, cudaEvent_t*);
template int blk_lu_factor<float>(float*, const BandLayout&, const BlkPlan&, int*, float*, int*, float*, cudaStream_t,
                                  cudaStream_t, cudaEvent_t*, cudaEvent_t*);
template int blk_inverses<double>(const double*, const BandLayout&, const BlkPlan&, bool, const int*,
                                          const double*, double*, cudaStream_t);
template int blk_inverses<float>(const float*, const BandLayout&, const BlkPlan&, bool, const int*, const float*,
                                         double*, cudaStream_t);
template int blk_backward<double>(const double*, const BlkPlan&, bool, double*, SolveWord*, int64_t&, int*, int&,
                                  cudaStream_t, WaitTest, const int*);
template int blk_backward<float>(const float*, const BlkPlan&, bool, double*, SolveWord*, int64_t&, int*, int&,
                                 cudaStream_t, WaitTest, const int*);
template int blk_backward_grid<double>();
template int blk_backward_grid<float>();
template int blk_forward<double>(const double*, const BandLayout&, const BlkPlan&, bool, const int*, const double*,
                                 const double*, double*, SolveWord*, int64_t&, int*, int&, cudaStream_t, WaitTest,
                                 const int*);
template int blk_forward<float>(const float*, const BandLayout&, const BlkPlan&, bool, const int*, const float*,
                                const double*, double*, SolveWord*, int64_t&, int*, int&, cudaStream_t, WaitTest,
                                const int*);

}  // namespace mafem

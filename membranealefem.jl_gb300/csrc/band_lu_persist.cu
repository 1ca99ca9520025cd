// band_lu_persist.cu -- the node-block pivoted banded LU (band_lu_blk.cu) as
// ONE persistent cooperative launch per factorisation.
//
// Roles.  CTA G-1 only factorises panels; CTA G-2 carries the right-hand side
// (when there is one).  Column c is owned by worker CTA c mod GW for the
// whole factorisation, so the updates of a column by successive panels run in
// order on one CTA without any flag; a worker has ~(ku + ndfp) / GW columns
// per panel.
//
// Per panel p every worker with columns in p's trailing range:
//   1. waits for a21cnt[p] (every column of p has its rows below the diagonal
//      block final) and has p's A21 and its own columns copied to shared memory,
//      beside the panel's factorisation,
//   2. waits for pdone[p] (panel p factorised) and loads a row of L11\U11 per
//      lane, with the permutation and 1/U(j,j), into registers,
//   3. runs its columns' triangular solves (one warp each),
//   4. for its column of panel p + 1 (at most one): updates the 32 rows the
//      next factorisation reads, bumps critcnt[p + 1], then the rows below,
//      bumps a21cnt[p + 1],
//   5. updates the rows of its other columns.
// The factorising CTA waits for critcnt[p + 1] = w(p + 1), factorises panel
// p + 1 in registers and publishes pdone[p + 1].  So the critical path per
// panel is: the block's load, one triangular solve, 32 rows of one column, the
// panel factorisation, and two flag hand-overs -- no kernel launches.
//
// Flags and counters go on across factorisations: pdone[t] holds the epoch that set
// it, critcnt[t] / a21cnt[t] reach epoch * w(t), modulo 2^32; a wait compares
// differences, so they may wrap.  All waits are bounded (kSpinLimit polls) and abort
// every CTA through *err; the host then starts the counters afresh (blk_persist_count).
//
// From both ends (FP64 with a right-hand side, and FP32; blk_two_plan).  A panel takes
// 19.2 us of dependent steps in FP64 (15 us in FP32) however narrow the band is, so
// the number of panels in a row is what bounds narrow bands, and a band's last unknowns can be eliminated beside its
// first ones: two chains, each on half of the CTAs with its own factorising CTA,
// meet in the middle.  The second numbers rows and columns from the last unknown,
// so it is the same code on descending addresses (its fill and Y lie below the
// diagonal).  Up to panel pm of the first one the two touch different entries; there
// all CTAs meet (*bdone) and share the columns of what is left, 2 kuf unknowns.
// The chain of dependent panels is n / 2 + kuf unknowns long instead of n.
// Factorisation, ms, one chain -> two (FP64; FP32):
//   ALEVB 17 x 17 (n 2410, kuf 310)     1.50 -> 1.01; 1.02 -> 0.65
//   ALEVB 32 x 32 (n 8410, kuf 550)     6.77 -> 5.86; 3.58 -> 2.21
//   ALEVB 64 x 64 (n 33242, kuf 1062)   94.3 -> 81.6
// In FP64 the last two are bound by the FP64 units (1.25 TFLOP/s: 4.0 and 60 ms for
// the 2 n kl kuf operations): there the gain is that one chain's hand-overs hide behind
// the other's updates.  A worker has twice the columns while the chains run beside
// each other (kMaxCols, and eight staged at once where shared memory allows).
//
// L1 coherence.  Band entries written by other SMs are read by TMA or with L2-only
// loads (__ldcg), as are the pivot data; flags with ld.acquire.

#include "band_lu_common.cuh"

namespace mafem {

namespace {

template <class T>
struct PersistArgs {
  T* ab;
  BlkChain c[2];              // two chains: c[0] forward, side by side on CTAs [0, split), c[1] backward on the others
  int split;
  int n, off, kl, kuf;
  int rmax, wmax, nslot;      // rmax = wmax + kl: rows of a staged panel column
  int pm;
  unsigned bdone_target;      // panel pm of c[0] and later ones: after *bdone has reached the target, but for
                              // the factorising CTA (pm's block lies clear of c[1], blk_two_plan)
  int* bdone;
  int* perm_all;
  T* rdiag;
  int* info;
  T* rhs;
  int* pdone;
  int* critcnt;
  int* a21cnt;
  unsigned epoch;
  int* err;
  int limit;        // polls before a wait gives up
  long long* trace;  // optional: kTraceSlots device-clock stamps per panel (diagnostics)
};
constexpr int kTraceSlots = 12;
constexpr int kMaxCols = 16;  // columns a worker handles per panel (more: the grid is too small)
__device__ __forceinline__ void stamp(long long* trace, int t, int slot) {
  if (trace && threadIdx.x == 0) {
    long long v;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v));
    trace[(size_t)t * kTraceSlots + slot] = v;
  }
}

// thread 0 waits until *p has reached target (modulo 2^32); false (uniform over the CTA) on timeout / abort
__device__ __forceinline__ bool wait_geq(const int* p, unsigned target, int* err, int limit, int* s_ok) {
  if (threadIdx.x == 0) {
    int ok = 1;
    for (int it = 0; (int)((unsigned)ld_acquire(p) - target) < 0; ++it) {
      if (it > limit || ((it & 31) == 31 && *(volatile int*)err)) {  // (a look at it delays the next poll)
        atomicCAS(err, 0, 1);
        ok = 0;
        break;
      }
      __nanosleep(32);
    }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

}  // namespace

enum Role { kWorker, kRhs, kFactor };
// Panels [p0, p1) of one chain by one CTA: worker `me` of GW, the CTA of the
// right-hand side or the factorising one.  REV: the chain that eliminates from the
// last unknown; rows and columns are numbered in the chain's order, so row i of a
// column (and of its copy in shared memory) lies at a descending address.  false
// after a wait ran out.
template <class T, bool REV, bool TWO>
__device__ __forceinline__ bool persist_panels(const PersistArgs<T>& a, const BlkChain& C, int p0, int p1, int me, int GW,
                                               Role role, unsigned char* smem_raw, uint64_t* s_bar, uint32_t& ph) {
  constexpr int SG = REV ? -1 : 1;  // address step from a row to the next
  __shared__ T s_l[2][32];
  __shared__ int s_p[2];
  __shared__ int s_ok;
  __shared__ int s_col[kMaxCols];  // this panel's columns (-1: the right-hand side)
  __shared__ T s_part[4][32];      // partial sums of the critical rows
  const int* __restrict__ ps = C.ps;
  const int npan = C.npan;
  const int64_t sj = C.sj;
  T* const ab = a.ab + C.org;                             // element (i, j) at ab[i SG + j sj]
  T* const rhs = a.rhs ? a.rhs + C.vorg : nullptr;        // element i at rhs[i SG]
  int* const pdone = a.pdone + C.pbase;
  int* const critcnt = a.critcnt + C.pbase;
  int* const a21cnt = a.a21cnt + C.pbase;
  int* const perm_all = a.perm_all + (size_t)C.pbase * kBlkW;
  T* const rdiag = a.rdiag + C.rbase;
  const bool rhs_cta = role == kRhs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  if (role == kFactor) {
    for (int t = p0; t < p1; ++t) {
      const int j0 = ps[t], wt = ps[t + 1] - j0;
      stamp(a.trace, t, 0);
      if (t > 0 && !wait_geq(critcnt + t, a.epoch * wt, a.err, a.limit, &s_ok)) return false;
      stamp(a.trace, t, 1);
      blk_panel_factor<T, true>(ab + j0 * SG + j0 * sj, SG, sj, j0, wt, REV ? a.n - j0 : j0 + 1, SG, C.blk_end + j0,
                                perm_all + (size_t)t * kBlkW, rdiag + j0, a.info, s_l, s_p);
      __syncthreads();
      if (tid == 0) st_release(pdone + t, (int)a.epoch);
      stamp(a.trace, t, 2);
    }
    return true;
  }

  // Shared memory.  Column slots of LDp elements: the panel's w columns (Lp)
  // and nslot column segments (S).  A segment starting at global element index
  // g is placed at slot offset g mod E (E elements = 16 bytes), so that its
  // 16-byte-aligned global elements land 16-byte-aligned in shared memory and
  // the bulk of it can be one TMA copy (cp.async.bulk); the at most E - 1
  // elements before and after the aligned bulk are loaded directly.
  constexpr int E = 16 / (int)sizeof(T);
  const int LDp = (a.rmax + 2 * E - 1) / E * E;
  T* Lp = reinterpret_cast<T*>(smem_raw) + (TWO ? 64 : 0);  // [kBlkW][LDp] (64 around it: chunk reads past R)
  T* S = Lp + (size_t)a.wmax * LDp + 64;              // [nslot][LDp] column segments
  T* Y = S + (size_t)a.nslot * LDp;                   // [nslot][32]
  __shared__ int s_sb[8];                             // row 0 of the segments, from S
  int R = 0;  // rows of the current panel's columns
  // panel column k, row 0 (row r: SG r further)
  auto lpa = [&](int k) -> T* {
    return REV ? Lp + k * LDp + ((a.off + k - R + 1) & (E - 1)) + R - 1 : Lp + k * LDp + ((a.off - k) & (E - 1));
  };
  // Copy of n elements src[0..n) -> dst[0..n) (same address phase mod 16 bytes): mode 0 returns the bytes
  // of the aligned bulk, mode 1 issues it as one TMA copy on `bar`, mode 2 loads the unaligned head and
  // tail (at most E - 1 elements each) directly -- after every TMA copy is in flight.
  auto seg_copy = [&](T* dst, const T* src, int n, uint64_t* bar, int mode) -> uint32_t {
    const int g = (int)(((uintptr_t)src / sizeof(T)) & (E - 1));
    const int h = min(n, (E - g) & (E - 1));
    const int nb = max(0, (n - h) / E * E);
    if (mode == 1 && nb > 0) tma_load_1d(dst + h, src + h, (uint32_t)(nb * sizeof(T)), bar);
    if (mode == 2) {
      T hv[E - 1], tv[E - 1];
#pragma unroll
      for (int i = 0; i < E - 1; ++i) {
        hv[i] = i < h ? __ldcg(src + i) : T(0);
        tv[i] = h + nb + i < n ? __ldcg(src + h + nb + i) : T(0);
      }
#pragma unroll
      for (int i = 0; i < E - 1; ++i) {
        if (i < h) dst[i] = hv[i];
        if (h + nb + i < n) dst[h + nb + i] = tv[i];
      }
    }
    return (uint32_t)(nb * sizeof(T));
  };
  auto wait_bar = [&](uint64_t* bar, uint32_t& ph) -> bool {
    int ok = 1;
    for (int it = 0; !mbar_try_wait(bar, ph); ++it)
      if (it > kSpinLimit) {
        ok = 0;
        atomicCAS(a.err, 0, 3);
        break;
      }
    ph ^= 1u;
    return __syncthreads_and(ok) != 0;
  };

  for (int p = p0; p < p1; ++p) {
    const int j0 = ps[p], j1 = ps[p + 1];
    const int w = j1 - j0;
    R = min(C.n - j0, w + a.kl);
    const int jend = min(C.n, j1 + a.kuf);
    const int jn = p + 1 < npan ? ps[p + 2] : j1;  // panel p + 1 = columns [j1, jn)
    const int cend = max(jend, jn);
    const bool is_rhs = rhs_cta;
    const int cfirst = rhs_cta ? cend : j1 + (((me - j1) % GW) + GW) % GW;
    if (cfirst >= cend && !is_rhs) continue;
    const bool tr_owner = !TWO && p + 1 < npan && me == j1 % GW;
    if (tr_owner) stamp(a.trace, p + 1, 3);
    if (p > 0 && !wait_geq(a21cnt + p, a.epoch * w, a.err, a.limit, &s_ok)) return false;
    const int nch = (R - w + 31) / 32;  // 32-row chunks below the diagonal block
    // columns of this panel: the one of panel p + 1 first, then the others, then the right-hand side
    const int nown = cfirst < cend ? (int)((cend - 1 - cfirst) / GW) + 1 : 0;
    const int ncol = nown + (is_rhs ? 1 : 0);
    if (ncol > kMaxCols || (nown > 1 && cfirst + GW < jn)) {  // grid too small (the host setup rules this out)
      if (tid == 0) atomicCAS(a.err, 0, 2);
      return false;
    }
    if (tid < nown) s_col[tid] = cfirst + tid * GW;
    if (tid == 0 && is_rhs) s_col[nown] = -1;
    fence_proxy_async_smem();  // earlier reads / writes of the buffers before the TMA writes below
    __syncthreads();
    // Warp 0 issues the copies, while the panel's diagonal block is still being
    // factorised: lane l the rows below it (A21) of panel column l and the segment of
    // this CTA's column l.
    auto issue_cols = [&](int b0, int nb, bool with_panel) {
      if (warp != 0) return;
      fence_proxy_async_global();  // data written by ordinary stores (here or, before a flag, elsewhere)
      T* sd = nullptr;
      const T* ss = nullptr;
      if (lane < nb) {
        const int c = s_col[b0 + lane];
        ss = c < 0 ? rhs + j0 * SG : ab + j0 * SG + c * sj;
        if (REV) ss -= R - 1;  // the segment's lowest address
        const int off = (int)(((uintptr_t)ss / sizeof(T)) & (E - 1));
        s_sb[lane] = lane * LDp + off + (REV ? R - 1 : 0);
        sd = S + lane * LDp + off;
      }
      const bool pc = with_panel && lane < w && R > w;
      const int lo = REV ? 1 - R : w;  // rows [w, R), from the lowest address
      T* const pd = lpa(lane) + lo;
      const T* const pd_src = ab + j0 * SG + (j0 + lane) * sj + lo;
      uint32_t bytes = 0;
      if (lane < nb) bytes += seg_copy(sd, ss, R, s_bar, 0);
      if (pc) bytes += seg_copy(pd, pd_src, R - w, s_bar, 0);
      for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(kFull, bytes, o);
      if (lane == 0) mbar_arrive_expect_tx(s_bar, bytes);
      __syncwarp();
      for (int mode = 1; mode <= 2; ++mode) {
        if (lane < nb) seg_copy(sd, ss, R, s_bar, mode);
        if (pc) seg_copy(pd, pd_src, R - w, s_bar, mode);
      }
    };
    issue_cols(0, min(a.nslot, ncol), true);
    if (!wait_geq(pdone + p, a.epoch, a.err, a.limit, &s_ok)) {
      wait_bar(s_bar, ph);  // no copy in flight when the CTA ends
      return false;
    }
    if (tr_owner) stamp(a.trace, p + 1, 4);

    for (int b0 = 0; b0 < ncol; b0 += a.nslot) {
      const int nb = min(a.nslot, ncol - b0);
      if (b0 > 0) {  // later batches (small grids only)
        fence_proxy_async_smem();
        __syncthreads();
        issue_cols(b0, nb, false);
      }
      // this lane's row of the diagonal block in registers (nothing to load on the
      // dependency chains): L(lane, k) for k < lane, U(lane, k) for k > lane
      T Tr[32], rl = T(0);
      int pr = 0;
      if (warp < nb) {
        const T* row = ab + (j0 + min(lane, w - 1)) * SG + j0 * sj;
#pragma unroll
        for (int k = 0; k < 32; ++k) Tr[k] = (k < w && lane < w) ? __ldcg(row + k * sj) : T(0);
        if (lane < w) {
          rl = __ldcg(rdiag + j0 + lane);
          pr = __ldcg(perm_all + (size_t)p * kBlkW + lane);
        }
      }
      if (!wait_bar(s_bar, ph)) return false;
      if (tr_owner && b0 == 0) stamp(a.trace, p + 1, 5);
      // triangular solves, one warp per column: u = L11^-1 P s[0:w], y = U11^-1 u (kept as Y in place of A12)
      if (warp < a.nslot) {
        T v = T(0);
        if (warp < nb) {
          const int c = s_col[b0 + warp];
          const T* s = S + s_sb[warp];
          T* dst = c < 0 ? rhs + j0 * SG : ab + j0 * SG + c * sj;
          T x = lane < w ? s[pr * SG] : T(0);  // row `lane` of the permuted top
#pragma unroll
          for (int k = 0; k < 32; ++k) {
            if (k < w) {
              const T xk = __shfl_sync(kFull, x, k);
              if (lane > k) x = fma(-Tr[k], xk, x);
            }
          }
          // y = U11^-1 u with this lane's U row pre-scaled by 1/U(lane, lane)
          // (unit diagonal): each step is one shuffle and one FMA
#pragma unroll
          for (int k = 0; k < 32; ++k)
            if (k > lane) Tr[k] *= rl;
          v = x * rl;
#pragma unroll
          for (int k = 31; k >= 0; --k) {
            if (k < w) {
              const T yk = __shfl_sync(kFull, v, k);
              if (lane < k) v = fma(-Tr[k], yk, v);
            }
          }
          if (lane < w) dst[lane * SG] = v;  // Y (the right-hand side: z); not read again by this kernel
        }
        Y[warp * 32 + lane] = (warp < nb && lane < w) ? v : T(0);
      }
      __syncthreads();
      if (tr_owner && b0 == 0) stamp(a.trace, p + 1, 6);
      // rows [w, R): s -= A21 y, 32-row chunks; tasks (column qq, chunk ci) in [q0, q1) x [c0, c1)
      auto rows = [&](int q0, int q1, int c0, int c1) {
        const int nq = q1 - q0, ntask = nq * (c1 - c0);
        for (int tk = warp; tk < ntask; tk += 8) {
          const int qq = q0 + tk % nq, ci = c0 + tk / nq;
          const int r = w + 32 * ci + lane;
          const T* s = S + s_sb[qq];
          const T* yq = Y + qq * 32;
          T acc = s[min(r, R - 1) * SG];
          for (int k = 0; k < w; ++k) acc = fma(-lpa(k)[r * SG], yq[k], acc);
          if (r < R) {
            const int c = s_col[b0 + qq];
            T* dst = c < 0 ? rhs + j0 * SG : ab + j0 * SG + c * sj;
            dst[r * SG] = acc;
          }
        }
        fence_proxy_async_global();  // these rows are read by TMA later
        __syncthreads();
      };
      int q0 = 0;
      if (b0 == 0 && s_col[0] >= j1 && s_col[0] < jn) {  // the column of panel p + 1
        const bool reach = s_col[0] < jend;
        if (reach && nch > 0) {  // chunk 0 (the rows panel p + 1 factorises): k split over 4 warps
          const int r = w + lane;
          if (warp < 4) {
            T part = T(0);
            for (int k = 8 * warp; k < min(w, 8 * warp + 8); ++k) part = fma(-lpa(k)[r * SG], Y[k], part);
            s_part[warp][lane] = part;
          }
          __syncthreads();
          if (warp == 0 && r < R) {
            T* dst = ab + j0 * SG + s_col[0] * sj;
            dst[r * SG] = S[s_sb[0] + min(r, R - 1) * SG] +
                     ((s_part[0][lane] + s_part[1][lane]) + (s_part[2][lane] + s_part[3][lane]));
          }
          __threadfence();  // read by the factorising CTA with L2-only loads (and rewritten by it before any TMA read)
          __syncthreads();
        }
        if (tid == 0) atomicAdd(critcnt + p + 1, 1);
        if (tr_owner) stamp(a.trace, p + 1, 7);
        if (reach) {
          rows(0, 1, min(1, nch), nch);
          __threadfence();
          __syncthreads();
        }
        if (tid == 0) atomicAdd(a21cnt + p + 1, 1);
        if (tr_owner) stamp(a.trace, p + 1, 8);
        q0 = 1;
      }
      if (q0 < nb) rows(q0, nb, 0, nch);
    }
  }
  return true;
}

// With a right-hand side the last CTA but one of a chain carries it alone (its extra
// column would otherwise make one worker late every few panels); the last factorises.
// kSideBySide: each chain on its own CTAs, the forward one up to panel pm, then the rest on all of them.
// kInTurn, on too few CTAs for that: all of them run the backward chain, meet, and run the forward one.  Every
// entry sees the same updates in the same order as side by side: the results do not depend on the number of
// CTAs.  (A batch keeps its patches on their smallest grids; one step of a batch of FP64 patches against the
// one chain there: 24 of 8 x 8 to 16 x 16 56 -> 29 ms, 12 of 17 x 17 ALEVB 55.6 -> 51.4 ms, 8 of 32 x 32 375 ->
// 334 ms.)  A kernel of its own: with both forms in one, side by side cost 64 x 64 ALEVB 82.5 instead of 81.6 ms
// and the FP32 32 x 32 patch 2.30 instead of 2.21.
enum Form { kOneChain, kSideBySide, kInTurn };
template <class T, Form FORM>
__global__ void __launch_bounds__(256, 1) blk_factor_persist_kernel(PersistArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t s_bar;  // completion of the TMA copies
  [[maybe_unused]] __shared__ int s_ok;
  const int G = (int)gridDim.x;
  const int nx = a.rhs ? 2 : 1;  // CTAs of a chain that own no columns
  int me = blockIdx.x;
  if (threadIdx.x == 0) {
    mbar_init(&s_bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  uint32_t ph = 0;
  auto role_of = [&](int i, int ctas) { return i == ctas - 1 ? kFactor : a.rhs && i == ctas - 2 ? kRhs : kWorker; };
  // between the chains: each side reads what the other one updated
  [[maybe_unused]] auto meet = [&]() {
    fence_proxy_async_global();
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(a.bdone, 1);
    return wait_geq(a.bdone, a.bdone_target, a.err, a.limit, &s_ok);
  };
  if constexpr (FORM == kOneChain) {
    persist_panels<T, false, false>(a, a.c[0], 0, a.c[0].npan, me, G - nx, role_of(me, G), smem_raw, &s_bar, ph);
  } else if constexpr (FORM == kInTurn) {
    const Role role = role_of(me, G);
    if (!persist_panels<T, true, true>(a, a.c[1], 0, a.c[1].npan, me, G - nx, role, smem_raw, &s_bar, ph)) return;
    if (!meet()) return;
    persist_panels<T, false, true>(a, a.c[0], 0, a.c[0].npan, me, G - nx, role, smem_raw, &s_bar, ph);
  } else {
    const bool rev = me >= a.split;
    const int G0 = rev ? G - a.split : a.split;
    if (rev) me -= a.split;
    Role role = role_of(me, G0);
    if (rev) {
      if (!persist_panels<T, true, true>(a, a.c[1], 0, a.c[1].npan, me, G0 - nx, role, smem_raw, &s_bar, ph)) return;
    }
    // the forward chain's factorising CTA goes on without the meeting: of its panels pm alone can come before
    // it (later ones wait for columns that are updated after it), and pm's block is out of c[1]'s reach
#pragma unroll 1
    for (int half = rev || role == kFactor ? 1 : 0; half < 2; ++half) {
      if (half == 1 && (rev || role != kFactor)) {
        if (!meet()) return;
        if (rev) {  // the columns change hands
          role = kWorker;
          me += a.split - nx;
        }
      }
      const int p0 = half == 1 && role != kFactor ? a.pm : 0, p1 = half == 0 ? a.pm : a.c[0].npan;
      if (!persist_panels<T, false, true>(a, a.c[0], p0, p1, me, half == 0 ? a.split - nx : G - nx, role, smem_raw, &s_bar,
                                          ph))
        return;
    }
  }
}

// ---------------------------------------------------------------------------
// host side
template <class T>
static size_t persist_smem(const BandLayout& L, int wmax, int nslot, bool two) {
  constexpr int E = 16 / (int)sizeof(T);
  const size_t rmax = (size_t)wmax + L.kl;
  const size_t ldp = (rmax + 2 * E - 1) / E * E;
  return ((two ? 64 : 0) + (size_t)wmax * ldp + 64 + nslot * (ldp + 32)) * sizeof(T);
}

// The kernel's limit of dynamic shared memory belongs to the process, not to a handle:
// it is always set to all that the device has (cap) beside the kernel's static part, so
// that no handle's set-up takes away what another one's launches ask for.
template <class T, Form FORM>
static bool persist_fits(size_t sm, int cap) {
  int per = 0;
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, blk_factor_persist_kernel<T, FORM>) != cudaSuccess) return false;
  const int dyn = cap - (int)fa.sharedSizeBytes;
  return sm <= (size_t)dyn &&
         cudaFuncSetAttribute(blk_factor_persist_kernel<T, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) ==
             cudaSuccess &&
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, blk_factor_persist_kernel<T, FORM>, 256, sm) ==
             cudaSuccess &&
         per >= 1;
}

template <class T>
int blk_persist_setup(const BandLayout& L, const BlkPlan& B, BlkPersist& S) {
  int dev = 0, sms = 0, cap = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  int coop = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  S.smem = persist_smem<T>(L, B.wmax, 4, false);
  if (!coop || S.smem + 12 * 1024 > (size_t)cap || B.wmax > kBlkW) return 0;  // + static shared memory
  if (!persist_fits<T, kOneChain>(S.smem, cap)) return 0;
  // The smallest grid: workers with at most kFewCols columns each per panel (columns c
  // of the trailing range, owned by c mod GW, plus the right-hand side), and at least
  // one per column of the widest panel (a worker owns at most one column of the next
  // panel); + the right-hand-side CTA + the factorising CTA
  constexpr int kFewCols = 8;
  S.grid = sms;
  S.min_grid = std::max((int)((B.kuf + B.wmax + 1 + kFewCols - 1) / kFewCols), B.wmax) + 2;
  if (S.grid < S.min_grid) return S.grid = 0;
  S.max_grid = S.grid;
  // two chains: each on half of the CTAs, a worker with up to kMaxCols columns per panel (on fewer CTAs one
  // chain after the other); not where the device is too small for them to run side by side
  S.min_two = 0;
  for (int nslot : {8, 4}) {
    if (!B.has_two) break;
    S.nslot2 = nslot;
    S.smem2 = persist_smem<T>(L, B.wmax, nslot, true);
    if (S.smem2 + 12 * 1024 <= (size_t)cap && persist_fits<T, kSideBySide>(S.smem2, cap)) {
      S.min_two = 2 * (std::max((int)((B.kuf + B.wmax + 1 + kMaxCols - 1) / kMaxCols), B.wmax) + 2);
      if (S.min_two > S.max_grid) S.min_two = 0;
      break;
    }
  }
  cudaGetLastError();
  return S.grid;
}

template <class T>
int blk_lu_factor_persist(T* ab, const BandLayout& L, const BlkPlan& B, BlkPersist& S, bool two, int* perm_all,
                          T* rdiag, int* info, T* rhs, int* err, cudaStream_t st, long long* trace) {
  if (S.refuse) return -1;
  PersistArgs<T> a;
  a.ab = ab;
  a.c[0] = two ? B.two[0] : B.one;
  a.c[1] = B.two[1];
  const int after = two ? B.npan() : 0;  // the two chains' flags stand after the one chain's
  const Form form = !two ? kOneChain : S.grid >= S.min_two ? kSideBySide : kInTurn;
  if (form == kInTurn && !S.turn_ready) {  // not at every handle's creation: the kernel is loaded by its first use
    int dev = 0, cap = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        !persist_fits<T, kInTurn>(S.smem2, cap))
      return -1;
    S.turn_ready = true;
  }
  a.split = (S.grid + 1) / 2;
  a.n = (int)L.n;
  a.off = (int)L.off;
  a.kl = L.kl;
  a.kuf = B.kuf;
  a.rmax = B.wmax + (int)L.kl;
  a.wmax = B.wmax;
  a.nslot = two ? S.nslot2 : 4;
  a.pm = B.pm;
  a.bdone = S.d_bdone;
  a.bdone_target = S.bdone + S.grid - (form == kSideBySide);  // all CTAs, side by side but the forward chain's factorising one
  a.perm_all = perm_all;
  a.rdiag = rdiag;
  a.info = info;
  a.rhs = rhs;
  a.pdone = S.d_pdone + after;
  a.critcnt = S.d_critcnt + after;
  a.a21cnt = S.d_a21cnt + after;
  a.epoch = S.epoch[two] + 1;
  a.err = err;
  a.limit = S.limit > 0 ? S.limit : kSpinLimit;
  a.trace = two ? nullptr : trace;
  void* args[] = {(void*)&a};
  const void* fn = form == kOneChain     ? (const void*)blk_factor_persist_kernel<T, kOneChain>
                   : form == kSideBySide ? (const void*)blk_factor_persist_kernel<T, kSideBySide>
                                         : (const void*)blk_factor_persist_kernel<T, kInTurn>;
  if (cudaLaunchCooperativeKernel(fn, dim3(S.grid), dim3(256), args, two ? S.smem2 : S.smem, st) != cudaSuccess) return -1;
  S.epoch[two] = a.epoch;
  if (two) S.bdone = a.bdone_target;
  return 1;
}

cudaError_t blk_persist_count(const BlkPlan& B, BlkPersist& S, unsigned count, unsigned missing, cudaStream_t st) {
  const std::vector<int>* ps[3] = {&B.ps, &B.ps0, &B.ps1};
  std::vector<unsigned> v[2];  // pdone; critcnt and a21cnt
  for (const auto* q : ps)
    for (size_t t = 0; t + 1 < q->size(); ++t) {
      v[0].push_back(count);
      v[1].push_back(count * (unsigned)((*q)[t + 1] - (*q)[t]));
    }
  S.epoch[0] = S.epoch[1] = S.bdone = count;
  const unsigned met = count - missing;
  cudaError_t e = cudaMemcpyAsync(S.d_bdone, &met, sizeof met, cudaMemcpyHostToDevice, st);
  int* dst[3] = {S.d_pdone, S.d_critcnt, S.d_a21cnt};
  for (int k = 0; k < 3 && e == cudaSuccess; ++k) {
    const auto& w = v[k > 0];
    e = cudaMemcpyAsync(dst[k], w.data(), w.size() * sizeof(unsigned), cudaMemcpyHostToDevice, st);
  }
  return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

template int blk_persist_setup<double>(const BandLayout&, const BlkPlan&, BlkPersist&);
template int blk_persist_setup<float>(const BandLayout&, const BlkPlan&, BlkPersist&);
template int blk_lu_factor_persist<double>(double*, const BandLayout&, const BlkPlan&, BlkPersist&, bool, int*, double*,
                                           int*, double*, int*, cudaStream_t, long long*);
template int blk_lu_factor_persist<float>(float*, const BandLayout&, const BlkPlan&, BlkPersist&, bool, int*, float*,
                                          int*, float*, int*, cudaStream_t, long long*);

}  // namespace mafem

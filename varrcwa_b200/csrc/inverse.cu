// Batched in-place matrix inversion: Gauss-Jordan with partial (row) pivoting.
//
// The reference inverts through Eigen PartialPivLU (explicit inverse of
// I - rdu*Rud, src/core/RedhefferIntegrator.cpp:267-270) and uses LU solves
// elsewhere; here every W^{-1}X / M^{-1}X of the hot path is an explicit
// inverse followed by a tensor-core GEMM (same 8n^3 flops as getrf+getrs).
//
// Small matrices stay in one CTA's registers; larger ones are reduced a panel
// at a time, the panel's accumulated row operations applied to every other
// column as one rank-w update on the tensor cores.
#include "common.cuh"
#include "kernels.h"

namespace vrc {
namespace {

// ---------------------------------------------------------------------------
// n <= 96: one CTA per matrix, the matrix in registers (rows over the lanes,
// columns over the warps).  Rows are never exchanged: step k takes as pivot row
// the largest entry of column k among the rows not yet used, and the permutation
// comes out with the stores.  A step passes one barrier: the warp that owns the
// next column updates it first, finds its pivot and the reciprocal while the
// others still update, and hands all three on through shared memory; the pivot's
// row comes from the lane that holds it.  Bound by the chain of a step (row,
// update of a column, search, reciprocal: 0.7 us at n = 25, 1.1 at 96), also with
// the SMs full (600 at n = 96: issue 40%, the FP64 pipe 34%, barriers first among
// the stalls).
// ---------------------------------------------------------------------------
constexpr int ZS_MAXN = 96;

// bits of infinity, 1e-150 and 1e150
constexpr unsigned long long INF_BITS = 0x7ff0000000000000ull, MID_LO = 0x20ca2fe76a3f9475ull,
                             MID_HI = 0x5f138d352e5096afull;

__device__ __forceinline__ cplx cinv_mid(cplx b) {  // the plain form of cinv_fast
  const double r = 1.0 / (b.x * b.x + b.y * b.y);
  return mk(b.x * r, -b.y * r);
}

template <int R, int W>
__global__ void __launch_bounds__(32 * W)
    zinv_small_kernel(cplx* const* __restrict__ mats, int n, int* __restrict__ status) {
  constexpr int C = 32 * R / W;  // columns of a warp: W c + warp
  __shared__ cplx col[2][32 * R], row[W][C], inv[2];
  __shared__ int prow[32 * R];
  cplx* g = mats[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const cplx zero = mk(0.0, 0.0);
  cplx a[R][C], x[R];
  bool used[R], bad = false;
  int step[R];  // the step that this row was the pivot of
  // the largest |re| + |im| of column k in x, by its high word, then its low
  // word; meanwhile each lane takes the reciprocal of its own candidate
  const auto search = [&](int k) {
    cplx xb = zero;
    unsigned long long best = 0;  // 1 + the bits of the candidate (as integers they order alike)
    int hb = 0;
#pragma unroll
    for (int h = 0; h < R; ++h) {
      col[k & 1][lane + 32 * h] = x[h];
      const unsigned long long bits = (unsigned long long)__double_as_longlong(cabs1(x[h]));
      const unsigned long long key = used[h] ? 0 : bits > INF_BITS ? 1 : bits + 1;  // (a NaN counts as zero)
      if (key > best) {
        best = key;
        xb = x[h];
        hb = h;
      }
    }
    const bool ok = best > 1 && best <= INF_BITS;
    const cplx ib = best - MID_LO < MID_HI - MID_LO ? cinv_mid(xb) : ok ? cinv(xb) : mk(1.0, 0.0);
    const unsigned hi = (unsigned)(best >> 32), lo = (unsigned)best;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    const int p = __ffs(__ballot_sync(0xffffffffu, hi == mh && lo == ml)) - 1;
    if (lane == p) {
      inv[k & 1] = ib;
      prow[k] = lane + 32 * hb;
      if (!ok) bad = true;
    }
  };
#pragma unroll
  for (int h = 0; h < R; ++h) {
    const int i = lane + 32 * h;
    used[h] = i >= n;
    step[h] = 0;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int j = W * c + warp;
      a[h][c] = i < n && j < n ? g[(size_t)j * n + i] : zero;
    }
    x[h] = a[h][0];
  }
  if (warp == 0) search(0);
  __syncthreads();
#pragma unroll
  for (int c = 0; c < C; ++c) {
    for (int w = 0; w < W; ++w) {
      const int k = W * c + w;
      if (k >= n) break;
      const int p = prow[k];
      const cplx ip = inv[k & 1];
      cplx nf[R];
#pragma unroll
      for (int h = 0; h < R; ++h) nf[h] = lane + 32 * h == p ? ip : cneg(cmul(col[k & 1][lane + 32 * h], ip));
      // the pivot's row, left empty (its lane adds 1 / pivot times it below)
#pragma unroll
      for (int h = 0; h < R; ++h) {
        const bool mine = lane + 32 * h == p;
        if (R > 1 && !__any_sync(0xffffffffu, mine)) continue;
        if (mine) {
#pragma unroll
          for (int d = 0; d < C; ++d) row[warp][d] = a[h][d];
        }
#pragma unroll
        for (int d = 0; d < C; ++d) a[h][d] = mine ? zero : a[h][d];
        used[h] = used[h] || mine;
        step[h] = mine ? k : step[h];
      }
      __syncwarp();
#pragma unroll
      for (int cc = 0; cc < C; ++cc) {
        const int d = (c + cc) % C;
        const cplx q = row[warp][d];
#pragma unroll
        for (int h = 0; h < R; ++h) a[h][d] = cfma(nf[h], q, a[h][d]);
        if (cc == 0 ? warp == w + 1 : cc == 1 && warp == 0 && w == W - 1) {
#pragma unroll
          for (int h = 0; h < R; ++h) x[h] = a[h][d];
          if (k + 1 < n) search(k + 1);
        }
      }
      if (warp == w) {
#pragma unroll
        for (int h = 0; h < R; ++h) a[h][c] = nf[h];
      }
      __syncthreads();
    }
  }
  // inverse(step of a row, pivot row of a column)
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = W * c + warp;
    if (j < n) {
      cplx* o = g + (size_t)prow[j] * n;
#pragma unroll
      for (int h = 0; h < R; ++h)
        if (lane + 32 * h < n) o[step[h]] = a[h][c];
    }
  }
  if (bad && status) status[blockIdx.x] = ST_ESINGULAR;
}

// ---------------------------------------------------------------------------
// Blocked form with the rank-w updates on the tensor cores.  Rows are never
// exchanged: step t takes as pivot row p_t the largest entry of column t among
// the rows not yet used, and the permutation comes out once at the end,
// inverse(t, p_u) = a(p_t, u).  Per panel of w columns zinv_panel_kernel
// reduces the panel, stores the update factor M = Tp - E (n x w; E the unit
// columns at the pivot rows) and extracts the pivot rows of the other columns,
// X (w x n, zero in the panel's columns); the batched GEMM then performs
// a += M X for all columns at once.
//
// The panel kernel holds a row (or RPT rows) per thread, so the multiplier of
// a step is the thread's own register and a pivot passes one barrier: the
// candidates are compared by their upper 32 bits (a pivot within 1e-6 of the
// largest is as good; magnitudes below 4.2e-314, whose reciprocal overflows,
// count as zero) with one warp reduction each side of it, and every warp's
// candidate puts out its row and the reciprocal of its pivot before it is known
// which one is taken.  Bound by that chain and by the loads, whose pivot rows
// are single entries of every column (64 matrices at n = 450: waits for memory
// first among the stalls, the FP64 pipe 12%).
// With rows split over two threads, exchanges, and every thread reducing the
// candidates and forming the reciprocal, a pivot took 4,700 cycles at n = 162,
// the row moves 25,000 cycles per panel and the final column exchanges one
// global round trip per column; above n = 256 the panel was in shared memory
// (n = 450: 4.0 ms per inversion of four matrices).
template <int THREADS, int RPT, int W>
__global__ void __launch_bounds__(THREADS, 1)
    zinv_panel_kernel(cplx* const* __restrict__ mats, cplx* __restrict__ scratch, size_t per, int n, int k, int w,
                      int* __restrict__ status) {
  // every warp's candidate of a step: key, row, and its entries with the
  // reciprocal of the first in front; two steps' worth
  __shared__ cplx s_cand[2][16][W];
  __shared__ unsigned s_key[2][16];
  __shared__ int s_row[2][16], s_piv[W], s_bad;

  cplx* a = mats[blockIdx.x];
  cplx* M = scratch + (size_t)blockIdx.x * per;  // [w][n] (room for W)
  cplx* X = M + (size_t)n * W;                   // [n][w]: X(s, j) at X[j * w + s]
  int* piv = reinterpret_cast<int*>(M + 2 * (size_t)n * W);  // [n]: pivot row of each column
  int* used = piv + n;                                       // [n]: rows that have been pivots
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nth >> 5;

  cplx r[RPT][W];
  bool open[RPT];
  int step[RPT];  // the step of this panel whose pivot the row was
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int i = tid + q * nth;
    step[q] = -1;
    open[q] = i < n && (k == 0 || used[i] == 0);
#pragma unroll
    for (int c = 0; c < W; ++c) r[q][c] = (i < n && c < w) ? a[(size_t)(k + c) * n + i] : mk(0.0, 0.0);
  }
  if (tid == 0) s_bad = 0;
  // The step loop stays rolled (unrolled, its code left the instruction cache:
  // 1,590 cycles per pivot at n = 98 with two barriers): a step's column is always r[.][0], and
  // the update writes every column one place down, the finished one last, so
  // that W steps bring them back into order.
#pragma unroll 1
  for (int s = 0; s < W; ++s) {
    if (s >= w) {  // columns beyond the matrix
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const cplx r0 = r[q][0];
#pragma unroll
        for (int c = 1; c < W; ++c) r[q][c - 1] = r[q][c];
        r[q][W - 1] = r0;
      }
      continue;
    }
    unsigned key = 0;  // rows that may be pivots have keys from 1 up
    int row = 0;
#pragma unroll
    for (int q = 0; q < RPT; ++q)
      if (open[q]) {
        const unsigned kq = max(1u, (unsigned)__double2hiint(cabs1(r[q][0])));
        if (kq > key) {
          key = kq;
          row = tid + q * nth;
        }
      }
    const int buf = s & 1;
    const unsigned wmax = __reduce_max_sync(0xffffffffu, key);
    const unsigned eq = __ballot_sync(0xffffffffu, key == wmax);
    if (lane == __ffs(eq) - 1) {  // this warp's candidate
      s_key[buf][warp] = key;
      s_row[buf][warp] = row;
#pragma unroll
      for (int q = 0; q < RPT; ++q)
        if (q == 0 || row == tid + q * nth) {
#pragma unroll
          for (int c = 1; c < W; ++c) s_cand[buf][warp][c] = r[q][c];
          s_cand[buf][warp][0] = (key <= 1u || key >= 0x7ff00000u) ? mk(1.0, 0.0) : cinv_fast(r[q][0]);
        }
    }
    __syncthreads();
    const unsigned kw = lane < nwarps ? s_key[buf][lane] : 0u;
    const unsigned top = __reduce_max_sync(0xffffffffu, kw);
    const int ww = __ffs(__ballot_sync(0xffffffffu, kw == top)) - 1;
    const int p = s_row[buf][ww];
    const cplx* prow = s_cand[buf][ww];
    const cplx ip = prow[0];
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      if (p == tid + q * nth) {
#pragma unroll
        for (int c = 1; c < W; ++c) r[q][c - 1] = cmul(r[q][c], ip);
        r[q][W - 1] = ip;
        step[q] = s;
        open[q] = false;
        s_piv[s] = p;
        if (top <= 1u || top >= 0x7ff00000u) s_bad = 1;
      } else {
        const cplx f = cneg(cmul(r[q][0], ip));
#pragma unroll
        for (int c = 1; c < W; ++c) r[q][c - 1] = cfma(f, prow[c], r[q][c]);
        r[q][W - 1] = f;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int i = tid + q * nth;
    if (i < n) {
#pragma unroll
      for (int c = 0; c < W; ++c)
        if (c < w) {
          const cplx v = r[q][c];
          a[(size_t)(k + c) * n + i] = v;
          M[(size_t)c * n + i] = step[q] == c ? mk(v.x - 1.0, v.y) : v;
        }
      if (k == 0 || step[q] >= 0) used[i] = step[q] >= 0 ? 1 : 0;
    }
  }
  __syncthreads();
  if (tid < w) piv[k + tid] = s_piv[tid];
  for (int j = tid; j < n; j += nth) {  // a thread per column, its gathers in flight together
    const bool own = j >= k && j < k + w;
    cplx x[W];
#pragma unroll
    for (int s = 0; s < W; ++s) x[s] = (own || s >= w) ? mk(0.0, 0.0) : a[(size_t)j * n + s_piv[s]];
#pragma unroll
    for (int s = 0; s < W; ++s)
      if (s < w) X[(size_t)j * w + s] = x[s];
  }
  if (tid == 0 && status && s_bad) status[blockIdx.x] = ST_ESINGULAR;
}

// The permutation at the end, in two passes that are each in place within a
// block's shared memory: entry t of a column is its entry p_t (four columns
// per block), then column u becomes column p_u (four rows per block).
constexpr int PERM_THREADS = 128;
template <bool COLS>
__global__ void __launch_bounds__(PERM_THREADS)
    zinv_permute_kernel(cplx* const* __restrict__ mats, const cplx* __restrict__ scratch, size_t per, int n, int W) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* buf = reinterpret_cast<cplx*>(smem_raw);  // [4 n]
  cplx* a = mats[blockIdx.y];
  const int* piv = reinterpret_cast<const int*>(scratch + (size_t)blockIdx.y * per + 2 * (size_t)n * W);
  const int v0 = blockIdx.x * 4, nv = min(4, n - v0), tid = threadIdx.x;
  if (COLS) {
    const int v = tid & 3;
    if (v < nv)
      for (int e = tid >> 2; e < n; e += PERM_THREADS / 4) buf[e * 4 + v] = a[(size_t)e * n + v0 + v];
    __syncthreads();
    if (v < nv)
      for (int e = tid >> 2; e < n; e += PERM_THREADS / 4) a[(size_t)piv[e] * n + v0 + v] = buf[e * 4 + v];
  } else {
    for (int e = tid; e < nv * n; e += PERM_THREADS) buf[e] = a[(size_t)v0 * n + e];
    __syncthreads();
    for (int v = 0; v < nv; ++v)
      for (int e = tid; e < n; e += PERM_THREADS) a[(size_t)(v0 + v) * n + e] = buf[v * n + piv[e]];
  }
}

}  // namespace

// One launch up to here, panels and updates above.  Measured, small against
// blocked, 1 / 148 / 600 matrices: n = 25 19 / 21 / 27 us against 52 / 56 / 124,
// n = 49 50 / 52 / 164 against 95 / 112 / 307, n = 96 109 / 115 / 548 against
// 153 / 251 / 880.  Four rows a lane would not fit the register file.
int zinv_small_maxn() { return ZS_MAXN; }

void zinv_small_batched(cplx* const* d_mats, int batch, int n, int* d_status, cudaStream_t stream) {
  if (batch <= 0) return;
  if (n <= 32) zinv_small_kernel<1, 4><<<batch, 128, 0, stream>>>(d_mats, n, d_status);
  else if (n <= 64) zinv_small_kernel<2, 8><<<batch, 256, 0, stream>>>(d_mats, n, d_status);
  else zinv_small_kernel<3, 16><<<batch, 512, 0, stream>>>(d_mats, n, d_status);
  VRC_CUDA_CHECK(cudaGetLastError());
}

// Panel columns: what a thread's registers hold (512 threads, 128 registers
// each) with a row per thread up to n = 512, two up to 1024, the largest order
// of a structure, and six above, where only matrices inverted by themselves
// (vrc_zinv) come in.
int zinv_blocked_width(int n) { return n <= 512 ? 16 : n <= 1024 ? 8 : 4; }

// The largest order taken: four columns of a matrix, the multipliers and the
// pivots in one CTA's shared memory, as a panel needed when it was kept there.
constexpr int ZB_MAXN = 2767;

size_t zinv_blocked_scratch(int n) {
  const int w = zinv_blocked_width(n);
  return (2 * (size_t)n * w + (2 * (size_t)n * 4 + 15) / 16) * 16;  // M, X, pivots, used rows
}

void zinv_blocked_batched(cplx* const* d_mats, int batch, int n, int* d_status, void* scratch,
                          const GemmDesc* d_descs, cudaStream_t stream) {
  if (batch <= 0) return;
  if (n > ZB_MAXN) throw StatusError(ST_EINVAL, "inversion: matrix too large");
  const int W = zinv_blocked_width(n);
  const size_t per = zinv_blocked_scratch(n) / 16;
  const size_t psm = (size_t)4 * n * sizeof(cplx);
  ensure_smem((const void*)zinv_permute_kernel<false>, psm);
  ensure_smem((const void*)zinv_permute_kernel<true>, psm);
  cplx* scr = static_cast<cplx*>(scratch);
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    const int nb = min(65535, batch - b0);
    cplx* sb = scr + (size_t)b0 * per;
    for (int k = 0; k < n; k += W) {
      const int w = min(W, n - k);
      int* st = d_status ? d_status + b0 : nullptr;
      const int rows = n <= 512 ? 1 : n <= 1024 ? 2 : 6, threads = ((n + rows - 1) / rows + 31) / 32 * 32;
      auto panel = n <= 256    ? zinv_panel_kernel<256, 1, 16>
                   : n <= 512  ? zinv_panel_kernel<512, 1, 16>
                   : n <= 1024 ? zinv_panel_kernel<512, 2, 8>
                               : zinv_panel_kernel<512, 6, 4>;
      panel<<<nb, threads, 0, stream>>>(d_mats + b0, sb, per, n, k, w, st);
      VRC_CUDA_CHECK(cudaGetLastError());
      // descriptor b: A = M (n x w, leading dimension n), B = X (w x n,
      // leading dimension w) at M + n W, C = Cin = the matrix
      zgemm_batched(d_descs + b0, nb, n, mk(1.0, 0.0), mk(1.0, 0.0), 0.0, stream, w);
    }
    const dim3 grid((n + 3) / 4, nb);
    zinv_permute_kernel<false><<<grid, PERM_THREADS, psm, stream>>>(d_mats + b0, sb, per, n, W);
    zinv_permute_kernel<true><<<grid, PERM_THREADS, psm, stream>>>(d_mats + b0, sb, per, n, W);
  }
  VRC_CUDA_CHECK(cudaGetLastError());
}

}  // namespace vrc

// Batched in-place matrix inversion: blocked Gauss-Jordan with partial
// (row) pivoting, one CTA per matrix.
//
// The reference inverts through Eigen PartialPivLU (explicit inverse of
// I - rdu*Rud, src/core/RedhefferIntegrator.cpp:267-270) and uses LU solves
// elsewhere; here every W^{-1}X / M^{-1}X of the hot path is an explicit
// inverse followed by a tensor-core GEMM (same 8n^3 flops as getrf+getrs).
//
// Blocking: a panel of nb columns is reduced in shared memory (pivot search
// by warp-shuffle max reduction); the nb accumulated row operations are then
// applied to every other column as one rank-nb update
//     a[:, j] <- P a[:, j];  a[:, j] += (Tp - E) a[k:k+nb, j]
// so the matrix is streamed once per panel instead of once per pivot.
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"

namespace vrc {
namespace {

constexpr int INV_THREADS = 512;

struct PivotCand {
  double v;
  int i;
};

__device__ __forceinline__ PivotCand warp_argmax(PivotCand c) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double ov = __shfl_xor_sync(0xffffffffu, c.v, o);
    int oi = __shfl_xor_sync(0xffffffffu, c.i, o);
    if (ov > c.v || (ov == c.v && oi < c.i)) {
      c.v = ov;
      c.i = oi;
    }
  }
  return c;
}

__global__ void __launch_bounds__(INV_THREADS)
    zinv_kernel(cplx* const* __restrict__ mats, int n, int nb, int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* panel = reinterpret_cast<cplx*>(smem_raw);  // [nb][n] column-major panel
  cplx* fcol = panel + (size_t)nb * n;                       // [n] multipliers
  int* piv = reinterpret_cast<int*>(fcol + n);                // [n]
  __shared__ PivotCand red[INV_THREADS / 32];
  __shared__ cplx s_inv;
  __shared__ int s_p;
  __shared__ int s_bad;

  cplx* a = mats[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = INV_THREADS / 32;
  if (tid == 0) s_bad = 0;

  for (int k = 0; k < n; k += nb) {
    const int w = min(nb, n - k);
    // Load panel columns k..k+w-1.
    for (int idx = tid; idx < w * n; idx += INV_THREADS) {
      int c = idx / n, r = idx - c * n;
      panel[c * n + r] = a[(size_t)(k + c) * n + r];
    }
    __syncthreads();
    for (int s = 0; s < w; ++s) {
      const int r0 = k + s;
      cplx* col = panel + s * n;
      // Pivot search over rows >= r0 (|re|+|im|, as izamax).
      PivotCand c{-1.0, n};
      for (int i = r0 + tid; i < n; i += INV_THREADS) {
        double v = cabs1(col[i]);
        if (v > c.v) { c.v = v; c.i = i; }
      }
      c = warp_argmax(c);
      if (lane == 0) red[warp] = c;
      __syncthreads();
      if (warp == 0) {
        PivotCand cc = lane < nwarps ? red[lane] : PivotCand{-1.0, n};
        cc = warp_argmax(cc);
        if (lane == 0) {
          int p = cc.i;
          cplx pv = col[p];
          if (!(cc.v > 0.0) || !isfinite(cc.v)) {
            s_bad = 1;
            pv = mk(1.0, 0.0);
            p = r0;
          }
          s_p = p;
          s_inv = cinv(pv);
          piv[r0] = p;
        }
      }
      __syncthreads();
      const int p = s_p;
      const cplx ip = s_inv;
      // Swap rows r0 and p inside the panel.
      if (p != r0) {
        for (int c2 = tid; c2 < w; c2 += INV_THREADS) {
          cplx t = panel[c2 * n + r0];
          panel[c2 * n + r0] = panel[c2 * n + p];
          panel[c2 * n + p] = t;
        }
      }
      __syncthreads();
      // Save the multipliers (column s), then scale the pivot row:
      // a[r0][s] := 1, row *= 1/piv.
      for (int i = tid; i < n; i += INV_THREADS) fcol[i] = col[i];
      __syncthreads();
      for (int c2 = tid; c2 < w; c2 += INV_THREADS) {
        cplx v = (c2 == s) ? mk(1.0, 0.0) : panel[c2 * n + r0];
        panel[c2 * n + r0] = cmul(v, ip);
      }
      __syncthreads();
      // Eliminate column s from the other rows (panel columns only).
      for (int idx = tid; idx < n * w; idx += INV_THREADS) {
        int c2 = idx / n, i = idx - c2 * n;
        if (i == r0) continue;
        cplx prow = panel[c2 * n + r0];
        cplx v = (c2 == s) ? mk(0.0, 0.0) : panel[c2 * n + i];
        panel[c2 * n + i] = csub(v, cmul(fcol[i], prow));
      }
      __syncthreads();
    }
    // Write the panel back.
    for (int idx = tid; idx < w * n; idx += INV_THREADS) {
      int c = idx / n, r = idx - c * n;
      a[(size_t)(k + c) * n + r] = panel[c * n + r];
    }
    // Rank-w update of all other columns: one warp per column.
    for (int j = warp; j < n; j += nwarps) {
      if (j >= k && j < k + w) continue;
      cplx* colj = a + (size_t)j * n;
      // Row swaps in order.
      if (lane == 0) {
        for (int s = 0; s < w; ++s) {
          int p = piv[k + s];
          if (p != k + s) {
            cplx t = colj[k + s];
            colj[k + s] = colj[p];
            colj[p] = t;
          }
        }
      }
      __syncwarp();
      cplx x[16];
#pragma unroll
      for (int s = 0; s < 16; ++s) x[s] = (s < w) ? colj[k + s] : mk(0.0, 0.0);
      __syncwarp();
      for (int i = lane; i < n; i += 32) {
        cplx v = colj[i];
        cplx acc = mk(0.0, 0.0);
#pragma unroll
        for (int s = 0; s < 16; ++s) {
          if (s < w) {
            cplx t = panel[s * n + i];
            if (i == k + s) t.x -= 1.0;
            acc = cfma(t, x[s], acc);
          }
        }
        colj[i] = cadd(v, acc);
      }
    }
    __syncthreads();
  }
  // Undo the row interchanges as column interchanges, in reverse order.
  for (int k = n - 1; k >= 0; --k) {
    int p = piv[k];
    if (p != k) {
      for (int i = tid; i < n; i += INV_THREADS) {
        cplx t = a[(size_t)k * n + i];
        a[(size_t)k * n + i] = a[(size_t)p * n + i];
        a[(size_t)p * n + i] = t;
      }
    }
    __syncthreads();
  }
  if (tid == 0 && status && s_bad) status[blockIdx.x] = ST_ESINGULAR;
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
// largest is as good) with one warp reduction each side of it, and every warp's
// candidate puts out its row and the reciprocal of its pivot before it is known
// which one is taken.  Bound by that chain for few matrices and by the FP64
// issue of the update for many.
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

int zinv_panel_width(int n) {
  // panel (nb x n complex) + pivots must fit comfortably in shared memory.
  int nb = 16;
  while (nb > 1 && (size_t)(nb + 1) * n * 16 + (size_t)n * 4 > 200 * 1024) nb >>= 1;
  return nb;
}

// Panel columns: what a thread's registers hold with a row per thread up to
// n = 512 and two above (512 threads, 128 registers each).
int zinv_blocked_width(int n) { return n <= 512 ? 16 : 8; }

size_t zinv_blocked_scratch(int n) {
  const int w = zinv_blocked_width(n);
  return (2 * (size_t)n * w + (2 * (size_t)n * 4 + 15) / 16) * 16;  // M, X, pivots, used rows
}

void zinv_blocked_batched(cplx* const* d_mats, int batch, int n, int* d_status, void* scratch,
                          const GemmDesc* d_descs, cudaStream_t stream) {
  if (batch <= 0) return;
  if (n > 1024) throw StatusError(ST_EINVAL, "blocked inversion: n <= 1024");
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
      const int threads = (n <= 512 ? n + 31 : (n + 1) / 2 + 31) / 32 * 32;
      auto panel = n <= 256   ? zinv_panel_kernel<256, 1, 16>
                   : n <= 512 ? zinv_panel_kernel<512, 1, 16>
                              : zinv_panel_kernel<512, 2, 8>;
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

void zinv_batched(cplx* const* d_mats, int batch, int n, int* d_status, cudaStream_t stream) {
  if (batch <= 0) return;
  int nb = zinv_panel_width(n);
  size_t smem = (size_t)(nb + 1) * n * 16 + (size_t)n * 4;
  ensure_smem((const void*)zinv_kernel, smem);
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    int nbat = batch - b0 < 65535 ? batch - b0 : 65535;
    zinv_kernel<<<nbat, INV_THREADS, smem, stream>>>(d_mats + b0, n, nb,
                                                      d_status ? d_status + b0 : nullptr);
  }
  VRC_CUDA_CHECK(cudaGetLastError());
}

}  // namespace vrc

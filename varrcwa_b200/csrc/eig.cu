// Batched FP64 complex non-Hermitian eigensolver (right eigenvectors), one
// CTA per matrix, replacing LAPACKE_zgeev / magma_zgeev of the reference
// (src/rcwa/MKLEigenSolver.hpp:45-55, src/gpu/RedhefferIntegratorGPU.cpp:220-223).
//
//   1. hess_smem_kernel, hess_kernel
//                    Householder reduction to upper Hessenberg form
//                    (H = Q^H A Q) with the left and right reflector
//                    applications fused into one rank-2 update per column,
//                    then backward accumulation of Q.
//   2. hqr_kernel    complex Schur form T = Z^H A Z (qr.cu: multi-bulge
//                    shifted QR with a rotation log replayed onto Z).
//   3. trevc_kernel  eigenvectors of T by back substitution (one warp per
//                    eigenvalue, near-singular diagonals perturbed to smin).
//   4. vecnorm_kernel  X = Z Y is formed by the GEMM; each column is scaled to
//                    unit 2-norm with its largest component real (the zgeev
//                    convention).
#include <cstdlib>

#include "common.cuh"
#include "householder.cuh"
#include "kernels.h"

namespace vrc {
namespace {

constexpr int HESS_THREADS = 256;
constexpr int HESS_WARPS = HESS_THREADS / 32;

__device__ __forceinline__ cplx warp_sum(cplx v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}
__device__ __forceinline__ double warp_sumd(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// 1. Hessenberg reduction + Q accumulation
// ---------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(HESS_THREADS)
    hess_kernel(cplx* const* __restrict__ Hs, cplx* const* __restrict__ Zs, int n) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* v = reinterpret_cast<cplx*>(smem_raw);  // [n]
  cplx* y = v + n;                              // [n]
  cplx* u = y + n;                              // [n]
  cplx* taus = u + n;                           // [n]
  cplx* yp = taus + n;                          // [HESS_WARPS][n]
  __shared__ double red[HESS_WARPS];
  __shared__ cplx s_tau, s_scale, s_s;

  cplx* H = Hs[blockIdx.x];
  cplx* Z = Zs[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  for (int k = 0; k + 2 < n; ++k) {
    const int j0 = k + 1;  // J = [j0, n)
    // --- reflector from x = H[j0:n, k]
    double part = 0.0;
    for (int i = j0 + 1 + tid; i < n; i += HESS_THREADS) part += cabs2(H[(size_t)k * n + i]);
    part = warp_sumd(part);
    if (lane == 0) red[warp] = part;
    __syncthreads();
    if (tid == 0) {
      double xn = 0.0;
      for (int w = 0; w < HESS_WARPS; ++w) xn += red[w];
      cplx alpha = H[(size_t)k * n + j0];
      double beta;
      cplx tau, scale;
      householder(alpha, xn, &beta, &tau, &scale);
      s_tau = tau;
      s_scale = scale;
      taus[k] = tau;
      H[(size_t)k * n + j0] = mk(beta, 0.0);
    }
    __syncthreads();
    const cplx tau = s_tau;
    for (int i = tid; i < n; i += HESS_THREADS) {
      cplx vi;
      if (i < j0) vi = mk(0.0, 0.0);
      else if (i == j0) vi = mk(1.0, 0.0);
      else {
        vi = cmul(H[(size_t)k * n + i], s_scale);
        H[(size_t)k * n + i] = vi;  // keep v below the subdiagonal for Q
      }
      v[i] = vi;
    }
    __syncthreads();
    if (tau.x == 0.0 && tau.y == 0.0) continue;
    // --- fused products: y = H[:, J] v (all rows), u_j = v^H H[J, j]
    cplx ypart[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) ypart[t] = mk(0.0, 0.0);
    for (int j = j0 + warp; j < n; j += HESS_WARPS) {
      const cplx vj = v[j];
      const cplx* col = H + (size_t)j * n;
      cplx up = mk(0.0, 0.0);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        int i = lane + 32 * t;
        if (i < n) {
          cplx h = col[i];
          ypart[t] = cfma(h, vj, ypart[t]);
          if (i >= j0) up = cadd(up, cmulc(v[i], h));
        }
      }
      up = warp_sum(up);
      if (lane == 0) u[j] = up;
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      int i = lane + 32 * t;
      if (i < n) yp[warp * n + i] = ypart[t];
    }
    __syncthreads();
    for (int i = tid; i < n; i += HESS_THREADS) {
      cplx s = mk(0.0, 0.0);
      for (int w = 0; w < HESS_WARPS; ++w) s = cadd(s, yp[w * n + i]);
      y[i] = s;
    }
    __syncthreads();
    // s = v^H y_J
    {
      cplx sp = mk(0.0, 0.0);
      for (int i = j0 + tid; i < n; i += HESS_THREADS) sp = cadd(sp, cmulc(v[i], y[i]));
      sp = warp_sum(sp);
      if (lane == 0) yp[warp] = sp;  // reuse
      __syncthreads();
      if (tid == 0) {
        cplx s = mk(0.0, 0.0);
        for (int w = 0; w < HESS_WARPS; ++w) s = cadd(s, yp[w]);
        s_s = s;
      }
      __syncthreads();
    }
    // z_j = u_j - tau * s * conj(v_j)
    const cplx ts = cmul(tau, s_s);
    for (int j = j0 + tid; j < n; j += HESS_THREADS) u[j] = csub(u[j], cmul(ts, cconj(v[j])));
    __syncthreads();
    // --- rank-2 update of H[:, J]
    const cplx tauc = cconj(tau);
    for (int j = j0 + warp; j < n; j += HESS_WARPS) {
      const cplx vjc = cconj(v[j]);
      const cplx zj = u[j];
      cplx* col = H + (size_t)j * n;
      const cplx tv = cmul(tau, vjc);
      const cplx tz = cmul(tauc, zj);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        int i = lane + 32 * t;
        if (i < n) {
          cplx h = col[i];
          h = csub(h, cmul(y[i], tv));
          if (i >= j0) h = csub(h, cmul(v[i], tz));
          col[i] = h;
        }
      }
    }
    __syncthreads();
  }
  // --- Q = H_0 H_1 ... H_{n-3}, accumulated backward into Z.
  for (int idx = tid; idx < n * n; idx += HESS_THREADS) {
    int c = idx / n, r = idx - c * n;
    Z[idx] = mk(r == c ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  for (int k = n - 3; k >= 0; --k) {
    const int j0 = k + 1;
    const cplx tau = taus[k];
    for (int i = tid; i < n; i += HESS_THREADS) {
      v[i] = (i < j0) ? mk(0.0, 0.0) : (i == j0 ? mk(1.0, 0.0) : H[(size_t)k * n + i]);
    }
    __syncthreads();
    if (!(tau.x == 0.0 && tau.y == 0.0)) {
      for (int j = j0 + warp; j < n; j += HESS_WARPS) {
        cplx* col = Z + (size_t)j * n;
        cplx wp = mk(0.0, 0.0);
        for (int i = j0 + lane; i < n; i += 32) wp = cadd(wp, cmulc(v[i], col[i]));
        wp = warp_sum(wp);
        const cplx tw = cmul(tau, wp);
        for (int i = j0 + lane; i < n; i += 32) col[i] = csub(col[i], cmul(v[i], tw));
      }
    }
    __syncthreads();
  }
  // Clear everything below the subdiagonal (the stored reflectors).
  for (int idx = tid; idx < n * n; idx += HESS_THREADS) {
    int c = idx / n, r = idx - c * n;
    if (r > c + 1) H[idx] = mk(0.0, 0.0);
  }
}

// The same reduction for n <= 115 with the matrix in shared memory, Q accumulated
// in its place.  Eight lanes take a column (a row in eight each, the rows padded
// with zeros to 8 RV) and the CTA 32 columns at a time: both products in one
// pass, v^H a_j kept in registers for the update, and every warp forms the
// reflector for itself.  A column passes three barriers (the warps' shares of
// A v, their sum, the next reflector's column).  Bound by that chain, with the
// SMs full too (600 at n = 61: issue and the shared-memory port 46%, FP64 33%).
// One / 600 matrices take 0.11 / 0.37 ms at n = 42, 0.21 / 0.73 at 61 (hess_kernel
// 0.51 for some 60) and 0.58 / 2.9 at 98 (panels and GEMM updates 0.93 / 4.1),
// 0.75 / 3.8 at 113 (1.00 / 5.1) and 0.76 / 3.9 at 115 (1.02 / 5.3).  RV = 15
// leaves the padding out, the only form that fits above 112 (a row more in a
// lane, padded, holds 111).
constexpr size_t hs_smem(int n, int rv) {
  return ((size_t)(n + HESS_WARPS + 2) * (rv == 15 ? n : 8 * rv) + HESS_WARPS) * sizeof(cplx);
}
constexpr int hs_maxn() {  // the largest order whose matrix a CTA's shared memory holds
  int n = 113;
  while (hs_smem(n + 1, 15) <= (size_t)227 * 1024) ++n;
  return n;
}
constexpr int HS_MAXN = hs_maxn();
static_assert(HS_MAXN <= 8 * 15 && hs_smem(112, 14) <= (size_t)227 * 1024, "rows of the widest forms");

__device__ __forceinline__ cplx shfl_xor(cplx z, int o) {
  return mk(__shfl_xor_sync(0xffffffffu, z.x, o), __shfl_xor_sync(0xffffffffu, z.y, o));
}

__device__ __forceinline__ cplx sum8(cplx z) {
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) z = cadd(z, shfl_xor(z, o));
  return z;
}

template <int RV>
__global__ void __launch_bounds__(HESS_THREADS, RV <= 10 ? 2 : 1)
    hess_smem_kernel(cplx* const* __restrict__ Hs, cplx* const* __restrict__ Zs, int n) {
  constexpr bool TIGHT = RV == 15;  // no room for padding: rows past n are the next column's
  const int LD = TIGHT ? n : 8 * RV;
  constexpr int RT = (RV + 3) / 4 * 4, NT = RT / 4;  // rows and column passes of a lane
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* A = reinterpret_cast<cplx*>(smem_raw);  // [n][LD]
  cplx* yp = A + n * LD;                        // [HESS_WARPS][LD]
  cplx* ys = yp + HESS_WARPS * LD;              // [LD]
  cplx* taus = ys + LD;                         // [LD]
  cplx* sp = taus + LD;                         // [HESS_WARPS]
  cplx* H = Hs[blockIdx.x];
  cplx* Z = Zs[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int l8 = lane & 7, col = 4 * warp + (lane >> 3);
  const bool b0 = lane & 8, b1 = lane & 16;
  const cplx zero = mk(0.0, 0.0);
  if (TIGHT)
    for (int r = tid; r < HESS_WARPS * LD; r += HESS_THREADS) yp[r] = zero;  // (past the last column)
  for (int c = warp; c < n; c += HESS_WARPS)
    for (int r = lane; r < LD; r += 32) A[c * LD + r] = r < n ? H[(size_t)c * n + r] : zero;
  __syncthreads();
  for (int k = 0; k + 2 < n; ++k) {
    const int j0 = k + 1;  // J = [j0, n)
    const cplx* x = A + k * LD;
    cplx v[RV];
    double part[2] = {0.0, 0.0};
#pragma unroll
    for (int t = 0; t < RV; ++t) {
      v[t] = !TIGHT || t < RV - 1 || l8 + 8 * t < n ? x[l8 + 8 * t] : zero;
      if (l8 + 8 * t > j0) part[t & 1] += cabs2(v[t]);
    }
    double x2 = part[0] + part[1];
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) x2 += __shfl_xor_sync(0xffffffffu, x2, o);
    double beta;
    cplx tau, scale;
    householder(x[j0], x2, &beta, &tau, &scale);
    if (tid == 0) taus[k] = tau;
    if (tau.x == 0.0 && tau.y == 0.0) continue;  // (every thread alike)
#pragma unroll
    for (int t = 0; t < RV; ++t) {
      const int i = l8 + 8 * t;
      v[t] = i > j0 ? cmul(v[t], scale) : mk(i == j0 ? 1.0 : 0.0, 0.0);
    }
    // shares of y = A[:, J] v and of s = v^H y, and u_j = v^H a_j
    cplx y[RT], u[NT], vj[NT], s = zero;
#pragma unroll
    for (int t = 0; t < RT; ++t) y[t] = zero;
#pragma unroll
    for (int p = 0; p < NT; ++p) {
      u[p] = vj[p] = zero;
      if (j0 + 32 * p + 4 * warp < n) {  // (a warp alike)
        const int j = j0 + 32 * p + col;
        const cplx* a = A + min(j, n - 1) * LD + l8;
        cplx u2[2] = {zero, zero};  // (two chains)
        if (j < n) vj[p] = j == j0 ? mk(1.0, 0.0) : cmul(x[j], scale);
#pragma unroll
        for (int t = 0; t < RV; ++t) {
          const cplx h = a[8 * t];
          y[t] = cfma(h, vj[p], y[t]);
          u2[t & 1] = cfma(cconj(v[t]), h, u2[t & 1]);
        }
        u[p] = sum8(cadd(u2[0], u2[1]));
        s = cfma(u[p], vj[p], s);
      }
    }
    // over the warp's four columns: each group of lanes ends with a row in four
    cplx half[RT / 2];
#pragma unroll
    for (int q = 0; q < RT / 2; ++q)
      half[q] = cadd(b1 ? y[2 * q + 1] : y[2 * q], shfl_xor(b1 ? y[2 * q] : y[2 * q + 1], 16));
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      const int t = 4 * q + 2 * b0 + b1;
      const cplx z =
          cadd(b0 ? half[2 * q + 1] : half[2 * q], shfl_xor(b0 ? half[2 * q] : half[2 * q + 1], 8));
      if (t < RV && (!TIGHT || t < RV - 1 || l8 + 8 * t < n)) yp[warp * LD + l8 + 8 * t] = z;
    }
    s = cadd(s, shfl_xor(s, 8));
    s = cadd(s, shfl_xor(s, 16));
    if (lane == 0) sp[warp] = s;
    __syncthreads();
    if (tid < LD) {
      cplx sum = zero;
#pragma unroll
      for (int w = 0; w < HESS_WARPS; ++w) sum = cadd(sum, yp[w * LD + tid]);
      ys[tid] = sum;
    }
    s = zero;
#pragma unroll
    for (int w = 0; w < HESS_WARPS; ++w) s = cadd(s, sp[w]);
    const cplx ts = cmul(tau, s), tauc = cconj(tau);
    if (warp == HESS_WARPS - 1 && lane < 8) {  // column k: its reflector stays below the subdiagonal
#pragma unroll
      for (int t = 0; t < RV; ++t)
        if (l8 + 8 * t >= j0 && (!TIGHT || t < RV - 1 || l8 + 8 * t < n)) A[k * LD + l8 + 8 * t] = l8 + 8 * t == j0 ? mk(beta, 0.0) : v[t];
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < RV; ++t) y[t] = ys[l8 + 8 * t];
    // rank-2 update
#pragma unroll
    for (int p = 0; p < NT; ++p) {
      const int j = j0 + 32 * p + col;
      if (j < n) {
        cplx* a = A + j * LD + l8;
        const cplx vc = cconj(vj[p]), tv = cmul(cneg(tau), vc),
                   tz = cmul(tauc, csub(cmul(ts, vc), u[p]));
#pragma unroll
        for (int t = 0; t < RV; ++t)
          if (!TIGHT || t < RV - 1 || l8 + 8 * t < n) a[8 * t] = cfma(y[t], tv, cfma(v[t], tz, a[8 * t]));
      }
    }
    __syncthreads();
  }
  __syncthreads();
  for (int c = warp; c < n; c += HESS_WARPS)
    for (int r = lane; r < n; r += 32) H[(size_t)c * n + r] = r <= c + 1 ? A[c * LD + r] : zero;
  __syncthreads();
  // Q = H_0 H_1 ... H_(n-3) backward, in place: step k turns column k + 1 into
  // Q's and leaves column k, which holds v_k, for the step after
  if (tid == 0) A[(n - 1) * LD + n - 1] = mk(1.0, 0.0);
  __syncthreads();
  for (int k = n - 3; k >= 0; --k) {
    const int j0 = k + 1;
    const cplx tau = taus[k];
    cplx v[RV];
#pragma unroll
    for (int t = 0; t < RV; ++t) {
      const int i = l8 + 8 * t;
      v[t] = i > j0 && (!TIGHT || t < RV - 1 || i < n) ? A[k * LD + i] : mk(i == j0 ? 1.0 : 0.0, 0.0);
    }
#pragma unroll
    for (int p = 0; p < NT; ++p) {
      if (j0 + 32 * p + 4 * warp < n) {  // (a warp alike)
        const int j = j0 + 32 * p + col;
        cplx* a = A + min(j, n - 1) * LD + l8;
        cplx h[RV], w[2] = {zero, zero};
#pragma unroll
        for (int t = 0; t < RV; ++t) {
          const int i = l8 + 8 * t;
          h[t] = j == j0 ? mk(i == j0 ? 1.0 : 0.0, 0.0) : i > j0 ? a[8 * t] : zero;
          w[t & 1] = cfma(cconj(v[t]), h[t], w[t & 1]);
        }
        const cplx z = sum8(cadd(w[0], w[1]));
        const cplx tw = cneg(j == j0 ? tau : cmul(tau, z));
#pragma unroll
        for (int t = 0; t < RV; ++t)
          if (j < n && l8 + 8 * t >= j0 && (!TIGHT || t < RV - 1 || l8 + 8 * t < n)) a[8 * t] = cfma(v[t], tw, h[t]);
      }
    }
    __syncthreads();
  }
  for (int c = warp; c < n; c += HESS_WARPS)
    for (int r = lane; r < n; r += 32)
      Z[(size_t)c * n + r] = (c == 0 || r == 0) ? mk(c == r ? 1.0 : 0.0, 0.0) : A[c * LD + r];
}

constexpr double ULP = EIG_ULP;
constexpr double SMLNUM_BASE = EIG_SAFMIN;

// ---------------------------------------------------------------------------
// 3. Eigenvectors of the triangular Schur factor
// ---------------------------------------------------------------------------
constexpr int TV_WARPS = 8;

__global__ void __launch_bounds__(TV_WARPS * 32)
    trevc_kernel(cplx* const* __restrict__ Ts, cplx* const* __restrict__ Ys, int n) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* work = reinterpret_cast<cplx*>(smem_raw) + (threadIdx.x >> 5) * n;
  const int lane = threadIdx.x & 31;
  const int mat = blockIdx.y;
  const cplx* T = Ts[mat];
  cplx* Y = Ys[mat];
  const int ki = blockIdx.x * TV_WARPS + (threadIdx.x >> 5);
  if (ki >= n) return;
  const cplx lam = T[(size_t)ki * n + ki];
  const double smin = fmax(ULP * cabs1(lam), SMLNUM_BASE * ((double)n / ULP));
  for (int r = lane; r < n; r += 32) work[r] = (r < ki) ? cneg(T[(size_t)ki * n + r]) : mk(0.0, 0.0);
  __syncwarp();
  for (int j = ki - 1; j >= 0; --j) {
    // x_j = work_j / (T_jj - lam)
    cplx dj = csub(T[(size_t)j * n + j], lam);
    if (cabs1(dj) < smin) dj = mk(smin, 0.0);
    cplx xj = cdiv(work[j], dj);
    __syncwarp();
    if (lane == 0) work[j] = xj;
    const cplx* colj = T + (size_t)j * n;
    for (int r = lane; r < j; r += 32) work[r] = csub(work[r], cmul(xj, colj[r]));
    __syncwarp();
  }
  cplx* y = Y + (size_t)ki * n;
  for (int r = lane; r < n; r += 32) y[r] = (r < ki) ? work[r] : (r == ki ? mk(1.0, 0.0) : mk(0.0, 0.0));
}

// ---------------------------------------------------------------------------
// 4. Column normalisation: unit 2-norm, largest-modulus component real.
// ---------------------------------------------------------------------------
__global__ void vecnorm_kernel(cplx* const* __restrict__ Xs, int n) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * (blockDim.x >> 5) + warp;
  if (col >= n) return;
  cplx* x = Xs[blockIdx.y] + (size_t)col * n;
  double s2 = 0.0, best = -1.0;
  int bi = 0;
  for (int r = lane; r < n; r += 32) {
    double a = cabs2(x[r]);
    s2 += a;
    if (a > best) { best = a; bi = r; }
  }
  s2 = warp_sumd(s2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double ob = __shfl_xor_sync(0xffffffffu, best, o);
    int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
  }
  cplx xm = x[bi];
  double am = sqrt(cabs2(xm));
  double nrm = sqrt(s2);
  cplx f = (am > 0.0 && nrm > 0.0) ? mk(xm.x / (am * nrm), -xm.y / (am * nrm)) : mk(1.0, 0.0);
  for (int r = lane; r < n; r += 32) x[r] = cmul(x[r], f);
  __syncwarp();
  if (lane == 0) x[bi] = mk(x[bi].x, 0.0);
}

template <int RV>
void launch_hess_smem(cplx* const* H, cplx* const* Z, int batch, int n, cudaStream_t st) {
  const size_t smem = hs_smem(n, RV);
  ensure_smem((const void*)hess_smem_kernel<RV>, smem);
  hess_smem_kernel<RV><<<batch, HESS_THREADS, smem, st>>>(H, Z, n);
}

template <int NT>
void launch_hess(cplx* const* H, cplx* const* Z, int batch, int n, cudaStream_t st) {
  size_t smem = (size_t)(4 + HESS_WARPS) * n * 16;
  ensure_smem((const void*)hess_kernel<NT>, smem);
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    int nb = min(65535, batch - b0);
    hess_kernel<NT><<<nb, HESS_THREADS, smem, st>>>(H + b0, Z + b0, n);
  }
}

}  // namespace

int hessenberg_smem_maxn() { return HS_MAXN; }

void hessenberg_batched(cplx* const* d_H, cplx* const* d_Z, int batch, int n, cudaStream_t st) {
  if (batch <= 0) return;
  // Cluster or single-CTA reduction, by measured crossovers on B200 (ms per
  // batch, both variants): a single CTA wins for n <= 128 at every
  // batch (4-9x at n = 50..98 once the batch fills the SMs, because eight
  // CTAs of a few columns each spend the reduction in cluster barriers); for
  // 128 < n <= 192 and 256 < n < 400 it wins only once the batch gives every
  // SM two matrices; the cluster kernel wins for 192 < n <= 256 at every batch
  // (matrix in shared memory) and for n >= 400, where the single-CTA
  // reduction's per-matrix latency dominates.
  static const int sms = [] {
    int dev = 0, v = 0;
    VRC_CUDA_CHECK(cudaGetDevice(&dev));
    VRC_CUDA_CHECK(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
    return v;
  }();
  const bool full = batch >= 2 * sms;
  const bool cluster = hessenberg_cluster_fits(n) && n > 128 &&
                       ((n > 192 && n <= 256) || n >= 400 || !full);
  if (cluster && !std::getenv("VRC_HESS_SINGLE_CTA")) {
    hessenberg_cluster_batched(d_H, d_Z, batch, n, st);
    return;
  }
  // Within it the kernel in shared memory, at every batch (its figures above).
  if (n <= HS_MAXN) {
    if (n <= 32) launch_hess_smem<4>(d_H, d_Z, batch, n, st);
    else if (n <= 48) launch_hess_smem<6>(d_H, d_Z, batch, n, st);
    else if (n <= 64) launch_hess_smem<8>(d_H, d_Z, batch, n, st);
    else if (n <= 80) launch_hess_smem<10>(d_H, d_Z, batch, n, st);
    else if (n <= 96) launch_hess_smem<12>(d_H, d_Z, batch, n, st);
    else if (n <= 112) launch_hess_smem<14>(d_H, d_Z, batch, n, st);
    else launch_hess_smem<15>(d_H, d_Z, batch, n, st);
    VRC_CUDA_CHECK(cudaGetLastError());
    return;
  }
  if (n <= 256) launch_hess<8>(d_H, d_Z, batch, n, st);
  else if (n <= 512) launch_hess<16>(d_H, d_Z, batch, n, st);
  else if (n <= 1024) launch_hess<32>(d_H, d_Z, batch, n, st);
  else throw StatusError(ST_EINVAL, "eigensolver supports n <= 1024");
  VRC_CUDA_CHECK(cudaGetLastError());
}

void trevc_batched(cplx* const* d_T, cplx* const* d_Y, int batch, int n, cudaStream_t st) {
  if (batch <= 0) return;
  size_t smem = (size_t)TV_WARPS * n * 16;
  ensure_smem((const void*)trevc_kernel, smem);
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    int nb = min(65535, batch - b0);
    dim3 grid((n + TV_WARPS - 1) / TV_WARPS, nb);
    trevc_kernel<<<grid, TV_WARPS * 32, smem, st>>>(d_T + b0, d_Y + b0, n);
  }
  VRC_CUDA_CHECK(cudaGetLastError());
}

void vecnorm_batched(cplx* const* d_X, int batch, int n, cudaStream_t st) {
  if (batch <= 0) return;
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    int nb = min(65535, batch - b0);
    dim3 grid((n + 7) / 8, nb);
    vecnorm_kernel<<<grid, 256, 0, st>>>(d_X + b0, n);
  }
  VRC_CUDA_CHECK(cudaGetLastError());
}

}  // namespace vrc

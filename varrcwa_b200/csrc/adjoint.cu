// Kernels of the layer-stack forward solve and its adjoint (gradients of
// per-order power with respect to permittivity pixels).
//
// Complex gradients follow dL = Re(sum(conj(G) * dZ)).  With every eigen
// basis held fixed, a perturbation (dP, dQ) of a z-uniform layer changes only
// the layer's own-basis blocks, by the first-order term of the perturbative
// segment (src/core/RedhefferIntegrator.cpp:317-399) with the z-integrals
// done exactly:
//   dtuu = dtdd =  K_E o (W^-1 dP V + V^-1 dQ W),
//   drud = drdu = -K_D o (W^-1 dP V - V^-1 dQ W),
//   K_E[i,j] = i/(2k0) int_0^d exp(i(g_i(d-z) + g_j z)/k0) dz,
//   K_D[i,j] = i/(2k0) int_0^d exp(i(g_i + g_j) z/k0) dz.
// These are divided differences of exponentials; nearly equal eigenvalues take
// the series form, so degenerate modes need no separate treatment.
#include "common.cuh"
#include "kernels.h"

namespace vrc {

namespace {

constexpr double PI_D = 3.1415926535897932;  // src/rcwa/defns.h:25

inline dim3 grid_for(long long total, int batch, int threads = 256) {
  long long bx = (total + threads - 1) / threads;
  if (bx > 1024) bx = 1024;
  if (bx < 1) bx = 1;
  return dim3((unsigned)bx, (unsigned)batch);
}

__device__ __forceinline__ cplx cexp(cplx x) {
  double s, c;
  sincos(x.y, &s, &c);
  const double e = exp(x.x);
  return mk(e * c, e * s);
}

// (exp(x) - 1) / x for |x| < 0.1 by its Taylor series (terms to x^10).
__device__ __forceinline__ cplx phi_series(cplx x) {
  cplx s = mk(1.0, 0.0), term = mk(1.0, 0.0);
#pragma unroll
  for (int k = 2; k < 12; ++k) {
    term = cscale(cmul(term, x), 1.0 / k);
    s = cadd(s, term);
  }
  return s;
}

// int_0^d exp(i (a (d - z) + b z) / k0) dz
__device__ cplx int_exp2(cplx a, cplx b, double d, double k0) {
  const double t = d / k0;
  const cplx ea = cexp_i(a, t);
  const cplx x = mk(-(b.y - a.y) * t, (b.x - a.x) * t);  // i (b - a) d / k0
  if (fabs(x.x) + fabs(x.y) < 0.1) return cscale(cmul(ea, phi_series(x)), d);
  const cplx eb = cexp_i(b, t);
  return cscale(cdiv(csub(eb, ea), x), d);
}

// int_0^d exp(i s z / k0) dz
__device__ cplx int_exp1(cplx s, double d, double k0) {
  const double t = d / k0;
  const cplx x = mk(-s.y * t, s.x * t);  // i s d / k0
  if (fabs(x.x) + fabs(x.y) < 0.1) return cscale(phi_series(x), d);
  return cscale(cdiv(csub(cexp(x), mk(1.0, 0.0)), x), d);
}

__global__ void scale_kernel(const cplx* const* __restrict__ As, const cplx* const* __restrict__ rss,
                             const cplx* const* __restrict__ css, cplx* const* __restrict__ outs, int n) {
  const cplx* a = As[blockIdx.y];
  const cplx* rs = rss ? rss[blockIdx.y] : nullptr;
  const cplx* cs = css ? css[blockIdx.y] : nullptr;
  cplx* o = outs[blockIdx.y];
  const long long total = (long long)n * n;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx % n), j = (int)(idx / n);
    cplx v = a[idx];
    if (rs) v = cmul(rs[i], v);
    if (cs) v = cmul(v, cs[j]);
    o[idx] = v;
  }
}

__global__ void phase_vec_kernel(const cplx* const* __restrict__ gams, const double* __restrict__ ts,
                                 cplx* const* __restrict__ outs, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) outs[blockIdx.y][i] = cexp_i(gams[blockIdx.y][i], ts[blockIdx.y]);
}

__global__ void layer_adjoint_kernel(const LayerAdjDesc* __restrict__ ds, int n) {
  const LayerAdjDesc d = ds[blockIdx.y];
  const long long total = (long long)n * n;
  const cplx c = mk(0.0, 0.5 / d.k0);  // i / (2 k0)
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx % n), j = (int)(idx / n);
    const cplx gi = d.gam[i], gj = d.gam[j];
    const cplx KE = cmul(c, int_exp2(gi, gj, d.d, d.k0));
    const cplx KD = cmul(c, int_exp1(cadd(gi, gj), d.d, d.k0));
    const cplx gA = cmulc(KE, cadd(d.gtdd[idx], d.gtuu[idx]));
    const cplx gB = cneg(cmulc(KD, cadd(d.grud[idx], d.grdu[idx])));
    d.gS[idx] = cadd(gA, gB);
    d.gD[idx] = csub(gA, gB);
  }
}

// The thickness enters a layer's own-basis blocks only through
// X = diag(exp(i gam d / k0)); dX/dd = (i gam / k0) X.
__global__ void thick_adjoint_kernel(const ThickAdjDesc* __restrict__ ds, int n) {
  const ThickAdjDesc d = ds[blockIdx.x];
  __shared__ double red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const size_t ii = (size_t)i * n + i;
    const cplx g = cadd(d.gtdd[ii], d.gtuu[ii]);
    const cplx dx = cmul(mk(-d.gam[i].y / d.k0, d.gam[i].x / d.k0), d.x[i]);  // (i gam / k0) x
    s += g.x * dx.x + g.y * dx.y;                                              // Re(conj(g) dx)
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    *d.out = t;
  }
}

__global__ void interface_e_kernel(const IfFieldDesc* __restrict__ ds, int n) {
  const IfFieldDesc d = ds[blockIdx.x];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    cplx s = mk(0.0, 0.0);
    for (int k = 0; k < n; ++k) s = cfma(d.W[(size_t)k * n + i], cadd(d.ap[k], d.am[k]), s);
    d.e[i] = s;
  }
}

// Ex, Ey at pixel (p, q) = sum over harmonics of e_k exp(i (alpha_k x_p + beta_k y_q))
__global__ void field_image_kernel(const IfFieldDesc* __restrict__ ds, int m, int ngx, int ngy) {
  const IfFieldDesc d = ds[blockIdx.y];
  if (!d.img) return;
  const int npix = ngx * ngy;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < npix; idx += gridDim.x * blockDim.x) {
    const int q = idx / ngx, p = idx - q * ngx;
    const double x = d.Lx * p / ngx, y = d.Ly * q / ngy;
    cplx ex = mk(0.0, 0.0), ey = mk(0.0, 0.0);
    for (int k = 0; k < m; ++k) {
      double sn, cs;
      sincos(d.alpha[k] * x + d.beta[k] * y, &sn, &cs);
      const cplx ph = mk(cs, sn);
      ex = cfma(d.e[k], ph, ex);
      ey = cfma(d.e[m + k], ph, ey);
    }
    d.img[idx] = ex;
    d.img[npix + idx] = ey;
  }
}

__global__ void vec_axpy_kernel(const cplx* const* __restrict__ as, const cplx* const* __restrict__ bs, cplx s,
                                cplx* const* __restrict__ ys, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) ys[blockIdx.y][i] = cfma(s, bs[blockIdx.y][i], as[blockIdx.y][i]);
}

// dL/dP, dL/dQ of Layer::waveEqnCoeff (src/rcwa/Layer.cpp:36-171, periodic)
// -> dL/dfe11, dL/dfe22 and Z = dL/dF1 Kx + dL/dF2 Ky (F = fe33^-1 [Kx Ky]).
__global__ void pq_adjoint_kernel(const PQAdjDesc* __restrict__ ds, int m) {
  const PQAdjDesc d = ds[blockIdx.y];
  const int n = 2 * m;
  const double k2 = d.k0 * d.k0;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < m * m; idx += gridDim.x * blockDim.x) {
    const int i = idx % m, j = idx / m;
    auto at = [&](const cplx* M, int r, int col) { return M[(size_t)col * n + r]; };
    d.g11[idx] = cscale(at(d.gQ, m + i, j), k2);
    d.g22[idx] = cscale(at(d.gQ, i, m + j), -k2);
    const double ai = d.alpha[i], bi = d.beta[i], aj = d.alpha[j], bj = d.beta[j];
    const cplx gF2 = cadd(cscale(at(d.gP, i, j), ai), cscale(at(d.gP, m + i, j), bi));
    const cplx gF1 = cneg(cadd(cscale(at(d.gP, i, m + j), ai), cscale(at(d.gP, m + i, m + j), bi)));
    d.Z[idx] = cadd(cscale(gF1, aj), cscale(gF2, bj));
  }
}

// Twiddle factor of FourierSolver1D (src/rcwa/FourierSolver1D.cpp:11-41) for
// harmonic p - half and cell [x0, x1] of a period D.
__device__ cplx twiddle(int p, int half, double x0, double x1, double D) {
  const int mm = p - half;
  const double w = x1 - x0;
  if (mm == 0) return mk(w / D, 0.0);
  double sn, cs;
  sincos(-(mm * PI_D * (x1 + x0) / D), &sn, &cs);
  const double amp = sin(PI_D * mm * w / D) / (PI_D * mm);
  return mk(amp * cs, amp * sn);
}

// In-place inverse of a t x t column-major matrix by one warp (Gauss-Jordan,
// partial pivoting).  Returns false on a zero pivot.
__device__ bool warp_inverse(cplx* a, cplx* fcol, int* piv, int t, int lane) {
  bool ok = true;
  for (int k = 0; k < t; ++k) {
    double best = -1.0;
    int p = t;
    for (int i = k + lane; i < t; i += 32) {
      double v = cabs1(a[k * t + i]);
      if (v > best) { best = v; p = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      double ob = __shfl_xor_sync(0xffffffffu, best, o);
      int op = __shfl_xor_sync(0xffffffffu, p, o);
      if (ob > best || (ob == best && op < p)) { best = ob; p = op; }
    }
    if (!(best > 0.0)) { ok = false; p = k; }
    if (lane == 0) piv[k] = p;
    if (p != k)
      for (int j = lane; j < t; j += 32) {
        cplx tmp = a[j * t + k];
        a[j * t + k] = a[j * t + p];
        a[j * t + p] = tmp;
      }
    __syncwarp();
    const cplx ip = (best > 0.0) ? cinv(a[k * t + k]) : mk(1.0, 0.0);
    for (int i = lane; i < t; i += 32) fcol[i] = a[k * t + i];
    __syncwarp();
    for (int j = lane; j < t; j += 32) {
      cplx v = (j == k) ? mk(1.0, 0.0) : a[j * t + k];
      a[j * t + k] = cmul(v, ip);
    }
    __syncwarp();
    for (int j = lane; j < t; j += 32) {
      const cplx prow = a[j * t + k];
      for (int i = 0; i < t; ++i) {
        if (i == k) continue;
        cplx v = (j == k) ? mk(0.0, 0.0) : a[j * t + i];
        a[j * t + i] = csub(v, cmul(fcol[i], prow));
      }
    }
    __syncwarp();
  }
  for (int k = t - 1; k >= 0; --k) {
    const int p = piv[k];
    if (p != k)
      for (int i = lane; i < t; i += 32) {
        cplx tmp = a[k * t + i];
        a[k * t + i] = a[p * t + i];
        a[p * t + i] = tmp;
      }
    __syncwarp();
  }
  return ok;
}

constexpr int PX_THREADS = 256, PX_WARPS = PX_THREADS / 32;

// dL/d(pixel) from dL/dfe11, dL/dfe22, dL/dfe33 on a uniform npy x npx grid
// (FourierSolver2D::solve, src/rcwa/FourierSolver2D.cpp:43-349: Laurent rule
// for fe33, Li's inverse rule for fe11 (y strips) and fe22 (x columns)).  First
// the Toeplitz-diagonal sums of the three (K11, K22, gf, in the layer's
// scratch), then one warp per strip: all rows of all layers, each row's pixels
// written (fe33 and fe11), then all columns, added to (fe22).  The per-strip
// Toeplitz inverses are recomputed.  Bound by the strips' serial inversions, so
// they are spread over the GPU: with one CTA per layer doing all its strips, a
// layer after the other, the four layers of one 9 x 9-order stack of 64 x 64
// pixels took 4.5 ms.
__global__ void pixel_sums_kernel(const PixAdjDesc* __restrict__ ds, int nx, int ny) {
  const PixAdjDesc d = ds[blockIdx.y];
  const int P = 2 * nx - 1, Q = 2 * ny - 1, m = nx * ny;
  cplx* K11 = d.kscr;                        // [Q][nx][nx]
  cplx* K22 = K11 + (size_t)Q * nx * nx;     // [P][ny][ny]
  cplx* gf = K22 + (size_t)P * ny * ny;      // [Q][P]
  auto G = [&](const cplx* M, int a, int c, int b, int dd) { return M[(size_t)(b * ny + dd) * m + a * ny + c]; };
  const int n1 = Q * nx * nx, n2 = P * ny * ny, n3 = P * Q;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n1 + n2 + n3; e += gridDim.x * blockDim.x) {
    cplx s = mk(0.0, 0.0);
    if (e < n1) {
      const int q = e / (nx * nx), rem = e - q * nx * nx, b = rem / nx, a = rem - b * nx;
      const int qq = q - (ny - 1);
      for (int c = max(0, qq); c < min(ny, ny + qq); ++c) s = cadd(s, G(d.g11, a, c, b, c - qq));
      K11[e] = s;
    } else if (e < n1 + n2) {
      const int idx = e - n1, p = idx / (ny * ny), rem = idx - p * ny * ny, dd = rem / ny, c = rem - dd * ny;
      const int pp = p - (nx - 1);
      for (int a = max(0, pp); a < min(nx, nx + pp); ++a) s = cadd(s, G(d.g22, a, c, a - pp, dd));
      K22[idx] = s;
    } else {
      const int idx = e - n1 - n2, q = idx / P, p = idx - q * P;
      const int pp = p - (nx - 1), qq = q - (ny - 1);
      for (int a = max(0, pp); a < min(nx, nx + pp); ++a)
        for (int c = max(0, qq); c < min(ny, ny + qq); ++c) s = cadd(s, G(d.g33, a, c, a - pp, c - qq));
      gf[idx] = s;
    }
  }
}

// Per-warp shared memory (complex elements) of a strip of `len` pixels with t
// harmonics along it and ho Fourier coefficients across it.
__host__ __device__ inline int px_strip_scratch(int t, int len, int ho) {
  return 3 * t * t + 3 * (2 * t - 1) + t + len + ho;
}

template <bool ROWS>
__global__ void __launch_bounds__(PX_THREADS)
    pixel_strip_kernel(const PixAdjDesc* __restrict__ ds, int nx, int ny, int npx, int npy) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PixAdjDesc d = ds[blockIdx.y];
  const int P = 2 * nx - 1, Q = 2 * ny - 1, NW = blockDim.x >> 5;
  // along the strip: t harmonics, H coefficients, len pixels; across: HO
  const int t = ROWS ? nx : ny, H = 2 * t - 1, HO = ROWS ? Q : P, len = ROWS ? npx : npy;
  const int strips = ROWS ? npy : npx, to = ROWS ? ny : nx;
  const double D = ROWS ? d.Lx : d.Ly, DO = ROWS ? d.Ly : d.Lx;
  const cplx* K = d.kscr + (ROWS ? 0 : (size_t)Q * nx * nx);  // [HO][t][t]
  const cplx* gf = d.kscr + (size_t)Q * nx * nx + (size_t)P * ny * ny;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  cplx* E = reinterpret_cast<cplx*>(smem_raw);  // [len][H]
  cplx* T = E + (size_t)len * H + (size_t)warp * px_strip_scratch(t, len, HO);
  cplx* gT = T + t * t;
  cplx* tmp = gT + t * t;
  cplx* gvec = tmp + t * t;  // H: Fourier coefficients of 1/eps
  cplx* gv = gvec + H;       // H: Toeplitz-diagonal adjoint
  cplx* v33 = gv + H;        // H: this row of dL/dfe33
  cplx* fcol = v33 + H;      // t
  cplx* w = fcol + t;        // len: 1/eps
  cplx* eo = w + len;        // HO: twiddles across the strip
  int* piv = reinterpret_cast<int*>(E + (size_t)len * H + (size_t)NW * px_strip_scratch(t, len, HO)) + warp * 32;
  for (int idx = tid; idx < len * H; idx += blockDim.x) {
    const int c = idx / H, p = idx - c * H;
    E[idx] = twiddle(p, t - 1, D * c / len, D * (c + 1) / len, D);
  }
  __syncthreads();
  const int r = blockIdx.x * NW + warp;  // this warp's strip
  if (r >= strips) return;
  const cplx* er = d.eps + (ROWS ? (size_t)r * npx : r);
  double* gr = d.grad + (ROWS ? (size_t)r * npx : r);
  const int st = ROWS ? 1 : npx;
  for (int c = lane; c < len; c += 32) w[c] = cinv(er[(size_t)c * st]);
  for (int q = lane; q < HO; q += 32) eo[q] = twiddle(q, to - 1, DO * r / strips, DO * (r + 1) / strips, DO);
  __syncwarp();
  for (int p = lane; p < H; p += 32) {
    cplx s = mk(0.0, 0.0), u = s;
    for (int c = 0; c < len; ++c) s = cadd(s, cmul(E[c * H + p], w[c]));
    gvec[p] = s;
    if (ROWS) {
      for (int q = 0; q < HO; ++q) u = cadd(u, cmulc(eo[q], gf[q * H + p]));
      v33[p] = u;
    }
  }
  __syncwarp();
  for (int idx = lane; idx < t * t; idx += 32) {
    const int k = idx / t, i = idx - k * t;
    T[k * t + i] = gvec[t - 1 + i - k];
  }
  __syncwarp();
  warp_inverse(T, fcol, piv, t, lane);
  // gT[a,b] = sum_q conj(eo[q]) K[q, b, a]
  for (int idx = lane; idx < t * t; idx += 32) {
    cplx s = mk(0.0, 0.0);
    for (int q = 0; q < HO; ++q) s = cadd(s, cmulc(eo[q], K[(size_t)q * t * t + idx]));
    gT[idx] = s;
  }
  __syncwarp();
  // tmp = T^H gT ; gT <- -tmp T^H
  for (int idx = lane; idx < t * t; idx += 32) {
    const int b = idx / t, a = idx - b * t;
    cplx s = mk(0.0, 0.0);
    for (int k = 0; k < t; ++k) s = cadd(s, cmulc(T[a * t + k], gT[b * t + k]));
    tmp[b * t + a] = s;
  }
  __syncwarp();
  for (int idx = lane; idx < t * t; idx += 32) {
    const int b = idx / t, a = idx - b * t;
    cplx s = mk(0.0, 0.0);
    for (int k = 0; k < t; ++k) s = cadd(s, cmul(tmp[k * t + a], cconj(T[k * t + b])));
    gT[b * t + a] = cneg(s);
  }
  __syncwarp();
  for (int k = lane; k < H; k += 32) {
    const int off = k - (t - 1);  // a - b
    cplx s = mk(0.0, 0.0);
    for (int b = max(0, -off); b < min(t, t - off); ++b) s = cadd(s, gT[b * t + b + off]);
    gv[k] = s;
  }
  __syncwarp();
  for (int c = lane; c < len; c += 32) {
    cplx s = mk(0.0, 0.0);
    double s33 = 0.0;
    for (int k = 0; k < H; ++k) {
      const cplx e = E[c * H + k];
      s = cadd(s, cmulc(e, gv[k]));
      if (ROWS) s33 += e.x * v33[k].x + e.y * v33[k].y;
    }
    const cplx w2 = cmul(w[c], w[c]);
    const double g = -(w2.x * s.x + w2.y * s.y);  // Re conj(-w^2) s
    gr[(size_t)c * st] = ROWS ? s33 + g : gr[(size_t)c * st] + g;
  }
}

// Per-order powers of a stack (RCWASolver::scatterPlaneWave,
// src/rcwa/RCWASolver.cpp:1636-1733, incidence from the z0 medium, flux
// normalised) and, with adj != 0, dL/dRdu and dL/dTuu for
// L = sum_k wR[k] REF[k] + wT[k] TRN[k] (rank-one: (W^H g) c^H).
__global__ void stack_power_kernel(const StackPowerDesc* __restrict__ ds, int m, int adj) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const StackPowerDesc d = ds[blockIdx.x];
  const int n = 2 * m;
  cplx* c = reinterpret_cast<cplx*>(smem_raw);
  cplx* u = c + n;
  cplx* v = u + n;
  cplx* r = v + n;
  cplx* tt = r + n;
  cplx* gr = tt + n;
  cplx* gt = gr + n;
  const int tid = threadIdx.x;
  const int ctr = (d.ny * (d.nx - 1)) / 2 + (d.ny - 1) / 2;
  for (int i = tid; i < n; i += blockDim.x)
    c[i] = cadd(cscale(d.W0inv[(size_t)ctr * n + i], d.px), cscale(d.W0inv[(size_t)(m + ctr) * n + i], d.py));
  __syncthreads();
  for (int i = tid; i < n; i += blockDim.x) {
    cplx a = mk(0.0, 0.0), b = mk(0.0, 0.0);
    for (int k = 0; k < n; ++k) {
      a = cfma(d.Tuu[(size_t)k * n + i], c[k], a);
      b = cfma(d.Rdu[(size_t)k * n + i], c[k], b);
    }
    u[i] = a;
    v[i] = b;
  }
  __syncthreads();
  for (int i = tid; i < n; i += blockDim.x) {
    cplx a = mk(0.0, 0.0), b = mk(0.0, 0.0);
    for (int k = 0; k < n; ++k) {
      a = cfma(d.W1[(size_t)k * n + i], u[k], a);
      b = cfma(d.W0[(size_t)k * n + i], v[k], b);
    }
    tt[i] = a;
    r[i] = b;
  }
  __syncthreads();
  const double norm = sqrt(d.eps_in.x) * d.k0;
  for (int i = tid; i < m; i += blockDim.x) {
    const double a = d.alpha[i], b = d.beta[i];
    const cplx kzr = cneg(csqrt(mk(d.k0 * d.k0 * d.eps_in.x - a * a - b * b, d.k0 * d.k0 * d.eps_in.y)));
    const cplx kzt = csqrt(mk(d.k0 * d.k0 * d.eps_out.x - a * a - b * b, d.k0 * d.k0 * d.eps_out.y));
    for (int side = 0; side < 2; ++side) {
      const cplx kz = side ? kzt : kzr;
      cplx* f = side ? tt : r;
      const cplx fx = f[i], fy = f[i + m];
      double Pw = 0.0;
      cplx ux = mk(0.0, 0.0), uy = mk(0.0, 0.0), fz = mk(0.0, 0.0);
      if (kz.x != 0.0 || kz.y != 0.0) {
        ux = cdiv(mk(a, 0.0), kz);
        uy = cdiv(mk(b, 0.0), kz);
        fz = cadd(cmul(ux, fx), cmul(uy, fy));
        Pw = fabs(kz.x) * (cabs2(fx) + cabs2(fy) + cabs2(fz)) / norm;
      }
      if (side) d.TRN[i] = Pw; else d.REF[i] = Pw;
      if (adj) {
        const double w = side ? d.wT[i] : d.wR[i];
        const double aw = 2.0 * w * fabs(kz.x) / norm;
        cplx* g = side ? gt : gr;
        g[i] = cscale(cadd(fx, cmulc(ux, fz)), aw);
        g[i + m] = cscale(cadd(fy, cmulc(uy, fz)), aw);
      }
    }
  }
  if (!adj) return;
  __syncthreads();
  // u <- W1^H gt, v <- W0^H gr
  for (int i = tid; i < n; i += blockDim.x) {
    cplx a = mk(0.0, 0.0), b = mk(0.0, 0.0);
    for (int k = 0; k < n; ++k) {
      a = cadd(a, cmulc(d.W1[(size_t)i * n + k], gt[k]));
      b = cadd(b, cmulc(d.W0[(size_t)i * n + k], gr[k]));
    }
    u[i] = a;
    v[i] = b;
  }
  __syncthreads();
  for (long long idx = tid; idx < (long long)n * n; idx += blockDim.x) {
    const int i = (int)(idx % n), j = (int)(idx / n);
    const cplx cj = cconj(c[j]);
    d.gTuu[idx] = cmul(u[i], cj);
    d.gRdu[idx] = cmul(v[i], cj);
  }
}

}  // namespace

void scale_batched(const cplx* const* A, const cplx* const* rs, const cplx* const* cs, cplx* const* out, int batch,
                   int n, cudaStream_t st) {
  if (batch <= 0) return;
  scale_kernel<<<grid_for((long long)n * n, batch), 256, 0, st>>>(A, rs, cs, out, n);
  VRC_CUDA_CHECK(cudaGetLastError());
}

void phase_vec_batched(const cplx* const* gam, const double* t, cplx* const* out, int batch, int n, cudaStream_t st) {
  if (batch <= 0) return;
  dim3 grid((n + 127) / 128, batch);
  phase_vec_kernel<<<grid, 128, 0, st>>>(gam, t, out, n);
  VRC_CUDA_CHECK(cudaGetLastError());
}

void layer_adjoint_batched(const LayerAdjDesc* d, int batch, int n, cudaStream_t st) {
  if (batch <= 0) return;
  layer_adjoint_kernel<<<grid_for((long long)n * n, batch), 256, 0, st>>>(d, n);
  VRC_CUDA_CHECK(cudaGetLastError());
}

void pq_adjoint_batched(const PQAdjDesc* d, int batch, int m, cudaStream_t st) {
  if (batch <= 0) return;
  pq_adjoint_kernel<<<grid_for((long long)m * m, batch), 256, 0, st>>>(d, m);
  VRC_CUDA_CHECK(cudaGetLastError());
}

void interface_fields_batched(const IfFieldDesc* d, int batch, int n, int ngx, int ngy, cudaStream_t st) {
  if (batch <= 0) return;
  interface_e_kernel<<<batch, 256, 0, st>>>(d, n);
  VRC_CUDA_CHECK(cudaGetLastError());
  if (ngx > 0 && ngy > 0) {
    field_image_kernel<<<grid_for((long long)ngx * ngy, batch), 256, 0, st>>>(d, n / 2, ngx, ngy);
    VRC_CUDA_CHECK(cudaGetLastError());
  }
}

void vec_axpy_batched(const cplx* const* a, const cplx* const* b, cplx s, cplx* const* y, int batch, int n,
                      cudaStream_t st) {
  if (batch <= 0) return;
  dim3 grid((n + 127) / 128, batch);
  vec_axpy_kernel<<<grid, 128, 0, st>>>(a, b, s, y, n);
  VRC_CUDA_CHECK(cudaGetLastError());
}

void thick_adjoint_batched(const ThickAdjDesc* d, int batch, int n, cudaStream_t st) {
  if (batch <= 0) return;
  thick_adjoint_kernel<<<batch, 256, 0, st>>>(d, n);
  VRC_CUDA_CHECK(cudaGetLastError());
}

// Rasters that stacks take, at most 32 harmonics an axis: the bound of a kernel
// that held both directions' twiddle tables, the coefficients, one strip's
// matrices and the raster's sums in one CTA's shared memory.  The strips above
// hold one direction's table and what a warp needs, less at every size within it.
bool pixel_adjoint_fits(int nx, int ny, int npx, int npy) {
  if (nx > 32 || ny > 32) return false;
  const int P = 2 * nx - 1, Q = 2 * ny - 1, t = nx > ny ? nx : ny;
  const size_t c = (size_t)P * npx + (size_t)Q * npy + (size_t)P * Q + (size_t)Q * npx +
                   (size_t)(3 * t * t + 2 * (2 * t - 1) + t);
  return c * 16 + (size_t)npy * npx * 8 + 32 * sizeof(int) <= 227 * 1024;
}

size_t pixel_adjoint_scratch(int nx, int ny) {
  const int P = 2 * nx - 1, Q = 2 * ny - 1;
  return ((size_t)Q * nx * nx + (size_t)P * ny * ny + (size_t)P * Q) * 16;
}

void pixel_adjoint_batched(const PixAdjDesc* d, int batch, int nx, int ny, int npx, int npy, cudaStream_t st) {
  if (batch <= 0) return;
  if (!pixel_adjoint_fits(nx, ny, npx, npy))
    throw StatusError(ST_EINVAL, "pixel adjoint: raster and harmonics exceed the shared-memory tile");
  // strips per CTA: the most (up to eight) that leave room
  auto smem = [&](bool rows, int nw) {
    const int t = rows ? nx : ny, len = rows ? npx : npy, ho = 2 * (rows ? ny : nx) - 1;
    return ((size_t)len * (2 * t - 1) + (size_t)nw * px_strip_scratch(t, len, ho)) * 16 + nw * 32 * sizeof(int);
  };
  auto warps = [&](bool rows) {
    int nw = PX_WARPS;
    while (nw > 1 && smem(rows, nw) > 227 * 1024) nw /= 2;
    return nw;
  };
  const int wr = warps(true), wc = warps(false);
  ensure_smem((const void*)pixel_strip_kernel<true>, smem(true, wr));
  ensure_smem((const void*)pixel_strip_kernel<false>, smem(false, wc));
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    const int nb = batch - b0 < 65535 ? batch - b0 : 65535;
    pixel_sums_kernel<<<dim3(8, nb), 256, 0, st>>>(d + b0, nx, ny);
    pixel_strip_kernel<true><<<dim3((npy + wr - 1) / wr, nb), wr * 32, smem(true, wr), st>>>(d + b0, nx, ny, npx, npy);
    pixel_strip_kernel<false><<<dim3((npx + wc - 1) / wc, nb), wc * 32, smem(false, wc), st>>>(d + b0, nx, ny, npx,
                                                                                            npy);
  }
  VRC_CUDA_CHECK(cudaGetLastError());
}

void stack_power_batched(const StackPowerDesc* d, int batch, int m, int adj, cudaStream_t st) {
  if (batch <= 0) return;
  const size_t smem = (size_t)7 * 2 * m * 16;
  if (smem > 227 * 1024) throw StatusError(ST_EINVAL, "stack powers: n too large");
  ensure_smem((const void*)stack_power_kernel, smem);
  stack_power_kernel<<<batch, 256, smem, st>>>(d, m, adj);
  VRC_CUDA_CHECK(cudaGetLastError());
}

}  // namespace vrc

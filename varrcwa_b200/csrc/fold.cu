// Mirror symmetry of a unit cell (eps(-x, y) = eps(x, -y) = eps(x, y)).
//
// The harmonics then split into even and odd combinations along x and along
// y, and the wave equation of the cell into four independent ones.  With the
// parity (sx, sy) of Ex, Ey and Hx have (-sx, -sy) and Hy has (sx, sy): P and
// Q of src/rcwa/Layer.cpp:91-138 change sign with alpha or beta exactly where
// they couple such components.  The four classes have (m+1)/2, (m-1)/2,
// (m-1)/2 and (m+1)/2 modes (m = nx ny), so an n x n eigenproblem becomes four
// of a quarter of its order.  The two smaller classes are filled up with one
// decoupled mode, constant along z, so that all four have the order
// d = (m+1)/2 and share every batched stage.
//
// Classes k = 0..3: (even, even), (even, odd), (odd, even), (odd, odd).  Within
// a class the first component's harmonics come before the second's (Ex before
// Ey, Hx before Hy), each ordered by |a|, then |b|, odd combinations starting
// at 1; combinations are normalised.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace vrc {
namespace {

struct Parity {
  int nx2, ny2;  // (nx-1)/2, (ny-1)/2
  __device__ __forceinline__ int count(int ox, int oy) const { return (nx2 + 1 - ox) * (ny2 + 1 - oy); }
};

// Basis element e of a class in field E (h = 0) or H (h = 1): component
// (0: x, 1: y), parities and orders.  False for the fill-up mode.
__device__ __forceinline__ bool element(const Parity& q, int cls, int h, int e, int* comp, int* ox, int* oy, int* a,
                                        int* b) {
  int px = cls >> 1, py = cls & 1;  // odd along x / y: Ex and Hy
  if (h) {
    px ^= 1;
    py ^= 1;  // Hx
  }
  int c = 0, cnt = q.count(px, py);
  if (e >= cnt) {
    e -= cnt;
    c = 1;
    px ^= 1;
    py ^= 1;
    if (e >= q.count(px, py)) return false;
  }
  const int nb = q.ny2 + 1 - py;
  *comp = c;
  *ox = px;
  *oy = py;
  *a = e / nb + px;
  *b = e % nb + py;
  return true;
}

// P (E rows, H columns) and Q (H rows, E columns) of one class from the full
// matrices: the row's combination of entries in the column of the
// representative (a, b) with a, b >= 0 (by symmetry its other members give the
// same).  One thread per entry; four scattered reads each, bound by memory
// latency (2% of an eigen-decomposition of the folded order).
__global__ void fold_kernel(const FoldDesc* __restrict__ descs, int nx, int ny, int d) {
  const FoldDesc f = descs[blockIdx.y];
  const Parity q{(nx - 1) / 2, (ny - 1) / 2};
  const int m = nx * ny, n = 2 * m;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < 2 * d * d; idx += gridDim.x * blockDim.x) {
    const bool isQ = idx >= d * d;
    const int e = isQ ? idx - d * d : idx, col = e / d, row = e - col * d;
    const cplx* full = isQ ? f.Qfull : f.Pfull;
    int rc, rx, ry, ra, rb, cc, cx, cy, ca, cb;
    const bool hr = element(q, f.cls, isQ ? 1 : 0, row, &rc, &rx, &ry, &ra, &rb);
    const bool hc = element(q, f.cls, isQ ? 0 : 1, col, &cc, &cx, &cy, &ca, &cb);
    cplx v = mk(0.0, 0.0);
    if (hr && hc) {
      const size_t j = (size_t)(cc * m + (q.nx2 + ca) * ny + q.ny2 + cb) * n;
      const int ka = ra ? 2 : 1, kb = rb ? 2 : 1;
      for (int sa = 0; sa < ka; ++sa)
        for (int sb = 0; sb < kb; ++sb) {
          const cplx x = full[j + rc * m + (q.nx2 + (sa ? -ra : ra)) * ny + q.ny2 + (sb ? -rb : rb)];
          const bool neg = ((sa && rx) != (sb && ry));
          v = neg ? csub(v, x) : cadd(v, x);
        }
      const int kc = (ca ? 2 : 1) * (cb ? 2 : 1);
      v = cscale(v, sqrt((double)kc / (double)(ka * kb)));
    } else if (row == col && !hr && !hc) {
      v = mk(isQ ? -2.0 * f.k0sq : f.k0sq, 0.0);  // an evanescent mode of its own
    }
    (isQ ? f.Q : f.P)[e] = v;
  }
}

// Harmonics (Ex then Ey, 2 m) of a folded E vector.
__global__ void unfold_kernel(const UnfoldDesc* __restrict__ descs, int nx, int ny, int d) {
  const UnfoldDesc f = descs[blockIdx.x];
  const Parity q{(nx - 1) / 2, (ny - 1) / 2};
  const int m = nx * ny;
  for (int i = threadIdx.x; i < 2 * m; i += blockDim.x) f.out[i] = mk(0.0, 0.0);
  __syncthreads();
  for (int e = threadIdx.x; e < d; e += blockDim.x) {
    int c, ox, oy, a, b;
    if (!element(q, f.cls, 0, e, &c, &ox, &oy, &a, &b)) continue;
    const int ka = a ? 2 : 1, kb = b ? 2 : 1;
    const cplx v = cscale(f.in[e], sqrt(1.0 / (ka * kb)));
    for (int sa = 0; sa < ka; ++sa)
      for (int sb = 0; sb < kb; ++sb) {
        const bool neg = ((sa && ox) != (sb && oy));
        f.out[c * m + (q.nx2 + (sa ? -a : a)) * ny + q.ny2 + (sb ? -b : b)] = neg ? cneg(v) : v;
      }
  }
}

// An operator on E from its classes: entry (i, j) is the sum over the classes
// of their entries between the combinations that hold harmonics i and j.
__global__ void unfold_mat_kernel(const UnfoldMatDesc* __restrict__ descs, int nx, int ny, int d) {
  const UnfoldMatDesc f = descs[blockIdx.y];
  const Parity q{(nx - 1) / 2, (ny - 1) / 2};
  const int m = nx * ny, n = 2 * m;
  // place of harmonic i in class k, its weight there (0: not in the class)
  auto place = [&](int i, int k, int* e) -> double {
    const int c = i / m, a = (i - c * m) / ny - q.nx2, b = (i - c * m) % ny - q.ny2;
    const int ox = (k >> 1) ^ c, oy = (k & 1) ^ c, ua = abs(a), ub = abs(b);
    if (ua < ox || ub < oy) return 0.0;
    *e = (c ? q.count(ox ^ 1, oy ^ 1) : 0) + (ua - ox) * (q.ny2 + 1 - oy) + ub - oy;
    const double w = sqrt(1.0 / ((ua ? 2 : 1) * (ub ? 2 : 1)));
    return ((a < 0 && ox) != (b < 0 && oy)) ? -w : w;
  };
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n * n; idx += gridDim.x * blockDim.x) {
    const int j = idx / n, i = idx - j * n;
    cplx v = mk(0.0, 0.0);
    for (int k = 0; k < 4; ++k) {
      int ei = 0, ej = 0;
      const double w = place(i, k, &ei) * place(j, k, &ej);
      if (w != 0.0) v = cadd(v, cscale(f.in[k][(size_t)ej * d + ei], w));
    }
    f.out[idx] = v;
  }
}

// status[s] = ST_ASYMMETRIC where a raster differs from one of its mirror images.
__global__ void mirror_check_kernel(const cplx* const* __restrict__ eps, int npx, int npy, int* __restrict__ status) {
  const cplx* e = eps[blockIdx.y];
  bool same = true;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < npx * npy; idx += gridDim.x * blockDim.x) {
    const int row = idx / npx, col = idx - row * npx;
    const cplx v = e[idx], x = e[(size_t)row * npx + npx - 1 - col], y = e[(size_t)(npy - 1 - row) * npx + col];
    same = same && v.x == x.x && v.y == x.y && v.x == y.x && v.y == y.y;
  }
  if (__syncthreads_or(!same) && threadIdx.x == 0) status[blockIdx.y] = ST_ASYMMETRIC;
}

}  // namespace

void fold_batched(const FoldDesc* d, int batch, int nx, int ny, cudaStream_t st) {
  if (batch <= 0) return;
  const int o = fold_order(nx, ny), blocks = std::min(256, (2 * o * o + 255) / 256);
  for (int b0 = 0; b0 < batch; b0 += 65535)
    fold_kernel<<<dim3(blocks, std::min(65535, batch - b0)), 256, 0, st>>>(d + b0, nx, ny, o);
  VRC_CUDA_CHECK(cudaGetLastError());
}
void unfold_batched(const UnfoldDesc* d, int batch, int nx, int ny, cudaStream_t st) {
  if (batch <= 0) return;
  unfold_kernel<<<batch, 128, 0, st>>>(d, nx, ny, fold_order(nx, ny));
  VRC_CUDA_CHECK(cudaGetLastError());
}
void unfold_matrices(const UnfoldMatDesc* d, int batch, int nx, int ny, cudaStream_t st) {
  if (batch <= 0) return;
  const int n = 2 * nx * ny, blocks = std::min(256, (n * n + 255) / 256);
  for (int b0 = 0; b0 < batch; b0 += 65535)
    unfold_mat_kernel<<<dim3(blocks, std::min(65535, batch - b0)), 256, 0, st>>>(d + b0, nx, ny, fold_order(nx, ny));
  VRC_CUDA_CHECK(cudaGetLastError());
}
void mirror_check(const cplx* const* d_eps, int batch, int npx, int npy, int* d_status, cudaStream_t st) {
  if (batch <= 0) return;
  const int blocks = std::min(64, (npx * npy + 255) / 256);
  for (int b0 = 0; b0 < batch; b0 += 65535)
    mirror_check_kernel<<<dim3(blocks, std::min(65535, batch - b0)), 256, 0, st>>>(d_eps + b0, npx, npy,
                                                                                  d_status + b0);
  VRC_CUDA_CHECK(cudaGetLastError());
}

}  // namespace vrc

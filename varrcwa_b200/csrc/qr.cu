// Complex Schur form by implicitly shifted QR with several bulges per sweep
// (FP64, one CTA per matrix), plus the replay of the logged rotations onto
// the Schur vectors and the parts of T outside the active window.
//
// Sweep on the active window [m, i] with nb shifts (the eigenvalues of the
// trailing nb x nb block; one Wilkinson or exceptional shift when nb = 1):
// bulge a (warp a) is introduced at round 3a and moves one position per
// round, so in round r it performs step k = m + r - 3a.  Bulges three apart
// use rotations on disjoint index pairs, so in a round every entry receives
// at most one row transform and one column transform.  Rounds run in chunks
// of QB inside a diagonal window D held in shared memory, in three steps with
// a CTA barrier after each: one warp forms all bulges' rotations (a lane per
// bulge), every warp transforms its bulge's rows, every warp transforms its
// bulge's columns.  (A barrier costs some 30 cycles; merging the steps, with
// every warp forming its own rotation and the entries that two bulges share
// handled apart, cost about 500 instructions per warp and round, and with
// two CTAs per SM the instruction issue is what a round is bound by: 1,900
// cycles per round at n = 242 then, 1,140 now.)  After a chunk the rest of
// the active window is updated from strips staged in shared memory
// (strip_rounds).  Rows above the
// window, columns right of it and all of Z are not touched here: every
// sweep's rotations are logged round-major and replayed afterwards
// (qr_replay_rows_kernel / qr_replay_cols_kernel).  For
// any entry, eager in-window updates precede deferred column transforms,
// which precede deferred row transforms (the window's bottom only moves up
// and windows never straddle a zero subdiagonal), so the replay reproduces
// the full transformation.
//
// Deflation: small subdiagonals (Ahues-Tisseur test) split the window;
// exceptional shifts at iterations 10 and 20; at most 30*max(10,n)
// iterations per eigenvalue and 30n+300 in total, else ST_ENOCONV.  Before
// a sweep, aggressive early deflation examines the trailing jw x jw block of
// the window (aed_* below): its converged eigenvalues deflate at once, and
// its unconverged ones are the sweep's shifts.  Its similarity transform U is
// applied eagerly inside the active window and logged as a dense block for
// the replay, in sequence with the sweeps' rotations.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "householder.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace vrc {
namespace {

constexpr int QR_THREADS = 256;
constexpr int NBMAX = QR_THREADS / 32;           // bulges per sweep (one warp each)
constexpr int QB = 40;                           // rounds per chunk
constexpr int QD = QB + 3 * (NBMAX - 1) + 3;     // diagonal window size (64: two entries per lane)
// leading dimension of the window: odd in 16-byte units, so that the lanes
// of a row access (stride QLD) fall in distinct shared-memory banks
constexpr int QLD = QD + 1;
// strips of the active window outside D: groups of FV vectors (rows or
// columns) per warp, at most FE entries each, double buffered in D's room
constexpr int FV = 4, FE = QB + 3 * (NBMAX - 1) + 1;
constexpr int QR_D = QD * QLD > NBMAX * 2 * FV * FE ? QD * QLD : NBMAX * 2 * FV * FE;
constexpr size_t QR_SMEM = (size_t)(QR_D + NBMAX * QB) * sizeof(cplx) + (size_t)NBMAX * QB * sizeof(double);

struct QrLogHeader {
  int nsweeps, nrot;
  int nrounds, naed;                           // statistics (naed: deflation-window blocks)
  long long t_defl, t_shift, t_rounds, t_far;  // statistics: SM clock cycles per phase
  long long t_wschur, t_wdefl;                 // statistics: window Schur form, window deflation
};
constexpr int QR_HDR = sizeof(QrLogHeader);  // 64
// A sweep on the active window [m, i] with nb bulges and R rounds; its
// rotations are stored round-major from rotation index start: round u,
// bulge b at start + u*nb + b, acting on the pair (k, k+1), k = m + u - 3b,
// when m <= k <= i - 1 (other slots are padding and never read).  A
// deflation-window block on the active window [m, i] has nb = -1: the
// unitary U of order R (columns and rows pad0..i) is stored column-major
// (leading dimension R) from rotation index start.
struct QrSweep {
  int m, i, nb, R;
  int start, pad0, pad1, pad2;
};

}  // namespace

long long schur_rot_cap(int n) { return 6LL * n * n + 64; }
int schur_sweep_cap(int n) { return 30 * n + 301; }  // the total iteration cap + 1
size_t schur_log_bytes(int n) {
  size_t b = QR_HDR + (size_t)schur_sweep_cap(n) * sizeof(QrSweep) + (size_t)schur_rot_cap(n) * 2 * sizeof(cplx);
  return (b + 255) / 256 * 256;
}

namespace {

__device__ __forceinline__ QrSweep* log_sweeps(char* logb) { return reinterpret_cast<QrSweep*>(logb + QR_HDR); }
__device__ __forceinline__ cplx* log_rot(char* logb, int sweep_cap) {
  return reinterpret_cast<cplx*>(logb + QR_HDR + (size_t)sweep_cap * sizeof(QrSweep));
}

// Complex Givens rotation G = [c s; -conj(s) c], c real, with
// G (f, g)^T = (r, 0)^T.  The whole rotation comes from one reciprocal square
// root, u = 1 / (|f| sqrt(|f|^2 + |g|^2)): c = |f|^2 u, s = f conj(g) u,
// r = f (|f|^2 + |g|^2) u.  A reflector (sqrt, two divisions, then seven
// dependent FMAs per application against three here) is a longer serial
// chain at every step.  Outside the range where the squares neither over- nor
// underflow the pair is scaled first.
struct Rot {
  double c;
  cplx s, r;
};
__device__ __forceinline__ Rot givens(cplx f, cplx g) {
  Rot o;
  const double f2 = cabs2(f), d2 = f2 + cabs2(g), u = rsqrt(f2 * d2);
  o.c = f2 * u;
  o.s = cscale(cmul(f, cconj(g)), u);
  o.r = cscale(f, d2 * u);
  if (!(f2 > 1e-140 && d2 < 1e140)) {  // f zero or far smaller than g, or squares out of range
    const double m = fmax(cabs1(f), cabs1(g)), sc = 1.0 / fmax(m, 1e-300);
    const cplx fs = cscale(f, sc), gs = cscale(g, sc);
    const double a2 = cabs2(fs), g2 = cabs2(gs);
    if (g2 < 1e-290) {
      o.c = 1.0;
      o.s = mk(0.0, 0.0);
      o.r = f;
    } else if (a2 < 1e-290) {
      const double ug = rsqrt(g2);
      o.c = 0.0;
      o.s = mk(gs.x * ug, -gs.y * ug);
      o.r = mk(g2 * ug * m, 0.0);
    } else {
      const double us = rsqrt(a2 * (a2 + g2));
      o.c = a2 * us;
      o.s = cscale(cmul(fs, cconj(gs)), us);
      o.r = cscale(f, (a2 + g2) * us);
    }
  }
  return o;
}

// The rotation on one pair (a, b): from the left (ROWOP, G) or, on a row of
// two columns, from the right (G^H).  The product with the pair's first
// entry, which a carried chain waits for, comes last.
template <bool ROWOP>
__device__ __forceinline__ void rotate2(cplx& a, cplx& b, double c, cplx s) {
  if (!ROWOP) s.y = -s.y;  // (p, w) -> (c p + conj(s) w, c w - s p)
  const cplx p = a, w = b;
  a = mk(fma(c, p.x, fma(s.x, w.x, -s.y * w.y)), fma(c, p.y, fma(s.x, w.y, s.y * w.x)));
  b = mk(fma(-s.y, p.y, fma(-s.x, p.x, c * w.x)), fma(s.y, p.x, fma(-s.x, p.y, c * w.y)));
}

// Principal square root of a value whose square is within range.
__device__ __forceinline__ cplx csqrt_inrange(cplx a) {
  const double a2 = cabs2(a);
  const double q = 0.5 * fma(a2, rsqrt(a2), fabs(a.x)), iq = rsqrt(q), t = q * iq;
  const double o = 0.5 * a.y * iq;
  return a.x >= 0.0 ? mk(t, o) : mk(fabs(o), copysign(t, a.y));
}

// Wilkinson's shift of the 2x2 block [p q; r t]: its eigenvalue closer to t,
// t - q r / (x +- sqrt(x^2 + q r)) with x = (p - t) / 2 and the sign that
// enlarges the denominator.  Out of range the entries are scaled first; a
// vanishing square root or denominator gives t.
__device__ __forceinline__ cplx wilkinson(cplx p, cplx q, cplx r, cplx t) {
  cplx x = cscale(csub(p, t), 0.5);
  double big = 1.0;
  cplx qr = cmul(q, r), z = cadd(cmul(x, x), qr);
  double z2 = cabs2(z);
  if (!(z2 > 1e-250 && z2 < 1e250)) {
    big = fmax(cabs1(x), fmax(cabs1(q), cabs1(r)));
    if (!(big > 1e-290)) return t;
    const double inv = 1.0 / big;
    x = cscale(x, inv);
    qr = cmul(cscale(q, inv), cscale(r, inv));
    z = cadd(cmul(x, x), qr);
    z2 = cabs2(z);
  }
  cplx w = z2 > 1e-280 ? csqrt_inrange(z) : mk(0.0, 0.0);
  if (x.x * w.x + x.y * w.y < 0.0) w = cneg(w);
  const cplx den = cadd(x, w);
  const double d2 = cabs2(den);
  if (!(d2 > 1e-280)) return t;
  const double rd = rsqrt(d2);
  return csub(t, cscale(cmul(qr, cconj(den)), big * rd * rd));
}

// Single shift for window [l, i]: exceptional at iterations 10 and 20, else
// Wilkinson's of the trailing 2x2 block.
__device__ __forceinline__ cplx single_shift(const cplx* H, int n, int l, int i, int its) {
  auto h = [&](int r, int c) { return H[(size_t)c * n + r]; };
  if (its == 10) return cadd(mk(0.75 * cabs1(h(l + 1, l)), 0.0), h(l, l));
  if (its == 20) return cadd(mk(0.75 * cabs1(h(i, i - 1)), 0.0), h(i, i));
  return wilkinson(h(i - 1, i - 1), h(i - 1, i), h(i, i - 1), h(i, i));
}

// cp.async copies of 16 bytes into shared memory, one commit group each; SHARED:
// past L1, for data that other CTAs of the cluster write.
template <bool SHARED = false>
__device__ __forceinline__ void cpa16(cplx* smem, const cplx* g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  if (SHARED)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(g) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(g) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpa_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// One chunk's rotations on FV vectors held in shared memory (entry e of vector
// v at e * FV + v), 8 lanes per vector, one per bulge.  In a round the bulges
// act on disjoint pairs, so the lanes work side by side: a lane carries its
// pair's second entry over to the next round, takes in the entry above it
// (left there by the leading bulge two rounds ago, so it is fetched a round
// ahead) and puts back the one it has passed.  p: this lane's first entry;
// rounds [ra0, ra1) of [r0, r1) are its own.  Bank conflict free: consecutive
// bulges are 3 FV entries apart.
//
// Bounded by issue with two CTAs per SM (12 FP64 instructions of about 30 per
// round and warp), else by a round's latency.  One thread per vector and bulge after bulge, straight from
// global memory, took 234 cycles per rotation at n = 242: on a row transform
// every lane walks a column of its own, so each access was 32 sectors, eight
// times over.
template <bool ROWOP>
__device__ __forceinline__ void strip_rounds(cplx* p, int r0, int r1, int ra0, int ra1, const double* cs,
                                             const cplx* ss) {
  if (__all_sync(0xffffffffu, ra0 == r0 && ra1 == r0 + QB)) {
    // a whole chunk inside the window for all bulges: no bounds to look at
    // (half the instructions of a round)
    cplx x = p[0], y = p[FV];
#pragma unroll 4
    for (int u = 0; u < QB; ++u) {
      const cplx nx = p[(min(u, QB - 2) + 2) * FV];
      rotate2<ROWOP>(x, y, cs[u * NBMAX], ss[u * NBMAX]);
      p[u * FV] = x;
      x = y;
      y = nx;
      __syncwarp();
    }
    p[QB * FV] = x;
    __syncwarp();
    return;
  }
  cplx x = mk(0.0, 0.0), y = x;
  for (int r = r0; r < r1; ++r, cs += NBMAX, ss += NBMAX) {
    if (r >= ra0 && r < ra1) {
      if (r == ra0) {
        x = p[0];
        y = p[FV];
      }
      const bool more = r + 1 < ra1;
      cplx nx = mk(0.0, 0.0);
      if (more) nx = p[2 * FV];
      rotate2<ROWOP>(x, y, cs[0], ss[0]);
      p[0] = x;
      if (!more) p[FV] = y;
      x = y;
      y = nx;
      p += FV;
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Aggressive early deflation (Braman, Byers & Mathias, "The multishift QR
// algorithm. Part II: aggressive early deflation", SIAM J. Matrix Anal.
// Appl. 23 (2002); LAPACK xLAQR3).  The trailing jw x jw block of the active
// window (jw <= AW, one lane per row or column) is brought to Schur form
// T = U^H H_w U by one warp in shared memory.  The subdiagonal entry s0 that
// couples the block to the rest becomes the spike s0 * conj(U[0, :]); an
// eigenvalue whose spike entry is negligible deflates, the others are moved
// to the top of T by swaps of adjacent diagonal entries.  If any deflated,
// the undeflated top block with its spike is returned to Hessenberg form
// (one reflector, then a Householder reduction) and U is applied to the rows
// of the active window above the block; the rest of H and Z receive U through
// the log (a dense entry, replayed like the sweeps).  The undeflated
// eigenvalues become the next sweep's shifts.
constexpr int AW = 32;       // largest deflation window
constexpr int ALD = AW + 1;  // its leading dimension in shared memory (odd in 16-byte units)

// Negligible subdiagonal entry sub = T[k][k-1] between the diagonal entries
// dkm = T[k-1][k-1] and dk = T[k][k], with sup = T[k-1][k] and the
// neighbouring subdiagonals below and above (Ahues-Tisseur, LAPACK xLAHQR).  The
// diagonal entries count as apart by their rounding at least: with equal ones
// and sub sup below its square the shift rounds to the diagonal and a step only
// exchanges the two, for ever.
__device__ __forceinline__ bool negligible(cplx sub, cplx dkm, cplx dk, cplx sup, cplx sub_up, cplx sub_dn,
                                           double smlnum) {
  const double cs = cabs1(sub);
  if (cs <= smlnum) return true;
  double tst = cabs1(dkm) + cabs1(dk);
  if (tst == 0.0) tst = cabs1(sub_up) + cabs1(sub_dn);
  if (cs > EIG_ULP * tst) return false;
  const double a2 = cabs1(sup);
  const double ab = fmax(cs, a2), ba = fmin(cs, a2);
  const double b1 = cabs1(dk), b2 = cabs1(csub(dkm, dk));
  const double aa = fmax(b1, b2), bb = fmin(b1, b2);
  return ba * ab <= fmax(smlnum * (aa + ab), EIG_ULP * aa * fmax(bb, EIG_ULP * aa));
}
__device__ __forceinline__ bool small_negligible(const cplx* T, int nw, int k, double smlnum) {
  auto t = [&](int r, int c) { return T[c * ALD + r]; };
  return negligible(t(k, k - 1), t(k - 1, k - 1), t(k, k), t(k - 1, k), k >= 2 ? t(k - 1, k - 2) : mk(0.0, 0.0),
                    k + 1 < nw ? t(k + 1, k) : mk(0.0, 0.0), smlnum);
}

__device__ __forceinline__ cplx shfl_c(cplx v, int src) {
  return mk(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// Schur form of the nw x nw upper Hessenberg T (shared memory, leading
// dimension ALD, nw <= AW) by single-shift QR with Wilkinson shifts
// (exceptional at iterations 10 and 20), accumulating the rotations into U
// (may be null).  One warp.  A step is explicit, T - sh I = Q R, then
// R Q + sh I (EISPACK's comqr), because its serial chain is the shortest: in
// the first half lane j carries column j's running entry in a register, so a
// rotation waits for one shuffle and one rotation of the step before; in the
// second every row is a chain of its own with all rotations known.  The
// implicit form hands two entries through shared memory twice per rotation
// and took 260,000 cycles for a 12 x 12 window with U.  rc, rs: room for AW
// rotations.  Returns false if an eigenvalue needs more than 30 * max(10, nw)
// iterations.
__device__ bool small_schur_warp(cplx* T, cplx* U, int nw, int lane, double smlnum, double* rc, cplx* rs) {
  auto t = [&](int r, int c) -> cplx& { return T[c * ALD + r]; };
  const cplx zero = mk(0.0, 0.0);
  const int itmax = 30 * max(10, nw);
  int hi = nw - 1, its = 0;
  while (hi > 0) {
    __syncwarp();
    // largest k <= hi with a negligible T[k][k-1] (lane k-1 tests k), else 0
    const bool negl = lane + 1 <= hi && small_negligible(T, nw, lane + 1, smlnum);
    const unsigned bal = __ballot_sync(0xffffffffu, negl);
    const int lo = bal ? 32 - __clz(bal) : 0;
    if (lo > 0 && lane == 0) t(lo, lo - 1) = zero;
    if (lo == hi) {
      --hi;
      its = 0;
      continue;
    }
    if (++its > itmax) return false;
    const cplx sh = single_shift(T, ALD, lo, hi, its);
    __syncwarp();  // every lane has read T
    {  // rows lo..hi, columns lo..nw-1; column j on lane j
      const int j = lane;
      const bool in = j < nw;
      cplx cur = (in && j >= lo) ? t(lo, j) : zero;
      if (j == lo) cur = csub(cur, sh);
      cplx b = (in && j > lo) ? t(lo + 1, j) : zero, y = t(lo + 1, lo);
      for (int k = lo; k < hi; ++k) {
        if (j == k + 1) b = csub(b, sh);
        cplx bn = zero, yn = zero;  // the next row's entries
        if (k + 1 < hi) {
          if (in && j > k + 1) bn = t(k + 2, j);
          yn = t(k + 2, k + 1);
        }
        const Rot g = givens(shfl_c(cur, k), y);
        rotate2<true>(cur, b, g.c, g.s);
        if (in && j >= k) t(k, j) = j == k ? g.r : cur;
        if (lane == 0) {
          rc[k] = g.c;
          rs[k] = g.s;
        }
        cur = b;
        b = bn;
        y = yn;
      }
      if (in && j >= hi) t(hi, j) = cur;
    }
    __syncwarp();
    // columns lo..hi of the rows of T and of U: row r of M as a chain
    auto chain = [&](cplx* M, int r, bool tri) {
      cplx p = (tri && r > lo) ? zero : M[lo * ALD + r];
      for (int k = lo; k < hi; ++k) {
        cplx w = (tri && r > k + 1) ? zero : M[(k + 1) * ALD + r];
        rotate2<false>(p, w, rc[k], rs[k]);
        M[k * ALD + r] = (tri && r == k) ? cadd(p, sh) : p;
        p = w;
      }
      M[hi * ALD + r] = (tri && r == hi) ? cadd(p, sh) : p;
    };
    if (nw <= 16) {  // both at once, on half a warp each
      const int r = lane & 15;
      const bool tri = lane < 16;
      if (tri ? r <= hi : (U != nullptr && r < nw)) chain(tri ? T : U, r, tri);
    } else {
      if (lane <= hi) chain(T, lane, true);
      if (U != nullptr && lane < nw) chain(U, lane, false);
    }
  }
  __syncwarp();
  return true;
}

// Swaps the adjacent diagonal entries k, k+1 of the upper triangular T and
// updates U (LAPACK xTREXC's step: T <- G T G^H, U <- U G^H).  One warp.
__device__ void schur_swap_warp(cplx* T, cplx* U, int nw, int k, int lane) {
  auto t = [&](int r, int c) -> cplx& { return T[c * ALD + r]; };
  auto u = [&](int r, int c) -> cplx& { return U[c * ALD + r]; };
  const cplx t11 = t(k, k), t22 = t(k + 1, k + 1), zero = mk(0.0, 0.0);
  const int j = k + 2 + lane;
  const bool row = j < nw, col = lane < k, uu = lane < nw;
  cplx a0 = zero, a1 = zero, b0 = zero, b1 = zero, u0 = zero, u1 = zero;
  if (row) a0 = t(k, j), a1 = t(k + 1, j);       // rows k, k+1 over columns k+2..nw-1
  if (col) b0 = t(lane, k), b1 = t(lane, k + 1);  // columns k, k+1 over rows 0..k-1
  if (uu) u0 = u(lane, k), u1 = u(lane, k + 1);
  const Rot g = givens(t(k, k + 1), csub(t22, t11));
  rotate2<true>(a0, a1, g.c, g.s);
  rotate2<false>(b0, b1, g.c, g.s);
  rotate2<false>(u0, u1, g.c, g.s);
  __syncwarp();
  if (row) t(k, j) = a0, t(k + 1, j) = a1;
  if (col) t(lane, k) = b0, t(lane, k + 1) = b1;
  if (uu) u(lane, k) = u0, u(lane, k + 1) = u1;
  if (lane == 0) t(k, k) = t22;
  if (lane == 1) t(k + 1, k + 1) = t11;
  __syncwarp();
}

// Reflector I - tau v v^H (v in shared memory, v[0] = 1) from the left,
// conjugated, on rows r0..r0+len-1 of T over columns c0..nc-1, and from the
// right on columns c0'..c0'+len-1 of a matrix over rows 0..nr-1.
__device__ __forceinline__ void refl_left_warp(cplx* T, const cplx* v, int r0, int len, cplx tau, int c0, int nc,
                                               int lane) {
  const int c = c0 + lane;
  if (c < nc) {
    cplx w = mk(0.0, 0.0);
    for (int q = 0; q < len; ++q) w = cadd(w, cmulc(v[q], T[c * ALD + r0 + q]));
    w = cmul(cconj(tau), w);
    for (int q = 0; q < len; ++q) T[c * ALD + r0 + q] = csub(T[c * ALD + r0 + q], cmul(v[q], w));
  }
}
__device__ __forceinline__ void refl_right_warp(cplx* M, const cplx* v, int c0, int len, cplx tau, int nr,
                                                int lane) {
  if (lane < nr) {
    cplx w = mk(0.0, 0.0);
    for (int q = 0; q < len; ++q) w = cadd(w, cmul(M[(c0 + q) * ALD + lane], v[q]));
    w = cmul(tau, w);
    for (int q = 0; q < len; ++q) M[(c0 + q) * ALD + lane] = csub(M[(c0 + q) * ALD + lane], cmul(w, cconj(v[q])));
  }
}

// Warp sum of a real value.
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// The deflation window's analysis by one warp (after small_schur_warp):
// deflation of the eigenvalues with negligible spike entries, reordering of
// the others to the top, their values into ev[0..ns-1], and, if anything
// deflated, the return of the top ns x ns block to Hessenberg form.
// Returns ns, the number of undeflated eigenvalues.
__device__ int aed_deflate_warp(cplx* T, cplx* U, cplx* v, cplx* ev, int nw, cplx s0, int lane, double smlnum) {
  auto t = [&](int r, int c) -> cplx& { return T[c * ALD + r]; };
  auto u = [&](int r, int c) -> cplx& { return U[c * ALD + r]; };
  int ns = nw;
  const double as0 = cabs1(s0);
  // bottom up: an entry that looks converged is brought to the bottom of the
  // undeflated block and tested there
  auto converged = [&](int j) {
    double foo = cabs1(t(j, j));
    if (foo == 0.0) foo = as0;
    return as0 * cabs1(u(0, j)) <= fmax(smlnum, EIG_ULP * foo);
  };
  for (int j = nw - 1; j >= 0; --j) {
    if (!converged(j)) continue;
    for (int k = j; k < ns - 1; ++k) schur_swap_warp(T, U, nw, k, lane);
    if (converged(ns - 1)) --ns;
  }
  if (lane < ns) ev[lane] = t(lane, lane);
  __syncwarp();
  if (ns == nw || ns <= 1 || (s0.x == 0.0 && s0.y == 0.0)) return ns;
  // reflector taking the spike's top ns entries to a multiple of e_0
  {
    const cplx sp = lane < ns ? cmul(s0, cconj(u(0, lane))) : mk(0.0, 0.0);
    const double xn2 = warp_sum(lane >= 1 ? cabs2(sp) : 0.0);
    const cplx alpha = mk(__shfl_sync(0xffffffffu, sp.x, 0), __shfl_sync(0xffffffffu, sp.y, 0));
    double beta;
    cplx tau, scale;
    householder(alpha, xn2, &beta, &tau, &scale);
    if (lane < ns) v[lane] = lane == 0 ? mk(1.0, 0.0) : cmul(sp, scale);
    __syncwarp();
    refl_left_warp(T, v, 0, ns, tau, 0, nw, lane);
    __syncwarp();
    refl_right_warp(T, v, 0, ns, tau, ns, lane);
    refl_right_warp(U, v, 0, ns, tau, nw, lane);
    __syncwarp();
  }
  // Householder reduction of the top ns x ns block to Hessenberg form
  for (int j = 0; j + 2 < ns; ++j) {
    const int len = ns - 1 - j;  // rows j+1..ns-1
    const cplx xr = (lane >= 1 && lane < len) ? t(j + 1 + lane, j) : mk(0.0, 0.0);
    const double xn2 = warp_sum(cabs2(xr));
    const cplx alpha = t(j + 1, j);
    double beta;
    cplx tau, scale;
    householder(alpha, xn2, &beta, &tau, &scale);
    __syncwarp();  // every lane has read column j
    if (lane < len) v[lane] = lane == 0 ? mk(1.0, 0.0) : cmul(xr, scale);
    if (lane == 0) t(j + 1, j) = mk(beta, 0.0);
    if (lane >= 1 && lane < len) t(j + 1 + lane, j) = mk(0.0, 0.0);
    __syncwarp();
    refl_left_warp(T, v, j + 1, len, tau, j + 1, nw, lane);
    __syncwarp();
    refl_right_warp(T, v, j + 1, len, tau, ns, lane);
    refl_right_warp(U, v, j + 1, len, tau, nw, lane);
    __syncwarp();
  }
  return ns;
}

// One chunk of a sweep, for the CTAs that transform what lies outside D.
struct Chunk {
  int m, i, nb, r0, r1, kmin, kmax, ds, de;  // m < 0: the matrix is done
};

// The rest of the active window: columns de+1..i (row transforms) and rows
// m..ds-1 (column transforms), FV vectors per warp at a time; every step-th
// group from first on.
__device__ __forceinline__ int far_groups(const Chunk& c) {
  return (c.i - c.de + FV - 1) / FV + (c.ds - c.m + FV - 1) / FV;
}
template <bool TEAM>
__device__ __forceinline__ void far_strips(cplx* H, int n, const Chunk& ch, cplx* D, const double* s_c,
                                           const cplx* s_s, int first, int step) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cnt = ch.kmax + 2 - ch.kmin;  // entries kmin..kmax+1 of each vector
  const int gr = (ch.i - ch.de + FV - 1) / FV, ng = far_groups(ch);
  cplx* buf = D + (size_t)warp * 2 * FV * FE;
  auto where = [&](int g, cplx*& x, size_t& es, size_t& vs, int& nv) {
    if (g < gr) {  // columns
      const int c0 = ch.de + 1 + g * FV;
      x = H + (size_t)c0 * n + ch.kmin;
      es = 1;
      vs = n;
      nv = min(FV, ch.i + 1 - c0);
    } else {  // rows
      const int q0 = ch.m + (g - gr) * FV;
      x = H + (size_t)ch.kmin * n + q0;
      es = n;
      vs = 1;
      nv = min(FV, ch.ds - q0);
    }
  };
  auto fetch = [&](int g, int half) {
    cplx* x;
    size_t es, vs;
    int nv;
    where(g, x, es, vs, nv);
    const int v = lane % FV;
    if (v < nv)
      for (int e = lane / FV; e < cnt; e += 32 / FV)
        cpa16<TEAM>(buf + half * FV * FE + e * FV + v, x + (size_t)e * es + (size_t)v * vs);
    cpa_commit();
  };
  const int b = lane / FV;  // this lane's bulge
  const int ra0 = max(ch.r0, 3 * b), ra1 = b < ch.nb ? min(ch.r1, 3 * b + (ch.i - ch.m)) : ch.r0;
  const int off = (ch.m + ra0 - 3 * b - ch.kmin) * FV + lane % FV;
  if (first < ng) fetch(first, 0);
  for (int g = first, half = 0; g < ng; g += step, half ^= 1) {
    if (g + step < ng) {
      fetch(g + step, half ^ 1);
      cpa_wait<1>();
    } else {
      cpa_wait<0>();
    }
    __syncwarp();
    cplx* vec = buf + half * FV * FE;
    if (g < gr)
      strip_rounds<true>(vec + off, ch.r0, ch.r1, ra0, ra1, s_c + b, s_s + b);
    else
      strip_rounds<false>(vec + off, ch.r0, ch.r1, ra0, ra1, s_c + b, s_s + b);
    cplx* x;
    size_t es, vs;
    int nv;
    where(g, x, es, vs, nv);
    const int v = lane % FV;
    if (v < nv)
      for (int e = lane / FV; e < cnt; e += 32 / FV) x[(size_t)e * es + (size_t)v * vs] = vec[e * FV + v];
    __syncwarp();  // the buffer is free for the group after next
  }
}

// Two CTAs per SM, which is what their shared memory allows.  TEAM: a cluster per
// matrix.  Its first CTA iterates; the others wait for its chunks and take their
// share of the strips outside D (at n = 450 on one CTA 44% of the iteration),
// which changes nothing in the arithmetic.
template <bool TEAM>
__global__ void __launch_bounds__(QR_THREADS, 2)
    hqr_kernel(cplx* const* __restrict__ Hs, void* const* __restrict__ logs, cplx* const* __restrict__ Ws, int n,
               int sweep_cap, long long rot_cap, int* __restrict__ status, int aed_min, int aed_w) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* D = reinterpret_cast<cplx*>(smem_raw);  // [QD][QLD] column-major window
  cplx* s_s = D + QR_D;                                       // [QB][NBMAX] rotations: s
  double* s_c = reinterpret_cast<double*>(s_s + NBMAX * QB);  // [QB][NBMAX] and c
  __shared__ cplx s_shift[NBMAX];
  __shared__ cplx s_small[NBMAX * ALD];
  __shared__ int s_red[QR_THREADS / 32];
  __shared__ int s_l, s_nb, s_nsw, s_nrot, s_over, s_nround, s_cur;
  // deflation window: reflector vector, undeflated eigenvalues, outcome
  // (undeflated count, or -1 when skipped), shifts it left for the next sweep
  __shared__ cplx s_aedv[AW], s_aedev[AW];
  __shared__ int s_aed_ns, s_pend, s_naed;
  __shared__ long long s_clk[7];  // statistics: phase timers (defl, shift, rounds, far), the last stamp,
                                  // window Schur form and window deflation

  __shared__ Chunk s_chunk;
  const int team = TEAM ? (int)cg::this_cluster().num_blocks() : 1;
  const int mat = blockIdx.x / team;
  // every CTA's writes to H are visible to the whole cluster
  auto team_sync = [&] {
    __threadfence();
    cg::this_cluster().sync();
    __threadfence();
  };
  cplx* H = Hs[mat];
  if (TEAM && cg::this_cluster().block_rank() != 0) {
    const int rank = (int)cg::this_cluster().block_rank(), wp = threadIdx.x >> 5;
    const Chunk* rc = cg::this_cluster().map_shared_rank(&s_chunk, 0);
    const cplx* rs = cg::this_cluster().map_shared_rank(s_s, 0);
    const double* rcs = cg::this_cluster().map_shared_rank(s_c, 0);
    for (;;) {
      team_sync();
      const Chunk ch = *rc;
      if (ch.m >= 0) {
        for (int q = threadIdx.x; q < NBMAX * (ch.r1 - ch.r0); q += QR_THREADS) {
          s_s[q] = rs[q];
          s_c[q] = rcs[q];
        }
        __syncthreads();
        far_strips<TEAM>(H, n, ch, D, s_c, s_s, NBMAX * rank + wp, NBMAX * team);
      }
      team_sync();
      if (ch.m < 0) return;
    }
  }
  char* logb = static_cast<char*>(logs[mat]);
  QrSweep* sweeps = log_sweeps(logb);
  cplx* rot = log_rot(logb, sweep_cap);
  cplx* W = Ws[mat];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double smlnum = EIG_SAFMIN * ((double)n / EIG_ULP);
  const int itmax = 30 * max(10, n);       // per eigenvalue
  const long long totmax = 30LL * n + 300;  // whole matrix
  long long tot = 0;
  auto h = [&](int r, int c) -> cplx& { return H[(size_t)c * n + r]; };
  if (tid == 0) {
    s_nsw = 0;
    s_pend = 0;
    s_naed = 0;
    s_nrot = 0;
    s_over = 0;
    s_nround = 0;
    for (int q = 0; q < 7; ++q) s_clk[q] = 0;
  }
  __syncthreads();
  // tid 0 only: charge the time since the last stamp to phase q
  auto stamp = [&](int q) {
    const long long t = clock64();
    if (q >= 0) s_clk[q] += t - s_clk[4];
    s_clk[4] = t;
  };
  int i = n - 1;
  int failed = 0;
  while (i >= 0) {
    int l = 0;
    int its;
    for (its = 0; its <= itmax && tot <= totmax; ++its, ++tot) {
      if (tid == 0) stamp(-1);
      // Deflation search: largest k in (l, i] with a negligible H[k][k-1].
      int best = l;
      for (int k = l + 1 + tid; k <= i; k += QR_THREADS) {
        const bool small =
            negligible(h(k, k - 1), h(k - 1, k - 1), h(k, k), h(k - 1, k), k >= 2 ? h(k - 1, k - 2) : mk(0.0, 0.0),
                       k + 1 < n ? h(k + 1, k) : mk(0.0, 0.0), smlnum);
        if (small && k > best) best = k;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
      if (lane == 0) s_red[warp] = best;
      __syncthreads();
      if (tid == 0) {
        int b = l;
        for (int w = 0; w < QR_THREADS / 32; ++w) b = max(b, s_red[w]);
        s_l = b;
        if (b > l) h(b, b - 1) = mk(0.0, 0.0);
      }
      // shifts left by the deflation window, read between two barriers: warp 0
      // takes them below while other warps may still be choosing their way
      const int pend0 = s_pend;
      __syncthreads();
      l = s_l;
      if (tid == 0) stamp(0);
      if (l >= i) break;  // H[i][i] isolated
      // Aggressive early deflation on the trailing block of the window
      // (skipped at the exceptional-shift iterations and while shifts from
      // the previous one are pending).
      const bool exceptional = its == 10 || its == 20;
      if (aed_min > 0 && !exceptional && pend0 == 0 && i - l + 1 >= aed_min) {
        const int jw = min(aed_w, i - l + 1), kw = i - jw + 1;
        const cplx s0 = kw > l ? h(kw, kw - 1) : mk(0.0, 0.0);
        cplx* T = D;               // [AW][ALD]
        cplx* U = D + AW * ALD;    // [AW][ALD]
        for (int idx = tid; idx < jw * jw; idx += QR_THREADS) {
          const int c = idx / jw, r = idx - c * jw;
          T[c * ALD + r] = (r <= c + 1) ? h(kw + r, kw + c) : mk(0.0, 0.0);
          U[c * ALD + r] = mk(r == c ? 1.0 : 0.0, 0.0);
        }
        __syncthreads();
        if (warp == 0) {
          int ns = -1;
          const long long c0 = clock64();
          const bool conv = small_schur_warp(T, U, jw, lane, smlnum, s_c, s_s);
          const long long c1 = clock64();
          if (conv) ns = aed_deflate_warp(T, U, s_aedv, s_aedev, jw, s0, lane, smlnum);
          if (lane == 0) {
            s_clk[5] += c1 - c0;
            s_clk[6] += clock64() - c1;
            // a deflation is logged as a dense jw x jw block; without room, skip it
            if (ns >= 0 && ns < jw &&
                (s_nsw + 1 > sweep_cap || (long long)s_nrot + (jw * jw + 1) / 2 > rot_cap))
              ns = -1;
            s_aed_ns = ns;
          }
        }
        __syncthreads();
        const int ns = s_aed_ns;
        if (ns >= 0 && ns < jw) {
          // write the block back, the spike's first entry left of it
          for (int idx = tid; idx < jw * jw; idx += QR_THREADS) {
            const int c = idx / jw, r = idx - c * jw;
            h(kw + r, kw + c) = T[c * ALD + r];
          }
          if (tid == 0 && kw > l) h(kw, kw - 1) = ns > 0 ? cmul(s0, cconj(U[0])) : mk(0.0, 0.0);
          // rows l..kw-1 of the window: H[r, kw:i] <- H[r, kw:i] U (a warp per row)
          for (int r = l + warp; r < kw; r += QR_THREADS / 32) {
            const cplx hv = lane < jw ? h(r, kw + lane) : mk(0.0, 0.0);
            cplx acc = mk(0.0, 0.0);
            for (int k = 0; k < jw; ++k) {
              const cplx x = mk(__shfl_sync(0xffffffffu, hv.x, k), __shfl_sync(0xffffffffu, hv.y, k));
              if (lane < jw) acc = cfma(x, U[lane * ALD + k], acc);
            }
            if (lane < jw) h(r, kw + lane) = acc;
          }
          // the dense log entry: U column-major (leading dimension jw)
          const int start = s_nrot;
          for (int idx = tid; idx < jw * jw; idx += QR_THREADS) {
            const int c = idx / jw, r = idx - c * jw;
            rot[2 * (size_t)start + idx] = U[c * ALD + r];
          }
          __syncthreads();
          if (tid == 0) {
            sweeps[s_nsw] = QrSweep{l, i, -1, jw, start, kw, 0, 0};
            s_nsw += 1;
            s_nrot += (jw * jw + 1) / 2;
            s_naed += 1;
          }
        }
        if (ns >= 0) {
          // shifts: up to NBMAX undeflated eigenvalues of the block, the
          // smallest in magnitude (LAPACK xLAQR0's choice); ranks by a warp
          const int ie = i - (jw - ns);
          const int want = min(NBMAX, max(1, (ie - l + 1 - 4) / 6));
          if (warp == 0 && ns >= 1) {
            const int nsh = min(want, ns);
            if (lane < ns) {
              const double me = cabs1(s_aedev[lane]);
              int rank = 0;
              for (int q = 0; q < ns; ++q) {
                const double o = cabs1(s_aedev[q]);
                rank += (o < me || (o == me && q < lane)) ? 1 : 0;
              }
              if (rank < nsh) s_shift[rank] = s_aedev[lane];
            }
            if (lane == 0) s_pend = nsh;
          }
          __syncthreads();
          // many deflations: skip the sweep and look again (LAPACK's 14%)
          if (ns < jw && 100 * (jw - ns) > 14 * jw) {
            if (tid == 0) s_pend = 0;
            __syncthreads();
          }
          // a deflation: isolate the deflated eigenvalues first (the shifts wait)
          if (ns < jw) {
            if (tid == 0) stamp(1);
            continue;
          }
        }
      }
      // Number of bulges and their shifts.
      if (warp == 0) {
        const int w = i - l + 1;
        const int pend = exceptional ? 0 : s_pend;  // shifts left by the deflation window
        const int nb0 = exceptional ? 1 : min(NBMAX, max(1, (w - 4) / 6));
        const int nb = pend > 0 ? min(nb0, pend) : nb0;
        if (pend > 0) {
        } else if (nb == 1) {
          if (lane == 0) s_shift[0] = single_shift(H, n, l, i, its);
        } else {
          const int b0 = i - nb + 1;
          for (int idx = lane; idx < nb * nb; idx += 32) {
            const int c = idx / nb, r = idx - c * nb;
            s_small[c * ALD + r] = (r <= c + 1) ? h(b0 + r, b0 + c) : mk(0.0, 0.0);
          }
          __syncwarp();
          // (on failure to converge the diagonal entries reached are used)
          small_schur_warp(s_small, nullptr, nb, lane, smlnum, s_c, s_s);
          __syncwarp();
          if (lane < nb) s_shift[lane] = s_small[lane * ALD + lane];
        }
        __syncwarp();  // every lane has read s_pend
        if (lane == 0) {
          s_nb = nb;
          s_pend = 0;
          stamp(1);
        }
      }
      __syncthreads();
      const int nb = s_nb, m = l;
      const int R = (i - m) + 3 * (nb - 1);  // rounds of this sweep
      if (tid == 0) {
        if (s_nsw + 1 > sweep_cap || (long long)s_nrot + (long long)R * nb > rot_cap) {
          s_over = 1;
        } else {
          sweeps[s_nsw] = QrSweep{m, i, nb, R, s_nrot, 0, 0, 0};
          s_cur = s_nrot;
          s_nsw += 1;
          s_nrot += R * nb;
          s_nround += R;
        }
      }
      const int a = warp;                      // this warp's bulge
      const bool mine = a < nb;
      for (int r0 = 0; r0 < R; r0 += QB) {
        const int r1 = min(r0 + QB, R);
        const int kmin = max(m, m + r0 - 3 * (nb - 1));
        const int kmax = min(i - 1, m + r1 - 1);
        const int ds = (kmin > m) ? kmin - 1 : m;
        const int de = min(kmax + 2, i);
        const int dn = de - ds + 1;
        for (int c = warp; c < dn; c += QR_THREADS / 32) {
          const cplx* hc = &h(ds, ds + c);
          for (int r = lane; r < dn; r += 32) cpa16<TEAM>(D + c * QLD + r, hc + r);
        }
        cpa_commit();
        cpa_wait<0>();
        __syncthreads();
        if (s_over) break;
        // A round in three steps, each ended by a CTA barrier: lane b of warp
        // 0 forms bulge b's rotation (while every warp fetches the rows it
        // will transform); each warp transforms its bulge's rows k, k+1 over
        // columns k..de; each warp transforms columns k, k+1 over rows
        // ds..min(k+2, i).  Both spans are at most QD, two entries per lane.
        const int kr0 = m + r0 - 3 * a;
        cplx* prow = D + (ptrdiff_t)(kr0 - ds) * (QLD + 1) + (ptrdiff_t)lane * QLD;
        cplx* pcol = D + (ptrdiff_t)(kr0 - ds) * QLD + lane;
        for (int r = r0; r < r1; ++r, prow += QLD + 1, pcol += QLD) {
          const int k = m + r - 3 * a, u = r - r0;
          const bool act = mine && k >= m && k <= i - 1;
          const bool row0 = act && lane <= de - k, row1 = act && lane + 32 <= de - k;
          cplx x0, y0, x1, y1;
          if (row0) {
            x0 = prow[0];
            y0 = prow[1];
          }
          if (row1) {
            x1 = prow[32 * QLD];
            y1 = prow[32 * QLD + 1];
          }
          if (tid < nb) {
            const int kb = m + r - 3 * tid;
            double c = 1.0;  // outside the window: the identity
            cplx sn = mk(0.0, 0.0);
            if (kb >= m && kb <= i - 1) {
              cplx* pb = D + (ptrdiff_t)(kb - ds) * (QLD + 1);  // (kb, kb)
              const bool first = kb == m;
              const cplx x = first ? csub(pb[0], s_shift[tid]) : pb[-QLD];
              const cplx y = first ? pb[1] : pb[1 - QLD];
              const Rot g = givens(x, y);
              if (!first) {
                pb[-QLD] = g.r;
                pb[1 - QLD] = mk(0.0, 0.0);
              }
              c = g.c;
              sn = g.s;
            }
            s_c[u * NBMAX + tid] = c;
            s_s[u * NBMAX + tid] = sn;
          }
          __syncthreads();
          const double c = s_c[u * NBMAX + a];
          const cplx sn = s_s[u * NBMAX + a];
          if (row0) {
            rotate2<true>(x0, y0, c, sn);
            prow[0] = x0;
            prow[1] = y0;
          }
          if (row1) {
            rotate2<true>(x1, y1, c, sn);
            prow[32 * QLD] = x1;
            prow[32 * QLD + 1] = y1;
          }
          __syncthreads();
          const int nc = min(k + 2, i) - ds;
          const bool col0 = act && lane <= nc, col1 = act && lane + 32 <= nc;
          if (col0) {
            x0 = pcol[0];
            y0 = pcol[QLD];
          }
          if (col1) {
            x1 = pcol[32];
            y1 = pcol[QLD + 32];
          }
          if (col0) {
            rotate2<false>(x0, y0, c, sn);
            pcol[0] = x0;
            pcol[QLD] = y0;
          }
          if (col1) {
            rotate2<false>(x1, y1, c, sn);
            pcol[32] = x1;
            pcol[QLD + 32] = y1;
          }
          __syncthreads();
        }
        if (tid == 0) stamp(2);
        // Write the window back and log this chunk's rotations (round-major).
        for (int c = warp; c < dn; c += QR_THREADS / 32) {
          cplx* hc = &h(ds, ds + c);
          for (int r = lane; r < dn; r += 32) hc[r] = D[c * QLD + r];
        }
        const int nr = r1 - r0;
        for (int idx = tid; idx < nb * nr; idx += QR_THREADS) {
          const int u = idx / nb, b = idx - u * nb;
          const size_t ri = (size_t)s_cur + (size_t)(r0 + u) * nb + b;
          rot[2 * ri] = mk(s_c[u * NBMAX + b], 0.0);  // (the identity where the bulge is outside the window)
          rot[2 * ri + 1] = s_s[u * NBMAX + b];
        }
        const Chunk ch{m, i, nb, r0, r1, kmin, kmax, ds, de};
        if (TEAM && far_groups(ch) > NBMAX) {
          if (tid == 0) s_chunk = ch;
          team_sync();  // D is free; the others read the chunk
          far_strips<TEAM>(H, n, ch, D, s_c, s_s, warp, NBMAX * team);
          team_sync();
        } else {
          __syncthreads();  // D is free
          far_strips<TEAM>(H, n, ch, D, s_c, s_s, warp, NBMAX);
          __syncthreads();
        }
        if (tid == 0) stamp(3);
      }
      if (s_over) {
        failed = 1;
        break;
      }
    }
    if (failed || its > itmax || tot > totmax) {
      failed = 1;
      break;
    }
    i = l - 1;
  }
  __syncthreads();
  for (int k = tid; k < n; k += QR_THREADS) W[k] = h(k, k);
  if (tid == 0) {
    QrLogHeader* hdr = reinterpret_cast<QrLogHeader*>(logb);
    hdr->nsweeps = s_nsw;
    hdr->nrot = s_nrot;
    hdr->nrounds = s_nround;
    hdr->naed = s_naed;
    hdr->t_defl = s_clk[0];
    hdr->t_shift = s_clk[1];
    hdr->t_rounds = s_clk[2];
    hdr->t_far = s_clk[3];
    hdr->t_wschur = s_clk[5];
    hdr->t_wdefl = s_clk[6];
    if (failed && status) status[mat] = ST_ENOCONV;
    s_chunk.m = -1;
  }
  if (TEAM) {
    team_sync();  // the others see that the matrix is done
    team_sync();  // and have read it
  }
}

// Replay kernels: every vector (column transforms: rows of Z for every sweep,
// rows of H above the sweep's window; row transforms: columns of H right of
// the window) stays in shared memory from the first sweep to the last, FV
// vectors per warp, and takes the log's rotations with eight lanes per vector
// as strip_rounds does.  The log is one stream: it comes in through a ring of
// four chunks, two ahead of the one in use, whatever sweep they belong to.
//
// Bounded by issue when several warps share a scheduler (600 matrices at n = 61:
// 75% of the slots, FP64 27%), by the latency of a round (some 50 cycles) when the
// batch is small or n leaves two blocks to an SM (n = 450: 32%).  One thread
// per vector with four bulges in a register ring, its entries streamed from
// global memory once per four bulges and sweep, took 525 cycles per round and
// four bulges, and two memory latencies at the start of every sweep.
constexpr int RG_CHUNK = 128, RG_CHUNKS = 4;            // rotations per chunk, chunks of the ring
constexpr int RG_SLOTS = RG_CHUNK * RG_CHUNKS;          // a power of two
constexpr int RG_DENSE = 16;  // deflation-window blocks up to this order are read from the ring (two chunks at most)
constexpr int RP_MAXW = 4;    // warps per block, at most

// Warps per block: the vectors of a warp take 64 n bytes.  Four warps let two
// blocks share an SM up to n = 376; three keep two blocks there up to n = 500
// and still fit one at n = 1024.
int replay_warps(int n) { return n <= 376 ? RP_MAXW : 3; }
size_t replay_smem(int n) {
  return (size_t)RG_SLOTS * 2 * sizeof(cplx) + (size_t)replay_warps(n) * FV * n * sizeof(cplx);
}

struct LogRing {
  const cplx* rot;  // the log's rotations (two complex numbers each)
  cplx* ring;
  int nrot, cur;  // rotations in the log, the chunk in use

  __device__ __forceinline__ void load(int chunk) {
    for (int e = threadIdx.x; e < RG_CHUNK * 2; e += blockDim.x)
      if (chunk * RG_CHUNK + e / 2 < nrot)
        cpa16(ring + (chunk % RG_CHUNKS) * RG_CHUNK * 2 + e, rot + (size_t)chunk * RG_CHUNK * 2 + e);
    cpa_commit();
  }
  __device__ __forceinline__ void begin() {
    cur = -1;
    load(0);
    load(1);
  }
  // every rotation up to `slot` is in the ring (and at least a chunk before
  // it).  All threads of the block call it alike.
  __device__ __forceinline__ void ensure(int slot) {
    while (cur < slot / RG_CHUNK) {
      ++cur;
      cpa_wait<1>();    // chunk cur has landed
      __syncthreads();  // for every thread; chunk cur - 2 is done with
      load(cur + 2);
    }
  }
};

template <bool ROWOP>
__device__ __forceinline__ void replay(cplx* X, size_t es, size_t vs, int sel, int v0, int n, char* logb,
                                       int sweep_cap, cplx* smem) {
  // vectors v0 + 4 warp .. of X (entry e of vector v at e es + v vs); sel: 0 =
  // every sweep, 1 = sweeps with v < m (rows of H above the window), 2 =
  // sweeps with v > i (columns of H right of the window)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = lane / FV, vl = lane % FV, v = v0 + warp * FV + vl;
  const QrLogHeader hdr = *reinterpret_cast<const QrLogHeader*>(logb);
  const QrSweep* sw = log_sweeps(logb);
  LogRing lr{log_rot(logb, sweep_cap), smem, hdr.nrot, -1};
  cplx* vec = smem + RG_SLOTS * 2 + (size_t)warp * FV * n + vl;
  lr.begin();
  if (v < n)
    for (int e = b; e < n; e += 32 / FV) vec[e * FV] = X[(size_t)e * es + (size_t)v * vs];
  __syncwarp();
  QrSweep next;
  if (hdr.nsweeps > 0) next = sw[0];
  for (int s = 0; s < hdr.nsweeps; ++s) {
    const QrSweep q = next;
    if (s + 1 < hdr.nsweeps) next = sw[s + 1];
    const bool mine = v < n && (sel == 0 || (sel == 1 ? v < q.m : v > q.i));
    const bool any = __any_sync(0xffffffffu, mine);
    if (q.nb < 0) {  // deflation-window block: x <- U^H x (row transforms) or x U
      const int jw = q.R;
      const bool ringed = jw <= RG_DENSE;
      if (ringed) lr.ensure(q.start + (jw * jw - 1) / 2);
      if (any) {
        cplx out[AW / 8];
#pragma unroll
        for (int t = 0; t < AW / 8; ++t) {
          const int j = b + 8 * t;
          cplx acc = mk(0.0, 0.0);
          if (j < jw)
            for (int k = 0; k < jw; ++k) {
              const int e = 2 * q.start + j * jw + k;
              const cplx u = ringed ? lr.ring[e & (2 * RG_SLOTS - 1)] : ld(lr.rot + e);
              const cplx x = vec[(q.pad0 + k) * FV];
              acc = ROWOP ? cadd(acc, cmulc(u, x)) : cfma(x, u, acc);
            }
          out[t] = acc;
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < AW / 8; ++t)
          if (mine && b + 8 * t < jw) vec[(q.pad0 + b + 8 * t) * FV] = out[t];
        __syncwarp();
      }
      continue;
    }
    const int nb = q.nb;
    const int ra0 = 3 * b, ra1 = (mine && b < nb) ? 3 * b + (q.i - q.m) : 0;
    cplx* p = vec + (size_t)q.m * FV;
    cplx x = mk(0.0, 0.0), y = x;
    for (int t0 = 0; t0 < q.R;) {
      lr.ensure(q.start + (t0 + 1) * nb - 1);
      const int t1 = min(q.R, ((lr.cur + 1) * RG_CHUNK - q.start) / nb);  // rounds whose rotations are in the ring
      if (any) {
        int slot = q.start + t0 * nb + b;
        auto rc = [&](int i) { return lr.ring[2 * (i & (RG_SLOTS - 1))].x; };
        auto rs = [&](int i) { return lr.ring[2 * (i & (RG_SLOTS - 1)) + 1]; };
        double c = rc(slot);
        cplx sn = rs(slot);
        for (int r = t0; r < t1; ++r) {
          slot += nb;
          const double cn = rc(slot);  // the next round's (stale past t1, then read again)
          const cplx sn2 = rs(slot);
          if (r >= ra0 && r < ra1) {
            if (r == ra0) {
              x = p[0];
              y = p[FV];
            }
            const bool more = r + 1 < ra1;
            cplx nx = mk(0.0, 0.0);
            if (more) nx = p[2 * FV];
            rotate2<ROWOP>(x, y, c, sn);
            p[0] = x;
            if (!more) p[FV] = y;
            x = y;
            y = nx;
            p += FV;
          }
          c = cn;
          sn = sn2;
          __syncwarp();
        }
      }
      t0 = t1;
    }
  }
  cpa_wait<0>();
  if (v < n)
    for (int e = b; e < n; e += 32 / FV) X[(size_t)e * es + (size_t)v * vs] = vec[e * FV];
}

__global__ void __launch_bounds__(RP_MAXW * 32)
    qr_replay_rows_kernel(cplx* const* __restrict__ Hs, cplx* const* __restrict__ Zs,
                          void* const* __restrict__ logs, int n, int sweep_cap, int row_blocks) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int mat = blockIdx.y;
  const bool isZ = blockIdx.x >= row_blocks;
  const int per = blockDim.x / 32 * FV;
  replay<false>(isZ ? Zs[mat] : Hs[mat], (size_t)n, 1, isZ ? 0 : 1,
                (isZ ? blockIdx.x - row_blocks : blockIdx.x) * per, n, static_cast<char*>(logs[mat]), sweep_cap,
                reinterpret_cast<cplx*>(smem_raw));
}

// Runs after qr_replay_rows_kernel: for any entry all column transforms
// precede all row transforms.
__global__ void __launch_bounds__(RP_MAXW * 32)
    qr_replay_cols_kernel(cplx* const* __restrict__ Hs, void* const* __restrict__ logs, int n, int sweep_cap) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int mat = blockIdx.y;
  replay<true>(Hs[mat], 1, (size_t)n, 2, blockIdx.x * (blockDim.x / 32 * FV), n, static_cast<char*>(logs[mat]),
               sweep_cap, reinterpret_cast<cplx*>(smem_raw));
}

}  // namespace

// CTAs per matrix of the iteration: clusters of 8 on half of the SMs, of 4 on four
// fifths, of 2 on half (with 66 matrices at n = 162 on all of them, beside another
// stream's work, 13.4 ms for 10.4 alone).
// ms for 1 / 2 / 4 / 8: n = 450, 4 matrices 72.7 / 61.3 / 56.5 / 52.4, 16 matrices
// 72.1 / 61.2 / 54.3 / 59.9; n = 242, 18 matrices 22.8 / 19.9 / 19.1 / 20.9; n = 162,
// 4 matrices 10.9 / 10.8 / 10.6 / 10.6; 37 matrices 10.8 / 10.7 / 11.3 / 20.3 (the
// clusters no longer fit side by side); below, the strips are too few: n = 120, 3
// matrices 5.98 / 6.10 / 6.07 / 6.12.
static int team_size(int n, int batch) {
  static const int sms = [] {
    int dev = 0, v = 0;
    VRC_CUDA_CHECK(cudaGetDevice(&dev));
    VRC_CUDA_CHECK(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
    return v;
  }();
  if (n < 160) return 1;
  return 2LL * batch * 8 <= sms ? 8 : 5LL * batch * 4 <= 4LL * sms ? 4 : 4LL * batch <= sms ? 2 : 1;
}

void schur_batched(cplx* const* d_H, cplx* const* d_Z, cplx* const* d_W, void* const* d_logs, int batch, int n,
                   int* d_status, cudaStream_t st, int parts) {
  if (batch <= 0) return;
  // Order of the deflation window (VRC_QR_AEDW, 4..32) and the order of the
  // active window from which it is taken (VRC_QR_AED; 0: never).  By default 10
  // and 48 for n > 128, never below: ms of iteration and replay for windows of
  // 0 / 8 / 10 / 12 / 16, n = 98 (11 matrices) 4.5 / 4.3 / 4.5 / 5.0 / 5.6, n = 162
  // (5) 10.1 / 9.5 / 9.3 / 10.2 / 11.3, n = 162 (74) 14.7 / 13.0 / 12.7 / 13.4 /
  // 14.5, n = 242 (8) 20.7 / 18.7 / 18.2 / 19.2 / 21.2, n = 450 (5) 71.2 / 64.2 /
  // 56.5 / 58.2 / 61.0: a window's cost (one warp) against the sweeps it saves.
  static const int aed_w_env = [] {
    const char* e = std::getenv("VRC_QR_AEDW");
    return e ? std::min(AW, std::max(4, std::atoi(e))) : 0;
  }();
  const int aed_w = aed_w_env ? aed_w_env : 10;
  static const int aed_env = [] {
    const char* e = std::getenv("VRC_QR_AED");
    return e ? std::max(0, std::atoi(e)) : -1;
  }();
  const int aed_min = aed_env >= 0 ? aed_env : (n <= 128 ? 0 : 48);
  ensure_smem((const void*)hqr_kernel<false>, QR_SMEM);
  const size_t rp_smem = replay_smem(n);
  const int rp_threads = 32 * replay_warps(n);
  ensure_smem((const void*)qr_replay_rows_kernel, rp_smem);
  ensure_smem((const void*)qr_replay_cols_kernel, rp_smem);
  const int cc = schur_sweep_cap(n);
  const long long rc = schur_rot_cap(n);
  const int row_blocks = (n + rp_threads / 32 * FV - 1) / (rp_threads / 32 * FV);
  for (int b0 = 0; b0 < batch; b0 += 65535) {
    const int nb = min(65535, batch - b0);
    if (parts & SCHUR_ITERATE) {
      int* stat = d_status ? d_status + b0 : nullptr;
      const int team = team_size(n, nb);
      if (team > 1) {
        ensure_smem((const void*)hqr_kernel<true>, QR_SMEM);
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)team;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(nb * team));
        cfg.blockDim = dim3(QR_THREADS);
        cfg.dynamicSmemBytes = QR_SMEM;
        cfg.stream = st;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        VRC_CUDA_CHECK(cudaLaunchKernelEx(&cfg, hqr_kernel<true>, d_H + b0, d_logs + b0, d_W + b0, n, cc, rc, stat,
                                          aed_min, aed_w));
      } else {
        hqr_kernel<false><<<nb, QR_THREADS, QR_SMEM, st>>>(d_H + b0, d_logs + b0, d_W + b0, n, cc, rc, stat, aed_min,
                                                           aed_w);
      }
    }
    if (parts & SCHUR_REPLAY) {
      qr_replay_rows_kernel<<<dim3(2 * row_blocks, nb), rp_threads, rp_smem, st>>>(d_H + b0, d_Z + b0, d_logs + b0,
                                                                                  n, cc, row_blocks);
      qr_replay_cols_kernel<<<dim3(row_blocks, nb), rp_threads, rp_smem, st>>>(d_H + b0, d_logs + b0, n, cc);
    }
  }
  VRC_CUDA_CHECK(cudaGetLastError());
}

}  // namespace vrc

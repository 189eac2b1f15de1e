// Particle-mesh Ewald reciprocal term and exclusion corrections.
//
// Reference: mdl/interface/force/nonbonded/Grid.h (anterpolateCharge :107-154, interpolateForce
// :158-189, scalarSum :236-341, initialize :498-586, dftmod :588-600), BSpline.cpp:55-105,
// NonbondedPMEwaldSystemForce.h (reciprocalTerm :812-864, correctionTerm :874-911).
//
// Pipeline per step (every kernel batched over the boxes of a system):
//   k_spread      B-spline weights, order^3 int64 fixed-point atomics per atom slot (two to eight
//                 threads per slot, one z-offset of the stencil each)
//   k_fft_z_fwd   z-lines of the fixed-point grid (cleared as it is read), two real lines packed
//                 per complex FFT, half spectrum written as [kz][x][y]
//   k_fft_plane   per kz plane, in shared memory: y- and x-lines forward, influence function
//                 multiply with energy and virial partials added to the box accumulators, x- and
//                 y-lines inverse (planes too large for that: k_fft_y, k_fft_x_infl, k_fft_y)
//   k_fft_z_inv   inverse z transform back to the real potential grid [x][y][z]
//   k_gather      the same threads per atom slot, fixed-point force atomics
// The transforms are unnormalised, as the reference's ZFFT/FFTW calls; r2c/c2r replace the
// reference's full complex transform of a real grid (identical result: the spectrum is Hermitian
// and the influence function even in m).
#include <functional>
#include <type_traits>

#include "pmb_internal.h"

namespace pmb {

namespace {

template <typename T>
struct C2;
template <>
struct C2<float> {
  using t = float2;
};
template <>
struct C2<double> {
  using t = double2;
};

__device__ __forceinline__ float2 cmk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 cmk(double a, double b) { return make_double2(a, b); }

template <typename T2>
__device__ __forceinline__ T2 cmul(T2 a, T2 b) {
  return cmk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename T2>
__device__ __forceinline__ T2 cadd(T2 a, T2 b) { return cmk(a.x + b.x, a.y + b.y); }
template <typename T2>
__device__ __forceinline__ T2 csub(T2 a, T2 b) { return cmk(a.x - b.x, a.y - b.y); }
// multiply by (i * sign)
template <typename T2>
__device__ __forceinline__ T2 cis(T2 a, int sign) { return sign > 0 ? cmk(-a.y, a.x) : cmk(a.y, -a.x); }
template <typename T2, typename S>
__device__ __forceinline__ T2 cscale(T2 a, S s) { return cmk(a.x * s, a.y * s); }

// Small DFTs X_k = sum_n x_n exp(sign 2 pi i n k / R).
template <int R, typename T2>
__device__ __forceinline__ void dft_small(T2 *v, int sign) {
  using S = decltype(v[0].x);
  if constexpr (R == 2) {
    T2 a = cadd(v[0], v[1]), b = csub(v[0], v[1]);
    v[0] = a; v[1] = b;
  } else if constexpr (R == 3) {
    const S h = S(0.86602540378443864676);
    T2 t1 = cadd(v[1], v[2]);
    T2 t2 = csub(v[0], cscale(t1, S(0.5)));
    T2 t3 = cis(cscale(csub(v[1], v[2]), h), sign);
    v[0] = cadd(v[0], t1);
    v[1] = cadd(t2, t3);
    v[2] = csub(t2, t3);
  } else if constexpr (R == 4) {
    T2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]);
    T2 d = cis(csub(v[1], v[3]), sign);
    v[0] = cadd(a, c); v[1] = cadd(b, d); v[2] = csub(a, c); v[3] = csub(b, d);
  } else if constexpr (R == 5) {
    const S c1 = S(0.30901699437494742410), c2 = S(-0.80901699437494742410),
            s1 = S(0.95105651629515357212), s2 = S(0.58778525229247312917);
    T2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]), t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
    T2 a1 = cadd(v[0], cadd(cscale(t1, c1), cscale(t2, c2)));
    T2 a2 = cadd(v[0], cadd(cscale(t1, c2), cscale(t2, c1)));
    T2 b1 = cis(cadd(cscale(t3, s1), cscale(t4, s2)), sign);
    T2 b2 = cis(csub(cscale(t3, s2), cscale(t4, s1)), sign);
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd(a1, b1); v[4] = csub(a1, b1);
    v[2] = cadd(a2, b2); v[3] = csub(a2, b2);
  }
}

// floor(a / d) for 0 <= a < 2^21 from r ~ 1/d (a few ulp suffice: (a + 1/2) / d stays at least
// 1/(2d) away from an integer), without an integer division.
__device__ __forceinline__ int divf(int a, float r) { return __float2int_rz(((float)a + 0.5f) * r); }
__device__ __forceinline__ float rcpf(int d) { return __fdividef(1.0f, (float)d); }

// One Stockham stage, out of place (src -> dst): each thread takes whole butterflies (R inputs
// read, twiddled, transformed and written), so only R values are live at a time.
template <int R, typename T2>
__device__ __forceinline__ void fft_stage(const T2 *__restrict__ src, T2 *__restrict__ dst, int n,
                                          int nlines, int lstride, int estride, int Ns,
                                          const T2 *tw, int sign) {
  const int nb = n / R, total = nb * nlines, step = n / (Ns * R);
  const float rnb = rcpf(nb), rnl = rcpf(nlines), rns = rcpf(Ns);
  for (int b = threadIdx.x; b < total; b += blockDim.x) {
    // contiguous lines: consecutive threads take consecutive butterflies of one line;
    // strided lines: consecutive threads take the same butterfly of consecutive lines
    int line, j;
    if (estride == 1) {
      line = divf(b, rnb);
      j = b - line * nb;
    } else {
      j = divf(b, rnl);
      line = b - j * nlines;
    }
    const T2 *Ls = src + line * lstride;
    T2 *Ld = dst + line * lstride;
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = Ls[(j + r * nb) * estride];
    const int jq = divf(j, rns), k = j - jq * Ns;
#pragma unroll
    for (int r = 1; r < R; r++) {
      T2 w = tw[r * k * step];
      if (sign > 0) w.y = -w.y;
      v[r] = cmul(v[r], w);
    }
    dft_small<R>(v, sign);
    const int out = jq * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; r++) Ld[(out + r * Ns) * estride] = v[r];
  }
  __syncthreads();
}

// Batched 1-D FFTs of length n over shared memory (element e of line l at
// buf[l*lstride + e*estride]); radices[0..nrad) multiply to n.  Stages alternate between buf
// and tmp (same layout); returns the buffer holding the result.
template <typename T2>
__device__ T2 *fft_lines(T2 *buf, T2 *tmp, int n, int nlines, int lstride, int estride,
                         const int *radices, int nrad, const T2 *tw, int sign) {
  int Ns = 1;
  T2 *src = buf, *dst = tmp;
  for (int s = 0; s < nrad; s++) {
    const int R = radices[s];
    if (R == 4) fft_stage<4>(src, dst, n, nlines, lstride, estride, Ns, tw, sign);
    else if (R == 2) fft_stage<2>(src, dst, n, nlines, lstride, estride, Ns, tw, sign);
    else if (R == 3) fft_stage<3>(src, dst, n, nlines, lstride, estride, Ns, tw, sign);
    else fft_stage<5>(src, dst, n, nlines, lstride, estride, Ns, tw, sign);
    Ns *= R;
    T2 *t = src;
    src = dst;
    dst = t;
  }
  return src;
}

// B-spline weights of order P at w (BSpline::set, BSpline.cpp:55-105).
template <typename T>
__device__ __forceinline__ void bspline(int P, T w, T *th, T *dth) {
  if (P == 2) {
    th[1] = w; th[0] = T(1) - w;
    if (dth) { dth[1] = T(1); dth[0] = T(-1); }
    return;
  }
  th[P - 1] = T(0);
  th[1] = w;
  th[0] = T(1) - w;
  #pragma unroll
  for (int k = 2; k < P - 1; k++) {
    T div = T(1) / T(k);
    th[k] = div * w * th[k - 1];
    #pragma unroll
    for (int j = 1; j < k; j++)
      th[k - j] = div * ((w + T(j)) * th[k - j - 1] + (T(k + 1 - j) - w) * th[k - j]);
    th[0] = div * (T(1) - w) * th[0];
  }
  if (dth) {
    dth[0] = -th[0];
    #pragma unroll
    for (int j = 1; j <= P - 1; j++) dth[j] = th[j - 1] - th[j];
  }
  T div = T(1) / (T(P) - T(1));
  th[P - 1] = div * w * th[P - 2];
  #pragma unroll
  for (int j = 1; j < P - 1; j++)
    th[P - 1 - j] = div * ((w + T(j)) * th[P - j - 2] + (T(P - j) - w) * th[P - 1 - j]);
  th[0] = div * (T(1) - w) * th[0];
}

// Grid coordinate of one dimension: base index (already offset by -(P-1)/2 and wrapped to
// [0, n)) and the fractional weight w.
template <bool MIXED>
__device__ __forceinline__ void grid_coord(unsigned fx, double x, double hr, int n, int P, int &base,
                                           typename std::conditional<MIXED, float, double>::type &w) {
  int iu;
  if constexpr (MIXED) {
    unsigned long long prod = (unsigned long long)fx * (unsigned)n;
    iu = (int)(prod >> 32);
    w = (float)(unsigned)(prod & 0xffffffffull) * 2.3283064365386963e-10f;
  } else {
    // Grid.h:110-121: u = x n / L wrapped into [0, n) by repeated +-n, then truncated.
    double u = x * hr;
    for (int it = 0; it < 4 && u < 0.0; it++) u += n;
    for (int it = 0; it < 4 && u >= n; it++) u -= n;
    if (!(u >= 0.0 && u < n)) {
      u -= n * floor(u / n);
      if (!(u >= 0.0 && u < n)) u = 0.0;
    }
    iu = (int)u;
    w = u - iu;
  }
  base = iu - (P - 1) / 2 + n;  // myNXOffset = -(order-1)/2 + n
}

// x mod n for 0 <= x < 3n (a stencil index: base in [n - (p-1)/2, 2n) plus an offset below p,
// with n >= p), without an integer division.
__device__ __forceinline__ int wrap3(int x, int n) {
  x = x >= n ? x - n : x;
  return x >= n ? x - n : x;
}

// B-spline weights and grid bases of one slot for order P (2, 4, 6 or 8).
template <bool MIXED, int P, bool DERIV>
__device__ __forceinline__ void slot_weights(const PmeBoxPlan &pl, uint4 f, double4 pq,
                                             typename std::conditional<MIXED, float, double>::type th[3][P],
                                             typename std::conditional<MIXED, float, double>::type dth[3][P],
                                             int base[3], typename std::conditional<MIXED, float, double>::type &q) {
  using T = typename std::conditional<MIXED, float, double>::type;
  if constexpr (MIXED) {
    const unsigned fx[3] = {f.x, f.y, f.z};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      T w;
      grid_coord<true>(fx[d], 0.0, 0.0, pl.n[d], P, base[d], w);
      bspline<T>(P, w, th[d], DERIV ? dth[d] : nullptr);
    }
    q = __uint_as_float(f.w);
  } else {
    const double x[3] = {pq.x, pq.y, pq.z};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      T w;
      grid_coord<false>(0u, x[d], pl.hr[d], pl.n[d], P, base[d], w);
      bspline<T>(P, w, th[d], DERIV ? dth[d] : nullptr);
    }
    q = pq.w;
  }
}

// v[p] for a run-time p in [0, P) without indexing a register array (which would go to local
// memory).
template <int P, typename T>
__device__ __forceinline__ T pick(const T v[P], int p) {
  T o = v[0];
#pragma unroll
  for (int k = 1; k < P; k++) o = p == k ? v[k] : o;
  return o;
}

// Threads of one atom slot: the order rounded up to a power of two.
template <int P>
constexpr int SLOT_THREADS = P <= 2 ? 2 : P <= 4 ? 4 : 8;

// SLOT_THREADS threads per atom slot: thread p adds the P^2 points of z-offset p of the stencil,
// so that at every step the slot's threads add to P consecutive grid words (one to three 32-byte
// sectors).  Bound by the L2's atomics.  Orders above 4 ran one thread per slot, with the order
// known at run time and the weights in local memory (19,200 atoms, order 6, FP64: 40 us, now 12; the
// gather 43 us, now 17).
template <bool MIXED, int P>
__global__ void k_spread(NbListDev nb, PmeDev pm) {
  using T = typename std::conditional<MIXED, float, double>::type;
  constexpr int W = SLOT_THREADS<P>;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int sl = (int)(t / W), p = (int)(t % W);
  if (sl >= nb.nslot || p >= P) return;
  // the slot's metadata and position are loaded together (one round trip)
  const int4 m = nb.slot_meta[sl];
  uint4 f4 = make_uint4(0, 0, 0, 0);
  double4 p4 = make_double4(0, 0, 0, 0);
  if constexpr (MIXED) f4 = nb.slot_fx[sl];
  else p4 = nb.slot_pq[sl];
  if (m.x < 0) return;
  const PmeBoxPlan &pl = pm.plan[m.w];
  T th[3][P];
  int base[3];
  T q;
  slot_weights<MIXED, P, false>(pl, f4, p4, th, th, base, q);
  const int nx = pl.n[0], ny = pl.n[1], nz = pl.n[2];
  long long *g = pm.qgrid + pl.grid0;
  const T c2 = pick<P>(th[2], p);
  long long *col = g + wrap3(p + base[2], nz);
#pragma unroll
  for (int i = 0; i < P; i++) {
    const T a = q * th[0][i];
    const int i1 = wrap3(i + base[0], nx);
#pragma unroll
    for (int j = 0; j < P; j++) {
      const int j1 = wrap3(j + base[1], ny);
      const long long v = f2fix(a * th[1][j] * c2, (T)GRID_SCALE);
      if (v) red_add(col + ((long long)i1 * ny + j1) * nz, v);
    }
  }
}

// The same threads read the stencil: thread p z-offset p, so that at every step the slot's threads
// read P consecutive grid words; the partial forces are summed over the slot's lanes.  Every lane
// takes part in the shuffles (slots out of range or padding, and lanes past the order, add zeros).
template <bool MIXED, int P>
__global__ void k_gather(const SystemDev s, NbListDev nb, PmeDev pm) {
  using T = typename std::conditional<MIXED, float, double>::type;
  constexpr int W = SLOT_THREADS<P>;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int sl = (int)(t / W), p = (int)(t % W);
  const bool in = sl < nb.nslot;
  const int4 m = in ? nb.slot_meta[sl] : make_int4(-1, -1, 0, 0);
  uint4 f4 = make_uint4(0, 0, 0, 0);
  double4 pq = make_double4(0, 0, 0, 0);
  if (in) {
    if constexpr (MIXED) f4 = nb.slot_fx[sl];
    else pq = nb.slot_pq[sl];
  }
  const bool ok = m.x >= 0;
  T fx = 0, fy = 0, fz = 0, q = 0;
  const PmeBoxPlan *pl = ok ? pm.plan + m.w : nullptr;
  if (ok && p < P) {
    T th[3][P], dth[3][P];
    int base[3];
    slot_weights<MIXED, P, true>(*pl, f4, pq, th, dth, base, q);
    const int nx = pl->n[0], ny = pl->n[1], nz = pl->n[2];
    const T *col = reinterpret_cast<const T *>(pm.rgrid) + pl->grid0 + wrap3(p + base[2], nz);
    const T tz = pick<P>(th[2], p), dz = pick<P>(dth[2], p);
#pragma unroll
    for (int i = 0; i < P; i++) {
      const int i1 = wrap3(i + base[0], nx);
#pragma unroll
      for (int j = 0; j < P; j++) {
        const int j1 = wrap3(j + base[1], ny);
        const T xij = dth[0][i] * th[1][j], yij = th[0][i] * dth[1][j], zij = th[0][i] * th[1][j];
        const T term = col[((long long)i1 * ny + j1) * nz];
        fx -= term * xij * tz;
        fy -= term * yij * tz;
        fz -= term * zij * dz;
      }
    }
  }
#pragma unroll
  for (int o = 1; o < W; o <<= 1) {
    fx += __shfl_xor_sync(0xffffffffu, fx, o);
    fy += __shfl_xor_sync(0xffffffffu, fy, o);
    fz += __shfl_xor_sync(0xffffffffu, fz, o);
  }
  if (ok && p == 0) {
    long long *f = s.facc + 3 * (long long)m.x;
    red_add(f, f2fix((double)(fx * T(pl->hr[0]) * q), FORCE_SCALE));
    red_add(f + 1, f2fix((double)(fy * T(pl->hr[1]) * q), FORCE_SCALE));
    red_add(f + 2, f2fix((double)(fz * T(pl->hr[2]) * q), FORCE_SCALE));
  }
}

template <int THREADS, typename T>
__device__ __forceinline__ double block_sum(double v, double *red) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x < 32) {
    r = threadIdx.x < THREADS / 32 ? red[threadIdx.x] : 0.0;
    r = warp_sum(r);
  }
  return r;
}

constexpr int LT = 128;          // threads of the y- and x-line kernels
constexpr int LMAXE = 2048;      // complex elements per line-kernel CTA, per ping-pong buffer

// y-lines of the half spectrum: rows C[kz][x][0..ny) of one work item are contiguous.
template <typename T>
__global__ void __launch_bounds__(LT, 8) k_fft_y(PmeDev pm, int sign) {
  using T2 = typename C2<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int4 wk = pm.ywork[blockIdx.x];  // box, kz, x0, rows
  const PmeBoxPlan &pl = pm.plan[wk.x];
  const int nx = pl.n[0], ny = pl.n[1], kz = wk.y, x0 = wk.z, rows = wk.w;
  T2 *tw = reinterpret_cast<T2 *>(smem_raw + 32 * sizeof(double));
  T2 *buf = tw + 256, *tmp = buf + pm.lbuf;
  for (int k = threadIdx.x; k < ny; k += LT) {
    if constexpr (sizeof(T) == 4) tw[k] = pm.twiddlef[pl.tw0[1] + k];
    else tw[k] = pm.twiddle[pl.tw0[1] + k];
  }
  T2 *C = reinterpret_cast<T2 *>(pm.cgrid) + pl.cgrid0 + ((long long)kz * nx + x0) * ny;
  const int ne = rows * ny;
  for (int e = threadIdx.x; e < ne; e += LT) buf[e] = C[e];
  __syncthreads();
  const T2 *res = fft_lines(buf, tmp, ny, rows, ny, 1, pm.radix + pl.rad0[1], pl.nrad[1], tw, sign);
  for (int e = threadIdx.x; e < ne; e += LT) C[e] = res[e];
}

// x-lines (columns y0..y0+cols of one kz plane): forward FFT, influence function with energy and
// virial (Grid.h:236-341, half spectrum kz <= nz/2 with the doubling of interior kz), inverse FFT.
template <typename T>
__global__ void __launch_bounds__(LT, 8) k_fft_x_infl(const SystemDev s, PmeDev pm) {
  using T2 = typename C2<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int4 wk = pm.xwork[blockIdx.x];  // box, kz, y0, cols
  const PmeBoxPlan &pl = pm.plan[wk.x];
  const int nx = pl.n[0], ny = pl.n[1], nz = pl.n[2], kz = wk.y, y0 = wk.z, cols = wk.w;
  double *red = reinterpret_cast<double *>(smem_raw);  // 32 doubles
  T2 *tw = reinterpret_cast<T2 *>(smem_raw + 32 * sizeof(double));
  T2 *buf = tw + 256, *tmp = buf + pm.lbuf;  // buf[x * cols + c]
  for (int k = threadIdx.x; k < nx; k += LT) {
    if constexpr (sizeof(T) == 4) tw[k] = pm.twiddlef[pl.tw0[0] + k];
    else tw[k] = pm.twiddle[pl.tw0[0] + k];
  }
  T2 *C = reinterpret_cast<T2 *>(pm.cgrid) + pl.cgrid0 + (long long)kz * nx * ny + y0;
  const int ne = nx * cols;
  const float rcols = rcpf(cols);
  for (int e = threadIdx.x; e < ne; e += LT) {
    const int x = divf(e, rcols), c = e - x * cols;
    buf[e] = C[(long long)x * ny + c];
  }
  __syncthreads();
  T2 *spec = fft_lines(buf, tmp, nx, cols, 1, cols, pm.radix + pl.rad0[0], pl.nrad[0], tw, -1);
  T2 *other = spec == buf ? tmp : buf;
  // influence function of this plane's columns (precomputed per plan, 0 at m = 0)
  const T *th = reinterpret_cast<const T *>(pm.theta) + pl.cgrid0 + (long long)kz * nx * ny + y0;
  const double mk = kz * pl.mr[2];
  const double wz = (kz > 0 && ((2 * kz != nz) || (nz & 1))) ? 2.0 : 1.0;
  double en = 0, vxx = 0, vxy = 0, vxz = 0, vyy = 0, vyz = 0, vzz = 0;
  for (int e = threadIdx.x; e < ne; e += LT) {
    const int i = divf(e, rcols), cc = e - i * cols;
    const T theta = th[(long long)i * ny + cc];
    T2 c = spec[e];
    double qq = (double)c.x * (double)c.x + (double)c.y * (double)c.y;
    double ee = wz * qq * (double)theta;
    en += ee;
    if (pm.virial && theta != T(0)) {
      const int j = y0 + cc;
      int i0 = i <= nx / 2 ? i : i - nx, j0 = j <= ny / 2 ? j : j - ny;
      double mi = i0 * pl.mr[0], mj = j0 * pl.mr[1];
      double m2 = mi * mi + mj * mj + mk * mk;
      double v = 2.0 * (1.0 / m2 + pl.fac);
      vxx += ee * (1.0 - v * mi * mi); vxy -= ee * (v * mi * mj); vxz -= ee * (v * mi * mk);
      vyy += ee * (1.0 - v * mj * mj); vyz -= ee * (v * mj * mk); vzz += ee * (1.0 - v * mk * mk);
    }
    spec[e] = cmk(c.x * theta, c.y * theta);
  }
  // the CTA's energy (x 0.5, Grid.h:319-337) and virial partials go to the box accumulators in
  // fixed point (a fixed reduction order per CTA, integer sums across CTAs)
  double part[7] = {en, vxx, vxy, vxz, vyy, vyz, vzz};
  const int np = pm.virial ? 7 : 1;
  long long *eb = s.eacc + (long long)wk.x * ACC_PER_BOX;
  const int slot[6][2] = {{0, 0}, {1, 3}, {2, 6}, {4, 4}, {5, 7}, {8, 8}};  // xx xy xz yy yz zz
  for (int c = 0; c < np; c++) {
    const double r = block_sum<LT, T>(part[c], red);
    if (threadIdx.x == 0) {
      const long long v = f2fix(r * 0.5, ENERGY_SCALE);
      if (c == 0) {
        red_add(eb + E_COUL, v);
      } else {
        red_add(eb + E_VIR + slot[c - 1][0], v);
        if (slot[c - 1][1] != slot[c - 1][0]) red_add(eb + E_VIR + slot[c - 1][1], v);
      }
    }
  }
  __syncthreads();
  const T2 *res = fft_lines(spec, other, nx, cols, 1, cols, pm.radix + pl.rad0[0], pl.nrad[0], tw, +1);
  for (int e = threadIdx.x; e < ne; e += LT) {
    const int x = divf(e, rcols), c = e - x * cols;
    C[(long long)x * ny + c] = res[e];
  }
}

// ------------------------------------------------------------ warp-shuffle transforms (n = 32 R)
// One line of n = 32 R points per warp, no shared-memory stages and no block barrier: lane l
// holds points l, l + 32, ..., l + 32 (R - 1) in registers.  Forward: an R-point DFT over the
// registers, the factors W_n^(l k1), then a 32-point decimation-in-frequency transform across
// the lanes (five xor-shuffle butterfly stages); register k1 of lane l then holds X[k1 + R b(l)],
// b = 5-bit reversal.  Inverse: consumes exactly that layout, decimation-in-time across the
// lanes, the conjugate factors, the R-point DFT over the registers, and leaves point
// l + 32 r in register r.  The factors come from the plan's table W_n^k = exp(-2 pi i k / n).
__device__ __forceinline__ int brev5(int l) { return (int)(__brev((unsigned)l) >> 27); }

template <typename T2>
__device__ __forceinline__ T2 shfl_xor2(T2 v, int d) {
  return cmk(__shfl_xor_sync(0xffffffffu, v.x, d), __shfl_xor_sync(0xffffffffu, v.y, d));
}
template <typename T2>
__device__ __forceinline__ T2 cmulc(T2 a, T2 w) {  // a * conj(w)
  return cmk(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y);
}

// Per-lane factors: st[s] = w_(2d)^(l mod d) for d = 16 >> s (w_m = exp(-2 pi i / m)), and
// rk[k1] = W_n^(l k1).
template <int R, typename T2>
struct WarpTw {
  T2 st[5], rk[R];
};
template <int R, typename T2, typename TW>
__device__ __forceinline__ WarpTw<R, T2> warp_twiddles(const TW *tw) {
  const int lane = threadIdx.x & 31;
  WarpTw<R, T2> w;
#pragma unroll
  for (int s = 0; s < 5; s++) {
    const int d = 16 >> s, j = lane & (d - 1);
    const TW t = tw[j * (16 / d) * R];
    w.st[s] = cmk(t.x, t.y);
  }
#pragma unroll
  for (int k = 0; k < R; k++) {
    const TW t = tw[lane * k];
    w.rk[k] = cmk(t.x, t.y);
  }
  return w;
}

template <int R, typename T2>
__device__ __forceinline__ void warp_fft_fwd(T2 v[R], const WarpTw<R, T2> &w) {
  const int lane = threadIdx.x & 31;
  dft_small<R>(v, -1);
#pragma unroll
  for (int k = 1; k < R; k++) v[k] = cmul(v[k], w.rk[k]);
#pragma unroll
  for (int s = 0; s < 5; s++) {
    const int d = 16 >> s;
    const bool up = (lane & d) != 0;
#pragma unroll
    for (int k = 0; k < R; k++) {
      const T2 p = shfl_xor2(v[k], d);
      v[k] = up ? cmul(csub(p, v[k]), w.st[s]) : cadd(v[k], p);
    }
  }
}

template <int R, typename T2>
__device__ __forceinline__ void warp_fft_inv(T2 v[R], const WarpTw<R, T2> &w) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 4; s >= 0; s--) {
    const int d = 16 >> s;
    const bool up = (lane & d) != 0;
#pragma unroll
    for (int k = 0; k < R; k++) {
      const T2 t = up ? cmulc(v[k], w.st[s]) : v[k];
      const T2 p = shfl_xor2(t, d);
      v[k] = up ? csub(p, t) : cadd(v[k], p);
    }
  }
#pragma unroll
  for (int k = 1; k < R; k++) v[k] = cmulc(v[k], w.rk[k]);
  dft_small<R>(v, +1);
}

constexpr int WT = 128;  // threads of the warp-transform y kernel (one row per warp)
constexpr int WX = PME_WX_THREADS;  // threads of the warp-transform x kernel (one column per warp)

// y-lines with n_y = 32 R: row C[kz][x][0..ny) per warp, up to WT / 32 rows per work item.
// The forward result is put back into natural order through a per-warp shared-memory line; the
// inverse reads its input in the forward's lane order through it.
template <typename T, int R>
__global__ void __launch_bounds__(WT) k_fft_y_warp(PmeDev pm, int sign) {
  using T2 = typename C2<T>::t;
  __shared__ T2 sline[WT / 32][32 * R];
  const int4 wk = pm.ywork[blockIdx.x];  // box, kz, x0, rows
  const PmeBoxPlan &pl = pm.plan[wk.x];
  const int nx = pl.n[0], w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (w >= wk.w) return;  // warp-uniform; no block barrier below
  constexpr int ny = 32 * R;
  T2 *row = reinterpret_cast<T2 *>(pm.cgrid) + pl.cgrid0 + ((long long)wk.y * nx + wk.z + w) * ny;
  WarpTw<R, T2> tw;
  if constexpr (sizeof(T) == 4) tw = warp_twiddles<R, T2>(pm.twiddlef + pl.tw0[1]);
  else tw = warp_twiddles<R, T2>(pm.twiddle + pl.tw0[1]);
  T2 *sl = sline[w];
  T2 v[R];
  const int b = brev5(lane);
  if (sign < 0) {
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = row[r * 32 + lane];
    warp_fft_fwd<R>(v, tw);
#pragma unroll
    for (int k = 0; k < R; k++) sl[k + R * b] = v[k];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; r++) row[r * 32 + lane] = sl[r * 32 + lane];
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) sl[r * 32 + lane] = row[r * 32 + lane];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < R; k++) v[k] = sl[k + R * b];
    warp_fft_inv<R>(v, tw);
#pragma unroll
    for (int r = 0; r < R; r++) row[r * 32 + lane] = v[r];
  }
}

// x-lines with n_x = 32 R (columns y0..y0+cols of one kz plane, one per warp): forward
// transform, influence function with energy and virial (as k_fft_x_infl), inverse transform.
// The block is staged through shared memory (coalesced rows in and out); between the two
// transforms each point stays in its lane's registers.
template <typename T, int R>
__global__ void __launch_bounds__(WX, 3) k_fft_x_warp(const SystemDev s, PmeDev pm) {
  using T2 = typename C2<T>::t;
  constexpr int nx = 32 * R, NW = WX / 32, SP = nx + 1;  // padded column stride
  __shared__ T2 sb[NW * SP];
  __shared__ T sth[NW * SP];  // the block's influence function, staged like the spectrum
  __shared__ double red[32];
  const int4 wk = pm.xwork[blockIdx.x];  // box, kz, y0, cols
  const PmeBoxPlan &pl = pm.plan[wk.x];
  const int ny = pl.n[1], nz = pl.n[2], kz = wk.y, y0 = wk.z, cols = wk.w;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T2 *C = reinterpret_cast<T2 *>(pm.cgrid) + pl.cgrid0 + (long long)kz * nx * ny + y0;
  const T *thg = reinterpret_cast<const T *>(pm.theta) + pl.cgrid0 + (long long)kz * nx * ny + y0;
  const float rcols = rcpf(cols);
  for (int e = threadIdx.x; e < nx * cols; e += WX) {
    const int x = divf(e, rcols), c = e - x * cols;
    sb[c * SP + x] = C[(long long)x * ny + c];
    sth[c * SP + x] = thg[(long long)x * ny + c];
  }
  __syncthreads();
  double en = 0, vxx = 0, vxy = 0, vxz = 0, vyy = 0, vyz = 0, vzz = 0;
  T2 v[R];
  if (w < cols) {
    WarpTw<R, T2> tw;
    if constexpr (sizeof(T) == 4) tw = warp_twiddles<R, T2>(pm.twiddlef + pl.tw0[0]);
    else tw = warp_twiddles<R, T2>(pm.twiddle + pl.tw0[0]);
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = sb[w * SP + r * 32 + lane];
    warp_fft_fwd<R>(v, tw);
    const T *th = sth + w * SP;
    const double mk = kz * pl.mr[2];
    const double wz = (kz > 0 && ((2 * kz != nz) || (nz & 1))) ? 2.0 : 1.0;
    const int j = y0 + w, j0 = j <= ny / 2 ? j : j - ny;
    const double mj = j0 * pl.mr[1];
    const int b = brev5(lane);
#pragma unroll
    for (int k = 0; k < R; k++) {
      const int i = k + R * b;
      const T theta = th[i];
      const T2 c = v[k];
      const double qq = (double)c.x * (double)c.x + (double)c.y * (double)c.y;
      const double ee = wz * qq * (double)theta;
      en += ee;
      if (pm.virial && theta != T(0)) {
        const int i0 = i <= nx / 2 ? i : i - nx;
        const double mi = i0 * pl.mr[0];
        const double m2 = mi * mi + mj * mj + mk * mk;
        const double vv = 2.0 * (1.0 / m2 + pl.fac);
        vxx += ee * (1.0 - vv * mi * mi); vxy -= ee * (vv * mi * mj); vxz -= ee * (vv * mi * mk);
        vyy += ee * (1.0 - vv * mj * mj); vyz -= ee * (vv * mj * mk); vzz += ee * (1.0 - vv * mk * mk);
      }
      v[k] = cmk(c.x * theta, c.y * theta);
    }
    warp_fft_inv<R>(v, tw);
#pragma unroll
    for (int r = 0; r < R; r++) sb[w * SP + r * 32 + lane] = v[r];
  }
  // the CTA's energy (x 0.5, Grid.h:319-337) and virial partials in fixed point, as k_fft_x_infl
  const double part[7] = {en, vxx, vxy, vxz, vyy, vyz, vzz};
  const int np = pm.virial ? 7 : 1;
  long long *eb = s.eacc + (long long)wk.x * ACC_PER_BOX;
  const int slot[6][2] = {{0, 0}, {1, 3}, {2, 6}, {4, 4}, {5, 7}, {8, 8}};  // xx xy xz yy yz zz
  for (int c = 0; c < np; c++) {
    const double r = block_sum<WX, T>(part[c], red);
    if (threadIdx.x == 0) {
      const long long q = f2fix(r * 0.5, ENERGY_SCALE);
      if (c == 0) {
        red_add(eb + E_COUL, q);
      } else {
        red_add(eb + E_VIR + slot[c - 1][0], q);
        if (slot[c - 1][1] != slot[c - 1][0]) red_add(eb + E_VIR + slot[c - 1][1], q);
      }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nx * cols; e += WX) {
    const int x = divf(e, rcols), c = e - x * cols;
    C[(long long)x * ny + c] = sb[c * SP + x];
  }
}

// ------------------------------------------------------------ plane transform (y, x, x, y)
// Composite DFTs in registers: R = R1 R2 points, index n = R2 n1 + n2 -> k = k1 + R1 k2.
// cos and sin of 2 pi k / N for the inner factors (N, k constant after unrolling).
__device__ __forceinline__ double2 unit_root(int N, int k) {
  switch (N * 16 + k) {
    case 97: return make_double2(0.50000000000000011, 0.8660254037844386);
    case 98: return make_double2(-0.49999999999999978, 0.86602540378443871);
    case 100: return make_double2(-0.50000000000000044, -0.86602540378443837);
    case 101: return make_double2(0.50000000000000011, -0.8660254037844386);
    case 129: return make_double2(0.70710678118654757, 0.70710678118654746);
    case 131: return make_double2(-0.70710678118654746, 0.70710678118654757);
    case 133: return make_double2(-0.70710678118654768, -0.70710678118654746);
    case 135: return make_double2(0.70710678118654735, -0.70710678118654768);
    default: return make_double2(0.0, 0.0);
  }
}
// a exp(SIGN 2 pi i k / N)
template <int SIGN, typename T2>
__device__ __forceinline__ T2 mul_root(T2 a, int N, int k) {
  using S = decltype(a.x);
  if (k == 0) return a;
  if (2 * k == N) return cmk(-a.x, -a.y);
  if (4 * k == N) return cis(a, SIGN);
  if (4 * k == 3 * N) return cis(a, -SIGN);
  const double2 w = unit_root(N, k);
  const S c = (S)w.x, s = (S)(SIGN * w.y);
  return cmk(a.x * c - a.y * s, a.x * s + a.y * c);
}
template <int R1, int R2, int SIGN, typename T2>
__device__ __forceinline__ void dft_composite(T2 *v) {
  T2 a[R1 * R2];
#pragma unroll
  for (int n2 = 0; n2 < R2; n2++) {
    T2 t[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; n1++) t[n1] = v[R2 * n1 + n2];
    dft_small<R1>(t, SIGN);
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) a[k1 * R2 + n2] = mul_root<SIGN>(t[k1], R1 * R2, n2 * k1);
  }
#pragma unroll
  for (int k1 = 0; k1 < R1; k1++) {
    dft_small<R2>(a + k1 * R2, SIGN);
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) v[k1 + R1 * k2] = a[k1 * R2 + k2];
  }
}
template <int R, int SIGN, typename T2>
__device__ __forceinline__ void dft_reg(T2 *v) {
  if constexpr (R <= 5) dft_small<R>(v, SIGN);
  else if constexpr (R == 6) dft_composite<2, 3, SIGN>(v);
  else dft_composite<2, 4, SIGN>(v);
}

// One in-place stage of a length-n transform on sub-blocks of m = R mq points, butterfly (b, j):
// the R points b m + j + r mq.  Forward (decimation in frequency): DFT, then the factors W_m^(j k)
// on output k; inverse: the conjugate factors on input k, then the DFT.  After the forward stages
// R0, R1, .. output k = k0 + R0 k1 + .. sits at k0 n / R0 + k1 n / (R0 R1) + ..; the inverse stages
// in reverse order take it from there.  tw: W_n^k; ts = n / m.
template <int R, int SIGN, typename T2>
__device__ __forceinline__ void stage_math(T2 *v, const T2 *tw, int j, int ts) {
  if constexpr (SIGN < 0) {
    dft_reg<R, SIGN>(v);
#pragma unroll
    for (int k = 1; k < R; k++) v[k] = cmul(v[k], tw[j * k * ts]);
  } else {
#pragma unroll
    for (int k = 1; k < R; k++) {
      const T2 w = tw[j * k * ts];
      v[k] = cmk(v[k].x * w.x + v[k].y * w.y, v[k].y * w.x - v[k].x * w.y);
    }
    dft_reg<R, SIGN>(v);
  }
}

// What one plane's transform works on.
template <typename T2>
struct PlaneCtx {
  T2 *buf;        // [nx][ld]
  const T2 *twx, *twy;
  T2 *C;          // the plane in memory, [nx][ny]
  int nx, ny, ld;
};

// Rows (y).  The outermost stage (m = ny) reads (forward) or writes (inverse) the plane in memory
// instead of the buffer, consecutive threads along the row; the others run consecutive threads
// down the rows (the odd row stride keeps them on different banks).
template <int R, int SIGN, bool OUTER, typename T2>
__device__ __forceinline__ void row_stage(const PlaneCtx<T2> &p, int m) {
  const int mq = m / R, ts = p.ny / m, total = p.nx * (p.ny / R);
  const float rq = rcpf(mq), rnx = rcpf(p.nx);
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    int row, b, j;
    if constexpr (OUTER) {
      row = divf(e, rq);
      j = e - row * mq;
      b = 0;
    } else {
      const int q = divf(e, rnx);
      row = e - q * p.nx;
      b = divf(q, rq);
      j = q - b * mq;
    }
    T2 *L = p.buf + row * p.ld + b * m + j;
    T2 *G = p.C + (long long)row * p.ny + j;
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = OUTER && SIGN < 0 ? G[r * mq] : L[r * mq];
    stage_math<R, SIGN>(v, p.twy, j, ts);
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (OUTER && SIGN > 0) G[r * mq] = v[r];
      else L[r * mq] = v[r];
    }
  }
}
// Columns (x), consecutive threads along a row.
template <int R, int SIGN, typename T2>
__device__ __forceinline__ void col_stage(const PlaneCtx<T2> &p, int m) {
  const int mq = m / R, ts = p.nx / m, total = p.ny * (p.nx / R);
  const float rq = rcpf(mq), rny = rcpf(p.ny);
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const int q = divf(e, rny), c = e - q * p.ny, b = divf(q, rq), j = q - b * mq;
    T2 *L = p.buf + (b * m + j) * p.ld + c;
    const int st = mq * p.ld;
    T2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = L[r * st];
    stage_math<R, SIGN>(v, p.twx, j, ts);
#pragma unroll
    for (int r = 0; r < R; r++) L[r * st] = v[r];
  }
}
// Energy and virial sums of the influence function whose value does not depend on the order: a box's
// energy must follow neither the block's size, which the other boxes of the system decide, nor which
// thread took what.  Each term is split into a multiple of 2^-20 and a rest rounded to a multiple of
// 2^-52 (by adding and taking away a number of that rounding unit), and the two kinds are summed apart:
// exact in FP64 while the sums stay below 2^33 and 2 kcal/mol.  Seven additions a term and no shuffles
// (a warp sum and a rounding per 32 terms instead: 20.4 for 19.2 us at 96^3).
template <bool VIR>
struct InflSums {
  static constexpr int N = VIR ? 7 : 1;  // energy, xx xy xz yy yz zz
  double hi[N] = {}, lo[N] = {};
  __device__ __forceinline__ void add(const double x[N]) {
    constexpr double UH = 1.5 * 4294967296.0, UL = 1.5;
#pragma unroll
    for (int c = 0; c < N; c++) {
      const double h = __dadd_rn(__dadd_rn(x[c], UH), -UH);
      hi[c] = __dadd_rn(hi[c], h);
      lo[c] = __dadd_rn(lo[c], __dadd_rn(__dadd_rn(__dadd_rn(x[c], -h), UL), -UL));
    }
  }
  // this warp's sums into 2 N shared words
  __device__ __forceinline__ void share(unsigned long long *acc) {
#pragma unroll
    for (int c = 0; c < N; c++) {
      const double h = warp_sum(hi[c]) * 1048576.0, l = warp_sum(lo[c]) * 4503599627370496.0;  // 2^20, 2^52
      if ((threadIdx.x & 31) == 0) {
        atomicAdd(acc + 2 * c, (unsigned long long)__double2ll_rn(h));
        atomicAdd(acc + 2 * c + 1, (unsigned long long)__double2ll_rn(l));
      }
    }
  }
  // word c of the block in the fixed point of the accumulators (x 0.5, Grid.h:319-337)
  __device__ static __forceinline__ long long fixed(const unsigned long long *acc, int c) {
    const double h = (double)(long long)acc[2 * c], l = (double)(long long)acc[2 * c + 1];
    return f2fix(0.5 * (h * (1.0 / 1048576.0) + l * (1.0 / 4503599627370496.0)), ENERGY_SCALE);
  }
};
// The columns' last forward stage, the influence function and their first inverse stage, in
// registers (m = R: no factors).  th: the plane's influence function in the order of the buffer;
// mx, my: the reciprocal vectors' components by buffer position (virial).
template <int R, bool VIR, typename T, typename T2>
__device__ __forceinline__ void col_infl(const PlaneCtx<T2> &p, const T *th, double wz, const double *mx, const double *my,
                                         double mk, double fac, InflSums<VIR> &s) {
  const int total = p.ny * (p.nx / R);
  const float rny = rcpf(p.ny);
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    double part[VIR ? 7 : 1] = {};
    const int b = divf(e, rny), c = e - b * p.ny;
    T2 *L = p.buf + b * R * p.ld + c;
    T2 v[R];
    T t[R];
#pragma unroll
    for (int r = 0; r < R; r++) t[r] = th[(b * R + r) * p.ny + c];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = L[r * p.ld];
    dft_reg<R, -1>(v);
#pragma unroll
    for (int r = 0; r < R; r++) {
      const double ee = wz * ((double)v[r].x * (double)v[r].x + (double)v[r].y * (double)v[r].y) * (double)t[r];
      part[0] += ee;
      if constexpr (VIR)
        if (t[r] != T(0)) {
          const double mi = mx[b * R + r], mj = my[c];
          const double vv = 2.0 * (1.0 / (mi * mi + mj * mj + mk * mk) + fac);
          part[1] += ee * (1.0 - vv * mi * mi); part[2] -= ee * (vv * mi * mj); part[3] -= ee * (vv * mi * mk);
          part[4] += ee * (1.0 - vv * mj * mj); part[5] -= ee * (vv * mj * mk); part[6] += ee * (1.0 - vv * mk * mk);
        }
      v[r] = cmk(v[r].x * t[r], v[r].y * t[r]);
    }
    dft_reg<R, +1>(v);
#pragma unroll
    for (int r = 0; r < R; r++) L[r * p.ld] = v[r];
    s.add(part);
  }
}

// (Radices of 9, 10 and 12 save a stage of most lengths, but the code of the stages then outgrew the
// instruction cache: fetches were the top stall, and a 98,304-atom run took 7308 us, now 7053.)
#define PLANE_RADIX(R, CALL) \
  switch (R) {               \
    case 2: CALL(2); break;  \
    case 3: CALL(3); break;  \
    case 4: CALL(4); break;  \
    case 5: CALL(5); break;  \
    case 6: CALL(6); break;  \
    default: CALL(8); break; \
  }

// One kz plane of the half spectrum per CTA, in shared memory between its two passes over memory:
// forward y and x transforms, influence function with energy and virial (Grid.h:236-341), inverse x
// and y.  Two or three register stages a direction (96 = 6 x 4 x 4), so about ten barriers; the
// three kernels before it had four or five each way and moved the spectrum through memory six
// times.  Few CTAs (49 at 96^3) of long latency, which suits running beside the pair kernel: alone
// 20 -> 13 us at 72^3, 36 -> 31 us at 125^3, 12 -> 8 us at 20^3 (22 -> 25 us at 96^3, where one line per
// warp replaced these stages, but those kernels waited for room on every SM), and two launches fewer.
template <typename T, bool VIR>
__global__ void __launch_bounds__(PLANE_MAX_THREADS) k_fft_plane(const SystemDev s, PmeDev pm) {
  using T2 = typename C2<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int2 wk = pm.pwork[blockIdx.x];  // box, kz
  const PmeBoxPlan &pl = pm.plan[wk.x];
  const int nx = pl.n[0], ny = pl.n[1], nz = pl.n[2], kz = wk.y;
  unsigned long long *acc = reinterpret_cast<unsigned long long *>(smem_raw);  // 16: the CTA's sums
  double *mx = reinterpret_cast<double *>(smem_raw) + 16, *my = mx + (VIR ? nx : 0);
  T2 *twx = reinterpret_cast<T2 *>(my + (VIR ? ny + (nx + ny) % 2 : 0)), *twy = twx + nx;
  PlaneCtx<T2> p;
  p.buf = twy + ny;
  p.twx = twx;
  p.twy = twy;
  p.C = reinterpret_cast<T2 *>(pm.cgrid) + pl.cgrid0 + (long long)kz * nx * ny;
  p.nx = nx;
  p.ny = ny;
  p.ld = ny | 1;
  if (threadIdx.x < 16) acc[threadIdx.x] = 0ull;
  for (int k = threadIdx.x; k < nx + ny; k += blockDim.x) {
    const int at = k < nx ? pl.tw0[0] + k : pl.tw0[1] + k - nx;
    if constexpr (sizeof(T) == 4) twx[k] = pm.twiddlef[at];
    else twx[k] = pm.twiddle[at];
    if constexpr (VIR) {  // components of the vector at buffer position k
      const int d = k < nx ? 0 : 1, n = pl.n[d], i = pm.perm[at];
      mx[k] = (i <= n / 2 ? i : i - n) * pl.mr[d];
    }
  }
  __syncthreads();
  const int *rx = pm.pradix + pl.prad0[0], *ry = pm.pradix + pl.prad0[1];
  const int sx = pl.npr[0], sy = pl.npr[1];
  int m = ny;
#define ROW_FIRST(R) row_stage<R, -1, true>(p, m)
  PLANE_RADIX(ry[0], ROW_FIRST)
  m /= ry[0];
  __syncthreads();
  for (int q = 1; q < sy; q++) {
#define ROW_FWD(R) row_stage<R, -1, false>(p, m)
    PLANE_RADIX(ry[q], ROW_FWD)
    m /= ry[q];
    __syncthreads();
  }
  m = nx;
  for (int q = 0; q + 1 < sx; q++) {
#define COL_FWD(R) col_stage<R, -1>(p, m)
    PLANE_RADIX(rx[q], COL_FWD)
    m /= rx[q];
    __syncthreads();
  }
  InflSums<VIR> sum;
  {
    const T *th = reinterpret_cast<const T *>(pm.theta) + pl.cgrid0 + (long long)kz * nx * ny;
    const double wz = (kz > 0 && ((2 * kz != nz) || (nz & 1))) ? 2.0 : 1.0;
#define COL_INFL(R) col_infl<R, VIR, T>(p, th, wz, mx, my, kz * pl.mr[2], pl.fac, sum)
    PLANE_RADIX(rx[sx - 1], COL_INFL)
  }
  sum.share(acc);
  __syncthreads();
  for (int q = sx - 2; q >= 0; q--) {  // (m = rx[sx - 1] here)
    m *= rx[q];
#define COL_INV(R) col_stage<R, +1>(p, m)
    PLANE_RADIX(rx[q], COL_INV)
    __syncthreads();
  }
  m = 1;
  for (int q = sy - 1; q > 0; q--) {
    m *= ry[q];
#define ROW_INV(R) row_stage<R, +1, false>(p, m)
    PLANE_RADIX(ry[q], ROW_INV)
    __syncthreads();
  }
#define ROW_LAST(R) row_stage<R, +1, true>(p, ny)
  PLANE_RADIX(ry[0], ROW_LAST)
#undef ROW_FIRST
#undef ROW_FWD
#undef COL_FWD
#undef COL_INFL
#undef COL_INV
#undef ROW_INV
#undef ROW_LAST
  // (added before the barrier that follows the influence function)
  if (threadIdx.x < (VIR ? 7 : 1)) {
    long long *eb = s.eacc + (long long)wk.x * ACC_PER_BOX;
    const int c = threadIdx.x;
    const long long q = InflSums<VIR>::fixed(acc, c);
    if (c == 0) {
      red_add(eb + E_COUL, q);
    } else {  // xx xy xz yy yz zz: words 0, 1 3, 2 6, 4, 5 7, 8
      const int w = c <= 3 ? c - 1 : c == 6 ? 8 : c, t = c == 2 ? 3 : c == 3 ? 6 : c == 5 ? 7 : w;
      red_add(eb + E_VIR + w, q);
      if (t != w) red_add(eb + E_VIR + t, q);
    }
  }
}

constexpr int ZT = 128;  // threads of the z-line kernels

// Shared memory of a z kernel: factors, positions, lines, radices (read before the first barrier with
// the rest, so that no stage waits for memory).
template <typename T2>
struct ZLines {
  PlaneCtx<T2> p;       // rows: the packed lines, of nz points
  const int *pos;       // position of index k in a transformed line
  const int *rad;
};
template <typename T, typename T2>
__device__ __forceinline__ ZLines<T2> z_lines(const PmeDev &pm, const PmeBoxPlan &pl, int npair, unsigned char *smem) {
  const int nz = pl.n[2];
  ZLines<T2> z;
  T2 *tw = reinterpret_cast<T2 *>(smem);
  int *pos = reinterpret_cast<int *>(tw + nz + (nz & 1));
  z.p.twx = nullptr;
  z.p.twy = tw;
  z.p.C = nullptr;
  z.p.nx = npair;
  z.p.ny = nz;
  z.p.ld = z_line_stride(nz, pm.zpairs, sizeof(T) == 4);
  z.p.buf = reinterpret_cast<T2 *>(pos + (nz + 3) / 4 * 4);
  z.pos = pos;
  __shared__ int rad[8];  // 2^a 3^b 5^c <= 256 in radices up to 8
  if (threadIdx.x < pl.npr[2]) rad[threadIdx.x] = pm.pradix[pl.prad0[2] + threadIdx.x];
  z.rad = rad;
  for (int k = threadIdx.x; k < nz; k += ZT) {
    if constexpr (sizeof(T) == 4) tw[k] = pm.twiddlef[pl.tw0[2] + k];
    else tw[k] = pm.twiddle[pl.tw0[2] + k];
    pos[k] = pm.perm[pl.tw0[2] + k];
  }
  return z;
}

// r2c: the work item's lines of the fixed-point charge grid, two real lines packed per complex line,
// in the plane kernel's in-place register stages; the half spectrum leaves as [kz][x][y].  Latency
// bound (load, two to four stages, store, with a barrier between each).  Against shared-memory stages
// with a table lookup per point (both directions): 14.6 + 12.1 -> 12.6 + 9.7 us at 125^3, 186 + 168
// -> 152 + 130 us for 256 boxes of 15 to 40 points; 9.2 + 16.9 -> 9.7 + 16.5 us at 96^3 beside the
// pair kernel (there the inverse had a form of one line per warp).  A box of 216 waters pays 0.6 us
// a step (38.5) for the larger code.
template <typename T>
__global__ void __launch_bounds__(ZT, sizeof(T) == 4 ? 8 : 4) k_fft_z_fwd(PmeDev pm) {
  using T2 = typename C2<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int4 wk = pm.zwork[blockIdx.x];
  const PmeBoxPlan &pl = pm.plan[wk.x];
  const int nx = pl.n[0], ny = pl.n[1], nz = pl.n[2], x = wk.y, y0 = wk.z, cnt = wk.w;
  const int npair = (cnt + 1) / 2;
  const ZLines<T2> z = z_lines<T, T2>(pm, pl, npair, smem_raw);
  long long *g = pm.qgrid + pl.grid0 + ((long long)x * ny + y0) * nz;
  const float rnz = rcpf(nz), rnp = rcpf(npair);
#pragma unroll 4
  for (int e = threadIdx.x; e < npair * nz; e += ZT) {
    const int pi = divf(e, rnz), k = e - pi * nz;
    long long *ga = g + e + pi * nz;
    const bool two = 2 * pi + 1 < cnt;
    const long long qa = __ldcs(ga), qb = two ? __ldcs(ga + nz) : 0ll;
    z.p.buf[pi * z.p.ld + k] = cmk(T((double)qa * (1.0 / GRID_SCALE)), T((double)qb * (1.0 / GRID_SCALE)));
  }
  __syncthreads();
  int m = nz;
  for (int q = 0; q < pl.npr[2]; q++) {
#define Z_FWD(R) row_stage<R, -1, false>(z.p, m)
    PLANE_RADIX(z.rad[q], Z_FWD)
#undef Z_FWD
    m /= z.rad[q];
    __syncthreads();
  }
  const int nh = nz / 2 + 1;
  T2 *C = reinterpret_cast<T2 *>(pm.cgrid) + pl.cgrid0;
  const bool vec = ((ny | cnt | pl.cgrid0) & 1) == 0;  // both lines of a pair at an aligned 16 bytes
  for (int e = threadIdx.x; e < npair * nh; e += ZT) {
    const int k = divf(e, rnp), pi = e - k * npair;
    const T2 *L = z.p.buf + pi * z.p.ld;
    const T2 zk = L[z.pos[k]], zn = L[z.pos[k == 0 ? 0 : nz - k]];
    // X = (Z_k + conj(Z_{n-k})) / 2, Y = -i/2 (Z_k - conj(Z_{n-k}))
    const T2 X = cmk(T(0.5) * (zk.x + zn.x), T(0.5) * (zk.y - zn.y));
    const T2 Y = cmk(T(0.5) * (zk.y + zn.y), T(-0.5) * (zk.x - zn.x));
    T2 *row = C + ((long long)k * nx + x) * ny + y0 + 2 * pi;
    if constexpr (sizeof(T) == 4) {
      if (vec) {
        *reinterpret_cast<float4 *>(row) = make_float4(X.x, X.y, Y.x, Y.y);
        continue;
      }
    }
    row[0] = X;
    if (2 * pi + 1 < cnt) row[1] = Y;
  }
  // the charge grid cleared for the next step
  for (int e = threadIdx.x; e < cnt * nz; e += ZT) g[e] = 0;
}

// c2r: the packed lines rebuilt from the half spectrum, in the order that the inverse stages take.
template <typename T>
__global__ void __launch_bounds__(ZT, sizeof(T) == 4 ? 8 : 4) k_fft_z_inv(PmeDev pm) {
  using T2 = typename C2<T>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int4 wk = pm.zwork[blockIdx.x];
  const PmeBoxPlan &pl = pm.plan[wk.x];
  const int nx = pl.n[0], ny = pl.n[1], nz = pl.n[2], x = wk.y, y0 = wk.z, cnt = wk.w;
  const int npair = (cnt + 1) / 2, nh = nz / 2 + 1;
  const ZLines<T2> z = z_lines<T, T2>(pm, pl, npair, smem_raw);
  const int *pos = pm.perm + pl.tw0[2];  // (not through shared memory: no barrier before the loads)
  const T2 *C = reinterpret_cast<const T2 *>(pm.cgrid) + pl.cgrid0;
  const float rnz = rcpf(nz), rnp = rcpf(npair);
  const bool vec = ((ny | cnt | pl.cgrid0) & 1) == 0;  // both lines of a pair at an aligned 16 bytes
#pragma unroll 2
  for (int e = threadIdx.x; e < npair * nh; e += ZT) {
    const int k = divf(e, rnp), pi = e - k * npair;
    const T2 *row = C + ((long long)k * nx + x) * ny + y0 + 2 * pi;
    T2 X, Y;
    if (sizeof(T) == 4 && vec) {
      const float4 v = *reinterpret_cast<const float4 *>(row);
      X = cmk(T(v.x), T(v.y));
      Y = cmk(T(v.z), T(v.w));
    } else {
      X = row[0];
      Y = (2 * pi + 1 < cnt) ? row[1] : cmk(T(0), T(0));
    }
    if (k == 0 || (2 * k == nz)) {
      X.y = T(0);
      Y.y = T(0);
    }
    // Z_k = X_k + i Y_k and Z_{n-k} = conj(X_k) + i conj(Y_k)
    T2 *L = z.p.buf + pi * z.p.ld;
    L[pos[k]] = cmk(X.x - Y.y, X.y + Y.x);
    if (k > 0 && 2 * k != nz) L[pos[nz - k]] = cmk(X.x + Y.y, Y.x - X.y);
  }
  __syncthreads();
  int m = 1;
  for (int q = pl.npr[2] - 1; q >= 0; q--) {
    m *= z.rad[q];
#define Z_INV(R) row_stage<R, +1, false>(z.p, m)
    PLANE_RADIX(z.rad[q], Z_INV)
#undef Z_INV
    __syncthreads();
  }
  T *R = reinterpret_cast<T *>(pm.rgrid) + pl.grid0 + ((long long)x * ny + y0) * nz;
  for (int e = threadIdx.x; e < npair * nz; e += ZT) {
    const int pi = divf(e, rnz), k = e - pi * nz;
    const T2 v = z.p.buf[pi * z.p.ld + k];
    R[e + pi * nz] = v.x;
    if (2 * pi + 1 < cnt) R[e + (pi + 1) * nz] = v.y;
  }
}

template <typename T>
int recip_t(const SystemDev &s, const NbListDev &nb, const PmeDev &pm, cudaStream_t st, cudaEvent_t head,
            StageMark mark, void *mctx) {
  using T2 = typename C2<T>::t;
  const int TB = 256;
  constexpr bool MIXED = sizeof(T) == 4;
  auto slots = [&](int w) { return (unsigned)(((long long)w * nb.nslot + TB - 1) / TB); };
  switch (pm.order) {  // (even, at most 8)
    case 2: k_spread<MIXED, 2><<<slots(SLOT_THREADS<2>), TB, 0, st>>>(nb, pm); break;
    case 4: k_spread<MIXED, 4><<<slots(SLOT_THREADS<4>), TB, 0, st>>>(nb, pm); break;
    case 6: k_spread<MIXED, 6><<<slots(SLOT_THREADS<6>), TB, 0, st>>>(nb, pm); break;
    default: k_spread<MIXED, 8><<<slots(SLOT_THREADS<8>), TB, 0, st>>>(nb, pm);
  }
  if (mark) mark(mctx, "pme_spread");
  // shared memory sized to the largest work item of the plan
  static bool zconf[PMB_MAX_DEVICES] = {}, lconf[PMB_MAX_DEVICES] = {};  // per device
  const int dev = device_slot();
  if (!zconf[dev]) {
    cudaFuncSetAttribute(k_fft_z_fwd<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, Z_SMEM_MAX);
    cudaFuncSetAttribute(k_fft_z_inv<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, Z_SMEM_MAX);
    zconf[dev] = true;
  }
  k_fft_z_fwd<T><<<pm.nzwork, ZT, pm.zsmem, st>>>(pm);
  if (head) cudaEventRecord(head, st);
  const size_t lsmem = 32 * sizeof(double) + sizeof(T2) * (256 + 2 * (size_t)pm.lbuf);
  if (!lconf[dev]) {
    const int lcap = (int)(32 * sizeof(double) + sizeof(T2) * (256 + 2 * (size_t)LMAXE));
    cudaFuncSetAttribute(k_fft_y<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, lcap);
    cudaFuncSetAttribute(k_fft_x_infl<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, lcap);
    lconf[dev] = true;
  }
  if (pm.npwork > 0) {  // y, x, influence, x, y of each kz plane in one kernel
    static bool pconf[2][PMB_MAX_DEVICES] = {};  // per device
    auto kern = pm.virial ? k_fft_plane<T, true> : k_fft_plane<T, false>;
    if (!pconf[pm.virial != 0][dev]) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PLANE_SMEM_MAX);
      pconf[pm.virial != 0][dev] = true;
    }
    kern<<<pm.npwork, pm.pthreads, pm.psmem, st>>>(s, pm);
  }
  // planes too large for that: y, x with the influence function, y, a launch per form of the lines
  // (lines are of at most 256 points, so such planes have lines of 64, in FP32 of 128 points or more:
  // WARP_R_MIN of the plan)
  auto fft_y = [&](int sign) {
    for (int r = 0; r < 6; r++) {
      const int n = pm.nywork[r + 1] - pm.nywork[r];
      if (n <= 0) continue;
      PmeDev q = pm;
      q.ywork += pm.nywork[r];
      if (r == 0) k_fft_y<T><<<n, LT, lsmem, st>>>(q, sign);
      else if (r == 5) k_fft_y_warp<T, 5><<<n, WT, 0, st>>>(q, sign);
      else if (r == 4) k_fft_y_warp<T, 4><<<n, WT, 0, st>>>(q, sign);
      else if constexpr (!MIXED) {
        if (r == 3) k_fft_y_warp<T, 3><<<n, WT, 0, st>>>(q, sign);
        else k_fft_y_warp<T, 2><<<n, WT, 0, st>>>(q, sign);
      }
    }
  };
  fft_y(-1);
  for (int r = 0; r < 6; r++) {
    const int n = pm.nxwork[r + 1] - pm.nxwork[r];
    if (n <= 0) continue;
    PmeDev q = pm;
    q.xwork += pm.nxwork[r];
    if (r == 0) k_fft_x_infl<T><<<n, LT, lsmem, st>>>(s, q);
    else if (r == 5) k_fft_x_warp<T, 5><<<n, WX, 0, st>>>(s, q);
    else if (r == 4) k_fft_x_warp<T, 4><<<n, WX, 0, st>>>(s, q);
    else if constexpr (!MIXED) {
      if (r == 3) k_fft_x_warp<T, 3><<<n, WX, 0, st>>>(s, q);
      else k_fft_x_warp<T, 2><<<n, WX, 0, st>>>(s, q);
    }
  }
  fft_y(+1);
  k_fft_z_inv<T><<<pm.nzwork, ZT, pm.zsmem, st>>>(pm);
  if (mark) mark(mctx, "pme_fft");
  switch (pm.order) {
    case 2: k_gather<MIXED, 2><<<slots(SLOT_THREADS<2>), TB, 0, st>>>(s, nb, pm); break;
    case 4: k_gather<MIXED, 4><<<slots(SLOT_THREADS<4>), TB, 0, st>>>(s, nb, pm); break;
    case 6: k_gather<MIXED, 6><<<slots(SLOT_THREADS<6>), TB, 0, st>>>(s, nb, pm); break;
    default: k_gather<MIXED, 8><<<slots(SLOT_THREADS<8>), TB, 0, st>>>(s, nb, pm);
  }
  if (mark) mark(mctx, "pme_gather");
  return 0;
}

}  // namespace

int pme_line_capacity() { return LMAXE; }

bool pme_plane_radices(int n, std::vector<int> &rad) {
  // the fewest stages, then the smallest sum of radices
  static const int R[] = {8, 6, 5, 4, 3, 2};
  std::vector<int> best, cur;
  int best_sum = 0;
  std::function<void(int, int, int)> search = [&](int m, int from, int sum) {
    if (m == 1) {
      if (!cur.empty() && (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && sum < best_sum))) {
        best = cur;
        best_sum = sum;
      }
      return;
    }
    if (!best.empty() && cur.size() >= best.size()) return;
    for (int k = from; k < 6; k++)
      if (m % R[k] == 0) {
        cur.push_back(R[k]);
        search(m / R[k], k, sum + R[k]);
        cur.pop_back();
      }
  };
  search(n, 0, 0);
  rad = best;
  return !best.empty();
}

size_t pme_z_smem(int nz, int lines, int precision) {
  const size_t c = precision ? sizeof(float2) : sizeof(double2);
  return c * (nz + (nz & 1)) + sizeof(int) * ((nz + 3) / 4 * 4) + c * (size_t)((lines + 1) / 2) * z_line_stride(nz, (lines + 1) / 2, precision);
}

size_t pme_plane_smem(int nx, int ny, int precision) {
  const size_t c = precision ? sizeof(float2) : sizeof(double2);
  return sizeof(double) * (16 + nx + ny + (nx + ny) % 2) + c * ((size_t)nx + ny + (size_t)nx * (ny | 1));
}

int pme_recip_launch(const SystemDev &s, const NbListDev &nb, const PmeDev &pm, cudaStream_t st, cudaEvent_t head,
                     StageMark mark, void *mctx) {
  return pm.precision ? recip_t<float>(s, nb, pm, st, head, mark, mctx)
                      : recip_t<double>(s, nb, pm, st, head, mark, mctx);
}

}  // namespace pmb

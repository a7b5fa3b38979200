// Initial conditions on the GPU in float64: PM3D.make_ic (pbhgr/pbhgr/pm3d.py:40-73) and the
// benchmark's Gaussian-peak recipe, both ending in the reference's Zel'dovich tail
// (pm3d.py:59-72): delta_k -> displacement potential -> psi = -grad phi -> CIC-interpolated
// displacements of the quiet-start lattice.
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <utility>
#include <vector>

#include "../../include/pmb200.h"
#include "common.cuh"

namespace {

constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr double kPi = 3.14159265358979323846264338328;
constexpr int kThreads = 256;

#define CU(x)                                         \
  do {                                                \
    cudaError_t e_ = (x);                             \
    if (e_ != cudaSuccess) { rc = -(int)e_; goto done; } \
  } while (0)
#define CF(x)                                         \
  do {                                                \
    cufftResult r_ = (x);                             \
    if (r_ != CUFFT_SUCCESS) { rc = -1000 - (int)r_; goto done; } \
  } while (0)

__device__ __forceinline__ double kline(int i, int N, double kf) { return kf * (double)(i < N / 2 ? i : i - N); }

// Piecewise cubic (scipy PPoly layout: c[k*m + i] multiplies (r - x_i)^(3-k)); interval by
// searchsorted(x, r, 'right') - 1 clipped to [0, m-1], as CubicSpline.__call__ does.
__device__ double spline_eval(const double* __restrict__ xs, const double* __restrict__ c, int m, double r) {
  int lo = 0, hi = m;  // find last i in [0, m] with xs[i] <= r
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (xs[mid] <= r) lo = mid; else hi = mid - 1;
  }
  int i = lo;
  if (i > m - 1) i = m - 1;
  if (i < 0) i = 0;
  const double t = r - xs[i];
  return ((c[i] * t + c[m + i]) * t + c[2 * m + i]) * t + c[3 * m + i];
}

// The curvature field amp * profile(min(r, x_m)) on the centred cell grid x = (i + 1/2) dx - L/2
// (pm3d.py:42-46); the noise (if any) is copied behind it on the way, so that one batched
// transform takes both.
__global__ void k_field(int N, double L, double amp, double a0, double a1, double a2, const double* __restrict__ xs,
                        const double* __restrict__ c, int m, const double* __restrict__ noise,
                        double* __restrict__ out) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long N3 = (long long)N * N * N;
  if (g >= N3) return;
  const int l2 = 31 - __clz(N), iz = (int)(g & (N - 1)), iy = (int)((g >> l2) & (N - 1)), ix = (int)(g >> (2 * l2));
  const double dx = L / N;
  const double X = (ix + 0.5) * dx - L / 2, Y = (iy + 0.5) * dx - L / 2, Z = (iz + 0.5) * dx - L / 2;
  const double r = sqrt((X / a0) * (X / a0) + (Y / a1) * (Y / a1) + (Z / a2) * (Z / a2));
  if (noise) out[N3 + g] = noise[g];
  out[g] = amp * spline_eval(xs, c, m, fmin(r, xs[m]));
}

// The Gaussian peak exp(-sum x_i^2 / 2 R_i^2) is a product over the axes, and so is its transform:
// out[axis][k] = sum_j exp(-x_j^2 / 2 R^2) W_N^(j k), one warp per value, instead of a field and a
// 3D transform (143 + 150 us at 256^3).
__global__ void __launch_bounds__(kThreads) k_gauss_lines(int N, double L, double r0, double r1, double r2,
                                                          double2* __restrict__ out) {
  const int w = (blockIdx.x * kThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= 3 * N) return;
  const int axis = w / N, k = w - axis * N;
  const double R = axis == 0 ? r0 : axis == 1 ? r1 : r2, dx = L / N;
  double re = 0.0, im = 0.0;
  for (int j = lane; j < N; j += 32) {
    const double X = (j + 0.5) * dx - L / 2;
    const double f = exp(-(X * X) / (2 * R * R));
    double sn, cs;
    sincospi(2.0 * (double)((j * k) & (N - 1)) / (double)N, &sn, &cs);
    re += f * cs;
    im -= f * sn;
  }
  for (int d = 16; d > 0; d >>= 1) {
    re += __shfl_xor_sync(0xffffffffu, re, d);
    im += __shfl_xor_sync(0xffffffffu, im, d);
  }
  if (lane == 0) out[w] = make_double2(re, im);
}

// Noise spectrum shape at |k| = kk.  kind 0: band-limited P flat in ln k (pm3d.py:49-54); kind 1:
// sqrt(P) = 1/k, P(0) = 0 (benchmark recipe).
struct Shape {
  int kind;
  double N3, L, tail_rms, k1, k2;
};
__device__ __forceinline__ double shape_at(const Shape& h, double kk, bool zero) {
  if (h.kind) return zero ? 0.0 : 1.0 / kk;
  if (!(kk >= h.k1 && kk <= h.k2)) return 0.0;
  const double km = fmax(kk, 1e-30);
  const double P = 2 * kPi * kPi * h.tail_rms * h.tail_rms / (km * km * km * log(h.k2 / h.k1));
  return sqrt(P * h.N3 / (h.L * h.L * h.L));
}

// Counter-based normal deviates for seeded noise generated on the device: Philox4x32-10
// (Salmon, Moraes, Dror & Shaw, SC'11: 10 rounds of the two 32x32->64 multiplies with a Weyl-
// sequence key schedule) feeding the Box-Muller transform.  Element i of the field is a
// deterministic function of (seed, i), so a run is reproducible and independent of launch shape.
__device__ __forceinline__ void philox_round(u32 (&c)[4], u32 k0, u32 k1) {
  const u32 M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  const u32 hi0 = __umulhi(M0, c[0]), lo0 = M0 * c[0];
  const u32 hi1 = __umulhi(M1, c[2]), lo1 = M1 * c[2];
  const u32 n0 = hi1 ^ c[1] ^ k0, n1 = lo1, n2 = hi0 ^ c[3] ^ k1, n3 = lo0;
  c[0] = n0;
  c[1] = n1;
  c[2] = n2;
  c[3] = n3;
}

__global__ void k_philox_normal(double* __restrict__ out, long long n, unsigned long long seed) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // one Philox call -> 4 normals
  if (4 * q >= n) return;
  u32 c[4] = {(u32)q, (u32)((unsigned long long)q >> 32), 0x5eedu, 0x1ce5u};
  u32 k0 = (u32)seed, k1 = (u32)(seed >> 32);
  for (int r = 0; r < 10; ++r) {
    philox_round(c, k0, k1);
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  // 53-bit uniforms in (0, 1] from pairs of words, then Box-Muller pairs.
  const double inv53 = 1.0 / 9007199254740992.0;
  const double u0 = ((double)((((unsigned long long)c[0] << 32) | c[1]) >> 11) + 1.0) * inv53;
  const double u1 = (double)((((unsigned long long)c[2] << 32) | c[3]) >> 11) * inv53;
  const double r = sqrt(-2.0 * log(u0));
  double sn, cs;
  sincospi(2.0 * u1, &sn, &cs);
  // The second pair reuses the words with halves swapped.
  const double v0 = ((double)((((unsigned long long)c[3] << 32) | c[2]) >> 11) + 1.0) * inv53;
  const double v1 = (double)((((unsigned long long)c[1] << 32) | c[0]) >> 11) * inv53;
  const double r2 = sqrt(-2.0 * log(v0));
  double sn2, cs2;
  sincospi(2.0 * v1, &sn2, &cs2);
  const double z[4] = {r * cs, r * sn, r2 * cs2, r2 * sn2};
  for (int k = 0; k < 4; ++k)
    if (4 * q + k < n) out[4 * q + k] = z[k];
}

// One mode of delta_k (kind 0: 0.4 k^2 zeta_k / H_i^2, pm3d.py:59), zero mode removed, and of the
// three displacements (see k_spectra).  Each spectrum carries numpy's 1/N^3 and, in the kz = 0 and
// kz = N/2 planes, its Hermitian part (numpy's irfftn uses only that part there).
__device__ __forceinline__ void four_spectra(const cufftDoubleComplex z, int kind, double kx, double ky, double kz,
                                            long long m, double* re, double* im) {
  const double k2 = m == 0 ? 1.0 : kx * kx + ky * ky + kz * kz;
  double dr = z.x, di = z.y;
  if (kind == 0) {
    const double f = 0.4 * k2 / (PM_H_I * PM_H_I);
    dr *= f;
    di *= f;
  }
  if (m == 0) dr = di = 0.0;
  const double pr = -dr / k2, pi = -di / k2;
  re[0] = dr;
  im[0] = di;
  const double kc[3] = {kx, ky, kz};
  for (int c = 0; c < 3; ++c) {  // -(i k phi) = (k pi, -k pr)
    re[c + 1] = kc[c] * pi;
    im[c + 1] = -kc[c] * pr;
  }
}

// Everything about the linear density spectrum before the potential: the peak's (gl: the Gaussian
// lines; spec: a transformed field) plus the shaped noise (ns), times its amplitude a.
struct Modes {
  int N, l2, kind;
  double kf, amp, a;
  const double2* gl;
  const cufftDoubleComplex *spec, *ns;
  Shape shape;
};
__device__ __forceinline__ cufftDoubleComplex mode_at(const Modes& g, int ix, int iy, int kz, double kx, double ky,
                                                      double kzv) {
  const int N = g.N, Nh = N / 2 + 1;
  const long long m = ((long long)ix * N + iy) * Nh + kz;
  cufftDoubleComplex z;
  if (g.kind) {
    const double2 a = g.gl[ix], b = g.gl[N + iy], c = g.gl[2 * N + kz];
    const double2 ab = make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
    z.x = g.amp * (ab.x * c.x - ab.y * c.y);
    z.y = g.amp * (ab.x * c.y + ab.y * c.x);
  } else {
    z = g.spec[m];
  }
  if (g.ns) {
    const double f = g.a * shape_at(g.shape, sqrt(kx * kx + ky * ky + kzv * kzv), m == 0);
    const cufftDoubleComplex n = g.ns[m];
    z.x += f * n.x;
    z.y += f * n.y;
  }
  return z;
}

// The nf spectra inverted at once: psi_c = -irfftn(i k_c phi) with phi = -dk / k^2 (pm3d.py:61-62),
// and (nf = 4) delta_lin = irfftn(dk) (pm3d.py:70).  noise_frac and stat (kind 1): the noise is scaled
// to noise_frac of the peak by its own rms, which is on the device.
__global__ void __launch_bounds__(kThreads) k_spectra(Modes g, double noise_frac, const double* __restrict__ stat, int nf,
                                                      cufftDoubleComplex* __restrict__ out) {
  const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int N = g.N, Nh = N / 2 + 1;
  const long long M = (long long)N * N * Nh;
  if (m >= M) return;
  g.a = g.kind ? noise_frac * g.amp / stat[0] : 1.0;
  const u32 row = (u32)m / (u32)Nh;  // M < 2^32: a mesh of 2048^3 does not fit the GPU
  const int kz = (int)(m - (long long)row * Nh), iy = (int)(row & (N - 1)), ix = (int)(row >> g.l2);
  const double kx = kline(ix, N, g.kf), ky = kline(iy, N, g.kf), kzv = g.kf * kz;
  double re[4], im[4];
  four_spectra(mode_at(g, ix, iy, kz, kx, ky, kzv), g.kind, kx, ky, kzv, m, re, im);
  if (kz == 0 || kz == N / 2) {
    const int px = (-ix) & (N - 1), py = (-iy) & (N - 1);
    const double qx = kline(px, N, g.kf), qy = kline(py, N, g.kf);
    double rp[4], ip[4];
    four_spectra(mode_at(g, px, py, kz, qx, qy, kzv), g.kind, qx, qy, kzv, ((long long)px * N + py) * Nh + kz, rp, ip);
    for (int c = 0; c < 4; ++c) {
      re[c] = 0.5 * (re[c] + rp[c]);
      im[c] = 0.5 * (im[c] - ip[c]);
    }
  }
  const double inv = 1.0 / g.shape.N3;
  for (int c = 1; c < 4; ++c) {
    out[(c - 1) * M + m].x = re[c] * inv;
    out[(c - 1) * M + m].y = im[c] * inv;
  }
  if (nf == 4) {
    out[3 * M + m].x = re[0] * inv;
    out[3 * M + m].y = im[0] * inv;
  }
}

// Rms of the shaped noise on the grid (numpy's std) from its spectrum (Parseval; the mean is the
// zero mode, left out; the half spectrum counts 0 < kz < N/2 twice), instead of transforming it
// back and reading the grid twice.  Partials per block, summed in a fixed order by the last one.
__global__ void __launch_bounds__(kThreads) k_noise_rms(Modes g, double* __restrict__ part, u32* __restrict__ count,
                                                        double* __restrict__ stat) {
  __shared__ double sh[kThreads / 32];
  __shared__ bool last;
  const int N = g.N, Nh = N / 2 + 1;
  const long long M = (long long)N * N * Nh;
  double s = 0.0;
  for (long long m = (long long)blockIdx.x * kThreads + threadIdx.x; m < M; m += (long long)gridDim.x * kThreads) {
    if (m == 0) continue;
    const u32 row = (u32)m / (u32)Nh;  // M < 2^32: a mesh of 2048^3 does not fit the GPU
    const int kz = (int)(m - (long long)row * Nh);
    const double kx = kline((int)(row >> g.l2), N, g.kf), ky = kline((int)(row & (N - 1)), N, g.kf), kzv = g.kf * kz;
    const double f = shape_at(g.shape, sqrt(kx * kx + ky * ky + kzv * kzv), false);
    const cufftDoubleComplex n = g.ns[m];
    const double p = (f * n.x) * (f * n.x) + (f * n.y) * (f * n.y);
    s += kz == 0 || kz == N / 2 ? p : 2.0 * p;
  }
  auto block_sum = [&](double v) {
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) t += sh[w];
    __syncthreads();
    return t;
  };
  const double t = block_sum(s);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = t;
    __threadfence();
    last = atomicAdd(count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double q = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kThreads) q += __ldcg(part + b);
  q = block_sum(q);
  if (threadIdx.x == 0) {
    *count = 0u;
    stat[0] = sqrt(q) / g.shape.N3;
  }
}

// Python's float modulo, x - L floor(x/L), for x / L in [-1, 2) without the general remainder (the
// same bits: both subtractions are exact there).
__device__ __forceinline__ double pymod(double x, double L) {
  if (x >= 0.0 && x < L) return x;
  if (x >= L && x < 2 * L) return x - L;
  if (x < 0.0 && x >= -L) return x + L;
  double r = fmod(x, L);
  if (r != 0.0 && ((r < 0) != (L < 0))) r += L;
  return r;
}

// One axis of the lattice: coordinate Q_j (pm3d.py:64-65), and the two mesh nodes and CIC weights at
// (Q_j + L/2) % L (pm3d.py:66).  A lattice point that lies on a node up to rounding (any Np that
// divides N into odd parts, Np = N above all) is put on it, so that the far node is not read.
struct LatticeAxis {
  double q, w0, w1;
  int i0, i1;
};
__global__ void k_lattice_axis(int N, int Np, double L, LatticeAxis* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= Np) return;
  const double dq = L / Np, dx = L / N;
  LatticeAxis a;
  a.q = (j + 0.5) * dq - L / 2;
  const double g = pymod(a.q + L / 2, L) / dx - 0.5, near = rint(g);
  const bool on = fabs(g - near) <= 4e-16 * N;
  const double fl = on ? near : floor(g);
  const long long c = (long long)fl;
  a.w1 = on ? 0.0 : g - fl;
  a.w0 = 1.0 - a.w1;
  a.i0 = (int)(((c % N) + N) % N);
  a.i1 = (int)(((c + 1) % N + N) % N);
  out[j] = a;
}

// Lattice and CIC displacement (pm3d.py:64-68): x and p of every particle.  A block takes kThreads
// consecutive particles, and their coordinates from the axis table (no division or remainder per
// particle); their 24-byte rows leave through shared memory, 8 bytes per lane in order.
__global__ void __launch_bounds__(kThreads) k_lattice(int N, int Np, double L, const LatticeAxis* __restrict__ ax,
                                                      const double* __restrict__ psi, double* __restrict__ x,
                                                      double* __restrict__ p) {
  __shared__ double sx[3 * kThreads], sp[3 * kThreads];
  const long long n = (long long)Np * Np * Np, b0 = (long long)blockIdx.x * kThreads;
  const long long i = b0 + threadIdx.x;
  if (i < n) {
    const u32 row = n < (1LL << 32) ? (u32)i / (u32)Np : (u32)(i / Np);  // jx Np + jy
    const u32 jx = row / (u32)Np;
    const LatticeAxis A[3] = {ax[jx], ax[row - jx * (u32)Np], ax[(u32)(i - (long long)row * Np)]};
    const long long N3 = (long long)N * N * N;
    double disp[3] = {0.0, 0.0, 0.0};
    for (int c = 0; c < 8; ++c) {
      const double w = (c & 4 ? A[0].w1 : A[0].w0) * (c & 2 ? A[1].w1 : A[1].w0) * (c & 1 ? A[2].w1 : A[2].w0);
      if (w == 0.0) continue;
      const long long o = ((long long)(c & 4 ? A[0].i1 : A[0].i0) * N + (c & 2 ? A[1].i1 : A[1].i0)) * N + (c & 1 ? A[2].i1 : A[2].i0);
      for (int d = 0; d < 3; ++d) disp[d] += psi[d * N3 + o] * w;
    }
    for (int d = 0; d < 3; ++d) {
      sx[3 * threadIdx.x + d] = pymod(A[d].q + disp[d] + L / 2, L);
      sp[3 * threadIdx.x + d] = PM_H_I * disp[d];
    }
  }
  __syncthreads();
  const long long m = min((long long)kThreads, n - b0) * 3;
  for (int k = threadIdx.x; k < m; k += kThreads) {
    x[3 * b0 + k] = sx[k];
    p[3 * b0 + k] = sp[k];
  }
}

constexpr int kRmsBlocks = 592;
// Entries of the axis table from the first call on: particles of more per side (48 bytes each, 412 GB)
// do not fit the GPU, so that no later call grows it.
constexpr int kAxis = 2048;

unsigned nblk(long long n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// Device buffers and FP64 cuFFT plans of pm_make_ic, kept per (device, N, path) after first use so
// that repeated calls (a request loop) neither allocate nor plan again.
struct ICWork {
  double* field = nullptr;               // [2][N^3] peak field, noise
  cufftDoubleComplex* spec = nullptr;    // [2][M] their spectra
  cufftDoubleComplex* spec4 = nullptr;   // [4][M] displacements, delta_lin
  double* real4 = nullptr;               // [4][N^3]
  double2* lines = nullptr;              // [3][N] Gaussian lines
  double* part = nullptr;                // kRmsBlocks partials, then stat[1] (noise rms)
  u32* count = nullptr;
  LatticeAxis* axis = nullptr;           // [axis_n]
  int axis_n = 0;
  double* spline = nullptr;              // [spline_n] knots, coefficients
  int spline_n = 0;
  cufftHandle d2z = 0, d2z2 = 0, z2d3 = 0, z2d4 = 0;
  bool ok = false;                       // the buffers are there
  bool gone = false;                     // released, or could not be made: not in the table any more
  // Held through a synchronous call, and by an asynchronous one while it plans, grows buffers and
  // enqueues (host threads that share a work area: their calls follow one another on the stream).
  std::mutex busy;
};
std::mutex g_ic_mu;  // the table; never held while an entry's `busy` is waited for
// Keyed by (device, N, path): the synchronous pm_make_ic and the stream-ordered
// pm_make_ic_async keep separate work areas, so the two never share buffers in flight.
std::map<std::tuple<int, int, int>, std::shared_ptr<ICWork>> g_ic;

void ic_free(ICWork& w) {
  cudaFree(w.field);
  cudaFree(w.spec);
  cudaFree(w.spec4);
  cudaFree(w.real4);
  cudaFree(w.lines);
  cudaFree(w.part);
  cudaFree(w.count);
  cudaFree(w.axis);
  cudaFree(w.spline);
  for (cufftHandle h : {w.d2z, w.d2z2, w.z2d3, w.z2d4})
    if (h) cufftDestroy(h);
}

// The work area, its `busy` held by the caller from here on.
int ic_work(int device, int N, int path, std::shared_ptr<ICWork>* out, std::unique_lock<std::mutex>* hold) {
  const std::tuple<int, int, int> key{device, N, path};
  auto make = [N](ICWork& w) {
    const long long N3 = (long long)N * N * N, M = (long long)N * N * (N / 2 + 1);
    int rc = 0;
    CU(cudaMalloc(&w.field, sizeof(double) * 2 * N3));
    CU(cudaMalloc(&w.spec, sizeof(cufftDoubleComplex) * 2 * M));
    CU(cudaMalloc(&w.spec4, sizeof(cufftDoubleComplex) * 4 * M));
    CU(cudaMalloc(&w.real4, sizeof(double) * 4 * N3));
    CU(cudaMalloc(&w.lines, sizeof(double2) * 3 * N));
    CU(cudaMalloc(&w.part, sizeof(double) * (kRmsBlocks + 1)));
    CU(cudaMalloc(&w.count, sizeof(u32)));
    CU(cudaMemset(w.count, 0, sizeof(u32)));
    CU(cudaStreamSynchronize(0));  // the caller's stream may not wait for the default one
    w.ok = true;
  done:
    return rc;
  };
  for (;;) {
    std::shared_ptr<ICWork> w;
    {
      std::lock_guard<std::mutex> lock(g_ic_mu);
      std::shared_ptr<ICWork>& e = g_ic[key];
      if (!e) e = std::make_shared<ICWork>();
      w = e;
    }
    std::unique_lock<std::mutex> busy(w->busy);
    if (w->gone) continue;  // released while this thread waited: a new one
    if (!w->ok) {
      if (int rc = make(*w)) {
        ic_free(*w);
        w->gone = true;
        std::lock_guard<std::mutex> lock(g_ic_mu);
        const auto it = g_ic.find(key);
        if (it != g_ic.end() && it->second == w) g_ic.erase(it);
        return rc;
      }
    }
    *out = std::move(w);
    *hold = std::move(busy);
    return 0;
  }
}

// A plan of the work area, made when it is first used (each holds cuFFT scratch of its own).
cufftResult use_plan(cufftHandle* h, int N, cufftType type, int batch, cudaStream_t s) {
  if (!*h) {
    int n3[3] = {N, N, N};
    const cufftResult r = cufftPlanMany(h, 3, n3, nullptr, 1, 0, nullptr, 1, 0, type, batch);
    if (r != CUFFT_SUCCESS) {
      *h = 0;
      return r;
    }
  }
  return cufftSetStream(*h, s);
}

// Grows a kept buffer to n elements; the stream is drained first, since earlier work on it may
// still read the old one.
template <class T>
cudaError_t grow(T** buf, int* have, int n, cudaStream_t s) {
  if (*have >= n) return cudaSuccess;
  cudaError_t e = cudaStreamSynchronize(s);
  if (e == cudaSuccess && *buf) e = cudaFree(*buf);
  *buf = nullptr;
  *have = 0;
  if (e == cudaSuccess) e = cudaMalloc((void**)buf, sizeof(T) * (size_t)n);
  if (e == cudaSuccess) *have = n;
  return e;
}

}  // namespace

extern "C" int pm_ic_release_cache(void) {
  std::map<std::tuple<int, int, int>, std::shared_ptr<ICWork>> all;
  {
    std::lock_guard<std::mutex> lock(g_ic_mu);
    all.swap(g_ic);
  }
  for (auto& kv : all) {
    std::lock_guard<std::mutex> busy(kv.second->busy);  // a call that has it finishes first
    if (kv.second->gone) continue;
    kv.second->gone = true;
    cudaSetDevice(std::get<0>(kv.first));
    cudaDeviceSynchronize();  // what asynchronous calls have enqueued
    ic_free(*kv.second);
  }
  return 0;
}

namespace {

int check_params(const pm_ic_params* prm, const double* x_out, const double* p_out) {
  if (!prm || !x_out || !p_out) return -2000;
  const int N = prm->N, Np = prm->Np;
  if (N < 4 || (N & (N - 1)) || Np < 1 || !(prm->L > 0)) return -2001;
  if (prm->kind == 0 && (!prm->spline_x || !prm->spline_c || prm->spline_m < 1)) return -2002;
  if (prm->kind != 0 && prm->kind != 1) return -2003;
  return 0;
}

// Bounded by the float64 transforms (cuFFT, 4 back and at most 2 forward: 1.05 of the 1.43 ms of a
// 256^3 call) and, up to 64^3, by its launches (eleven at 64^3, six of them cuFFT's).  Before the lines, the Parseval sum, the
// fused spectra and the axis table (a field transform, an inverse transform with two grid
// reductions for the rms, four passes over the spectra, 64-bit remainders per particle):
// 2.51 ms at 256^3 with noise and delta_lin, 270 -> 147 us for a 64^3 curvature profile.
//
// The IC pipeline on stream s with work area w (kind 0: w->spline holds the spline).  The noise rms
// is left in w->part[kRmsBlocks].
int make_ic_on(const pm_ic_params* prm, double* x_out, double* p_out, double* delta_lin_out, ICWork* w, cudaStream_t s) {
  const int N = prm->N, Np = prm->Np, nf = delta_lin_out ? 4 : 3;
  const long long N3 = (long long)N * N * N, M = (long long)N * N * (N / 2 + 1);
  const double L = prm->L;
  int rc = 0;
  double* stat = w->part + kRmsBlocks;
  const bool want_noise = (prm->kind == 0 && prm->tail_rms > 0) || (prm->kind == 1 && prm->noise_frac > 0);
  const bool noisy = want_noise && (prm->noise || prm->noise_seed);
  cufftHandle& inverse = nf == 4 ? w->z2d4 : w->z2d3;
  Modes g{};
  g.N = N;
  while ((1 << g.l2) < N) ++g.l2;
  g.kind = prm->kind;
  g.kf = kTwoPi / L;
  g.amp = prm->amp;
  g.gl = w->lines;
  g.spec = w->spec;
  g.ns = noisy ? w->spec + M : nullptr;
  g.shape = Shape{prm->kind, (double)N3, L, prm->tail_rms, prm->k1, prm->k2};
  CU(grow(&w->axis, &w->axis_n, std::max(Np, kAxis), s));
  k_lattice_axis<<<nblk(Np), kThreads, 0, s>>>(N, Np, L, w->axis);
  if (noisy && !prm->noise) {  // seeded device noise
    k_philox_normal<<<nblk((N3 + 3) / 4), kThreads, 0, s>>>(w->field + N3, N3, prm->noise_seed);
    CU(cudaGetLastError());
  }
  if (prm->kind == 0) {
    const int m = prm->spline_m;
    k_field<<<nblk(N3), kThreads, 0, s>>>(N, L, prm->amp, prm->axes[0], prm->axes[1], prm->axes[2], w->spline,
                                          w->spline + m + 1, m, noisy ? prm->noise : nullptr, w->field);
    CU(cudaGetLastError());
    cufftHandle& forward = noisy ? w->d2z2 : w->d2z;
    CF(use_plan(&forward, N, CUFFT_D2Z, noisy ? 2 : 1, s));
    CF(cufftExecD2Z(forward, w->field, w->spec));
  } else {
    k_gauss_lines<<<nblk(3LL * N * 32), kThreads, 0, s>>>(N, L, prm->axes[0], prm->axes[1], prm->axes[2], w->lines);
    CU(cudaGetLastError());
    if (noisy) {
      CF(use_plan(&w->d2z, N, CUFFT_D2Z, 1, s));
      CF(cufftExecD2Z(w->d2z, prm->noise ? (double*)prm->noise : w->field + N3, w->spec + M));
    }
  }
  if (noisy) {
    k_noise_rms<<<(unsigned)std::min<long long>(kRmsBlocks, nblk(M)), kThreads, 0, s>>>(g, w->part, w->count, stat);
    CU(cudaGetLastError());
  } else {
    CU(cudaMemsetAsync(stat, 0, sizeof(double), s));
  }
  k_spectra<<<nblk(M), kThreads, 0, s>>>(g, prm->noise_frac, stat, nf, w->spec4);
  CU(cudaGetLastError());
  CF(use_plan(&inverse, N, CUFFT_Z2D, nf, s));
  CF(cufftExecZ2D(inverse, w->spec4, w->real4));
  k_lattice<<<nblk((long long)Np * Np * Np), kThreads, 0, s>>>(N, Np, L, w->axis, w->real4, x_out, p_out);
  CU(cudaGetLastError());
  if (delta_lin_out)
    CU(cudaMemcpyAsync(delta_lin_out, w->real4 + 3 * N3, sizeof(double) * N3, cudaMemcpyDeviceToDevice, s));
done:
  return rc;
}

}  // namespace

extern "C" int pm_make_ic(const pm_ic_params* prm, double* x_out, double* p_out, double* delta_lin_out,
                          double* noise_rms_out) {
  if (int r = check_params(prm, x_out, p_out)) return r;
  int rc = 0, device = 0;
  double rms = 0.0;
  std::shared_ptr<ICWork> w;
  std::unique_lock<std::mutex> hold;  // released before w
  CU(cudaGetDevice(&device));
  rc = ic_work(device, prm->N, 0, &w, &hold);
  if (rc) return rc;
  if (prm->kind == 0) {
    const int m = prm->spline_m;
    CU(grow(&w->spline, &w->spline_n, 5 * m + 1, 0));
    CU(cudaMemcpyAsync(w->spline, prm->spline_x, sizeof(double) * (m + 1), cudaMemcpyHostToDevice, 0));
    CU(cudaMemcpyAsync(w->spline + m + 1, prm->spline_c, sizeof(double) * 4 * m, cudaMemcpyHostToDevice, 0));
  }
  rc = make_ic_on(prm, x_out, p_out, delta_lin_out, w.get(), 0);
  if (rc) goto done;
  CU(cudaMemcpyAsync(&rms, w->part + kRmsBlocks, sizeof(rms), cudaMemcpyDeviceToHost, 0));
  CU(cudaDeviceSynchronize());
  if (noise_rms_out) *noise_rms_out = rms;
done:
  return rc;
}

extern "C" int pm_make_ic_async(const pm_ic_params* prm, double* x_out, double* p_out, void* stream) {
  if (int r = check_params(prm, x_out, p_out)) return r;
  if (prm->kind != 1) return -2003;  // the curvature-profile ICs copy a host spline: pm_make_ic
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return -(int)e;
  std::shared_ptr<ICWork> w;
  std::unique_lock<std::mutex> hold;  // released before w
  if (int r = ic_work(device, prm->N, 1, &w, &hold)) return r;
  cufftResult f = use_plan(&w->d2z, prm->N, CUFFT_D2Z, 1, (cudaStream_t)stream);  // both now, noise or not
  if (f == CUFFT_SUCCESS) f = use_plan(&w->z2d3, prm->N, CUFFT_Z2D, 3, (cudaStream_t)stream);
  if (f != CUFFT_SUCCESS) return -1000 - (int)f;
  return make_ic_on(prm, x_out, p_out, nullptr, w.get(), (cudaStream_t)stream);
}

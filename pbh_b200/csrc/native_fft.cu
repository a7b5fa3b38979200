// Native 3D real FFT for meshes of 64^3 to 512^3 (sm_100a), and the Poisson solve built from it
// (pm3d.py:104-112: transform, Green's function, gradient, inverse transforms).
//
// Layouts (one field; fields of a batch are consecutive), N = 64, 128, 256 or 512:
//   real field      r[x][y][z]          N^3 float (the deposit's delta, the force grids)
//   spectrum        s[kz][kx][ky]       (N/2+1) x N x N complex ("plane-major")
// numpy's rfftn(r)[kx][ky][kz] is s[kz][kx][ky]: the same transform, stored with kz outermost.
//
// Every 1D transform is a two-factor (Cooley-Tukey "four-step") transform held in registers:
// a line of length L = 16 T is owned by T threads, thread t holding the 16 elements
// n = T n1 + t, n1 = 0..15.  Each thread runs a 16-point DFT over n1 in registers and scales by
// W_L^{t k1}; one shared-memory exchange hands the threads the T values of each k1 for the
// T-point DFTs of the second factor; output k = k1 + 16 k2.  For T <= 16 a thread does 16/T
// DFTs of T points; for T = 32 a pair of threads shares each 32-point DFT (two 16-point halves
// and a radix-2 step across the pair by warp shuffle).  Register DFTs are radix-2
// decimation in frequency, so their outputs sit in bit-reversed register order (compile-time).
// Exchange layouts are XOR-swizzled and rows padded so that both the write and the read side of
// every exchange hit distinct shared-memory banks within each half-warp (for the 64^3 Z pass,
// at most two-way).
//
// The engine's Poisson solve (delta -> three force grids).  The inverse along x comes first, so the
// x transform, the Green multiply and the inverse x transform of a column need no pass over
// memory between them; and because the y and z gradients multiply by factors that do not depend on
// kx, only two fields leave that pass (A = -i G delta_k and B = g(kx) A; the y and z components are
// g(ky) A and g(kz) A, multiplied where A is next read) instead of three.  256^3 and 512^3:
//   k_fft_z_r2c   a real FFT along z of CTA/T consecutive (x, y) lines per CTA (T = N/32): a complex
//                 FFT of the N/2 packed (even, odd) pairs, then the split into N/2+1 outputs,
//                 written transposed into the kz planes
//   k_fft_rows    forward Y of the planes' rows, in place
//   k_solve_cols  per column of a plane: forward X, the Green multiply, inverse X of two fields
//   k_solve_rows  inverse Y of the three components
//   k_fft_z_c2r   the real inverse along z of the three components, written as force rows
// Up to 128^3 the y-z slab of one x fits an SM:
//   k_slab_fwd    Z and Y of a slab (in engines of a few meshes up to 64^3, after finishing delta)
//   k_solve_cols  as above
//   k_slab_inv    inverse Y and Z of a slab, one component
// Per cell the five passes move 8 + 8 + 12 + 20 + 24 = 72 bytes, the three 8 + 12 + 20 = 40; the six
// passes they replace (Y before X on the way back) moved 88 and did the multiply once per
// component.  Whole solve by events, six passes, five, three: 296, 244, - us at 256^3; 2431, 2062, -
// at 512^3; 72, 47, 43 at 128^3; 42, 25, 22 at 64^3 (eight of them: -, 55, 46).  Errors against
// float64 are the same.  HBM bounds the row and Z passes (5.1-6.9 TB/s of these bytes at 256^3);
// the column pass (55 us for 202 MB) waits on its exchanges.
// Chaining the plane passes in one persistent kernel, plane by plane so that L2 holds a plane from
// pass to pass, was slower (350 us at 256^3: its item claims, waits and fences cost more than
// the HBM traffic they save).
// The plain transforms (pm_rfft3_native, pm_irfft3_native) are three launches each: the Z passes
// above and one launch per axis of the planes (k_fft_rows, k_fft_cols), in place.
// No kernel communicates between CTAs.
// Twiddles come from a 512-entry table of W_512^e computed in double precision on the host; the
// register DFTs use the exact constants cos(pi/8), cos(pi/4), cos(3 pi/8).
// Transforms are unnormalised like cuFFT's; the Green factor carries numpy's 1/N^3.
#include <cmath>
#include <cstdint>

#include <mutex>

#include "pm_kernels.cuh"

namespace {

constexpr int TWN = 512;           // entries of the twiddle table

// Threads per CTA for mesh N: 256, fewer where the mesh has few lines, so that a single small mesh
// still spreads over the SMs (a pass over the planes of one 64^3 mesh is 132 CTAs of 64 threads
// rather than 33 of 256; a solve of five such passes, before the slab kernels, 34.8 -> 33.7 us, 58 ->
// 55 us at 128^3).
template <int N>
__host__ __device__ constexpr int cta() { return N <= 64 ? 64 : N == 128 ? 128 : 256; }

__device__ float2 g_tw[TWN];       // exp(-2 pi i e / 512) of this device

__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// times W_4 = -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 mul_w4(float2 a) { return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x); }

__host__ __device__ constexpr int brev(int p, int bits) {
  int r = 0;
  for (int i = 0; i < bits; ++i) r |= ((p >> i) & 1) << (bits - 1 - i);
  return r;
}

// W_L^e from the table (conjugated for the inverse); L divides 512.
template <bool INV, int L>
__device__ __forceinline__ float2 tw_global(int e) {
  const float2 w = g_tw[(e * (TWN / L)) & (TWN - 1)];
  return INV ? cconj(w) : w;
}

// x W_16^e (conjugate twiddle for the inverse).  e is a compile-time constant wherever this is
// called from the unrolled register DFTs, so the branches and constants fold away.
template <bool INV>
__device__ __forceinline__ float2 mul_w16(float2 x, int e) {
  e &= 15;
  if (e == 0) return x;
  if (e == 8) return make_float2(-x.x, -x.y);
  if (e == 4) return mul_w4<INV>(x);
  if (e == 12) return mul_w4<!INV>(x);
  constexpr float C1 = 0.923879532511286756f, C2 = 0.707106781186547524f, C3 = 0.382683432365089772f;
  const int q = e >> 2, r = e & 3;
  const float cb = r == 1 ? C1 : (r == 2 ? C2 : C3), sb = r == 1 ? C3 : (r == 2 ? C2 : C1);
  // (cos, sin) of 2 pi e / 16: the base angle r pi / 8 turned by q quarter turns
  const float c = q == 0 ? cb : (q == 1 ? -sb : (q == 2 ? -cb : sb));
  const float s = q == 0 ? sb : (q == 1 ? cb : (q == 2 ? -sb : -cb));
  return cmul(x, make_float2(c, INV ? s : -s));
}

// Radix-2 DIF DFT of length L on v[OFF .. OFF + L - 1] in registers: afterwards v[OFF + p] holds
// output brev(p, log2 L).
template <bool INV, int L, int OFF, int NV>
__device__ __forceinline__ void dft_reg(float2 (&v)[NV]) {
  if constexpr (L > 1) {
#pragma unroll
    for (int j = 0; j < L / 2; ++j) {
      const float2 a = v[OFF + j], b = v[OFF + j + L / 2];
      v[OFF + j] = cadd(a, b);
      v[OFF + j + L / 2] = mul_w16<INV>(csub(a, b), j * (16 / L));
    }
    dft_reg<INV, L / 2, OFF, NV>(v);
    dft_reg<INV, L / 2, OFF + L / 2, NV>(v);
  }
}

template <int T>
__host__ __device__ constexpr int log2i() { return T <= 1 ? 0 : 1 + log2i<T / 2>(); }

// T-point DFTs of the 16 / T consecutive groups of u.
template <bool INV, int T, int S = 0>
__device__ __forceinline__ void dft_groups(float2 (&u)[16]) {
  if constexpr (S < 16 / T) {
    dft_reg<INV, T, T * S, 16>(u);
    dft_groups<INV, T, S + 1>(u);
  }
}

// Output element held in u[p] by thread t of a line of T threads after line_fft: for T <= 16
// group s = p / T of the thread's 16 / T groups, element q = p % T of its T-point DFT.
template <int T>
__device__ __forceinline__ int line_k(int t, int p) {
  if constexpr (T <= 16) return t + T * (p / T) + 16 * brev(p % T, log2i<T>());
  else return (t >> 1) + 16 * brev(p, 4) + 256 * (t & 1);
}

// Swizzled position of Y[k1][t] in a line's exchange row.
template <int T>
__device__ __forceinline__ int line_slot(int k1, int t) {
  if constexpr (T <= 16) return k1 * T + (t ^ (k1 & (T - 1)));
  else return k1 * 32 + (t ^ (2 * k1));
}

// The transform of one line of L = 16 T points shared by its T threads: thread t holds v[n1] =
// x[T n1 + t] on entry and u[p] = X[line_k<T>(t, p)] on exit.  row: the line's exchange row in
// shared memory (16 T values); tl: W_L^{t k1} at [k1 * T + t] (the forward ones, conjugated here
// for the inverse).  The threads of a line are
// consecutive lanes of one warp (T = 32: the whole warp), so the exchange needs no CTA barrier; the
// rows must not overlap.  Ends after the exchange has been read: the caller synchronizes the warp
// before it writes the row again.
template <bool INV>
__device__ __forceinline__ float2 twc(float2 w) { return INV ? cconj(w) : w; }

template <bool INV, int T>
__device__ __forceinline__ void line_fft(float2 (&v)[16], float2 (&u)[16], float2* row, const float2* tl, int t) {
  dft_reg<INV, 16, 0, 16>(v);
#pragma unroll
  for (int p = 0; p < 16; ++p) {
    const int k1 = brev(p, 4);
    row[line_slot<T>(k1, t)] = k1 ? cmul(v[p], twc<INV>(tl[k1 * T + t])) : v[p];
  }
  __syncwarp();  // the T threads of a line are lanes of one warp
  if constexpr (T <= 16) {
    // this thread's k1 = t + T s, s < 16 / T: one T-point DFT each
#pragma unroll
    for (int s = 0; s < 16 / T; ++s)
#pragma unroll
      for (int j = 0; j < T; ++j) u[T * s + j] = row[line_slot<T>(t + T * s, j)];
    dft_groups<INV, T>(u);
  } else {
    // k1 = t / 2; this thread's half t0 = t & 1 of the 32 values: Y[k1][2 t1 + t0], t1 = 0..15
    const int k1 = t >> 1, t0 = t & 1;
#pragma unroll
    for (int j = 0; j < 16; ++j) u[j] = row[line_slot<32>(k1, 2 * j + t0)];
    dft_reg<INV, 16, 0, 16>(u);  // u[p] = A_t0[m], m = brev(p)
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      if (t0) u[p] = cmul(u[p], twc<INV>(tl[brev(p, 4) * 32 + 16]));  // W_32^m = W_512^{16 m}
      const float ox = __shfl_xor_sync(0xffffffffu, u[p].x, 1), oy = __shfl_xor_sync(0xffffffffu, u[p].y, 1);
      // X[k1 + 16 m] = A_0 + W_32^m A_1 (even lane), X[k1 + 16 m + 256] = A_0 - W_32^m A_1 (odd lane)
      u[p] = t0 ? make_float2(ox - u[p].x, oy - u[p].y) : make_float2(u[p].x + ox, u[p].y + oy);
    }
  }
}

// Z pass geometry for mesh N: a z line is M = N/2 packed pairs shared by T = M/16 threads.
template <int N>
struct ZGeo {
  static constexpr int CTA = cta<N>(), M = N / 2, NH = N / 2 + 1, T = M / 16, L = CTA / T;  // L lines per CTA
  // Row stride (float2) of a line in shared memory and the swizzle of its natural-order row,
  // chosen so that the exchange, the row writes and the column reads of the split are free of
  // bank conflicts (T = 2: at most two-way).
  static constexpr int X = M + (T >= 8 ? 8 : T);
  static constexpr int C = L + 2;       // stride of the kz-major input tile of the inverse
  static constexpr int TILE = (NH * C > L * X) ? NH * C : L * X;
  static constexpr long long N2 = (long long)N * N, N3 = N2 * N;
  static_assert(L <= N * N, "lines per CTA");
  __device__ static int sw(int l) { return T >= 8 ? (l >> 1) & 7 : (l & 15); }
};

// Shared twiddle tables of the Z passes: tw[e] = W_N^e (e <= N/2, conjugated for the inverse),
// tl[k1 * T + t] = W_M^{t k1}.
template <bool INV, int N>
__device__ __forceinline__ void load_ztw(float2* tw, float2* tl) {
  using G = ZGeo<N>;
  for (int i = threadIdx.x; i <= G::M; i += G::CTA) tw[i] = tw_global<INV, N>(i);
  for (int i = threadIdx.x; i < 16 * G::T; i += G::CTA) tl[i] = tw_global<false, G::M>((i / G::T) * (i % G::T));
}

__device__ __forceinline__ void cpa16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Whether the peak of an engine slot deposited this step (only then have its density and, after
// the solve, its forces changed).
__device__ __forceinline__ bool slot_active(const StepArgs& A, const int* slot_peak, int slot) {
  return (A.plan[slot_peak[slot]].flags & PLAN_DEP) != 0;
}

// Pass Z forward: fields in[f][x][y][z] -> planes out[f][kz][x][y].  A CTA takes L consecutive
// (x, y) lines.  grid (N^2/L, nf).  slot_peak (engine solve): field f is slot f's density, idle
// slots are skipped.
template <int N>
__global__ void __launch_bounds__(cta<N>(), 1024 / cta<N>()) k_fft_z_r2c(const float* __restrict__ in, float2* __restrict__ out,
                                                       StepArgs A, const int* slot_peak) {
  using G = ZGeo<N>;
  __shared__ float2 tw[G::M + 1], tl[16 * G::T];
  __shared__ __align__(16) float2 xb[G::L * G::X];
  load_ztw<false, N>(tw, tl);
  pdl_wait();
  if (slot_peak && !slot_active(A, slot_peak, blockIdx.y)) return;
  const int t = threadIdx.x % G::T, l = threadIdx.x / G::T;
  const long long g0 = (long long)blockIdx.x * G::L;  // first line (x N + y) of this CTA
  const int f = blockIdx.y;
  const float2* src = reinterpret_cast<const float2*>(in + (long long)f * G::N3 + (g0 + l) * N);
  float2 v[16], u[16];
#pragma unroll
  for (int n1 = 0; n1 < 16; ++n1) v[n1] = __ldcg(src + G::T * n1 + t);  // (r[2n], r[2n+1]), n = T n1 + t
  __syncthreads();  // tables
  float2* row = xb + l * G::X;
  line_fft<false, G::T>(v, u, row, tl, t);
  __syncwarp();
  // Z_k into the line's row in natural order, swizzled so that the column reads below are
  // conflict-free: Z_k at row[k ^ sw(l)].
  const int sw = G::sw(l);
#pragma unroll
  for (int p = 0; p < 16; ++p) row[line_k<G::T>(t, p) ^ sw] = u[p];
  __syncthreads();
  // X_k = E_k + W_N^k O_k with E = (Z_k + conj Z_{M-k})/2, O = -i (Z_k - conj Z_{M-k})/2
  float2* dst = out + (long long)f * G::NH * G::N2 + g0;
  for (int e = threadIdx.x; e < G::NH * G::L; e += G::CTA) {
    const int k = e / G::L, ll = e - k * G::L, sl = G::sw(ll);
    const float2* zr = xb + ll * G::X;
    const float2 zk = zr[(k & (G::M - 1)) ^ sl];
    const float2 zm = cconj(zr[((G::M - k) & (G::M - 1)) ^ sl]);
    const float2 E = cscale(cadd(zk, zm), 0.5f);
    const float2 O = cscale(mul_w4<false>(csub(zk, zm)), 0.5f);
    dst[(long long)k * G::N2 + ll] = cadd(E, cmul(tw[k], O));
  }
}

template <int N>
__device__ __forceinline__ float kl(int i, float kf) { return kf * (float)(i < N / 2 ? i : i - N); }
// Gradient factor of line index i: the spectral k (gtab null), or the tabulated transfer function
// of a finite difference (a table, because sinf unrolled over a thread's 16 values would fill the
// instruction cache).
template <int N>
__device__ __forceinline__ float gfac(int i, float kf, const float* __restrict__ gtab) {
  return gtab ? __ldg(gtab + i) : kl<N>(i, kf);
}

// Pass Z inverse: planes in[f][kz][x][y] -> fields out[f][x][y][z].  A CTA takes L consecutive
// (x, y) lines.  grid (N^2/L, nf).  slot_peak (engine solve): field 3 s + c is component c of
// slot s, idle slots are skipped, and the z component arrives without its gradient factor g(kz),
// which is applied to each line here.
template <int N>
__global__ void __launch_bounds__(cta<N>(), 1024 / cta<N>()) k_fft_z_c2r(const float2* __restrict__ in, float* __restrict__ out,
                                                       StepArgs A, const int* slot_peak) {
  using G = ZGeo<N>;
  __shared__ float2 tw[G::M + 1], tl[16 * G::T];
  __shared__ __align__(16) float2 xb[G::TILE];  // the kz-major tile, later the exchange rows
  const long long g0 = (long long)blockIdx.x * G::L;
  const int f = blockIdx.y;
  load_ztw<true, N>(tw, tl);
  pdl_wait();
  if (slot_peak && !slot_active(A, slot_peak, f / 3)) return;
  const float2* src = in + (long long)f * G::NH * G::N2 + g0;
  for (int e = threadIdx.x; e < G::NH * G::L / 2; e += G::CTA) {  // two complex values (16 bytes) per copy
    const int k = e / (G::L / 2), ll = 2 * (e - k * (G::L / 2));
    cpa16(xb + k * G::C + ll, src + (long long)k * G::N2 + ll);
  }
  const bool zgrad = slot_peak && f % 3 == 2;
  float kf = 0.f;
  const float* gtab = nullptr;
  if (zgrad) {
    const PeakDesc& P = A.peaks[slot_peak[f / 3]];
    kf = (float)(2.0 * M_PI / P.L);
    gtab = P.gtab;
  }
  cpa_wait();
  __syncthreads();
  const int t = threadIdx.x % G::T, l = threadIdx.x / G::T;
  // Z_n = E_n + i O_n with E = X_n + conj X_{M-n}, O = (X_n - conj X_{M-n}) W_N^{-n}; a C2R
  // reads only the real parts of X_0 and X_M (numpy's irfftn does the same after its complex
  // transforms along x and y).
  float2 v[16], u[16];
#pragma unroll
  for (int n1 = 0; n1 < 16; ++n1) {
    const int n = G::T * n1 + t;
    float2 xk = xb[n * G::C + l], xm = cconj(xb[(G::M - n) * G::C + l]);
    if (zgrad) {
      xk = cscale(xk, gtab ? __ldg(gtab + n) : kf * (float)n);
      xm = cscale(xm, gtab ? __ldg(gtab + G::M - n) : kf * (float)(G::M - n));
    }
    if (n == 0) {
      xk.y = 0.f;
      xm.y = 0.f;
    }
    const float2 O = cmul(csub(xk, xm), tw[n]);
    v[n1] = cadd(cadd(xk, xm), make_float2(-O.y, O.x));
  }
  __syncthreads();  // the tile is read; its memory becomes the exchange rows
  line_fft<true, G::T>(v, u, xb + l * G::X, tl, t);
  float2* dst = reinterpret_cast<float2*>(out + (long long)f * G::N3 + (g0 + l) * N);
#pragma unroll
  for (int p = 0; p < 16; ++p) dst[line_k<G::T>(t, p)] = u[p];  // (r[2n], r[2n+1])
}

// Plane-pass geometry for mesh N: a line (row or column) of N points shared by T = N/16 threads,
// B = CTA/T lines per CTA, R = N/B blocks of lines per plane.
template <int N>
struct PGeo {
  static constexpr int CTA = cta<N>(), T = N / 16, B = CTA / T, NH = N / 2 + 1, R = N / B;
  static constexpr int RS = N + (T <= 8 ? T : 0);  // row stride in shared memory (bank-conflict free)
  static constexpr size_t COLS_SMEM = sizeof(float2) * (16 * T * B + 16 * CTA + 16 * T);  // k_solve_cols
  static constexpr long long N2 = (long long)N * N, N3 = N2 * N;
  static_assert(B <= N, "a CTA's rows (columns) lie in one plane");
};

template <int N>
__device__ __forceinline__ void load_ptw(float2* tl) {
  constexpr int T = PGeo<N>::T;
  for (int i = threadIdx.x; i < 16 * T; i += cta<N>()) tl[i] = tw_global<false, N>((i / T) * (i % T));
}

// The transform of a column shared by T threads of different warps (consecutive lanes hold
// consecutive columns): v[n1] = x[T n1 + t] on entry, u[p] = X[line_k<T>(t, p)] on exit.  buf:
// [k1][t][j], the whole CTA's.  LEAD: a barrier first, when buf may still be read.
template <bool INV, int T, int B, bool LEAD>
__device__ __forceinline__ void col_fft(float2 (&v)[16], float2 (&u)[16], float2* buf, const float2* tl, int t, int j) {
  dft_reg<INV, 16, 0, 16>(v);
  if (LEAD) __syncthreads();
#pragma unroll
  for (int p = 0; p < 16; ++p) {
    const int k1 = brev(p, 4);
    buf[(k1 * T + t) * B + j] = k1 ? cmul(v[p], twc<INV>(tl[k1 * T + t])) : v[p];
  }
  __syncthreads();
  if constexpr (T <= 16) {
    // this thread's k1 = t + T s, s < 16 / T: one T-point DFT each
#pragma unroll
    for (int s = 0; s < 16 / T; ++s)
#pragma unroll
      for (int i = 0; i < T; ++i) u[T * s + i] = buf[((t + T * s) * T + i) * B + j];
    dft_groups<INV, T>(u);
  } else {
    static_assert(T <= 32, "column pass for N <= 512");
    const int k1 = t >> 1, t0 = t & 1;
#pragma unroll
    for (int i = 0; i < 16; ++i) u[i] = buf[(k1 * 32 + 2 * i + t0) * B + j];
    dft_reg<INV, 16, 0, 16>(u);
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      if (t0) u[p] = cmul(u[p], twc<INV>(tl[brev(p, 4) * 32 + 16]));  // W_32^m
      // partner: thread t ^ 1 of the same column, B lanes away
      const float ox = __shfl_xor_sync(0xffffffffu, u[p].x, B), oy = __shfl_xor_sync(0xffffffffu, u[p].y, B);
      u[p] = t0 ? make_float2(ox - u[p].x, oy - u[p].y) : make_float2(u[p].x + ox, u[p].y + oy);
    }
  }
}

// Rows x = B rb + r of kz planes, T threads per row, [f][kz][.][.] (in place allowed: a CTA reads its
// rows before it writes them).  slot_peak (engine solve): field f is slot f's spectrum, idle slots are
// skipped.  grid (N/B * nplanes).
template <int N, bool INV>
__global__ void __launch_bounds__(cta<N>(), 1024 / cta<N>()) k_fft_rows(const float2* in, float2* out,
                                                                           const __grid_constant__ StepArgs A,
                                                                           const int* slot_peak) {
  using G = PGeo<N>;
  constexpr int T = G::T;
  __shared__ float2 tl[16 * T];
  __shared__ __align__(16) float2 buf[G::B * G::RS];
  load_ptw<N>(tl);
  pdl_wait();
  const int rb = blockIdx.x % G::R, pl = blockIdx.x / G::R;
  if (slot_peak && !slot_active(A, slot_peak, pl / G::NH)) return;
  const int t = threadIdx.x % T, r = threadIdx.x / T;
  const long long o = (long long)pl * G::N2 + (long long)(G::B * rb + r) * N;
  float2 v[16], u[16];
#pragma unroll
  for (int n1 = 0; n1 < 16; ++n1) v[n1] = in[o + T * n1 + t];
  __syncthreads();  // table
  line_fft<INV, T>(v, u, buf + r * G::RS, tl, t);
#pragma unroll
  for (int p = 0; p < 16; ++p) out[o + line_k<T>(t, p)] = u[p];
}

// Columns ky = B cb + j of kz planes, in place (the plain transforms).  Each warp access covers 32/B
// rows, B columns (8 B bytes) of each.  grid (N/B * nplanes).
template <int N, bool INV>
__global__ void __launch_bounds__(cta<N>(), 1024 / cta<N>()) k_fft_cols(float2* io) {
  using G = PGeo<N>;
  constexpr int T = G::T, B = G::B;
  __shared__ float2 tl[16 * T];
  __shared__ __align__(16) float2 buf[16 * T * B];
  load_ptw<N>(tl);
  pdl_wait();
  const int cb = blockIdx.x % G::R, pl = blockIdx.x / G::R;
  const int j = threadIdx.x % B, t = threadIdx.x / B;
  float2* plane = io + (long long)pl * G::N2 + B * cb + j;
  float2 v[16], u[16];
#pragma unroll
  for (int n1 = 0; n1 < 16; ++n1) v[n1] = plane[(long long)(T * n1 + t) * N];
  __syncthreads();
  col_fft<INV, T, B, false>(v, u, buf, tl, t, j);
#pragma unroll
  for (int p = 0; p < 16; ++p) plane[(long long)line_k<T>(t, p) * N] = u[p];
}

// ------------------------------------------------------------------------------------------
// Column pass of the solve: columns ky = B cb + j of one kz plane, T threads per column: forward X,
// A = -i G delta_k, inverse X of B = g(kx) A (to the x component's plane) and of A (in place).
// A waits in shared memory while B is transformed: kept in registers (32 more) it would leave two
// CTAs of 256 threads per SM instead of three.  Planes in descending order: the row pass before
// took them in ascending order, so the ones it left in L2 come first.  grid (N/B * nplanes).
template <int N>
__global__ void __launch_bounds__(cta<N>(), 768 / cta<N>())
    k_solve_cols(float2* spec, float2* gspec, const __grid_constant__ StepArgs A, const int* slot_peak) {
  using G = PGeo<N>;
  constexpr int T = G::T, B = G::B, R = G::R;
  extern __shared__ __align__(16) float2 s_cols[];
  float2* const buf = s_cols;                              // exchange buffer
  float2* const keep = buf + 16 * T * B + threadIdx.x;     // this thread's 16 values of A
  float2* const tl = buf + 16 * T * B + 16 * G::CTA;
  const int idx = blockIdx.x % R, pl = gridDim.x / R - 1 - blockIdx.x / R;
  const int slot = pl / G::NH, kz = pl - slot * G::NH, pk = slot_peak[slot];
  load_ptw<N>(tl);
  pdl_wait();
  if (!(A.plan[pk].flags & PLAN_DEP)) return;
  const int tid = threadIdx.x, j = tid % B, t = tid / B, ky = B * idx + j;
  float2* const col = spec + (long long)pl * G::N2 + ky;
  float2 v[16], u[16];
#pragma unroll
  for (int n1 = 0; n1 < 16; ++n1) v[n1] = col[(T * n1 + t) * N];
  __syncthreads();  // table
  col_fft<false, T, B, false>(v, u, buf, tl, t, j);
  // The spectrum of this thread's kx = T n1 + t into v.
  if constexpr (T <= 16) {
#pragma unroll
    for (int p = 0; p < 16; ++p) v[p / T + (16 / T) * brev(p % T, log2i<T>())] = u[p];
  } else {  // a thread's outputs are not its inputs' places: through the exchange buffer
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 16; ++p) buf[line_k<T>(t, p) * B + j] = u[p];
    __syncthreads();
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) v[n1] = buf[(T * n1 + t) * B + j];
  }
  const PeakDesc& P = A.peaks[pk];
  const float s_c = (float)(-1.5 * PM_H_I * PM_H_I / A.clocks[pk].a_grid / (double)G::N3);
  const float kf = (float)(2.0 * M_PI / P.L);
  const float sd2 = P.smooth > 0 ? (float)(P.smooth * P.dx) * (float)(P.smooth * P.dx) : 0.f;
  const float kyv = kl<N>(ky, kf), kzv = kf * (float)kz, yz2 = kyv * kyv + kzv * kzv;
  double w = 0.0;  // the modes' potential energy: terms in FP32, summed in FP64
#pragma unroll
  for (int n1 = 0; n1 < 16; ++n1) {
    const float kx = kf * (float)(T * n1 + t - (n1 < 8 ? 0 : N)), k2 = kx * kx + yz2;
    float Gk = s_c / k2;
    if (sd2 > 0.f) Gk *= expf(-0.5f * k2 * sd2);
    if (n1 == 0) Gk = k2 == 0.f ? 0.f : Gk;  // the mean
    const float2 d = v[n1];
    w += (double)(Gk * (d.x * d.x + d.y * d.y));
    const float2 a = make_float2(Gk * d.y, -Gk * d.x);  // -i G delta_k
    keep[n1 * G::CTA] = a;
    v[n1] = cscale(a, kx);
  }
  if (const float* const gtab = P.gtab) {
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) v[n1] = cscale(keep[n1 * G::CTA], __ldg(gtab + T * n1 + t));
  }
  for (int d = 16; d > 0; d >>= 1) w += __shfl_down_sync(0xffffffffu, w, d);
  if ((tid & 31) == 0)
    A.wpart[P.mode_base * (PM_THREADS / 32) + ((long long)kz * R + idx) * (G::CTA / 32) + (tid >> 5)] =
        (kz == 0 || kz == N / 2) ? w : 2.0 * w;  // the half spectrum counts 0 < kz < N/2 twice
  col_fft<true, T, B, true>(v, u, buf, tl, t, j);
  float2* const outx = gspec + ((long long)(3 * slot) * G::NH + kz) * G::N2 + ky;
#pragma unroll
  for (int p = 0; p < 16; ++p) outx[line_k<T>(t, p) * N] = u[p];
  asm volatile("" ::: "memory");  // A is fetched after B is stored (registers)
#pragma unroll
  for (int n1 = 0; n1 < 16; ++n1) v[n1] = keep[n1 * G::CTA];
  col_fft<true, T, B, true>(v, u, buf, tl, t, j);
#pragma unroll
  for (int p = 0; p < 16; ++p) col[line_k<T>(t, p) * N] = u[p];
}

// Row pass of the solve, one component: inverse Y of rows x = B rb + r of one kz plane, the x
// component from B in place, the y component from g(ky) A, the z component from A (its factor g(kz)
// is applied by the inverse Z pass).  The three components of a row block are adjacent in the
// grid, so that A is read from HBM once.  grid (3 * N/B * nplanes).
template <int N>
__global__ void __launch_bounds__(cta<N>(), 1024 / cta<N>())
    k_solve_rows(const float2* spec, float2* gspec, const __grid_constant__ StepArgs A, const int* slot_peak) {
  using G = PGeo<N>;
  constexpr int T = G::T, B = G::B, R = G::R;
  __shared__ float2 tl[16 * T];
  __shared__ __align__(16) float2 buf[G::B * G::RS];
  const int comp = blockIdx.x % 3, q = blockIdx.x / 3, rb = q % R, pl = q / R;
  const int slot = pl / G::NH, kz = pl - slot * G::NH, pk = slot_peak[slot];
  load_ptw<N>(tl);
  pdl_wait();
  if (!(A.plan[pk].flags & PLAN_DEP)) return;
  const int t = threadIdx.x % T, r = threadIdx.x / T, o = (B * rb + r) * N;
  float2* const dst = gspec + ((long long)(3 * slot + comp) * G::NH + kz) * G::N2 + o;
  const float2* const src = comp == 0 ? dst : spec + (long long)pl * G::N2 + o;
  float2 v[16], u[16];
#pragma unroll
  for (int n1 = 0; n1 < 16; ++n1) v[n1] = src[T * n1 + t];
  if (comp == 1) {
    const PeakDesc& P = A.peaks[pk];
    const float kf = (float)(2.0 * M_PI / P.L);
    const float* const gtab = P.gtab;
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) v[n1] = cscale(v[n1], gfac<N>(T * n1 + t, kf, gtab));
  }
  __syncthreads();  // table
  line_fft<true, T>(v, u, buf + r * G::RS, tl, t);
#pragma unroll
  for (int p = 0; p < 16; ++p) dst[line_k<T>(t, p)] = u[p];
}

// ------------------------------------------------------------------------------------------
// Meshes up to 128^3: the y and z transforms of one x slab in one kernel, the slab (NH x N complex,
// 70 KB at 128^3) in shared memory between them.  Three launches a solve instead of five, and per
// cell 8 + 12 + 20 bytes instead of 72.  A larger slab does not fit an SM.
template <int N>
struct SGeo {
  static constexpr int M = N / 2, NH = M + 1, TZ = M / 16, TY = N / 16;
  static constexpr int THREADS = (NH * TY + 31) / 32 * 32;  // one thread per 16 elements of a (kz) line
  static_assert(N * TZ <= THREADS, "a thread per 16 pairs of a z line");
  static constexpr int X = M + TZ;   // row stride (float2) of the z lines
  static constexpr int C = N + TY;   // row stride of the kz lines
  static constexpr int BUF = NH * C > N * X ? NH * C : N * X;
  static constexpr size_t SMEM = sizeof(float2) * (BUF + 16 * TZ + 16 * TY + M + 1);
  static constexpr int MINB = N == 128 ? 2 : 4;  // CTAs per SM
  // The inverse runs at 64 registers; two CTAs of 128^3 then have 512 threads each, and its one line
  // too many takes a second round.
  static constexpr int ITHREADS = N == 128 ? 512 : THREADS;
  // The forward kernel that finishes the deposit: more threads than lines, for the node sums.
  static constexpr bool SUMS = N <= 64;
  static constexpr int STHREADS = N == 64 ? 256 : 128;
  static constexpr long long N2 = (long long)N * N;
};
template <bool INV, int N, int THREADS>
__device__ __forceinline__ void load_slab_tw(float2* tz, float2* ty, float2* tw) {
  using G = SGeo<N>;
  for (int i = threadIdx.x; i < 16 * G::TZ; i += THREADS) tz[i] = tw_global<false, G::M>((i / G::TZ) * (i % G::TZ));
  for (int i = threadIdx.x; i < 16 * G::TY; i += THREADS) ty[i] = tw_global<false, N>((i / G::TY) * (i % G::TY));
  for (int i = threadIdx.x; i <= G::M; i += THREADS) tw[i] = tw_global<INV, N>(i);
}

// The plane x of a mesh out of its node sums S (PeakDesc::rho, written by the deposit's adds): delta =
// S / n_mean - 1 to the mesh and to the rows of buf (X float2 apart), the sums cleared for the next
// step.  Latency is all of it, so a thread has all its loads in flight (four at a time, with the
// clearing stores between them, took 5 us longer at 64^3).  And, as k_fixup does for other meshes, the next push's arrival counts and overflow area
// emptied and this step's gates closed.  dsum, smax: the thread's part of the mass defect and of
// the largest sum.
template <int N, int THREADS, int X>
__device__ __forceinline__ void finish_nodes(const StepArgs& A, int pk, int x, float2* buf, long long& dsum,
                                             long long& smax) {
  constexpr int PAIRS = N * N / 2, PER = PAIRS / THREADS;  // pairs per thread, all in flight at once
  static_assert(PAIRS % THREADS == 0 && PER <= 8, "");
  const PeakDesc& P = A.peaks[pk];
  const long long nmf = P.n_mean_fix;
  const double inv = P.inv_fix_nmean;
  ulonglong2* const src = reinterpret_cast<ulonglong2*>(P.rho + (long long)x * N * N);
  float2* const dst = reinterpret_cast<float2*>(P.delta + (long long)x * N * N);
  ulonglong2 S[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) S[k] = __ldcg(src + threadIdx.x + k * THREADS);
  dsum = smax = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + k * THREADS;
    const long long a = (long long)S[k].x, b = (long long)S[k].y, da = a - nmf, db = b - nmf;
    const float2 d = make_float2((float)((double)da * inv), (float)((double)db * inv));
    buf[i / (N / 2) * X + i % (N / 2)] = d;
    dst[i] = d;
    src[i] = make_ulonglong2(0, 0);
    dsum += da + db;
    smax = max(smax, max(a, b));
  }
  BinFill* const next = (A.plan[pk].flags & PLAN_SBUF ? A.fill[0] : A.fill[1]) + P.st_base;
  for (int i = x * THREADS + threadIdx.x; i < P.nst; i += N * THREADS) next[i].moved = 0u;
  if (x == 0 && threadIdx.x == 0) {
    A.ovf_n[pk] = 0u;
    *A.sort_gate = *A.layout_gate = *A.refresh_gate = 0u;
  }
}

// Forward: densities in[slot][x][y][z] (ADDS: made here from the deposit's node sums) -> spectra
// out[slot][kz][x][ky].  grid (N, nslots).
template <int N, int THREADS, bool ADDS>
__global__ void __launch_bounds__(THREADS, ADDS ? 3 : SGeo<N>::MINB)
    k_slab_fwd(const float* in, float2* out, const __grid_constant__ StepArgs A, const int* slot_peak) {
  using G = SGeo<N>;
  extern __shared__ __align__(16) float2 s_slab[];
  float2 *const xb = s_slab, *const tz = xb + G::BUF, *const ty = tz + 16 * G::TZ, *const tw = ty + 16 * G::TY;
  load_slab_tw<false, N, THREADS>(tz, ty, tw);
  const int x = blockIdx.x, slot = blockIdx.y;
  pdl_wait();
  if (!slot_active(A, slot_peak, slot)) return;
  float2 v[16], u[16];
  [[maybe_unused]] long long dsum, smax;
  const int tid = threadIdx.x;
  const bool zt = tid < N * G::TZ;  // whole warps
  const int t = tid % G::TZ, y = tid / G::TZ;
  float2* const row = xb + y * G::X;
  if constexpr (ADDS) {
    finish_nodes<N, THREADS, G::X>(A, slot_peak[slot], x, xb, dsum, smax);
    __syncthreads();  // density rows and tables
    if (zt) {
#pragma unroll
      for (int n1 = 0; n1 < 16; ++n1) v[n1] = row[G::TZ * n1 + t];
      __syncwarp();
    }
  } else {
    if (zt) {
      const float2* src = reinterpret_cast<const float2*>(in + ((long long)slot * N + x) * G::N2 + y * N);
#pragma unroll
      for (int n1 = 0; n1 < 16; ++n1) v[n1] = __ldcg(src + G::TZ * n1 + t);
    }
    __syncthreads();  // tables
  }
  if (zt) {
    line_fft<false, G::TZ>(v, u, row, tz, t);
    __syncwarp();
#pragma unroll
    for (int p = 0; p < 16; ++p) row[line_k<G::TZ>(t, p)] = u[p];
  }
  __syncthreads();
  // Line kz: X_k = E_k + W_N^k O_k of every row, E = (Z_k + conj Z_{M-k})/2, O = -i (Z_k - conj Z_{M-k})/2
  // (threads beyond the last line repeat it)
  const int k = min(tid / G::TY, G::M), ty_ = tid % G::TY;
  const float2 wk = tw[k];
#pragma unroll
  for (int n1 = 0; n1 < 16; ++n1) {
    const float2* zr = xb + (G::TY * n1 + ty_) * G::X;
    const float2 zk = zr[k & (G::M - 1)], zm = cconj(zr[(G::M - k) & (G::M - 1)]);
    const float2 E = cscale(cadd(zk, zm), 0.5f), O = cscale(mul_w4<false>(csub(zk, zm)), 0.5f);
    v[n1] = cadd(E, cmul(wk, O));
  }
  __syncthreads();  // the z lines are read; their memory becomes the exchange rows
  if ((tid & ~31) / G::TY <= G::M) line_fft<false, G::TY>(v, u, xb + k * G::C, ty, ty_);  // whole warps
  if (tid / G::TY <= G::M) {
    float2* dst = out + ((long long)slot * G::NH + k) * G::N2 + x * N;
#pragma unroll
    for (int p = 0; p < 16; ++p) dst[line_k<G::TY>(ty_, p)] = u[p];
  }
  if constexpr (ADDS) {  // the peak's statistics, off the path of the transform
    for (int d = 16; d > 0; d >>= 1) {
      dsum += __shfl_xor_sync(0xffffffffu, dsum, d);
      smax = max(smax, __shfl_xor_sync(0xffffffffu, smax, d));
    }
    if ((tid & 31) == 0) {
      atomicAdd((u64*)&A.stats[slot_peak[slot]].mass_defect, (u64)dsum);
      atomicMax(&A.stats[slot_peak[slot]].max_fix, (u64)smax);
    }
  }
}

// Inverse of one component: the x component from B (gspec's first field), y and z from A (spec) times
// their gradient factors -> force grids out[slot][comp][x][y][z].  The three components of a slab
// are adjacent in the grid, so that A is read from HBM once.  grid (3 N, nslots).
template <int N>
__global__ void __launch_bounds__(SGeo<N>::ITHREADS, SGeo<N>::MINB)
    k_slab_inv(const float2* spec, const float2* gspec, float* out, const __grid_constant__ StepArgs A,
               const int* slot_peak) {
  using G = SGeo<N>;
  extern __shared__ __align__(16) float2 s_slab[];
  float2 *const xb = s_slab, *const tz = xb + G::BUF, *const ty = tz + 16 * G::TZ, *const tw = ty + 16 * G::TY;
  load_slab_tw<true, N, G::ITHREADS>(tz, ty, tw);
  const int comp = blockIdx.x % 3, x = blockIdx.x / 3, slot = blockIdx.y;
  const int tid = threadIdx.x, ty_ = tid % G::TY;
  const PeakDesc& P = A.peaks[slot_peak[slot]];
  const float kf = (float)(2.0 * M_PI / P.L);
  const float* const gtab = P.gtab;
  pdl_wait();
  if (!slot_active(A, slot_peak, slot)) return;
  __syncthreads();  // tables
  float2 v[16], u[16];
  const float2* src = (comp == 0 ? gspec + (long long)3 * slot * G::NH * G::N2 : spec + (long long)slot * G::NH * G::N2) + x * N;
  // Whole warps take part; threads beyond the last line repeat it.
#pragma unroll 1
  for (int l0 = (tid & ~31) / G::TY; l0 <= G::M; l0 += G::ITHREADS / G::TY) {
    const int k = min(l0 + (tid & 31) / G::TY, G::M);
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) v[n1] = src[k * (int)G::N2 + G::TY * n1 + ty_];
    if (comp == 1) {
#pragma unroll
      for (int n1 = 0; n1 < 16; ++n1) v[n1] = cscale(v[n1], gfac<N>(G::TY * n1 + ty_, kf, gtab));
    } else if (comp == 2) {
      const float gz = gtab ? __ldg(gtab + k) : kf * (float)k;
#pragma unroll
      for (int n1 = 0; n1 < 16; ++n1) v[n1] = cscale(v[n1], gz);
    }
    float2* const line = xb + k * G::C;
    line_fft<true, G::TY>(v, u, line, ty, ty_);
    __syncwarp();
#pragma unroll
    for (int p = 0; p < 16; ++p) line[line_k<G::TY>(ty_, p)] = u[p];
  }
  __syncthreads();
  // Row y: Z_n = E_n + i O_n with E = X_n + conj X_{M-n}, O = (X_n - conj X_{M-n}) W_N^{-n}; only the
  // real parts of X_0 and X_M count (see k_fft_z_c2r).
  const bool zt = tid < N * G::TZ;  // whole warps
  const int t = tid % G::TZ, y = tid / G::TZ;
  if (zt) {
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) {
      const int n = G::TZ * n1 + t;
      float2 xk = xb[n * G::C + y], xm = cconj(xb[(G::M - n) * G::C + y]);
      if (n == 0) {
        xk.y = 0.f;
        xm.y = 0.f;
      }
      const float2 O = cmul(csub(xk, xm), tw[n]);
      v[n1] = cadd(cadd(xk, xm), make_float2(-O.y, O.x));
    }
  }
  __syncthreads();  // the kz lines are read; their memory becomes the exchange rows
  if (zt) {
    line_fft<true, G::TZ>(v, u, xb + y * G::X, tz, t);
    float2* dst = reinterpret_cast<float2*>(out + ((long long)(3 * slot + comp) * N + x) * G::N2 + y * N);
#pragma unroll
    for (int p = 0; p < 16; ++p) dst[line_k<G::TZ>(t, p)] = u[p];  // (r[2n], r[2n+1])
  }
}

template <int N>
int r2c_n(const float* x, float2* spec, int nfields, cudaStream_t s) {
  using Z = ZGeo<N>;
  using G = PGeo<N>;
  const unsigned blocks = (unsigned)G::R * (unsigned)(nfields * G::NH);
  pdl_launch(k_fft_z_r2c<N>, dim3((unsigned)(Z::N2 / Z::L), nfields), G::CTA, 0, s, x, spec, StepArgs{}, nullptr);
  pdl_launch(k_fft_rows<N, false>, dim3(blocks), G::CTA, 0, s, spec, spec, StepArgs{}, nullptr);
  pdl_launch(k_fft_cols<N, false>, dim3(blocks), G::CTA, 0, s, spec);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

template <int N>
int solve_n(const float* delta, float2* spec, float2* gspec, float* force, const StepArgs& A, const int* slot_peak,
            int nslots, bool sums, cudaStream_t s) {
  using G = PGeo<N>;
  const unsigned blocks = (unsigned)G::R * (unsigned)(nslots * G::NH);
  if constexpr (N <= 128) {
    using S = SGeo<N>;
    if constexpr (S::SUMS) {
      if (sums) pdl_launch(k_slab_fwd<N, S::STHREADS, true>, dim3(N, nslots), S::STHREADS, S::SMEM, s, delta, spec, A, slot_peak);
    }
    if (!S::SUMS || !sums)
      pdl_launch(k_slab_fwd<N, S::THREADS, false>, dim3(N, nslots), S::THREADS, S::SMEM, s, delta, spec, A, slot_peak);
    pdl_launch(k_solve_cols<N>, dim3(blocks), G::CTA, G::COLS_SMEM, s, spec, gspec, A, slot_peak);
    pdl_launch(k_slab_inv<N>, dim3(3 * N, nslots), S::ITHREADS, S::SMEM, s, spec, gspec, force, A, slot_peak);
  } else {
    using Z = ZGeo<N>;
    pdl_launch(k_fft_z_r2c<N>, dim3((unsigned)(Z::N2 / Z::L), nslots), G::CTA, 0, s, delta, spec, A, slot_peak);
    pdl_launch(k_fft_rows<N, false>, dim3(blocks), G::CTA, 0, s, spec, spec, A, slot_peak);
    pdl_launch(k_solve_cols<N>, dim3(blocks), G::CTA, G::COLS_SMEM, s, spec, gspec, A, slot_peak);
    pdl_launch(k_solve_rows<N>, dim3(3 * blocks), G::CTA, 0, s, spec, gspec, A, slot_peak);
    pdl_launch(k_fft_z_c2r<N>, dim3((unsigned)(Z::N2 / Z::L), 3 * nslots), G::CTA, 0, s, gspec, force, A, slot_peak);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

template <int N>
int c2r_n(const float2* spec, float2* work, float* out, int nfields, cudaStream_t s) {
  using Z = ZGeo<N>;
  using G = PGeo<N>;
  const unsigned blocks = (unsigned)G::R * (unsigned)(nfields * G::NH);
  pdl_launch(k_fft_rows<N, true>, dim3(blocks), G::CTA, 0, s, spec, work, StepArgs{}, nullptr);
  pdl_launch(k_fft_cols<N, true>, dim3(blocks), G::CTA, 0, s, work);
  pdl_launch(k_fft_z_c2r<N>, dim3((unsigned)(Z::N2 / Z::L), nfields), G::CTA, 0, s, work, out, StepArgs{}, nullptr);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

}  // namespace

bool fft_native_size(int N) { return N == 64 || N == 128 || N == 256 || N == 512; }
bool fft_solve_size(int N) { return N == 32 || fft_native_size(N); }

bool fft_solve_adds_nodes(int N) { return N == 32 || N == 64; }
// Potential-energy partials of a solve: one per warp of k_solve_cols, N / 16 threads per column.
long long fft_solve_partials(int N) { return (long long)(N / 2 + 1) * N * (N / 16) / 32; }

// Per-device set-up: the twiddle table and the shared-memory limits.  Call with the device current.
int fft_native_init() {
  float2 h[TWN];
  for (int k = 0; k < TWN; ++k) {
    const double a = -2.0 * M_PI * (double)k / (double)TWN;
    h[k] = make_float2((float)cos(a), (float)sin(a));
  }
  cudaError_t e = cudaMemcpyToSymbol(g_tw, h, sizeof(h));
  // The copy may return before it has landed, and the first transform may be on a stream that does
  // not wait for the default one.
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  auto smem = [&](auto* kernel, size_t bytes) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  smem(k_solve_cols<32>, PGeo<32>::COLS_SMEM);
  smem(k_solve_cols<64>, PGeo<64>::COLS_SMEM);
  smem(k_solve_cols<128>, PGeo<128>::COLS_SMEM);
  smem(k_solve_cols<256>, PGeo<256>::COLS_SMEM);
  smem(k_solve_cols<512>, PGeo<512>::COLS_SMEM);
  smem(k_slab_fwd<128, SGeo<128>::THREADS, false>, SGeo<128>::SMEM);
  smem(k_slab_inv<128>, SGeo<128>::SMEM);
  return e == cudaSuccess ? 0 : -(int)e;
}

// delta fields [slot][x][y][z] -> 3 force grids per slot [slot][comp][x][y][z] (the Poisson solve);
// spec [slot][kz][.][.] and gspec [slot][comp][kz][.][.] are work space.
int fft_native_solve(int N, const float* delta, float2* spec, float2* gspec, float* force, const StepArgs& A,
                     const int* slot_peak, int nslots, bool sums, cudaStream_t s) {
  if (nslots <= 0) return 0;
  switch (N) {
    case 32: return solve_n<32>(delta, spec, gspec, force, A, slot_peak, nslots, sums, s);
    case 64: return solve_n<64>(delta, spec, gspec, force, A, slot_peak, nslots, sums, s);
    case 128: return solve_n<128>(delta, spec, gspec, force, A, slot_peak, nslots, sums, s);
    case 256: return solve_n<256>(delta, spec, gspec, force, A, slot_peak, nslots, sums, s);
    case 512: return solve_n<512>(delta, spec, gspec, force, A, slot_peak, nslots, sums, s);
    default: return -2000;
  }
}

namespace {
// Plain unnormalised forward: fields [f][x][y][z] -> spectra [f][kz][kx][ky].
int fft_native_r2c(int N, const float* delta, float2* spec, int nslots, cudaStream_t s) {
  if (nslots <= 0) return 0;
  switch (N) {
    case 64: return r2c_n<64>(delta, spec, nslots, s);
    case 128: return r2c_n<128>(delta, spec, nslots, s);
    case 256: return r2c_n<256>(delta, spec, nslots, s);
    case 512: return r2c_n<512>(delta, spec, nslots, s);
    default: return -2000;
  }
}

// Plain unnormalised inverse: spectra [f][kz][kx][ky] -> fields [f][x][y][z]; gwork as spec.
int fft_native_c2r(int N, const float2* spec, float2* gwork, float* out, int nfields, cudaStream_t s) {
  if (nfields <= 0) return 0;
  switch (N) {
    case 64: return c2r_n<64>(spec, gwork, out, nfields, s);
    case 128: return c2r_n<128>(spec, gwork, out, nfields, s);
    case 256: return c2r_n<256>(spec, gwork, out, nfields, s);
    case 512: return c2r_n<512>(spec, gwork, out, nfields, s);
    default: return -2000;
  }
}

// Per-device set-up of the twiddle table, once per device; the lock keeps two host threads that
// make their first call on one device at the same time from racing on it.
std::mutex g_init_mu;
int ensure_native_init() {
  static int done[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return -(int)e;
  if (dev < 0 || dev >= 64) return -2004;
  std::lock_guard<std::mutex> lock(g_init_mu);
  if (!done[dev]) {
    if (int r = fft_native_init()) return r;
    done[dev] = 1;
  }
  return 0;
}
}  // namespace

extern "C" int pm_rfft3_native(int n, const float* x, void* spec, int nfields, void* stream) {
  if (!fft_native_size(n)) return -2000;
  if (!x || !spec) return -2001;
  if (nfields < 0) return -2003;
  if (((uintptr_t)x | (uintptr_t)spec) & 15) return -2001;  // 16-byte copies
  if (int r = ensure_native_init()) return r;
  return fft_native_r2c(n, x, (float2*)spec, nfields, (cudaStream_t)stream);
}

extern "C" int pm_irfft3_native(int n, const void* spec, void* work, float* x, int nfields, void* stream) {
  if (!fft_native_size(n)) return -2000;
  if (!spec || !work || !x) return -2001;
  if (nfields < 0) return -2004;
  if (((uintptr_t)x | (uintptr_t)spec | (uintptr_t)work) & 15) return -2001;
  if (int r = ensure_native_init()) return r;
  return fft_native_c2r(n, (const float2*)spec, (float2*)work, x, nfields, (cudaStream_t)stream);
}

extern "C" int pm_rfft3_256(const float* x, void* spec, int nfields, void* stream) {
  return pm_rfft3_native(256, x, spec, nfields, stream);
}

extern "C" int pm_irfft3_256(const void* spec, void* work, float* x, int nfields, void* stream) {
  return pm_irfft3_native(256, spec, work, x, nfields, stream);
}

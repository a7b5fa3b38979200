// Step kernels of the pm3d engine: push (CIC gather + kicks + drift, each particle written into
// the bin of its new super-tile), clock advance, regrouping (bin layouts and relayouts, the
// priming radix-sort permutation, the optional per-super-tile re-sort), halo-exchange CIC
// deposit with its face fix-up, Green's function + gradient, and particle I/O.
#include <algorithm>
#include <type_traits>

#include "pm_kernels.cuh"

namespace {

constexpr double kTwoPi = 6.283185307179586476925286766559;

// Shared-memory layout of a (TS+1)^3 node patch: node (lx, ly, lz) at lx*PS + ly*RS + lz.  The
// strides are padded so that the 8 corners read (push) or added to (deposit) by a warp of 32
// Morton-consecutive cells fall in 32 distinct banks, and so that rows start on 16 bytes
// (asynchronous 16-byte copies).
__host__ __device__ constexpr int patch_rs(int TS) { return TS == 4 ? 8 : TS == 8 ? 12 : 20; }
__host__ __device__ constexpr int patch_ps(int TS) { return TS == 4 ? 44 : TS == 8 ? 112 : 368; }
__host__ __device__ constexpr int patch_size(int TS) { return (TS + 1) * patch_ps(TS); }

__device__ __forceinline__ void cp_async16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(unsigned dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Asks L2 for `n` 16-byte elements from p on (one thread; nothing waits for it).
__device__ __forceinline__ void prefetch_l2(const void* p, int n) {
  if (n > 0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(n * 16) : "memory");
}

__device__ __forceinline__ u32 lanemask_lt() {
  u32 m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}


// Bin buffers, layouts and fills selected by a per-peak bit without indexing the
// kernel-parameter arrays dynamically (which would copy the parameter struct to local memory).
__device__ __forceinline__ int4* bpos(const StepArgs& A, int b) { return b ? A.pos1 : A.pos0; }
__device__ __forceinline__ float4* bmom(const StepArgs& A, int b) { return b ? A.mom1 : A.mom0; }
__device__ __forceinline__ BinLayout* blay(const StepArgs& A, int g) { return g ? A.lay[1] : A.lay[0]; }
__device__ __forceinline__ BinFill* bfill(const StepArgs& A, int b) { return b ? A.fill[1] : A.fill[0]; }

// The two runs of a filled bin: slots [b0, b0 + n0) (stayers) and [b1 + n0, b1 + n0 + n1)
// (arrivals), i.e. particle k < n0 + n1 of the bin sits at slot (k < n0 ? b0 : b1) + k.  The
// fill's counts are clamped into the bin, so a corrupted fill can never address outside it.
struct BinRuns {
  long long b0, b1;
  int n0, n1;
  __device__ __forceinline__ int total() const { return n0 + n1; }
  __device__ __forceinline__ long long slot(int k) const { return (k < n0 ? b0 : b1) + k; }
};
__device__ __forceinline__ BinRuns bin_runs(const BinLayout& L, const BinFill& F) {
  const u32 gap = min(F.gap, L.cap);
  const u32 stay = min(F.stay, gap);
  const u32 moved = min(F.moved, L.cap - gap);
  BinRuns r;
  r.b0 = L.base;
  r.n0 = (int)stay;
  r.b1 = (long long)L.base + gap - stay;
  r.n1 = (int)moved;
  return r;
}
// Particles in a bin: stayers plus the arrivals that found room.
__device__ __forceinline__ u32 bin_count(const BinLayout& L, const BinFill& F) {
  const u32 gap = min(F.gap, L.cap);
  return min(F.stay, gap) + min(F.moved, L.cap - gap);
}

// Locate the peak and the peak-local index of this CTA (uniform across the block).
struct TileRef {
  int pk, t, TS;
};

__device__ __forceinline__ TileRef find_tile(const int2* st_ref, int tile) {
  const int2 v = __ldg(st_ref + tile);  // the same for every thread of the CTA
  return TileRef{v.x & 0xFFFF, v.y, v.x >> 16};
}

// The digest of a clock (see PeakPlan).
__device__ __forceinline__ PeakPlan plan_of(const PeakClock& c, const PeakDesc& P) {
  PeakPlan p{};
  const bool run = c.state == PS_RUN, push = run || c.state == PS_FINALIZE;
  p.flags = (push ? PLAN_PUSH : 0u) | (run ? PLAN_RUN : 0u) | (c.sbuf ? PLAN_SBUF : 0u) | (c.lgen ? PLAN_LGEN : 0u) |
            (c.dep ? PLAN_DEP : 0u);
  p.a = c.a;
  if (push) {
    // H(a) = H_I a^(-3/2): the kick 0.5 da / (a H) and the drift da / (a^3 H) at the middle
    // (pm3d.py:122-124).
    const double a = c.a, da = c.da, amid = a + 0.5 * da;
    p.kA = (float)c.kpend;
    p.kB = run ? (float)(0.5 / PM_H_I * da * sqrt(a)) : 0.f;
    p.D = run ? (float)(da / (PM_H_I * amid * sqrt(amid) * P.dx)) : 0.f;
    p.gscale = c.a_grid == a ? 1.0f : (float)(c.a_grid / a);
  }
  return p;
}
__device__ __forceinline__ PeakPlan load_plan(const StepArgs& A, int pk) {
  union {
    int4 v[2];
    PeakPlan p;
  } u;
  const int4* src = reinterpret_cast<const int4*>(A.plan + pk);
  u.v[0] = __ldcg(src);
  u.v[1] = __ldcg(src + 1);
  return u.p;
}

// ------------------------------------------------------------------------------------------
// Push: CIC gather of the three force grids (pm3d.py:91-99) fused with the pending closing
// kick of the previous step, the opening kick and the drift of this one (pm3d.py:122-127).
// One CTA per super-tile: the (TS+1)^3 node patch of all three grids is staged in shared
// memory, and the particles of the super-tile's bin read their 8 corners from there.  Each
// result goes straight into the bin of the super-tile it is now in, in the other buffer:
// stayers take ranks from a shared-memory counter (one add per warp), arrivals from an atomic on
// the destination's `moved` count, placed after the destination's count before the step (which
// no stayer rank reaches).  An arrival that finds no room, which the spare capacity makes rare,
// goes to the peak's overflow area and the peak relayouts this step.
// Where a particle that leaves its super-tile goes: a slot of the bin of its new cell's super-tile
// (after that bin's count before the step, which no stayer rank reaches), else the peak's
// overflow area; returns false when even that is full (the bins were corrupted).
template <int T, int SB>
__device__ __forceinline__ bool push_move(const StepArgs& A, const PeakDesc& P, int pk, const BinLayout* lay, int4 np,
                                          float4 nm) {
  const int l2 = P.log2N, m = P.N - 1;
  constexpr int s = T == 4 ? 2 : T == 8 ? 3 : 4;
  const long long gD =
      P.st_base + pm_morton3((u32)(np.x >> (2 * l2)) >> s, (u32)((np.x >> l2) & m) >> s, (u32)(np.x & m) >> s);
  const BinLayout L = lay[gD];
  const u32 cnt = bin_count(L, A.fill[SB][gD]);
  const u32 r = atomicAdd(&A.fill[SB ^ 1][gD].moved, 1u);
  if (r < L.cap - cnt) {
    const u32 dst = L.base + cnt + r;
    (SB ? A.pos0 : A.pos1)[dst] = np;
    (SB ? A.mom0 : A.mom1)[dst] = nm;
    return true;
  }
  const u32 o = atomicAdd(&A.ovf_n[pk], 1u);
  if (o >= (u32)P.n) return false;
  A.lpos[P.p_off + o] = np;
  A.lmom[P.p_off + o] = nm;
  atomicAdd(&A.ovf_in[gD], 1u);
  return true;
}

// SB: the bin buffer read (its arrays are then kernel parameters, not per-thread selects).
template <int T, int SB, int PT>
__device__ __forceinline__ void push_super(const StepArgs& A, const PeakDesc& P, int pk, u32 st, float* s_f, u32* s_stay,
                                           const PeakPlan& K, const BinLayout& L, const BinFill& F) {
  constexpr int T1 = T + 1, RS = patch_rs(T), PS = patch_ps(T), CS = patch_size(T);
  constexpr int CH = T / 4 + 1;  // per patch row: T/4 copies of 16 bytes, then the (wrapped) last node
  const int N = P.N, l2 = P.log2N;
  const int sx = pm_compact3(st >> 2), sy = pm_compact3(st >> 1), sz = pm_compact3(st);
  const long long gS = P.st_base + st;
  const BinLayout* const lay = blay(A, K.flags & PLAN_LGEN);
  const BinRuns R = bin_runs(L, F);
  const int n = R.total();
  const long long N3 = (long long)N * N * N;
  // One particle per thread per sweep, the next two sweeps' particles in flight meanwhile (the
  // first two already while the patch is staged); 32-bit indices inside the bin's two runs:
  // particle k sits at [k] in the first run, at [k + d1] in the second.
  const int4* __restrict__ pp = (SB ? A.pos1 : A.pos0) + R.b0;
  const float4* __restrict__ mp = (SB ? A.mom1 : A.mom0) + R.b0;
  const int n0 = R.n0, d1 = (int)(R.b1 - R.b0);
  int k = threadIdx.x;
  int4 pa = make_int4(0, 0, 0, 0), pb = pa;
  float4 ma = make_float4(0.f, 0.f, 0.f, 0.f), mb = ma;
  if (k < n) {
    const int j = k < n0 ? k : k + d1;
    pa = pp[j];
    ma = mp[j];
  }
  if (k + PT < n) {
    const int j = k + PT < n0 ? k + PT : k + PT + d1;
    pb = pp[j];
    mb = mp[j];
  }
  if (n > 0) {
    // Asynchronous copies of the patch rows (every row start is 16-byte aligned on both sides:
    // z0 = sz*T is a multiple of 4 and the grids are 256-byte aligned).
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(s_f);
    const int z0 = sz * T, zl = (sz * T + T) & (N - 1);
    // Thread t copies piece t % CH of the patch rows t / CH, t / CH + RSTEP, ..., of all three grids
    // at once (one address computation for three copies).
    constexpr int NTH = PT - PT % CH, RSTEP = NTH / CH;
    if (threadIdx.x < NTH) {
      const int part = threadIdx.x % CH;
      const float *f0 = P.force + (part < T / 4 ? z0 + 4 * part : zl), *f1 = f0 + N3, *f2 = f1 + N3;
      const unsigned d0 = sbase + 16u * (unsigned)part;
      for (int row = threadIdx.x / CH; row < T1 * T1; row += RSTEP) {
        const int lx = row / T1, ly = row - lx * T1;
        const u32 off = ((u32)((sx * T + lx) & (N - 1)) << (2 * l2)) + ((u32)((sy * T + ly) & (N - 1)) << l2);
        const unsigned dst = d0 + 4u * (unsigned)(lx * PS + ly * RS);
        if (part < T / 4) {
          cp_async16(dst, f0 + off);
          cp_async16(dst + 4u * CS, f1 + off);
          cp_async16(dst + 8u * CS, f2 + off);
        } else {
          cp_async4(dst, f0 + off);
          cp_async4(dst + 4u * CS, f1 + off);
          cp_async4(dst + 8u * CS, f2 + off);
        }
      }
    }
    cp_async_wait_all();
  }
  __syncthreads();
  // A cell index belongs to this super-tile iff its bits outside the local ones equal the
  // super-tile's: one mask and one compare (negative or out-of-mesh values never match).
  const int local = ((T - 1) << (2 * l2)) | ((T - 1) << l2) | (T - 1);
  const int tile_bits = ((sx * T) << (2 * l2)) | ((sy * T) << l2) | (sz * T);
  const int mz = N - 1, my = mz << l2, mx = my << l2;  // the fields of a cell index
  const u32 lt = lanemask_lt();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bool bad = false, lost = false;
  double ex = 0.0, ey = 0.0, ez = 0.0, ep = 0.0;  // this thread's momentum and p^2 sums
  for (; k - lane < n; k += PT) {  // uniform across a warp, so that its votes see all lanes
    int4 ps = pa;
    float4 m = ma;
    pa = pb;
    ma = mb;
    const int k2 = k + 2 * PT;
    if (k2 < n) {
      const int j = k2 < n0 ? k2 : k2 + d1;
      pb = pp[j];
      mb = mp[j];
    }
    const bool valid = k < n;
    const int c = ps.x;
    // A particle outside this super-tile (bins and state disagree) is flagged and moved on
    // unchanged to the bin its cell names; nothing indexes outside the patch.
    const bool inside = (c & ~local) == tile_bits;
    bool stay = valid && inside;
    if (stay) {
      const float fx = __int_as_float(ps.y), fy = __int_as_float(ps.z), fz = __int_as_float(ps.w);
      const float gx = 1.0f - fx, gy = 1.0f - fy, gz = 1.0f - fz;
      const int o = ((c >> (2 * l2)) & (T - 1)) * PS + ((c >> l2) & (T - 1)) * RS + (c & (T - 1));
      float ax = 0.f, ay = 0.f, az = 0.f;
#define PM_CORNER(w, d)                       \
  {                                           \
    const float w_ = (w);                     \
    ax = fmaf(w_, s_f[o + (d)], ax);          \
    ay = fmaf(w_, s_f[CS + o + (d)], ay);     \
    az = fmaf(w_, s_f[2 * CS + o + (d)], az); \
  }
      const float w00 = gx * gy, w01 = gx * fy, w10 = fx * gy, w11 = fx * fy;
      PM_CORNER(w00 * gz, 0)
      PM_CORNER(w00 * fz, 1)
      PM_CORNER(w01 * gz, RS)
      PM_CORNER(w01 * fz, RS + 1)
      PM_CORNER(w10 * gz, PS)
      PM_CORNER(w10 * fz, PS + 1)
      PM_CORNER(w11 * gz, PS + RS)
      PM_CORNER(w11 * fz, PS + RS + 1)
#undef PM_CORNER
      ax *= K.gscale;
      ay *= K.gscale;
      az *= K.gscale;
      float px = m.x + K.kA * ax, py = m.y + K.kA * ay, pz = m.z + K.kA * az;
      // Momentum synchronised with the positions (after the closing kick): energy and momentum sums.
      {
        const double dx = px, dy = py, dz = pz;
        ex += dx;
        ey += dy;
        ez += dz;
        ep += dx * dx + dy * dy + dz * dz;
      }
      const bool finite = fabsf(px) < INFINITY && fabsf(py) < INFINITY && fabsf(pz) < INFINITY;
      if ((K.flags & PLAN_RUN) && finite) {  // a non-finite particle stays where it is (the peak is flagged)
        px += K.kB * ax;
        py += K.kB * ay;
        pz += K.kB * az;
        int cx, cy, cz;  // cells crossed
#define PM_DRIFT(f, p, i, out)    \
  {                               \
    float fn = f + K.D * p;       \
    float fl = floorf(fn);        \
    fn -= fl;                     \
    if (fn >= 1.0f) {             \
      fn -= 1.0f;                 \
      fl += 1.0f;                 \
    }                             \
    out = __float_as_int(fn);     \
    i = (int)fl;                  \
  }
        PM_DRIFT(fx, px, cx, ps.y)
        PM_DRIFT(fy, py, cy, ps.z)
        PM_DRIFT(fz, pz, cz, ps.w)
#undef PM_DRIFT
        // Each field of the cell index advanced modulo N in place (carries fall outside its mask).
        ps.x = ((c + (int)((u32)cx << (2 * l2))) & mx) | ((c + (int)((u32)cy << l2)) & my) | ((c + cz) & mz);
        stay = (ps.x & ~local) == tile_bits;
        bad |= !(fabsf(px) < INFINITY && fabsf(py) < INFINITY && fabsf(pz) < INFINITY);
      }
      bad |= !finite;
      m.x = px;
      m.y = py;
      m.z = pz;
    }
    const u32 sm = __ballot_sync(0xffffffffu, stay);
    u32 r = 0;
    if (lane == 0) r = atomicAdd(s_stay, (u32)__popc(sm));
    r = L.base + __shfl_sync(0xffffffffu, r, 0) + (u32)__popc(sm & lt);
    if (stay) {
      if (r < L.base + L.cap) {  // always: the stayers are at most the bin's count
        (SB ? A.pos0 : A.pos1)[r] = ps;
        (SB ? A.mom0 : A.mom1)[r] = m;
      } else {
        lost = true;
      }
    } else if (valid) {
      bad |= !inside;
      if (!inside && !(c >= 0 && c < N3)) ps.x = tile_bits;  // a cell outside the mesh names no bin: this one
      lost |= !push_move<T, SB>(A, P, pk, lay, ps, m);
    }
  }
  // Super-tile partials of the momentum and p^2 sums, in a fixed order: a plain FP64 tree over
  // the 32 lanes of a warp (about 5e-16 of the sum of magnitudes; compensating it cost 4 % of the
  // push), then compensated merges across the warps here and across super-tiles in the energy CTAs.
  __shared__ double s_e[PT / 32][4];
  const double ea[4] = {ex, ey, ez, ep};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    double v = ea[q];
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    if (lane == 0) s_e[warp][q] = v;
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&A.stats[pk].status, 1u);
  if (__any_sync(0xffffffffu, lost) && lane == 0) atomicOr(&A.stats[pk].status, 4u);
  __syncthreads();
  if (threadIdx.x == PT - 1) {
    // This bin's fill in the buffer written: its stayers, and where its arrivals start.
    A.fill[SB ^ 1][gS].stay = *s_stay;
    A.fill[SB ^ 1][gS].gap = (u32)n;
  }
  if (warp < 4) {  // one warp per sum
    static_assert(PT >= 128 && PT <= 1024, "four warps for the sums, one lane per warp of the CTA");
    CSum t = csum_warp(CSum{lane < PT / 32 ? s_e[lane][warp] : 0.0, 0.0});
    if (lane == 0) A.epart[gS * 4 + warp] = make_double2(t.s, t.c);
  }
}

// PT threads per CTA (push_threads).  TS16: the engine has super-tiles of 16^3 cells.
template <int PT, bool TS16>
__global__ void __launch_bounds__(PT, 1024 / PT) k_push(const __grid_constant__ StepArgs A) {
  extern __shared__ __align__(16) float s_f[];
  __shared__ u32 s_stay;
  // A CTA's work is a chain of memory round trips (its tile, its peak and bin, then its particles
  // and force patch): as few as possible, because only two CTAs share an SM to hide them.  Both
  // candidates of the bin's layout and fill are fetched beside the plan that selects them.
  const TileRef tr = find_tile(A.st_ref, blockIdx.x);
  if (threadIdx.x == 0) s_stay = 0u;
  pdl_wait();
  const PeakPlan K = load_plan(A, tr.pk);
  const int4 F0 = __ldcg(reinterpret_cast<const int4*>(A.fill[0] + blockIdx.x)),
             F1 = __ldcg(reinterpret_cast<const int4*>(A.fill[1] + blockIdx.x));
  const int2 L0 = __ldcg(reinterpret_cast<const int2*>(A.lay[0] + blockIdx.x)),
             L1 = __ldcg(reinterpret_cast<const int2*>(A.lay[1] + blockIdx.x));
  const PeakDesc P = A.peaks[tr.pk];
  const int4 f = K.flags & PLAN_SBUF ? F1 : F0;
  const int2 l = K.flags & PLAN_LGEN ? L1 : L0;
  const BinFill F{(u32)f.x, (u32)f.y, (u32)f.z, 0u};
  const BinLayout L{(u32)l.x, (u32)l.y};
  if (threadIdx.x == 0 && tr.t == 0) A.pushed_a[tr.pk] = K.flags & PLAN_PUSH ? K.a : -1.0;
  if (!(K.flags & PLAN_PUSH)) return;
  const u32 st = (u32)tr.t;
  const bool sb = K.flags & PLAN_SBUF;
  switch (P.TS) {
    case 4:
      if (sb) push_super<4, 1, PT>(A, P, tr.pk, st, s_f, &s_stay, K, L, F);
      else push_super<4, 0, PT>(A, P, tr.pk, st, s_f, &s_stay, K, L, F);
      break;
    case 8:
      if (sb) push_super<8, 1, PT>(A, P, tr.pk, st, s_f, &s_stay, K, L, F);
      else push_super<8, 0, PT>(A, P, tr.pk, st, s_f, &s_stay, K, L, F);
      break;
    default:
      if (!TS16) break;
      if (sb) push_super<16, 1, PT>(A, P, tr.pk, st, s_f, &s_stay, K, L, F);
      else push_super<16, 0, PT>(A, P, tr.pk, st, s_f, &s_stay, K, L, F);
      break;
  }
}

// Bin layout of a peak that primes or relayouts this step, by one CTA of LAYOUT_THREADS.  The new count
// of each super-tile comes from the sorted keys when priming; else it is the bin the push filled
// plus its arrivals in the overflow area.  A bin's base capacity is count + count/8 +
// BIN_SLACK_MIN (the peak's bin_shift and bin_min), rounded up to BIN_ALIGN.  On a relayout a
// bin also asks for room for BIN_ARRIVALS times the arrivals of this step plus bin_grow steps
// of its net growth in this step (a bin that particles stream through needs room for its
// arrivals even when its count stays put), so that collapsing and infalling regions do not
// relayout every step.
//   Partial relayout (clock.relayout = 1): when the free space after the last bin of the peak's
// region holds, with their base capacity and wanted room, every overflowed bin and every bin
// whose remaining room is below another step of its arrivals, only those bins move there (in
// the buffer the push filled, which stays current); the others keep their place and their two
// runs.  The old places stay unused until the next full relayout.
//   Full relayout (clock.relayout = 2): every bin is laid out again from the start of the
// region, the wanted room shared out of the region's spare beyond the base capacities in
// proportion to the wants, and every particle is copied into the other buffer, which becomes
// current.  The region, n + n/8 + n/8 + (BIN_SLACK_MIN + BIN_ALIGN) nst slots, covers every base
// layout.
// The layout goes into generation clock.lgen (the clock advance switched to it).  When priming,
// the fills are set to the counts, which the placement then provides.  On a relayout the counts go
// to new_count, and every bin that moves gets its new fill here, and its particles go as pieces of
// at most MOVE_PIECE into the peak's list for the relayout copies.
__device__ __forceinline__ void layout_peak(const StepArgs& A, int pk, const PeakClock& C) {
  static_assert(LAYOUT_THREADS == 1024, "one lane per warp of the CTA");
  __shared__ u32 s_w[2][LAYOUT_THREADS / 32];
  __shared__ unsigned long long s_r[4][LAYOUT_THREADS / 32];
  __shared__ u32 s_moves;
  const PeakDesc& P = A.peaks[pk];
  const BinLayout* old = blay(A, C.lgen ^ 1) + P.st_base;
  BinLayout* lay = blay(A, C.lgen) + P.st_base;
  const BinFill* pushed = bfill(A, C.sbuf) + P.st_base;  // relayout: the buffer the push filled
  BinFill* cur = bfill(A, C.sbuf) + P.st_base;
  BinFill* nxt = bfill(A, C.sbuf ^ 1) + P.st_base;
  const u32* ss = A.sstart + P.sst_off;
  const u32* ovf_in = A.ovf_in + P.st_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // Count, base capacity and wanted extra capacity of bin i.
  auto bin = [&](int i, u32& cnt, u32& cap, u32& want) {
    want = 0u;
    u32 need = 0u;
    if (C.sortstep) {
      cnt = !A.sorted ? A.load_count[P.st_base + i] : ss[i + 1] >= ss[i] ? ss[i + 1] - ss[i] : 0u;
    } else {
      const u32 prev = min(pushed[i].gap, old[i].cap);  // the bin's count before the push
      cnt = bin_count(old[i], pushed[i]) + ovf_in[i];
      const u32 grow = cnt > prev ? cnt - prev : 0u;
      const unsigned long long nd =
          (unsigned long long)pushed[i].moved * BIN_ARRIVALS + (unsigned long long)grow * (unsigned)P.bin_grow;
      need = (u32)min(nd, (unsigned long long)P.n);
    }
    cnt = min(cnt, (u32)P.n);
    cap = (cnt + (P.bin_shift < 32 ? cnt >> P.bin_shift : 0u) + (u32)P.bin_min + BIN_ALIGN - 1) & ~(u32)(BIN_ALIGN - 1);
    if (P.bin_grow > 0 && need > cap - cnt) want = need - (cap - cnt);
  };
  // Whether a partial relayout moves bin i (new count cnt): it overflowed, or (with spare capacity
  // in use) its remaining room is below another step of its arrivals, so that its neighbours'
  // overflows do not relayout the peak again in the next steps.
  auto moves = [&](int i, u32 cnt) -> bool {
    if (ovf_in[i]) return true;
    if (P.bin_grow == 0) return false;
    const u32 room = old[i].cap > cnt ? old[i].cap - cnt : 0u;
    return (unsigned long long)room < (unsigned long long)pushed[i].moved * BIN_ARRIVALS;
  };
  // Capacity of a bin moved by a partial relayout: base capacity plus its want.
  auto moved_cap = [&](u32 cap, u32 want) -> u32 {
    return (u32)min((unsigned long long)cap + want + BIN_ALIGN - 1, (unsigned long long)P.r_size) &
           ~(u32)(BIN_ALIGN - 1);
  };
  // Relayout: the base capacities' total, the total want, the space the overflowed bins need when
  // moved, and the end of the last bin of the current layout; then partial or full.
  bool partial = false;
  unsigned long long spare = 0, want_tot = 0, tail = 0;
  if (C.relayout) {
    unsigned long long sc = 0, sg = 0, sp = 0, mt = 0;
    for (int i = threadIdx.x; i < P.nst; i += LAYOUT_THREADS) {
      u32 cnt, cap, want;
      bin(i, cnt, cap, want);
      sc += cap;
      sg += want;
      if (moves(i, cnt)) sp += moved_cap(cap, want);
      const unsigned long long e = (unsigned long long)old[i].base + old[i].cap - (unsigned long long)P.r_off;
      mt = e > mt ? e : mt;
    }
    for (int d = 16; d > 0; d >>= 1) {
      sc += __shfl_xor_sync(0xffffffffu, sc, d);
      sg += __shfl_xor_sync(0xffffffffu, sg, d);
      sp += __shfl_xor_sync(0xffffffffu, sp, d);
      const unsigned long long o = __shfl_xor_sync(0xffffffffu, mt, d);
      mt = o > mt ? o : mt;
    }
    if (lane == 0) {
      s_r[0][warp] = sc;
      s_r[1][warp] = sg;
      s_r[2][warp] = sp;
      s_r[3][warp] = mt;
    }
    __syncthreads();
    sc = sg = sp = mt = 0;
    for (int w = 0; w < LAYOUT_THREADS / 32; ++w) {
      sc += s_r[0][w];
      sg += s_r[1][w];
      sp += s_r[2][w];
      mt = s_r[3][w] > mt ? s_r[3][w] : mt;
    }
    tail = mt;
    partial = tail + sp <= (unsigned long long)P.r_size;
    if (!partial && P.bin_grow > 0) {
      spare = (long long)sc < P.r_size ? (unsigned long long)(P.r_size - (long long)sc) : 0ull;
      want_tot = sg;
    }
  }
  if (threadIdx.x == 0) s_moves = 0u;
  __syncthreads();
  bool bad = false;
  // The particles of bin i's old place as pieces to its new one, then its new fill.
  auto move = [&](int i, const BinLayout& to, u32 cnt) {
    const BinRuns R = bin_runs(old[i], pushed[i]);
    const int n = min(R.total(), (int)to.cap);
    const int n0 = min(R.n0, n);
    const u32 p0 = (u32)(n0 + MOVE_PIECE - 1) / MOVE_PIECE, p1 = (u32)(n - n0 + MOVE_PIECE - 1) / MOVE_PIECE;
    u32 q = atomicAdd(&s_moves, p0 + p1);
    if (!piece_fits(q, p0 + p1, piece_room(P.n, P.nst))) {  // more particles than the peak has: corrupted bins
      bad = true;
      return;
    }
    auto run = [&](int from, int end, long long src) {
      for (int k = from; k < end; k += MOVE_PIECE, ++q)
        A.moves[P.mv_off + q] = make_uint4((u32)(src + k), to.base + (u32)k, (u32)min(MOVE_PIECE, end - k), 0u);
    };
    run(0, n0, R.b0);
    run(n0, n, R.b1);
    cnt = min(cnt, to.cap);
    (partial ? cur : nxt)[i] = BinFill{cnt, cnt, 0u, 0u};  // a full relayout fills the other buffer
  };
  // One bin per thread and round, placed by a prefix sum over the CTA.  (Four consecutive bins per
  // thread, for fewer rounds, read the tables in 64-byte strides and took 1.4 times as long.)
  long long carry = partial ? (long long)tail : 0;
  for (int base = 0, round = 0; base < P.nst; base += LAYOUT_THREADS, round ^= 1) {
    const int i = base + threadIdx.x;
    u32 cnt = 0, cap = 0;
    if (i < P.nst) {
      u32 want;
      bin(i, cnt, cap, want);
      if (partial) {
        cap = moves(i, cnt) ? moved_cap(cap, want) : 0u;  // only the moved bins take new space
      } else if (want && want_tot) {  // the wanted extra, or its share of the spare
        const unsigned long long share = (unsigned long long)want * spare / want_tot;
        cap += (u32)(min(share, (unsigned long long)want) & ~(unsigned long long)(BIN_ALIGN - 1));
      }
    }
    u32 incl = cap;
    for (int d = 1; d < 32; d <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    if (lane == 31) s_w[round][warp] = incl;
    __syncthreads();
    u32 total = s_w[round][lane], before = lane < warp ? total : 0u;
    for (int d = 16; d > 0; d >>= 1) {
      before += __shfl_xor_sync(0xffffffffu, before, d);
      total += __shfl_xor_sync(0xffffffffu, total, d);
    }
    if (i < P.nst) {
      if (partial && cap == 0u) {
        lay[i] = old[i];  // not overflowed: stays where it is
      } else {
        long long b = carry + before + incl - cap;  // bin start inside the peak's region
        if (b + cap > P.r_size) {                   // counts above the particle total: never past the region
          bad = true;
          b = min(b, P.r_size);
          cap = (u32)(P.r_size - b);
          cnt = min(cnt, cap);
        }
        const BinLayout to{(u32)(P.r_off + b), cap};
        lay[i] = to;
        if (C.relayout) move(i, to, cnt);
      }
      if (C.sortstep) {
        cur[i] = BinFill{cnt, cnt, 0u, 0u};
        nxt[i] = BinFill{0u, 0u, 0u, 0u};
        A.ovf_in[P.st_base + i] = 0u;
        A.load_count[P.st_base + i] = 0u;  // ready for the next load
        A.new_count[P.st_base + i] = 0u;   // k_load_place counts it up
      } else {
        A.new_count[P.st_base + i] = cnt;
      }
    }
    carry += total;
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(&A.stats[pk].status, 4u);
  if (threadIdx.x == 0) {
    if (C.sortstep) A.ovf_n[pk] = 0u;
    if (C.relayout) {
      A.n_moves[pk] = pieces_published(s_moves, piece_room(P.n, P.nst));
      A.clocks[pk].relayout = partial ? 1 : 2;
      if (!partial) {  // the full relayout fills the other buffer, which becomes current
        A.clocks[pk].sbuf = C.sbuf ^ 1;
        A.plan[pk].flags ^= PLAN_SBUF;
        A.stats[pk].relayouts_full += 1u;
      }
    }
  }
}

// Layouts of the priming peaks (one CTA per peak; only in steps that prime).
__global__ void __launch_bounds__(LAYOUT_THREADS) k_layout(StepArgs A) {
  const int pk = blockIdx.x;
  const PeakClock C = A.clocks[pk];
  if (C.dep && C.sortstep) layout_peak(A, pk, C);
}

// ------------------------------------------------------------------------------------------
// Energy and momentum of a peak that was just pushed: the push partials give K and sum p at the
// positions' a, the previous step's Green partials give W at the same a (the grids were computed
// there).  The deposit's launch carries these CTAs beside its own, because nothing in the step
// waits for the result; what they need of the clock the push has put aside (pushed_a), since the
// clock has moved on by then.  Each CTA reduces a slice of the partials (about eight per thread for
// the engine's largest peak); the last one to finish (atomic ticket) merges the slices in slice
// order and updates the statistics.  All sums are compensated, every order fixed.  The
// Layzer-Irvine integral int K da advances by the trapezoid rule between samples.
__device__ __forceinline__ void energy_slice(const StepArgs& A, int pk, int sl, CSum& tot) {
  const PeakDesc& P = A.peaks[pk];
  __shared__ CSum s_w[ENERGY_THREADS / 32][5];
  CSum v[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) v[q] = CSum{0.0, 0.0};
  const long long t0 = (long long)P.nst * sl / A.eslices, t1 = (long long)P.nst * (sl + 1) / A.eslices;
  for (long long t = t0 + threadIdx.x; t < t1; t += ENERGY_THREADS) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double2 e = A.epart[(P.st_base + t) * 4 + q];
      csum_merge(v[q], CSum{e.x, e.y});
    }
  }
  // Green partials: one per warp of the kernel that multiplies by the Green's function.
  const long long g0 = P.nwpart * sl / A.eslices, g1 = P.nwpart * (sl + 1) / A.eslices;
  const double* wp = A.wpart + P.mode_base * (PM_THREADS / 32);
  for (long long t = g0 + threadIdx.x; t < g1; t += ENERGY_THREADS) csum_add(v[4], wp[t]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const CSum r = csum_warp(v[q]);
    if (lane == 0) s_w[warp][q] = r;
  }
  __syncthreads();
  if (threadIdx.x < 5) {
    CSum t = s_w[0][threadIdx.x];
    for (int w = 1; w < ENERGY_THREADS / 32; ++w) csum_merge(t, s_w[w][threadIdx.x]);
    tot = t;
  }
}

// The merged slices into the peak's statistics (one thread; s_tot: momentum (3), p^2, Green sum).
__device__ __forceinline__ void energy_stats(const StepArgs& A, int pk, double a, const double* s_tot) {
  const PeakDesc& P = A.peaks[pk];
  PeakStats& S = A.stats[pk];
  const double kin = P.m_part / (2.0 * a * a) * s_tot[3];
  const double pot = 0.5 * (3.0 * PM_H_I * PM_H_I / (8.0 * M_PI)) * P.dx * P.dx * P.dx * s_tot[4];
  if (S.nsamples == 0) {
    S.li_int = 0.0;
    S.li_e0 = a * (kin + pot);
  } else {
    S.li_int += 0.5 * (S.kin + kin) * (a - S.a_e);
  }
  S.a_e = a;
  S.mom[0] = P.m_part * s_tot[0];
  S.mom[1] = P.m_part * s_tot[1];
  S.mom[2] = P.m_part * s_tot[2];
  S.kin = kin;
  S.pot = pot;
  S.nsamples += 1;
}

__device__ __noinline__ void energy_cta(const StepArgs& A, int pk, int sl) {
  __shared__ u32 s_last;
  __shared__ double s_tot[5];
  const double a = A.pushed_a[pk];
  if (a < 0.0) return;  // not pushed
  CSum t;  // threads 0 to 4: the sum each merges
  energy_slice(A, pk, sl, t);
  if (A.eslices > 1) {
    if (threadIdx.x < 5) {
      A.eslice[((long long)pk * ENERGY_SLICES + sl) * 5 + threadIdx.x] = make_double2(t.s, t.c);
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&A.ecount[pk], 1u) == (u32)A.eslices - 1 ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x < 5) {
      t = CSum{0.0, 0.0};
      for (int q = 0; q < A.eslices; ++q) {
        const double2 e = __ldcg(A.eslice + ((long long)pk * ENERGY_SLICES + q) * 5 + threadIdx.x);
        csum_merge(t, CSum{e.x, e.y});
      }
    }
    if (threadIdx.x == 0) A.ecount[pk] = 0u;
  }
  if (threadIdx.x < 5) s_tot[threadIdx.x] = t.s + t.c;
  __syncthreads();
  if (threadIdx.x == 0) energy_stats(A, pk, a, s_tot);
}

// Clock advance of a peak (one thread): applies the step that the push just made, selects the next
// step size, whether this step primes by sort, relayouts (the push overflowed a bin) or re-sorts
// the super-tiles by cell, and whether the peak re-deposits.  A running peak's particles are now
// in the other bin buffer; one that relayouts switches to a new layout generation.  The gate
// words are raised here; the face fix-up, which runs after the kernels they gate, lowers them.
// Returns whether the peak relayouts.
__device__ __forceinline__ bool advance_clock(const StepArgs& A, int pk) {
  const PeakDesc& P = A.peaks[pk];
  PeakClock c = A.clocks[pk];
  const u64 max_fix = A.stats[pk].max_fix;  // (fetched with the clock, not after it)
  const u32 n_ovf = A.ovf_n[pk];
  int dep = 0;
  // Collapse detection on the deposit made by the previous step, i.e. of the positions at c.a.
  // This step's push has already moved a running peak on to c.a + c.da, so a stop takes
  // effect after the step is booked below: the next step applies its closing kick and ends.
  bool stop_now = false;
  if (c.has_delta && c.delta_collapse > 0 && c.a_collapse < 0 && c.state != PS_PRIME) {
    if ((double)max_fix / (double)PM_FIX_ONE / P.n_mean - 1.0 >= c.delta_collapse) {
      c.a_collapse = c.a;
      stop_now = c.stop_on_collapse && c.state == PS_RUN;
    }
  }
  const bool pushed = c.state == PS_RUN || c.state == PS_FINALIZE;
  const int ovf = pushed && n_ovf != 0u ? 1 : 0;
  switch (c.state) {
    case PS_PRIME:
      dep = 1;
      c.sortstep = 1;
      c.relayout = 0;
      c.refresh = 0;
      c.lgen ^= 1;
      c.kpend = 0.0;
      c.a_grid = c.a;
      c.has_delta = 1;
      c.state = c.mode == SCHED_EXPLICIT ? PS_HOLD : PS_RUN;
      break;
    case PS_RUN: {
      const double an = c.a + c.da;
      c.kpend = 0.5 / PM_H_I * c.da * sqrt(an);  // 0.5 da / (a H(a))
      c.a = an;
      c.a_grid = an;
      c.nsteps += 1;
      c.sortstep = 0;
      c.refresh = P.full_every > 0 && (c.nsteps % P.full_every) == 0 ? 1 : 0;
      dep = 1;
      if (c.mode == SCHED_RATIO) {
        if (c.nsteps >= c.max_steps) c.state = PS_FINALIZE;
        else c.da = c.a * c.param;
      } else if (c.mode == SCHED_FRAC) {
        if (c.a >= c.a_end) c.state = PS_FINALIZE;
        else c.da = fmin(c.param * c.a, c.a_end - c.a);
      } else {
        c.state = PS_HOLD;
      }
      if (stop_now && c.state == PS_RUN) c.state = PS_FINALIZE;
      break;
    }
    case PS_FINALIZE:
      c.kpend = 0.0;
      c.sortstep = 0;
      c.refresh = 0;
      dep = 1;
      c.state = PS_IDLE;
      break;
    default:
      break;
  }
  if (pushed) {  // the particles are now in the buffer the push wrote
    if (ovf) A.stats[pk].relayouts += 1u;
    c.relayout = ovf;
    c.sbuf ^= 1;
    if (ovf) c.lgen ^= 1;
  }
  c.dep = dep;
  A.clocks[pk] = c;
  A.plan[pk] = plan_of(c, P);
  A.sortseg[pk].active = dep && c.sortstep;
  if (dep) {
    A.stats[pk].max_fix = 0;
    A.stats[pk].mass_defect = 0;
    if (c.sortstep) atomicExch(A.sort_gate, 1u);
    if (c.relayout) atomicExch(A.layout_gate, 1u);
    if (c.refresh) atomicExch(A.refresh_gate, 1u);
  }
  return dep && c.relayout;
}

// One CTA per peak: its clock, then (when the push overflowed a bin) its new bin layout.
__global__ void __launch_bounds__(LAYOUT_THREADS) k_tick(const __grid_constant__ StepArgs A) {
  __shared__ int s_relayout;
  const int pk = blockIdx.x;
  pdl_wait();
  if (threadIdx.x == 0) s_relayout = advance_clock(A, pk);
  __syncthreads();
  if (s_relayout) layout_peak(A, pk, A.clocks[pk]);
}

// ------------------------------------------------------------------------------------------
// Priming (particles loaded into the loading area): counts per super-tile (k_load_count), the bin
// layout from them (k_layout), then every particle to the next free slot of its bin of the
// current buffer (k_load_place).  Nothing needs an order inside a bin, so 4 + 64 bytes per particle
// do.  A warp takes a 2 x 4 x 4 block of the lattice (load_index), whose nodes the patch strides of
// the push and the deposit put in distinct shared-memory banks; in the lattice's own order the
// push was 3.5 % slower afterwards.  At 256^3 the step that primes took 1617 us with the full radix
// sort of the cell keys, 737 with this; at 512^3 15.3 and 5.7 ms.
// An engine with a refresh period, whose bins are to be in cell order, primes by that sort
// instead: the Morton-key radix sort, the super-tile starts in the sorted keys, the layout, then
// the gather of the loading area into the bins in sorted order (so does one whose sort test hook
// is set).  All are grid-stride loops that return at once on the steps where no peak primes.

// Calls f(pk) for the peaks with pick(clock), in order, by a whole CTA of PM_THREADS: the clocks are
// read PM_THREADS at a time instead of one after the other.
template <class Pick, class F>
__device__ __forceinline__ void for_peaks(const StepArgs& A, Pick pick, F f) {
  __shared__ u32 s_mask[PM_THREADS / 32];
  for (int base = 0; base < A.npeaks; base += PM_THREADS) {
    const int i = base + threadIdx.x;
    const u32 m = __ballot_sync(0xffffffffu, i < A.npeaks && pick(A.clocks[i]));
    if ((threadIdx.x & 31) == 0) s_mask[threadIdx.x >> 5] = m;
    __syncthreads();
    for (int w = 0; w < PM_THREADS / 32; ++w)
      for (u32 b = s_mask[w]; b; b &= b - 1) f(base + 32 * w + __ffs(b) - 1);
    __syncthreads();
  }
}

// Place in the loading area of a warp's lane: the warp-th 2 x 4 x 4 block of an Np^3 lattice (Np a
// multiple of 4), else the warp-th 32 particles.
__device__ __forceinline__ long long load_index(const PeakDesc& P, long long warp, int lane) {
  if (!P.np4) return warp * 32 + lane;
  const u32 q = (u32)P.np4, w = (u32)warp, row = w / q, bz = w - row * q, bx = row / q, by = row - bx * q;
  return ((long long)(2 * bx + (lane >> 4)) * (4 * q) + 4 * by + ((lane >> 2) & 3)) * (4 * q) + 4 * bz + (lane & 3);
}

__global__ void __launch_bounds__(PM_THREADS) k_load_count(const __grid_constant__ StepArgs A) {
  if (*A.sort_gate == 0u) return;
  for_peaks(A, [](const PeakClock& c) { return c.dep && c.sortstep; }, [&](int pk) {
    const PeakDesc& P = A.peaks[pk];
    const long long n = P.n, nw = (n + 31) / 32;
    for (long long w = (long long)blockIdx.x * (PM_THREADS / 32) + (threadIdx.x >> 5); w < nw;
         w += (long long)gridDim.x * (PM_THREADS / 32)) {
      const long long j = load_index(P, w, threadIdx.x & 31);
      const u32 S = j < n ? min(A.keys_push[P.p_off + j] >> P.st_shift, (u32)(P.nst - 1)) : 0xffffffffu;
      const u32 peers = __match_any_sync(0xffffffffu, S);
      if (j < n && (peers & lanemask_lt()) == 0) atomicAdd(&A.load_count[P.st_base + S], (u32)__popc(peers));
    }
  });
}

__global__ void __launch_bounds__(PM_THREADS) k_load_place(const __grid_constant__ StepArgs A) {
  if (*A.sort_gate == 0u) return;
  for_peaks(A, [](const PeakClock& c) { return c.dep && c.sortstep; }, [&](int pk) {
    const PeakDesc& P = A.peaks[pk];
    const int sbuf = A.clocks[pk].sbuf;
    const BinLayout* lay = blay(A, A.clocks[pk].lgen);
    int4* opos = bpos(A, sbuf);
    float4* omom = bmom(A, sbuf);
    const long long n = P.n, nw = (n + 31) / 32;
    for (long long w = (long long)blockIdx.x * (PM_THREADS / 32) + (threadIdx.x >> 5); w < nw;
         w += (long long)gridDim.x * (PM_THREADS / 32)) {
      const long long j = load_index(P, w, threadIdx.x & 31);
      const bool v = j < n;
      const u32 S = v ? min(A.keys_push[P.p_off + j] >> P.st_shift, (u32)(P.nst - 1)) : 0xffffffffu;
      int4 ps;
      float4 m;
      if (v) {
        ps = A.lpos[P.p_off + j];
        m = A.lmom[P.p_off + j];
      }
      const u32 peers = __match_any_sync(0xffffffffu, S);
      const int leader = __ffs(peers) - 1;
      u32 r = 0;
      if (v && (int)(threadIdx.x & 31) == leader) r = atomicAdd(&A.new_count[P.st_base + S], (u32)__popc(peers));
      r = __shfl_sync(0xffffffffu, r, leader) + (u32)__popc(peers & lanemask_lt());
      if (!v) continue;
      const BinLayout L = lay[P.st_base + S];
      if (r >= L.cap) {  // counts that disagree: never write outside the bin
        atomicOr(&A.stats[pk].status, 4u);
        continue;
      }
      opos[L.base + r] = ps;
      omom[L.base + r] = m;
    }
  });
}

__global__ void k_st_starts(StepArgs A, long long ntot) {
  if (*A.sort_gate == 0u) return;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < ntot; j += (long long)gridDim.x * blockDim.x) {
    const int pk = pm_find(A.p_base, A.npeaks, j);
    const PeakClock C = A.clocks[pk];
    if (!(C.dep && C.sortstep)) continue;
    const PeakDesc P = A.peaks[pk];
    u32* ss = A.sstart + P.sst_off;
    // Super-tile of each sorted key; a key outside the peak's key range (a failed sort) is
    // clamped, so no start is ever written outside the peak's table.
    const u32 kb = A.keys_sorted[j] >> P.st_shift;
    if (kb >= (u32)P.nst) atomicOr(&A.stats[pk].status, 2u);
    const int b = (int)min(kb, (u32)(P.nst - 1));
    const int bprev = j == P.p_off ? -1 : (int)min(A.keys_sorted[j - 1] >> P.st_shift, (u32)(P.nst - 1));
    for (int bb = bprev + 1; bb <= b; ++bb) ss[bb] = (u32)j;
    if (j == P.p_off + P.n - 1)
      for (int bb = b + 1; bb <= P.nst; ++bb) ss[bb] = (u32)(P.p_off + P.n);
  }
}

__global__ void k_permute(StepArgs A, long long ntot) {
  if (*A.sort_gate == 0u) return;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < ntot; j += (long long)gridDim.x * blockDim.x) {
    const int pk = pm_find(A.p_base, A.npeaks, j);
    const PeakClock C = A.clocks[pk];
    if (!(C.dep && C.sortstep)) continue;
    const PeakDesc& P = A.peaks[pk];
    const u32 q = A.perm[j];
    const u32 S = min(A.keys_sorted[j] >> P.st_shift, (u32)(P.nst - 1));
    const BinLayout L = blay(A, C.lgen)[P.st_base + S];
    const long long r = j - (long long)A.sstart[P.sst_off + S];
    // A failed sort (a value outside the peak, a rank outside the bin): never read or write outside.
    if ((long long)q < P.p_off || (long long)q >= P.p_off + P.n || r < 0 || r >= (long long)L.cap) {
      atomicOr(&A.stats[pk].status, 2u);
      continue;
    }
    bpos(A, C.sbuf)[L.base + r] = A.lpos[q];
    bmom(A, C.sbuf)[L.base + r] = A.lmom[q];
  }
}

// Relayout copies of the peaks whose push overflowed a bin, a grid-stride loop that returns at once
// in the steps without one.  Full relayout (clock.relayout = 2): every bin is copied from the
// buffer the push filled to its place in the current buffer.  Partial (1): only the bins that got
// a new place after the last bin move there, inside the current buffer.  The list of pieces spreads
// a dense bin over many CTAs (one CTA per bin took 78 us a step through a 256^3 collapse, whose
// densest bins hold tens of thousands of particles; the pieces take 9).  Then each particle of the peak's
// overflow area goes to the end of its new bin (ovf_in counts down to zero, one rank per
// particle).  The two parts write disjoint slots and read nothing the other writes, so they need
// no order between them.
__global__ void __launch_bounds__(PM_THREADS) k_relayout(const __grid_constant__ StepArgs A) {
  pdl_wait();
  if (*A.layout_gate == 0u) return;
  for_peaks(A, [](const PeakClock& c) { return c.dep && c.relayout; }, [&](int pk) {
    const PeakClock& C = A.clocks[pk];
    const int kind = C.relayout, sbuf = C.sbuf, lgen = C.lgen;
    const PeakDesc& P = A.peaks[pk];
    const int src = kind == 2 ? (sbuf ^ 1) : sbuf;
    const int4* ip = bpos(A, src);
    const float4* im = bmom(A, src);
    int4* op = bpos(A, sbuf);
    float4* om = bmom(A, sbuf);
    const u32 nmv = min(A.n_moves[pk], (u32)piece_room(P.n, P.nst));
    for (u32 q = blockIdx.x; q < nmv; q += gridDim.x) {
      const uint4 mv = A.moves[P.mv_off + q];
      if (!piece_inside(mv.x, mv.y, mv.z, P.r_off, P.r_size)) {  // never outside the peak's bins
        if (threadIdx.x == 0) atomicOr(&A.stats[pk].status, 4u);
        continue;
      }
      static_assert(MOVE_PIECE % (4 * PM_THREADS) == 0, "four particles per thread and round");
      for (u32 k = threadIdx.x; k < mv.z; k += 4 * PM_THREADS) {  // old and new places never overlap
        int4 p[4];
        float4 m[4];
#pragma unroll
        for (int d = 0; d < 4; ++d)
          if (k + d * PM_THREADS < mv.z) {
            p[d] = ip[mv.x + k + d * PM_THREADS];
            m[d] = im[mv.x + k + d * PM_THREADS];
          }
#pragma unroll
        for (int d = 0; d < 4; ++d)
          if (k + d * PM_THREADS < mv.z) {
            op[mv.y + k + d * PM_THREADS] = p[d];
            om[mv.y + k + d * PM_THREADS] = m[d];
          }
      }
    }
    const long long novf = (long long)min(A.ovf_n[pk], (u32)P.n);
    for (long long o = (long long)blockIdx.x * PM_THREADS + threadIdx.x; o < novf;
         o += (long long)gridDim.x * PM_THREADS) {
      const long long j = P.p_off + o;
      const int4 ps = A.lpos[j];
      const int N = P.N, l2 = P.log2N, s = P.log2TS;
      const u32 S = pm_morton3(((ps.x >> (2 * l2)) & (N - 1)) >> s, ((ps.x >> l2) & (N - 1)) >> s, (ps.x & (N - 1)) >> s);
      const long long g = P.st_base + S;
      const BinLayout L = blay(A, lgen)[g];
      const u32 cnt = A.new_count[g];  // arrivals from the overflow area included
      const u32 v = atomicSub(&A.ovf_in[g], 1u);
      if (v == 0u || v > cnt || cnt > L.cap) {  // counts that disagree: never write outside the bin
        atomicOr(&A.stats[pk].status, 4u);
        continue;
      }
      bpos(A, sbuf)[L.base + cnt - v] = ps;
      bmom(A, sbuf)[L.base + cnt - v] = A.lmom[j];
    }
  });
}

// ------------------------------------------------------------------------------------------
// Refresh (optional, off by default): every full_every steps each super-tile's particles are
// re-sorted by cell (local
// Morton code of the cell inside the super-tile), so the deposit's and the push's warps see
// neighbouring cells and same-cell runs again, and the bin's two runs become one.  A counting
// sort per super-tile: the order inside one cell is not kept (nothing downstream depends on it;
// the deposit sums integers).  Up to TSORT_CAP particles the super-tile is staged in shared
// memory and written back to the start of its bin, coalesced (64 bytes of traffic per particle);
// denser super-tiles are copied to the same bin of the other buffer (free until the next push)
// and placed back from there.  Persistent grid (one CTA per SM) over the super-tiles; every
// launch returns at once when no peak refreshes this step.
template <int TS>
__device__ __forceinline__ void tile_sort(const StepArgs& A, const PeakDesc& P, const PeakClock& C, u32 st,
                                          unsigned char* smem) {
  constexpr int NCELL = TS * TS * TS;
  u32* hist = (u32*)smem;                                           // [NCELL], then its prefix
  int4* spos = (int4*)(smem + sizeof(u32) * 16 * 16 * 16);          // [TSORT_CAP]
  float4* smom = (float4*)(spos + TSORT_CAP);                       // [TSORT_CAP]
  u32* cr = (u32*)(smom + TSORT_CAP);                               // [TSORT_CAP] cell << 16 | rank
  unsigned short* inv = (unsigned short*)(cr + TSORT_CAP);          // [TSORT_CAP] slot -> particle
  __shared__ u32 s_wsum[TSORT_THREADS / 32];
  const long long g = P.st_base + st;
  const BinLayout L = blay(A, C.lgen)[g];
  BinFill* F = bfill(A, C.sbuf) + g;
  const BinRuns R = bin_runs(L, *F);
  const int n = R.total();
  int4* pos = bpos(A, C.sbuf);
  float4* mom = bmom(A, C.sbuf);
  int4* tpos = bpos(A, C.sbuf ^ 1);
  float4* tmom = bmom(A, C.sbuf ^ 1);
  const long long b = L.base;
  __syncthreads();  // every thread has read the fill before it is rewritten
  if (threadIdx.x == 0) *F = BinFill{(u32)n, (u32)n, 0u, 0u};  // one run from here on
  if (n < 2 && R.n0 == n) return;  // uniform: nothing to move
  const int N = P.N, l2 = P.log2N;
  const int sx = pm_compact3(st >> 2), sy = pm_compact3(st >> 1), sz = pm_compact3(st);
  // Local cell code; masked into the super-tile so a corrupted grouping cannot index outside.
  auto cell_of = [&](int c) -> u32 {
    const int ix = c >> (2 * l2), iy = (c >> l2) & (N - 1), iz = c & (N - 1);
    return pm_morton3((ix - sx * TS) & (TS - 1), (iy - sy * TS) & (TS - 1), (iz - sz * TS) & (TS - 1));
  };
  for (int i = threadIdx.x; i < NCELL; i += TSORT_THREADS) hist[i] = 0u;
  __syncthreads();
  const bool staged = n <= TSORT_CAP;
  if (staged) {
    for (int i = threadIdx.x; i < n; i += TSORT_THREADS) {
      const long long j = R.slot(i);
      const int4 p = pos[j];
      spos[i] = p;
      smom[i] = mom[j];
      const u32 c = cell_of(p.x);
      cr[i] = (c << 16) | atomicAdd(&hist[c], 1u);
    }
  } else {
    for (int i = threadIdx.x; i < n; i += TSORT_THREADS) {
      const long long j = R.slot(i);
      const int4 p = pos[j];
      tpos[b + i] = p;
      tmom[b + i] = mom[j];
      atomicAdd(&hist[cell_of(p.x)], 1u);
    }
  }
  __syncthreads();
  // Exclusive prefix of the cell counts (NCELL <= 4096 = 4 per thread).
  {
    constexpr int PER = (NCELL + TSORT_THREADS - 1) / TSORT_THREADS;
    u32 v[PER];
    u32 tot = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = threadIdx.x * PER + k;
      v[k] = i < NCELL ? hist[i] : 0u;
      tot += v[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u32 incl = tot;
    for (int d = 1; d < 32; d <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    u32 off = 0;
    for (int w = 0; w < warp; ++w) off += s_wsum[w];
    u32 run = off + incl - tot;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = threadIdx.x * PER + k;
      if (i < NCELL) hist[i] = run;
      run += v[k];
    }
  }
  __syncthreads();
  if (staged) {
    for (int i = threadIdx.x; i < n; i += TSORT_THREADS) {
      const u32 x = cr[i];
      inv[hist[x >> 16] + (x & 0xFFFFu)] = (unsigned short)i;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < n; o += TSORT_THREADS) {
      const int i = inv[o];
      pos[b + o] = spos[i];
      mom[b + o] = smom[i];
    }
  } else {
    // The copies in the other buffer are visible to the block after the barrier above; each
    // particle takes the next rank of its cell (order inside a cell arbitrary).
    for (int i = threadIdx.x; i < n; i += TSORT_THREADS) {
      const int4 p = tpos[b + i];
      const u32 o = atomicAdd(&hist[cell_of(p.x)], 1u);
      if (o < (u32)n) {
        pos[b + o] = p;
        mom[b + o] = tmom[b + i];
      }
    }
  }
  __syncthreads();  // shared arrays are reused by the next super-tile
}

__global__ void __launch_bounds__(TSORT_THREADS) k_tile_sort(StepArgs A, long long nst) {
  extern __shared__ __align__(16) unsigned char s_ts[];
  __shared__ int s_pk;
  pdl_wait();
  if (*A.refresh_gate == 0u) return;
  for (long long t = blockIdx.x; t < nst; t += gridDim.x) {
    if (threadIdx.x == 0) s_pk = pm_find(A.st_base, A.npeaks, t);
    __syncthreads();
    const int pk = s_pk;
    __syncthreads();
    const PeakClock C = A.clocks[pk];
    if (!(C.dep && C.refresh)) continue;
    const PeakDesc P = A.peaks[pk];
    const u32 st = (u32)(t - A.st_base[pk]);
    switch (P.TS) {
      case 4: tile_sort<4>(A, P, C, st, s_ts); break;
      case 8: tile_sort<8>(A, P, C, st, s_ts); break;
      default: tile_sort<16>(A, P, C, st, s_ts); break;
    }
  }
}

// ------------------------------------------------------------------------------------------
// Deterministic CIC deposit (pm3d.py:81-89, 103-104).  One CTA per super-tile deposits its own
// particles (one contiguous range) onto the (TS+1)^3 nodes they touch.  Per particle the 8 CIC
// weights are formed in 64-bit fixed point with 38 fractional bits, the 8th corner taking the
// remainder so each particle deposits exactly 2^38.  Each node accumulates in shared memory as two
// native 32-bit words (the signed weight's bits >= 19 and its low 19 bits), exact within a chunk
// of up to 8191 particles, and is folded into a 64-bit register accumulator after every chunk.
// Interior nodes are then final and written as FP32 delta = S/n_mean - 1; nodes on the three
// lower faces (which neighbours also reach) and on the upper halo (which belongs to the
// neighbours) are written as 64-bit partials.
//
// The face fix-up (k_fixup, the next launch) completes the face nodes: own partial plus the
// lower neighbours' halo partials.  (Engines of a few small meshes: see add_nodes.)
// Integer sums make the result independent of particle order, bit for bit; no float atomics.
__device__ __forceinline__ int face_index(int lx, int ly, int lz, int T) {
  if (lx == 0) return ly * T + lz;
  if (ly == 0) return T * T + (lx - 1) * T + lz;
  return T * T + (T - 1) * T + (lx - 1) * (T - 1) + (ly - 1);
}
__device__ __forceinline__ int halo_index(int lx, int ly, int lz, int T) {
  if (lx == T) return ly * (T + 1) + lz;
  if (ly == T) return (T + 1) * (T + 1) + lx * (T + 1) + lz;
  return (T + 1) * (T + 1) + T * (T + 1) + lx * T + ly;
}
// Finish the face nodes of super-tile Y (whole CTA of FIX_THREADS): each face node's own
// partial plus the halo partials of the lower neighbours Y - o, o = (ox, oy, oz) in {0,1}^3 \ 0,
// that reach it (node (lx + TS ox, ...) of the neighbour, which lies on its upper halo, for a
// face node with (lx, ly, lz) zero where o is one).  nb[o]: the neighbours' halo partials.
// Adds to the caller's statistics.
template <int TS>
__device__ __forceinline__ bool fixup_faces(const StepArgs& A, int pk, u32 Y, int only, double* rho64, long long& dsum,
                                            long long& smax) {
  // Where this super-tile's face partials and its lower neighbours' halo partials start: a table, so
  // that the partials are two memory round trips away (the kernel is bound by their latency) and
  // are on their way before the peak's plan has arrived.
  const long long* const ref = A.fix_ref + 8LL * blockIdx.x;
  const long long* const face = A.face + __ldg(ref);
  auto nb = [&](int o) { return A.halo + __ldg(ref + o); };
  // Three face nodes per thread, one of each face (x: TS x TS nodes; y: without lx = 0; z: without
  // lx = 0 and ly = 0), so that coordinates are shifts and the neighbours that reach a node are
  // known: always the face's own, the others only for edge and corner nodes.  All own partials and
  // first neighbours are loaded together.  Integer sums: the order does not change a bit.
  static_assert(TS * TS <= FIX_THREADS, "one node of each face per thread");
  const int u = threadIdx.x / TS, v = threadIdx.x % TS;
  const bool in = threadIdx.x < TS * TS, on[3] = {in, in && u > 0, in && u > 0 && v > 0};
  const int cx[3] = {0, u, u}, cy[3] = {u, 0, v}, cz[3] = {v, v, 0};
  long long S[3] = {0, 0, 0};
  constexpr int H1 = (TS + 1) * (TS + 1), H2 = H1 + TS * (TS + 1);  // starts of the y and z planes in the halo
  if (on[0]) S[0] = __ldcg(face + u * TS + v) + __ldcg(nb(1) + u * (TS + 1) + v);
  if (on[1]) S[1] = __ldcg(face + TS * TS + (u - 1) * TS + v) + __ldcg(nb(2) + H1 + u * (TS + 1) + v);
  if (on[2]) S[2] = __ldcg(face + TS * TS + (TS - 1) * TS + (u - 1) * (TS - 1) + v - 1) + __ldcg(nb(4) + H2 + u * TS + v);
  if (on[0] && u == 0) S[0] += __ldcg(nb(2) + H1 + v) + __ldcg(nb(3) + TS * (TS + 1) + v);
  if (on[0] && v == 0) S[0] += __ldcg(nb(4) + H2 + u) + __ldcg(nb(5) + u * (TS + 1) + TS);
  if (on[0] && u == 0 && v == 0) S[0] += __ldcg(nb(6) + H1 + TS) + __ldcg(nb(7) + TS * (TS + 1) + TS);
  if (on[1] && v == 0) S[1] += __ldcg(nb(4) + H2 + u * TS) + __ldcg(nb(6) + H1 + u * (TS + 1) + TS);
  const u32 flags = __ldcg(&A.plan[pk].flags);
  if (only < 0 ? !(flags & PLAN_DEP) : pk != only) return false;
  if (threadIdx.x == 0) {
    // Ready for the next push, which fills the other buffer: no arrivals yet, overflow area
    // empty.  (Here rather than in the deposit, whose particle loop is register-bound.)
    bfill(A, flags & PLAN_SBUF ? 0 : 1)[blockIdx.x].moved = 0u;
    if (Y == 0) {
      A.ovf_n[pk] = 0u;
      *A.sort_gate = *A.layout_gate = *A.refresh_gate = 0u;  // this step's gated kernels have run
    }
  }
  const PeakDesc& P = A.peaks[pk];
  const int N = P.N;
  const int sx = pm_compact3(Y >> 2), sy = pm_compact3(Y >> 1), sz = pm_compact3(Y);
  const long long nmf = P.n_mean_fix;
  const double inv = P.inv_fix_nmean;
  float* const delta = P.delta;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (!on[k]) continue;
    const long long Dv = S[k] - nmf;
    const long long node = ((long long)(sx * TS + cx[k]) * N + (sy * TS + cy[k])) * N + (sz * TS + cz[k]);
    delta[node] = (float)((double)Dv * inv);
    if (rho64) rho64[node] = (double)S[k] * (1.0 / (double)PM_FIX_ONE);
    dsum += Dv;
    smax = S[k] > smax ? S[k] : smax;
  }
  return true;
}

// Nearest integer to the exact product a*b for 0 <= a*b < 2^51: one FMA with 2^52 rounds the
// product to an integer in the mantissa (round half to even), whose low 52 bits are read off.
// The same rounding as __double2ll_rn of the exact product, on the FP64 pipe instead of the
// conversion unit.
__device__ __forceinline__ u64 fix_round(double a, double b) {
  return (u64)__double_as_longlong(fma(a, b, 4503599627370496.0)) & 0xFFFFFFFFFFFFFull;
}

// Shared-memory address of node number `node` (z fastest) of a (TS+1)^3 patch.
template <int TS>
__device__ __forceinline__ int dep_addr(int node) {
  constexpr int T1 = TS + 1;
  const int lx = node / (T1 * T1), r = node - lx * (T1 * T1), ly = r / T1, lz = r - ly * T1;
  return lx * patch_ps(TS) + ly * patch_rs(TS) + lz;
}
// A node's chunk sum S from its two accumulator words (see deposit_super): S lies within
// [2^19 hi - DEP_BIAS, 2^19 hi - DEP_BIAS + 2^32), and its low 32 bits are lo.
#define DEP_BIAS 32764u
__device__ __forceinline__ u32 chunk_rest(u32 hi, u32 lo) { return lo - (hi << 19) + DEP_BIAS; }
__device__ __forceinline__ long long chunk_sum(u32 hi, u32 lo) {
  return ((long long)hi << 19) + (long long)chunk_rest(hi, lo) - (long long)DEP_BIAS;
}

// Adds a full chunk's node sums into the fold scratch (first chunk: stores) and clears the
// chunk accumulators.  Kept out of line: it runs only for super-tiles of more than one chunk.
template <int TS>
__device__ __noinline__ void fold_chunk(u64* acc64, u32* acc_hi, u32* acc_lo, bool add) {
  constexpr int NN = (TS + 1) * (TS + 1) * (TS + 1);
  for (int node = threadIdx.x; node < NN; node += DEP_THREADS) {
    const int ad = dep_addr<TS>(node);
    acc64[node] = (add ? acc64[node] : 0ull) + (u64)chunk_sum(acc_hi[ad], acc_lo[ad]);
    acc_hi[ad] = 0u;
    acc_lo[ad] = 0u;
  }
}

// Engines of a few small meshes (PeakDesc::rho): all (TS+1)^3 node sums of a super-tile added to the
// mesh's grid of 64-bit sums, which the solve's first kernel turns into delta and clears
// (finish_nodes), so that no fix-up is launched: deposit and fix-up 13.7 -> 10.8 us at 32^3, 17.4 ->
// 12.7 at 64^3, against 2 and 1 more in the solve.  Integer adds: the same sums in any order.  Out of
// line: the particle loop is register-bound.
template <int TS>
__device__ __noinline__ void add_nodes(const u32* acc_hi, const u32* acc_lo, const u64* fold, u64* rho, int x0, int y0,
                                       int z0, int l2) {
  constexpr int T1 = TS + 1, RS = patch_rs(TS), PS = patch_ps(TS);
  const int m = (1 << l2) - 1;
  for (int node = threadIdx.x; node < T1 * T1 * T1; node += DEP_THREADS) {
    const int lx = node / (T1 * T1), r = node - lx * (T1 * T1), ly = r / T1, lz = r - ly * T1;
    const int ad = lx * PS + ly * RS + lz;
    long long S = chunk_sum(acc_hi[ad], acc_lo[ad]);
    if (fold) S += (long long)fold[node];
    if (S) atomicAdd(rho + (((((x0 + lx) & m) << l2 | ((y0 + ly) & m)) << l2) | ((z0 + lz) & m)), (u64)S);
  }
}

// One corner weight W (the nearest integer of a product in units of 2^-38, 0 <= W < 2^39, see
// fix_round): W >> 19, and W modulo 2^32.  The FMA's result has the bits 0x4330000000000000 + W, so
// the first is one funnel shift of its two words (the exponent bits shift out) and the second its
// low word as it is.
struct Split {
  u32 hi, lo;
};
__device__ __forceinline__ Split fix_split(double a, double b) {
  const double r = fma(a, b, 4503599627370496.0);
  const u32 wl = (u32)__double2loint(r), wh = (u32)__double2hiint(r);
  return Split{__funnelshift_r(wl, wh, 19), wl};
}

// The nodes of a super-tile itself out of the accumulators: delta of interior nodes, partials of
// face nodes; dsum and smax: the sum of S - n_mean_fix and the largest S over the interior nodes.
// GENERAL: 64-bit integers throughout, with the sums of folded chunks and the float64 counts.
// Otherwise (one chunk, n_mean < 2^10) S - n_mean_fix is formed in FP64, exactly: both accumulator
// words are brought in by bit construction (2^52 + word) and one FMA joins them, so that the
// conversion to FP32 delta is the same as from the integer; sums of up to TS^3 such terms of one
// chunk stay below 2^53.
template <int TS, bool GENERAL>
__device__ __forceinline__ void write_nodes(const u32* acc_hi, const u32* acc_lo, const u64* fold, float* delta,
                                            double* rho64, long long* face, int N, long long nmf, double inv,
                                            long long& dsum, long long& smax) {
  constexpr int RS = patch_rs(TS), PS = patch_ps(TS), G4 = TS / 4, T1 = TS + 1;
  const double c_lo = 4503599627370496.0 + (double)((long long)DEP_BIAS + nmf);  // exact below 2^53
  long long isum = 0, imax = 0;
  double fsum = 0.0, fmaxd = -9007199254740992.0;
  for (int item = threadIdx.x; item < TS * TS * G4; item += DEP_THREADS) {
    const int g = item % G4, ly = (item / G4) % TS, lx = item / (G4 * TS);
    const int ad = lx * PS + ly * RS + 4 * g;
    const uint4 h = *reinterpret_cast<const uint4*>(acc_hi + ad);
    const uint4 l = *reinterpret_cast<const uint4*>(acc_lo + ad);
    const u32 hv[4] = {h.x, h.y, h.z, h.w}, lv[4] = {l.x, l.y, l.z, l.w};
    const bool row_face = lx == 0 || ly == 0;
    if (row_face || g == 0) {
      const int nf = row_face ? 4 : 1;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < nf) {
          long long S = chunk_sum(hv[k], lv[k]);
          if (GENERAL && fold) S += (long long)fold[(lx * T1 + ly) * T1 + 4 * g + k];
          face[face_index(lx, ly, 4 * g + k, TS)] = S;
        }
    }
    if (row_face) continue;
    float4 d;
    float* dv = &d.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (GENERAL) {
        long long S = chunk_sum(hv[k], lv[k]);
        if (fold) S += (long long)fold[(lx * T1 + ly) * T1 + 4 * g + k];
        const long long D = S - nmf;
        dv[k] = (float)((double)D * inv);
        if (g > 0 || k > 0) {
          isum += D;
          imax = S > imax ? S : imax;
          if (rho64) rho64[((long long)lx * N + ly) * N + 4 * g + k] = (double)S * (1.0 / (double)PM_FIX_ONE);
        }
      } else {
        const double hd = __hiloint2double(0x43300000, (int)hv[k]) - 4503599627370496.0;
        const double ld = __hiloint2double(0x43300000, (int)chunk_rest(hv[k], lv[k])) - c_lo;
        const double D = fma(hd, 524288.0, ld);
        dv[k] = (float)(D * inv);
        if (k > 0 || g > 0) {
          fsum += D;
          fmaxd = D > fmaxd ? D : fmaxd;
        }
      }
    }
    *reinterpret_cast<float4*>(delta + ((long long)lx * N + ly) * N + 4 * g) = d;
  }
  if (GENERAL) {
    dsum = isum;
    smax = imax;
  } else {
    dsum = (long long)fsum;
    const long long m = (long long)fmaxd + nmf;
    smax = m > 0 ? m : 0;
  }
}

template <int TS, int SB>
__device__ __forceinline__ void deposit_super(const StepArgs& A, const PeakDesc& P, int pk, u32 st,
                                              const BinLayout& L, const BinFill& F, u32* smem, double* rho64) {
  constexpr int T1 = TS + 1, NN = T1 * T1 * T1;
  constexpr int RS = patch_rs(TS), PS = patch_ps(TS), SZ = patch_size(TS);
  constexpr int FC = TS * TS * TS - (TS - 1) * (TS - 1) * (TS - 1);
  static_assert(RS % 4 == 0 && PS % 4 == 0, "patch rows are read 16 bytes at a time");
  u32* acc_hi = smem;
  u32* acc_lo = smem + SZ;
  __shared__ long long s_red[DEP_THREADS / 32];
  __shared__ long long s_max[DEP_THREADS / 32];
  const int N = P.N, l2 = P.log2N;
  const int sx = pm_compact3(st >> 2), sy = pm_compact3(st >> 1), sz = pm_compact3(st);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const BinRuns R = bin_runs(L, F);
  // A cell index belongs to this super-tile iff its bits outside the local ones equal the
  // super-tile's: one mask and one compare (negative or out-of-mesh values never match).
  const int local = ((TS - 1) << (2 * l2)) | ((TS - 1) << l2) | (TS - 1);
  const int tile_bits = ((sx * TS) << (2 * l2)) | ((sy * TS) << l2) | (sz * TS);
  __syncthreads();
  // Nodes' sums of the chunks folded so far, only for a super-tile of more than one chunk: kept
  // in the same bin of the other buffer (free until the next push; a bin of more than one chunk
  // of 16-byte entries holds the NN 8-byte sums several times over).
  static_assert((8191 / DEP_THREADS) * DEP_THREADS * sizeof(int4) >= NN * sizeof(u64), "fold scratch too small");
  bool folded = false;
  // Two accumulator words per node.  A weight W (at most 2^38) adds W >> 19 to hi and W to lo
  // modulo 2^32; the eighth corner, whose weight is the remainder 2^38 - (the other seven), adds
  // the hi of its own product, which the remainder differs from by less than 4.  A node takes at
  // most one contribution per particle of a chunk of n <= 8191 particles, so hi stays below 2^32,
  // and the node's sum S differs from 2^19 hi by more than -4 n >= -DEP_BIAS and less than
  // n (2^19 + 4) <= 2^32 - DEP_BIAS: S is the one value in that interval whose low 32 bits are lo.
  // Exact, and neither word needs a mask or a carry (the split into two 19-bit fields that this
  // replaced took 14 more integer instructions per particle).  A typical super-tile (about TS^3
  // particles) is a single chunk.
  constexpr int CH_IT = 8191 / DEP_THREADS;  // sweeps of DEP_THREADS particles per chunk
  static_assert(CH_IT >= 1 && CH_IT * DEP_THREADS <= 8191, "chunk too large for the split accumulators");
  static_assert(PM_FIX_BITS == 38, "the two accumulator words assume 38 fractional bits");
  static_assert(CH_IT * DEP_THREADS * 4 <= (int)DEP_BIAS, "bias of the interval");
  // 32-bit indices inside the bin's two runs (fewer integer instructions and live registers than
  // 64-bit pointers): particle k sits at pp[k] in the first run, at pp[k + d1] in the second.
  const int4* __restrict__ pp = (SB ? A.pos1 : A.pos0) + R.b0;
  const int n = R.total(), n0 = R.n0, d1 = (int)(R.b1 - R.b0);
  u64* const fold = reinterpret_cast<u64*>((SB ? A.pos0 : A.pos1) + L.base);
  if (threadIdx.x == 0) {
    prefetch_l2(pp, n0);
    prefetch_l2(pp + n0 + d1, n - n0);
  }
  bool bad = false;
  for (int c0 = 0; c0 < n; c0 += CH_IT * DEP_THREADS) {  // chunks; almost always one
    if (c0) {  // fold the chunk before into `fold`
      __syncthreads();
      fold_chunk<TS>(fold, acc_hi, acc_lo, folded);
      folded = true;
      __syncthreads();
    }
    const int c1 = min(n, c0 + CH_IT * DEP_THREADS);
    auto add = [&](const int4& ps) {
      const int c = ps.x;
      const double one = (double)PM_FIX_ONE;
      const double fx = __int_as_float(ps.y), fy = __int_as_float(ps.z), fz = __int_as_float(ps.w);
      const double Fx = fx * one, Gx = one - Fx;   // exact: fx has 24 significant bits
      const double gy = 1.0 - fy, gz = 1.0 - fz;
      const double w00 = Gx * gy, w01 = Gx * fy, w10 = Fx * gy, w11 = Fx * fy;
      // Seven corners rounded to integers in units of 2^-38; the eighth takes the remainder so
      // the particle deposits exactly 2^38 (0 modulo 2^32).
      Split w[8] = {fix_split(w00, gz), fix_split(w00, fz), fix_split(w01, gz), fix_split(w01, fz),
                    fix_split(w10, gz), fix_split(w10, fz), fix_split(w11, gz), fix_split(w11, fz)};
      w[7].lo = 0u - (w[0].lo + w[1].lo + w[2].lo + w[3].lo + w[4].lo + w[5].lo + w[6].lo);
      if ((c & ~local) == tile_bits) {
        const int nb = ((c >> (2 * l2)) & (TS - 1)) * PS + ((c >> l2) & (TS - 1)) * RS + (c & (TS - 1));
        const int off[8] = {0, 1, RS, RS + 1, PS, PS + 1, PS + RS, PS + RS + 1};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          atomicAdd(&acc_hi[nb + off[q]], w[q].hi);
          atomicAdd(&acc_lo[nb + off[q]], w[q].lo);
        }
      } else {
        bad = true;
      }
    };
    // Two sweeps per round, the next two sweeps' loads in flight meanwhile, and two rounds unrolled:
    // one sweep per round took 192 instructions per particle and 134 us at 256^3, this 160 and 123.
    int k = c0 + threadIdx.x;
    int4 na = make_int4(0, 0, 0, 0), nb = na;
    if (k < c1) na = pp[k < n0 ? k : k + d1];
    if (k + DEP_THREADS < c1) nb = pp[k + DEP_THREADS < n0 ? k + DEP_THREADS : k + DEP_THREADS + d1];
#pragma unroll 2
    while (k < c1) {
      const int4 pa = na, pb = nb;
      const bool two = k + DEP_THREADS < c1;
      k += 2 * DEP_THREADS;
      if (k < c1) na = pp[k < n0 ? k : k + d1];
      if (k + DEP_THREADS < c1) nb = pp[k + DEP_THREADS < n0 ? k + DEP_THREADS : k + DEP_THREADS + d1];
      add(pa);
      if (two) add(pb);
    }
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(&A.stats[pk].status, 1u);
  if (P.rho && !rho64) {
    add_nodes<TS>(acc_hi, acc_lo, folded ? fold : nullptr, P.rho, sx * TS, sy * TS, sz * TS, l2);
    return;
  }
  // Write-out of the last chunk (plus the folded ones).  First the TS^3 nodes of the super-tile,
  // four of a row at a time: interior nodes final as FP32 delta (16-byte stores; the first node
  // of an interior row is a face node, stored here from this super-tile's own sum and completed by
  // k_fixup), nodes on the lower faces as 64-bit partials; then the upper halo, partials in their
  // storage order.
  const long long gbase = ((long long)sx * TS * N + (long long)sy * TS) * N + sz * TS;
  long long* face = A.face + P.face_off + (long long)st * FC;
  long long* halo = A.halo + P.halo_off + (long long)st * P.hc;
  const long long nmf = P.n_mean_fix;
  const double inv = P.inv_fix_nmean;
  long long dsum, smax;
  if (folded || rho64 || nmf >= (1LL << 48))
    write_nodes<TS, true>(acc_hi, acc_lo, folded ? fold : nullptr, P.delta + gbase, rho64 ? rho64 + gbase : nullptr,
                          face, N, nmf, inv, dsum, smax);
  else
    write_nodes<TS, false>(acc_hi, acc_lo, nullptr, P.delta + gbase, nullptr, face, N, nmf, inv, dsum, smax);
  {
    // The three upper planes: their TS x TS parts with coordinates from shifts, then the 3 TS + 1
    // nodes of their common edges.
    auto put = [&](int lx, int ly, int lz) {
      const int ad = lx * PS + ly * RS + lz;
      long long S = chunk_sum(acc_hi[ad], acc_lo[ad]);
      if (folded) S += (long long)fold[(lx * T1 + ly) * T1 + lz];
      halo[halo_index(lx, ly, lz, TS)] = S;
    };
    for (int f = threadIdx.x; f < TS * TS; f += DEP_THREADS) {
      const int u = f / TS, v = f % TS;
      put(TS, u, v);
      put(u, TS, v);
      put(u, v, TS);
    }
    for (int f = threadIdx.x; f < 3 * TS + 1; f += DEP_THREADS) {
      const int e = f / TS, u = f % TS;  // e = 3: the corner
      put(e == 0 ? u : TS, e == 1 ? u : TS, e == 2 ? u : TS);
    }
  }
  for (int d = 16; d > 0; d >>= 1) {
    dsum += __shfl_xor_sync(0xffffffffu, dsum, d);
    const long long om = __shfl_xor_sync(0xffffffffu, smax, d);
    smax = om > smax ? om : smax;
  }
  if (lane == 0) {
    s_red[warp] = dsum;
    s_max[warp] = smax;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long ts = 0, tm = 0;
    for (int w = 0; w < DEP_THREADS / 32; ++w) {
      ts += s_red[w];
      tm = s_max[w] > tm ? s_max[w] : tm;
    }
    atomicAdd((unsigned long long*)&A.stats[pk].mass_defect, (unsigned long long)ts);
    atomicMax(&A.stats[pk].max_fix, (u64)tm);
  }
}


__global__ void __launch_bounds__(DEP_THREADS, 4)
    k_deposit(const __grid_constant__ StepArgs A, double* rho64, int only, int necta) {
  extern __shared__ __align__(16) u32 s_dep[];
  if ((int)blockIdx.x < necta) {  // the energies' CTAs (in front, so that they start at once)
    pdl_wait();
    energy_cta(A, (int)blockIdx.x / A.eslices, (int)blockIdx.x % A.eslices);
    return;
  }
  const int tile = (int)blockIdx.x - necta;
  const TileRef tr = find_tile(A.st_ref, tile);
  const PeakDesc P = A.peaks[tr.pk];
  {  // clear the accumulators
    const int words = 2 * (tr.TS == 4 ? patch_size(4) : tr.TS == 8 ? patch_size(8) : patch_size(16));
    static_assert((2 * patch_size(4)) % 4 == 0 && (2 * patch_size(8)) % 4 == 0 && (2 * patch_size(16)) % 4 == 0, "");
    for (int i = threadIdx.x; i < words / 4; i += DEP_THREADS)
      reinterpret_cast<uint4*>(s_dep)[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  pdl_wait();
  // The plan and both candidates of the bin's layout and fill in one round trip (as in k_push).
  const u32 flags = __ldcg(&A.plan[tr.pk].flags);
  const int4 F0 = __ldcg(reinterpret_cast<const int4*>(A.fill[0] + tile)),
             F1 = __ldcg(reinterpret_cast<const int4*>(A.fill[1] + tile));
  const int2 L0 = __ldcg(reinterpret_cast<const int2*>(A.lay[0] + tile)),
             L1 = __ldcg(reinterpret_cast<const int2*>(A.lay[1] + tile));
  const bool sb = flags & PLAN_SBUF;
  const int4 f = sb ? F1 : F0;
  const int2 l = flags & PLAN_LGEN ? L1 : L0;
  const BinFill F{(u32)f.x, (u32)f.y, (u32)f.z, 0u};
  const BinLayout L{(u32)l.x, (u32)l.y};
  if (only < 0 ? !(flags & PLAN_DEP) : tr.pk != only) return;
  const u32 st = (u32)tr.t;
  switch (P.TS) {
    // The bin buffer as a template argument: its pointers are then kernel parameters, not a
    // per-thread select (the particle loop is register-bound).
    case 4:
      if (sb) deposit_super<4, 1>(A, P, tr.pk, st, L, F, s_dep, rho64);
      else deposit_super<4, 0>(A, P, tr.pk, st, L, F, s_dep, rho64);
      break;
    case 8:
      if (sb) deposit_super<8, 1>(A, P, tr.pk, st, L, F, s_dep, rho64);
      else deposit_super<8, 0>(A, P, tr.pk, st, L, F, s_dep, rho64);
      break;
    default:
      if (sb) deposit_super<16, 1>(A, P, tr.pk, st, L, F, s_dep, rho64);
      else deposit_super<16, 0>(A, P, tr.pk, st, L, F, s_dep, rho64);
      break;
  }
}

// Face fix-up: one CTA per super-tile whose peak deposited this step.  Small and
// latency-bound, so many CTAs per SM.
__global__ void __launch_bounds__(FIX_THREADS) k_fixup(const __grid_constant__ StepArgs A, double* rho64, int only) {
  __shared__ long long s_red[FIX_THREADS / 32];
  __shared__ long long s_max[FIX_THREADS / 32];
  const TileRef tr = find_tile(A.st_ref, blockIdx.x);
  pdl_wait();
  long long dsum = 0, smax = 0;
  const bool active = tr.TS == 4   ? fixup_faces<4>(A, tr.pk, (u32)tr.t, only, rho64, dsum, smax)
                      : tr.TS == 8 ? fixup_faces<8>(A, tr.pk, (u32)tr.t, only, rho64, dsum, smax)
                                   : fixup_faces<16>(A, tr.pk, (u32)tr.t, only, rho64, dsum, smax);
  if (!active) return;  // the whole CTA
  for (int d = 16; d > 0; d >>= 1) {
    dsum += __shfl_xor_sync(0xffffffffu, dsum, d);
    const long long om = __shfl_xor_sync(0xffffffffu, smax, d);
    smax = om > smax ? om : smax;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    s_red[warp] = dsum;
    s_max[warp] = smax;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long ts = 0, tm = 0;
    for (int w = 0; w < FIX_THREADS / 32; ++w) {
      ts += s_red[w];
      tm = s_max[w] > tm ? s_max[w] : tm;
    }
    atomicAdd((unsigned long long*)&A.stats[tr.pk].mass_defect, (unsigned long long)ts);
    atomicMax(&A.stats[tr.pk].max_fix, (u64)tm);
  }
}

// ------------------------------------------------------------------------------------------
// Green's function and gradient in k-space (pm3d.py:105-112): for every mode
//   Phi_k = -(3/2) H_i^2 delta_k / (a k^2) [* exp(-k^2 (smooth dx)^2 / 2)],  Phi_0 = 0,
//   G_i   = -i k_i Phi_k / N^3    (the 1/N^3 of numpy's inverse transform),
// written as three spectra for one batched C2R.  numpy's irfftn keeps the Nyquist
// wavenumbers (-pi/dx) and, in the kz = 0 and kz = N/2 planes, uses only the Hermitian part
// of its input (it takes the real part after the two complex inverse transforms).  Those two
// planes are therefore written as (G(k) + conj G(-k))/2, which any correct C2R turns into
// exactly numpy's field.
__device__ __forceinline__ float kline(int i, int N, float kf) { return kf * (float)(i < N / 2 ? i : i - N); }

// Gradient operator in k-space: spectral -i k (the reference), or the transfer function of the
// 2-point / 4-point central differences.
__device__ __forceinline__ float grad_k(float k, float dx, int mode) {
  if (mode == 1) return sinf(k * dx) / dx;
  if (mode == 2) return (8.0f * sinf(k * dx) - sinf(2.0f * k * dx)) / (6.0f * dx);
  return k;
}

// Per-peak constants of the Green kernel, read once into registers.
struct GreenCtx {
  int N, log2N, Nh, gm;
  long long M;
  u32 nh_magic;
  int nh_shift;
  float kf, dx, sd2, s_c;
  const float2* spec;
  float2* out;
};

__device__ __forceinline__ double green_mode(const GreenCtx& g, long long m, float2 d) {
  const int N = g.N, Nh = g.Nh;
  // m = row * Nh + kz (m < N^2 Nh < 2^32 for N <= 1024): division by the invariant Nh.
  const u32 rest = pm_div_by((u32)m, g.nh_magic, g.nh_shift);
  const int kz = (int)((u32)m - rest * (u32)Nh);
  const int iy = (int)(rest & (N - 1)), ix = (int)(rest >> g.log2N);
  const float kx = kline(ix, N, g.kf), ky = kline(iy, N, g.kf), kzv = g.kf * (float)kz;
  const float k2 = kx * kx + ky * ky + kzv * kzv;
  const long long M = g.M;
  if (m == 0) {
    g.out[0] = g.out[M] = g.out[2 * M] = make_float2(0.f, 0.f);
    return 0.0;
  }
  float G = g.s_c / k2;
  if (g.sd2 > 0.f) G *= expf(-0.5f * k2 * g.sd2);
  const float gx = grad_k(kx, g.dx, g.gm) * G, gy = grad_k(ky, g.dx, g.gm) * G, gz = grad_k(kzv, g.dx, g.gm) * G;
  // -i k G d = (k G d.y, -k G d.x)
  float2 ox = make_float2(gx * d.y, -gx * d.x), oy = make_float2(gy * d.y, -gy * d.x),
         oz = make_float2(gz * d.y, -gz * d.x);
  if (kz == 0 || kz == N / 2) {
    const int px = (-ix) & (N - 1), py = (-iy) & (N - 1);
    const float2 dp = g.spec[((long long)px * N + py) * Nh + kz];
    const float hx = grad_k(kline(px, N, g.kf), g.dx, g.gm) * G, hy = grad_k(kline(py, N, g.kf), g.dx, g.gm) * G;
    // (v + conj(v_partner)) / 2 with v_partner = (h dp.y, -h dp.x)
    ox = make_float2(0.5f * (ox.x + hx * dp.y), 0.5f * (ox.y + hx * dp.x));
    oy = make_float2(0.5f * (oy.x + hy * dp.y), 0.5f * (oy.y + hy * dp.x));
    oz = make_float2(0.5f * (oz.x + gz * dp.y), 0.5f * (oz.y + gz * dp.x));
  }
  g.out[m] = ox;
  g.out[M + m] = oy;
  g.out[2 * M + m] = oz;
  // Potential-energy term: sum_x delta Phi = sum_k |delta_k|^2 G_k over the full spectrum; the
  // half spectrum counts each kz in (0, N/2) twice.
  // The term in FP32 (relative rounding ~1e-7, independent from mode to mode), summed in FP64.
  const float wk = (kz == 0 || kz == N / 2) ? 1.0f : 2.0f;
  return (double)(wk * G * (d.x * d.x + d.y * d.y));
}

// Grid: the Green blocks of the peaks in A.green_peak (those without the native transform).
__global__ void __launch_bounds__(PM_THREADS) k_green(StepArgs A) {
  __shared__ int s_pk;
  __shared__ long long s_lb;
  pdl_wait();
  if (threadIdx.x == 0) {
    const int gi = pm_find(A.green_base, A.ngreen, (long long)blockIdx.x);
    s_pk = A.green_peak[gi];
    s_lb = (long long)blockIdx.x - A.green_base[gi];
  }
  __syncthreads();
  const int pk = s_pk;
  const long long lb = s_lb;  // block within the peak
  const PeakClock& C = A.clocks[pk];
  if (!C.has_delta) return;
  const PeakDesc& P = A.peaks[pk];
  GreenCtx g;
  g.N = P.N;
  g.log2N = P.log2N;
  g.Nh = P.N / 2 + 1;
  g.gm = P.gradient;
  g.M = P.nmodes;
  g.nh_magic = P.nh_magic;
  g.nh_shift = P.nh_shift;
  g.kf = (float)(kTwoPi / P.L);
  g.dx = (float)P.dx;
  g.sd2 = P.smooth > 0 ? (float)(P.smooth * P.dx) * (float)(P.smooth * P.dx) : 0.f;
  g.s_c = (float)(-1.5 * PM_H_I * PM_H_I / C.a_grid / ((double)P.N * P.N * P.N));
  g.spec = P.spec;
  g.out = P.gspec;
  const long long m0 = lb * (PM_THREADS * GREEN_MODES) + threadIdx.x;
  // All loads of the block's modes first (the stores below could alias them as far as the
  // compiler knows), then the arithmetic and the stores.
  float2 d[GREEN_MODES];
#pragma unroll
  for (int k = 0; k < GREEN_MODES; ++k) {
    const long long m = m0 + k * PM_THREADS;
    d[k] = m < g.M ? __ldg(g.spec + m) : make_float2(0.f, 0.f);
  }
  double w = 0.0;
#pragma unroll
  for (int k = 0; k < GREEN_MODES; ++k) {
    const long long m = m0 + k * PM_THREADS;
    if (m < g.M) w += green_mode(g, m, d[k]);
  }
  // Within a warp a plain FP64 tree (128 terms); one partial per warp, no block barrier; the
  // energy kernel merges the partials with the compensated sum.
  for (int dd = 16; dd > 0; dd >>= 1) w += __shfl_down_sync(0xffffffffu, w, dd);
  if ((threadIdx.x & 31) == 0) A.wpart[(P.mode_base + lb) * (PM_THREADS / 32) + (threadIdx.x >> 5)] = w;
}

__global__ void k_reset_peak(StepArgs A, int pk, double a0, int mode, double param, double a_end, int max_steps,
                             int set_thr, double delta_collapse, int stop) {
  PeakClock c = A.clocks[pk];
  c.a = a0;
  c.a_grid = a0;
  c.kpend = 0.0;
  c.mode = mode;
  c.param = param;
  c.a_end = a_end;
  c.max_steps = max_steps;
  c.nsteps = 0;
  c.state = PS_PRIME;
  c.has_delta = 0;
  c.dep = 0;
  c.sortstep = 0;
  c.refresh = 0;
  c.a_collapse = -1.0;
  c.stop_on_collapse = set_thr ? (stop ? 1 : 0) : 0;
  if (set_thr) c.delta_collapse = delta_collapse;
  if (mode == SCHED_RATIO) c.da = a0 * param;
  else if (mode == SCHED_FRAC) c.da = fmin(param * a0, a_end - a0);
  else c.da = 0.0;
  A.clocks[pk] = c;
  A.plan[pk] = plan_of(c, A.peaks[pk]);
  A.stats[pk].status = 0;
  A.stats[pk].nsamples = 0;
  A.stats[pk].relayouts = 0;
  A.stats[pk].relayouts_full = 0;
  A.sort_err[pk] = 0;
}

__global__ void k_release_peak(StepArgs A, int pk) {
  PeakClock c = A.clocks[pk];
  c.state = PS_IDLE;
  c.has_delta = 0;
  c.dep = 0;
  c.kpend = 0.0;
  A.clocks[pk] = c;
  A.plan[pk] = plan_of(c, A.peaks[pk]);
}

__global__ void k_tables(const PeakDesc* peaks, const long long* st_base, int npeaks, long long nst, int2* st_ref,
                         long long* fix_ref) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nst) return;
  const int pk = pm_find(st_base, npeaks, g);
  const PeakDesc& P = peaks[pk];
  const u32 t = (u32)(g - st_base[pk]), m = (u32)P.NS - 1;
  const u32 sx = pm_compact3(t >> 2), sy = pm_compact3(t >> 1), sz = pm_compact3(t);
  st_ref[g] = make_int2(pk | P.TS << 16, (int)t);
  fix_ref[8 * g] = P.face_off + (long long)t * P.fc;
  for (u32 o = 1; o < 8; ++o)
    fix_ref[8 * g + o] =
        P.halo_off + (long long)pm_morton3((sx - (o & 1)) & m, (sy - ((o >> 1) & 1)) & m, (sz - (o >> 2)) & m) * P.hc;
}

// A held peak's next explicit step.
__global__ void k_begin_step(StepArgs A, int pk, double da) {
  PeakClock c = A.clocks[pk];
  c.mode = SCHED_EXPLICIT;
  c.da = da;
  c.state = PS_RUN;
  A.clocks[pk] = c;
  A.plan[pk] = plan_of(c, A.peaks[pk]);
}

__global__ void k_write_clock(StepArgs A, int pk, PeakClock c) {
  A.clocks[pk] = c;
  A.plan[pk] = plan_of(c, A.peaks[pk]);
}

// Particles (n,3) float64 in lattice order -> split state + cell keys (pm3d.py:76-79 convention).
__global__ void k_set_particles(StepArgs A, int pk, PeakDesc P, const double* __restrict__ x,
                                const double* __restrict__ p) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  int ii[3];
  float ff[3];
  for (int d = 0; d < 3; ++d) {
    const double g = x[3 * i + d] / P.dx - 0.5;
    const double fl = floor(g);
    long long c = (long long)fl;
    float f = (float)(g - fl);
    if (f >= 1.0f) {
      f = 0.0f;
      c += 1;
    }
    ii[d] = (int)(((c % P.N) + P.N) % P.N);
    ff[d] = f;
  }
  const int cell = (ii[0] << (2 * P.log2N)) | (ii[1] << P.log2N) | ii[2];
  const long long g = P.p_off + i;
  // Loaded into the loading area in lattice order; the priming step sorts it into bins.
  A.lpos[g] = make_int4(cell, __float_as_int(ff[0]), __float_as_int(ff[1]), __float_as_int(ff[2]));
  A.lmom[g] = make_float4((float)p[3 * i], (float)p[3 * i + 1], (float)p[3 * i + 2], __int_as_float((int)i));
  A.keys_push[g] = pm_cell_key(ii[0], ii[1], ii[2]);
}

// Re-priming an existing state: copy it back to the loading area with its sort keys.  One CTA
// per super-tile of the peak; places in the loading area from a per-peak counter (ovf_n, zeroed
// by the host before the launch; the priming step zeroes it again), one add per warp.
__global__ void __launch_bounds__(PM_THREADS) k_reload(StepArgs A, int pk, PeakDesc P) {
  const PeakClock C = A.clocks[pk];
  const long long g = P.st_base + blockIdx.x;
  const BinRuns R = bin_runs(blay(A, C.lgen)[g], bfill(A, C.sbuf)[g]);
  const int4* ip = bpos(A, C.sbuf);
  const float4* im = bmom(A, C.sbuf);
  const int N = P.N, l2 = P.log2N;
  const int n = R.total();
  for (int base = 0; base < n; base += PM_THREADS) {  // uniform trip count: the ballot sees whole warps
    const int k = base + threadIdx.x;
    const bool v = k < n;
    const u32 vm = __ballot_sync(0xffffffffu, v);
    u32 o0 = 0;
    if ((threadIdx.x & 31) == 0 && vm) o0 = atomicAdd(&A.ovf_n[pk], (u32)__popc(vm));
    o0 = __shfl_sync(0xffffffffu, o0, 0);
    if (!v) continue;
    const u32 o = o0 + (u32)__popc(vm & lanemask_lt());
    if (o >= (u32)P.n) {
      atomicOr(&A.stats[pk].status, 4u);
      continue;
    }
    const long long j = R.slot(k);
    const int4 ps = ip[j];
    A.lpos[P.p_off + o] = ps;
    A.lmom[P.p_off + o] = im[j];
    A.keys_push[P.p_off + o] = pm_cell_key((ps.x >> (2 * l2)) & (N - 1), (ps.x >> l2) & (N - 1), ps.x & (N - 1));
  }
}

// Current state -> float64 x, p (lattice order).  p includes the pending closing kick; acc
// (optional) receives -grad Phi at the particles evaluated for expansion factor a_acc.  One CTA
// per super-tile of the peak walks its bin; a peak loaded but not yet primed has its particles in
// the loading area instead, where CTA t takes the t-th slice.
//
// What a particle's output rows are made of.  id: its row, -1 when there is none.
struct ReadRow {
  int id, ii[3];
  float f[3], mv[3];
  double g[3];
};
__device__ __forceinline__ ReadRow read_row(const StepArgs& A, int pk, const PeakDesc& P, bool valid, bool need_g, int4 ps,
                                            float4 m) {
  const int N = P.N;
  ReadRow r{valid ? __float_as_int(m.w) : -1,
            {(ps.x >> (2 * P.log2N)) & (N - 1), (ps.x >> P.log2N) & (N - 1), ps.x & (N - 1)},
            {__int_as_float(ps.y), __int_as_float(ps.z), __int_as_float(ps.w)},
            {m.x, m.y, m.z},
            {0.0, 0.0, 0.0}};
  if (valid && (r.id < 0 || r.id >= P.n)) {  // never write through an id that is not a lattice index
    atomicOr(&A.stats[pk].status, 8u);
    r.id = -1;
  }
  if (need_g && r.id >= 0) {
    const long long N3 = (long long)N * N * N;
    for (int c = 0; c < 8; ++c) {
      const int cx = c >> 2, cy = (c >> 1) & 1, cz = c & 1;
      const float w = (cx ? r.f[0] : 1.0f - r.f[0]) * (cy ? r.f[1] : 1.0f - r.f[1]) * (cz ? r.f[2] : 1.0f - r.f[2]);
      const long long o =
          ((long long)((r.ii[0] + cx) & (N - 1)) * N + ((r.ii[1] + cy) & (N - 1))) * N + ((r.ii[2] + cz) & (N - 1));
      r.g[0] += w * P.force[o];
      r.g[1] += w * P.force[N3 + o];
      r.g[2] += w * P.force[2 * N3 + o];
    }
  }
  return r;
}
__device__ __forceinline__ double row_x(const PeakDesc& P, const ReadRow& r, int d) {
  const double X = ((double)r.ii[d] + (double)r.f[d] + 0.5) * P.dx;
  return X >= P.L ? X - P.L : X;
}
// kick: the pending closing kick for forces of unit expansion factor; scale: the forces' factor.
struct ReadScale {
  double kick, scale;
  bool need_g;
};
__device__ __forceinline__ ReadScale read_scale(const PeakClock& C, const double* p, const double* acc, double a_acc) {
  const bool kick = p && C.kpend != 0.0;
  return ReadScale{kick ? C.kpend * (C.a_grid / C.a) : 0.0, acc ? C.a_grid / a_acc : 0.0, C.has_delta && (kick || acc)};
}

// One particle, its lane writing the rows.
__device__ __forceinline__ void get_one(const StepArgs& A, int pk, const PeakDesc& P, const ReadScale& S, int4 ps, float4 m,
                                        double* __restrict__ x, double* __restrict__ p, double* __restrict__ acc) {
  const ReadRow r = read_row(A, pk, P, true, S.need_g, ps, m);
  if (r.id < 0) return;
  const long long o = 3LL * r.id;
  for (int d = 0; d < 3; ++d) {
    if (x) x[o + d] = row_x(P, r, d);
    if (p) p[o + d] = (double)r.mv[d] + S.kick * r.g[d];
    if (acc) acc[o + d] = r.g[d] * S.scale;
  }
}

// A warp takes 32 particles (`valid` lanes) and writes their 24-byte rows of each output through
// `row` (96 doubles of shared memory per warp), eight bytes per lane in the rows' own order: a
// bin's neighbours are lattice neighbours, so this covers whole sectors, where one row per lane and
// one column at a time touched each of them three times (256^3: 679 -> 303 us, 658 -> 507
// with a pending kick, whose gather from the force grids then dominates).  STAGED false: each lane writes
// its own row (see k_get_particles).
template <bool STAGED>
__device__ __forceinline__ void get_warp(const StepArgs& A, int pk, const PeakDesc& P, const ReadScale& S, bool valid,
                                         int4 ps, float4 m, double* row, double* __restrict__ x,
                                         double* __restrict__ p, double* __restrict__ acc) {
  const int lane = threadIdx.x & 31;
  const ReadRow r = read_row(A, pk, P, valid, S.need_g, ps, m);
  auto put = [&](double* __restrict__ out, const double (&v)[3]) {
    if (!STAGED) {
      if (r.id >= 0)
        for (int d = 0; d < 3; ++d) out[3LL * r.id + d] = v[d];
      return;
    }
    __syncwarp();
    for (int d = 0; d < 3; ++d) row[3 * lane + d] = v[d];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int e = 32 * k + lane, q = e / 3;
      const int to = __shfl_sync(0xffffffffu, r.id, q);
      if (to >= 0) out[3LL * to + (e - 3 * q)] = row[e];
    }
  };
  double v[3];
  if (x) {
    for (int d = 0; d < 3; ++d) v[d] = row_x(P, r, d);
    put(x, v);
  }
  if (p) {
    for (int d = 0; d < 3; ++d) v[d] = (double)r.mv[d] + S.kick * r.g[d];
    put(p, v);
  }
  if (acc) {
    for (int d = 0; d < 3; ++d) v[d] = r.g[d] * S.scale;
    put(acc, v);
  }
}

// DENSE: bins of more than a few warps (READ_MEAN particles in the mean).  Many such bins share the
// memory system, and their rows go through shared memory.  A bin denser than READ_DENSE times the mean,
// and each of a few (READ_BINS), is alone with its CTA's latency, where lanes that write their own rows are
// faster.  us with own and staged rows: 262144 particles in one bin 569 and 724, in 1/1000 of a 64^3 mesh
// 568 and 722, eight bins of 32768 107 and 121; 512 bins of 1728 56 and 44, 256^3 483 and 349.  Smaller bins
// (a 128^3 mesh of 4^3 super-tiles, 64 particles each) need many CTAs on an SM: 48 registers and no shared
// memory 116, own rows in the larger kernel 129, staged 132.
#define READ_DENSE 32
#define READ_BINS 128
#define READ_MEAN 128
template <bool DENSE>
__global__ void __launch_bounds__(PM_THREADS) k_get_particles(StepArgs A, int pk, PeakDesc P, double* __restrict__ x,
                                                              double* __restrict__ p, double* __restrict__ acc,
                                                              double a_acc) {
  __shared__ double s_row[DENSE ? PM_THREADS * 3 : 1];
  double* const row = s_row + (DENSE ? (threadIdx.x >> 5) * 96 : 0);
  const int lane = threadIdx.x & 31;
  const PeakClock C = A.clocks[pk];
  const ReadScale S = read_scale(C, p, acc, a_acc);
  if (C.state == PS_PRIME) {  // still in the loading area
    const long long per = (P.n + P.nst - 1) / P.nst, i0 = per * blockIdx.x, i1 = min(P.n, i0 + per);
    for (long long i = i0 + threadIdx.x; i - (DENSE ? lane : 0) < i1; i += PM_THREADS) {
      const bool v = !DENSE || i < i1;
      const long long j = P.p_off + (v ? i : i0);
      if (DENSE) get_warp<true>(A, pk, P, S, v, A.lpos[j], A.lmom[j], row, x, p, acc);
      else get_one(A, pk, P, S, A.lpos[j], A.lmom[j], x, p, acc);
    }
    return;
  }
  const long long g = P.st_base + blockIdx.x;
  const BinRuns R = bin_runs(blay(A, C.lgen)[g], bfill(A, C.sbuf)[g]);
  const int4* ip = bpos(A, C.sbuf);
  const float4* im = bmom(A, C.sbuf);
  const int n = R.total();
  if (DENSE && P.nst >= READ_BINS && (long long)n * P.nst <= READ_DENSE * P.n) {
    for (int k = threadIdx.x; k - lane < n; k += PM_THREADS) {
      const bool v = k < n;
      const long long j = R.slot(v ? k : 0);
      get_warp<true>(A, pk, P, S, v, ip[j], im[j], row, x, p, acc);
    }
  } else {
    for (int k = threadIdx.x; k < n; k += PM_THREADS) {
      const long long j = R.slot(k);
      if (DENSE) get_warp<false>(A, pk, P, S, true, ip[j], im[j], row, x, p, acc);
      else get_one(A, pk, P, S, ip[j], im[j], x, p, acc);
    }
  }
}

// Reference-exact float64 CIC gather of an arbitrary field (pm3d.py:91-99).
__global__ void k_interp64(const double* __restrict__ F, const double* __restrict__ X, long long n, int N, double dx,
                           double* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  long long i0[3], i1[3];
  double f[3];
  for (int d = 0; d < 3; ++d) {
    const double g = X[3 * i + d] / dx - 0.5;
    const double fl = floor(g);
    const long long c = (long long)fl;
    f[d] = g - fl;
    i0[d] = ((c % N) + N) % N;
    i1[d] = (((c + 1) % N) + N) % N;
  }
  double s = 0.0;
  for (int c = 0; c < 8; ++c) {
    const int cx = c >> 2, cy = (c >> 1) & 1, cz = c & 1;
    const long long o = ((cx ? i1[0] : i0[0]) * N + (cy ? i1[1] : i0[1])) * N + (cz ? i1[2] : i0[2]);
    s += F[o] * ((cx ? f[0] : 1.0 - f[0]) * (cy ? f[1] : 1.0 - f[1]) * (cz ? f[2] : 1.0 - f[2]));
  }
  out[i] = s;
}

// CIC counts of arbitrary float64 positions (pm3d.py:81-89) without an engine: per particle the
// eight corner weights in 64-bit fixed point (38 fractional bits, the eighth corner taking the
// remainder, as in the engine's deposit) added with integer atomics, so the sums do not depend
// on the order; then k_fix_counts turns them into float64 counts.
__global__ void k_deposit64(const double* __restrict__ X, long long n, int N, double dx, u64* __restrict__ work) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  long long i0[3], i1[3];
  double f[3];
  for (int d = 0; d < 3; ++d) {
    const double g = X[3 * i + d] / dx - 0.5;
    const double fl = floor(g);
    const long long c = (long long)fl;
    f[d] = g - fl;
    i0[d] = ((c % N) + N) % N;
    i1[d] = (((c + 1) % N) + N) % N;
  }
  const double one = (double)PM_FIX_ONE;
  const double Fx = f[0] * one, Gx = one - Fx, gy = 1.0 - f[1], gz = 1.0 - f[2];
  const double pl[4] = {Gx * gy, Gx * f[1], Fx * gy, Fx * f[1]};
  u64 w[8], sum = 0;
  for (int c = 0; c < 7; ++c) {
    w[c] = fix_round(pl[c >> 1], (c & 1) ? f[2] : gz);
    sum += w[c];
  }
  w[7] = PM_FIX_ONE - sum;
  for (int c = 0; c < 8; ++c) {
    const int cx = c >> 2, cy = (c >> 1) & 1, cz = c & 1;
    const long long o = ((cx ? i1[0] : i0[0]) * N + (cy ? i1[1] : i0[1])) * N + (cz ? i1[2] : i0[2]);
    atomicAdd((unsigned long long*)&work[o], (unsigned long long)w[c]);
  }
}

__global__ void k_fix_counts(const u64* __restrict__ work, long long n3, double* __restrict__ counts) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) counts[i] = (double)(long long)work[i] * (1.0 / (double)PM_FIX_ONE);
}

}  // namespace

// Dynamic shared memory of the largest super-tile in use (the smaller ones fit inside).
size_t pm_deposit_smem(int TSmax) { return sizeof(u32) * 2 * (size_t)patch_size(TSmax); }
size_t pm_push_smem(int TSmax) { return sizeof(float) * 3 * (size_t)patch_size(TSmax); }

size_t pm_tile_sort_smem() {
  return sizeof(u32) * 16 * 16 * 16 + (size_t)TSORT_CAP * (sizeof(int4) + sizeof(float4) + sizeof(u32) + sizeof(unsigned short));
}

int pm_kernels_init() {
  cudaError_t e =
      cudaFuncSetAttribute(k_push<PUSH_THREADS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_deposit, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_tile_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pm_tile_sort_smem());
  return e == cudaSuccess ? 0 : -(int)e;
}

static unsigned nb(long long n, int t) { return (unsigned)((n + t - 1) / t); }

static int num_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      sms = 148;
  }
  return sms;
}

// Grid of a grid-stride kernel: enough CTAs to fill every SM `per_sm` times, fewer for small n.
static unsigned stride_grid(long long n, int t, int per_sm) {
  const long long g = std::min<long long>((long long)nb(n, t), (long long)num_sms() * per_sm);
  return (unsigned)std::max<long long>(g, 1);
}

// Threads of a push CTA when no super-tile is larger than 8^3 cells.  Narrow CTAs let more super-tiles
// reside at once, and 512 particles are then several sweeps whose loads overlap; wide ones take a
// dense super-tile (collapse, many particles per cell) in fewer sweeps.  So wide ones where all reside
// at once anyway (1024 threads an SM) and the particles fill them.  us a step with 128, 256, 512 threads:
// 64 super-tiles (one 32^3 peak) 28.8, 26.9, 27.0, of 64 particles 27.0, 27.0, 29.0, of 4096 46.0, 40.3,
// 39.3, of 32768 257, 190, 167; 512 (one 64^3 peak) 37.5, 37.1, 42.3 or, on another GPU, 37.7, 39.4, -, of 4096
// 88.9, 85.8, 89.4; 1024 (two 64^3 peaks) 47.2, 49.3, 55.6; 4096 (a 128^3 mesh of 8^3 super-tiles) 137, 145,
// 175.  What stays is that a cloud in a few of many super-tiles waits for its 128 threads: a 64^3 peak
// in collapse (maximum density contrast 450) 65.5, 57.1, 55.1; 2e6 particles in 2 % of the side of a 128^3
// box 25.7 ms, 16.0 with 512.
static int push_threads(long long nst, long long ntot) {
  const long long sms = num_sms();
  if (nst <= 2 * sms) return ntot >= 512 * nst ? 512 : 256;
  return nst <= 4 * sms && ntot >= 2048 * nst ? 256 : 128;
}
void launch_push(const StepArgs& A, long long nst, long long ntot, size_t smem, cudaStream_t s) {
  const dim3 grid((unsigned)nst);
  if (smem > pm_push_smem(8)) {
    pdl_launch(k_push<PUSH_THREADS, true>, grid, PUSH_THREADS, smem, s, A);
    return;
  }
  switch (push_threads(nst, ntot)) {
    case 512: pdl_launch(k_push<512, false>, grid, 512, smem, s, A); break;
    case 256: pdl_launch(k_push<256, false>, grid, 256, smem, s, A); break;
    default: pdl_launch(k_push<128, false>, grid, 128, smem, s, A); break;
  }
}
void launch_tick(const StepArgs& A, cudaStream_t s) {
  pdl_launch(k_tick, dim3(A.npeaks), LAYOUT_THREADS, 0, s, A);
}
void launch_load_count(const StepArgs& A, long long ntot, cudaStream_t s) {
  k_load_count<<<stride_grid(ntot, PM_THREADS, 8), PM_THREADS, 0, s>>>(A);
}
void launch_load_place(const StepArgs& A, long long ntot, cudaStream_t s) {
  k_load_place<<<stride_grid(ntot, PM_THREADS, 8), PM_THREADS, 0, s>>>(A);
}
void launch_permute(const StepArgs& A, long long ntot, cudaStream_t s) {
  k_permute<<<stride_grid(ntot, PM_THREADS, 8), PM_THREADS, 0, s>>>(A, ntot);
}
void launch_st_starts(const StepArgs& A, long long ntot, cudaStream_t s) {
  k_st_starts<<<stride_grid(ntot, PM_THREADS, 8), PM_THREADS, 0, s>>>(A, ntot);
}
void launch_tile_sort(const StepArgs& A, long long nst, cudaStream_t s) {
  pdl_launch(k_tile_sort, dim3(stride_grid(nst, 1, 1)), TSORT_THREADS, pm_tile_sort_smem(), s, A, nst);
}
void launch_layout(const StepArgs& A, cudaStream_t s) { k_layout<<<(unsigned)A.npeaks, LAYOUT_THREADS, 0, s>>>(A); }
void launch_relayout(const StepArgs& A, long long ntot, cudaStream_t s) {
  pdl_launch(k_relayout, dim3(stride_grid(ntot, MOVE_PIECE, RELAYOUT_CTAS_PER_SM)), PM_THREADS, 0, s, A);
}
void launch_deposit(const StepArgs& A, long long nst, size_t smem, double* rho64, int only, cudaStream_t s) {
  const int necta = only < 0 ? A.npeaks * A.eslices : 0;
  pdl_launch(k_deposit, dim3((unsigned)(nst + necta)), DEP_THREADS, smem, s, A, rho64, only, necta);
}
void launch_fixup(const StepArgs& A, long long nst, double* rho64, int only, cudaStream_t s) {
  pdl_launch(k_fixup, dim3((unsigned)nst), FIX_THREADS, 0, s, A, rho64, only);
}
void launch_green(const StepArgs& A, long long nblocks, cudaStream_t s) {
  pdl_launch(k_green, dim3((unsigned)nblocks), PM_THREADS, 0, s, A);
}
void launch_reset_peak(const StepArgs& A, int pk, double a0, int mode, double param, double a_end,
                       int max_steps, int set_thr, double delta_collapse, int stop, cudaStream_t s) {
  k_reset_peak<<<1, 1, 0, s>>>(A, pk, a0, mode, param, a_end, max_steps, set_thr, delta_collapse, stop);
}
void launch_tables(const PeakDesc* peaks, const long long* st_base, int npeaks, long long nst, int2* st_ref,
                   long long* fix_ref, cudaStream_t s) {
  k_tables<<<nb(nst, PM_THREADS), PM_THREADS, 0, s>>>(peaks, st_base, npeaks, nst, st_ref, fix_ref);
}
void launch_begin_step(const StepArgs& A, int pk, double da, cudaStream_t s) { k_begin_step<<<1, 1, 0, s>>>(A, pk, da); }
void launch_write_clock(const StepArgs& A, int pk, const PeakClock& c, cudaStream_t s) {
  k_write_clock<<<1, 1, 0, s>>>(A, pk, c);
}
void launch_release_peak(const StepArgs& A, int pk, cudaStream_t s) { k_release_peak<<<1, 1, 0, s>>>(A, pk); }
void launch_set_particles(const StepArgs& A, int pk, const PeakDesc& P, const double* x, const double* p,
                          cudaStream_t s) {
  k_set_particles<<<nb(P.n, PM_THREADS), PM_THREADS, 0, s>>>(A, pk, P, x, p);
}
void launch_reload(const StepArgs& A, int pk, const PeakDesc& P, cudaStream_t s) {
  cudaMemsetAsync(A.ovf_n + pk, 0, sizeof(u32), s);
  k_reload<<<(unsigned)P.nst, PM_THREADS, 0, s>>>(A, pk, P);
}
void launch_get_particles(const StepArgs& A, int pk, const PeakDesc& P, double* x, double* p, double* acc,
                          double a_acc, cudaStream_t s) {
  auto* kernel = P.n >= (long long)READ_MEAN * P.nst ? k_get_particles<true> : k_get_particles<false>;
  kernel<<<(unsigned)P.nst, PM_THREADS, 0, s>>>(A, pk, P, x, p, acc, a_acc);
}
void launch_interp64(const double* F, const double* X, long long n, int N, double dx, double* out, cudaStream_t s) {
  k_interp64<<<nb(n, PM_THREADS), PM_THREADS, 0, s>>>(F, X, n, N, dx, out);
}
void launch_deposit64(const double* X, long long n, int N, double dx, u64* work, double* counts, cudaStream_t s) {
  const long long n3 = (long long)N * N * N;
  cudaMemsetAsync(work, 0, sizeof(u64) * (size_t)n3, s);
  if (n > 0) k_deposit64<<<nb(n, PM_THREADS), PM_THREADS, 0, s>>>(X, n, N, dx, work);
  k_fix_counts<<<nb(n3, PM_THREADS), PM_THREADS, 0, s>>>(work, n3, counts);
}

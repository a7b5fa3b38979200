// Kernels of one PM step (pbhgr/pbhgr/pm3d.py:101-129) over a batch of peaks.
//
// Particles live in bins, one per super-tile (TS^3 cells), in two bin buffers that alternate
// every step.  Both buffers share a bin layout: super-tile S of a peak owns slots
// [base[S], base[S] + cap[S]) of each buffer, with spare capacity (an eighth of its count plus
// 32, and room for further growth after a relayout, set whenever the layout is made).  A filled bin holds two runs: the particles that stayed
// in S, from base[S] up, and the particles that arrived from other super-tiles, from
// base[S] + (the bin's count before the step) up (BinFill).  One step:
//   push       per super-tile: CIC gather of the forces, kicks, drift; each particle appended
//              to the bin of the super-tile it is now in, in the other buffer (stayers ranked in
//              shared memory, arrivals by an atomic on the destination's count); a particle
//              for which the destination bin has no room goes to the peak's overflow area
//   tick       per peak: the clock; a peak whose push overflowed gets a new layout and the list of
//              pieces to move
//   relayout   gated: those pieces, and the overflow area, into the buffer the push read (with a
//              refresh period each super-tile's particles are then re-sorted by cell)
//   deposit    per super-tile: CIC density of its particles into (TS+1)^3 nodes; interior nodes
//              final, face and upper-halo nodes as 64-bit partials.  In front of its grid the
//              energy CTAs: momentum, kinetic and potential energy, Layzer-Irvine integral
//   fixup      per super-tile: face nodes = own partial + the lower neighbours' halo partials
//   solve      delta -> three force grids (native_fft.cu; other sizes: cuFFT and k_green)
// A step that primes a peak places its loaded particles before the relayout (k_load_count, k_layout,
// k_load_place; with a refresh period a full Morton-key radix sort and a permutation).
// Engines of a few small meshes have no fixup: the deposit adds every node sum to a grid
// (NODE_SUMS_MAX_CELLS).
#pragma once
#include "common.cuh"
#include "sort.cuh"

#define PM_THREADS 256
#define PUSH_THREADS 512
#define DEP_THREADS 256    // deposit CTA (4 per SM)
#define GREEN_MODES 4      // modes per thread of the Green kernel (a block covers PM_THREADS * GREEN_MODES)
// Most cells of an engine whose deposit adds its node sums to the meshes (PeakDesc::rho) instead of
// leaving face partials to a fix-up launch.  Per step, fix-up and sums: 30.8 and 28.9 us for one
// 32^3 peak, 41.0 and 37.0 for eight, 39.2 and 37.0-39.0 for one of 64^3, 51.3 and 47.3 for two
// (2^19 cells), 72.1 and 72.1 for four, 117.6 and 121.5 for eight: the sums' 16 bytes per cell and
// wider loads then cost more than the launch that they save.  At 128^3: 109 and 123.
#define NODE_SUMS_MAX_CELLS (1LL << 19)
#define ENERGY_SLICES 128  // most CTAs per peak of the energy reduction
#define ENERGY_THREADS DEP_THREADS  // they ride in the deposit's launch
#define FIX_THREADS 256    // face fix-up CTA
#define TSORT_THREADS 1024 // super-tile sort (refresh) CTA
#define TSORT_CAP 5120     // particles of a super-tile sorted in shared memory; denser ones via global
// Bin capacities: count + (count >> BIN_SLACK_SHIFT) + BIN_SLACK_MIN, rounded up to BIN_ALIGN;
// a relayout adds room for BIN_ARRIVALS times the arrivals of the step plus BIN_GROW_STEPS times
// its net growth, out of a further (n >> BIN_SPARE_SHIFT) slots of the peak's bin region.
#ifndef BIN_SLACK_SHIFT
#define BIN_SLACK_SHIFT 3
#endif
#ifndef BIN_SPARE_SHIFT
#define BIN_SPARE_SHIFT 3
#endif
#ifndef BIN_ARRIVALS
#define BIN_ARRIVALS 1
#endif
#ifndef BIN_GROW_STEPS
#define BIN_GROW_STEPS 4
#endif
#define BIN_SLACK_MIN 32
#define BIN_ALIGN 8        // bin bases and capacities are multiples of 8 slots (128 bytes)
#define LAYOUT_THREADS 1024
#define MOVE_PIECE 1024        // most particles of one piece of a relayout
#define RELAYOUT_CTAS_PER_SM 4  // grid of the relayout copies

// Fill of one bin in one buffer: the stayers occupy [base, base + stay), the arrivals
// [base + gap, base + gap + min(moved, cap - gap)); gap is the bin's count before the push
// that filled it (no stayer rank reaches it).  `moved` is incremented atomically by the pushes
// of all source super-tiles and may exceed the room; the excess went to the overflow area.
struct BinFill {
  u32 stay, gap, moved, pad;
};
struct BinLayout {
  u32 base, cap;  // slot offset in a bin buffer, capacity
};

// The list of pieces of a peak's relayout (StepArgs::moves).  Bins that hold together what the peak
// has fit piece_room entries: two runs per bin, each rounded up to whole pieces.  Bins that disagree with
// their peak (corrupted fills) may ask for more: a bin that finds no room writes no entry, and
// then the list is not published at all, so that no entry is copied that was not written.
__host__ __device__ __forceinline__ long long piece_room(long long n, long long nst) { return n / MOVE_PIECE + 2 * nst; }
__host__ __device__ __forceinline__ bool piece_fits(u32 first, u32 pieces, long long room) {
  return (long long)first + pieces <= room;
}
__host__ __device__ __forceinline__ u32 pieces_published(u32 asked, long long room) { return asked <= room ? asked : 0u; }
// Whether a piece reads and writes inside the peak's bin region [r_off, r_off + r_size).
__host__ __device__ __forceinline__ bool piece_inside(u32 src, u32 dst, u32 count, long long r_off, long long r_size) {
  return src >= r_off && dst >= r_off && (long long)src + count <= r_off + r_size && (long long)dst + count <= r_off + r_size;
}

// Views of the engine's device arrays handed to every kernel.
struct StepArgs {
  const PeakDesc* peaks;
  PeakClock* clocks;
  PeakStats* stats;
  SortSeg* sortseg;            // sort activity flags, written by k_tick
  u32* sort_gate;              // 1 when any peak primes by sort this step (k_tick)
  u32* layout_gate;            // 1 when any peak primes or relayouts this step (k_tick)
  u32* refresh_gate;           // 1 when any peak re-sorts its super-tiles this step (k_tick)
  const long long* st_base;    // [npeaks + 1] prefix of super-tiles
  const int2* st_ref;          // [super-tile] {its peak | side << 16, its index in the peak} (one load, no search)
  const long long* fix_ref;    // [super-tile][8] offsets: its face partials, then the halo partials of its
                               // lower neighbours o = 1..7 (bit 0: x - 1, bit 1: y - 1, bit 2: z - 1)
  PeakPlan* plan;              // [peak] digest of the clock (see PeakPlan)
  const long long* p_base;     // [npeaks + 1] prefix of particles
  const long long* mode_base;  // [npeaks + 1] prefix of Green blocks
  const long long* green_base; // [ngreen + 1] prefix of Green blocks over the peaks k_green serves
  const int* green_peak;       // [ngreen] those peaks (the others use the native transform)
  int npeaks;
  int ngreen;
  int4* pos0;                  // bin buffers 0 and 1 (clock.sbuf: the current one)
  float4* mom0;
  int4* pos1;
  float4* mom1;
  int4* lpos;                  // loading area (set_particles, reload) and overflow area of the push,
  float4* lmom;                // [p_off, p_off + n) per peak
  BinLayout* lay[2];           // [super-tile] bin layouts, two generations (clock.lgen selects)
  BinFill* fill[2];            // [super-tile] bin fills of buffers 0 and 1
  u32* ovf_n;                  // [peak] particles in the overflow area (push), reset by the deposit
  u32* ovf_in;                 // [super-tile] overflowed particles whose destination it is
  u32* new_count;              // [super-tile] particles after a relayout; particles placed so far (priming)
  uint4* moves;                // pieces of a relayout, from mv_off: {source slot, destination slot, particles, -}
  u32* n_moves;                // [peak] their number
  u32* load_count;             // [super-tile] loaded particles (zero outside a priming step)
  int sorted;                  // this step primes by the radix sort
  u32* keys_push;              // Morton keys written by set_particles / reload (priming sort input)
  const u32* keys_sorted;      // sort output keys
  const u32* perm;             // sort output permutation
  u32* sstart;                 // [peak][nst + 1] starts of the super-tiles in the sorted keys
  long long* face;             // face partials
  long long* halo;             // upper-halo partials
  double2* epart;              // [super-tile][4] push partials (sum, compensation): p_x, p_y, p_z, p^2
  double* wpart;               // [Green block][warp] partials of sum_k w_k |delta_k|^2 G_k
  double2* eslice;             // [peak][ENERGY_SLICES][5] slice partials of the energy kernel
  u32* ecount;                 // [peak] energy slices finished this step (0 between steps)
  int eslices;                 // energy CTAs per peak
  double* pushed_a;            // [peak] expansion factor the push started from, -1 when it did not push
  int* sort_err;               // [peak] the priming sort's bounded look-back gave up (sort plan)
};

// Binary search: largest i in [0, n) with base[i] <= v.
__device__ __forceinline__ int pm_find(const long long* base, int n, long long v) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (base[mid] <= v) lo = mid; else hi = mid - 1;
  }
  return lo;
}

int pm_kernels_init();  // kernel attributes; call once per device before launching
size_t pm_deposit_smem(int TSmax);
size_t pm_push_smem(int TSmax);

void launch_push(const StepArgs& A, long long nst, long long ntot, size_t smem, cudaStream_t s);
void launch_tick(const StepArgs& A, cudaStream_t s);
void launch_load_count(const StepArgs& A, long long ntot, cudaStream_t s);
void launch_load_place(const StepArgs& A, long long ntot, cudaStream_t s);
void launch_permute(const StepArgs& A, long long ntot, cudaStream_t s);
void launch_st_starts(const StepArgs& A, long long ntot, cudaStream_t s);
void launch_layout(const StepArgs& A, cudaStream_t s);                     // priming peaks
void launch_relayout(const StepArgs& A, long long ntot, cudaStream_t s);    // gated
void launch_tile_sort(const StepArgs& A, long long nst, cudaStream_t s);
// only >= 0: deposit that peak alone, whether or not its clock asks for it.
void launch_deposit(const StepArgs& A, long long nst, size_t smem, double* rho64, int only, cudaStream_t s);
void launch_fixup(const StepArgs& A, long long nst, double* rho64, int only, cudaStream_t s);
void launch_green(const StepArgs& A, long long nblocks, cudaStream_t s);

// The native Poisson solve of 32^3 to 512^3 meshes and plain transforms of 64^3 to 512^3
// (native_fft.cu).  fft_native_init: once per device before use.
bool fft_native_size(int N);
bool fft_solve_size(int N);
long long fft_solve_partials(int N);
bool fft_solve_adds_nodes(int N);
int fft_native_init();
int fft_native_solve(int N, const float* delta, float2* spec, float2* gspec, float* force, const StepArgs& A,
                     const int* slot_peak, int nslots, bool sums, cudaStream_t s);

// The per-super-tile tables st_ref and fix_ref (see StepArgs).
void launch_tables(const PeakDesc* peaks, const long long* st_base, int npeaks, long long nst, int2* st_ref,
                   long long* fix_ref, cudaStream_t s);

// Host-requested per-peak operations.  reset: new schedule from a0, status and sort error
// cleared; set_thr = 1 also sets the collapse threshold and its stop flag (else they are kept).
void launch_reset_peak(const StepArgs& A, int pk, double a0, int mode, double param, double a_end,
                       int max_steps, int set_thr, double delta_collapse, int stop, cudaStream_t s);
// begin_step: a held peak runs one explicit step of da next.  write_clock: the host's clock for a peak, on the stream.
void launch_begin_step(const StepArgs& A, int pk, double da, cudaStream_t s);
void launch_write_clock(const StepArgs& A, int pk, const PeakClock& c, cudaStream_t s);
// release: the peak goes idle (no pending kick, no grids), on the stream, without a host round trip.
void launch_release_peak(const StepArgs& A, int pk, cudaStream_t s);
void launch_set_particles(const StepArgs& A, int pk, const PeakDesc& P, const double* x, const double* p,
                          cudaStream_t s);
void launch_reload(const StepArgs& A, int pk, const PeakDesc& P, cudaStream_t s);  // bins -> loading area + keys
void launch_get_particles(const StepArgs& A, int pk, const PeakDesc& P, double* x, double* p, double* acc,
                          double a_acc, cudaStream_t s);
void launch_interp64(const double* F, const double* X, long long n, int N, double dx, double* out, cudaStream_t s);
void launch_deposit64(const double* X, long long n, int N, double dx, u64* work, double* counts, cudaStream_t s);

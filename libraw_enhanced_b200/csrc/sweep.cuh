// sweep.cuh -- in-order (Gauss-Seidel) sweeps over an image on the GPU.
//
// Several demosaic passes of the reference rewrite a plane in place while
// reading neighbours that the same row-major loop has already rewritten
// (DCB's nyquist, pp, refinement clamp and last color_full loop; AAHD's
// hot-pixel pass and direction refinement).  Their result is defined by that
// order.  k_gs_sweep reproduces it exactly:
//   * a warp owns a band of 32 rows (lane = row) and walks the columns with
//     a skew of SKEW columns per row (per PAIR rows), so every neighbour that
//     precedes a site in row-major order is already updated and every one
//     that follows is not;
//   * the band's rows, its halo rows and the read-only inputs are staged
//     through a shared-memory ring of kRing columns; the next group's columns
//     are copied with cp.async while the current group runs;
//   * bands are chained through per-band progress counters in global memory
//     (release by the band above after its stores, acquire by the band below
//     before it stages the upper halo); band numbers are handed out in CTA
//     start order by an atomic ticket, so a band only waits for one that is
//     already running;
//   * every wait is bounded: on time-out the kernel raises an error flag and
//     stops waiting, and the host reports the failure.
// That in-order form is the fallback: k_blk_sweep (below) runs the same ops on
// independent blocks and checks that the result is the in-order one.
//
// An op supplies NS state planes + inputs (NP planes per warp), HALO, SKEW,
// PAIR, NCH (independent channels run as separate warps), LAG (how many
// columns behind its walk position a cell may still write), RING (ring
// columns, a power of two), BLK_WARPS (warps of a block), BLK_PER_SM (resident
// blocks per SM), BLK_ROWS and BLK_COLS (a block's overlap), BLK_FROM (how large a
// plane has to be for blocks, sweeps_in_order), BLK_SKEW and BLK_PAIR (a block's own skew),
// UNROLL (whether a block's group of steps is unrolled), STEP2 (a block visits
// every second step only, from phase(r0, g) on), IDLE0 (sites whose inputs are
// zero keep their values, so a group without others is skipped), site(r, c, g) (whether the
// pass visits the site) and cell(t, c, g), which updates the site that the
// accessor t stands on.
#pragma once

#include <algorithm>
#include <climits>
#include <string>
#include <type_traits>

#include "common.cuh"
#include "lre_internal.h"

namespace lre {
namespace {

constexpr int kRing = 128;  // default shared-memory ring width in columns (power of two)

struct Geo {
  int W, H;
  uint32_t filters;
  float maxv;
  const float* aux;  // optional device scalars an op reads (nullptr when unused)
  const float* ex[3];  // optional planes an op reads at its own sites only
  float* ex_out;       // and where it writes for the sites its block owns
  float auxv[2];       // aux[0], aux[1], read once by a block
  __device__ __forceinline__ unsigned fc(int r, int c) const { return fcol3((unsigned)r, (unsigned)c, filters); }
  __device__ __forceinline__ size_t at(int r, int c) const { return (size_t)r * W + c; }
};

// 2D launch helper: (32 x 8) threads, grid-strided in y.  Along x a block
// covers 64 columns and each thread takes two of them of the same parity in
// two half-passes (lane l: columns 2l, then 2l + 1), so the 32 lanes of a
// warp see one Bayer colour at a time and do not diverge on it.  Launch with
// (W + 63) / 64 blocks in x.
#define GS_FOR_PIXELS(g)                                                                        \
  for (int r = blockIdx.y * blockDim.y + threadIdx.y; r < (g).H; r += gridDim.y * blockDim.y)   \
    for (int gs_half = 0; gs_half < 2; gs_half++)                                                \
      for (int c = 2 * (blockIdx.x * blockDim.x + threadIdx.x) + gs_half; c < (g).W;             \
           c += 2 * gridDim.x * blockDim.x)

struct SweepArgs {
  float* plane[4];  // state planes first, then read-only inputs
  Geo g;
  int r_lo, r_hi, c_lo, c_hi;  // updated rectangle (inclusive)
  int* ticket;
  int* err;
  int* progress;  // per band: columns < progress[b] of band b are final in HBM
  const int* skip_if_zero;  // optional: every band returns at once when *skip_if_zero == 0
  const int* run_if;        // optional: likewise when *run_if == 0
  long long wait_cycles;    // bound of one wait for the band above (SM clock cycles)
  int hold_ticket;          // fault injection: this band never publishes (-1: none)
};

// The sweep's shared-memory ring, addressed through the __shared__ symbol
// itself so every access compiles to a shared-memory instruction.
extern __shared__ float sweep_smem[];

template <int NP, int HALO, int PAD, int RING>
struct Ring {
  static constexpr int ROWS = 32 + 2 * HALO;
  static constexpr int PITCH = RING + PAD;
  static constexpr int PLANE = ROWS * PITCH;
  static constexpr size_t BYTES = (size_t)NP * PLANE * sizeof(float);
  int rbase;
  __device__ __forceinline__ float& operator()(int p, int r, int c) const {
    return sweep_smem[p * PLANE + (r - rbase) * PITCH + (c & (RING - 1))];
  }
};

// One site of the ring as an op sees it: get(p, dr, dc) is state plane p at
// (r + dr, c + dc), input(p) input plane p at the site, set(p, v) writes the
// site, off(dc) is the site dc columns away.
template <class R>
struct RingCell {
  R t;
  int r, c;
  __device__ __forceinline__ float get(int p, int dr, int dc) const { return t(p, r + dr, c + dc); }
  __device__ __forceinline__ float input(int p) const { return t(p, r, c); }
  __device__ __forceinline__ void set(int p, float v) const { t(p, r, c) = v; }
  __device__ __forceinline__ RingCell off(int dc) const { return RingCell{t, r, c + dc}; }
};

// Row padding so the 32 lanes of a step hit 32 different banks: lane l
// reads row l + k at column t - SKEW * (l / PAIR), so with PAIR = 1 a pitch
// of SKEW + 1 (mod 32) gives bank l + const; with PAIR = 2 and an odd SKEW a
// pitch of 16 (mod 32) gives bank (32 - SKEW) * (l / 2) + 16 * (l & 1) +
// const, 32 distinct banks.
template <class Op>
using RingOf = Ring<Op::NP, Op::HALO, (Op::PAIR == 2 ? 16 : Op::SKEW + 1), Op::RING>;

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ints of a call's sync table before the per-band progress: [1] error flag,
// [2] gave-up flag, the last one the ticket
constexpr int kSyncInts = 64;
constexpr long long kWaitCycles = 4000000000LL;  // default wait bound: ~2 s at 1.9 GHz

__device__ __forceinline__ void cp_async4(float* s, const float* g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Steps per group.  Each group first makes the columns it needs resident
// (copies issued one group earlier), then issues the copies for the next
// group, then runs its GS steps while those copies are in flight.
constexpr int kGroup = 16;

// Groups staged ahead of the one being computed.
constexpr int kAhead = 1;
// Warps per CTA: one runs the steps, three move data.
constexpr int kSweepWarps = 4;

// One CTA per band (and channel), four warps:
//   * warp 0 runs the GS-step groups, touching only shared memory;
//   * warp 1 handles the band boundaries: in iteration g (while warp 0 runs
//     group g) it flushes the columns that became final with group g - 1,
//     publishes them at once (a release after the stores), then waits for
//     the band above as far as group g + kAhead needs and loads those
//     upper-halo rows into the ring;
//   * warps 2 and 3 copy group g + kAhead's band-local rows and inputs with
//     cp.async and wait for them.
// The warps meet at a named barrier once per group, so global-memory latency
// overlaps the steps.  Ring capacity: a group reads columns down to
// t0 - SPAN - HALO - LAG while the copies reach t0 + (kAhead + 1) * GS + HALO.
template <class Op>
__global__ void __launch_bounds__(kSweepWarps * 32) k_gs_sweep(SweepArgs a) {
  using R = RingOf<Op>;
  constexpr int HALO = Op::HALO, NS = Op::NS, NP = Op::NP, NCH = Op::NCH, GS = kGroup;
  constexpr int SPAN = Op::SKEW * (31 / Op::PAIR);  // column lag of lane 31 behind lane 0
  static_assert((kAhead + 1) * GS + SPAN + 2 * HALO + Op::LAG <= Op::RING, "sweep ring too small for this op");
  if (a.skip_if_zero && *a.skip_if_zero == 0) return;
  if (a.run_if && *a.run_if == 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lc = lane & 15, lr = lane >> 4;
  __shared__ int s_ticket;
  if (threadIdx.x == 0) s_ticket = atomicAdd(a.ticket, 1);
  __syncthreads();
  // Tickets go out in CTA start order; ticket k is band k / NCH, channel
  // k % NCH, and waits only for ticket k - NCH (same channel, band above).
  const int ticket = s_ticket;
  const int band = ticket / NCH, ch = ticket % NCH;
  const int r0 = a.r_lo + band * 32;
  const int W = a.g.W, H = a.g.H;
  const R t{r0 - HALO};
  const int t_end = a.c_hi + SPAN;
  const int ngroups = (t_end - a.c_lo) / GS + 1;
  auto group_barrier = []() { asm volatile("bar.sync 1, %0;" ::"n"(kSweepWarps * 32) : "memory"); };

  if (warp == 0) {
    const int r = r0 + lane;
    const bool row_on = r <= a.r_hi;
    __syncthreads();  // prologue staged
    for (int g = 0; g < ngroups; g++) {
      const int t0 = a.c_lo + g * GS;
#pragma unroll 4
      for (int s = 0; s < GS; s++) {
        const int c = t0 + s - Op::SKEW * (lane / Op::PAIR);
        if (row_on && c >= a.c_lo && c <= a.c_hi && Op::site(r, c, a.g)) Op::cell(RingCell<R>{t, r, c}, c, a.g);
        __syncwarp();
      }
      group_barrier();
    }
    return;
  }

  // ---- data movement
  // Per-CTA plane pointers (with NCH = 2 the argument holds
  // {state ch0, state ch1, input ch0, input ch1}).
  const float* src[NP];
  float* dst[NS];
#pragma unroll
  for (int p = 0; p < NP; p++) {
    if (NCH == 1) src[p] = a.plane[p];
    else src[p] = p < NS ? (ch ? a.plane[1] : a.plane[0]) : (ch ? a.plane[3] : a.plane[2]);
  }
#pragma unroll
  for (int p = 0; p < NS; p++) dst[p] = NCH == 1 ? a.plane[p] : (ch ? a.plane[1] : a.plane[0]);
  const int st_r0 = max(r0 - HALO, 0), st_r1 = min(r0 + 31 + HALO, H - 1);
  const int out_r1 = min(r0 + 31, a.r_hi);
  const int c_stop = a.c_hi + HALO + 1;  // staging never reaches past this column
  // Rows above r0 belong to the band above: its state planes are read by
  // warp 1 only after that band has published the columns, with L2-coherent
  // loads.  Everything else is band-local or read-only and goes through
  // warps 2 and 3.
  auto upper = [&](int p, int rr) { return band > 0 && p < NS && rr < r0; };
  int staged = a.c_lo - HALO;

  if (warp >= 2) {
    const int sub = warp - 2;  // rows st_r0 + 2 * sub + lr, step 4
    auto stage_local = [&](int hi) {
      hi = min(hi, c_stop);
      if (hi <= staged) return;
#pragma unroll
      for (int p = 0; p < NP; p++)
        for (int c = staged + lc; c < hi; c += 16)
          for (int rr = st_r0 + 2 * sub + lr; rr <= st_r1; rr += 4)
            if (!upper(p, rr)) cp_async4(&t(p, rr, c), src[p] + (size_t)rr * W + c);
      staged = hi;
    };
    stage_local(a.c_lo + kAhead * GS + HALO);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    for (int g = 0; g < ngroups; g++) {
      const int t0 = a.c_lo + g * GS;
      stage_local(t0 + (kAhead + 1) * GS + HALO);
      cp_async_commit();
      asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");  // group g + 1 resident
      group_barrier();
    }
    cp_async_wait_all();
    return;
  }

  // ---- warp 1: band boundaries
  int flushed = a.c_lo, published = a.c_lo;
  bool waiting = band > 0;
  int above = 0;
  // Progress of the band above as last observed by lane 0 (acquire loads;
  // the shuffle after the wait orders every lane's later loads).
  auto wait_above = [&](int need) {
    if (!waiting) return;
    int ok = 1;
    if (lane == 0 && above < need) {
      const long long start = clock64();
      while ((above = ld_acquire(a.progress + ticket - NCH)) < need) {
        __nanosleep(32);
        if (clock64() - start > a.wait_cycles) {
          atomicExch(a.err, 1);
          ok = 0;
          break;
        }
      }
    }
    if (!__shfl_sync(0xffffffffu, ok, 0)) waiting = false;
  };
  // Upper-halo rows of the band above, read once it has published them.
  auto stage_upper = [&](int hi) {
    hi = min(hi, c_stop);
    if (hi <= staged) return;
    if (band > 0) {
      wait_above(min(hi, a.c_hi + 1));
#pragma unroll
      for (int p = 0; p < NS; p++)
        for (int c = staged + lc; c < hi; c += 16)
          for (int rr = st_r0 + lr; rr < r0; rr += 2) t(p, rr, c) = __ldcg(src[p] + (size_t)rr * W + c);
    }
    staged = hi;
  };
  auto flush = [&](int hi) {
    if (hi <= flushed) return;
#pragma unroll
    for (int p = 0; p < NS; p++)
      for (int c = flushed + lc; c < hi; c += 16)
        for (int rr = r0 + lr; rr <= out_r1; rr += 2) __stcg(dst[p] + (size_t)rr * W + c, t(p, rr, c));
    flushed = hi;
  };
  // Release by lane 0 after a warp barrier, so it covers every lane's stores.
  auto publish = [&](int upto) {
    if (upto <= published) return;
    __syncwarp();
    if (lane == 0 && ticket != a.hold_ticket) st_release(a.progress + ticket, upto > a.c_hi ? INT_MAX : upto);
    published = upto;
  };

  stage_upper(a.c_lo + kAhead * GS + HALO);
  __syncwarp();
  __syncthreads();
  for (int g = 0; g < ngroups; g++) {
    const int t0 = a.c_lo + g * GS;
    flush(min(t0 - SPAN - Op::LAG, a.c_hi + 1));
    publish(flushed);
    stage_upper(t0 + (kAhead + 1) * GS + HALO);
    __syncwarp();
    group_barrier();
  }
  flush(a.c_hi + 1);
  publish(flushed);
}


// ---------------------------------------------------------------- blocks
// The same sweep on independent blocks, checked.
//
// A site's new value depends on values far above and to the left of it only
// through a chain of sites each of which passes on a fraction of a change (an
// average, a clamp that mostly does not bind).  So a block that starts
// BLK_ROWS rows above and BLK_COLS steps left of the sites it owns, from the
// pass's input values, arrives at its own sites with the in-order values, bit
// for bit, although what it started from was wrong.  That is not assumed but
// checked: each block keeps the values of the sites just outside its own that
// its own sites read (HALO rows above, REACH steps left), and
// k_blk_check compares them with what the owners of those sites produced.
// Where all agree, every site is its op's value of its final predecessors and
// its original successors, which is the in-order result (by induction in
// row-major order from the first block, which starts at the frame).  A block
// that disagrees runs once more from its neighbours' values (k_blk_sweep,
// repair), is checked again, and if that disagrees too the in-order sweep
// below runs on the untouched input.  The result is the in-order one always.
//
// Which frames disagree: those with flat areas larger than the overlap, clipped
// ones or synthetic ones, where a mean of equal values passes on a unit in the
// last place for ever, and runs of sites that each decide the next one.  Such a
// pass costs the blocks and the whole in-order sweep, so where a call runs the
// same op several times (DCB's nyquist) one that gave way sends the later ones
// in order at once (two iterations of DCB on clipped waves, 24, 1.5 and 0.17 MP:
// 17.5, 4.0 and 1.9 ms without that, 15.0, 3.6 and 1.5 ms; before the blocks 16.1,
// 3.2 and 1.2 ms).
// (Mending the blocks one after another instead is slower: a chain of changes
// passes through whole blocks, 250 us each, where the in-order sweep's links are
// 32 rows by 16 columns: 25.5 ms against 11.6 for DCB of 24 MP of clipped waves.)
//
// Block geometry: BLK_WARPS warps of 32 rows walk the steps tau = c + SKEW *
// (row / PAIR) of the block in groups of kBlkGroup, each warp one group behind
// the warp above; a barrier per group.  The state planes live in a
// shared-memory ring of kBlkRing steps indexed by tau (the skew is in the
// index, so the ring needs no columns for it); the inputs, read at the site
// only, in one group's buffer per warp.  With the group's steps unrolled,
// every access of a cell is one instruction: the group's place in the ring is
// in a register, the rest in the immediate.  What bounds it is the latency of
// a warp's steps (shared memory, then a chain of dependent operations), so the
// buffers are kept small enough for two blocks per SM.
//
// Why: the in-order form chains its 32-row bands through global memory and
// leaves most SMs waiting; a sweep of 24 MP took 1.9 to 2.8 ms (44 ms for the
// LoCA lift) whatever its arithmetic.  Blocks at 24 MP: nyquist 1930 -> 252 us,
// pp 2810 -> 324, refinement 2360 -> 186, color_full 2800 -> 378, LoCA 44470
// -> 1270 (with its terms as state, three blocks of four warps per SM); direction refinement at 12 MP 2210 ->
// 104, hot pixels 2000 -> 205.  Staging through registers and keeping the
// inputs in one group's buffer (two blocks per SM instead of one) was worth
// 1.9x; 4-byte cp.async into a full ring of every plane had given 620 us for
// nyquist.
//
// Overlap: an average of four updated neighbours passes on 3/7 of a change
// per row and 1/1.5 per step (pp); from a difference of 2^18 ulps, 64 rows
// and 96 steps leave fewer than 2^-20 ulps.  The noisy 12 and 24 MP scenes of the
// measured calls have no block that disagrees (lre_sweep_counts).
constexpr int kBlkGroup = 8;    // steps per group
constexpr int kBlkRing = 64;    // ring steps (power of two): groups g-2 .. g+5

struct BlkArgs {
  const float* in[4];  // state planes first, then read-only inputs (NCH = 2: as SweepArgs::plane)
  float* out[4];       // where the state planes' result goes (every site of the plane)
  Geo g;
  int r_lo, r_hi, c_lo, c_hi;  // updated rectangle (inclusive)
  int S, nbj, nbi;             // owned steps per block, blocks per row of blocks, rows of blocks
  float* side;                 // per block: the kept outside values
  int* bad;                    // [0], [1]: a block disagreed in the first / second check; [2..]: per block
  unsigned* counts;            // of the context: blocks that disagreed, passes that gave way (lre_sweep_counts)
  int* gave_up;                // optional: an earlier pass of the call gave way, and this one is to
  const int* skip_if_zero;
};

template <class Op>
struct Blk {
  static constexpr int NW = Op::BLK_WARPS, ROWS = NW * 32, OWN = ROWS - Op::BLK_ROWS;
  static constexpr int PITCH = kBlkRing + 1;  // odd: the 32 rows of a step are on 32 banks
  static constexpr int PLANE = (ROWS + 2 * Op::HALO) * PITCH;
  static constexpr int NI = Op::NP - Op::NS, IPITCH = kBlkGroup + 1, IPLANE = ROWS * IPITCH;
  static constexpr int INPUTS = Op::NS * PLANE;  // where the input buffers start
  static constexpr size_t BYTES = (size_t)(INPUTS + NI * IPLANE) * sizeof(float);
  static constexpr int PER_SM = Op::BLK_PER_SM;  // resident blocks, by shared memory and registers
  static_assert(PER_SM * (BYTES + 1024) <= 227 * 1024, "blocks per SM");
  static constexpr int SKEW = Op::BLK_SKEW, PAIR = Op::BLK_PAIR;
  // skew of a row relative to the block's first one (floor division)
  __host__ __device__ static constexpr int skew(int lr) { return SKEW * (PAIR == 2 ? (lr >> 1) : lr); }
  // columns read left of a site or above it reach this many steps back
  static constexpr int REACH = Op::HALO * SKEW + Op::HALO + Op::LAG;
  static_assert(REACH <= kBlkGroup + Op::LAG, "the ring keeps two groups behind");
  static_assert(Op::BLK_ROWS % 32 == 0 && Op::BLK_COLS % kBlkGroup == 0 && OWN > 0, "row pairs and groups stay together");
  // side buffer of one block: per state plane HALO rows of S + REACH steps,
  // then OWN rows of REACH steps
  static size_t side_floats(int S) { return (size_t)Op::NS * (Op::HALO * (S + REACH) + OWN * REACH); }
};

// The accessor of a block's cells.  b[q] is the ring place of group g - 2 + q
// in this lane's row and s the step in the group, a constant after unrolling,
// so the group a neighbour falls into is known at compile time.
template <class Op>
struct BlkCell {
  unsigned b[5], in;
  int s;
  __device__ __forceinline__ unsigned at(int p, int dr, int dc) const {
    using B = Blk<Op>;
    const int dt = s + dc + B::SKEW * (B::PAIR == 2 ? dr / 2 : dr) + 2 * kBlkGroup;
    return b[dt >> 3] + p * B::PLANE + dr * B::PITCH + (dt & 7);
  }
  __device__ __forceinline__ float get(int p, int dr, int dc) const { return sweep_smem[at(p, dr, dc)]; }
  __device__ __forceinline__ float input(int p) const { return sweep_smem[in + (p - Op::NS) * Blk<Op>::IPLANE + s]; }
  __device__ __forceinline__ void set(int p, float v) const { sweep_smem[at(p, 0, 0)] = v; }
  __device__ __forceinline__ BlkCell off(int dc) const {
    BlkCell o = *this;
    o.s += dc;
    return o;
  }
};
// Without unrolling: the step is a run-time value.
template <class Op>
struct BlkCellAny {
  unsigned row, in;  // this lane's row in the ring and in the input buffer
  int lr, tau;
  size_t px;  // the site's index in the image
  bool own;   // the block owns the site
  __device__ __forceinline__ unsigned at(int p, int dr, int dc) const {
    using B = Blk<Op>;
    const int dt = dc + (B::PAIR == 2 ? B::skew(lr + dr) - B::skew(lr) : B::SKEW * dr);
    return row + p * B::PLANE + dr * B::PITCH + ((tau + dt) & (kBlkRing - 1));
  }
  __device__ __forceinline__ float get(int p, int dr, int dc) const { return sweep_smem[at(p, dr, dc)]; }
  __device__ __forceinline__ float input(int p) const {
    return sweep_smem[in + (p - Op::NS) * Blk<Op>::IPLANE + (tau & (kBlkGroup - 1))];
  }
  __device__ __forceinline__ void set(int p, float v) const { sweep_smem[at(p, 0, 0)] = v; }
};

template <class Op, bool REPAIR>
__global__ void __launch_bounds__(Blk<Op>::NW * 32, Blk<Op>::PER_SM) k_blk_sweep(BlkArgs a) {
  using B = Blk<Op>;
  constexpr int G = kBlkGroup, NP = Op::NP, NS = Op::NS, HALO = Op::HALO, NCH = Op::NCH, KR = Op::BLK_ROWS;
  if (a.skip_if_zero && *a.skip_if_zero == 0) return;
  const int ch = blockIdx.z, bi = blockIdx.y, bj = blockIdx.x;
  const int blk = (ch * a.nbi + bi) * a.nbj + bj;
  if (a.gave_up && *a.gave_up != 0) {
    if (!REPAIR && blk == 0 && threadIdx.x == 0) {
      a.bad[1] = 1;
      atomicAdd(a.counts + 1, 1u);
    }
    return;
  }
  if (REPAIR && a.bad[2 + blk] == 0) return;
  const int W = a.g.W, H = a.g.H;
  const int own_r = bi * B::OWN, r0 = own_r - KR;
  const int own_lo = B::skew(KR) + bj * a.S, own_hi = own_lo + a.S;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int l8 = lane & 7, l4 = lane >> 3;
  const float* src[NP];
  float* dst[NS];
#pragma unroll
  for (int p = 0; p < NP; p++)
    src[p] = NCH == 1 ? a.in[p] : (p < NS ? (ch ? a.in[1] : a.in[0]) : (ch ? a.in[3] : a.in[2]));
#pragma unroll
  for (int p = 0; p < NS; p++) dst[p] = NCH == 1 ? a.out[p] : (ch ? a.out[1] : a.out[0]);
  const int g_lo = (REPAIR ? own_lo : own_lo - Op::BLK_COLS) >> 3;  // first group walked
  const int g_hi = (own_hi - 1 + Op::LAG) >> 3;                    // last one
  const int ng = g_hi - g_lo + 1;

  // Rows this warp stages: its 32, eight steps of rows k, k + 8, k + 16 and
  // k + 24 per instruction (32 distinct banks), and, at the block's ends, the
  // halo rows.  Loaded into registers in one phase and stored to shared memory
  // at the start of the next: state for group g + 5, inputs for group g.
  const int lr8 = warp * 32 + 8 * l4;  // even, so row lr8 + k has skew skew(lr8) + skew(k)
  const int lrh = warp == 0 && l4 < HALO ? l4 - HALO : (warp == B::NW - 1 && l4 < HALO ? B::ROWS + l4 : INT_MAX);
  const unsigned slr = (lr8 + HALO) * B::PITCH;
  float v[8][NP], vh[NS];
  // every row and column of group g inside the image (the same in every lane)
  auto inside = [&](int g) {
    return r0 + warp * 32 >= 0 && r0 + warp * 32 + 32 <= H && g * G - B::skew(warp * 32 + 31) >= 0 &&
           g * G + G - B::skew(warp * 32) <= W;
  };
  // planes [P0, P1) of group g
  auto load = [&](int g, auto p0, auto p1) {
    constexpr int P0 = decltype(p0)::value, P1 = decltype(p1)::value;
    const int tau = g * G + l8;
    const int c0 = tau - B::skew(lr8);
    const ptrdiff_t i0 = (ptrdiff_t)(r0 + lr8) * W + c0;
    if (!REPAIR && inside(g)) {
#pragma unroll
      for (int k = 0; k < 8; k++)
#pragma unroll
        for (int p = P0; p < P1; p++) v[k][p] = __ldg(src[p] + i0 + ((ptrdiff_t)k * W - B::skew(k)));
    } else {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int r = r0 + lr8 + k, c = c0 - B::skew(k);
        const bool on = r >= 0 && r < H && c >= 0 && c < W;
#pragma unroll
        for (int p = P0; p < P1; p++) {
          // a repair starts from what the neighbours before it produced
          const float* q = REPAIR && p < NS && (lr8 + k < KR || tau < own_lo) ? dst[p] : src[p];
          v[k][p] = on ? __ldcg(q + i0 + ((ptrdiff_t)k * W - B::skew(k))) : 0.f;
        }
      }
    }
    if (P0 == 0 && lrh != INT_MAX) {
      const int r = r0 + lrh, c = tau - B::skew(lrh);
      const bool on = r >= 0 && r < H && c >= 0 && c < W;
#pragma unroll
      for (int p = 0; p < NS; p++) {
        const float* q = REPAIR && lrh < KR ? dst[p] : src[p];
        vh[p] = on ? __ldcg(q + (ptrdiff_t)r * W + c) : 0.f;
      }
    }
  };
  auto store = [&](int g) {  // state planes
    const unsigned tr = (g * G + l8) & (kBlkRing - 1);
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
      for (int p = 0; p < NS; p++) sweep_smem[p * B::PLANE + slr + tr + k * B::PITCH] = v[k][p];
    if (lrh != INT_MAX) {
#pragma unroll
      for (int p = 0; p < NS; p++) sweep_smem[p * B::PLANE + (lrh + HALO) * B::PITCH + tr] = vh[p];
    }
  };
  // Returns whether any input of the warp's group is non-zero (g: that group).
  auto store_inputs = [&](int g) {
    const unsigned sl = B::INPUTS + lr8 * B::IPITCH + l8;
    bool any = false;
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
      for (int p = NS; p < NP; p++) {
        sweep_smem[sl + (p - NS) * B::IPLANE + k * B::IPITCH] = v[k][p];
        any |= v[k][p] != 0.f;
        if (Op::IDLE0 && v[k][p] != 0.f) {
          // what the op will read at this site, on its way to L1
          const ptrdiff_t px = (ptrdiff_t)(r0 + lr8 + k) * W + g * G + l8 - B::skew(lr8 + k);
#pragma unroll
          for (int e = 0; e < 3; e++) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.g.ex[e] + px));
        }
      }
    return Op::IDLE0 ? __any_sync(0xffffffffu, any) != 0 : true;
  };
  const std::integral_constant<int, 0> z0{};
  const std::integral_constant<int, NS> zs{};
  const std::integral_constant<int, NP> zp{};

  const int top_len = a.S + B::REACH;
  float* side = a.side + (size_t)blk * (NS * (HALO * top_len + B::OWN * B::REACH));
  // final values of group g: the owned ones to the result, the outside ones
  // that owned sites read to the side buffer
  auto flush = [&](int g) {
    const int tau = g * G + l8;
    const int c0 = tau - B::skew(lr8);
    const ptrdiff_t i0 = (ptrdiff_t)(r0 + lr8) * W + c0;
    const unsigned sl = slr + (tau & (kBlkRing - 1));
    if (warp * 32 >= KR && g * G >= own_lo && g * G + G <= own_hi && inside(g)) {
#pragma unroll
      for (int k = 0; k < 8; k++)
#pragma unroll
        for (int p = 0; p < NS; p++)
          dst[p][i0 + ((ptrdiff_t)k * W - B::skew(k))] = sweep_smem[p * B::PLANE + sl + k * B::PITCH];
      return;
    }
    if (g * G + G <= own_lo - B::REACH || (warp * 32 + 32 <= KR - HALO)) return;
    const bool own_c = tau >= own_lo && tau < own_hi;
#pragma unroll 1
    for (int k = 0; k < 8; k++) {
      const int lr = lr8 + k, r = r0 + lr, c = c0 - B::skew(k);
      if (r < 0 || r >= H || c < 0 || c >= W) continue;
      const unsigned q = sl + k * B::PITCH;
      if (lr >= KR) {
        if (own_c) {
#pragma unroll
          for (int p = 0; p < NS; p++) dst[p][(size_t)r * W + c] = sweep_smem[p * B::PLANE + q];
        } else if (tau < own_lo && tau >= own_lo - B::REACH) {
#pragma unroll
          for (int p = 0; p < NS; p++)
            side[NS * HALO * top_len + (p * B::OWN + lr - KR) * B::REACH + tau - (own_lo - B::REACH)] =
                sweep_smem[p * B::PLANE + q];
        }
      } else if (lr >= KR - HALO && tau >= own_lo - B::REACH && tau < own_hi) {
#pragma unroll
        for (int p = 0; p < NS; p++)
          side[(p * HALO + lr - (KR - HALO)) * top_len + tau - (own_lo - B::REACH)] = sweep_smem[p * B::PLANE + q];
      }
    }
  };

  for (int g = g_lo - 2; g <= g_lo + 4; g++) {
    load(g, z0, zs);
    store(g);
  }
  load(g_lo, zs, zp);
  load(g_lo + 5, z0, zs);
  __syncthreads();
  if (REPAIR) {  // the outside values a repair starts from are the ones it uses
    flush(g_lo - 2);
    flush(g_lo - 1);
  }
  if (a.g.aux) {
    a.g.auxv[0] = a.g.aux[0];
    a.g.auxv[1] = a.g.aux[1];
  }
  const int lr = warp * 32 + lane, r = r0 + lr;
  const bool row_on = r >= a.r_lo && r <= a.r_hi && (!REPAIR || lr >= KR);
  const unsigned srow = (lr + HALO) * B::PITCH, irow = B::INPUTS + lr * B::IPITCH;
  for (int k = 0; k < ng + B::NW; k++) {
    const int g = g_lo + k - warp;
    if (k >= warp && k - warp < ng) {
      store(g + 5);
      const bool busy = store_inputs(g);
      __syncwarp();
      load(g + 1, zs, zp);
      load(g + 6, z0, zs);
      const int c0 = g * G - B::skew(lr);
      if constexpr (Op::UNROLL) {
        BlkCell<Op> t;
        t.in = irow;
#pragma unroll
        for (int q = 0; q < 5; q++) t.b[q] = srow + (((g - 2 + q) * G) & (kBlkRing - 1));
        // which steps the pass visits: all, or (STEP2) every second one
        const int ph = Op::STEP2 ? Op::phase(r0, a.g) & 1 : 0;
        auto steps = [&](auto all, auto first) {
          constexpr bool ALL = decltype(all)::value;
          constexpr int F = decltype(first)::value;
#pragma unroll
          for (int s = F; s < G; s += Op::STEP2 ? 2 : 1) {
            t.s = s;
            const int c = c0 + s;
            if (ALL || (row_on && c >= a.c_lo && c <= a.c_hi)) Op::cell(t, c, a.g);
            __syncwarp();
          }
        };
        // every site of the group is updated (the same answer in every lane)
        const bool all = !REPAIR && r0 + warp * 32 >= a.r_lo && r0 + warp * 32 + 31 <= a.r_hi &&
                         g * G - B::skew(warp * 32 + 31) >= a.c_lo && g * G + G - 1 - B::skew(warp * 32) <= a.c_hi;
        const std::true_type yes{};
        const std::false_type no{};
        const std::integral_constant<int, 0> f0{};
        const std::integral_constant<int, Op::STEP2 ? 1 : 0> f1{};
        if (all) {
          if (ph) steps(yes, f1); else steps(yes, f0);
        } else {
          if (ph) steps(no, f1); else steps(no, f0);
        }
      } else if (busy) {
        const size_t px = (size_t)r * W + c0;
#pragma unroll 1
        for (int s = 0; s < G; s++) {
          const int c = c0 + s, tau = g * G + s;
          if (row_on && c >= a.c_lo && c <= a.c_hi && Op::site(r, c, a.g))
            Op::cell(BlkCellAny<Op>{srow, irow, lr, tau, px + s, lr >= KR && tau >= own_lo && tau < own_hi}, c, a.g);
          __syncwarp();
        }
      }
      if (k > warp) flush(g - 1);
    } else if (k - warp == ng) {
      flush(g_hi);
    }
    __syncthreads();
  }
}

// Compares every block's kept outside values with the owners' results.
// ROUND 0 is the first check; ROUND 1 runs only where round 0 found a block
// bad, after the repair.
template <class Op, int ROUND>
__global__ void __launch_bounds__(256) k_blk_check(BlkArgs a) {
  using B = Blk<Op>;
  constexpr int NS = Op::NS, HALO = Op::HALO, NCH = Op::NCH;
  if (a.skip_if_zero && *a.skip_if_zero == 0) return;
  if (ROUND == 1 && a.bad[0] == 0) return;
  if (a.gave_up && *a.gave_up != 0) return;
  const int ch = blockIdx.z, bi = blockIdx.y, bj = blockIdx.x;
  const int blk = (ch * a.nbi + bi) * a.nbj + bj;
  const int own_r = bi * B::OWN, r0 = own_r - Op::BLK_ROWS;
  const int own_lo = B::skew(Op::BLK_ROWS) + bj * a.S;
  const int top_len = a.S + B::REACH;
  const size_t per = NS * (HALO * top_len + B::OWN * B::REACH);
  const float* side = a.side + (size_t)blk * per;
  int bad = 0;
  for (int e = threadIdx.x; e < (int)per; e += blockDim.x) {
    int p, lr, tau;
    if (e < NS * HALO * top_len) {
      p = e / (HALO * top_len);
      const int q = e - p * HALO * top_len;
      lr = Op::BLK_ROWS - HALO + q / top_len;
      tau = own_lo - B::REACH + q % top_len;
    } else {
      const int q = e - NS * HALO * top_len;
      p = q / (B::OWN * B::REACH);
      const int z = q - p * B::OWN * B::REACH;
      lr = Op::BLK_ROWS + z / B::REACH;
      tau = own_lo - B::REACH + z % B::REACH;
    }
    const int r = r0 + lr, c = tau - B::skew(lr);
    if (r < a.r_lo || r > a.r_hi || c < a.c_lo || c > a.c_hi) continue;
    const float* o = NCH == 1 ? (p == 0 ? a.out[0] : (p == 1 ? a.out[1] : a.out[2])) : (ch ? a.out[1] : a.out[0]);
    bad |= __float_as_int(o[(size_t)r * a.g.W + c]) != __float_as_int(side[e]);
  }
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    if (ROUND == 0) a.bad[2 + blk] = bad;
    if (bad) {
      if (ROUND == 0) {
        atomicExch(a.bad, 1);
        atomicAdd(a.counts, 1u);
      }
      // an op that also writes behind its walk position is not repaired: a
      // repair would update the last site of the block before it twice
      if ((ROUND == 1 || Op::LAG > 0) && atomicExch(a.bad + 1, 1) == 0) {
        atomicAdd(a.counts + 1, 1u);
        if (a.gave_up) *a.gave_up = 1;
      }
    }
  }
}

// out = in where the in-order sweep ran in place on `in` (run_if), or, for a
// sweep whose result stays in its input planes, in = out where it did not.
template <int NPL>
__global__ void k_blk_copy(BlkArgs a, const int* run_if, int back) {
  if (a.skip_if_zero && *a.skip_if_zero == 0) return;
  if ((*run_if != 0) == (back != 0)) return;
  const size_t n = (size_t)a.g.W * a.g.H;
#pragma unroll
  for (int p = 0; p < NPL; p++) {
    const float* s = back ? a.out[p] : a.in[p];
    float* d = back ? const_cast<float*>(a.in[p]) : a.out[p];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) d[i] = s[i];
  }
}

// Owned steps per block: what takes the fewest phases over all waves of
// blocks (PER_SM per SM, two for most ops).  A wide block spends less on overlap, a narrow one
// fills the last wave: at 24 MP (21 rows of blocks) 512 gives one wave of 84
// phases, 256 two of 52.
constexpr int kBlkSms = 148;  // the grid shape is also planned without a device
template <class Op>
void blk_grid(int W, int H, int* S, int* nbj, int* nbi) {
  using B = Blk<Op>;
  *nbi = (H + B::OWN - 1) / B::OWN;
  const int steps = W + B::skew(B::ROWS - 1) - B::skew(Op::BLK_ROWS);
  long long best = LLONG_MAX;
  for (int t = 64; t <= 2048; t += 64) {
    const long long n = (long long)((steps + t - 1) / t) * *nbi * Op::NCH;
    constexpr long long places = (long long)B::PER_SM * kBlkSms;
    const long long cost = (n + places - 1) / places * ((t + Op::BLK_COLS) / kBlkGroup + B::NW);
    if (cost < best) {
      best = cost;
      *S = t;
    }
  }
  *nbj = (steps + *S - 1) / *S;
}

// Workspace of block sweeps of a w x h plane, whichever of the ops runs.
template <class... Ops>
size_t blk_ws_bytes(size_t w, size_t h) {
  size_t m = 0;
  auto one = [&](auto* op) {
    using Op = std::remove_pointer_t<decltype(op)>;
    int S, nbj, nbi;
    blk_grid<Op>((int)w, (int)h, &S, &nbj, &nbi);
    const size_t n = (size_t)nbj * nbi * Op::NCH;
    m = std::max(m, n * Blk<Op>::side_floats(S) * sizeof(float) + (n + 2) * sizeof(int) + 1024);
  };
  (one(static_cast<Ops*>(nullptr)), ...);
  return m;
}

template <class Op>
lre_status sweep_in_order(Context* c, const SweepArgs& base, int* sync, int nb_max, const char* what) {
  if (base.r_hi < base.r_lo || base.c_hi < base.c_lo) return LRE_OK;
  using R = RingOf<Op>;
  const int nb = (base.r_hi - base.r_lo + 32) / 32 * Op::NCH;
  if (nb > nb_max) return fail(c, LRE_ERR_CUDA, std::string(what) + ": band table too small");
  SweepArgs a = base;
  a.ticket = sync + kSyncInts - 1;  // cleared together with the table
  a.progress = sync + kSyncInts;
  a.wait_cycles = c->sweep_wait_cycles > 0 ? c->sweep_wait_cycles : kWaitCycles;
  // a held band (host-side fault injection, one sweep only) never reports
  // its progress, so the band below it waits until its bound runs out
  a.hold_ticket = c->sweep_hold_band >= 0 ? c->sweep_hold_band * Op::NCH : -1;
  c->sweep_hold_band = -1;
  LRE_CUDA_TRY(c, cudaMemsetAsync(a.ticket, 0, (size_t)(nb + 1) * sizeof(int), c->stream));
  LRE_CUDA_TRY(c, cudaFuncSetAttribute(k_gs_sweep<Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R::BYTES));
  k_gs_sweep<Op><<<nb, kSweepWarps * 32, R::BYTES, c->stream>>>(a);
  count_launch(c);
  return check_launch(c, what);
}

// The block sweep with its checks and the repair.  *run_if (device) is then
// non-zero when the in-order sweep has to run instead.
template <class Op>
lre_status blk_sweep(Context* c, BlkArgs& b, void* ws, size_t ws_len, const int** run_if, const char* what) {
  using B = Blk<Op>;
  blk_grid<Op>(b.g.W, b.g.H, &b.S, &b.nbj, &b.nbi);
  const size_t n = (size_t)b.nbj * b.nbi * Op::NCH;
  if (n * B::side_floats(b.S) * sizeof(float) + (n + 2) * sizeof(int) > ws_len || b.nbi > 65535)
    return fail(c, LRE_ERR_CUDA, std::string(what) + ": block table too small");
  b.bad = reinterpret_cast<int*>(ws);
  b.counts = sweep_counts(c);
  b.side = reinterpret_cast<float*>(reinterpret_cast<char*>(ws) + (((n + 2) * sizeof(int) + 255) & ~size_t(255)));
  *run_if = b.bad + 1;
  LRE_CUDA_TRY(c, cudaMemsetAsync(b.bad, 0, 2 * sizeof(int), c->stream));
  const dim3 grid((unsigned)b.nbj, (unsigned)b.nbi, Op::NCH);
  auto k0 = k_blk_sweep<Op, false>;
  auto k1 = k_blk_sweep<Op, true>;
  LRE_CUDA_TRY(c, cudaFuncSetAttribute(k0, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)B::BYTES));
  LRE_CUDA_TRY(c, cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)B::BYTES));
  k0<<<grid, B::NW * 32, B::BYTES, c->stream>>>(b);
  k_blk_check<Op, 0><<<grid, 256, 0, c->stream>>>(b);
  count_launch(c, 2);
  if (Op::LAG == 0) {
    k1<<<grid, B::NW * 32, B::BYTES, c->stream>>>(b);
    k_blk_check<Op, 1><<<grid, 256, 0, c->stream>>>(b);
    count_launch(c, 2);
  }
  return check_launch(c, what);
}

// Whether a pass runs in order without trying blocks: where a wait limit or an
// injected stall asks for it, and on planes so small that the blocks' latency (43
// to 52 us a pass, whatever the size) is more than that of the few bands, which
// grows with the width and 2.5 times the height.  Blocks and in order, us: DCB (one
// iteration, six passes) 64x64 496 and 285, 128x128 507 and 440, 256x128 508 and
// 524; AAHD without hot pixels 64x64 136 and 110, 128x128 147 and 146, with them
// 64x128 213 and 219.  LoCA's blocks are the faster ones from 48x48 on.
template <class Op>
bool sweeps_in_order(Context* c, int W, int H) {
  return c->sweep_hold_band >= 0 || c->sweep_wait_cycles > 0 || 2 * W + 5 * H < Op::BLK_FROM;
}

// The sweep of base.plane[0 .. NS * NCH).  The result is in out[0 .. NS * NCH)
// (whole planes; the input planes are then scratch) if *moved says so, else where
// the input was.  keep: it is to end in the input planes.  ws: blk_ws_bytes of the
// plane.
template <class Op>
lre_status sweep(Context* c, const SweepArgs& base, float* const* out, bool keep, void* ws, size_t ws_len, int* sync,
                 int nb_max, const char* what, bool* moved, int* gave_up = nullptr) {
  constexpr int NPL = Op::NS * Op::NCH;
  *moved = false;
  if (base.r_hi < base.r_lo || base.c_hi < base.c_lo) return LRE_OK;  // nothing to update
  if (sweeps_in_order<Op>(c, base.g.W, base.g.H)) return sweep_in_order<Op>(c, base, sync, nb_max, what);
  *moved = !keep;
  BlkArgs b{};
  for (int p = 0; p < 4; p++) b.in[p] = base.plane[p];
  for (int p = 0; p < NPL; p++) b.out[p] = out[p];
  b.g = base.g;
  b.r_lo = base.r_lo;
  b.r_hi = base.r_hi;
  b.c_lo = base.c_lo;
  b.c_hi = base.c_hi;
  b.skip_if_zero = base.skip_if_zero;
  b.gave_up = gave_up;
  SweepArgs a = base;
  LRE_TRY(blk_sweep<Op>(c, b, ws, ws_len, &a.run_if, what));
  LRE_TRY(sweep_in_order<Op>(c, a, sync, nb_max, what));
  const unsigned cg = grid_for((size_t)b.g.W * b.g.H, 256, c->sm_count * 4);
  k_blk_copy<NPL><<<cg, 256, 0, c->stream>>>(b, a.run_if, keep ? 1 : 0);
  count_launch(c);
  return check_launch(c, what);
}

bool bayer_2x2(uint32_t filters) {
  // DCB's loops address non-green sites by column parity; that is the
  // reference's intent only for 2x2 Bayer layouts with green on a
  // checkerboard and R/B on the other two sites.
  for (unsigned r = 0; r < 8; r++) {
    const unsigned a = fcol3(r, 0, filters), b = fcol3(r, 1, filters);
    if ((a == 1) == (b == 1)) return false;
    if (fcol3(r, 2, filters) != a || fcol3((r + 2) & 7, 0, filters) != a || fcol3((r + 2) & 7, 1, filters) != b)
      return false;
  }
  const unsigned n0 = fcol3(0, 0, filters) == 1 ? fcol3(0, 1, filters) : fcol3(0, 0, filters);
  const unsigned n1 = fcol3(1, 0, filters) == 1 ? fcol3(1, 1, filters) : fcol3(1, 0, filters);
  if (fcol3(0, 0, filters) == 1 && fcol3(1, 0, filters) == 1) return false;
  return n0 + n1 == 2 && n0 != n1;
}

}  // namespace
}  // namespace lre

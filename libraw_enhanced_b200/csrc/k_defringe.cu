// k_defringe.cu -- edge-gated chroma-ratio defringe.
//
// Semantics: core/cpu_accelerator.cpp:3939-5064 (CPUAccelerator::defringe).
// Every per-pixel expression below is the reference's, in the reference's
// operation order (the library is built with --fmad=false), so results match
// bit for bit except where glibc's logf/expf and the device's differ by an
// ulp (see log_cr / exp_cr).
//
// Stage plan on the device (planes are float W x H in the workspace):
//   R0  max(0, G) reduction                       -> max_guide
//   K1  ratios + Sobel on sqrt(G/max)             -> lrg, lbg, edge_raw, max_edge
//   K2  5 separable Gaussian blurs (one kernel)   -> bg, blrg, blbg, be, ber
//   K3  fringe-support seed                       -> fs
//   K4  blur(fs)                                  -> bfs
//   K5  line-linked support + solo seeds          -> lfs, srs, sbs
//   K6  blur(srs), blur(sbs)                      -> srb, sbb
//   K7  classification + correction (in-place safe)
// Blurs walk column strips (k_df_blur_strip); the line-link kernel stages a
// +-14 px clamped halo.
#include <algorithm>
#include <cmath>

#include "lre_internal.h"
#include "stencil.cuh"

namespace lre {

GaussTaps make_defringe_taps(float radius) {
  GaussTaps t{};
  const float sigma = std::max(radius / 3.f, 0.5f);
  int ks = static_cast<int>(std::ceil(3.f * sigma));
  if (ks > GAUSS_MAX_KS) ks = GAUSS_MAX_KS;  // caller rejects larger radii first
  t.ks = ks;
  float ksum = 0.f;
  for (int k = -ks; k <= ks; k++) {
    float v = std::exp(-0.5f * (float)(k * k) / (sigma * sigma));
    t.w[k + ks] = v;
    ksum += v;
  }
  for (int k = 0; k < 2 * ks + 1; k++) t.w[k] /= ksum;
  return t;
}

namespace {

struct DfScalars {
  float max_guide_raw;  // max(0, G) over the image
  float max_edge;       // max Sobel magnitude (interior)
  int nonfinite;        // a log ratio of the image is infinite or NaN
};

struct DfPlanes {
  float *lrg, *lbg, *er, *bg, *blrg, *blbg, *be, *ber, *fs, *bfs, *lfs, *srs, *sbs, *srb, *sbb;
};

__device__ __forceinline__ float df_max_guide(const DfScalars* s) { return smax(s->max_guide_raw, 1e-6f); }

// ---------------------------------------------------------------- K1
// K1: log ratios and Sobel magnitude of the guide signal.  A warp walks up to
// PW_ROWS rows of 30 columns (and one beside them on either side): the guide
// signal, a square root and a divide, is formed once per pixel, its neighbours
// come from the lanes beside and the two rows before, and the next two rows are
// on their way meanwhile.  Bound by instructions: two logarithms in double, two
// divides and the guide.  51 MP 448 us, 26 MP odd 237 us, 1.9 MP 20 us; on 32 x 8
// tiles with the guide in shared memory, a barrier before and after, 783, 402 and
// 24 us, and with CUDA's log in double besides 856, 441 and 27 us.
constexpr int PW_ROWS = 32, PW_COLS = 30;

__global__ void __launch_bounds__(256) k_df_prep(const float* __restrict__ src, int W, int H, int rows, DfScalars* sc,
                                                 float* __restrict__ lrg, float* __restrict__ lbg,
                                                 float* __restrict__ er) {
  __shared__ __align__(16) double2 s_log[LOG_TAB_N];
  log_tab_fill(s_log);
  __syncthreads();
  const float max_guide = df_max_guide(sc);
  const float ratio_eps = smax(max_guide * 1e-4f, 1e-6f);
  const int limit_y = (H > 1) ? H - 1 : 1;
  const int limit_x = (W > 1) ? W - 1 : 1;
  const int strips = (W + PW_COLS - 1) / PW_COLS;
  const long long items = (long long)strips * ((H + rows - 1) / rows);
  const int lane = threadIdx.x & 31;
  auto guide = [&](float g) { return sqrtf(sclamp(smax(g, 0.f) / max_guide, 0.f, 1.f)); };
  bool odd = false;
  float local_max = 0.f;
  for (long long it = blockIdx.x * 8LL + (threadIdx.x >> 5); it < items; it += gridDim.x * 8LL) {
    const int chunk = (int)(it / strips), x = (int)(it - (long long)chunk * strips) * PW_COLS + lane - 1;
    const int y0 = chunk * rows, y1 = min(y0 + rows, H);
    const float* col = src + (size_t)min(max(x, 0), W - 1) * 3;
    auto row = [&](int y) { return col + (size_t)min(max(y, 0), H - 1) * W * 3; };
    struct Px {
      float r, g, b;
    };
    auto load = [&](int y) {
      const float* p = row(y);
      return Px{p[0], p[1], p[2]};
    };
    // a: the row above, b: this row, c: the row below; 0 left, 1 here, 2 right
    auto across = [&](float v, float& l, float& r) {
      l = __shfl_up_sync(~0u, v, 1);
      r = __shfl_down_sync(~0u, v, 1);
    };
    Px cur = load(y0), nxt = load(y0 + 1);
    float a00, a01 = guide(row(y0 - 1)[1]), a02, a10, a11 = guide(cur.g), a12, a20, a21, a22;
    across(a01, a00, a02);
    across(a11, a10, a12);
    const bool mine = lane >= 1 && lane <= PW_COLS && x < W;
    const bool inside = mine && x >= 1 && x < limit_x;
#pragma unroll 2
    for (int y = y0; y < y1; y++) {
      const Px aft = load(y + 2);
      a21 = guide(nxt.g);
      across(a21, a20, a22);
      const float gg = smax(cur.g, 0.f);
      const float lr = log_tab(s_log, (smax(cur.r, 0.f) + ratio_eps) / (gg + ratio_eps));
      const float lb = log_tab(s_log, (smax(cur.b, 0.f) + ratio_eps) / (gg + ratio_eps));
      float mag = 0.f;
      if (inside && y >= 1 && y < limit_y) {
        const float gx = -a00 + a02 - 2.f * a10 + 2.f * a12 - a20 + a22;
        const float gy = -a00 - 2.f * a01 - a02 + a20 + 2.f * a21 + a22;
        mag = sqrtf(gx * gx + gy * gy);
        local_max = smax(local_max, mag);
      }
      if (mine) {
        const size_t i = (size_t)y * W + x;
        odd |= !(isfinite(lr) && isfinite(lb));
        lrg[i] = lr;
        lbg[i] = lb;
        er[i] = mag;
      }
      cur = nxt;
      nxt = aft;
      a00 = a10;
      a01 = a11;
      a02 = a12;
      a10 = a20;
      a11 = a21;
      a12 = a22;
    }
  }
  if (odd) sc->nonfinite = 1;
  local_max = warp_max(local_max);
  if (lane == 0) atomic_max_float(&sc->max_edge, local_max);
}

// ---------------------------------------------------------------- blurs
// Source modes for a blur input plane.
enum BlurSrc : int { BS_PLANE = 0, BS_PLANE_EDGE_NORM = 1, BS_GUIDE_LINEAR = 2 };

struct BlurJob {
  const float* in[5];
  float* out[5];
  int mode[5];
  int np;
  unsigned long long nz = 0x8000000080000000ull;  // {-0.f, -0.f} (f2_mul)
};

constexpr int BT = 32;  // output tile edge

__device__ __forceinline__ void ld4(const float* p, float* o) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  o[0] = t.x;
  o[1] = t.y;
  o[2] = t.z;
  o[3] = t.w;
}
__device__ __forceinline__ void st4(float* p, const float* o) {
  *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
}

// Element p of a small parameter array through constant indices only: a
// run-time index into a kernel parameter would copy the whole parameter block
// to local memory.
template <typename T>
__device__ __forceinline__ T pick5(const T (&a)[5], int p) {
  switch (p) {
    case 0: return a[0];
    case 1: return a[1];
    case 2: return a[2];
    case 3: return a[3];
    default: return a[4];
  }
}

__device__ __forceinline__ float blur_src(const float* in, int mode, const DfScalars* sc, int x, int y, int W) {
  size_t i = (size_t)y * W + x;
  switch (mode) {
    case BS_GUIDE_LINEAR:
      return smax(in[i * 3 + 1], 0.f);
    case BS_PLANE_EDGE_NORM: {
      float f = smax(sc->max_edge, 1e-6f);
      float inv = 1.f / f;
      return in[i] * inv;
    }
    default:
      return in[i];
  }
}

// One CTA = BT x BT outputs of one plane of the job (blockIdx.z); the clamped
// input halo and the horizontal-pass rows live in shared memory, 48 KB at the
// largest tap radius.  (With the job's five planes in one CTA it was 222 KB at
// tap radius 30 and more than a CTA may have at 31 and 32.)
__global__ void __launch_bounds__(256) k_df_blur(BlurJob job, GaussTaps taps, int W, int H, const DfScalars* sc) {
  extern __shared__ __align__(16) float sm[];
  const int ks = taps.ks;
  const int E = BT + 2 * ks;  // halo tile edge
  const int x0 = blockIdx.x * BT, y0 = blockIdx.y * BT;
  float* s_in = sm;         // [E][E]
  float* s_h = sm + E * E;  // [E][BT]
  const float* in = pick5(job.in, blockIdx.z);
  const int mode = pick5(job.mode, blockIdx.z);
  for (int i = threadIdx.x; i < E * E; i += blockDim.x) {
    int gy = min(max(y0 - ks + i / E, 0), H - 1);
    int gx = min(max(x0 - ks + i % E, 0), W - 1);
    s_in[i] = blur_src(in, mode, sc, gx, gy, W);
  }
  __syncthreads();
  // horizontal pass over all E halo rows (rows are the clamped image rows)
  for (int i = threadIdx.x; i < E * BT; i += blockDim.x) {
    int j = i / BT, k = i % BT;
    const float* row = s_in + j * E + k;
    float acc = 0.f;
    for (int t = 0; t <= 2 * ks; t++) acc += taps.w[t] * row[t];
    s_h[i] = acc;
  }
  __syncthreads();
  // vertical pass
  float* out = pick5(job.out, blockIdx.z);
  for (int i = threadIdx.x; i < BT * BT; i += blockDim.x) {
    int j = i / BT, k = i % BT;
    int gy = y0 + j, gx = x0 + k;
    if (gx >= W || gy >= H) continue;
    float acc = 0.f;
    for (int t = 0; t <= 2 * ks; t++) acc += taps.w[t] * s_h[(j + t) * BT + k];
    out[(size_t)gy * W + gx] = acc;
  }
}

// Two floats in one 64-bit register.
__device__ __forceinline__ unsigned long long f2_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// The product of a tap per lane, rounded to nearest, and its sum: the
// reference rounds every multiply and every add.  A packed multiply feeding a
// packed add is not safe: ptxas contracts that pair into a fused multiply-add
// (one rounding).  The product is therefore fma(w, x, nz) with nz = {-0, -0}
// from a kernel parameter: adding -0 changes no product, not even a zero's
// sign, the compiler cannot know the value, and a fused multiply-add followed
// by an add has nothing left to contract.
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long w, unsigned long long x, unsigned long long nz) {
  unsigned long long p;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(w), "l"(x), "l"(nz));
  return p;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Separable blur of one plane for a compile-time tap radius KS, on strips of
// 128 columns.  A thread owns two columns and walks down the strip in batches
// of P = 2 KS + 1 rows:
//   1. the horizontal sums of the thread's two columns, packed, go to shared
//      memory of the thread's own;
//   2. the next batch's rows are on their way to shared memory (cp.async)
//      over this one's;
//   3. the vertical sums: P accumulators in registers, one per output row in
//      flight.  A new row is multiplied once by each of the KS + 1 distinct
//      weights (the kernel is symmetric) and the products are added to the
//      accumulators, each of which gets its taps in ascending order from 0,
//      the reference's order.  Unrolled over P rows, the accumulators rotate
//      by name.
// What bounds it: the FP32 pipe.  A packed operation takes the pipe twice as
// long as a scalar one, so it is the operations per output that count:
// 4 KS + 2 horizontally and 3 KS + 2 vertically (74 at KS = 10) against 97 in
// 64 x 64 tiles, whose halo the horizontal pass ran too.  One plane of 51 MP
// takes 206 us (tiles: 263 us); the pipe's time is 102 us, and register moves that
// line up the odd taps' pairs, chunk overlap and dependent adds take the rest.
// One staged batch, seven CTAs per SM: with a second one, on its way from the
// horizontal sums on, six fit, and the blurs of 51 MP took 1730 us, not 1647, of
// 26 MP at radius 7 790 us, not 733.  (Eight CTAs 1650 and 740 us, nine, which
// spill, 1607 and 764 us; 24 MP 790, 780 and 818 us.)
constexpr int BS_X = 128;  // output columns per strip
constexpr int BS_THREADS = BS_X / 2;

template <int KS>
struct BlurStrip {
  static constexpr int P = 2 * KS + 1;              // accumulators, rows per batch
  static constexpr int PAD = (KS + 3) & ~3;         // staged columns left and right of the strip
  static constexpr int C = BS_X + 2 * PAD;
  static constexpr int IN = (P + 1) * C;            // floats of the staged batch (one row more is read)
  static constexpr size_t SMEM = (size_t)(IN + (P + 1) * BS_X) * sizeof(float);
  // resident CTAs per SM: what the registers are bounded for, fewer where shared
  // memory (228 KB, 1 KB of it a CTA's own) holds fewer: six at tap radii 14 and 15
  static constexpr int PER_SM = 228 * 1024 / (SMEM + 1024) < 7 ? (int)(228 * 1024 / (SMEM + 1024)) : 7;
};
static_assert(BlurStrip<13>::PER_SM == 7 && BlurStrip<14>::PER_SM == 6 && BlurStrip<15>::PER_SM == 6, "blocks per SM");

__device__ __forceinline__ void cp_async(float* dst, const float* src, int bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

template <int KS>
__global__ void __launch_bounds__(BS_THREADS, BlurStrip<KS>::PER_SM) k_df_blur_strip(BlurJob job, GaussTaps taps, int W, int H, int batches,
                                                              const DfScalars* sc) {
  using B = BlurStrip<KS>;
  constexpr int P = B::P, C = B::C, PAD = B::PAD;
  extern __shared__ __align__(16) float sm_strip[];
  float* s_h = sm_strip + B::IN;  // [P + 1 rows][BS_X]
  const int tid = threadIdx.x;
  const float* __restrict__ in = pick5(job.in, blockIdx.z);
  float* __restrict__ out = pick5(job.out, blockIdx.z);
  const int mode = pick5(job.mode, blockIdx.z);
  const unsigned long long nz = job.nz;
  const int rows = batches * P - 2 * KS;  // output rows per strip chunk
  const int x0 = blockIdx.x * BS_X, y0 = blockIdx.y * rows, y1 = min(y0 + rows, H);
  const int x = x0 + 2 * tid;
  unsigned long long w[KS + 1];  // distinct weights, outermost first
#pragma unroll
  for (int t = 0; t <= KS; t++) w[t] = f2_pack(taps.w[t], taps.w[t]);
  const int step = mode == BS_GUIDE_LINEAR ? 3 : 1;  // the guide is read out of the RGB image
  const float* src = in + (mode == BS_GUIDE_LINEAR ? 1 : 0);
  // 16-byte copies where the plane's rows are aligned and the strip with its
  // halo lies inside the image; else sample by sample with the column clamped
  const bool wide = step == 1 && (W & 3) == 0 && x0 >= PAD && x0 + BS_X + PAD <= W;
  auto stage = [&](int b) {
    float* dst = sm_strip;
    const int yb = y0 - KS + b * P;
    if (wide) {
      for (int i = tid; i < P * (C / 4); i += BS_THREADS) {
        const int r = i / (C / 4), q = i - r * (C / 4);
        cp_async(dst + r * C + 4 * q, src + (size_t)min(max(yb + r, 0), H - 1) * W + x0 - PAD + 4 * q, 16);
      }
    } else {
#pragma unroll
      for (int k = 0; k < (C + BS_THREADS - 1) / BS_THREADS; k++) {
        const int q = tid + k * BS_THREADS;
        const int gx = min(max(x0 - PAD + q, 0), W - 1) * step;
        if (q < C)
          for (int r = 0; r < P; r++)
            cp_async(dst + r * C + q, src + (size_t)min(max(yb + r, 0), H - 1) * W * step + gx, 4);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const float inv = mode == BS_PLANE_EDGE_NORM ? 1.f / smax(sc->max_edge, 1e-6f) : 0.f;
  const bool vec = (W & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;

  unsigned long long acc[P];
#pragma unroll
  for (int j = 0; j < P; j++) acc[j] = 0ull;
  stage(0);
  for (int b = 0; b < batches; b++) {
    const int yb = y0 - KS + b * P;  // image row of the batch's first row
    if (yb - KS >= y1) break;
    float* cur = sm_strip;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (mode != BS_PLANE) {
      for (int i = tid; i < P * C; i += BS_THREADS) cur[i] = mode == BS_GUIDE_LINEAR ? smax(cur[i], 0.f) : cur[i] * inv;
      __syncthreads();
    }
    // horizontal sums of rows j, j + 1 at columns 2 tid, 2 tid + 1 (row P, read
    // with row P - 1, is not used)
#pragma unroll 1
    for (int j = 0; j < P; j += 2) {
      unsigned long long h[2];
      float e[2][P + 2];
      constexpr int O = PAD - KS;  // the window starts O columns into the pair
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const float2* q = reinterpret_cast<const float2*>(cur + (j + k) * C + 2 * tid + (O & ~1));
#pragma unroll
        for (int i = 0; i < (P + 1 + (O & 1) + 1) / 2; i++) {
          const float2 f = q[i];
          if (2 * i - (O & 1) >= 0) e[k][2 * i - (O & 1)] = f.x;
          if (2 * i + 1 - (O & 1) <= P) e[k][2 * i + 1 - (O & 1)] = f.y;
        }
        h[k] = 0ull;
      }
#pragma unroll
      for (int t = 0; t < P; t++) {
        const unsigned long long wt = w[t <= KS ? t : 2 * KS - t];
#pragma unroll
        for (int k = 0; k < 2; k++) h[k] = f2_add(h[k], f2_mul(wt, f2_pack(e[k][t], e[k][t + 1]), nz));
      }
#pragma unroll
      for (int k = 0; k < 2; k++)
        *reinterpret_cast<unsigned long long*>(&s_h[(j + k) * BS_X + 2 * tid]) = h[k];
    }
    __syncthreads();  // every thread has read the batch
    if (b + 1 < batches) stage(b + 1);
    // vertical sums (the thread reads only what it wrote)
#pragma unroll
    for (int s = 0; s < P; s++) {
      const unsigned long long v = *reinterpret_cast<const unsigned long long*>(&s_h[s * BS_X + 2 * tid]);
      unsigned long long m[KS + 1];
#pragma unroll
      for (int t = 0; t <= KS; t++) m[t] = f2_mul(w[t], v, nz);
      // accumulator (s + j) % P belongs to the output row KS - j above this
      // one and gets tap 2 KS - j; the last one starts here
#pragma unroll
      for (int j = 0; j < P; j++) {
        const int t = 2 * KS - j;
        unsigned long long& A = acc[(s + j) % P];
        A = f2_add(j == 2 * KS ? 0ull : A, m[t <= KS ? t : 2 * KS - t]);
      }
      const int o = yb + s - KS;
      if (o >= y0 && o < y1 && x < W) {
        float a, c;
        f2_unpack(acc[s], a, c);
        float* d = out + (size_t)o * W + x;
        if (vec) {
          *reinterpret_cast<float2*>(d) = make_float2(a, c);
        } else {
          d[0] = a;
          if (x + 1 < W) d[1] = c;
        }
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int KS>
lre_status run_blur_strip(Context* c, const BlurJob& job, const GaussTaps& taps, int W, int H, const DfScalars* sc) {
  using B = BlurStrip<KS>;
  LRE_CUDA_TRY(c, cudaFuncSetAttribute(k_df_blur_strip<KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)B::SMEM));
  // Batches per chunk: a chunk's first 2 KS rows produce nothing, so tall
  // chunks, halved while the grid has less than two waves of resident CTAs (seven
  // per SM at most tap radii).  Where even halves leave fewer than that,
  // what takes the fewest batch steps over all waves, a nearly empty last one
  // counting as much as a full one.  With six CTAs per SM the three blurs of
  // 1.9 MP took 104 us halved and 88 us so (82 us with seven); those of 24 and
  // 51 MP 839 and 1732 us halved and 859 and 1774 us by waves, whose CTAs don't
  // run in step when there are many.
  int batches = c->tune.blur_tile == 64 ? 32 : 16;
  const int tallest = batches;
  const int strips = (W + BS_X - 1) / BS_X;
  auto chunks = [&](int n) { return (H + n * B::P - 2 * KS - 1) / (n * B::P - 2 * KS); };
  auto ctas = [&](int n) { return (long long)strips * chunks(n) * job.np; };
  const long long places = (long long)B::PER_SM * c->sm_count;
  while (batches > 2 && ctas(batches) < 2 * places) batches /= 2;
  if (batches <= 4) {
    double least = 1e300;
    for (int n = 2; n <= tallest; n++) {
      const double cost = (double)((ctas(n) + places - 1) / places) * (n + 0.5);
      if (cost <= least) {
        least = cost;
        batches = n;
      }
    }
  }
  const dim3 grid((unsigned)strips, (unsigned)chunks(batches), (unsigned)job.np);
  k_df_blur_strip<KS><<<grid, BS_THREADS, B::SMEM, c->stream>>>(job, taps, W, H, batches, sc);
  count_launch(c);
  return check_launch(c, "defringe blur");
}

// ---------------------------------------------------------------- K3
struct DfConst {
  float edge_thr, chroma_thr, strength, green_scale;
  int green;
};

// smoothstep with edges that are the same for every pixel.  The quotient
// (x - e0) / d is formed from the reciprocal y = RN(1 / d), known before the
// launch, by Markstein's scheme (IBM J. Res. Dev. 34, 1990): a product, then
// two corrections by the exact residual, the last of which rounds the true
// quotient: with y correctly rounded and q within an ulp, RN(q + r y) is the
// correctly rounded quotient.  The numerator is clamped to [0, d] first, which
// gives the same t as clamping the quotient to [0, 1] (NaN stays NaN), so
// nothing overflows, and x - e0 is 0 or at least half an ulp of e0, so no
// residual underflows.  12 instructions against about 22 with an IEEE
// division.  FAST needs d and e0 in [2^-60, 2^60]; otherwise (a zero or
// negative threshold) the division itself runs.
struct DfEdge {
  float e0, e1, d, y;
};
template <bool FAST>
__device__ __forceinline__ float ss(const DfEdge& E, float x) {
  if (!FAST) return ssmooth(E.e0, E.e1, x);
  float n = x - E.e0;
  asm("max.NaN.f32 %0, %0, 0f00000000;" : "+f"(n));
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(n) : "f"(E.d));
  float q = n * E.y;
  q = __fmaf_rn(__fmaf_rn(-E.d, q, n), E.y, q);
  q = __fmaf_rn(__fmaf_rn(-E.d, q, n), E.y, q);
  return q * q * (3.0f - 2.0f * q);
}
// Edges written as literals: the compiler folds d and y.
__device__ __forceinline__ float ssl(float e0, float e1, float x) {
  const float d = e1 - e0;
  return ss<true>(DfEdge{e0, e1, d, 1.0f / d}, x);
}

// The edges that depend on the call's parameters, in the reference's
// expressions (factor * threshold * inv_s), formed on the host.
enum DfEdgeId : int {
  DE_CORE, DE_CORE_RAW, DE_LOW, DE_LOW_RAW, DE_BRIGHT, DE_CHROMA, DE_HUE, DE_RP_HUE, DE_ABS, DE_LOWC, DE_SOFT, DE_GATE,
  DE_PEAK, DE_HALO, DE_SOLO, DE_SEED_SOLO, DE_N
};
struct DfTab {
  DfEdge e[DE_N];
  float inv_s, mask_cutoff;
  float soften;      // 1 - 0.86 smoothstep(0.22, 0.40, chroma_thr)
  float solo_enable; // smoothstep(1.25, 3, strength)
  float release, surface;  // smoothstep(2, 6, strength), smoothstep(3, 8, strength)
};

// Fringe-support seed of pixel i (core/cpu_accelerator.cpp:4158-4205).
template <bool FAST>
__device__ __forceinline__ float support_at(const float* __restrict__ src, size_t i, const DfPlanes& P, const DfTab& T,
                                            bool enable_green) {
  const float rg = P.lrg[i];
  const float bgr = P.lbg[i];
  const float dr = rg - P.blrg[i];
  const float db = bgr - P.blbg[i];
  const float* s = src + i * 3;
  const float r0 = smax(s[0], 0.f);
  const float g0 = smax(s[1], 0.f);
  const float b0 = smax(s[2], 0.f);
  const float blur_guide = P.bg[i];
  const float purple_excess = smin(smax(0.f, dr), smax(0.f, db));
  const float denom_support = smax(blur_guide, 0.05f);
  const float g_over_min_support = smax(0.f, g0 - smin(r0, b0)) / denom_support;
  const float green_dom_support = ssl(0.010f, 0.060f, g_over_min_support);
  const float green_excess = smax(smax(0.f, -dr), smax(0.f, -db)) * green_dom_support;
  const bool is_purple = purple_excess >= green_excess;
  const float excess_support = is_purple ? purple_excess : green_excess;
  const float min_dir = is_purple ? smax(0.f, smin(rg, bgr)) : smax(0.f, smin(-rg, -bgr));
  const float max_dir = is_purple ? smax(1e-4f, smax(rg, bgr)) : smax(1e-4f, smax(-rg, -bgr));
  const float balance = min_dir / max_dir;
  const float c_edge = ss<FAST>(T.e[DE_CORE], P.be[i]) *
                       ss<FAST>(T.e[DE_CORE_RAW], P.ber[i]);
  const float c_bright = ss<FAST>(T.e[DE_BRIGHT], blur_guide);
  const float c_chroma = ss<FAST>(T.e[DE_CHROMA], excess_support);
  const float red_strength = smax(0.f, r0 - smax(g0, b0)) / smax(r0, 1e-4f);
  const float red_blue_balance = b0 / smax(r0, 1e-4f);
  const float blue_lift = smax(0.f, b0 - g0) / smax(r0 - g0, 1e-4f);
  const float red_purple = smax(ssl(0.55f, 0.78f, red_blue_balance), ssl(0.16f, 0.34f, blue_lift));
  const float red_purple_hue_signal = ssl(0.50f, 0.72f, red_blue_balance) * ssl(0.24f, 0.42f, blue_lift);
  const float balanced_hue = ss<FAST>(T.e[DE_HUE], min_dir) * ssl(0.35f, 0.75f, balance);
  const float red_purple_hue = is_purple ? smin(1.f, red_purple_hue_signal * 1.50f) *
                                               ss<FAST>(T.e[DE_RP_HUE], min_dir) *
                                               ssl(0.18f, 0.58f, balance)
                                         : 0.f;
  const float c_hue = smax(balanced_hue, red_purple_hue);
  const float natural_guard = 1.f - ssl(0.08f, 0.25f, red_strength) * (1.f - red_purple);
  const float green_enable = (enable_green || is_purple) ? 1.f : 0.f;
  return c_edge * c_bright * c_hue * c_chroma * natural_guard * green_enable;
}

// K3 per pixel, four consecutive pixels per thread.  A pixel whose blurred
// edge planes are at or below the lower smoothstep edges has an edge factor of
// exactly 0 and so a seed of 0: where all four are such, every log ratio of the
// image is finite and every pair of edges is apart (FAST; a chroma threshold of 0
// makes 0 / 0 of a pixel without excess), so no factor is NaN, the other planes
// are not read.
// At 51 MP 258 us; fused behind the blur of the five planes it had taken
// about 880 us of that kernel's 2200.
template <bool FAST>
__global__ void __launch_bounds__(256) k_df_support(const float* __restrict__ src, size_t n, DfPlanes P, DfConst k,
                                                    DfTab T, const DfScalars* sc) {
  const bool enable_green = k.green != 0;
  const float e0_edge = T.e[DE_CORE].e0, e0_raw = T.e[DE_CORE_RAW].e0;
  const bool can_skip = FAST && sc->nonfinite == 0 && k.edge_thr > 0.f;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (n + 3) / 4; q += stride) {
    const size_t i = q * 4;
    float be[4], ber[4], fs[4];
    if (i + 4 <= n) {
      ld4(P.be + i, be);
      ld4(P.ber + i, ber);
    } else {
      for (int t = 0; t < 4; t++) {
        be[t] = i + t < n ? P.be[i + t] : 0.f;
        ber[t] = i + t < n ? P.ber[i + t] : 0.f;
      }
    }
    unsigned need = 0;
#pragma unroll
    for (int t = 0; t < 4; t++)
      if (i + t < n && !(can_skip && (be[t] <= e0_edge || ber[t] <= e0_raw))) need |= 1u << t;
#pragma unroll
    for (int t = 0; t < 4; t++) fs[t] = 0.f;
#pragma unroll
    for (int t = 0; t < 4; t++)
      if (need >> t & 1u) fs[t] = support_at<FAST>(src, i + t, P, T, enable_green);
    if (i + 4 <= n) {
      st4(P.fs + i, fs);
    } else {
      for (int t = 0; t < 4; t++)
        if (i + t < n) P.fs[i + t] = fs[t];
    }
  }
}

// ---------------------------------------------------------------- K5
constexpr int LT = 32;   // line-link output tile
constexpr int LH = 14;   // max step along a line
constexpr int LE = LT + 2 * LH;

constexpr int LN_THREADS = 320;
static_assert(LE % (LN_THREADS / 32) == 0 && LE <= 64, "whole rows, two columns to a lane");
constexpr int LPAD = 16;  // floats around the sources: runs that begin or end beside the tile read up to 4 beyond

// A direction's share of a pixel's line support, from the largest source along
// the line on either side.
template <int TX, int TY>
__device__ __forceinline__ void line_dir(const float* s_fs, int c, float along, float& best) {
  // along == 0 contributes 0 * thin (thin in [0, 1], or NaN which
  // std::max ignores) to a running max that is already >= 0
  if (along == 0.f) return;
  constexpr int NX = -TY, NY = TX;  // across-direction normal
  const float across = smax(s_fs[c + (NY * LE + NX) * 2], s_fs[c - (NY * LE + NX) * 2]);
  const float thin = 1.f - ssmooth(along * 0.45f, along * 0.95f, across);
  best = smax(best, along * thin);
}

// Four neighbouring pixels of a line share most of their windows: v holds the
// line from STEPS before the first to STEPS behind the last.  The maximum starts
// at 0 and the samples are finite or NaN: std::max(along, v) then equals
// fmaxf(along, v) (neither ever yields NaN) in whatever order.
template <int STEPS>
__device__ __forceinline__ void line_windows(const float (&v)[2 * STEPS + 4], float (&along)[4]) {
  float back = 0.f, ahead = 0.f;
#pragma unroll
  for (int k = 3; k < STEPS; k++) back = fmaxf(back, v[k]);
#pragma unroll
  for (int k = STEPS + 4; k <= 2 * STEPS; k++) ahead = fmaxf(ahead, v[k]);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    float a = fmaxf(back, ahead);
#pragma unroll
    for (int k = j; k < 3; k++) a = fmaxf(a, fmaxf(v[k], v[k + STEPS + 1]));
#pragma unroll
    for (int k = 0; k < j; k++) a = fmaxf(a, fmaxf(v[STEPS + k], v[2 * STEPS + 1 + k]));
    along[j] = a;
  }
}

// One direction over the tile, a thread per run of four pixels along it,
// (x + DX j, y + DY j); (TX, TY) is the reference's sense of the direction.
// Runs that leave the tile sideways hold fewer pixels of it.
template <int DX, int DY, int STEPS, int TX, int TY>
__device__ __forceinline__ void line_runs(const float* s_ls, const float* s_fs, float* s_best) {
  constexpr int AX = DX < 0 ? -DX : DX, NS = LT + 3 * AX, STEP = DY * LE + DX;
  for (int i = threadIdx.x; i < 8 * NS; i += LN_THREADS) {
    const int g = i / NS, x = i - g * NS - (DX > 0 ? 3 * AX : 0);
    const int y = DY == 1 ? 4 * g : 8 * (g >> 1) + (g & 1);
    const int c = (y + LH) * LE + x + LH;
    float v[2 * STEPS + 4], along[4];
#pragma unroll
    for (int k = 0; k < 2 * STEPS + 4; k++) v[k] = s_ls[c + (k - STEPS) * STEP];
    line_windows<STEPS>(v, along);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (AX && (unsigned)(x + DX * j) >= (unsigned)LT) continue;
      float& best = s_best[(y + DY * j) * LT + x + DX * j];
      line_dir<TX, TY>(s_fs, c + j * STEP, along[j], best);
    }
  }
  __syncthreads();
}

// K5: line-linked support, then the solo seeds.  Bound by instructions and, a
// little, by the wait for the staged rows:
// * the eight directions' maxima are formed for four pixels of a line at a time
//   (of a pixel each: 160 loads and 160 maxima), with enough threads that every
//   direction's runs, up to 304 of a tile, take one turn;
// * a warp stages whole rows, all of its loads in flight (an element's place by
//   two divisions and four clamps, two in flight: about 105 instructions a pixel);
// * a pixel whose blurred edge planes are at or below the lower smoothstep edges
//   has solo seeds of exactly 0 where no factor is NaN (K3's rule), without the
//   two exponentials in double.
// 51 MP: 1223 us before, 768 us; 26 MP odd 664 and 470 us; 1.9 MP 55 and 45 us.
// (256 threads 926 us at 51 MP; two rows in flight 853 us; five CTAs per SM, which
// spill, 769 us.)
template <bool FAST>
__global__ void __launch_bounds__(LN_THREADS, 4)
    k_df_line(const float* __restrict__ src, int W, int H, DfPlanes P, DfConst k, DfTab T, const DfScalars* sc) {
  __shared__ __align__(16) float s_src[LPAD + LE * LE + LPAD];
  __shared__ float s_fs[LE * LE];
  __shared__ __align__(16) float s_best[LT * LT];
  __shared__ int s_any;
  float* s_ls = s_src + LPAD;
  const int x0 = blockIdx.x * LT, y0 = blockIdx.y * LT;
  if (threadIdx.x == 0) s_any = 0;
  __syncthreads();
  int any = 0;
  {
    const int lane = threadIdx.x & 31, gx0 = min(max(x0 - LH + lane, 0), W - 1), gx1 = min(x0 - LH + lane + 32, W - 1);
#pragma unroll
    for (int j = 0; j < LE / (LN_THREADS / 32); j++) {
      const int r = (threadIdx.x >> 5) + j * (LN_THREADS / 32);
      const size_t gr = (size_t)min(max(y0 - LH + r, 0), H - 1) * W;
      const float f0 = P.fs[gr + gx0], b0 = P.bfs[gr + gx0];
      const float f1 = P.fs[gr + gx1], b1 = P.bfs[gr + gx1];
      const float l0 = smax(f0, b0 * 0.55f), l1 = smax(f1, b1 * 0.55f);
      s_fs[r * LE + lane] = f0;
      s_ls[r * LE + lane] = l0;
      any |= l0 != 0.f;
      if (lane < LE - 32) {
        s_fs[r * LE + lane + 32] = f1;
        s_ls[r * LE + lane + 32] = l1;
        any |= l1 != 0.f;
      }
    }
  }
  if (__any_sync(0xffffffffu, any) && (threadIdx.x & 31) == 0) s_any = 1;
  __syncthreads();
  // a tile whose line sources are all zero has every `along` zero, so every
  // line-linked support value is exactly 0
  const bool tile_active = s_any != 0;
  if (tile_active) {
    // directions and step counts of core/cpu_accelerator.cpp:4290-4318; along
    // a row first, from vector loads, which sets every pixel's value
    if (threadIdx.x < 256) {
      const int y = threadIdx.x >> 3, x = (threadIdx.x & 7) * 4, c = (y + LH) * LE + x + LH;
      float v[32], along[4], best[4];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const float4 t = *reinterpret_cast<const float4*>(s_ls + c - LH + 4 * q);
        v[4 * q] = t.x;
        v[4 * q + 1] = t.y;
        v[4 * q + 2] = t.z;
        v[4 * q + 3] = t.w;
      }
      line_windows<14>(v, along);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        best[j] = 0.f;
        line_dir<1, 0>(s_fs, c + j, along[j], best[j]);
      }
      *reinterpret_cast<float4*>(s_best + y * LT + x) = make_float4(best[0], best[1], best[2], best[3]);
    }
    __syncthreads();
    line_runs<0, 1, 14, 0, 1>(s_ls, s_fs, s_best);
    line_runs<1, 1, 14, 1, 1>(s_ls, s_fs, s_best);
    line_runs<-1, 1, 14, 1, -1>(s_ls, s_fs, s_best);
    line_runs<2, 1, 6, 2, 1>(s_ls, s_fs, s_best);
    line_runs<1, 2, 6, 1, 2>(s_ls, s_fs, s_best);
    line_runs<-2, 1, 6, 2, -1>(s_ls, s_fs, s_best);
    line_runs<-1, 2, 6, 1, -2>(s_ls, s_fs, s_best);
  }
  const float e0_edge = T.e[DE_CORE].e0, e0_raw = T.e[DE_CORE_RAW].e0;
  const bool can_skip = FAST && sc->nonfinite == 0 && k.edge_thr > 0.f;
  for (int i = threadIdx.x; i < LT * LT; i += blockDim.x) {
    int ly = i / LT, lx = i % LT;
    int y = y0 + ly, x = x0 + lx;
    if (x >= W || y >= H) continue;
    const size_t gi = (size_t)y * W + x;
    const float best = tile_active ? s_best[i] : 0.f;
    const float be = P.be[gi], ber = P.ber[gi];
    P.lfs[gi] = best;
    if (can_skip && (be <= e0_edge || ber <= e0_raw)) {
      P.srs[gi] = 0.f;
      P.sbs[gi] = 0.f;
      continue;
    }
    const float* s = src + gi * 3;
    const float s0 = s[0], s1 = s[1], s2 = s[2];
    const float blur_guide = P.bg[gi];
    const float blrg = P.blrg[gi], blbg = P.blbg[gi];
    const float bfs = P.bfs[gi];

    // solo seeds (core/cpu_accelerator.cpp:4325-4374)
    const float g = smax(s1, 0.f);
    const float target_r = g * exp_cr(blrg);
    const float target_b = g * exp_cr(blbg);
    const float solo_r = smax(0.f, s0 - target_r) / smax(blur_guide, 0.05f);
    const float solo_b = smax(0.f, s2 - target_b) / smax(blur_guide, 0.05f);
    const float linked_fringe = ssl(0.004f, 0.045f, smax(bfs, best * 0.90f));
    const float c_edge_solo = ss<FAST>(T.e[DE_CORE], be) *
                              ss<FAST>(T.e[DE_CORE_RAW], ber);
    const float c_bright_solo = ss<FAST>(T.e[DE_BRIGHT], blur_guide);
    const float solo_enable = T.solo_enable;
    const float r0 = smax(s0, 0.f);
    const float g0 = smax(s1, 0.f);
    const float b0 = smax(s2, 0.f);
    const float red_strength_solo = smax(0.f, r0 - smax(g0, b0)) / smax(r0, 1e-4f);
    const float solo_red_guard = 1.f - 0.90f * ssl(0.12f, 0.32f, red_strength_solo);
    P.srs[gi] = solo_enable * c_edge_solo * c_bright_solo * linked_fringe * solo_red_guard *
                ss<FAST>(T.e[DE_SEED_SOLO], solo_r);
    P.sbs[gi] = solo_enable * c_edge_solo * c_bright_solo *
                ss<FAST>(T.e[DE_SEED_SOLO], solo_b);
  }
}

// ---------------------------------------------------------------- K7
// Constants of the main pass (core/cpu_accelerator.cpp:4376-4706), formed
// once per thread.
struct DfMainK {
  float mask_cutoff, scene_highlight_gate, strength, green_strength_scale;
  float e0_edge, e0_raw;
  bool enable_green, can_skip;
};

// The eleven planes the main pass reads at one pixel.
struct DfPx {
  float be, ber, srb, sbb, bg, blrg, blbg, bfs, lfs, lrg, lbg;
};

// Pixels that provably keep their input: with green correction off, either
// edge factor at or below its lower smoothstep edge zeroes both edge weights
// (the other factor is finite, or NaN, and a NaN mask never passes the
// cutoff), so no ratio/direct correction applies; zero solo blurs make the
// solo masks zero.  The output is then the input whatever the other planes
// hold, so those pixels need 4 planes instead of 11 and skip the rest.
__device__ __forceinline__ bool df_keeps_input(const DfMainK& K, float be, float ber, float srb, float sbb) {
  return K.can_skip && (be <= K.e0_edge || ber <= K.e0_raw) && srb == 0.f && sbb == 0.f;
}

// The correction of one pixel (s0, s1, s2) -> (d0, d1, d2).
template <bool FAST>
__device__ __forceinline__ void df_main_px(float s0, float s1, float s2, const DfPx& v, const DfMainK& K, const DfTab& T, float& d0,
                                           float& d1, float& d2) {
  const float mask_cutoff = K.mask_cutoff;
  const float scene_highlight_gate = K.scene_highlight_gate;
  const bool enable_green = K.enable_green;
  const float strength = K.strength;
  const float green_strength_scale = K.green_strength_scale;
  d0 = s0;
  d1 = s1;
  d2 = s2;
  const float blur_guide = v.bg;
  const float blur_log_rg = v.blrg;
  const float blur_log_bg = v.blbg;
  const float blur_fringe_support = v.bfs;
  const float line_support = v.lfs;

  const float rg = v.lrg;
  const float bg = v.lbg;
  const float dr = rg - blur_log_rg;
  const float db = bg - blur_log_bg;
  const float r0 = smax(s0, 0.f);
  const float g0 = smax(s1, 0.f);
  const float b0 = smax(s2, 0.f);
  const float rb_avg_pre = 0.5f * (r0 + b0);
  const float purple_r = smax(0.f, dr);
  const float purple_b = smax(0.f, db);
  const float green_r = smax(0.f, -dr);
  const float green_b = smax(0.f, -db);
  const float purple_excess = smin(purple_r, purple_b);
  const float denom = smax(blur_guide, 0.05f);
  const float g_over_min = smax(0.f, g0 - smin(r0, b0)) / denom;
  const float green_dom = ssl(0.010f, 0.060f, g_over_min);
  const float green_excess = smax(green_r, green_b) * green_dom;
  const bool is_purple = purple_excess >= green_excess;
  const float excess = is_purple ? purple_excess : green_excess;
  const float min_dir = is_purple ? smax(0.f, smin(rg, bg)) : smax(0.f, smin(-rg, -bg));
  const float max_dir = is_purple ? smax(1e-4f, smax(rg, bg)) : smax(1e-4f, smax(-rg, -bg));
  const float balance = min_dir / max_dir;
  const float c_edge_core = ss<FAST>(T.e[DE_CORE], v.be) *
                            ss<FAST>(T.e[DE_CORE_RAW], v.ber);
  const float c_edge_low = ss<FAST>(T.e[DE_LOW], v.be) *
                           ss<FAST>(T.e[DE_LOW_RAW], v.ber);
  const float linked_fringe = ssl(0.004f, 0.045f, smax(blur_fringe_support, line_support * 0.90f));
  const float c_bright = ss<FAST>(T.e[DE_BRIGHT], blur_guide);
  const float c_chroma = ss<FAST>(T.e[DE_CHROMA], excess);
  const float red_blue_balance_hue = b0 / smax(r0, 1e-4f);
  const float blue_lift_hue = smax(0.f, b0 - g0) / smax(r0 - g0, 1e-4f);
  const float red_purple_hue_signal = ssl(0.50f, 0.72f, red_blue_balance_hue) * ssl(0.24f, 0.42f, blue_lift_hue);
  const float balanced_hue = ss<FAST>(T.e[DE_HUE], min_dir) * ssl(0.35f, 0.75f, balance);
  const float red_purple_hue_gate = is_purple ? smin(1.f, red_purple_hue_signal * 1.50f) *
                                                    ss<FAST>(T.e[DE_RP_HUE], min_dir) *
                                                    ssl(0.18f, 0.58f, balance)
                                              : 0.f;
  const float green_unbalanced_hue =
      (enable_green && !is_purple) ? ss<FAST>(T.e[DE_RP_HUE], max_dir) : 0.f;
  const float c_hue = smax(balanced_hue, smax(red_purple_hue_gate, green_unbalanced_hue));
  const float rb_avg = rb_avg_pre;
  const float purple_abs = smin(smax(0.f, r0 - g0), smax(0.f, b0 - g0)) / smax(blur_guide, 0.05f);
  const float green_abs_base = smax(0.f, g0 - rb_avg) / smax(blur_guide, 0.05f);
  const float green_abs_alt = smax(0.f, g0 - smin(r0, b0)) / smax(blur_guide, 0.05f);
  const float green_abs = smax(green_abs_base, 0.55f * green_abs_alt);
  const bool abs_is_purple = purple_abs >= green_abs;
  const float abs_excess = abs_is_purple ? purple_abs : green_abs;
  const float c_abs = ss<FAST>(T.e[DE_ABS], abs_excess);
  const float low_contrast_color =
      ss<FAST>(T.e[DE_LOWC], abs_excess);
  const float green_soft_edge_boost =
      (enable_green && !is_purple) ? c_edge_low * ss<FAST>(T.e[DE_SOFT], max_dir) : 0.f;
  const float c_edge = smax(c_edge_core, smax(c_edge_low * linked_fringe * 1.45f,
                                              smax(c_edge_low * low_contrast_color * 0.35f, green_soft_edge_boost)));
  const float ratio_mask = c_edge * c_bright * c_hue * c_chroma;
  const float direct_mask = c_edge * c_bright * c_hue * c_abs;
  const bool use_direct = direct_mask > ratio_mask;
  float mask = smax(ratio_mask, direct_mask) * scene_highlight_gate;
  const bool correct_purple = use_direct ? abs_is_purple : is_purple;
  float local_gate = 0.f;
  if (correct_purple) {
    local_gate = ss<FAST>(T.e[DE_GATE], purple_abs);
    mask *= local_gate;
  } else {
    local_gate = ss<FAST>(T.e[DE_GATE], green_abs);
    if (enable_green) {
      const float peak_chroma_signal =
          ss<FAST>(T.e[DE_PEAK], green_abs);
      const float peak_neighbourhood = ssl(0.005f, 0.030f, blur_fringe_support);
      const float green_peak_mask = peak_chroma_signal * peak_neighbourhood * c_bright * c_hue;
      mask = smax(mask, green_peak_mask * scene_highlight_gate);
    }
    const float green_highlight_protect = 1.f - 0.85f * ssl(0.62f, 0.88f, blur_guide);
    const float rb_to_green = rb_avg / smax(g0, 1e-4f);
    const float natural_green_highlight = ssl(0.22f, 0.46f, rb_to_green) * ssl(0.30f, 0.55f, g0);
    const float natural_green_suppress = 1.f - 0.99f * natural_green_highlight;
    const float natural_green_suppress_sq = natural_green_suppress * natural_green_suppress;
    const float green_halo_strength =
        ss<FAST>(T.e[DE_HALO], green_abs);
    const float green_gain_base = enable_green ? 0.60f : 0.35f;
    const float green_gain_slope = enable_green ? 1.10f : 0.95f;
    const float green_gain = green_gain_base + green_gain_slope * green_halo_strength;
    const float min_ratio_ref = smin(blur_log_rg, blur_log_bg);
    const float green_neighbour = ssl(0.02f, 0.10f, smax(0.f, -min_ratio_ref));
    const float src_max = smax(r0, smax(g0, b0));
    const float src_min = smin(r0, smin(g0, b0));
    const float src_chroma = src_max - src_min;
    const float src_sat = src_chroma / smax(src_max, 1e-4f);
    const float whiteish = 1.f - ssl(0.05f, 0.13f, src_sat);
    const float foliage_guard =
        green_neighbour * whiteish * ssl(0.35f, 0.75f, blur_guide) * (1.f - green_halo_strength);
    const float strength_release = enable_green ? T.release : 0.f;
    const float green_line_evidence = ssl(0.004f, 0.030f, line_support) *
                                      ssl(0.20f, 0.55f, green_halo_strength) * ssl(0.05f, 0.15f, src_sat);
    const float not_natural_green = 1.f - natural_green_highlight;
    const float guard_release = strength_release * green_line_evidence * not_natural_green;
    const float released_highlight_protect = green_highlight_protect + (1.f - green_highlight_protect) * guard_release;
    const float released_natural_suppress =
        natural_green_suppress_sq + (1.f - natural_green_suppress_sq) * guard_release;
    const float foliage_term = 1.f - 0.999f * foliage_guard;
    const float released_foliage_term = foliage_term + (1.f - foliage_term) * guard_release;
    mask *= local_gate * green_gain * released_highlight_protect * released_natural_suppress * released_foliage_term;
    const float line_kill_evidence = ssl(0.04f, 0.15f, line_support);
    const float natural_blob =
        sqrtf(smax(0.f, natural_green_highlight)) * (1.f - line_kill_evidence) * green_neighbour;
    mask *= 1.f - 0.999f * natural_blob;
    if (!enable_green) mask = 0.f;
  }

  bool skip_rest = false;
  if (mask > mask_cutoff) {
    const float g = smax(s1, 0.f);
    const float red_strength = smax(0.f, r0 - smax(g0, b0)) / smax(r0, 1e-4f);
    const float red_blue_balance = b0 / smax(r0, 1e-4f);
    const float blue_lift = smax(0.f, b0 - g0) / smax(r0 - g0, 1e-4f);
    const float red_purple_balance = ssl(0.55f, 0.78f, red_blue_balance);
    const float red_purple_lift = ssl(0.16f, 0.34f, blue_lift);
    const float red_purple = smax(red_purple_balance, red_purple_lift);
    const float red_strength_guard = ssl(0.08f, 0.25f, red_strength);
    float red_purple_context = 0.f;
    float contextual_red_purple = 0.f;
    float red_magenta_surface = 0.f;
    if (red_purple > 0.50f) {
      red_purple_context = linked_fringe;
      contextual_red_purple = red_purple * red_purple_context;
      if (red_purple_context < 0.20f && red_strength_guard < 0.50f && red_purple > 0.50f) {
        red_magenta_surface = ssl(0.02f, 0.12f, purple_abs) * (1.f - red_purple_context);
      }
    }
    float neutral_gray_surface = 0.f;
    if (strength > 3.f && red_purple_context > 0.80f && line_support > 0.012f && red_strength_guard < 0.98f &&
        blue_lift > 1.10f && red_blue_balance > 0.82f && purple_abs > 0.015f) {
      const float neutral_gray_edge = ssl(1.10f, 1.80f, blue_lift) * ssl(0.82f, 1.05f, red_blue_balance) *
                                      (1.f - red_strength_guard);
      neutral_gray_surface = neutral_gray_edge * ssl(0.015f, 0.08f, purple_abs) * T.surface;
    }
    const float red_object_strength = smax(red_strength_guard, red_magenta_surface);
    const float natural_warm_guard_base = 1.f - red_object_strength * (1.f - contextual_red_purple);
    const float natural_warm_guard_sq =
        natural_warm_guard_base * natural_warm_guard_base * natural_warm_guard_base * natural_warm_guard_base;
    const float natural_warm_guard = natural_warm_guard_sq * natural_warm_guard_sq;
    const float line_purple_relief = ssl(0.012f, 0.06f, line_support) * ssl(0.10f, 0.24f, blue_lift);
    const float red_object_guard = ssl(0.55f, 0.90f, red_object_strength);
    const float linked_override = linked_fringe * 1.05f * (1.f - 0.85f * red_object_guard);
    const float line_override = line_purple_relief * (1.f - 0.85f * red_object_guard);
    const bool force_warm_guard = (red_object_guard > 0.75f) && (linked_fringe < 0.65f) && (line_purple_relief < 0.45f);
    const float warm_protect = correct_purple
                                   ? (force_warm_guard ? natural_warm_guard
                                                       : smax(natural_warm_guard, smax(linked_override, line_override)))
                                   : 1.f;
    const float red_without_support =
        ssl(0.22f, 0.45f, red_strength) * (1.f - ssl(0.02f, 0.12f, blur_fringe_support));
    const float protect = correct_purple ? red_without_support : 0.f;
    const float smooth_mask = ssmooth(mask_cutoff, mask_cutoff * 5.0f, mask);
    const float threshold_soften = T.soften;
    const float src_max = smax(r0, smax(g0, b0));
    const float src_min = smin(r0, smin(g0, b0));
    const float src_chroma = src_max - src_min;
    const float src_sat = src_chroma / smax(src_max, 1e-4f);
    const float neutral_guard_base = ssl(0.008f, 0.030f, src_sat);
    const float neutral_guard = 1.f - (1.f - neutral_guard_base) * ssl(0.35f, 0.80f, red_object_strength);
    float amount = sclamp(smooth_mask * strength * 1.90f * (1.f - protect) * warm_protect * neutral_guard *
                              threshold_soften,
                          0.f, 1.f);
    const float warm_edge_surface = ssl(0.006f, 0.035f, purple_abs) * ssl(0.25f, 0.65f, red_purple) *
                                    ssl(0.15f, 0.65f, red_purple_context) * (1.f - 0.55f * red_strength_guard) *
                                    T.surface;
    const float safe_surface = smax(neutral_gray_surface, warm_edge_surface);
    if (correct_purple && safe_surface > 1e-4f) {
      const float safe_amount_cap = 1.f - 0.99f * safe_surface;
      amount = smin(amount, safe_amount_cap);
    }
    if (amount <= 1e-4f) {
      skip_rest = true;
    } else {
      const float e_rg = exp_cr(blur_log_rg);
      const float e_bg = exp_cr(blur_log_bg);
      const float target_r = smin(g, g * e_rg);
      const float target_b = smin(g, g * e_bg);
      if (correct_purple) {
        float corrected_r = sclamp(s0 * (1.f - amount) + target_r * amount, 0.f, s0);
        float corrected_g = s1;
        float corrected_b = sclamp(s2 * (1.f - amount) + target_b * amount, 0.f, s2);
        if (safe_surface > 1e-4f) {
          const float luma_before = 0.2126f * s0 + 0.7152f * s1 + 0.0722f * s2;
          const float luma_after = 0.2126f * corrected_r + 0.7152f * corrected_g + 0.0722f * corrected_b;
          const float max_luma_drop = luma_before * 0.02f * (1.f - neutral_gray_surface);
          const float min_luma = smax(0.f, luma_before - max_luma_drop);
          if (luma_after < min_luma) {
            const float lift = min_luma - luma_after;
            const float channel_ceil = smax(s0, smax(s1, s2));
            corrected_r = smin(s0, corrected_r + lift);
            corrected_g = smin(channel_ceil, corrected_g + lift);
            corrected_b = smin(s2, corrected_b + lift);
          }
          const float smx = smax(s0, smax(s1, s2));
          const float smn = smin(s0, smin(s1, s2));
          const float cmx = smax(corrected_r, smax(corrected_g, corrected_b));
          const float cmn = smin(corrected_r, smin(corrected_g, corrected_b));
          const float sch = smx - smn;
          const float cch = cmx - cmn;
          const float min_chroma = sch * (1.f - 0.12f * safe_surface);
          if (sch > 1e-4f && cch < min_chroma) {
            const float dn = smax(sch - cch, 1e-4f);
            const float keep = sclamp((sch - min_chroma) / dn, 0.f, 1.f);
            corrected_r = s0 * (1.f - keep) + corrected_r * keep;
            corrected_g = s1 * (1.f - keep) + corrected_g * keep;
            corrected_b = s2 * (1.f - keep) + corrected_b * keep;
          }
        }
        d0 = corrected_r;
        d1 = corrected_g;
        d2 = corrected_b;
      } else {
        float target_g = s1;
        const float rg_ref = e_rg;
        const float bg_ref = e_bg;
        if (rg_ref > 1e-4f && bg_ref > 1e-4f) {
          const float g_from_r = smax(s0, 0.f) / rg_ref;
          const float g_from_b = smax(s2, 0.f) / bg_ref;
          target_g = 0.5f * (g_from_r + g_from_b);
        }
        const float rb_avg_target = 0.5f * (smax(s0, 0.f) + smax(s2, 0.f));
        target_g = smax(target_g, rb_avg_target);
        const float green_amount = sclamp(amount * green_strength_scale, 0.f, 1.f);
        d0 = s0;
        d1 = sclamp(s1 * (1.f - green_amount) + target_g * green_amount, 0.f, s1);
        d2 = s2;
      }
    }
  }

  if (!skip_rest) {
    const float solo_enable = T.solo_enable;
    if (solo_enable > 0.f) {
      const float g = smax(s1, 0.f);
      const float target_r = g * exp_cr(blur_log_rg);
      const float target_b = g * exp_cr(blur_log_bg);
      const float solo_r = smax(0.f, s0 - target_r) / smax(blur_guide, 0.05f);
      const float solo_b = smax(0.f, s2 - target_b) / smax(blur_guide, 0.05f);
      const float local_solo_r =
          ss<FAST>(T.e[DE_SOLO], solo_r);
      const float local_solo_b =
          ss<FAST>(T.e[DE_SOLO], solo_b);
      const float rr0 = smax(s0, 0.f);
      const float gg0 = g;
      const float bb0 = smax(s2, 0.f);
      const float g_over_min2 = smax(0.f, gg0 - smin(rr0, bb0)) / smax(blur_guide, 0.05f);
      const float green_dom2 = ssl(0.010f, 0.060f, g_over_min2);
      const float denom_solo = smax(blur_guide, 0.05f);
      const float purpleish =
          ssl(0.010f, 0.060f, smax(smax(0.f, rr0 - gg0), smax(0.f, bb0 - gg0)) / denom_solo);
      const float solo_allow = 1.f - green_dom2 * (1.f - purpleish);
      const float solo_r_mask = v.srb * local_solo_r * solo_allow;
      const float solo_b_mask = v.sbb * local_solo_b * solo_allow;
      if (solo_r_mask > mask_cutoff) {
        const float amount = sclamp(solo_r_mask * strength * 0.85f, 0.f, 0.85f);
        d0 = sclamp(d0 * (1.f - amount) + target_r * amount, 0.f, d0);
      }
      if (solo_b_mask > mask_cutoff) {
        const float amount = sclamp(solo_b_mask * strength * 0.95f, 0.f, 0.90f);
        d2 = sclamp(d2 * (1.f - amount) + target_b * amount, 0.f, d2);
      }
    }
  }
}

// Four consecutive pixels per thread and step, read and written as float4
// (src/dst 16-byte aligned; the planes are 256-byte aligned), so every load
// of a step is issued before the first use; the one-pixel loop was bound by
// load latency.  The keep-input test reads 4 planes; the other 7 are read
// only when a pixel of the group needs them.  The group's operands are then
// staged in shared memory (one column per thread) and one copy of the
// per-pixel code runs over the four pixels.
// Bound by the instructions of the pixels that don't keep their input, in warps
// where the others wait.  PACK: a warp lists its pixels with work and deals them
// to its lanes (51 MP 1008 us without, 853 us with; 1.9 MP 72 and 59 us; seven
// CTAs per SM, which spill more, 863 us).
constexpr int DFM_THREADS = 128;
constexpr int DFM_VALS = 14;  // s0 s1 s2 be ber srb sbb bg blrg blbg bfs lfs lrg lbg

template <bool FAST, bool PACK>
__global__ void __launch_bounds__(DFM_THREADS, 6)
    k_df_main(const float* src, float* dst, int W, int H, DfPlanes P, DfConst k, DfTab T, const DfScalars* sc,
              float* out_max_g) {
  __shared__ float S[DFM_VALS * 4][DFM_THREADS];
  __shared__ unsigned char s_list[PACK ? 4 * DFM_THREADS : 1];
  DfMainK K;
  K.mask_cutoff = T.mask_cutoff;
  const float max_guide = df_max_guide(sc);
  K.scene_highlight_gate = ssmooth(0.55f, 0.75f, max_guide);
  K.enable_green = k.green != 0;
  K.strength = k.strength;
  K.green_strength_scale = sclamp(k.green_scale, 0.f, 1.f);
  K.e0_edge = T.e[DE_LOW].e0;
  K.e0_raw = T.e[DE_LOW_RAW].e0;
  K.can_skip = !K.enable_green && k.edge_thr > 0.f;  // smoothstep edges strictly ordered
  const size_t n = (size_t)W * H;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
  const size_t n4 = vec ? n / 4 : 0;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const int tid = threadIdx.x;
  float mg = 0.f;  // max(0, G) of what this thread writes (fmaxf drops NaN)
  const int lane = tid & 31, wb = tid - lane;
  unsigned char* list = s_list + 4 * wb;
  for (size_t q0 = blockIdx.x * (size_t)blockDim.x + wb; q0 < n4; q0 += stride) {
    const size_t i = (q0 + lane) * 4;
    unsigned keep = 0xFu;
    if (q0 + lane < n4) {
      float s[12], be[4], ber[4], srb[4], sbb[4];
      ld4(src + i * 3, s);
      ld4(src + i * 3 + 4, s + 4);
      ld4(src + i * 3 + 8, s + 8);
      ld4(P.be + i, be);
      ld4(P.ber + i, ber);
      ld4(P.srb + i, srb);
      ld4(P.sbb + i, sbb);
      keep = 0;
#pragma unroll
      for (int t = 0; t < 4; t++) keep |= df_keeps_input(K, be[t], ber[t], srb[t], sbb[t]) ? 1u << t : 0u;
      if (keep == 0xFu) {
        st4(dst + i * 3, s);
        st4(dst + i * 3 + 4, s + 4);
        st4(dst + i * 3 + 8, s + 8);
        mg = fmaxf(mg, fmaxf(fmaxf(s[1], s[4]), fmaxf(s[7], s[10])));
      } else {
        float pl[7][4];
        ld4(P.bg + i, pl[0]);
        ld4(P.blrg + i, pl[1]);
        ld4(P.blbg + i, pl[2]);
        ld4(P.bfs + i, pl[3]);
        ld4(P.lfs + i, pl[4]);
        ld4(P.lrg + i, pl[5]);
        ld4(P.lbg + i, pl[6]);
        // S[v * 4 + t][tid]: value v of pixel t
#pragma unroll
        for (int t = 0; t < 4; t++) {
          S[0 * 4 + t][tid] = s[3 * t];
          S[1 * 4 + t][tid] = s[3 * t + 1];
          S[2 * 4 + t][tid] = s[3 * t + 2];
          S[3 * 4 + t][tid] = be[t];
          S[4 * 4 + t][tid] = ber[t];
          S[5 * 4 + t][tid] = srb[t];
          S[6 * 4 + t][tid] = sbb[t];
#pragma unroll
          for (int v = 0; v < 7; v++) S[(7 + v) * 4 + t][tid] = pl[v][t];
        }
      }
    }
    if (PACK) {
      // the warp's pixels with work, dealt to its lanes
      int count = 0;
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const bool work = !(keep >> t & 1u);
        const unsigned m = __ballot_sync(~0u, work);
        if (work) list[count + __popc(m & ((1u << lane) - 1))] = (unsigned char)(t << 5 | lane);
        count += __popc(m);
      }
      __syncwarp();
#pragma unroll 1
      for (int j = lane; j < count; j += 32) {
        const int t = list[j] >> 5, x = wb + (list[j] & 31);
        const DfPx v{S[3 * 4 + t][x],  S[4 * 4 + t][x],  S[5 * 4 + t][x],  S[6 * 4 + t][x],
                     S[7 * 4 + t][x],  S[8 * 4 + t][x],  S[9 * 4 + t][x],  S[10 * 4 + t][x],
                     S[11 * 4 + t][x], S[12 * 4 + t][x], S[13 * 4 + t][x]};
        float r0, r1, r2;
        df_main_px<FAST>(S[0 * 4 + t][x], S[1 * 4 + t][x], S[2 * 4 + t][x], v, K, T, r0, r1, r2);
        S[0 * 4 + t][x] = r0;
        S[1 * 4 + t][x] = r1;
        S[2 * 4 + t][x] = r2;
      }
      __syncwarp();
    } else {
#pragma unroll 1
      for (int t = 0; t < 4; t++) {
        if (keep >> t & 1u) continue;
        const DfPx v{S[3 * 4 + t][tid],  S[4 * 4 + t][tid],  S[5 * 4 + t][tid],  S[6 * 4 + t][tid],
                     S[7 * 4 + t][tid],  S[8 * 4 + t][tid],  S[9 * 4 + t][tid],  S[10 * 4 + t][tid],
                     S[11 * 4 + t][tid], S[12 * 4 + t][tid], S[13 * 4 + t][tid]};
        float r0, r1, r2;
        df_main_px<FAST>(S[0 * 4 + t][tid], S[1 * 4 + t][tid], S[2 * 4 + t][tid], v, K, T, r0, r1, r2);
        S[0 * 4 + t][tid] = r0;
        S[1 * 4 + t][tid] = r1;
        S[2 * 4 + t][tid] = r2;
      }
    }
    if (keep != 0xFu) {
      float d[12];
#pragma unroll
      for (int t = 0; t < 4; t++) {
        d[3 * t] = S[0 * 4 + t][tid];
        d[3 * t + 1] = S[1 * 4 + t][tid];
        d[3 * t + 2] = S[2 * 4 + t][tid];
      }
      st4(dst + i * 3, d);
      st4(dst + i * 3 + 4, d + 4);
      st4(dst + i * 3 + 8, d + 8);
      mg = fmaxf(mg, fmaxf(fmaxf(d[1], d[4]), fmaxf(d[7], d[10])));
    }
    if (PACK) __syncwarp();
  }
  for (size_t i = n4 * 4 + blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    const float s0 = src[i * 3 + 0], s1 = src[i * 3 + 1], s2 = src[i * 3 + 2];
    float d0 = s0, d1 = s1, d2 = s2;
    if (!df_keeps_input(K, P.be[i], P.ber[i], P.srb[i], P.sbb[i])) {
      const DfPx v{P.be[i], P.ber[i], P.srb[i], P.sbb[i], P.bg[i],  P.blrg[i],
                   P.blbg[i], P.bfs[i], P.lfs[i], P.lrg[i], P.lbg[i]};
      df_main_px<FAST>(s0, s1, s2, v, K, T, d0, d1, d2);
    }
    dst[i * 3 + 0] = d0;
    dst[i * 3 + 1] = d1;
    dst[i * 3 + 2] = d2;
    mg = fmaxf(mg, d1);
  }
  if (out_max_g) {  // every thread of the block gets here
    mg = warp_max(mg);
    if ((tid & 31) == 0) atomic_max_float(out_max_g, mg);
  }
}

// Four pixels a step where src is 16-byte aligned (of a one-pixel load's sectors a
// third was of use) and one atomic a block: 26 MP 102 us before, 53 us so, of
// which its 12 B a pixel take 48 us; 1.9 MP 6.6 and 3.8 us.
__global__ void __launch_bounds__(256) k_df_maxg(const float* __restrict__ src, size_t n, DfScalars* sc) {
  float m = 0.f;
  const size_t at = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  const size_t n4 = (reinterpret_cast<uintptr_t>(src) & 15) == 0 ? n / 4 : 0;
  const float4* s4 = reinterpret_cast<const float4*>(src);
#pragma unroll 2
  for (size_t q = at; q < n4; q += stride) {
    const float4 a = __ldg(s4 + 3 * q), b = __ldg(s4 + 3 * q + 1), c = __ldg(s4 + 3 * q + 2);
    m = smax(smax(m, smax(0.f, a.y)), smax(smax(0.f, b.x), smax(smax(0.f, b.w), smax(0.f, c.z))));
  }
  for (size_t i = n4 * 4 + at; i < n; i += stride) m = smax(m, smax(0.f, src[i * 3 + 1]));
  m = warp_max(m);
  __shared__ float s_m[8];
  if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 8) {
    m = s_m[threadIdx.x];
#pragma unroll
    for (int o = 4; o; o >>= 1) m = smax(m, __shfl_xor_sync(0xffu, m, o));
    if (threadIdx.x == 0) atomic_max_float(&sc->max_guide_raw, m);
  }
}

// Tap radii 3 to 15 run the strip kernel compiled for them, others the tile
// kernel with the radius at run time (all eight planes of 12 MP: radius 3 253 us
// and 15 634 us in strips, 2 678 us and 15.5 2257 us in tiles).  The strips'
// 2 KS + 1 accumulators take two registers each: 62 of 168 at 15.
template <int KS>
lre_status blur_for(Context* c, const BlurJob& job, const GaussTaps& taps, int W, int H, const DfScalars* sc, bool* done) {
  if constexpr (KS >= 3) {
    if (taps.ks == KS) {
      *done = true;
      return run_blur_strip<KS>(c, job, taps, W, H, sc);
    }
    return blur_for<KS - 1>(c, job, taps, W, H, sc, done);
  }
  return LRE_OK;
}

lre_status run_blur(Context* c, const BlurJob& job, const GaussTaps& taps, int W, int H, const DfScalars* sc) {
  bool done = false;
  LRE_TRY(blur_for<15>(c, job, taps, W, H, sc, &done));
  if (done) return LRE_OK;
  const int E = BT + 2 * taps.ks;
  const size_t smem = ((size_t)E * E + (size_t)E * BT) * sizeof(float);
  LRE_CUDA_TRY(c, cudaFuncSetAttribute(k_df_blur, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const dim3 grid((W + BT - 1) / BT, (H + BT - 1) / BT, job.np);
  k_df_blur<<<grid, 256, smem, c->stream>>>(job, taps, W, H, sc);
  count_launch(c);
  return check_launch(c, "defringe blur");
}

float host_ssmooth(float e0, float e1, float x) {
  float t = (x - e0) / (e1 - e0);
  t = t < 0.0f ? 0.0f : (1.0f < t ? 1.0f : t);
  return t * t * (3.0f - 2.0f * t);
}

// The table of a call, and whether every edge is in the range of ss<true>.
bool make_tab(const DfConst& k, DfTab* T) {
  const float st = k.strength < 1.0f ? 1.0f : k.strength;
  const float root = std::sqrt(st);
  const float sensitivity = root < 1.0f ? 1.0f : (2.5f < root ? 2.5f : root);
  const float i = 1.0f / sensitivity, e = k.edge_thr, c = k.chroma_thr;
  T->inv_s = i;
  T->mask_cutoff = 0.02f * i;
  T->soften = 1.f - 0.86f * host_ssmooth(0.22f, 0.40f, c);
  T->solo_enable = host_ssmooth(1.25f, 3.0f, k.strength);
  T->release = host_ssmooth(2.0f, 6.0f, k.strength);
  T->surface = host_ssmooth(3.f, 8.f, k.strength);
  bool fast = true;
  auto set = [&](int id, float e0, float e1) {
    const float d = e1 - e0;
    T->e[id] = DfEdge{e0, e1, d, 1.0f / d};
    const float lo = 8.6e-19f, hi = 1.1e18f;  // 2^-60, 2^60
    fast = fast && e0 >= lo && e0 <= hi && d >= lo && d <= hi;
  };
  set(DE_CORE, e * 0.35f * i, e * 1.50f * i);
  set(DE_CORE_RAW, 0.55f * i, 1.35f * i);
  set(DE_LOW, e * 0.10f * i, e * 0.80f * i);
  set(DE_LOW_RAW, 0.20f * i, 0.90f * i);
  set(DE_BRIGHT, 0.24f * i, 0.52f * i);
  set(DE_CHROMA, c * 0.45f * i, c * 1.60f * i);
  set(DE_HUE, 0.06f * i, 0.22f * i);
  set(DE_RP_HUE, 0.035f * i, 0.16f * i);
  set(DE_ABS, c * 0.35f * i, c * 1.20f * i);
  set(DE_LOWC, c * 1.20f * i, c * 2.40f * i);
  set(DE_SOFT, 0.05f * i, 0.20f * i);
  set(DE_GATE, c * 0.10f * i, c * 0.55f * i);
  set(DE_PEAK, c * 0.80f * i, c * 2.50f * i);
  set(DE_HALO, c * 0.55f * i, c * 1.65f * i);
  set(DE_SOLO, c * 0.12f * i, c * 0.65f * i);
  set(DE_SEED_SOLO, c * 0.22f * i, c * 0.95f * i);
  return fast;
}

}  // namespace

size_t ws_bytes_defringe(size_t w, size_t h, float radius) {
  (void)radius;
  return 15 * ((w * h * sizeof(float) + 255) & ~size_t(255)) + 256;
}

lre_status launch_defringe(Context* c, const float* in, float* out, size_t w, size_t h, float radius,
                           float edge_thr, float chroma_thr, float strength, bool green, float green_scale,
                           const float* in_max_g, float* out_max_g) {
  GaussTaps taps = make_defringe_taps(radius);
  {
    const float sigma = std::max(radius / 3.f, 0.5f);
    if (static_cast<int>(std::ceil(3.f * sigma)) > GAUSS_MAX_KS)
      return fail(c, LRE_ERR_INVALID_ARGUMENT, "defringe: radius > 32 is not supported");
  }
  const int W = (int)w, H = (int)h;
  const size_t plane = (w * h * sizeof(float) + 255) & ~size_t(255);
  DfPlanes P;
  float** slots[15] = {&P.lrg, &P.lbg, &P.er, &P.bg, &P.blrg, &P.blbg, &P.be, &P.ber,
                       &P.fs,  &P.bfs, &P.lfs, &P.srs, &P.sbs, &P.srb, &P.sbb};
  for (int i = 0; i < 15; i++) {
    *slots[i] = reinterpret_cast<float*>(c->ws.take(plane));
    if (!*slots[i]) return fail(c, LRE_ERR_OUT_OF_MEMORY, "defringe: workspace too small");
  }
  DfScalars* sc = reinterpret_cast<DfScalars*>(c->ws.take(sizeof(DfScalars)));
  if (!sc) return fail(c, LRE_ERR_OUT_OF_MEMORY, "defringe: workspace too small");
  DfConst k{edge_thr, chroma_thr, strength, green_scale, green ? 1 : 0};
  DfTab T;
  const bool fast = make_tab(k, &T);
  const size_t n = w * h;

  LRE_CUDA_TRY(c, cudaMemsetAsync(sc, 0, sizeof(DfScalars), c->stream));
  if (out_max_g) LRE_CUDA_TRY(c, cudaMemsetAsync(out_max_g, 0, sizeof(float), c->stream));
  if (in_max_g)
    LRE_CUDA_TRY(c, cudaMemcpyAsync(&sc->max_guide_raw, in_max_g, sizeof(float), cudaMemcpyDeviceToDevice, c->stream));
  if (!in_max_g) {
    k_df_maxg<<<grid_for((n + 3) / 4, 256, c->sm_count * 8), 256, 0, c->stream>>>(in, n, sc);
    count_launch(c);
  }
  // Rows of a walk: 32, fewer while the SMs have less than 32 warps each (two
  // rows beside a walk are formed for it alone).
  const size_t prep_strips = (W + PW_COLS - 1) / PW_COLS;
  int prep_rows = PW_ROWS;
  while (prep_rows > 4 && prep_strips * ((H + prep_rows - 1) / prep_rows) < (size_t)c->sm_count * 32) prep_rows /= 2;
  const size_t prep_blocks = (prep_strips * ((H + prep_rows - 1) / prep_rows) + 7) / 8;
  k_df_prep<<<(unsigned)std::min<size_t>(prep_blocks, (size_t)c->sm_count * 24), 256, 0, c->stream>>>(
      in, W, H, prep_rows, sc, P.lrg, P.lbg, P.er);
  count_launch(c);
  LRE_TRY(check_launch(c, "defringe prep"));

  BlurJob j1{};
  j1.np = 5;
  j1.in[0] = in;    j1.mode[0] = BS_GUIDE_LINEAR;    j1.out[0] = P.bg;
  j1.in[1] = P.lrg; j1.mode[1] = BS_PLANE;           j1.out[1] = P.blrg;
  j1.in[2] = P.lbg; j1.mode[2] = BS_PLANE;           j1.out[2] = P.blbg;
  j1.in[3] = P.er;  j1.mode[3] = BS_PLANE_EDGE_NORM; j1.out[3] = P.be;
  j1.in[4] = P.er;  j1.mode[4] = BS_PLANE;           j1.out[4] = P.ber;
  LRE_TRY(run_blur(c, j1, taps, W, H, sc));
  auto support = fast ? k_df_support<true> : k_df_support<false>;
  support<<<grid_for((n + 3) / 4, 256, c->sm_count * 8), 256, 0, c->stream>>>(in, n, P, k, T, sc);
  count_launch(c);
  LRE_TRY(check_launch(c, "defringe support"));

  BlurJob j2{};
  j2.np = 1;
  j2.in[0] = P.fs; j2.mode[0] = BS_PLANE; j2.out[0] = P.bfs;
  LRE_TRY(run_blur(c, j2, taps, W, H, sc));

  dim3 lgrid((W + LT - 1) / LT, (H + LT - 1) / LT);
  auto line = fast ? k_df_line<true> : k_df_line<false>;
  line<<<lgrid, LN_THREADS, 0, c->stream>>>(in, W, H, P, k, T, sc);
  count_launch(c);
  LRE_TRY(check_launch(c, "defringe line"));

  BlurJob j3{};
  j3.np = 2;
  j3.in[0] = P.srs; j3.mode[0] = BS_PLANE; j3.out[0] = P.srb;
  j3.in[1] = P.sbs; j3.mode[1] = BS_PLANE; j3.out[1] = P.sbb;
  LRE_TRY(run_blur(c, j3, taps, W, H, sc));

  // Eight times the resident CTAs: the work of a pixel depends on what it shows,
  // and CTAs that took a sixth of an SM's share each left SMs idle at the end
  // (51 MP 1110 us with 6 per SM, 997 us with 48; 26 MP odd 1261 and 1183 us;
  // before packing).
  // Packing pays where pixels keep their input; with green correction none does
  // (24 MP 589 us without, 485 us with it; 26 MP with green 1181 and 1279 us).
  const bool pack = !k.green && k.edge_thr > 0.f;
  auto main_pass = fast ? (pack ? k_df_main<true, true> : k_df_main<true, false>)
                        : (pack ? k_df_main<false, true> : k_df_main<false, false>);
  main_pass<<<grid_for((n + 3) / 4, DFM_THREADS, c->sm_count * 48), DFM_THREADS, 0, c->stream>>>(in, out, W, H, P, k,
                                                                                                T, sc, out_max_g);
  count_launch(c);
  return check_launch(c, "defringe main");
}

}  // namespace lre

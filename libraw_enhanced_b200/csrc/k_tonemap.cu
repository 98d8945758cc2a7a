// k_tonemap.cu -- detail-preserving tone map and highlight micro-contrast.
//
// Detail-preserving tone map: core/libraw_wrapper.cpp:1389-1471 with the
// separable box filter box_filter_normalized (:45-116), as two passes of
// sliding window sums over column strips (k_dt_box), or in the reference's
// scan order (k_box_rows2, k_box_cols2) where the last bit matters.
//
// Micro-contrast: core/cpu_accelerator.cpp:3074-3319.  The 9x9 Gaussian
// (sigma 5/3.7, clamp-to-edge) is a non-separable 81-tap sum in (ky, kx)
// order; it runs out of a shared-memory halo tile with the reference's tap
// order.  The global max of the local standard deviation needs a grid-wide
// reduction, so the stage is two kernels: statistics (+ atomic max), then the
// per-pixel enhancement.
#include <algorithm>
#include <cmath>

#include "lre_internal.h"
#include "stencil.cuh"

namespace lre {

namespace {

__device__ __forceinline__ float aces_tm(float x) {
  const float a = 2.51f, b = 0.03f, c = 2.43f, d = 0.59f, e = 0.14f;
  return (x * (a * x + b)) / (x * (c * x + d) + e);
}

// -------------------------------------------------------- detail tone map
// Box means over the (2R+1)^2 window cut at the frame, two quantities at a
// time, on column strips: 160 threads hold the vertical window sums of 152
// columns (128 outputs and R halo columns each side) and walk down a chunk of
// rows, four rows per step.  A step adds the entering samples and subtracts
// the leaving ones (kept in a shared-memory ring, so global memory is read
// once), puts the four rows' vertical sums in shared memory, and four warps
// then slide the horizontal sums over four adjacent outputs per lane.
//
// What bounds it: shared-memory reads of the horizontal sums (56 B per pixel
// and quantity pair) beside 20 B/px of HBM traffic per pass.  The form before
// (one thread per row, then one per column, each walking the whole image with
// a running sum) left the GPU to H or W threads: 18.97 ms at 8256x5504; this
// one takes 0.63 ms (0.74 ms with eight divisions a lane and row by the number of
// samples, whose reciprocals a lane now keeps).  A sum restarts at every chunk of
// rows and every four columns, so a vertical sum carries the roundings of at most
// 2 * 256 + 2R additions and subtractions (a row enters and one leaves), not of
// the whole column's; 24 more form a window's, and a product with a rounded
// reciprocal its mean.  Measured against 64 bits: 2e-7, where the whole-image
// running sums had 1.7e-6.  Samples above 1.8e19, whose squares are infinite,
// spoil the sums of their window and, behind them, of the chunk (there the whole
// column).
constexpr int DT_R = 12;               // box radius (core/libraw_wrapper.cpp:1424)
constexpr int DT_X = 128;              // output columns per strip
constexpr int DT_C = DT_X + 2 * DT_R;  // columns whose vertical sums a strip holds
constexpr int DT_THREADS = 160;
constexpr int DT_STEP = 4;             // rows per step
constexpr int DT_RING = 2 * DT_R + 1 + DT_STEP + 3;  // rows kept: the window and a step's entering rows (32)
static_assert(DT_RING == 32 && DT_C <= DT_THREADS, "ring index is masked");

__device__ __forceinline__ float dt_guide(const float* __restrict__ p) {
  return smax(0.0f, smax(p[0], smax(p[1], p[2])));
}

// PASS 0: quantities (guide, guide^2) of rgb -> a, b of the guided filter.
// PASS 1: quantities (a, b) -> the tone-mapped rgb_out (may be rgb).
template <int PASS>
__global__ void __launch_bounds__(DT_THREADS) k_dt_box(const float* rgb, const float* __restrict__ pa,
                                                       const float* __restrict__ pb, float* __restrict__ a_out,
                                                       float* __restrict__ b_out, float* rgb_out, int W, int H,
                                                       int pitch, int rows, int vec) {
  __shared__ float ring0[DT_RING][DT_C];
  __shared__ float ring1[PASS ? DT_RING : 1][DT_C];
  __shared__ __align__(16) float v0[DT_STEP][DT_THREADS], v1[DT_STEP][DT_THREADS];
  constexpr float eps = 0.0025f, edge0 = 0.55f, edge1 = 0.90f;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = blockIdx.x * DT_X, y0 = blockIdx.y * rows, y1 = min(y0 + rows, H);
  const int cx = x0 - DT_R + tid;  // this thread's column
  const bool col_on = tid < DT_C && cx >= 0 && cx < W;
  // the sample of (row y, this column), zero outside the frame
  auto fetch = [&](int y, float& q0, float& q1) {
    q0 = q1 = 0.f;
    if (col_on && y >= 0 && y < H) {
      if (PASS == 0) {
        q0 = dt_guide(rgb + ((size_t)y * W + cx) * 3);
      } else {
        q0 = pa[(size_t)y * pitch + cx];
        q1 = pb[(size_t)y * pitch + cx];
      }
    }
  };
  float s0 = 0.f, s1 = 0.f;
  // rows [y0 - R, y0 + R) enter before the first step
  for (int y = y0 - DT_R; y < y0 + DT_R; y += 4) {
    float q0[4], q1[4];
#pragma unroll
    for (int k = 0; k < 4; k++) fetch(y + k, q0[k], q1[k]);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (tid < DT_C) {
        ring0[(y + k) & (DT_RING - 1)][tid] = q0[k];
        if (PASS == 1) ring1[(y + k) & (DT_RING - 1)][tid] = q1[k];
      }
      s0 += q0[k];
      s1 += PASS == 0 ? q0[k] * q0[k] : q1[k];
    }
  }
  // 1 / (samples of a window) for the lane's four columns, formed anew where the
  // number of rows changes
  float inv[4], held = 0.f;
  float n0[DT_STEP], n1[DT_STEP];  // the next step's entering samples
#pragma unroll
  for (int k = 0; k < DT_STEP; k++) fetch(y0 + DT_R + k, n0[k], n1[k]);
  for (int y = y0; y < y1; y += DT_STEP) {
#pragma unroll
    for (int k = 0; k < DT_STEP; k++) {
      const float q0 = n0[k], q1 = n1[k];
      s0 += q0;
      s1 += PASS == 0 ? q0 * q0 : q1;
      v0[k][tid] = s0;
      v1[k][tid] = s1;
      if (tid < DT_C) {
        // only this thread touches its ring column
        const int in = (y + k + DT_R) & (DT_RING - 1), out = (y + k - DT_R) & (DT_RING - 1);
        const float l0 = ring0[out][tid];
        s0 -= l0;
        s1 -= PASS == 0 ? l0 * l0 : ring1[out][tid];
        ring0[in][tid] = q0;
        if (PASS == 1) ring1[in][tid] = q1;
      }
    }
    __syncthreads();
    if (y + DT_STEP < y1) {
#pragma unroll
      for (int k = 0; k < DT_STEP; k++) fetch(y + DT_STEP + DT_R + k, n0[k], n1[k]);
    }
    const int oy = y + warp;
    if (warp < DT_STEP && oy < y1) {
      // window sums of the lane's four adjacent columns
      float h0[4], h1[4];
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const float4* v = reinterpret_cast<const float4*>(q ? v1[warp] : v0[warp]) + lane;
        float e[4 + 2 * DT_R];
#pragma unroll
        for (int k = 0; k < 1 + DT_R / 2; k++) {
          const float4 f = v[k];
          e[4 * k] = f.x;
          e[4 * k + 1] = f.y;
          e[4 * k + 2] = f.z;
          e[4 * k + 3] = f.w;
        }
        // the 22 samples that all four windows share, then each window's own
        float m[4] = {e[3], e[4], e[5], e[6]};
#pragma unroll
        for (int k = 7; k <= 2 * DT_R; k++) m[(k - 3) & 3] += e[k];
        const float mid = (m[0] + m[1]) + (m[2] + m[3]);
        float* h = q ? h1 : h0;
        h[0] = mid + ((e[0] + e[1]) + e[2]);
        h[1] = mid + ((e[1] + e[2]) + e[25]);
        h[2] = mid + ((e[2] + e[25]) + e[26]);
        h[3] = mid + ((e[25] + e[26]) + e[27]);
      }
      const float cy = (float)(min(H - 1, oy + DT_R) - max(0, oy - DT_R) + 1);
      const int x = x0 + 4 * lane;
      if (cy != held) {
        held = cy;
#pragma unroll
        for (int k = 0; k < 4; k++) inv[k] = 1.0f / (cy * (float)(min(W - 1, x + k + DT_R) - max(0, x + k - DT_R) + 1));
      }
      float o0[4], o1[4];
      if (PASS == 0) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          // m0 = mean(guide), m1 = mean(guide^2)  (core/libraw_wrapper.cpp:1431-1436)
          const float m0 = h0[k] * inv[k], m1 = h1[k] * inv[k];
          const float var = smax(0.0f, m1 - m0 * m0);
          o0[k] = var / (var + eps);
          o1[k] = m0 * (1.0f - o0[k]);
        }
        // the planes' rows are padded to four columns
        if (x < W) {
          const size_t i = (size_t)oy * pitch + x;
          *reinterpret_cast<float4*>(a_out + i) = make_float4(o0[0], o0[1], o0[2], o0[3]);
          *reinterpret_cast<float4*>(b_out + i) = make_float4(o1[0], o1[1], o1[2], o1[3]);
        }
      } else {
        const size_t i = ((size_t)oy * W + x) * 3;
        const bool v4 = vec && x < W;  // W is then a multiple of four
        float c[12];
        if (v4) {
#pragma unroll
          for (int k = 0; k < 3; k++) {
            const float4 f = reinterpret_cast<const float4*>(rgb + i)[k];
            c[4 * k] = f.x;
            c[4 * k + 1] = f.y;
            c[4 * k + 2] = f.z;
            c[4 * k + 3] = f.w;
          }
        } else {
#pragma unroll
          for (int k = 0; k < 12; k++) c[k] = x + k / 3 < W ? rgb[i + k] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
          // m0 = mean(a), m1 = mean(b)  (core/libraw_wrapper.cpp:1442-1465)
          const float m0 = h0[k] * inv[k], m1 = h1[k] * inv[k];
          const float guide = dt_guide(c + 3 * k);
          const float base = smax(1e-6f, m0 * guide + m1);
          float w = (base - edge0) * (1.0f / (edge1 - edge0));
          w = sclamp(w, 0.0f, 1.0f);
          w = w * w * (3.0f - 2.0f * w);
          if (w > 0.0f) {
            const float mapped = aces_tm(base);
            const float gain = 1.0f + (sclamp(mapped / base, 0.0f, 1.0f) - 1.0f) * w;
            c[3 * k] *= gain;
            c[3 * k + 1] *= gain;
            c[3 * k + 2] *= gain;
          }
        }
        if (v4) {
#pragma unroll
          for (int k = 0; k < 3; k++)
            reinterpret_cast<float4*>(rgb_out + i)[k] = make_float4(c[4 * k], c[4 * k + 1], c[4 * k + 2], c[4 * k + 3]);
        } else {
#pragma unroll
          for (int k = 0; k < 12; k++)
            if (x + k / 3 < W) rgb_out[i + k] = c[k];
        }
      }
    }
    __syncthreads();
  }
}

// The same tone map with the reference's own running sums, one thread per
// row, then per column, in its scan order: last bit for last bit the
// reference's floats.  It serves the develops, where a difference in the last
// bits could become a visible one (16-bit codes, and the thresholds of defringe
// and lateral CA after the tone map) and where 16 bits are to be the quantised
// 32 of the same chain; 18.97 ms at 8256x5504 against 0.63 of the strips.
// Horizontal running box sums of two planes at once.  mode 0: the planes are
// derived from RGB (guide = max(0, maxRGB), guide^2); mode 1: plain planes.
__global__ void k_box_rows2(const float* __restrict__ rgb, const float* __restrict__ p0, const float* __restrict__ p1,
                            float* __restrict__ t0, float* __restrict__ t1, int W, int H, int R, int mode) {
  int y = blockIdx.x * blockDim.x + threadIdx.x;
  if (y >= H) return;
  const size_t row = (size_t)y * W;
  auto val = [&](int x, float& a, float& b) {
    if (mode == 0) {
      const float* p = rgb + (row + x) * 3;
      float g = smax(0.0f, smax(p[0], smax(p[1], p[2])));
      a = g;
      b = g * g;
    } else {
      a = p0[row + x];
      b = p1[row + x];
    }
  };
  float s0 = 0.f, s1 = 0.f;
  const int first_right = min(W - 1, R);
  for (int x = 0; x <= first_right; x++) {
    float a, b;
    val(x, a, b);
    s0 += a;
    s1 += b;
  }
  for (int x = 0; x < W; x++) {
    const int left = x > R ? x - R : 0;
    const int right = min(W - 1, x + R);
    const float cnt = (float)(right - left + 1);
    t0[row + x] = s0 / cnt;
    t1[row + x] = s1 / cnt;
    const int remove_x = x >= R ? x - R : W;
    const int add_x = x + R + 1;
    if (remove_x < W) {
      float a, b;
      val(remove_x, a, b);
      s0 -= a;
      s1 -= b;
    }
    if (add_x < W) {
      float a, b;
      val(add_x, a, b);
      s0 += a;
      s1 += b;
    }
  }
}

// Vertical running box sums of two planes; `emit(x, y, m0, m1)` consumes the
// means.  mode 0: produce a, b of the guided filter; mode 1: final apply.
__global__ void k_box_cols2(const float* __restrict__ t0, const float* __restrict__ t1, int W, int H, int R, int mode,
                            float* __restrict__ a_out, float* __restrict__ b_out, const float* __restrict__ rgb_in,
                            float* __restrict__ rgb_out) {
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= W) return;
  const float eps = 0.0025f, edge0 = 0.55f, edge1 = 0.90f;
  float s0 = 0.f, s1 = 0.f;
  const int first_bottom = min(H - 1, R);
  for (int y = 0; y <= first_bottom; y++) {
    s0 += t0[(size_t)y * W + x];
    s1 += t1[(size_t)y * W + x];
  }
  for (int y = 0; y < H; y++) {
    const int top = y > R ? y - R : 0;
    const int bottom = min(H - 1, y + R);
    const float cnt = (float)(bottom - top + 1);
    const float m0 = s0 / cnt, m1 = s1 / cnt;
    const size_t i = (size_t)y * W + x;
    if (mode == 0) {
      // m0 = mean(guide), m1 = mean(guide^2)  (core/libraw_wrapper.cpp:1431-1436)
      const float var = smax(0.0f, m1 - m0 * m0);
      const float a = var / (var + eps);
      a_out[i] = a;
      b_out[i] = m0 * (1.0f - a);
    } else {
      // m0 = mean(a), m1 = mean(b)  (core/libraw_wrapper.cpp:1442-1465)
      const float* p = rgb_in + i * 3;
      const float r = p[0], g = p[1], bl = p[2];
      const float guide = smax(0.0f, smax(r, smax(g, bl)));
      const float base = smax(1e-6f, m0 * guide + m1);
      const float mapped = aces_tm(base);
      float gain = sclamp(mapped / base, 0.0f, 1.0f);
      float w = (base - edge0) / (edge1 - edge0);
      w = sclamp(w, 0.0f, 1.0f);
      w = w * w * (3.0f - 2.0f * w);
      float* q = rgb_out + i * 3;
      if (w <= 0.0f) {
        q[0] = r;
        q[1] = g;
        q[2] = bl;
      } else {
        gain = 1.0f + (gain - 1.0f) * w;
        q[0] = r * gain;
        q[1] = g * gain;
        q[2] = bl * gain;
      }
    }
    const int remove_y = y >= R ? y - R : H;
    const int add_y = y + R + 1;
    if (remove_y < H) {
      s0 -= t0[(size_t)remove_y * W + x];
      s1 -= t1[(size_t)remove_y * W + x];
    }
    if (add_y < H) {
      s0 += t0[(size_t)add_y * W + x];
      s1 += t1[(size_t)add_y * W + x];
    }
  }
}

// -------------------------------------------------------- micro-contrast
// Local mean and standard deviation of one channel: the 81-tap sums of v and
// v^2, each product and each sum rounded, in (ky, kx) order from 0.
//
// A thread owns one column of a 64-column strip of one channel and walks down
// a chunk of rows; nine accumulator pairs (v and v^2 packed in one 64-bit
// register) are in flight, one per output row.  A staged sample is multiplied
// once per distinct |ky| (five packed products for nine rows) and the row's
// nine samples are taken in kx order, so every accumulator gets its taps in
// the reference's order.  The accumulators rotate by name over nine rows.
// What bounds it: the FP32 pipe.  Per channel and pixel 2 x (45 + 81)
// operations against 2 x 162 + 81 with every tap multiplied (and v squared)
// on its own.  4032x3024: 384 us (611 with tiles);
// the pipe's time is 290 us.
constexpr int MC_R = 4;
constexpr int MC_X = 64;                  // output columns per CTA
constexpr int MC_C = MC_X + 2 * MC_R;     // staged columns
constexpr int MC_P = 9;                   // the accumulators' period in rows
constexpr int MC_B = 2 * MC_P;            // rows per batch
constexpr int MC_THREADS = 3 * MC_X;      // one thread per column and channel

struct McTaps {
  float w[81];
  unsigned long long nz = 0x8000000080000000ull;  // {-0.f, -0.f}
};

__device__ __forceinline__ unsigned long long mc_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}

__global__ void __launch_bounds__(MC_THREADS) k_mc_stats(const float* __restrict__ in, int W, int H, int periods,
                                                         McTaps taps, float* __restrict__ mean3,
                                                         float* __restrict__ std3, float* d_max) {
  __shared__ __align__(16) float s[2][MC_B][MC_C * 3];
  const int x0 = blockIdx.x * MC_X, rows = periods * MC_P - 2 * MC_R;
  const int batches = (periods + 1) / 2;
  const int y0 = blockIdx.y * rows, y1 = min(y0 + rows, H);
  const int tid = threadIdx.x, ch = tid % 3, col = tid / 3, x = x0 + col;
  const unsigned long long nz = taps.nz;
  auto mul = [&](unsigned long long w, unsigned long long v) {  // the rounded product, not contracted with the sum
    unsigned long long p;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(w), "l"(v), "l"(nz));
    return p;
  };
  auto add = [](unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
  };
  auto stage = [&](int b) {
    const int yb = y0 - MC_R + b * MC_B;
    const int n = (periods - 2 * b) * MC_P;  // rows of the chunk from yb
    for (int i = tid; i < MC_C * 3; i += MC_THREADS) {
      const int gx = min(max(x0 - MC_R + i / 3, 0), W - 1), c = i % 3;
#pragma unroll
      for (int r = 0; r < MC_B; r++) {
        if (r == MC_P && n == MC_P) break;
        const float* g = in + ((size_t)min(max(yb + r, 0), H - 1) * W + gx) * 3 + c;
        const unsigned d = (unsigned)__cvta_generic_to_shared(&s[b & 1][r][i]);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(g) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // The weight of (ky, kx) depends on (ky - 4)^2 + (kx - 4)^2 only: 15 distinct
  // ones, in registers.
  auto widx = [](int a, int b) { return a <= b ? a * 5 - a * (a - 1) / 2 + b - a : b * 5 - b * (b - 1) / 2 + a - b; };
  unsigned long long w15[15];
#pragma unroll
  for (int i = 0; i < 5; i++)
#pragma unroll
    for (int j = i; j < 5; j++) w15[widx(i, j)] = mc_pack(taps.w[i * 9 + j], taps.w[i * 9 + j]);
  unsigned long long acc[MC_P];
#pragma unroll
  for (int j = 0; j < MC_P; j++) acc[j] = 0ull;
  float local_max = 0.f;
  stage(0);
  for (int b = 0; b < batches; b++) {
    const int yb = y0 - MC_R + b * MC_B;
    if (yb - MC_R >= y1) break;
    if (b + 1 < batches) {
      stage(b + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
#pragma unroll 1
    for (int half = 0; half < min(2, periods - 2 * b); half++)
#pragma unroll
    for (int r = 0; r < MC_P; r++) {
      const float* row = &s[b & 1][half * MC_P + r][col * 3 + ch];
#pragma unroll
      for (int kx = 0; kx < 9; kx++) {
        const float v = row[3 * kx];
        const unsigned long long v2 = mc_pack(v, v * v);
        unsigned long long m[MC_R + 1];  // products with the weights of |ky - 4| = 4 .. 0
#pragma unroll
        for (int k = 0; k <= MC_R; k++) m[k] = mul(w15[widx(k, kx <= MC_R ? kx : 8 - kx)], v2);
        // accumulator (r + j) % 9 belongs to the output row 4 - j above this
        // one: its tap ky = 8 - j
#pragma unroll
        for (int j = 0; j < MC_P; j++) {
          const int ky = 8 - j;
          unsigned long long& A = acc[(r + j) % MC_P];
          A = add(j == 8 && kx == 0 ? 0ull : A, m[ky <= MC_R ? ky : 8 - ky]);
        }
      }
      const int o = yb + half * MC_P + r - MC_R;
      if (o >= y0 && o < y1 && x < W) {
        float m, q;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(m), "=f"(q) : "l"(acc[r]));
        const float var = q - m * m;
        const float sd = sqrtf(smax(var, 0.f));
        const size_t i = ((size_t)o * W + x) * 3 + ch;
        mean3[i] = m;
        std3[i] = sd;
        local_max = smax(local_max, sd);
      }
    }
    __syncthreads();
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  block_max_atomic(local_max, d_max);
}

__global__ void k_mc_apply(const float* in, float* out, const float* __restrict__ mean3,
                           const float* __restrict__ std3, const float* __restrict__ mask, size_t n, float threshold,
                           float strength, float target, const float* d_max) {
  const float max_std = *d_max;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float* p = in + i * 3;
    const float I0 = p[0], I1 = p[1], I2 = p[2];
    float rgb[3];
    const float Iv[3] = {I0, I1, I2};
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float m = mean3[i * 3 + c];
      const float contrast = std3[i * 3 + c] / max_std;
      const float ef = (contrast < target) ? strength * (target - contrast) / target : 0.f;
      const float hf = Iv[c] - m;
      const float ehf = hf * (1.f + ef);
      rgb[c] = m + ehf;
    }
    float r = rgb[0], g = rgb[1], b = rgb[2];
    float* q = out + i * 3;
    if (mask) {
      const float w = sclamp(mask[i], 0.f, 1.f);
      const float maxc = smax(r, smax(g, b));
      if (maxc > 1.f) {
        const float scale = 1.f / maxc;
        r *= scale;
        g *= scale;
        b *= scale;
      }
      q[0] = I0 + (r - I0) * w;
      q[1] = I1 + (g - I1) * w;
      q[2] = I2 + (b - I2) * w;
    } else if (I1 >= threshold) {
      const float maxc = smax(r, smax(g, b));
      if (maxc > 1.f) {
        const float scale = 1.f / maxc;
        r *= scale;
        g *= scale;
        b *= scale;
      }
      q[0] = r;
      q[1] = g;
      q[2] = b;
    } else {
      q[0] = I0;
      q[1] = I1;
      q[2] = I2;
    }
  }
}

McTaps make_mc_taps() {
  // create_gaussian_kernel(9, 5/3.7) of core/cpu_accelerator.cpp:3077-3098,
  // evaluated with the host libm exactly as the reference does.
  McTaps t{};
  const float sigma = 5.f / 3.7f;
  const int size = 9, center = size / 2;
  float k[9][9];
  float sum = 0.0f;
  for (int i = 0; i < size; i++)
    for (int j = 0; j < size; j++) {
      float x = (float)(i - center);
      float y = (float)(j - center);
      k[i][j] = std::exp(-(x * x + y * y) / (2.0f * sigma * sigma));
      sum += k[i][j];
    }
  for (int i = 0; i < size; i++)
    for (int j = 0; j < size; j++) k[i][j] /= sum;
  for (int ky = 0; ky < 9; ky++)
    for (int kx = 0; kx < 9; kx++) t.w[ky * 9 + kx] = k[ky][kx];
  return t;
}

}  // namespace

// the a and b planes, rows padded to four columns
size_t dt_plane_bytes(size_t w, size_t h) { return (((w + 3) & ~size_t(3)) * h * 4 + 255) & ~size_t(255); }
size_t ws_bytes_detail_tonemap(size_t w, size_t h) {
  return std::max(2 * dt_plane_bytes(w, h), 4 * ((w * h * 4 + 255) & ~size_t(255)));
}
size_t ws_bytes_micro_contrast(size_t w, size_t h) { return 2 * ((w * h * 12 + 255) & ~size_t(255)) + 256; }

lre_status launch_detail_tonemap(Context* c, const float* in, float* out, size_t w, size_t h, bool reference_order) {
  const int W = (int)w, H = (int)h;
  if (reference_order) {
    const size_t plane = w * h;
    float* t0 = reinterpret_cast<float*>(c->ws.take(plane * 4));
    float* t1 = reinterpret_cast<float*>(c->ws.take(plane * 4));
    float* ra = reinterpret_cast<float*>(c->ws.take(plane * 4));
    float* rb = reinterpret_cast<float*>(c->ws.take(plane * 4));
    if (!t0 || !t1 || !ra || !rb) return fail(c, LRE_ERR_OUT_OF_MEMORY, "detail_tonemap: workspace too small");
    const int tb = 64, R = DT_R;
    k_box_rows2<<<(H + tb - 1) / tb, tb, 0, c->stream>>>(in, nullptr, nullptr, t0, t1, W, H, R, 0);
    k_box_cols2<<<(W + tb - 1) / tb, tb, 0, c->stream>>>(t0, t1, W, H, R, 0, ra, rb, nullptr, nullptr);
    k_box_rows2<<<(H + tb - 1) / tb, tb, 0, c->stream>>>(nullptr, ra, rb, t0, t1, W, H, R, 1);
    k_box_cols2<<<(W + tb - 1) / tb, tb, 0, c->stream>>>(t0, t1, W, H, R, 1, nullptr, nullptr, in, out);
    count_launch(c, 4);
    return check_launch(c, "detail_tonemap");
  }
  const int pitch = (W + 3) & ~3;
  float* pa = reinterpret_cast<float*>(c->ws.take(dt_plane_bytes(w, h)));
  float* pb = reinterpret_cast<float*>(c->ws.take(dt_plane_bytes(w, h)));
  if (!pa || !pb) return fail(c, LRE_ERR_OUT_OF_MEMORY, "detail_tonemap: workspace too small");
  // Rows per chunk: the 2R rows that a chunk reads ahead of its first output
  // cost the less the taller it is, so 256 rows, halved down to 16 while the
  // grid has fewer than eight CTAs per SM.
  const int strips = (W + DT_X - 1) / DT_X;
  int rows = 256;
  while (rows > 16 && (long long)strips * ((H + rows - 1) / rows) < 8LL * c->sm_count) rows /= 2;
  const dim3 grid((unsigned)strips, (unsigned)((H + rows - 1) / rows));
  const int vec = W % 4 == 0 && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  k_dt_box<0><<<grid, DT_THREADS, 0, c->stream>>>(in, nullptr, nullptr, pa, pb, nullptr, W, H, pitch, rows, 0);
  k_dt_box<1><<<grid, DT_THREADS, 0, c->stream>>>(in, pa, pb, nullptr, nullptr, out, W, H, pitch, rows,
                                                        vec);
  count_launch(c, 2);
  return check_launch(c, "detail_tonemap");
}

lre_status launch_micro_contrast(Context* c, const float* in, float* out, size_t w, size_t h, float threshold,
                                 float strength, float target, const float* mask) {
  const int W = (int)w, H = (int)h;
  float* mean3 = reinterpret_cast<float*>(c->ws.take(w * h * 12));
  float* std3 = reinterpret_cast<float*>(c->ws.take(w * h * 12));
  float* dmax = reinterpret_cast<float*>(c->ws.take(sizeof(float)));
  if (!mean3 || !std3 || !dmax) return fail(c, LRE_ERR_OUT_OF_MEMORY, "enhance_micro_contrast: workspace too small");
  static const McTaps taps = make_mc_taps();
  LRE_CUDA_TRY(c, cudaMemsetAsync(dmax, 0, sizeof(float), c->stream));
  // A chunk of n periods of nine rows writes 9n - 8 of them.  n by the time that the
  // fullest SM takes: its CTAs share the FP32 pipe, a quarter of a microsecond each
  // per row of theirs, and one alone waits for its own chain besides (0.42 us a row
  // with one CTA on the SM, 0.67 with two, 1.17 with four); more than one batch
  // begins with the loads of two.  Up to eight batches.
  // 530x530 19.1 us, 1536x1024 62.8, 4032x3024 384; halving from eight batches until
  // there were eight CTAs per SM 21.2, 81.0, 398; a tile per CTA 18.7, 87.1, 611.
  const int strips = (W + MC_X - 1) / MC_X;
  auto chunks = [&](int n) { return (H + n * MC_P - 2 * MC_R - 1) / (n * MC_P - 2 * MC_R); };
  auto cost = [&](int n) {
    const long long ctas = (long long)strips * chunks(n);
    return n * (2 + 3 * ((ctas + c->sm_count - 1) / c->sm_count)) + (n > 2 ? 2 : 0);
  };
  int periods = 2;
  for (int n = 3; n <= 16; n++)
    if (cost(n) < cost(periods)) periods = n;
  const dim3 grid((unsigned)strips, (unsigned)chunks(periods));
  k_mc_stats<<<grid, MC_THREADS, 0, c->stream>>>(in, W, H, periods, taps, mean3, std3, dmax);
  k_mc_apply<<<grid_for(w * h, 256, c->sm_count * 8), 256, 0, c->stream>>>(in, out, mean3, std3, mask, w * h,
                                                                            threshold, strength, target, dmax);
  count_launch(c, 2);
  return check_launch(c, "enhance_micro_contrast");
}

}  // namespace lre

// k_lateral.cu -- lateral chromatic-aberration registration: pyramidal
// Lucas-Kanade of R and B against G per cell, confidence gate, 3x3 cell
// smoothing, bilinear remap.
//
// Semantics: core/cpu_accelerator.cpp:3496-3673 (ca_register_lateral) with
// downsample_2x_box (:3369-3384), lk_estimate_level (:3390-3471),
// smooth_3x3_cells (:3474-3492) and bilinear_sample_plane (:3328-3346).
//
// Device plan: planar split + 2x box pyramid (one kernel per level); per
// level ONE launch estimates every cell of both channels, one CTA per
// (cell, channel): the CTA sweeps the cell's pixels, reduces the 2x2 normal
// equations in double with warp shuffles, and thread 0 solves and broadcasts
// the step, so all LK iterations of a cell stay on chip.  Gate + smoothing
// run in one small kernel; the remap is a streaming kernel.
//
// The estimate waits for its nine loads of a pixel.  What bought time was more
// of them in flight: four pixels per turn of the loop, five CTAs per SM, no
// clamps where the whole displaced cell lies inside, the pixel's row by a
// multiply-high, and the matrix summed in the first iteration only.  The three
// levels of 26 MP: 945 us before, 682 us now; of 1.9 MP 89 us, 70 us.
// (Three CTAs per SM with the same loop: 1135 us, the loads no longer hidden.)
#include <algorithm>
#include <cmath>

#include "lre_internal.h"
#include "stencil.cuh"

namespace lre {

namespace {

constexpr int LK_THREADS = 256;

__global__ void k_split_planes(const float* __restrict__ rgb, float* __restrict__ R, float* __restrict__ G,
                               float* __restrict__ B, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    R[i] = rgb[i * 3 + 0];
    G[i] = rgb[i * 3 + 1];
    B[i] = rgb[i * 3 + 2];
  }
}

// Split and the first 2x box in one pass, a thread per 2x2 block (the last one
// of an odd side holds one column or row, which has no box): the box no longer
// reads the planes back.  Bound by its 27 B per pixel.  vec: rgb is 8-byte
// aligned, so a row that starts at an even pixel moves in pairs of floats.
// 26 MP: split and boxes 105 + 90 us before, 130 us.
__global__ void __launch_bounds__(256) k_split_down(const float* __restrict__ rgb, float* __restrict__ R,
                                                    float* __restrict__ G, float* __restrict__ B,
                                                    float* __restrict__ r2, float* __restrict__ g2,
                                                    float* __restrict__ b2, int W, int H, bool vec) {
  const int W2 = W / 2, H2 = H / 2;
  float* const out[3] = {R, G, B};
  float* const box[3] = {r2, g2, b2};
  for (int y = blockIdx.y * blockDim.y + threadIdx.y; y < H - H2; y += gridDim.y * blockDim.y)
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < W - W2; x += gridDim.x * blockDim.x) {
      const bool two_x = x < W2, two_y = y < H2;
      float v[2][6];
#pragma unroll
      for (int r = 0; r < 2; r++) {
        if (r == 1 && !two_y) break;
        const size_t i = (size_t)(2 * y + r) * W + 2 * x;
        if (vec && two_x && (i & 1) == 0) {
#pragma unroll
          for (int q = 0; q < 3; q++) {
            const float2 t = __ldg(reinterpret_cast<const float2*>(rgb + 3 * i) + q);
            v[r][2 * q] = t.x;
            v[r][2 * q + 1] = t.y;
          }
        } else {
#pragma unroll
          for (int q = 0; q < 6; q++) v[r][q] = q < 3 || two_x ? __ldg(rgb + 3 * i + q) : 0.f;
        }
      }
#pragma unroll
      for (int r = 0; r < 2; r++) {
        if (r == 1 && !two_y) break;
        const size_t i = (size_t)(2 * y + r) * W + 2 * x;
#pragma unroll
        for (int q = 0; q < 3; q++) {
          if (two_x && (i & 1) == 0) {
            *reinterpret_cast<float2*>(out[q] + i) = make_float2(v[r][q], v[r][q + 3]);
          } else {
            out[q][i] = v[r][q];
            if (two_x) out[q][i + 1] = v[r][q + 3];
          }
        }
      }
      if (two_x && two_y)
#pragma unroll
        for (int q = 0; q < 3; q++)
          box[q][(size_t)y * W2 + x] = 0.25f * (v[0][q] + v[0][q + 3] + v[1][q] + v[1][q + 3]);
    }
}

struct Planes3 {
  const float* in[3];
  float* out[3];
};

__global__ void k_downsample3(Planes3 p, int W, int H, int W2, int H2) {
  size_t n = (size_t)W2 * H2;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int y = (int)(i / W2), x = (int)(i % W2);
    int y0 = 2 * y, y1 = min(y0 + 1, H - 1);
    int x0 = 2 * x, x1 = min(x0 + 1, W - 1);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float* in = p.in[c];
      p.out[c][i] = 0.25f * (in[(size_t)y0 * W + x0] + in[(size_t)y0 * W + x1] + in[(size_t)y1 * W + x0] +
                             in[(size_t)y1 * W + x1]);
    }
  }
}

__device__ __forceinline__ float bilinear_plane(const float* __restrict__ plane, int W, int H, float x, float y) {
  if (x < 0.f) x = 0.f;
  if (y < 0.f) y = 0.f;
  if (x > (float)(W - 1)) x = (float)(W - 1);
  if (y > (float)(H - 1)) y = (float)(H - 1);
  const int x0 = (int)x;
  const int y0 = (int)y;
  const int x1 = min(x0 + 1, W - 1);
  const int y1 = min(y0 + 1, H - 1);
  const float fx = x - (float)x0;
  const float fy = y - (float)y0;
  const float v00 = plane[(size_t)y0 * W + x0];
  const float v01 = plane[(size_t)y0 * W + x1];
  const float v10 = plane[(size_t)y1 * W + x0];
  const float v11 = plane[(size_t)y1 * W + x1];
  return (v00 * (1.f - fx) + v01 * fx) * (1.f - fy) + (v10 * (1.f - fx) + v11 * fx) * fy;
}

struct LkMaps {
  float* dx[2];
  float* dy[2];
  float* conf[2];
};

// One CTA per (cell, channel).  blockIdx.x = cell, blockIdx.y = channel
// (0: R, 1: B).
// PER_SM: resident CTAs that the registers are bounded for, five where there are
// CTAs enough, two where not (a CTA is then the faster by itself).
template <int PER_SM>
__global__ void __launch_bounds__(LK_THREADS, PER_SM)
    k_lk_level(const float* __restrict__ G, const float* __restrict__ Rt, const float* __restrict__ Bt, int W, int H,
               int map_w, int map_h, int max_iterations, float max_shift, float scale_down, float scale_up,
               LkMaps maps) {
  __shared__ double red[5][LK_THREADS / 32];
  __shared__ float s_acc[2];
  __shared__ int s_done;
  const int ch = blockIdx.y;
  const float* T = ch == 0 ? Rt : Bt;
  const int cell = blockIdx.x;
  const int cy = cell / map_w, cx = cell % map_w;
  const float cell_w_f = (float)W / (float)map_w;
  const float cell_h_f = (float)H / (float)map_h;
  const size_t x0 = (size_t)(cx * cell_w_f);
  const size_t y0 = (size_t)(cy * cell_h_f);
  size_t x1 = (size_t)((cx + 1) * cell_w_f);
  size_t y1 = (size_t)((cy + 1) * cell_h_f);
  x1 = x1 < (size_t)W ? x1 : (size_t)W;
  y1 = y1 < (size_t)H ? y1 : (size_t)H;
  float* dxm = maps.dx[ch];
  float* dym = maps.dy[ch];
  float* cfm = maps.conf[ch];
  float accum_dx = dxm[cell] * scale_down;
  float accum_dy = dym[cell] * scale_down;
  if (x1 <= x0 + 4 || y1 <= y0 + 4) {
    if (threadIdx.x == 0) {
      dxm[cell] = accum_dx * scale_up;
      dym[cell] = accum_dy * scale_up;
    }
    return;
  }
  const int iw = (int)(x1 - x0) - 2, ih = (int)(y1 - y0) - 2;  // interior extent
  const int npx = iw * ih;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // k / iw by a multiply-high: exact while npx * iw < 2^32, which holds for
  // every cell whose sides are below 1600 px (beyond, the division itself)
  const unsigned iw_m = 0xFFFFFFFFu / (unsigned)iw + 1u;
  const bool small = iw > 1 && iw < 1600 && ih < 1600;
  float min_eig_final = 0.f;
  // The matrix of the normal equations depends on G alone, so the first
  // iteration forms it for all (a lane's sums of later ones would be the same,
  // bit for bit); later iterations sum the right-hand side only.
  double A00 = 0.0, A01 = 0.0, A11 = 0.0;
  for (int iter = 0; iter < max_iterations; iter++) {
    double bx = 0.0, by = 0.0;
    // A pixel whose whole displaced cell lies inside the image needs no clamps.
    const bool inside = (float)x0 + accum_dx >= 0.f && (float)(x1 + 1) + accum_dx < (float)W &&
                        (float)y0 + accum_dy >= 0.f && (float)(y1 + 1) + accum_dy < (float)H;
    auto sweep = [&](auto in, auto first) {
      constexpr bool IN = decltype(in)::value, FIRST = decltype(first)::value;
#pragma unroll 4
      for (int k = threadIdx.x; k < npx; k += LK_THREADS) {
        const int yy = small ? (int)__umulhi((unsigned)k, iw_m) : k / iw;
        const int x = (int)x0 + 1 + k - yy * iw, y = (int)y0 + 1 + yy;
        const size_t i = (size_t)y * W + x;
        const float gc = G[i];
        const float gx = G[i + 1] - G[i - 1];
        const float gy = G[i + W] - G[i - W];
        const float tx = (float)x + accum_dx, ty = (float)y + accum_dy;
        float t_warp;
        if (IN) {
          const int xi = (int)tx, yi = (int)ty;
          const float fx = tx - (float)xi, fy = ty - (float)yi;
          const float* q = T + ((size_t)yi * W + xi);
          t_warp = (q[0] * (1.f - fx) + q[1] * fx) * (1.f - fy) + (q[W] * (1.f - fx) + q[W + 1] * fx) * fy;
        } else {
          t_warp = bilinear_plane(T, W, H, tx, ty);
        }
        const float err = t_warp - gc;
        const double dx = (double)gx, dy = (double)gy, de = (double)err;
        if (FIRST) {
          A00 += dx * dx;
          A01 += dx * dy;
          A11 += dy * dy;
        }
        bx -= dx * de;
        by -= dy * de;
      }
    };
    const std::true_type yes{};
    const std::false_type no{};
    if (inside) {
      if (iter == 0) sweep(yes, yes); else sweep(yes, no);
    } else {
      if (iter == 0) sweep(no, yes); else sweep(no, no);
    }
    if (iter == 0) {
      A00 = warp_sum_d(A00);
      A01 = warp_sum_d(A01);
      A11 = warp_sum_d(A11);
    }
    bx = warp_sum_d(bx);
    by = warp_sum_d(by);
    if (lane == 0) {
      red[0][wid] = A00;
      red[1][wid] = A01;
      red[2][wid] = A11;
      red[3][wid] = bx;
      red[4][wid] = by;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double s[5] = {0, 0, 0, 0, 0};
      for (int w = 0; w < LK_THREADS / 32; w++)
        for (int q = 0; q < 5; q++) s[q] += red[q][w];
      int done = 0;
      if (npx < 32) {
        done = 1;
      } else {
        const double det = s[0] * s[2] - s[1] * s[1];
        const double trace = s[0] + s[2];
        const double disc = fmax(0.0, trace * trace - 4.0 * det);
        const double sq = sqrt(disc);
        min_eig_final = (float)(0.5 * (trace - sq));
        if (det <= 1e-12) {
          done = 1;
        } else {
          const double inv = 1.0 / det;
          const double step_x = inv * (s[2] * s[3] - s[1] * s[4]);
          const double step_y = inv * (-s[1] * s[3] + s[0] * s[4]);
          accum_dx += (float)step_x;
          accum_dy += (float)step_y;
          if (accum_dx > max_shift) accum_dx = max_shift;
          if (accum_dx < -max_shift) accum_dx = -max_shift;
          if (accum_dy > max_shift) accum_dy = max_shift;
          if (accum_dy < -max_shift) accum_dy = -max_shift;
          if (fabs(step_x) < 0.005 && fabs(step_y) < 0.005) done = 1;
        }
      }
      s_acc[0] = accum_dx;
      s_acc[1] = accum_dy;
      s_done = done;
    }
    __syncthreads();
    accum_dx = s_acc[0];
    accum_dy = s_acc[1];
    const int done = s_done;
    __syncthreads();
    if (done) break;
  }
  if (threadIdx.x == 0) {
    dxm[cell] = accum_dx * scale_up;
    dym[cell] = accum_dy * scale_up;
    cfm[cell] = fmaxf(0.f, min_eig_final);
  }
}

// Confidence gate (relative to the strongest cell) and one 3x3 smoothing
// pass of each map.  One CTA; `tmp` holds 4 * n floats.
__global__ void k_lk_gate_smooth(LkMaps maps, int map_w, int map_h, float min_conf, float* tmp) {
  __shared__ float s_max[2][32];
  const int n = map_w * map_h;
  for (int ch = 0; ch < 2; ch++) {
    float m = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = smax(m, maps.conf[ch][i]);
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) s_max[ch][threadIdx.x >> 5] = m;
  }
  __syncthreads();
  for (int ch = 0; ch < 2; ch++) {
    float maxc = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) maxc = smax(maxc, s_max[ch][w]);
    if (maxc <= 0.f) continue;
    const float thr = maxc * min_conf;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      if (maps.conf[ch][i] < thr) {
        maps.dx[ch][i] = 0.f;
        maps.dy[ch][i] = 0.f;
      }
  }
  __syncthreads();
  float* m4[4] = {maps.dx[0], maps.dy[0], maps.dx[1], maps.dy[1]};
  for (int q = 0; q < 4; q++) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int cy = i / map_w, cx = i % map_w;
      float acc = 0.f;
      int cnt = 0;
      for (int dy = -1; dy <= 1; dy++)
        for (int dx = -1; dx <= 1; dx++) {
          const int yy = cy + dy, xx = cx + dx;
          if (yy < 0 || yy >= map_h || xx < 0 || xx >= map_w) continue;
          acc += m4[q][yy * map_w + xx];
          cnt++;
        }
      tmp[q * n + i] = cnt > 0 ? acc / (float)cnt : 0.f;
    }
  }
  __syncthreads();
  for (int q = 0; q < 4; q++)
    for (int i = threadIdx.x; i < n; i += blockDim.x) m4[q][i] = tmp[q * n + i];
}

struct ShiftMaps {
  const float* dx;
  const float* dy;
};

// The two map cells around a coordinate, and how far between them it lies.
__device__ __forceinline__ void map_place(float p, float cell, int n, int& g0, int& g1, float& f) {
  const float g_f = (p / cell) - 0.5f;
  g0 = (int)floorf(g_f);
  if (g0 < 0) g0 = 0;
  if (g0 >= n - 1) g0 = n - 2;
  if (g0 < 0) g0 = 0;
  f = sclamp(g_f - g0, 0.f, 1.f);
  g1 = min(g0 + 1, n - 1);
}

constexpr int RM_B = 4;  // rows in flight

// A warp's 32 columns over ROWS rows.  The shift is bilinear in the map, so
// its two horizontal means (of either map row, for four maps) stay in registers
// while the rows stay between the same two map rows, and a pixel costs the
// vertical mean alone, not 16 map loads and two divisions each way; the rows'
// divisions are one, a row to a lane.  Four rows are sampled together without
// clamps or branches where all their samples lie inside (a warp's vote): what
// bounds the pass is the wait for its loads.  The interleaved rows go out
// through shared memory, in whole sectors.
// 26 MP: 288 us before, 177 us; its 24 B per pixel take 95 us.  (One row at a
// time 287 us; three CTAs per SM 206 us, five, which spill, 201 us.)
template <int ROWS>
__global__ void __launch_bounds__(256, 4)
    k_lk_remap(const float* __restrict__ R0, const float* __restrict__ G0, const float* __restrict__ B0,
               float* __restrict__ dst, int W, int H, ShiftMaps mr, ShiftMaps mb, int map_w, int map_h, float cell,
               float clamp_shift) {
  __shared__ float stage[8][RM_B][96];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const float* const m[4] = {mr.dx, mr.dy, mb.dx, mb.dy};
  const float xe = (float)(W - 1), ye = (float)(H - 1);
  for (int yb = (blockIdx.y * 8 + wid) * ROWS; yb < H; yb += gridDim.y * 8 * ROWS)
    for (int xb = blockIdx.x * 32; xb < W; xb += gridDim.x * 32) {
      const int x = min(xb + lane, W - 1), live = min(32, W - xb) * 3;
      int gx0, gx1, ly0, ly1, held = -1;
      float fx, lfy, up[4], dn[4];
      map_place((float)x, cell, map_w, gx0, gx1, fx);
      map_place((float)(yb + lane), cell, map_h, ly0, ly1, lfy);
      const int y_end = min(yb + ROWS, H);
      for (int y0 = yb; y0 < y_end; y0 += RM_B) {
        float sx[RM_B][2], sy[RM_B][2];
        bool in = true;
#pragma unroll
        for (int j = 0; j < RM_B; j++) {
          const int y = min(y0 + j, y_end - 1);
          const int gy0 = __shfl_sync(~0u, ly0, y - yb);
          const float fy = __shfl_sync(~0u, lfy, y - yb);
          if (gy0 != held) {
            held = gy0;
            const int gy1 = min(gy0 + 1, map_h - 1);
#pragma unroll
            for (int q = 0; q < 4; q++) {
              up[q] = m[q][gy0 * map_w + gx0] * (1.f - fx) + m[q][gy0 * map_w + gx1] * fx;
              dn[q] = m[q][gy1 * map_w + gx0] * (1.f - fx) + m[q][gy1 * map_w + gx1] * fx;
            }
          }
#pragma unroll
          for (int q = 0; q < 2; q++) {
            sx[j][q] = (float)x + sclamp(up[2 * q] * (1.f - fy) + dn[2 * q] * fy, -clamp_shift, clamp_shift);
            sy[j][q] = (float)y + sclamp(up[2 * q + 1] * (1.f - fy) + dn[2 * q + 1] * fy, -clamp_shift, clamp_shift);
            in = in && sx[j][q] >= 0.f && sy[j][q] >= 0.f && sx[j][q] < xe && sy[j][q] < ye;
          }
        }
        const float* const src[2] = {R0, B0};
        if (__all_sync(~0u, in)) {
          float v[RM_B][2][4], g[RM_B];
#pragma unroll
          for (int j = 0; j < RM_B; j++) {
            g[j] = G0[(size_t)min(y0 + j, y_end - 1) * W + x];
#pragma unroll
            for (int q = 0; q < 2; q++) {
              const float* p = src[q] + ((size_t)(int)sy[j][q] * W + (int)sx[j][q]);
              v[j][q][0] = p[0];
              v[j][q][1] = p[1];
              v[j][q][2] = p[W];
              v[j][q][3] = p[W + 1];
            }
          }
#pragma unroll
          for (int j = 0; j < RM_B; j++) {
            stage[wid][j][lane * 3 + 1] = g[j];
#pragma unroll
            for (int q = 0; q < 2; q++) {
              const float tx = sx[j][q] - (float)(int)sx[j][q], ty = sy[j][q] - (float)(int)sy[j][q];
              stage[wid][j][lane * 3 + 2 * q] = (v[j][q][0] * (1.f - tx) + v[j][q][1] * tx) * (1.f - ty) +
                                                (v[j][q][2] * (1.f - tx) + v[j][q][3] * tx) * ty;
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < RM_B; j++) {
            stage[wid][j][lane * 3 + 1] = G0[(size_t)min(y0 + j, y_end - 1) * W + x];
#pragma unroll
            for (int q = 0; q < 2; q++)
              stage[wid][j][lane * 3 + 2 * q] = bilinear_plane(src[q], W, H, sx[j][q], sy[j][q]);
          }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < RM_B; j++)
#pragma unroll
          for (int k = 0; k < 3; k++)
            if (y0 + j < y_end && lane + 32 * k < live)
              dst[((size_t)(y0 + j) * W + xb) * 3 + lane + 32 * k] = stage[wid][j][lane + 32 * k];
        __syncwarp();
      }
    }
}

__global__ void k_zero(float* p, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = 0.f;
}

int effective_levels(size_t W0, size_t H0, int levels) {
  int e = levels;
  while (e > 1 && ((W0 >> (e - 1)) < 32 || (H0 >> (e - 1)) < 32)) e--;
  return e;
}

}  // namespace

size_t ws_bytes_lateral(size_t w, size_t h, int cell, int levels, bool in_place) {
  (void)in_place;
  if (cell < 16) cell = 16;
  if (levels < 1) levels = 1;
  size_t total = 0;
  size_t lw = w, lh = h;
  for (int l = 0; l < levels; l++) {
    total += 3 * (((lw * lh * 4) + 255) & ~size_t(255));
    lw /= 2;
    lh /= 2;
  }
  size_t mw = std::max<size_t>(2, (w + cell - 1) / cell), mh = std::max<size_t>(2, (h + cell - 1) / cell);
  total += 10 * (((mw * mh * 4) + 255) & ~size_t(255));
  return total + 4096;
}

lre_status launch_lateral_ca(Context* c, const float* in, float* out, size_t w, size_t h, int cell, int iters,
                             float max_shift, float min_conf, int levels) {
  if (cell < 16) cell = 16;
  if (iters < 1) iters = 1;
  if (levels < 1) levels = 1;
  const int eff = effective_levels(w, h, levels);
  std::vector<float*> Rl(eff), Gl(eff), Bl(eff);
  std::vector<int> Wl(eff), Hl(eff);
  Wl[0] = (int)w;
  Hl[0] = (int)h;
  for (int l = 1; l < eff; l++) {
    Wl[l] = Wl[l - 1] / 2;
    Hl[l] = Hl[l - 1] / 2;
  }
  for (int l = 0; l < eff; l++) {
    size_t n = (size_t)Wl[l] * Hl[l];
    Rl[l] = reinterpret_cast<float*>(c->ws.take(n * 4));
    Gl[l] = reinterpret_cast<float*>(c->ws.take(n * 4));
    Bl[l] = reinterpret_cast<float*>(c->ws.take(n * 4));
    if (!Rl[l] || !Gl[l] || !Bl[l]) return fail(c, LRE_ERR_OUT_OF_MEMORY, "ca_register_lateral: workspace too small");
  }
  const int map_w = (int)std::max<size_t>(2, (w + cell - 1) / cell);
  const int map_h = (int)std::max<size_t>(2, (h + cell - 1) / cell);
  const size_t ncell = (size_t)map_w * map_h;
  LkMaps maps;
  float* mapmem = reinterpret_cast<float*>(c->ws.take(10 * ncell * 4));
  if (!mapmem) return fail(c, LRE_ERR_OUT_OF_MEMORY, "ca_register_lateral: workspace too small");
  maps.dx[0] = mapmem;
  maps.dy[0] = mapmem + ncell;
  maps.conf[0] = mapmem + 2 * ncell;
  maps.dx[1] = mapmem + 3 * ncell;
  maps.dy[1] = mapmem + 4 * ncell;
  maps.conf[1] = mapmem + 5 * ncell;
  float* tmp = mapmem + 6 * ncell;

  if (eff > 1) {
    const dim3 g((unsigned)std::min<size_t>((w + 63) / 64, 1024), (unsigned)std::min<size_t>((h + 15) / 16, 8192));
    k_split_down<<<g, dim3(32, 8), 0, c->stream>>>(in, Rl[0], Gl[0], Bl[0], Rl[1], Gl[1], Bl[1], (int)w, (int)h,
                                                   reinterpret_cast<uintptr_t>(in) % 8 == 0);
  } else {
    k_split_planes<<<grid_for(w * h, 256, c->sm_count * 8), 256, 0, c->stream>>>(in, Rl[0], Gl[0], Bl[0], w * h);
  }
  k_zero<<<grid_for(6 * ncell, 256, 64), 256, 0, c->stream>>>(mapmem, 6 * ncell);
  count_launch(c, 2);
  for (int l = 2; l < eff; l++) {
    Planes3 p{{Rl[l - 1], Gl[l - 1], Bl[l - 1]}, {Rl[l], Gl[l], Bl[l]}};
    k_downsample3<<<grid_for((size_t)Wl[l] * Hl[l], 256, c->sm_count * 8), 256, 0, c->stream>>>(p, Wl[l - 1], Hl[l - 1],
                                                                                                Wl[l], Hl[l]);
    count_launch(c);
  }
  // Up to two CTAs per SM, or five of large cells, the form for few CTAs: 511x341,
  // cell 96 (48 CTAs) 36 us, 44 with the other; 1200x800 (234) 53 and 59; 1536x1024
  // (352) 83 and 73; cells of 400 at 26 MP (352) 1066 and 1522, of 200 at 12 MP (600)
  // 408 and 420, at 26 MP (1344) 819 and 803.
  const bool few = 2 * ncell <= (size_t)c->sm_count * (cell >= 160 ? 5 : 2);
  for (int L = eff - 1; L >= 0; L--) {
    const float scale_down = 1.f / (float)(1 << L);
    const float level_max_shift = max_shift * scale_down + (float)(1 << L) * 0.5f;
    const float scale_up = (float)(1 << L);
    dim3 grid((unsigned)ncell, 2);
    auto level = few ? k_lk_level<2> : k_lk_level<5>;
    level<<<grid, LK_THREADS, 0, c->stream>>>(Gl[L], Rl[L], Bl[L], Wl[L], Hl[L], map_w, map_h, iters, level_max_shift,
                                              scale_down, scale_up, maps);
    count_launch(c);
  }
  k_lk_gate_smooth<<<1, 1024, 0, c->stream>>>(maps, map_w, map_h, min_conf, tmp);
  const float clamp_shift = max_shift * (float)(1 << (eff - 1));
  // Sixteen rows a thread where that leaves eight CTAs per SM, else four: 0.2 MP 4.4
  // us, 10.0 with sixteen; 3 MP 24.8 and 26.2; 6 MP 46.8 and 46.4; 26 MP 193 and 177.
  const size_t strips = (w + 31) / 32;
  const bool tall = strips * ((h + 127) / 128) >= (size_t)c->sm_count * 8;
  const int rows = tall ? 16 : 4;
  const dim3 rg((unsigned)std::min<size_t>(strips, 1024), (unsigned)std::min<size_t>((h + 8 * rows - 1) / (8 * rows), 8192));
  auto remap = tall ? k_lk_remap<16> : k_lk_remap<4>;
  remap<<<rg, 256, 0, c->stream>>>(
      Rl[0], Gl[0], Bl[0], out, (int)w, (int)h, ShiftMaps{maps.dx[0], maps.dy[0]}, ShiftMaps{maps.dx[1], maps.dy[1]},
      map_w, map_h, (float)cell, clamp_shift);
  count_launch(c, 2);
  return check_launch(c, "ca_register_lateral");
}

}  // namespace lre

// k_xtrans.cu -- X-Trans demosaic: fast 1-pass interpolation and the 3-pass
// Markesteijn interpolation (RawTherapee's algorithm as ported in
// libraw_enhanced, YPbPr derivative variant), plus the X-Trans border fill.
//
// Semantics: core/cpu_accelerator.cpp:1664-2762 (XTrans_Processor):
//   xtrans_border_interpolate (:1806-1861), run_3pass (:1870-2676),
//   run_1pass (:2679-2762).
//
// 3-pass device design: the reference's 114 x 114 tiles (step 98, origin 3)
// are kept -- its homogeneity maps read outside the rows a tile computes at
// the first/last tile rows and columns, so the tiling is part of the result.
// One CTA runs one tile at a time; positions a tile reads without computing
// read zeros (a freshly allocated reference buffer).  Two kernels:
// * k_xtrans_3pass_planes, for every pattern whose row scans a host replay
//   reduces to "every site of the class" (the X-Trans layouts and their
//   shifts): one direction plane at a time in shared memory, every step one
//   site per thread;
// * k_xtrans_3pass, for any other pattern: the reference's row scans, one
//   row per thread in its column order, with the whole tile (8 directions x
//   114^2 RGB, derivatives, homogeneity maps) in a per-CTA global slab.
#include <cfloat>
#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "lre_internal.h"

namespace lre {

namespace {

constexpr int XTS = 114;
constexpr int NDIR = 8;
constexpr int XT_THREADS = 512;
constexpr int kXtCtasPerSm = 2;
constexpr int kXtMaxCtas = 148 * kXtCtasPerSm;

struct XtParams {
  char xt[6][6];
  short allhex0[3][3][8];
  short allhex1[3][3][8];
  int sgrow, sgcol;
  int right_shift[3];
};

struct XtArgs {
  const float* raw;
  const float* norm;  // dense raw / maximum (plane-resident kernel)
  int cstride;
  float* rgb_out;
  int W, H;
  float maximum;
  int n_top, n_left;
  unsigned char* scratch;
  int* tile_counter;
  int refill;  // clear and refill the plane for each direction (plane-resident kernel)
  XtParams P;
};

struct XtSlab {
  float* rgb;           // [NDIR][XTS][XTS][3]
  float2* gmm;          // [XTS][XTS/2] (min, max)
  float* drv;           // [NDIR][XTS-10][XTS-10]
  unsigned char* homo;  // [NDIR][XTS][XTS]
  unsigned char* homosum;
  unsigned char* homosummax;  // [XTS][XTS]
};

constexpr size_t kRgbBytes = (size_t)NDIR * XTS * XTS * 3 * 4;
constexpr size_t kGmmBytes = (size_t)XTS * (XTS / 2) * 8;
constexpr size_t kDrvBytes = (size_t)NDIR * (XTS - 10) * (XTS - 10) * 4;
constexpr size_t kHomoBytes = (size_t)NDIR * XTS * XTS;
constexpr size_t kHmaxBytes = (size_t)XTS * XTS;
constexpr size_t kXtSlabBytes = ((kRgbBytes + kGmmBytes + kDrvBytes + 2 * kHomoBytes + kHmaxBytes + 255) / 256) * 256;

__device__ XtSlab make_xt_slab(unsigned char* base) {
  XtSlab s;
  s.rgb = reinterpret_cast<float*>(base);
  base += kRgbBytes;
  s.gmm = reinterpret_cast<float2*>(base);
  base += kGmmBytes;
  s.drv = reinterpret_cast<float*>(base);
  base += kDrvBytes;
  s.homo = base;
  base += kHomoBytes;
  s.homosum = base;
  base += kHomoBytes;
  s.homosummax = base;
  return s;
}

__device__ __forceinline__ int xfc(const XtParams& P, int row, int col) { return P.xt[(row + 6) % 6][(col + 6) % 6]; }
__device__ __forceinline__ int xisgreen(const XtParams& P, int row, int col) { return P.xt[row % 3][col % 3] & 1; }

__device__ __forceinline__ float xraw(const XtArgs& A, int row, int col) {
  const size_t i = (size_t)row * A.W + col;
  const float v = A.cstride == 1 ? A.raw[i] : A.raw[i * 3 + xfc(A.P, row, col)];
  return v / A.maximum;
}
// raw_buffer_hex (:1691-1695): linear offset from (row, col), colour of the
// landing site.
__device__ __forceinline__ float xraw_hex(const XtArgs& A, int row, int col, int hex) {
  const long long pos = (long long)row * A.W + col + hex;
  float v;
  if (A.cstride == 1) {
    v = A.raw[pos];
  } else {  // the landing site's colour needs its (row, col)
    const int r = (int)(pos / A.W), c = (int)(pos % A.W);
    v = A.raw[pos * 3 + xfc(A.P, r, c)];
  }
  return v / A.maximum;
}

// n / d by a multiply-high, exact while n * d < 2^32 (every loop here); the
// per-site loops map a flat index to (row, column) every iteration.
struct XDiv {
  unsigned m;
  int d;
  __device__ explicit XDiv(int d_) : m(d_ > 1 ? 0xFFFFFFFFu / (unsigned)d_ + 1u : 0u), d(d_) {}
  __device__ __forceinline__ int div(int n) const { return (int)__umulhi((unsigned)n, m) + (d == 1 ? n : 0); }
};

// std::max(low, std::min(val, high)) -- LIM of core/metal/shader_common.h.
__device__ __forceinline__ float LIMf(float val, float low, float high) {
  float m = (high < val) ? high : val;
  return (low < m) ? m : low;
}
__device__ __forceinline__ float SQRf(float x) { return x * x; }

// --------------------------------------------------------- border fill
__device__ void xtrans_border_px(const XtArgs& A, int row, int col) {
  const float weight[3][3] = {{0.25f, 0.5f, 0.25f}, {0.5f, 0.f, 0.5f}, {0.25f, 0.5f, 0.25f}};
  const int W = A.W, H = A.H;
  float sum[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int v = (row == 0) ? 0 : -1;
  for (int y = (row > 0) ? row - 1 : 0; y < row + 2 && y < H; y++, v++) {
    int h = (col == 0) ? 0 : -1;
    for (int x = (col > 0) ? col - 1 : 0; x < col + 2 && x < W; x++, h++) {
      const int f = xfc(A.P, y, x);
      sum[f] += xraw(A, y, x) * weight[v + 1][h + 1];
      sum[f + 3] += weight[v + 1][h + 1];
    }
  }
  float* o = A.rgb_out + ((size_t)row * W + col) * 3;
  switch (xfc(A.P, row, col)) {
    case 0:
      o[0] = xraw(A, row, col);
      o[1] = (sum[1] / sum[4]);
      o[2] = (sum[2] / sum[5]);
      break;
    case 1:
      if (sum[3] == 0.f) {
        const float r = xraw(A, row, col);
        o[0] = o[1] = o[2] = r;
      } else {
        o[0] = (sum[0] / sum[3]);
        o[1] = xraw(A, row, col);
        o[2] = (sum[2] / sum[5]);
      }
      break;
    case 2:
      o[0] = (sum[0] / sum[3]);
      o[1] = (sum[1] / sum[4]);
      o[2] = xraw(A, row, col);
      break;
  }
}

__global__ void k_xtrans_border(XtArgs A, int border) {
  const int W = A.W, H = A.H;
  const long long n_tb = 2LL * border * W;
  const long long n_lr = 2LL * border * (H - 2 * border > 0 ? H - 2 * border : 0);
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n_tb + n_lr; k += (long long)gridDim.x * blockDim.x) {
    int row, col;
    if (k < n_tb) {
      const int b = (int)(k / W);
      col = (int)(k % W);
      row = b < border ? b : H - 2 * border + b;
    } else {
      const long long q = k - n_tb;
      const int b = (int)(q % (2 * border));
      row = border + (int)(q / (2 * border));
      col = b < border ? b : W - 2 * border + b;
    }
    if (row < 0 || row >= H || col < 0 || col >= W) continue;
    if (col >= border && col < W - border && row >= border && row < H - border) continue;
    xtrans_border_px(A, row, col);
  }
}

// --------------------------------------------------------- 1-pass (:2679-2762)
__global__ void k_xtrans_1pass(XtArgs A) {
  const float weight[3][3] = {{0.25f, 0.5f, 0.25f}, {0.5f, 0.0f, 0.5f}, {0.25f, 0.5f, 0.25f}};
  const int W = A.W, H = A.H;
  const long long n = (long long)(H - 2) * (W - 2);
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int row = 1 + (int)(k / (W - 2)), col = 1 + (int)(k % (W - 2));
    float sum[3] = {0.f, 0.f, 0.f};
    for (int v = -1; v <= 1; v++)
      for (int h = -1; h <= 1; h++) {
        const int sr = row + v, sc = col + h;
        const int c = xfc(A.P, sr, sc);
        const float raw_val = xraw(A, sr, sc);
        sum[c] += raw_val * weight[v + 1][h + 1];
      }
    float rgb[3];
    switch (xfc(A.P, row, col)) {
      case 0:
        rgb[0] = xraw(A, row, col);
        rgb[1] = sum[1] * 0.5f;
        rgb[2] = sum[2];
        break;
      case 1: {
        rgb[1] = xraw(A, row, col);
        if (xfc(A.P, row, col - 1) == xfc(A.P, row, col + 1)) {
          rgb[0] = sum[0];
          rgb[2] = sum[2];
        } else {
          rgb[0] = sum[0] * 1.3333333f;
          rgb[2] = sum[2] * 1.3333333f;
        }
      } break;
      default:
        rgb[0] = sum[0];
        rgb[1] = sum[1] * 0.5f;
        rgb[2] = xraw(A, row, col);
        break;
    }
    float* o = A.rgb_out + ((size_t)row * W + col) * 3;
    o[0] = rgb[0];
    o[1] = rgb[1];
    o[2] = rgb[2];
  }
}

// --------------------------------------------------------- 3-pass
__global__ void __launch_bounds__(XT_THREADS, kXtCtasPerSm) k_xtrans_3pass(XtArgs Ain) {
  const int ts = XTS;
  const int tid = threadIdx.x, nth = blockDim.x;
  // The pattern tables are indexed at run time; read from the kernel's
  // parameter block that would force a local-memory copy of it per thread,
  // so one copy goes to shared memory (constant-offset parameter loads).
  __shared__ XtArgs sA;
  {
    constexpr int NW = (int)(sizeof(XtArgs) / 4);
    const int* from = reinterpret_cast<const int*>(&Ain);
    int* to = reinterpret_cast<int*>(&sA);
#pragma unroll
    for (int k = 0; k < NW; k++)
      if (k % XT_THREADS == tid) to[k] = from[k];
  }
  __syncthreads();
  const XtArgs& A = sA;
  const XtParams& P = A.P;
  XtSlab S = make_xt_slab(A.scratch + (size_t)blockIdx.x * kXtSlabBytes);
  __shared__ int s_tile;
  const int W = A.W, H = A.H;
  bool zeroed_once = false;

  for (;;) {
    if (tid == 0) s_tile = atomicAdd(A.tile_counter, 1);
    __syncthreads();
    const int tile = s_tile;
    __syncthreads();
    if (tile >= A.n_top * A.n_left) break;
    const int top = 3 + (tile / A.n_left) * (ts - 16);
    const int left = 3 + (tile % A.n_left) * (ts - 16);
    const int mrow_g = min(top + ts, H - 3);  // global row bound of the computations
    const int mcol_g = min(left + ts, W - 3);

    // Fresh scratch (zeros) for tiles on the image border: only their
    // outputs read positions the tile never computes (the homogeneity maps
    // of the first/last tile rows and columns).  Interior tiles clear only
    // direction plane 0, as the reference does for every tile; they write
    // every other position before reading it.
    const bool border_tile = tile / A.n_left == 0 || tile / A.n_left == A.n_top - 1 || tile % A.n_left == 0 ||
                             tile % A.n_left == A.n_left - 1;
    if (border_tile || !zeroed_once) {
      float4* z = reinterpret_cast<float4*>(S.rgb);
      const size_t n4 = kXtSlabBytes / 16;
      for (size_t i = tid; i < n4; i += nth) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      zeroed_once = true;
    } else {
      // direction plane 0 is cleared for every tile (:2058)
      float4* z = reinterpret_cast<float4*>(S.rgb);
      for (int i = tid; i < XTS * XTS * 3 / 4; i += nth) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    float* rgb = S.rgb;
    auto RGB = [&](int d, int lr, int lc) -> float* { return rgb + (((size_t)d * ts + lr) * ts + lc) * 3; };

    // (a) green min / max per row (:1968-2053), one row per thread
    for (int row = top + tid; row < mrow_g; row += nth) {
      int leftstart = left;
      for (; leftstart < mcol_g; leftstart++)
        if (!xisgreen(P, row, leftstart)) break;
      int coloffset = (P.right_shift[row % 3] == 1 ? 3 : 1 + (xfc(P, row, leftstart + 1) & 1));
      float2* g = S.gmm + (size_t)(row - top) * (ts / 2);
      auto mm = [&](int col, const short* hex) {
        float minval = FLT_MAX, maxval = 0.f;
        for (int c = 0; c < 6; c++) {
          const float val = xraw_hex(A, row, col, hex[c]);
          minval = minval < val ? minval : val;
          maxval = maxval > val ? maxval : val;
        }
        return make_float2(minval, maxval);
      };
      if (coloffset == 3) {
        const short* hex = P.allhex0[row % 3][leftstart % 3];
        for (int col = leftstart; col < mcol_g; col += coloffset) g[(col - left) >> 1] = mm(col, hex);
      } else {
        int col = leftstart;
        if (coloffset == 2) {
          const short* hex = P.allhex0[row % 3][col % 3];
          g[(col - left) >> 1] = mm(col, hex);
          col += 2;
        }
        const short* hex = P.allhex0[row % 3][col % 3];
        for (; col < mcol_g - 1; col += 3) {
          const float2 v = mm(col, hex);
          g[(col - left) >> 1] = v;
          g[(col + 1 - left) >> 1] = v;
        }
        if (col < mcol_g) g[(col - left) >> 1] = mm(col, hex);
      }
    }
    // native samples into direction 0 (:2055-2061)
    const XDiv fdn(mcol_g - left);
    for (int i = tid; i < (mrow_g - top) * (mcol_g - left); i += nth) {
      const int lr = fdn.div(i), lc = i - lr * (mcol_g - left);
      const int row = top + lr, col = left + lc;
      RGB(0, lr, lc)[xfc(P, row, col)] = xraw(A, row, col);
    }
    __syncthreads();
    // copy direction 0 to 1..3, all but the last float (:2067-2069); the
    // planes are 16-byte aligned (ts*ts*3 floats apart), so 4 floats a step
    {
      constexpr int NF = XTS * XTS * 3 - 1;
      const float4* s4 = reinterpret_cast<const float4*>(rgb);
      for (int i = tid; i < NF / 4; i += nth) {
        const float4 v = s4[i];
        reinterpret_cast<float4*>(rgb + (size_t)1 * XTS * XTS * 3)[i] = v;
        reinterpret_cast<float4*>(rgb + (size_t)2 * XTS * XTS * 3)[i] = v;
        reinterpret_cast<float4*>(rgb + (size_t)3 * XTS * XTS * 3)[i] = v;
      }
      for (int i = (NF / 4) * 4 + tid; i < NF; i += nth) {
        const float v = rgb[i];
        rgb[(size_t)1 * XTS * XTS * 3 + i] = v;
        rgb[(size_t)2 * XTS * XTS * 3 + i] = v;
        rgb[(size_t)3 * XTS * XTS * 3 + i] = v;
      }
    }
    __syncthreads();
    // (b) green in 4 directions (:2071-2127), one row per thread
    for (int row = top + tid; row < mrow_g; row += nth) {
      int leftstart = left;
      for (; leftstart < mcol_g; leftstart++)
        if (!xisgreen(P, row, leftstart)) break;
      int coloffset = (P.right_shift[row % 3] == 1 ? 3 : 1 + (xfc(P, row, leftstart + 1) & 1));
      const float2* g = S.gmm + (size_t)(row - top) * (ts / 2);
      auto colors = [&](int col, const short* hex, float* color) {
        color[0] = 0.6796875f * (xraw_hex(A, row, col, hex[1]) + xraw_hex(A, row, col, hex[0])) -
                   0.1796875f * (xraw_hex(A, row, col, 2 * hex[1]) + xraw_hex(A, row, col, 2 * hex[0]));
        color[1] = 0.87109375f * xraw_hex(A, row, col, hex[3]) + xraw_hex(A, row, col, hex[2]) * 0.12890625f +
                   0.359375f * (xraw_hex(A, row, col, 0) - xraw_hex(A, row, col, -hex[2]));
        for (int c = 0; c < 2; c++)
          color[2 + c] = 0.640625f * xraw_hex(A, row, col, hex[4 + c]) + 0.359375f * xraw_hex(A, row, col, -2 * hex[4 + c]) +
                         0.12890625f * (2.f * xraw_hex(A, row, col, 0) - xraw_hex(A, row, col, 3 * hex[4 + c]) -
                                        xraw_hex(A, row, col, -3 * hex[4 + c]));
      };
      if (coloffset == 3) {
        const short* hex = P.allhex0[row % 3][leftstart % 3];
        for (int col = leftstart; col < mcol_g; col += coloffset) {
          float color[4];
          colors(col, hex, color);
          const float2 mmv = g[(col - left) >> 1];
          for (int c = 0; c < 4; c++) RGB(c, row - top, col - left)[1] = LIMf(color[c], mmv.x, mmv.y);
        }
      } else {
        const short* hexmod[2] = {P.allhex0[row % 3][leftstart % 3], P.allhex0[row % 3][(leftstart + coloffset) % 3]};
        for (int col = leftstart, hexindex = 0; col < mcol_g; col += coloffset, coloffset ^= 3, hexindex ^= 1) {
          const short* hex = hexmod[hexindex];
          float color[4];
          colors(col, hex, color);
          const float2 mmv = g[(col - left) >> 1];
          for (int c = 0; c < 4; c++) RGB(c ^ 1, row - top, col - left)[1] = LIMf(color[c], mmv.x, mmv.y);
        }
      }
    }
    __syncthreads();

    for (int pass = 0; pass < 3; pass++) {
      if (pass == 1) {
        // copy directions 0..3 into 4..7, all but the last float (:2131-2136)
        constexpr int NF = 4 * XTS * XTS * 3 - 1;
        const float4* s4 = reinterpret_cast<const float4*>(S.rgb);
        float4* d4 = reinterpret_cast<float4*>(S.rgb + (size_t)4 * XTS * XTS * 3);
        for (int i = tid; i < NF / 4; i += nth) d4[i] = s4[i];
        for (int i = (NF / 4) * 4 + tid; i < NF; i += nth) S.rgb[(size_t)4 * XTS * XTS * 3 + i] = S.rgb[i];
        __syncthreads();
        rgb = S.rgb + (size_t)4 * ts * ts * 3;
      }
      // (c) recalculate green from closer pixels (:2138-2183)
      if (pass) {
        for (int row = top + 2 + tid; row < mrow_g - 2; row += nth) {
          int leftstart = left + 2;
          for (; leftstart < mcol_g - 2; leftstart++)
            if (!xisgreen(P, row, leftstart)) break;
          int coloffset = (P.right_shift[row % 3] == 1 ? 3 : 1 + (xfc(P, row, leftstart + 1) & 1));
          const float2* g = S.gmm + (size_t)(row - top) * (ts / 2);
          // A site's three directions write three different planes and
          // read only their own plane, so all fifteen operands are loaded
          // before the three stores; sites stay in the reference's order.
          auto site = [&](int col, int f, const short* hex, int flip) {
            float v[3][5];
#pragma unroll
            for (int d = 3; d < 6; d++) {
              const float* rix = RGB((d - 2) ^ flip, row - top, col - left);
              const int o1 = hex[d] * 3, o2 = -2 * hex[d] * 3;
              v[d - 3][0] = rix[o2 + 1];
              v[d - 3][1] = rix[o1 + 1];
              v[d - 3][2] = rix[o1 + f];
              v[d - 3][3] = rix[o2 + f];
              v[d - 3][4] = rix[f];
            }
            const float2 mmv = g[(col - left) >> 1];
#pragma unroll
            for (int d = 3; d < 6; d++) {
              const float* q = v[d - 3];
              const float val = 0.33333333f * (q[0] + 2 * (q[1] - q[2]) - q[3]) + q[4];
              RGB((d - 2) ^ flip, row - top, col - left)[1] = LIMf(val, mmv.x, mmv.y);
            }
          };
          if (coloffset == 3) {
            int f = xfc(P, row, leftstart);
            const short* hex = P.allhex1[row % 3][leftstart % 3];
            for (int col = leftstart; col < mcol_g - 2; col += coloffset, f ^= 2) site(col, f, hex, 0);
          } else {
            int f = xfc(P, row, leftstart);
            const short* hexmod[2] = {P.allhex1[row % 3][leftstart % 3], P.allhex1[row % 3][(leftstart + coloffset) % 3]};
            for (int col = leftstart, hexindex = 0; col < mcol_g - 2;
                 col += coloffset, coloffset ^= 3, f = f ^ (coloffset & 2), hexindex ^= 1)
              site(col, f, hexmod[hexindex], 1);
          }
        }
        __syncthreads();
      }
      // (d) R/B at solitary green pixels (:2185-2222)
      {
        const int sgstartcol = (left - P.sgcol + 4) / 3 * 3 + P.sgcol;
        const int row0 = (top - P.sgrow + 4) / 3 * 3 + P.sgrow;
        // One solitary green per thread: along a row the scan toggles h once
        // per site (its inner loops toggle it an even number of times), so
        // the k-th site starts from h0 ^ 2 (k & 1); sites are independent.
        const int nrow = row0 < mrow_g - 2 ? (mrow_g - 2 - row0 + 2) / 3 : 0;
        const int ncol = sgstartcol < mcol_g - 2 ? (mcol_g - 2 - sgstartcol + 2) / 3 : 0;
        for (int item = tid; item < nrow * ncol; item += nth) {
          const int row = row0 + 3 * (item / ncol), k = item % ncol;
          const int col = sgstartcol + 3 * k;
          float color[3][6];
          {
            int h = xfc(P, row, sgstartcol + 1) ^ ((k & 1) << 1);
            float* rix = RGB(0, row - top, col - left);
            float diff[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int i = 1, d = 0; d < 6; d++, i ^= ts ^ 1, h ^= 2) {
              for (int c = 0; c < 2; c++, h ^= 2) {
                const int op = i * (1 << c) * 3, om = -i * (1 << c) * 3;
                const float g = rix[1] + rix[1] - rix[op + 1] - rix[om + 1];
                color[h][d] = g + rix[op + h] + rix[om + h];
                if (d > 1) diff[d] += SQRf(rix[op + 1] - rix[om + 1] - rix[op + h] + rix[om + h]) + SQRf(g);
              }
              if (d > 2 && (d & 1))
                if (diff[d - 1] < diff[d])
                  for (int c = 0; c < 2; c++) color[c * 2][d] = color[c * 2][d - 1];
              if ((d & 1) || d < 2) {
                for (int c = 0; c < 2; c++) rix[c * 2] = 0.5f * color[c * 2][d];
                rix += (size_t)ts * ts * 3;
              }
            }
          }
        }
      }
      __syncthreads();
      // (e) red for blue pixels and vice versa (:2224-2264), one row per
      // thread in the reference's column order
      for (int row = top + 3 + tid; row < mrow_g - 3; row += nth) {
        int leftstart = left + 3;
        for (; leftstart < mcol_g - 1; leftstart++)
          if (!xisgreen(P, row, leftstart)) break;
        int coloffset = (P.right_shift[row % 3] == 1 ? 3 : 1);
        const int c = ((row - P.sgrow) % 3) ? ts : 1;
        const int h = 3 * (c ^ ts ^ 1);
        auto body = [&](int col, int f) {
          float* rix = RGB(0, row - top, col - left);
          for (int d = 0; d < 4; d++, rix += (size_t)ts * ts * 3) {
            const int i = d > 1 || ((d ^ c) & 1) ||
                                  ((fabsf(rix[1] - rix[c * 3 + 1]) + fabsf(rix[1] - rix[-c * 3 + 1])) <
                                   2.f * (fabsf(rix[1] - rix[h * 3 + 1]) + fabsf(rix[1] - rix[-h * 3 + 1])))
                              ? c
                              : h;
            rix[f] = rix[1] + 0.5f * (rix[i * 3 + f] + rix[-i * 3 + f] - rix[i * 3 + 1] - rix[-i * 3 + 1]);
          }
        };
        if (coloffset == 3) {
          int f = 2 - xfc(P, row, leftstart);
          for (int col = leftstart; col < mcol_g - 3; col += coloffset, f ^= 2) body(col, f);
        } else {
          coloffset = xfc(P, row, leftstart + 1) == 1 ? 2 : 1;
          int f = 2 - xfc(P, row, leftstart);
          for (int col = leftstart; col < mcol_g - 3; col += coloffset, coloffset ^= 3, f = f ^ (coloffset & 2)) body(col, f);
        }
      }
      __syncthreads();
      // (f) R and B for 2x2 green blocks (:2266-2310), one row per thread in
      // the reference's column order
      int topstart = top + 2;
      for (; topstart < mrow_g - 2; topstart++)
        if ((topstart - P.sgrow) % 3) break;
      int leftstart = left + 2;
      for (; leftstart < mcol_g - 2; leftstart++)
        if ((leftstart - P.sgcol) % 3) break;
      const int coloffsetstart = 2 - (xfc(P, topstart, leftstart + 1) & 1);
      for (int row = topstart + tid; row < mrow_g - 2; row += nth) {
        if (!((row - P.sgrow) % 3)) continue;
        const short* hexmod[2] = {P.allhex1[row % 3][leftstart % 3], P.allhex1[row % 3][(leftstart + coloffsetstart) % 3]};
        for (int col = leftstart, coloffset = coloffsetstart, hexindex = 0; col < mcol_g - 2;
             col += coloffset, coloffset ^= 3, hexindex ^= 1) {
          float* rix = RGB(0, row - top, col - left);
          const short* hex = hexmod[hexindex];
          for (int d = 0; d < NDIR; d += 2, rix += (size_t)ts * ts * 3) {
            const int o0 = hex[d] * 3, o1 = hex[d + 1] * 3;
            if (hex[d] + hex[d + 1]) {
              const float g = 3 * rix[1] - 2 * rix[o0 + 1] - rix[o1 + 1];
              for (int c = 0; c < 4; c += 2) rix[c] = (g + 2 * rix[o0 + c] + rix[o1 + c]) * 0.33333333f;
            } else {
              const float g = 2 * rix[1] - rix[o0 + 1] - rix[o1 + 1];
              for (int c = 0; c < 4; c += 2) rix[c] = (g + rix[o0 + c] + rix[o1 + c]) * 0.5f;
            }
          }
        }
      }
      __syncthreads();
    }
    rgb = S.rgb;
    int mrow = mrow_g - top;
    int mcol = mcol_g - left;

    // (g) YPbPr derivatives (:2346-2405), yuv recomputed at the 3 taps
    {
      const int dn = XTS - 10;
      const int rows = mrow - 10, cols = mcol - 10;
      const XDiv fdrc(rows * cols), fdcl(cols);
      const int n = NDIR * rows * cols;
      // four items per thread and step: their 36 loads are issued before the
      // first store (a store to the derivative planes could otherwise alias
      // the next item's loads for the compiler)
      constexpr int U = 4;
      for (int i0 = tid; i0 < n; i0 += U * nth) {
        float res[U];
        int at[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int i = i0 + u * nth;
          at[u] = -1;
          if (i < n) {
            const int d = fdrc.div(i);
            const int rem = i - d * (rows * cols);
            const int q_ = fdcl.div(rem);
            const int row = 5 + q_, col = 5 + rem - q_ * cols;
            const int dv = d & 3;
            // direction steps 1, ts, ts + 1, ts - 1 of directions 0..3 (and 4..7)
            int f = dv == 0 ? 1 : (dv == 1 ? ts : (dv == 2 ? ts + 1 : ts - 1));
            f = f == 1 ? 1 : f - 8;
            // yuv buffer offset f (width ts-8) -> tile offset
            const int fr = (f == 1) ? 0 : 1, fc = (f == 1) ? 1 : (f - (XTS - 8));
            auto yuv = [&](int r, int c, float& y, float& uu, float& v) {
              const float* p = RGB(d, r, c);
              y = 0.2627f * p[0] + 0.6780f * p[1] + 0.0593f * p[2];
              uu = (p[2] - y) * 0.56433f;
              v = (p[0] - y) * 0.67815f;
            };
            float y0, u0, v0, yp, up, vp, ym, um, vm;
            yuv(row, col, y0, u0, v0);
            yuv(row + fr, col + fc, yp, up, vp);
            yuv(row - fr, col - fc, ym, um, vm);
            res[u] = SQRf(2 * y0 - yp - ym) + SQRf(2 * u0 - up - um) + SQRf(2 * v0 - vp - vm);
            at[u] = (d * dn + (row - 5)) * dn + (col - 5);
          }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
          if (at[u] >= 0) S.drv[at[u]] = res[u];
      }
    }
    __syncthreads();
    // (h) homogeneity maps (:2407-2496)
    {
      const int dn = XTS - 10;
      const int rows = mrow - 12, cols = mcol - 12;
      const XDiv fdh(cols);
      for (int i = tid; i < rows * cols; i += nth) {
        const int q_ = fdh.div(i), row = 6 + q_, col = 6 + i - q_ * cols;
        auto D = [&](int d, int r, int c) { return S.drv[((size_t)d * dn + (r - 5)) * dn + (c - 5)]; };
        float tr = D(0, row, col) < D(1, row, col) ? D(0, row, col) : D(1, row, col);
        for (int d = 2; d < NDIR; d++) tr = (D(d, row, col) < tr ? D(d, row, col) : tr);
        tr *= 8;
        // all eight counts first, then the stores: a byte store may alias
        // any load for the compiler, which would otherwise wait for each
        // direction's loads in turn
        unsigned char temp[NDIR];
#pragma unroll
        for (int d = 0; d < NDIR; d++) {
          temp[d] = 0;
          for (int v = -1; v <= 1; v++)
            for (int h = -1; h <= 1; h++) temp[d] += (D(d, row + v, col + h) <= tr ? 1 : 0);
        }
#pragma unroll
        for (int d = 0; d < NDIR; d++) S.homo[((size_t)d * ts + row) * ts + col] = temp[d];
      }
    }
    __syncthreads();
    if (H - top < ts + 4) mrow = H - top + 2;
    if (W - left < ts + 4) mcol = W - left + 2;
    // (j) 5x5 homogeneity sums and their max (:2504-2612).  Integer sums
    // (at most 25 * 9 = 225, no wrap), so they are formed separably: row
    // 5-sums first, into the derivative planes' memory (dead after (h)).
    const int r0 = min(top, 8), c0 = min(left, 8);
    unsigned char* hs5 = reinterpret_cast<unsigned char*>(S.drv);  // [NDIR][ts][ts]
    {
      const int rows = mrow - 8 - r0 + 4, cols = mcol - 8 - c0;
      const XDiv fdr(rows * cols), fdc(cols);
      for (int i = tid; i < NDIR * rows * cols; i += nth) {
        const int d = fdr.div(i), rem = i - d * (rows * cols);
        const int q_ = fdc.div(rem), row = r0 - 2 + q_, col = c0 + rem - q_ * cols;
        const unsigned char* hp = S.homo + ((size_t)d * ts + row) * ts + col;
        hs5[((size_t)d * ts + row) * ts + col] = (unsigned char)(hp[-2] + hp[-1] + hp[0] + hp[1] + hp[2]);
      }
    }
    __syncthreads();
    {
      const int rows = mrow - 8 - r0, cols = mcol - 8 - c0;
      const XDiv fdj(cols);
      for (int i = tid; i < rows * cols; i += nth) {
        const int q_ = fdj.div(i), row = r0 + q_, col = c0 + i - q_ * cols;
        unsigned char maxval = 0;
        for (int d = 0; d < NDIR; d++) {
          int s = 0;
          for (int v = -2; v <= 2; v++) s += hs5[((size_t)d * ts + row + v) * ts + col];
          const unsigned char hs = (unsigned char)s;
          S.homosum[((size_t)d * ts + row) * ts + col] = hs;
          if (d == 0 || maxval < hs) maxval = hs;
        }
        maxval -= maxval >> 3;
        S.homosummax[(size_t)row * ts + col] = maxval;
      }
    }
    __syncthreads();
    // (l) average the most homogeneous directions (:2614-2650)
    {
      const int rows = mrow - 8 - r0, cols = mcol - 8 - c0;
      const XDiv fdj(cols);
      for (int i = tid; i < rows * cols; i += nth) {
        const int q_ = fdj.div(i), row = r0 + q_, col = c0 + i - q_ * cols;
        unsigned char hm[8];
        for (int d = 0; d < 4; d++) hm[d] = S.homosum[((size_t)d * ts + row) * ts + col];
        for (int d = 4; d < NDIR; d++) {
          hm[d] = S.homosum[((size_t)d * ts + row) * ts + col];
          if (hm[d - 4] < hm[d]) hm[d - 4] = 0;
          else if (hm[d - 4] > hm[d]) hm[d] = 0;
        }
        float avg[4] = {0.f, 0.f, 0.f, 0.f};
        const unsigned char maxval = S.homosummax[(size_t)row * ts + col];
        for (int d = 0; d < NDIR; d++)
          if (hm[d] >= maxval) {
            const float* p = RGB(d, row, col);
            for (int c = 0; c < 3; c++) avg[c] += p[c];
            avg[3] += 1.f;
          }
        float* o = A.rgb_out + ((size_t)(row + top) * W + (col + left)) * 3;
        o[0] = fmaxf(0.f, avg[0] / avg[3]);
        o[1] = fmaxf(0.f, avg[1] / avg[3]);
        o[2] = fmaxf(0.f, avg[2] / avg[3]);
      }
    }
    __syncthreads();
  }
}

// --------------------------------------------------------- 3-pass, one plane on chip
// The interpolation steps (b) to (f) never mix direction planes: each
// direction's reads and writes stay in its own plane, and passes 1 and 2
// continue planes 4..7 from copies of planes 0..3 (:2131-2136).  So one CTA
// carries one plane at a time in shared memory through all of its passes:
// plane k through pass 0, whose derivatives (g) and RGB then go to the CTA's
// global scratch, and on in place as plane k + 4 through passes 1 and 2.  The
// green min/max table stays in shared memory for the whole tile.  The
// homogeneity steps stage the eight derivative planes back from the scratch
// and keep their byte maps in shared memory, and the final average reads the
// RGB planes back.  Every step visits each site of its class once and reads
// no value that the same step writes (xt_sites_ok replays the reference's
// scans), so each step runs one site per thread; sites stay in fresh-buffer
// semantics (zeros where a tile computes nothing).
//
// What bounds the kernel is the issue of instructions around a few shared
// loads per site, with 32 warps on the SM and a barrier after every step.  So:
// * A class of sites is one (row mod 3, column mod 3) of the tile, at most four
//   classes to a step.  256 threads take a class and a thread takes six of its
//   38 x 38 sites, whose places within the 3x3 blocks are the same for every
//   step: they stay in registers, and the class's hexagon offsets, directions
//   and strides are the same for a whole warp.  (A list of the sites in shared
//   memory, with the class looked up at each site in each step: twice the
//   instructions and four dependent loads ahead of the first sample.)
// * A step loads the samples of three sites before it stores one.
// * The plane is cleared once per tile, not once per plane: a slot that no step
//   writes stays zero, and one that a step writes is written before it is read
//   (xt_fresh_once looks at the pattern for that; any other is cleared for each
//   plane).
// * (g) walks along its direction and forms each pixel's luma and chroma once,
//   not three times; a pixel's own sample is the same in every plane, so two
//   floats per pixel of the tile's outputs go to the scratch, not three per
//   pixel of the tile (1.0 MB per CTA and tile, not 1.6).
// * The homogeneity counts read staged rows, and the 5x5 sums add four byte
//   columns per word.
// 26 MP: 4614 us before, 2805 us.  A tile takes about 295,000 cycles: (c) to (f)
// 84,000, (g) and the scratch's stores 61,000, (b) 20,000, (h) 49,000, (j) 11,000,
// (l) 45,000, of which most waits for the chosen samples: the CTAs' scratches
// together (142 MB) are more than L2 holds.  (Fetching them ahead, and stores
// that leave L2 first, moved that wait to other steps.)
constexpr int XS_THREADS = 1024;
constexpr int kXsMaxCtas = 148;
constexpr int XDN = XTS - 10;  // derivative plane edge
constexpr int XBS = XTS / 3;   // 3x3 blocks across a tile
constexpr int XS_CLS = 4;      // site classes of a step, at most
constexpr int XS_S = 6;        // sites per thread and class
constexpr int XS_B = 3;        // sites in flight
constexpr int XS_SAFE = 8 * XTS + 8;  // a site of every tile, for the mosaic loads of slots without one
constexpr size_t kPlaneFloats = (size_t)XTS * XTS * 3;
constexpr size_t kPlaneBytes = kPlaneFloats * 4;  // 155,952
// Samples of a site at the plane's edge may lie before the plane (they are
// loaded and not used): up to four rows and four columns, (c).
constexpr size_t kXsPad = ((4 * XTS + 5) * 12 + 15) / 16 * 16;
constexpr int XHS = 116;                          // byte-map row, whole words
constexpr size_t kXsMapBytes = (size_t)NDIR * XTS * XHS;
constexpr int XH_R = 13;  // rows of a homogeneity strip, XH_R + 2 staged
constexpr size_t kXsStageFloats = (size_t)NDIR * (XH_R + 2) * XDN;
constexpr size_t kXsOwn = (kXsPad + kPlaneBytes + kGmmBytes + 15) / 16 * 16;  // the own colours lie behind
constexpr size_t kXsSmemBytes = kXsOwn + (size_t)XTS * XTS;  // 226,468
constexpr size_t kXsSpillBytes = (((size_t)NDIR * XTS * XTS * 8 + kDrvBytes + 255) / 256) * 256;
static_assert(XTS % 3 == 0 && XBS == 38 && XS_S % XS_B == 0, "xs_site; five fields of site bits in a word");
static_assert(2 * kXsMapBytes <= kXsOwn, "byte maps");
static_assert(kXsMapBytes + 2 * kXsStageFloats * 4 + (size_t)XH_R * XDN * 4 <= kXsOwn, "homogeneity strips");
static_assert(kPlaneBytes % 16 == 0 && kXsMapBytes % 16 == 0 && XDN % 4 == 0 && XHS % 4 == 0, "vector accesses");

// raw / maximum for every mosaic site, in the reference's IEEE division
// (xraw), once per image: the plane-resident kernel reads each sample in
// several steps and for each of its four plane pairs.
__global__ void k_xt_normalize(XtArgs A, float* norm) {
  const long long n = (long long)A.W * A.H;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    norm[i] = A.cstride == 1 ? A.raw[i] / A.maximum : xraw(A, (int)(i / A.W), (int)(i % A.W));
}

__device__ __forceinline__ void xs_cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

__device__ __forceinline__ float2 xs_load_if(const float2* p, bool on) {
  float2 v = make_float2(0.f, 0.f);
  asm volatile("{.reg .pred q; setp.ne.s32 q, %3, 0; @q ld.global.v2.f32 {%0, %1}, [%2];}"
               : "+f"(v.x), "+f"(v.y)
               : "l"(p), "r"((int)on));
  return v;
}

struct XsPixel {
  float r, g, b, y, u, v;
  __device__ __forceinline__ void of(const float* p) {
    r = p[0];
    g = p[1];
    b = p[2];
    y = 0.2627f * r + 0.6780f * g + 0.0593f * b;
    u = (b - y) * 0.56433f;
    v = (r - y) * 0.67815f;
  }
};
__device__ __forceinline__ float xs_second(float m, float o, float p) { return SQRf(2 * o - p - m); }
// The two samples of a pixel that its own colour is not.
__device__ __forceinline__ float2 xs_two(float r, float g, float b, int own) {
  return make_float2(own == 0 ? g : r, own == 2 ? g : b);
}

// Block corner of slot s of a thread (of the 256 of its class), -1 where there
// is none.  Floats of neighbouring blocks lie 9 banks apart along a row and 2
// along a column, so a warp takes 32 blocks of one row, and the six columns left
// over four rows at a time, picked so that no two lanes meet in a bank: rows
// r, r + 1, r + 4, r + 5.  (Blocks in running order: two wavefronts to most
// loads, as a row ends within the warp.)
__device__ __forceinline__ int xs_site(int slot_warp, int lane) {
  if (slot_warp < XBS) return 3 * (slot_warp * XTS + lane);
  const int g = slot_warp - XBS, r = lane / 6;
  const int i = (g >> 1) * 8 + (g & 1) * 2 + (r & 1) + (r & 2) * 2, j = 32 + lane - 6 * r;
  return r < 4 && i < XBS ? 3 * (i * XTS + j) : -1;
}

struct XsTile {
  int nr, nc;          // computed extent
  int r0, r1, c0, c1;  // outputs
};

// (g) YPbPr derivatives of one finished direction plane D (:2346-2405) and
// the two interpolated samples of its outputs, into the CTA's scratch.  Reads
// the plane only.  ALONG: the direction's column step per row (0, 1, -1), or 2
// for the direction along the row.
template <int ALONG>
__device__ __forceinline__ void xs_derivatives(const float* pl, const unsigned char* own, float2* two, float* out,
                                               const XsTile& T) {
  constexpr int ts = XTS;
  const int rows = T.nr - 10, cols = T.nc - 10;
  static_assert(XDN + XH_R - 1 <= 128 && XDN <= 8 * XH_R && XDN <= 4 * 30, "four warps across, eight walks down");
  // A thread's pixels, from (row0, col0) in steps of (DR, DC): which of them have
  // a derivative and which are outputs, a bit each.
  constexpr int DR = ALONG == 2 ? 8 : 1, DC = ALONG == 2 ? 0 : ALONG;
  constexpr int OUT = ALONG == 1 || ALONG == -1 ? XH_R - 1 : 0;
  const int lane = threadIdx.x & 31, across = threadIdx.x & 127, down = threadIdx.x >> 7;
  const int row0 = 5 + (ALONG == 2 ? down : down * XH_R);
  const int col0 = ALONG == 2 ? 4 + 30 * (across >> 5) + lane : 5 + across - (ALONG == 1 ? OUT : 0);
  const int own_at = row0 * ts + col0;
  const float* p = pl + own_at * 3;
  auto bits = [&](int ra, int rb, int ca, int cb) {  // of the t with ra <= row < rb and ca <= col < cb
    int lo = row0 < ra ? (ra - row0 + DR - 1) / DR : 0, hi = min(XH_R, row0 < rb ? (rb - row0 + DR - 1) / DR : 0);
    if (DC == 0) {
      if (col0 < ca || col0 >= cb) hi = 0;
    } else if (DC == 1) {
      lo = max(lo, ca - col0);
      hi = min(hi, cb - col0);
    } else {
      lo = max(lo, col0 - cb + 1);
      hi = min(hi, col0 - ca + 1);
    }
    return hi > lo ? (1u << hi) - (1u << lo) : 0u;
  };
  unsigned m_d = bits(5, 5 + rows, 5, 5 + cols), m_o = m_d & bits(T.r0, T.r1, T.c0, T.c1);
  if (ALONG == 2 && (lane == 0 || lane == 31)) m_d = m_o = 0;
  out += (row0 - 5) * XDN + col0 - 5;
  two += own_at;
  auto emit = [&](int t, const XsPixel& o, float d) {
    if (m_d >> t & 1) out[t * (DR * XDN + DC)] = d;
    if (m_o >> t & 1) two[t * (DR * ts + DC)] = xs_two(o.r, o.g, o.b, own[own_at + t * (DR * ts + DC)]);
  };
  if (ALONG == 2) {
    // a warp per 30 pixels of a row; the neighbours' luma and chroma by shuffle
#pragma unroll
    for (int t = 0; t < XH_R; t++) {
      if (row0 + t * DR >= 5 + rows) break;
      XsPixel o;
      o.of(p + t * DR * ts * 3);
      const float d = xs_second(__shfl_up_sync(~0u, o.y, 1), o.y, __shfl_down_sync(~0u, o.y, 1)) +
                      xs_second(__shfl_up_sync(~0u, o.u, 1), o.u, __shfl_down_sync(~0u, o.u, 1)) +
                      xs_second(__shfl_up_sync(~0u, o.v, 1), o.v, __shfl_down_sync(~0u, o.v, 1));
      emit(t, o, d);
    }
  } else {
    // a thread walks XH_R rows; on a diagonal the columns shift with the rows,
    // so walks start up to XH_R - 1 columns outside (those pixels lie in the
    // rows above or below: read, not stored)
    if (m_d == 0) return;
    constexpr int STEP = (ts + ALONG) * 3;
    XsPixel m, o, nx;
    m.of(p - STEP);
    o.of(p);
#pragma unroll
    for (int t = 0; t < XH_R; t++) {
      if (row0 + t >= 5 + rows) break;
      nx.of(p + (t + 1) * STEP);
      emit(t, o, xs_second(m.y, o.y, nx.y) + xs_second(m.u, o.u, nx.u) + xs_second(m.v, o.v, nx.v));
      m = o;
      o = nx;
    }
  }
}

__device__ __forceinline__ void xs_plane_out(const float* pl, const unsigned char* own, float2* srgb, float* sdrv, int D,
                                             const XsTile& T) {
  float2* two = srgb + (size_t)D * XTS * XTS;
  float* out = sdrv + (size_t)D * XDN * XDN;
  // direction steps 1, ts, ts + 1, ts - 1 of directions 0..3 (and 4..7)
  switch (D & 3) {
    case 0: xs_derivatives<2>(pl, own, two, out, T); break;
    case 1: xs_derivatives<0>(pl, own, two, out, T); break;
    case 2: xs_derivatives<1>(pl, own, two, out, T); break;
    default: xs_derivatives<-1>(pl, own, two, out, T); break;
  }
  // outputs beyond the derivatives: tiles at the image's border
  if (T.r0 < 5 || T.c0 < 5 || T.r1 > T.nr - 5 || T.c1 > T.nc - 5) {
    const XDiv fd(T.c1 - T.c0);
    for (int i = threadIdx.x; i < (T.r1 - T.r0) * (T.c1 - T.c0); i += XS_THREADS) {
      const int q = fd.div(i), row = T.r0 + q, col = T.c0 + i - q * (T.c1 - T.c0);
      if (row >= 5 && row < T.nr - 5 && col >= 5 && col < T.nc - 5) continue;
      const int e = row * XTS + col;
      two[e] = xs_two(pl[e * 3], pl[e * 3 + 1], pl[e * 3 + 2], own[e]);
    }
  }
}

__global__ void __launch_bounds__(XS_THREADS, 1) k_xtrans_3pass_planes(XtArgs Ain) {
  constexpr int ts = XTS;
  extern __shared__ __align__(16) unsigned char xs_smem[];
  float* pl = reinterpret_cast<float*>(xs_smem + kXsPad);  // [XTS][XTS][3]
  float2* gmm = reinterpret_cast<float2*>(xs_smem + kXsPad + kPlaneBytes);  // [XTS][XTS/2] (min, max)
  unsigned char* own = xs_smem + kXsOwn;                           // [XTS][XTS] colour of the sample
  __shared__ int s_tile, s_cls[2 * XS_CLS];
  const int tid = threadIdx.x, nth = XS_THREADS;
  __shared__ XtArgs sA;
  {
    constexpr int NW = (int)(sizeof(XtArgs) / 4);
    const int* from = reinterpret_cast<const int*>(&Ain);
    int* to = reinterpret_cast<int*>(&sA);
#pragma unroll
    for (int k = 0; k < NW; k++)
      if (k % XS_THREADS == tid) to[k] = from[k];
  }
  const XtArgs& A = sA;
  const XtParams& P = A.P;
  // the corners of this thread's blocks, for either class list
  const int warp = tid >> 5, lane = tid & 31, nwarps = nth >> 5;
  constexpr int CW = XS_THREADS / XS_CLS / 32;  // warps of a class
  int e0[XS_S];
#pragma unroll
  for (int s = 0; s < XS_S; s++) e0[s] = xs_site((warp & (CW - 1)) + CW * s, lane);
  // Opaque before each step: the addresses that the steps derive from them, kept
  // over the loops by the compiler, would spill.
  auto fresh = [&]() {
#pragma unroll
    for (int s = 0; s < XS_S; s++) asm volatile("" : "+r"(e0[s]));
  };
  const int my = warp / CW;  // this thread's class

  if (tid == 0) s_tile = atomicAdd(Ain.tile_counter, 1);
  __syncthreads();
  for (;;) {
    const int tile = s_tile;
    if (tile >= A.n_top * A.n_left) break;
    const int W = A.W, H = A.H;
    float2* srgb = reinterpret_cast<float2*>(A.scratch + (size_t)blockIdx.x * kXsSpillBytes);  // [NDIR][XTS][XTS]
    float* sdrv = reinterpret_cast<float*>(srgb + (size_t)NDIR * ts * ts);                     // [NDIR][XDN][XDN]
    const int top = 3 + (tile / A.n_left) * (ts - 16);
    const int left = 3 + (tile % A.n_left) * (ts - 16);
    const int mrow_g = min(top + ts, H - 3);  // global row bound of the computations
    const int mcol_g = min(left + ts, W - 3);
    XsTile T;
    const int nr = T.nr = mrow_g - top, nc = T.nc = mcol_g - left;
    T.r0 = min(top, 8);
    T.c0 = min(left, 8);
    T.r1 = (H - top < ts + 4 ? H - top + 2 : nr) - 8;
    T.c1 = (W - left < ts + 4 ? W - left + 2 : nc) - 8;

    // the classes: non-green sites, and greens off the solitary ones' rows and
    // columns, by their place in a 3x3 block of the tile
    if (warp == 0) {
      const int r = top + lane / 3, c = left + lane % 3;
      const bool ng = lane < 9 && !(P.xt[r % 3][c % 3] & 1);
      const bool gg = lane < 9 && (r - P.sgrow) % 3 != 0 && (c - P.sgcol) % 3 != 0;
      const unsigned mn = __ballot_sync(~0u, ng), mg = __ballot_sync(~0u, gg), lt = (1u << lane) - 1;
      if (lane < 2 * XS_CLS) s_cls[lane] = -1;
      __syncwarp();
      if (ng) s_cls[__popc(mn & lt)] = lane;
      if (gg) s_cls[XS_CLS + __popc(mg & lt)] = lane;
    }
    __syncthreads();
    if (tid == 0) s_tile = atomicAdd(Ain.tile_counter, 1);  // the next one, read after this tile's barriers
    const int qn = s_cls[my], qg = s_cls[XS_CLS + my];
    const int an = qn < 0 ? 0 : qn / 3, bn = qn < 0 ? 0 : qn % 3, ag = qg < 0 ? 0 : qg / 3, bg = qg < 0 ? 0 : qg % 3;
    const int on = an * ts + bn, og = ag * ts + bg;
    const int r3 = (top + an) % 3, c3 = (left + bn) % 3;
    const int flip = P.right_shift[r3] == 1 ? 0 : 1;
    // six sites' bits each: in the tile, two and three off its edge, the own
    // colour being blue; two off the edge in the other list
    unsigned bits = 0;
    {
      unsigned blue = 0;  // by the parities of the block's row and column
#pragma unroll
      for (int q = 0; q < 4; q++)
        blue |= (P.xt[(top + an + 3 * (q >> 1)) % 6][(left + bn + 3 * (q & 1)) % 6] == 2 ? 1u : 0u) << q;
#pragma unroll
      for (int s = 0; s < XS_S; s++) {
        if (e0[s] < 0) continue;
        const int i = e0[s] / ts, j = e0[s] - i * ts;  // multiples of three
        auto edge = [&](int r, int c) { return min(min(r, nr - 1 - r), min(c, nc - 1 - c)); };
        if (qn >= 0) {
          const int d = edge(i + an, j + bn);
          if (d >= 0) bits |= 1u << s;
          if (d >= 2) bits |= 1u << (s + XS_S);
          if (d >= 3) bits |= 1u << (s + 2 * XS_S);
          bits |= (blue >> ((i & 1) * 2 + (j & 1)) & 1) << (s + 3 * XS_S);
        }
        if (qg >= 0 && edge(i + ag, j + bg) >= 2) bits |= 1u << (s + 4 * XS_S);
      }
    }
    const float* tb = A.norm + (size_t)top * W + left;

    // (a) green min / max (:1968-2053).  The scan stores a site's hexagon
    // min/max at its half-column slot; on rows with adjacent non-green pairs
    // it stores the first site's values at both sites' slots and computes
    // none for the second.
    {
      const bool second = !(P.xt[r3][(c3 + 2) % 3] & 1), first = !(P.xt[r3][(c3 + 1) % 3] & 1);
      int hex[6];
#pragma unroll
      for (int c = 0; c < 6; c++) hex[c] = P.allhex0[r3][c3][c];
      fresh();
#pragma unroll
      for (int s = 0; s < XS_S; s++) {
        const bool in = bits >> s & 1;
        const int e = in ? e0[s] + on : XS_SAFE, lr = e / ts, lc = e - lr * ts;
        const float* q = tb + ((size_t)lr * W + lc);
        float minval = FLT_MAX, maxval = 0.f;
#pragma unroll
        for (int c = 0; c < 6; c++) {
          const float val = __ldg(q + hex[c]);
          minval = minval < val ? minval : val;
          maxval = maxval > val ? maxval : val;
        }
        if (in && !(second && lc > 0)) {
          const float2 v = make_float2(minval, maxval);
          gmm[e >> 1] = v;  // = row * (ts / 2) + column / 2: ts is even
          if (first && lc + 1 < nc) gmm[(e + 1) >> 1] = v;
        }
      }
    }
    // the solitary greens of (d), a site per thread and round, with their first
    // colour; -1: none
    int ed[2];
    {
      const int sgstartcol = (left - P.sgcol + 4) / 3 * 3 + P.sgcol;
      const int row0 = (top - P.sgrow + 4) / 3 * 3 + P.sgrow;
      const int nrow = row0 < mrow_g - 2 ? (mrow_g - 2 - row0 + 2) / 3 : 0;
      const int ncol = sgstartcol < mcol_g - 2 ? (mcol_g - 2 - sgstartcol + 2) / 3 : 0;
      const XDiv fd(ncol);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int item = tid + q * nth;
        ed[q] = -1;
        if (item < nrow * ncol) {
          const int i = fd.div(item), row = row0 + 3 * i, kk = item - i * ncol;
          const int h0 = xfc(P, row, sgstartcol + 1) ^ ((kk & 1) << 1);
          ed[q] = ((row - top) * ts + (sgstartcol + 3 * kk - left)) | h0 << 16;
        }
      }
    }

    for (int k = 0; k < 4; k++) {
      // the plane's zeros and native samples (:2055-2061)
      if (k == 0 || A.refill) {
        for (int lc = lane; lc < ts; lc += 32) {
          const int c6 = (left + lc) % 6;
#pragma unroll
          for (int j = 0; j < (ts + 31) / 32; j++) {
            const int lr = warp + j * nwarps;
            if (lr >= ts) break;
            const int f = P.xt[(top + lr) % 6][c6];
            const float v = lr < nr && lc < nc ? __ldg(tb + (size_t)lr * W + lc) : 0.f;
            float* o = pl + (lr * ts + lc) * 3;
            o[0] = f == 0 ? v : 0.f;
            o[1] = f == 1 ? v : 0.f;
            o[2] = f == 2 ? v : 0.f;
            own[lr * ts + lc] = (unsigned char)f;
          }
        }
        __syncthreads();
      }
      // planes 1..3 are copies of plane 0 without its last float (:2067-2069)
      if (k && tid == 0) pl[kPlaneFloats - 1] = 0.f;
      // (b) the green of direction k at every non-green site (:2071-2127)
      {
        const int cdir = k ^ flip;
        const short* hex = P.allhex0[r3][c3];
        fresh();
        auto green = [&](auto color) {
#pragma unroll
          for (int s = 0; s < XS_S; s++) {
            const bool in = bits >> s & 1;
            const int e = in ? e0[s] + on : XS_SAFE, lr = e / ts, lc = e - lr * ts;
            const float v = color(tb + ((size_t)lr * W + lc));
            const float2 mmv = gmm[e >> 1];
            if (in) pl[e * 3 + 1] = LIMf(v, mmv.x, mmv.y);
          }
        };
        if (cdir == 0) {
          const int h0 = hex[0], h1 = hex[1];
          green([&](const float* q) {
            return 0.6796875f * (__ldg(q + h1) + __ldg(q + h0)) - 0.1796875f * (__ldg(q + 2 * h1) + __ldg(q + 2 * h0));
          });
        } else if (cdir == 1) {
          const int h2 = hex[2], h3 = hex[3];
          green([&](const float* q) {
            return 0.87109375f * __ldg(q + h3) + __ldg(q + h2) * 0.12890625f + 0.359375f * (__ldg(q) - __ldg(q - h2));
          });
        } else {
          const int h4 = hex[cdir + 2];
          green([&](const float* q) {
            return 0.640625f * __ldg(q + h4) + 0.359375f * __ldg(q - 2 * h4) +
                   0.12890625f * (2.f * __ldg(q) - __ldg(q + 3 * h4) - __ldg(q - 3 * h4));
          });
        }
      }
      __syncthreads();

      for (int pass = 0; pass < 3; pass++) {
        // (c) recalculate green from closer pixels (:2138-2183): direction
        // d = 3..5 updates plane (d - 2) ^ flip, reading green sites only
        if (pass) {
          const int dd = k ^ flip;
          if (dd) {
            const int hx = P.allhex1[r3][c3][dd + 2] * 3;
            fresh();
#pragma unroll
            for (int s0 = 0; s0 < XS_S; s0 += XS_B) {
              float val[XS_B];
#pragma unroll
              for (int j = 0; j < XS_B; j++) {
                const int s = s0 + j, e = e0[s] + on;
                const float *p = pl + e * 3, *p1 = p + hx, *p2 = p1 - 3 * hx;
                const int f = bits >> (s + 3 * XS_S) & 1 ? 2 : 0;
                const float2 mmv = gmm[e >> 1];
                val[j] = LIMf(0.33333333f * (p2[1] + 2 * (p1[1] - p1[f]) - p2[f]) + p[f], mmv.x, mmv.y);
              }
#pragma unroll
              for (int j = 0; j < XS_B; j++)
                if (bits >> (s0 + j + XS_S) & 1) pl[(e0[s0 + j] + on) * 3 + 1] = val[j];
            }
          }
          __syncthreads();
        }
        // (d) R/B at solitary green pixels (:2185-2222): plane k carries
        // direction k (k < 2), directions 2 and 3 (k = 2) or 4 and 5 (k = 3),
        // the second of a pair falling back to the first where its
        // difference is larger
        {
          // along i (1 or ts), the colour h at distance 1 and h ^ 2 at 2
          auto along = [&](const float* rix, int i, int h, float& r, float& b) {
            const float g1 = rix[1] + rix[1];
            const float p1 = rix[3 * i + 1], m1 = rix[-3 * i + 1], ph = rix[3 * i + h], mh = rix[-3 * i + h];
            const int h2 = h ^ 2;
            const float p2 = rix[6 * i + 1], m2 = rix[-6 * i + 1], qh = rix[6 * i + h2], nh = rix[-6 * i + h2];
            const float ga = g1 - p1 - m1, gb = g1 - p2 - m2;
            const float va = ga + ph + mh, vb = gb + qh + nh;
            r = h == 0 ? va : vb;
            b = h == 0 ? vb : va;
            float df = 0.f;
            df += SQRf(p1 - m1 - ph + mh) + SQRf(ga);
            df += SQRf(p2 - m2 - qh + nh) + SQRf(gb);
            return df;
          };
#pragma unroll
          for (int q = 0; q < 2; q++) {
            if (ed[q] < 0) continue;
            float* rix = pl + (ed[q] & 0xffff) * 3;
            const int h0 = ed[q] >> 16;
            float r, b;
            if (k < 2) {
              along(rix, k ? ts : 1, k ? h0 ^ 2 : h0, r, b);
            } else {
              float r1, b1;
              const float d0 = along(rix, 1, h0, r, b), d1 = along(rix, ts, h0 ^ 2, r1, b1);
              if (!(d0 < d1)) r = r1, b = b1;
            }
            rix[0] = 0.5f * r;
            rix[2] = 0.5f * b;
          }
        }
        __syncthreads();
        // (e) red for blue pixels and vice versa (:2224-2264): every non-green
        // site writes its other colour f = 2 - own
        {
          const bool off = (top + an - P.sgrow) % 3 != 0;
          const bool ask = !(k > 1 || ((k ^ (off ? ts : 1)) & 1));
          fresh();
          auto sites = [&](auto c_, auto h_) {
            constexpr int c = decltype(c_)::value, h = decltype(h_)::value;  // steps, as floats; h = 0: not asked for
#pragma unroll
            for (int s0 = 0; s0 < XS_S; s0 += XS_B) {
              float val[XS_B];
#pragma unroll
              for (int j = 0; j < XS_B; j++) {
                const int s = s0 + j;
                const float *p = pl + (e0[s] + on) * 3, *pf = p + (bits >> (s + 3 * XS_S) & 1 ? 0 : 2);
                const float g0 = p[1];
                float gp = p[c + 1], gm = p[1 - c], fp = pf[c], fm = pf[-c];
                if (h) {
                  const float hp = p[h + 1], hm = p[1 - h], qp = pf[h], qm = pf[-h];
                  if (!((fabsf(g0 - gp) + fabsf(g0 - gm)) < 2.f * (fabsf(g0 - hp) + fabsf(g0 - hm)))) {
                    gp = hp;
                    gm = hm;
                    fp = qp;
                    fm = qm;
                  }
                }
                val[j] = g0 + 0.5f * (fp + fm - gp - gm);
              }
#pragma unroll
              for (int j = 0; j < XS_B; j++) {
                const int s = s0 + j;
                if (bits >> (s + 2 * XS_S) & 1) pl[(e0[s] + on) * 3 + (bits >> (s + 3 * XS_S) & 1 ? 0 : 2)] = val[j];
              }
            }
          };
          using Row = std::integral_constant<int, 3 * ts>;
          using Col = std::integral_constant<int, 3>;
          using Row3 = std::integral_constant<int, 9 * ts>;
          using Col3 = std::integral_constant<int, 9>;
          using None = std::integral_constant<int, 0>;
          if (off) {
            if (ask) sites(Row{}, Col3{});
            else sites(Row{}, None{});
          } else {
            if (ask) sites(Col{}, Row3{});
            else sites(Col{}, None{});
          }
        }
        __syncthreads();
        // (f) R and B for 2x2 green blocks (:2266-2310): greens off the
        // solitary-green row and column classes, hexagon allhex1
        {
          const short* hex = P.allhex1[(top + ag) % 3][(left + bg) % 3];
          const int o0 = hex[2 * k] * 3, o1 = hex[2 * k + 1] * 3;
          const bool two = o0 + o1 != 0;
          const float wv = two ? 3.f : 2.f, wa = two ? 2.f : 1.f, wo = two ? 0.33333333f : 0.5f;
          fresh();
#pragma unroll
          for (int s0 = 0; s0 < XS_S; s0 += XS_B) {
            float v0[XS_B], v2[XS_B];
#pragma unroll
            for (int j = 0; j < XS_B; j++) {
              const float *p = pl + (e0[s0 + j] + og) * 3, *pa = p + o0, *pb = p + o1;
              // a factor of one leaves a value as it is: one form for both
              const float g = wv * p[1] - wa * pa[1] - pb[1];
              v0[j] = (g + wa * pa[0] + pb[0]) * wo;
              v2[j] = (g + wa * pa[2] + pb[2]) * wo;
            }
#pragma unroll
            for (int j = 0; j < XS_B; j++)
              if (bits >> (s0 + j + 4 * XS_S) & 1) {
                pl[(e0[s0 + j] + og) * 3] = v0[j];
                pl[(e0[s0 + j] + og) * 3 + 2] = v2[j];
              }
          }
        }
        __syncthreads();
        // plane k, and after passes 1 and 2 plane k + 4, is final: (g) its
        // derivatives and its RGB go to the scratch; it continues in place
        if (pass != 1) {
          xs_plane_out(pl, own, srgb, sdrv, pass ? k + 4 : k, T);
          __syncthreads();
        }
      }
    }

    // (h) homogeneity maps (:2407-2496) from the derivative planes, in strips of
    // XH_R rows staged a strip ahead
    unsigned char* homo = xs_smem;                 // [NDIR][XTS][XHS]
    unsigned char* hs5 = xs_smem + kXsMapBytes;    // [NDIR][XTS][XHS], after the strips
    float* stage = reinterpret_cast<float*>(hs5);  // 2 x [NDIR][XH_R + 2][XDN]
    float* tr = stage + 2 * kXsStageFloats;        // [XH_R][XDN]
    {
      const int rows = nr - 12, cols = nc - 12;  // >= 5: a tile computes 17 rows and columns at least
      const int strips = (rows + XH_R - 1) / XH_R;
      // the last strip begins early enough to be whole, if there are rows for it
      auto first = [&](int st) { return max(0, min(st * XH_R, rows - XH_R)); };
      auto fetch = [&](int st) {
        const int n = min(XH_R + 2, rows + 2) * (XDN / 4);
        float* to = stage + (st & 1) * kXsStageFloats;
        const float* from = sdrv + (size_t)first(st) * XDN;
        const XDiv fd(n);
        for (int i = tid; i < NDIR * n; i += nth) {
          const int d = fd.div(i), o = (i - d * n) * 4;
          xs_cp16(to + (size_t)d * (XH_R + 2) * XDN + o, from + (size_t)d * XDN * XDN + o);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      fetch(0);
      float4* z = reinterpret_cast<float4*>(homo);
      for (int i = tid; i < (int)(kXsMapBytes / 16); i += nth) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      const XDiv fd(cols);
      for (int st = 0; st < strips; st++) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // this strip is here; the last one's buffer and thresholds are free
        if (st + 1 < strips) fetch(st + 1);
        const float* b = stage + (st & 1) * kXsStageFloats;
        const int n = min(XH_R, rows);
        constexpr int DP = (XH_R + 2) * XDN;
        for (int i = tid; i < n * (XDN / 2); i += nth) {
          const int q = i / (XDN / 2), c = (i - q * (XDN / 2)) * 2;
          const float* dp = b + (q + 1) * XDN + c;
          float2 v[NDIR];
#pragma unroll
          for (int d = 0; d < NDIR; d++) v[d] = *reinterpret_cast<const float2*>(dp + d * DP);
          float x = v[0].x < v[1].x ? v[0].x : v[1].x, y = v[0].y < v[1].y ? v[0].y : v[1].y;
#pragma unroll
          for (int d = 2; d < NDIR; d++) {
            x = v[d].x < x ? v[d].x : x;
            y = v[d].y < y ? v[d].y : y;
          }
          *reinterpret_cast<float2*>(tr + q * XDN + c) = make_float2(x * 8, y * 8);
        }
        __syncthreads();
        for (int i = tid; i < NDIR * cols; i += nth) {
          const int d = fd.div(i), c = i - d * cols;
          const float* dp = b + d * DP + c;
          unsigned char* o = homo + (d * ts + 6 + first(st)) * XHS + 6 + c;
          float w[3][3];
#pragma unroll
          for (int v = 0; v < 2; v++)
#pragma unroll
            for (int h = 0; h < 3; h++) w[v + 1][h] = dp[v * XDN + h];
#pragma unroll
          for (int r = 0; r < XH_R; r++) {
            if (r >= n) break;
#pragma unroll
            for (int h = 0; h < 3; h++) {
              w[0][h] = w[1][h];
              w[1][h] = w[2][h];
              w[2][h] = dp[(r + 2) * XDN + h];
            }
            const float t = tr[r * XDN + c + 1];
            // counted in a float's low bits: the adds go to another pipe than
            // the comparisons
            float count = 8388608.f;
#pragma unroll
            for (int v = 0; v < 3; v++)
#pragma unroll
              for (int h = 0; h < 3; h++)
                if (w[v][h] <= t) count += 1.f;
            o[r * XHS] = (unsigned char)__float_as_int(count);
          }
        }
      }
    }
    __syncthreads();
    // (j) 5x5 homogeneity sums (:2504-2612), separably and four columns per
    // word: a byte counts to 9, its row sum to 45 and the whole to 225, so no
    // byte carries into the next (bytes beyond the outputs may; they carry
    // away from them).  Row sums first:
    const int rows = T.r1 - T.r0, cols = T.c1 - T.c0;
    const int q0 = T.c0 >> 2, nq = ((T.c1 - 1) >> 2) - q0 + 1;
    if (rows > 0 && cols > 0) {
      const XDiv fq(nq), fr(rows + 4);
      for (int i = tid; i < NDIR * (rows + 4) * nq; i += nth) {
        const int line = fq.div(i), d = fr.div(line);
        const int at = (d * ts + T.r0 - 2 + line - d * (rows + 4)) * XHS + (q0 + i - line * nq) * 4;
        const unsigned* hp = reinterpret_cast<const unsigned*>(homo + at);
        const unsigned w0 = hp[-1], w1 = hp[0], w2 = hp[1];
        *reinterpret_cast<unsigned*>(hs5 + at) = __funnelshift_r(w0, w1, 16) + __funnelshift_r(w0, w1, 24) + w1 +
                                                 __funnelshift_r(w1, w2, 8) + __funnelshift_r(w1, w2, 16);
      }
    }
    __syncthreads();
    // then columns, a thread down a quarter of them, over the counts' memory
    if (rows > 0 && cols > 0) {
      const XDiv fq(nq);
      const int seg = (rows + 3) / 4;
      for (int i = tid; i < NDIR * 4 * nq; i += nth) {
        const int line = fq.div(i), d = line >> 2, ra = T.r0 + (line & 3) * seg, rb = min(ra + seg, T.r1);
        const int at = d * ts * XHS + (q0 + i - line * nq) * 4;
        auto in = [&](int r) { return *reinterpret_cast<const unsigned*>(hs5 + at + r * XHS); };
        if (ra >= rb) continue;
        unsigned sum = in(ra - 2) + in(ra - 1) + in(ra) + in(ra + 1);
#pragma unroll 2
        for (int r = ra; r < rb; r++) {
          sum += in(r + 2);
          *reinterpret_cast<unsigned*>(homo + at + r * XHS) = sum;
          sum -= in(r - 2);
        }
      }
    }
    __syncthreads();
    // their max, and (l) the average of the most homogeneous directions
    // (:2614-2650), one output pixel per thread: which directions first, a bit
    // each over the row sums' memory, so that the second loop's loads wait for
    // one byte only
    if (rows > 0 && cols > 0) {
      const XDiv fd(cols);
      unsigned char* chosen = hs5;
#pragma unroll 2
      for (int i = tid; i < rows * cols; i += nth) {
        const int q = fd.div(i);
        const unsigned char* hp = homo + (T.r0 + q) * XHS + T.c0 + i - q * cols;
        int hm[NDIR], maxval = 0;
#pragma unroll
        for (int d = 0; d < NDIR; d++) {
          hm[d] = hp[d * ts * XHS];
          maxval = max(maxval, hm[d]);
        }
        maxval -= maxval >> 3;
        unsigned m = 0;
#pragma unroll
        for (int d = 0; d < NDIR / 2; d++) {
          // the lesser of a pair counts as zero
          if ((hm[d] < hm[d + 4] ? 0 : hm[d]) >= maxval) m |= 1u << d;
          if ((hm[d] > hm[d + 4] ? 0 : hm[d + 4]) >= maxval) m |= 16u << d;
        }
        chosen[i] = (unsigned char)m;
      }
      // (own writes: this thread's pixels)
#pragma unroll 2
      for (int i = tid; i < rows * cols; i += nth) {
        const int q = fd.div(i), row = T.r0 + q, col = T.c0 + i - q * cols;
        const unsigned m = chosen[i];
        const float nat = __ldg(tb + (size_t)row * W + col);
        const int f = own[row * ts + col];
        const float2* px = srgb + (row * ts + col);
        float2 p[NDIR];
#pragma unroll
        for (int d = 0; d < NDIR; d++) p[d] = xs_load_if(px + d * ts * ts, m & 1u << d);
        float ax = 0.f, ay = 0.f, an_ = 0.f;
#pragma unroll
        for (int d = 0; d < NDIR; d++) {
          ax += p[d].x;  // (a zero added changes no sum)
          ay += p[d].y;
          if (m & 1u << d) an_ += nat;
        }
        const float n = (float)__popc(m);
        ax = fmaxf(0.f, ax / n);
        ay = fmaxf(0.f, ay / n);
        an_ = fmaxf(0.f, an_ / n);
        float* o = A.rgb_out + ((size_t)(row + top) * W + (col + left)) * 3;
        o[0] = f == 0 ? an_ : ax;
        o[1] = f == 0 ? ax : (f == 1 ? an_ : ay);
        o[2] = f == 2 ? an_ : ay;
      }
    }
    __syncthreads();
  }
}

// allhex / solitary green / RightShift tables (:1887-1940), host side.
XtParams make_xt_params(const char* xtrans, int width) {
  XtParams P;
  memcpy(P.xt, xtrans, 36);
  const short orth[12] = {1, 0, 0, 1, -1, 0, 0, -1, 1, 0, 0, 1};
  const short patt[2][16] = {{0, 1, 0, -1, 2, 0, -1, 0, 1, 1, 1, -1, 0, 0, 0, 0},
                             {0, 1, 0, -2, 1, 0, -2, 0, 1, 1, -2, -2, 1, -1, -1, 1}};
  auto isg = [&](int row, int col) { return P.xt[row % 3][col % 3] & 1; };
  memset(P.allhex0, 0, sizeof(P.allhex0));
  memset(P.allhex1, 0, sizeof(P.allhex1));
  unsigned short sgrow = 0, sgcol = 0;
  for (int row = 0; row < 3; row++)
    for (int col = 0; col < 3; col++) {
      const int gint = isg(row, col);
      for (int ng = 0, d = 0; d < 10; d += 2) {
        if (isg(row + orth[d] + 6, col + orth[d + 2] + 6)) ng = 0;
        else ng++;
        if (ng == 4) {
          sgrow = row;
          sgcol = col;
        }
        if (ng == gint + 1)
          for (int c = 0; c < 8; c++) {
            const int v = orth[d] * patt[gint][c * 2] + orth[d + 1] * patt[gint][c * 2 + 1];
            const int h = orth[d + 2] * patt[gint][c * 2] + orth[d + 3] * patt[gint][c * 2 + 1];
            P.allhex0[row][col][c ^ (gint * 2 & d)] = (short)(h + v * width);
            P.allhex1[row][col][c ^ (gint * 2 & d)] = (short)(h + v * XTS);
          }
      }
    }
  P.sgrow = sgrow;
  P.sgcol = sgcol;
  for (int row = 0; row < 3; row++) {
    int greencount = 0;
    for (int col = 0; col < 3; col++) greencount += isg(row, col);
    P.right_shift[row] = (greencount == 2);
  }
  return P;
}

// Whether the reference's row scans of phases (a), (b), (c), (e) and (f)
// reduce to "every site of the class" for this pattern (true for the X-Trans
// layouts and their shifts), so the site-parallel kernels apply.  Checked by
// replaying the scans over every tile-origin residue.
bool xt_sites_ok(const XtParams& P) {
  auto isg = [&](int r, int c) { return P.xt[((r % 3) + 3) % 3][((c % 3) + 3) % 3] & 1; };
  auto fc = [&](int r, int c) { return (int)P.xt[(r + 6) % 6][(c + 6) % 6]; };
  // the plane kernel's site lists hold at most 4 non-green sites per 3x3
  int greens = 0;
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++) greens += isg(r, c);
  if (9 - greens > 4) return false;
  for (int t0 = 0; t0 < 6; t0++)
    for (int l0 = 0; l0 < 6; l0++) {
      const int top = 6 + t0, left = 6 + l0, mrow = top + 30, mcol = left + 30;
      for (int row = top; row < mrow; row++) {
        // (b): visits from the first non-green site
        int ls = left;
        while (ls < mcol && isg(row, ls)) ls++;
        int co = P.right_shift[row % 3] == 1 ? 3 : 1 + (fc(row, ls + 1) & 1);
        int expect = ls;
        for (int col = ls; col < mcol; col += co, co = (co == 3) ? 3 : (co ^ 3)) {
          while (expect < mcol && isg(row, expect)) expect++;
          if (col != expect) return false;
          expect++;
        }
        while (expect < mcol && isg(row, expect)) expect++;
        if (expect < mcol) return false;
        // (e): the written colour is 2 - own colour at every visit
        ls = left;
        while (ls < mcol - 1 && isg(row, ls)) ls++;
        int f = 2 - fc(row, ls);
        if (P.right_shift[row % 3] == 1) {
          for (int col = ls; col < mcol; col += 3, f ^= 2)
            if (isg(row, col) || f != 2 - fc(row, col)) return false;
        } else {
          co = fc(row, ls + 1) == 1 ? 2 : 1;
          for (int col = ls; col < mcol; col += co, co ^= 3, f ^= (co & 2))
            if (isg(row, col) || f != 2 - fc(row, col)) return false;
        }
      }
      // (a): the slot a non-green site reads holds the min/max of the site
      // itself, or of its left neighbour when that is a non-green site of
      // the tile (the second site of a pair); replayed in the scan's write
      // order
      for (int row = top; row < mrow; row++) {
        int src[40];
        for (int j = 0; j < 40; j++) src[j] = -1;
        int ls = left;
        while (ls < mcol && isg(row, ls)) ls++;
        const int co = P.right_shift[row % 3] == 1 ? 3 : 1 + (fc(row, ls + 1) & 1);
        if (co == 3) {
          for (int col = ls; col < mcol; col += 3) src[(col - left) >> 1] = col;
        } else {
          int col = ls;
          if (co == 2) {
            src[(col - left) >> 1] = col;
            col += 2;
          }
          for (; col < mcol - 1; col += 3) src[(col - left) >> 1] = src[(col + 1 - left) >> 1] = col;
          if (col < mcol) src[(col - left) >> 1] = col;
        }
        for (int col = left; col < mcol; col++) {
          if (isg(row, col)) continue;
          const int expect_src = (col > left && !isg(row, col - 1)) ? col - 1 : col;
          if (src[(col - left) >> 1] != expect_src) return false;
        }
      }
      // (c): visits every non-green site from left + 2 with f = own colour
      // and hexagon allhex1[row % 3][col % 3], and reads green sites only
      // (which the step does not write)
      for (int row = top + 2; row < mrow - 2; row++) {
        int ls = left + 2;
        while (ls < mcol - 2 && isg(row, ls)) ls++;
        int co = P.right_shift[row % 3] == 1 ? 3 : 1 + (fc(row, ls + 1) & 1);
        int f = fc(row, ls);
        int expect = ls;
        for (int col = ls; col < mcol - 2;) {
          while (expect < mcol - 2 && isg(row, expect)) expect++;
          if (col != expect || f != fc(row, col)) return false;
          expect++;
          for (int d = 3; d < 6; d++)
            for (int m = -2; m <= 1; m += 3) {
              const int x = m * P.allhex1[row % 3][col % 3][d];
              int v = -7, h = 0;
              for (int vv = -6; vv <= 6; vv++)
                if (x - vv * XTS >= -6 && x - vv * XTS <= 6) v = vv, h = x - vv * XTS;
              if (v < -6 || !isg(row + v, col + h)) return false;
            }
          if (co == 3) {
            col += 3;
            f ^= 2;
          } else {
            col += co;
            co ^= 3;
            f ^= (co & 2);
          }
        }
        while (expect < mcol - 2 && isg(row, expect)) expect++;
        if (expect < mcol - 2) return false;
      }
      // (f): visited columns are those off the solitary-green column class
      int ts_ = top;
      while (ts_ < mrow && !((ts_ - P.sgrow + 6) % 3)) ts_++;
      int lsf = left;
      while (lsf < mcol && !((lsf - P.sgcol + 6) % 3)) lsf++;
      const int cos = 2 - (fc(ts_, lsf + 1) & 1);
      for (int col = lsf, co = cos; col < mcol; col += co, co ^= 3)
        if (!((col - P.sgcol + 6) % 3)) return false;
      int visits = 0, expect_n = 0;
      for (int col = lsf, co = cos; col < mcol; col += co, co ^= 3) visits++;
      for (int col = lsf; col < mcol; col++) expect_n += ((col - P.sgcol + 6) % 3) != 0;
      if (visits != expect_n) return false;
    }
  return true;
}

// Whether a plane may keep the last one's values: every slot that a step of
// pass 0 reads is then native, never written, or written by an earlier step of
// the same plane ((b) greens, (d) solitary greens, (e) non-green sites).  True
// for the X-Trans layouts and their shifts.
bool xt_fresh_once(const XtParams& P) {
  auto fc = [&](int r, int c) { return (int)P.xt[(r + 12) % 6][(c + 12) % 6]; };
  auto isg = [&](int r, int c) { return P.xt[(r + 12) % 3][(c + 12) % 3] & 1; };
  auto sol = [&](int r, int c) { return (r + 12 - P.sgrow) % 3 == 0 && (c + 12 - P.sgcol) % 3 == 0; };
  for (int r = 0; r < 6; r++)
    for (int c = 0; c < 6; c++) {
      if ((fc(r, c) == 1) != (isg(r, c) != 0)) return false;
      if (sol(r, c)) {
        // (d): the colour at distance 1 along the row, the other at 2, and the
        // other way round along the column
        const int h = fc(r, c + 1);
        if (h == 1 || !isg(r, c)) return false;
        for (int s = -1; s <= 1; s += 2)
          if (fc(r, c + s) != h || fc(r, c + 2 * s) != (h ^ 2) || fc(r + s, c) != (h ^ 2) || fc(r + 2 * s, c) != h)
            return false;
      } else if (!isg(r, c)) {
        // (e): its other colour at distance 1 across or along, and 3
        const int f = 2 - fc(r, c);
        const bool off = (r + 12 - P.sgrow) % 3 != 0;
        for (int s = -3; s <= 3; s += 2) {
          const bool down = off == (s == 1 || s == -1);
          const int rr = down ? r + s : r, cc = down ? c : c + s;
          if (fc(rr, cc) != f && !sol(rr, cc)) return false;
        }
      } else {
        // (f): its hexagon holds no site of its own step
        for (int d = 0; d < 8; d++)
          for (int v = -2; v <= 2; v++) {
            const int h = P.allhex1[r % 3][c % 3][d] - v * XTS;
            if (h < -2 || h > 2) continue;
            if (isg(r + v, c + h) && !sol(r + v, c + h)) return false;
          }
      }
    }
  return true;
}

// The plane-resident kernel runs where the replay accepts the pattern,
// unless LRE_XTRANS_ROWSCAN=1 asks for the row-scan kernel (a test hook:
// it keeps the fallback path covered on the X-Trans layouts).
bool xt_use_planes(const XtParams& P) {
  const char* force = std::getenv("LRE_XTRANS_ROWSCAN");
  if (force && force[0] == '1') return false;
  return xt_sites_ok(P);
}

}  // namespace

size_t ws_bytes_xtrans(size_t w, size_t h, int passes, const char* xtrans) {
  if (passes == 1) return 0;
  const size_t planes = (size_t)kXsMaxCtas * kXsSpillBytes + ((w * h * sizeof(float) + 255) / 256) * 256;
  const size_t rowscan = (size_t)kXtMaxCtas * kXtSlabBytes;
  if (xtrans) return (xt_use_planes(make_xt_params(xtrans, (int)w)) ? planes : rowscan) + 4096;
  return std::max(rowscan, planes) + 4096;
}

lre_status launch_xtrans(Context* c, const float* raw, int cstride, float* rgb, size_t w, size_t h, const char* xtrans,
                         float maximum_value, int passes) {
  XtArgs A;
  A.raw = raw;
  A.norm = nullptr;
  A.cstride = cstride;
  A.rgb_out = rgb;
  A.W = (int)w;
  A.H = (int)h;
  A.maximum = maximum_value;
  // hexagon offsets are 16-bit (h + v * width, |v| <= 2), as in the reference
  if (2 * w + 2 > 32767 && passes != 1)
    return fail(c, LRE_ERR_INVALID_ARGUMENT, "demosaic_xtrans_3pass: width above 16382 overflows the hexagon offsets");
  A.P = make_xt_params(xtrans, (int)w);
  A.refill = !xt_fresh_once(A.P);
  if (passes == 1) {
    // border (1 px) first, then the interior (:2681-2760)
    k_xtrans_border<<<grid_for(4 * (w + h), 256, c->sm_count * 2), 256, 0, c->stream>>>(A, 1);
    if (w > 2 && h > 2)
      k_xtrans_1pass<<<grid_for((w - 2) * (h - 2), 256, c->sm_count * 8), 256, 0, c->stream>>>(A);
    count_launch(c, 2);
    return check_launch(c, "demosaic_xtrans_1pass");
  }
  // tile grid of :1968-1969
  int n_top = 0, n_left = 0;
  for (int top = 3; top < (int)h - 19; top += XTS - 16) n_top++;
  for (int left = 3; left < (int)w - 19; left += XTS - 16) n_left++;
  A.n_top = n_top;
  A.n_left = n_left;
  const int tiles = n_top * n_left;
  if (tiles > 0) {
    // Patterns whose scans the replay confirms run the plane-resident kernel:
    // one 1024-thread CTA per SM.  Others run the row-scan kernel, two
    // 512-thread CTAs per SM, each with its whole tile in a global slab.
    const bool sites = xt_use_planes(A.P);
    if (sites) {
      float* norm = reinterpret_cast<float*>(c->ws.take(w * h * sizeof(float)));
      if (!norm) return fail(c, LRE_ERR_OUT_OF_MEMORY, "demosaic_xtrans_3pass: workspace too small");
      k_xt_normalize<<<grid_for(w * h, 256, c->sm_count * 8), 256, 0, c->stream>>>(A, norm);
      count_launch(c);
      A.norm = norm;
    }
    const int nblk = sites ? std::min(std::min(tiles, c->sm_count), kXsMaxCtas)
                           : std::min(std::min(tiles, c->sm_count * kXtCtasPerSm), kXtMaxCtas);
    A.scratch = reinterpret_cast<unsigned char*>(c->ws.take((size_t)nblk * (sites ? kXsSpillBytes : kXtSlabBytes)));
    A.tile_counter = reinterpret_cast<int*>(c->ws.take(256));
    if (!A.scratch || !A.tile_counter) return fail(c, LRE_ERR_OUT_OF_MEMORY, "demosaic_xtrans_3pass: workspace too small");
    LRE_CUDA_TRY(c, cudaMemsetAsync(A.tile_counter, 0, sizeof(int), c->stream));
    if (sites) {
      LRE_CUDA_TRY(c, cudaFuncSetAttribute(k_xtrans_3pass_planes, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)kXsSmemBytes));
      k_xtrans_3pass_planes<<<nblk, XS_THREADS, kXsSmemBytes, c->stream>>>(A);
    } else {
      k_xtrans_3pass<<<nblk, XT_THREADS, 0, c->stream>>>(A);
    }
    count_launch(c);
  }
  k_xtrans_border<<<grid_for(16 * (w + h), 256, c->sm_count * 2), 256, 0, c->stream>>>(A, 8);
  count_launch(c);
  return check_launch(c, "demosaic_xtrans_3pass");
}

}  // namespace lre

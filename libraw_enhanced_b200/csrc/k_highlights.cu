// k_highlights.cu -- highlight recovery (the develop pipeline's
// recover_highlights, core/libraw_wrapper.cpp:1095-1383, run for
// highlight_mode > 2 at :1677-1683, and the standalone
// LibRawWrapper::recover_highlights_numpy, :3066-3096).
//
// The reference runs five loops over an interleaved float[3] image:
//   1. per pixel: the optional soft highlight mask, the highlight test
//      (R and B >= threshold) and, for unclipped highlights, the float sums
//      of R/G and B/G in pixel order;
//   2. per highlight pixel: max over channels, G from R and B through the
//      mean ratios, R and B pulled toward G, the white test;
//   3. per white pixel off the 1-px frame: the 8-neighbour mean, all
//      computed before any is written;
//   4. per highlight pixel off the 2-px frame, in pixel order, in place: the
//      LoCA green lift, which reads 3x3 and 5x5 neighbourhoods that earlier
//      pixels of the same loop may have rewritten.
//
// Here:
//   * loop 1 is one thread per pixel; its two float sums are sequential in
//     the reference, so the terms are compacted in pixel order (block counts,
//     one scan, an order-preserving scatter) and one warp adds them in that
//     order, bit for bit;
//   * loops 2 and 3 are one thread per pixel on R/G/B planes;
//   * loop 4 is an in-order sweep (sweep.cuh): a pixel reads rewritten
//     pixels up to two rows up and two columns right, so rows walk three
//     columns apart (skew 3) through a 256-column shared-memory ring.
// Arithmetic is the reference's operation for operation (--fmad=false; the
// 5x5 ratio sums in double).
#include <cfloat>

#include "common.cuh"
#include "lre_internal.h"
#include "stencil.cuh"
#include "sweep.cuh"

namespace lre {

namespace {

constexpr int kHlBlock = 256;

struct HlParams {
  float thr;
  float chroma_lo, chroma_inv;
  float inv_wb[3];
  float mask_inv;
};

// Loop 1 per pixel (:1150-1191): mask, highlight flag, candidate flag.
__global__ void k_hl_pass1(const float* __restrict__ in, size_t n, HlParams P, float* __restrict__ mask,
                           uint8_t* __restrict__ flags, int* __restrict__ block_counts, int* total) {
  const size_t i = (size_t)blockIdx.x * kHlBlock + threadIdx.x;
  int cand = 0;
  if (i < n) {
    const float p0 = in[i * 3], p1 = in[i * 3 + 1], p2 = in[i * 3 + 2];
    if (mask) {
      float t = (p1 - 0.95f) * P.mask_inv;
      if (t < 0.f) t = 0.f; else if (t > 1.f) t = 1.f;
      const float w_g = t * t * (3.f - 2.f * t);
      const float r_n = p0 * P.inv_wb[0], g_n = p1 * P.inv_wb[1], b_n = p2 * P.inv_wb[2];
      const float mx = smax(r_n, smax(g_n, b_n));
      const float mn = smin(r_n, smin(g_n, b_n));
      const float chroma = (mx > 1e-6f) ? (mx - mn) / mx : 0.f;
      float ct = (chroma - P.chroma_lo) * P.chroma_inv;
      if (ct < 0.f) ct = 0.f; else if (ct > 1.f) ct = 1.f;
      const float neutrality = 1.f - ct * ct * (3.f - 2.f * ct);
      mask[i] = w_g * neutrality;
    }
    uint8_t f = 0;
    if (p0 >= P.thr && p2 >= P.thr) {
      f = 1;
      if (p0 < 0.95f && p1 >= P.thr && p1 < 0.95f && p2 < 0.95f) {
        f = 3;
        cand = 1;
      }
    }
    flags[i] = f;
  }
  const int c = __syncthreads_count(cand);
  if (threadIdx.x == 0) {
    block_counts[blockIdx.x] = c;
    if (c) atomicAdd(total, c);
  }
}

// Exclusive scan of the per-block candidate counts (one CTA, eight counts per
// thread and step; the total goes to block_off[nb]).
__global__ void __launch_bounds__(1024) k_hl_scan(const int* __restrict__ counts, int nb, int* __restrict__ off,
                                                   const int* __restrict__ total) {
  if (*total == 0) {  // no terms: the usual case, as few highlights lie below 0.95
    if (threadIdx.x == 0) off[nb] = 0;
    return;
  }
  __shared__ int warp_sums[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nb; base += 8192) {
    const int i0 = base + 8 * threadIdx.x;
    int v[8], t = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      v[k] = i0 + k < nb ? counts[i0 + k] : 0;
      t += v[k];
    }
    int x = t;
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, d);
      if ((threadIdx.x & 31) >= d) x += y;
    }
    if ((threadIdx.x & 31) == 31) warp_sums[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
      int w = warp_sums[threadIdx.x];
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, d);
        if (threadIdx.x >= d) w += y;
      }
      warp_sums[threadIdx.x] = w;
    }
    __syncthreads();
    const int wp = (threadIdx.x >> 5) ? warp_sums[(threadIdx.x >> 5) - 1] : 0;
    int o = carry + wp + x - t;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      if (i0 + k < nb) off[i0 + k] = o;
      o += v[k];
    }
    __syncthreads();
    if (threadIdx.x == 1023) carry += wp + x;
    __syncthreads();
  }
  if (threadIdx.x == 0) off[nb] = carry;
}

// The candidates' R/G and B/G terms, scattered in pixel order.
__global__ void k_hl_compact(const float* __restrict__ in, size_t n, const uint8_t* __restrict__ flags,
                             const int* __restrict__ block_off, float* __restrict__ t_rg,
                             float* __restrict__ t_bg, const int* __restrict__ total, int nb) {
  __shared__ int warp_base[kHlBlock / 32];
  if (*total == 0) return;
  for (int blk = blockIdx.x; blk < nb; blk += gridDim.x) {
    if (block_off[blk + 1] == block_off[blk]) continue;  // none here
    const size_t i = (size_t)blk * kHlBlock + threadIdx.x;
    const bool cand = i < n && flags[i] == 3;
    const unsigned b = __ballot_sync(0xffffffffu, cand);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) warp_base[warp] = __popc(b);
    __syncthreads();
    if (threadIdx.x == 0) {
      int s = 0;
      for (int k = 0; k < kHlBlock / 32; k++) {
        const int c = warp_base[k];
        warp_base[k] = s;
        s += c;
      }
    }
    __syncthreads();
    if (cand) {
      const int pos = block_off[blk] + warp_base[warp] + __popc(b & ((1u << lane) - 1));
      const float p0 = in[i * 3], p1 = in[i * 3 + 1], p2 = in[i * 3 + 2];
      t_rg[pos] = p0 / p1;
      t_bg[pos] = p2 / p1;
    }
    __syncthreads();
  }
}

// grf / gbf / count as the reference accumulates them (:1182-1196): float
// sums in pixel order.  Lanes stage 32 terms at a time in shared memory;
// lane 0 adds them in order.  scal[0] = grf, scal[1] = gbf.
__global__ void k_hl_ratio_sums(const float* __restrict__ t_rg, const float* __restrict__ t_bg,
                                const int* __restrict__ total, float* __restrict__ scal) {
  __shared__ float a[32], b[32];
  const int k = *total;
  float grf = 0.f, gbf = 0.f, count = 0.f;
  for (int base = 0; base < k; base += 32) {
    const int m = min(32, k - base);
    if ((int)threadIdx.x < m) {
      a[threadIdx.x] = t_rg[base + threadIdx.x];
      b[threadIdx.x] = t_bg[base + threadIdx.x];
    }
    __syncwarp();
    if (threadIdx.x == 0)
      for (int j = 0; j < m; j++) {
        grf += a[j];
        gbf += b[j];
        count += 1.f;
      }
    __syncwarp();
  }
  if (threadIdx.x == 0) {
    if (count > 0.f) {
      grf /= count;
      gbf /= count;
    } else {
      grf = 1.f;
      gbf = 1.f;
    }
    scal[0] = grf;
    scal[1] = gbf;
  }
}

// Loop 2 (:1207-1251) on every highlight pixel, writing planes (non-highlight
// pixels copy through); flag bit 2 marks white pixels.  scal[2] = max_val.
__global__ void k_hl_pass2(const float* __restrict__ in, size_t n, HlParams P, uint8_t* __restrict__ flags,
                           float* __restrict__ R, float* __restrict__ G, float* __restrict__ B,
                           float* __restrict__ scal) {
  const float grf = scal[0], gbf = scal[1];
  float local_max = 0.f;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float p0 = in[i * 3], p1 = in[i * 3 + 1], p2 = in[i * 3 + 2];
    uint8_t f = flags[i];
    if (f & 1) {
      local_max = smax(local_max, smax(p0, smax(p1, p2)));
      p1 = (p0 / grf + p2 / gbf) * 0.5f;
      const float sp = (p0 < p2) ? p0 : p2;
      const float sl = (smin(sp, 1.f) - P.thr) / (P.thr);
      p0 = p0 * (1.f - sl) + (p1 * grf) * sl;
      p2 = p2 * (1.f - sl) + (p1 * gbf) * sl;
      p1 = (p0 / grf + p2 / gbf) * 0.5f;
      if (p1 >= 0.95f) flags[i] = f | 4;
    }
    R[i] = p0;
    G[i] = p1;
    B[i] = p2;
  }
  block_max_atomic(local_max, scal + 2);
}

// The neighbour terms of a pixel: its largest channel, and its G / RB ratio
// where the pixel takes part in its neighbours' ratio means, -1 where not.
__device__ __forceinline__ float loca_ratio(float n0, float n1, float n2, float nl, float thr) {
  const float nrb = 0.5f * (n0 + n2);
  if (nl < thr * 0.75f || nrb <= 1e-6f) return -1.f;
  const float ratio = n1 / nrb;
  return (ratio < 0.70f || ratio > 1.35f) ? -1.f : ratio;
}

// Loop 3 (:1259-1296): white pixels off the 1-px frame take the mean of their
// 8 neighbours, all read before any is written (out of place).
__global__ void k_hl_white(const float* __restrict__ R, const float* __restrict__ G, const float* __restrict__ B,
                           const uint8_t* __restrict__ flags, float* __restrict__ R2, float* __restrict__ G2,
                           float* __restrict__ B2, float* __restrict__ cand, float* __restrict__ nl,
                           float* __restrict__ rt, float* out, int W, int H, float thr) {
  const size_t n = (size_t)W * H;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int y = (int)(i / W), x = (int)(i % W);
    const float* src[3] = {R, G, B};
    const bool white = (flags[i] & 4) && x > 0 && x < W - 1 && y > 0 && y < H - 1;
    float v[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float* s = src[c];
      v[c] = white ? (s[i - W - 1] + s[i - W] + s[i - W + 1] + s[i - 1] + s[i + 1] + s[i + W - 1] + s[i + W] +
                           s[i + W + 1]) *
                              (1.f / 8.f)
                   : s[i];
    }
    // Loop 4 changes a highlight pixel only from its own value, and only when
    // that value passes these two tests (:1307-1329), so they are decided
    // here, once, for all pixels.
    const float l = smax(v[0], smax(v[1], v[2]));
    const float rb = 0.5f * (v[0] + v[2]);
    nl[i] = l;
    rt[i] = loca_ratio(v[0], v[1], v[2], l, thr);
    out[i * 3] = v[0];
    out[i * 3 + 1] = v[1];
    out[i * 3 + 2] = v[2];
    const bool changes = (flags[i] & 1) && !(l < thr * 0.90f) && !(rb <= v[1] * 1.04f);
    cand[i] = changes ? 1.f : 0.f;
    if (changes) {  // loop 4 reads a candidate's own value while its result may already be in `out`
      R2[i] = v[0];
      G2[i] = v[1];
      B2[i] = v[2];
    }
  }
}

// A candidate's new value from its own value and its neighbours' terms, or
// false where it keeps its value.  nl(dy, dx) and ratio(dy, dx) read the terms.
template <class NL, class RT>
__device__ __forceinline__ bool loca_lift(NL nl, RT ratio, float thr, float max_val, float& p0, float& p1, float& p2) {
  float local_max = 0.0f, local_min = FLT_MAX;
#pragma unroll
  for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
    for (int dx = -1; dx <= 1; ++dx) {
      const float n = nl(dy, dx);
      local_max = smax(local_max, n);
      local_min = smin(local_min, n);
    }
  if ((local_max - local_min) < 0.015f) return false;
  const float l = smax(p0, smax(p1, p2));
  const float rb = 0.5f * (p0 + p2);
  // Unrolled, so each weight 1.0 / (1 + |dx| + |dy|) is the same correctly
  // rounded double, folded at compile time.
  double ratio_sum = 0.0, ratio_w = 0.0;
#pragma unroll
  for (int dy = -2; dy <= 2; ++dy)
#pragma unroll
    for (int dx = -2; dx <= 2; ++dx) {
      // selected, not branched to: adding 0.0 changes neither sum
      const float q = ratio(dy, dx);
      const bool in = q != -1.f;
      const double w = 1.0 / (double)(1 + abs(dx) + abs(dy));
      ratio_sum += in ? (double)q * w : 0.0;
      ratio_w += in ? w : 0.0;
    }
  const float local_ratio = (float)(ratio_w > 0.0 ? ratio_sum / ratio_w : 1.0);
  const float desired_g = rb * sclamp(local_ratio, 0.95f, 1.08f);
  const float g_missing = desired_g - p1;
  if (g_missing <= 0.0f) return false;
  const float sat_w = sclamp((l - thr) / smax(1e-6f, smax(1.0f, max_val) - thr), 0.0f, 1.0f);
  const float edge_w = sclamp((local_max - local_min) / 0.08f, 0.0f, 1.0f);
  const float alpha = sclamp(0.30f + 0.55f * sat_w * edge_w, 0.0f, 0.90f);
  const float g_boost = alpha * smin(g_missing, (rb - p1) * 0.90f);
  p1 += g_boost;
  const float rb_residual = smax(0.0f, 0.5f * (p0 + p2) - p1);
  if (rb_residual > 0.0f) {
    const float trim = smin(rb_residual * alpha * 0.45f, 0.5f * (p0 + p2) * 0.12f);
    p0 = smax(0.0f, p0 - trim);
    p2 = smax(0.0f, p2 - trim);
  }
  p1 = smax(0.0f, p1);
  return true;
}

// Loop 4 (:1301-1377), in pixel order: state R, G, B; input the candidate
// flag (k_hl_white).  aux[0] = threshold, aux[1] = max_val.
struct OpLoca {
  static constexpr int NS = 3, NP = 4, HALO = 2, SKEW = 3, PAIR = 1, NCH = 1, LAG = 0, RING = 256;
  __device__ static bool site(int, int, const Geo&) { return true; }
  template <class T>
  __device__ static void cell(const T& t, int, const Geo& g) {
    if (t.input(3) == 0.f) return;
    const float thr = g.aux[0];
    float p0 = t.get(0, 0, 0), p1 = t.get(1, 0, 0), p2 = t.get(2, 0, 0);
    auto nl = [&](int dy, int dx) { return smax(t.get(0, dy, dx), smax(t.get(1, dy, dx), t.get(2, dy, dx))); };
    auto rt = [&](int dy, int dx) {
      return loca_ratio(t.get(0, dy, dx), t.get(1, dy, dx), t.get(2, dy, dx), nl(dy, dx), thr);
    };
    if (!loca_lift(nl, rt, thr, g.aux[1], p0, p1, p2)) return;
    t.set(0, p0);
    t.set(1, p1);
    t.set(2, p2);
  }
};

// The same loop for blocks.  A pixel's neighbours see only two terms of it,
// so those are the state (two planes instead of three, and no division per
// neighbour: each pixel's ratio is formed once).  The pixel's own RGB is read
// from the planes where it is a candidate, and its result goes straight into
// the interleaved image.
struct OpLocaBlk {
  static constexpr int NS = 2, NP = 3, HALO = 2, SKEW = 3, PAIR = 1, NCH = 1, LAG = 0, BLK_WARPS = 4, BLK_PER_SM = 3;
  static constexpr int BLK_SKEW = 3, BLK_PAIR = 1, BLK_ROWS = 32, BLK_COLS = 96, BLK_FROM = 0;
  static constexpr bool UNROLL = false, STEP2 = false, IDLE0 = true;
  __device__ static bool site(int, int, const Geo&) { return true; }
  template <class T>
  __device__ static void cell(const T& t, int, const Geo& g) {
    if (t.input(2) == 0.f) return;
    const float thr = g.auxv[0];
    float p0 = __ldg(g.ex[0] + t.px), p1 = __ldg(g.ex[1] + t.px), p2 = __ldg(g.ex[2] + t.px);
    if (loca_lift([&](int dy, int dx) { return t.get(0, dy, dx); }, [&](int dy, int dx) { return t.get(1, dy, dx); },
                  thr, g.auxv[1], p0, p1, p2)) {
      const float n = smax(p0, smax(p1, p2));
      t.set(0, n);
      t.set(1, loca_ratio(p0, p1, p2, n, thr));
    }
    if (t.own) {  // also where it keeps its value: a repair may undo a first run's change
      float* o = g.ex_out + t.px * 3;
      o[0] = p0;
      o[1] = p1;
      o[2] = p2;
    }
  }
};

// Loop 4's scalars for the sweep: aux[0] = threshold, aux[1] = max_val.
__global__ void k_hl_aux(float* scal, float thr) {
  scal[3] = thr;
  scal[4] = scal[2];
}

// The planes of the in-order sweep at the pixels that loop 4 leaves alone
// (`out` holds those; the candidates' are there), where it has to run.
__global__ void k_hl_planes(const float* __restrict__ out, const float* __restrict__ cand, float* __restrict__ R,
                            float* __restrict__ G, float* __restrict__ B, size_t n, const int* __restrict__ run_if) {
  if (run_if && *run_if == 0) return;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    if (cand[i] != 0.f) continue;
    R[i] = out[i * 3];
    G[i] = out[i * 3 + 1];
    B[i] = out[i * 3 + 2];
  }
}

// The in-order sweep's planes into the result, where it had to run.
__global__ void k_hl_interleave(const float* __restrict__ R, const float* __restrict__ G,
                                const float* __restrict__ B, float* __restrict__ out, size_t n,
                                const int* __restrict__ run_if) {
  if (run_if && *run_if == 0) return;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    out[i * 3] = R[i];
    out[i * 3 + 1] = G[i];
    out[i * 3 + 2] = B[i];
  }
}

size_t plane(size_t n) { return (n * sizeof(float) + 255) & ~size_t(255); }

}  // namespace

size_t ws_bytes_highlights(size_t w, size_t h) {
  const size_t n = w * h;
  const size_t nb = (n + kHlBlock - 1) / kHlBlock;
  const size_t bands = (h + 31) / 32 + 1;
  return 9 * plane(n) + ((n + 255) & ~size_t(255)) + 2 * ((nb + 1) * sizeof(int) + 256) + 256 +
         (kSyncInts + bands) * sizeof(int) + 1024 + blk_ws_bytes<OpLocaBlk>(w, h);
}

lre_status launch_recover_highlights(Context* c, const float* in, float* out, size_t w, size_t h,
                                     float saturation_threshold, float* mask_out, const float* wb_rgb,
                                     float* d_max_val_out, int* d_err) {
  const size_t n = w * h;
  const size_t nb = (n + kHlBlock - 1) / kHlBlock;
  if (nb > (size_t)INT_MAX - 1) return fail(c, LRE_ERR_INVALID_ARGUMENT, "recover_highlights: image too large");
  float* R = reinterpret_cast<float*>(c->ws.take(plane(n)));
  float* G = reinterpret_cast<float*>(c->ws.take(plane(n)));
  float* B = reinterpret_cast<float*>(c->ws.take(plane(n)));
  float* R2 = reinterpret_cast<float*>(c->ws.take(plane(n)));
  float* G2 = reinterpret_cast<float*>(c->ws.take(plane(n)));
  float* B2 = reinterpret_cast<float*>(c->ws.take(plane(n)));
  float* HL = reinterpret_cast<float*>(c->ws.take(plane(n)));
  float* NL = reinterpret_cast<float*>(c->ws.take(plane(n)));
  float* RT = reinterpret_cast<float*>(c->ws.take(plane(n)));
  uint8_t* flags = reinterpret_cast<uint8_t*>(c->ws.take((n + 255) & ~size_t(255)));
  int* counts = reinterpret_cast<int*>(c->ws.take((nb + 1) * sizeof(int) + 256));
  int* offs = reinterpret_cast<int*>(c->ws.take((nb + 1) * sizeof(int) + 256));
  float* scal = reinterpret_cast<float*>(c->ws.take(256));
  const int nb_max = (int)((h + 31) / 32 + 1);
  int* sync = reinterpret_cast<int*>(c->ws.take((kSyncInts + nb_max) * sizeof(int)));
  const size_t blk_len = blk_ws_bytes<OpLocaBlk>(w, h);
  void* blk_ws = c->ws.take(blk_len);
  if (!R || !G || !B || !R2 || !G2 || !B2 || !HL || !NL || !RT || !flags || !counts || !offs || !scal || !sync || !blk_ws)
    return fail(c, LRE_ERR_CUDA, "recover_highlights: workspace not reserved");

  HlParams P{};
  P.thr = saturation_threshold;
  P.mask_inv = 1.f / std::max(1e-6f, 1.00f - 0.95f);
  P.chroma_lo = wb_rgb ? 0.30f : 0.50f;
  const float chroma_hi = wb_rgb ? 0.60f : 0.70f;
  P.chroma_inv = 1.f / std::max(1e-6f, chroma_hi - P.chroma_lo);
  for (int k = 0; k < 3; k++) P.inv_wb[k] = wb_rgb ? 1.f / std::max(1e-6f, wb_rgb[k]) : 1.f;

  cudaStream_t s = c->stream;
  auto ck = [&](const char* what) {
    count_launch(c);
    return check_launch(c, what);
  };
  LRE_CUDA_TRY(c, cudaMemsetAsync(scal, 0, 256, s));
  int* total = reinterpret_cast<int*>(scal + 8);  // terms of the ratio means
  k_hl_pass1<<<(unsigned)nb, kHlBlock, 0, s>>>(in, n, P, mask_out, flags, counts, total);
  LRE_TRY(ck("recover_highlights"));
  k_hl_scan<<<1, 1024, 0, s>>>(counts, (int)nb, offs, total);
  LRE_TRY(ck("recover_highlights"));
  // the compacted terms live in R2/G2, which are free until loop 3
  k_hl_compact<<<(unsigned)std::min<size_t>(nb, (size_t)c->sm_count * 8), kHlBlock, 0, s>>>(in, n, flags, offs, R2, G2,
                                                                                       total, (int)nb);
  LRE_TRY(ck("recover_highlights"));
  k_hl_ratio_sums<<<1, 32, 0, s>>>(R2, G2, offs + nb, scal);
  LRE_TRY(ck("recover_highlights"));
  const unsigned g1 = grid_for(n, 256, c->sm_count * 8);
  k_hl_pass2<<<g1, 256, 0, s>>>(in, n, P, flags, R, G, B, scal);
  LRE_TRY(ck("recover_highlights"));
  k_hl_white<<<g1, 256, 0, s>>>(R, G, B, flags, R2, G2, B2, HL, NL, RT, out, (int)w, (int)h, P.thr);
  LRE_TRY(ck("recover_highlights"));
  // loop 4 reads the threshold and max_val from the device
  k_hl_aux<<<1, 1, 0, s>>>(scal, P.thr);
  LRE_TRY(ck("recover_highlights"));
  int* err = d_err ? d_err : sync + 1;
  SweepArgs sa{};
  sa.g = Geo{(int)w, (int)h, 0u, 1.0f, scal + 3};
  sa.err = err;
  sa.plane[0] = R2;
  sa.plane[1] = G2;
  sa.plane[2] = B2;
  sa.plane[3] = HL;
  sa.r_lo = 2;
  sa.r_hi = (int)h - 3;
  sa.c_lo = 2;
  sa.c_hi = (int)w - 3;
  if (!d_err) LRE_CUDA_TRY(c, cudaMemsetAsync(err, 0, sizeof(int), s));
  BlkArgs b{};
  b.g = sa.g;
  b.g.ex[0] = R2;
  b.g.ex[1] = G2;
  b.g.ex[2] = B2;
  b.g.ex_out = out;
  b.in[0] = NL;
  b.in[1] = RT;
  b.in[2] = HL;
  b.out[0] = R;  // dead since loop 3
  b.out[1] = G;
  b.r_lo = sa.r_lo;
  b.r_hi = sa.r_hi;
  b.c_lo = sa.c_lo;
  b.c_hi = sa.c_hi;
  if (sa.r_hi < sa.r_lo || sa.c_hi < sa.c_lo) {  // no pixel is off the 2-px frame
    if (d_max_val_out)
      LRE_CUDA_TRY(c, cudaMemcpyAsync(d_max_val_out, scal + 2, sizeof(float), cudaMemcpyDeviceToDevice, s));
    if (!d_err) LRE_CUDA_TRY(c, cudaStreamSynchronize(s));
    return LRE_OK;
  }
  if (!sweeps_in_order<OpLocaBlk>(c, (int)w, (int)h))
    LRE_TRY(blk_sweep<OpLocaBlk>(c, b, blk_ws, blk_len, &sa.run_if, "recover_highlights_loca"));
  k_hl_planes<<<g1, 256, 0, s>>>(out, HL, R2, G2, B2, n, sa.run_if);
  LRE_TRY(ck("recover_highlights"));
  LRE_TRY(sweep_in_order<OpLoca>(c, sa, sync, nb_max, "recover_highlights_loca"));
  k_hl_interleave<<<g1, 256, 0, s>>>(R2, G2, B2, out, n, sa.run_if);
  LRE_TRY(ck("recover_highlights"));
  if (d_max_val_out) LRE_CUDA_TRY(c, cudaMemcpyAsync(d_max_val_out, scal + 2, sizeof(float), cudaMemcpyDeviceToDevice, s));
  if (d_err) return LRE_OK;  // the caller reads the flag after its own synchronisation
  int e = 0;
  LRE_CUDA_TRY(c, cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, s));
  LRE_CUDA_TRY(c, cudaStreamSynchronize(s));
  if (e) return fail(c, LRE_ERR_TIMEOUT, "recover_highlights: a sweep band timed out waiting for the band above");
  return LRE_OK;
}

}  // namespace lre

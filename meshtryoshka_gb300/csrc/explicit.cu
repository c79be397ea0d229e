// Explicit render mode for sm_103a: per-shell first-hit rasterization,
// barycentric interpolation (forward / backward) and the per-pixel shell
// compositing loop (forward / backward).
//
// Follows triangle_rasterization/intersect.slang:86-182,
// interpolate.slang:19-76 and composite.slang:60-218. The hit test is the
// same fixed-order barycentric solve as the fused kernel (bary.cuh).
//
// composite backward has the same two gradient-routing modes as the fused
// kernel: the reference's (the outer sample's signed-distance gradient goes
// to slot shell_index - 1 and the last one to slot num_shells - 1,
// composite.slang:197,212) or the exact adjoint (the previous and last *hit*
// shells).

#include "bary.cuh"
#include "mt_common.cuh"

namespace mt {
namespace {

// ---------------------------------------------------------------------------
// First hit of every pixel in its shell's list (intersect.slang:86-182). A
// list belongs to a (camera, shell, tile); a CTA has one thread per pixel of a
// tile and takes every gridDim-th list, reading the ranges of 32 of them at a
// time: most tiles of a scene are empty, and with a CTA to each list the
// launch was mostly CTAs that waited for one range. A list goes by in chunks
// of a triangle to each thread.
//
// A thread tests its own triangle at the pixel centres inside the triangle's
// accept box (bary.cuh: outside it hit_test's fast reject fires), and a
// pixel's first hit is the least list position that was accepted there
// (atomicMin in shared memory). A fine mesh's triangles reach one to nine
// pixels of a tile, where every pixel testing every triangle of its list, in
// order, up to its first hit, made some hundred tests for each of them.
// Triangles whose box covers more than kOwnPixels centres of the tile (and
// those without a finite one) are left to the pixels, which take them in list
// order and stop at the first. 4 x 800^2, 8 shells of a 256^3 mesh, 16x16
// tiles: 711 us with the pixels testing everything, now 275 us.
// ---------------------------------------------------------------------------
constexpr int kOwnPixels = 32;

struct ExplicitFace {
  TriGeom g;
  int32_t face;
};

// Shared memory: a chunk's triangles, each pixel's best list position in the
// chunk, and a bit per triangle that is left to the pixels.
__host__ __device__ constexpr size_t intersect_smem(int bs) {
  return (size_t)bs * (sizeof(ExplicitFace) + sizeof(int)) + (size_t)((bs + 31) / 32) * sizeof(uint32_t);
}

template <auto kValue>
struct Constant {
  static constexpr auto value = kValue;
};

constexpr int kRanges = 32;  // list ranges read at a time

// kThreads: the most threads of a launch (256 leaves four CTAs to an SM).
template <int kThreads>
__global__ void __launch_bounds__(kThreads, kThreads <= 256 ? 4 : 1)
    intersect_kernel(const float* __restrict__ xy, int64_t V, const int32_t* __restrict__ faces,
                                 const int32_t* __restrict__ tri, const int64_t* __restrict__ bounds, int64_t lists,
                                 int S, int rows, int cols, int tile_h, int tile_w, int H, int W,
                                 float* __restrict__ out_uv, int32_t* __restrict__ out_index) {
  extern __shared__ float4 smem_f4[];
  const int bs = blockDim.x;
  ExplicitFace* sf = reinterpret_cast<ExplicitFace*>(smem_f4);
  int* best = reinterpret_cast<int*>(sf + bs);
  uint32_t* left_bits = reinterpret_cast<uint32_t*>(best + bs);
  __shared__ int64_t range[kRanges][2];
  const int tid = threadIdx.x;
  const int lx = tid % tile_w, ly = tid / tile_w;
  // The last warp of a tile may be partial.
  const int rest = bs - (tid & ~31);
  const uint32_t warp_mask = rest >= 32 ? 0xffffffffu : (1u << rest) - 1u;
  const int64_t T = (int64_t)rows * cols;
  constexpr int kNone = 0x7fffffff;
  int turn = 0;
  for (int64_t list = blockIdx.x; list < lists; list += gridDim.x, ++turn) {
    if (turn % kRanges == 0) {
      __syncthreads();
      for (int k = tid; k < kRanges; k += bs) {
        const int64_t ahead = list + k * (int64_t)gridDim.x;
        range[k][0] = ahead < lists ? bounds[2 * ahead] : 0;
        range[k][1] = ahead < lists ? bounds[2 * ahead + 1] : 0;
      }
      __syncthreads();
    }
    const int64_t start = range[turn % kRanges][0], end = range[turn % kRanges][1];
    const int64_t batch = list / T;  // camera * S + shell
    const int tile = (int)(list - batch * T);
    const int tx = tile % cols * tile_w, ty = tile / cols * tile_h;
    const int px = tx + lx, py = ty + ly;
    const float fx = (float)px + 0.5f, fy = (float)py + 0.5f;
    const int64_t o = (batch * H + py) * W + px;
    bool active = px < W && py < H;
    if (start < end) {
      const float2* xyc = reinterpret_cast<const float2*>(xy) + batch / S * V;
      const float bx = (float)tx + 0.5f, by = (float)ty + 0.5f;
      best[tid] = active ? kNone : -1;  // -1: nothing is below it
      for (int64_t chunk = start; chunk < end; chunk += bs) {
        if (__syncthreads_count(active) == 0) break;
        const int n = (int)min((int64_t)bs, end - chunk);
        bool left = false;
        if (tid < n) {
          const int32_t f = tri[chunk + tid];
          const float2 pa = xyc[faces[3 * (int64_t)f]], pb = xyc[faces[3 * (int64_t)f + 1]],
                       pc = xyc[faces[3 * (int64_t)f + 2]];
          ExplicitFace e;
          setup_geometry(pa.x, pa.y, pb.x, pb.y, pc.x, pc.y, e.g);
          e.g.shell = 0;
          e.face = f;
          sf[tid] = e;
          // Columns and rows of the tile inside the box: ceil / floor of
          // numbers clamped to just outside the tile.
          const CullBox box = cull_box(e.g, pa.x, pa.y, pb.x, pb.y, pc.x, pc.y);
          const int c0 = max((int)ceilf(fmaxf(box.x0 - bx, -1.0f)), 0);
          const int c1 = min((int)floorf(fminf(box.x1 - bx, (float)tile_w)), tile_w - 1);
          const int r0 = max((int)ceilf(fmaxf(box.y0 - by, -1.0f)), 0);
          const int r1 = min((int)floorf(fminf(box.y1 - by, (float)tile_h)), tile_h - 1);
          const int count = c1 >= c0 && r1 >= r0 ? (c1 - c0 + 1) * (r1 - r0 + 1) : 0;
          left = count > kOwnPixels;
          if (!left) {
            int c = c0, r = r0;
            for (int k = 0; k < count; ++k) {
              const int p = r * tile_w + c;
              float u, v, w;
              if (best[p] > tid && hit_test(e.g, bx + (float)c, by + (float)r, u, v, w)) atomicMin(&best[p], tid);
              if (++c > c1) c = c0, ++r;
            }
          }
        }
        const uint32_t leaving = __ballot_sync(warp_mask, left);
        if ((tid & 31) == 0) left_bits[tid >> 5] = leaving;
        __syncthreads();
        if (active) {
          int first = best[tid];
          for (int word = 0; word < (n + 31) >> 5 && 32 * word < first; ++word) {
            for (uint32_t m = left_bits[word]; m; m &= m - 1) {
              const int i = 32 * word + __ffs(m) - 1;
              if (i >= first) break;
              float u, v, w;
              if (hit_test(sf[i].g, fx, fy, u, v, w)) first = i;  // later ones are past it
            }
          }
          if (first != kNone) {
            float u, v, w;
            hit_test(sf[first].g, fx, fy, u, v, w);
            out_uv[2 * o] = u;
            out_uv[2 * o + 1] = v;
            out_index[o] = sf[first].face;
            active = false;
            best[tid] = -1;
          }
        }
      }
      __syncthreads();  // the next list's chunks overwrite the shared ones
    }
    if (active) {
      out_uv[2 * o] = 0.f;
      out_uv[2 * o + 1] = 0.f;
      out_index[o] = -1;
    }
  }
}

// interpolate.slang:22-76. (u, v, w = 1 - u - v) weights of the hit face.
__global__ void interpolate_forward_kernel(const float* __restrict__ uv, const int32_t* __restrict__ index,
                                           const int32_t* __restrict__ faces, const float* __restrict__ sdf,
                                           const float* __restrict__ colors, int64_t V, int S, int64_t BS,
                                           int64_t HW, float* __restrict__ out_sdf, float* __restrict__ out_colors) {
  const int64_t total = BS * HW;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t f = index[i];
    if (f < 0) {
      out_colors[3 * i] = 0.f;
      out_colors[3 * i + 1] = 0.f;
      out_colors[3 * i + 2] = 0.f;
      out_sdf[i] = 0.f;
      continue;
    }
    const int64_t b = (i / HW) / S;
    const float u = uv[2 * i], v = uv[2 * i + 1];
    const float w = __fsub_rn(__fsub_rn(1.0f, u), v);
    const int32_t ia = faces[3 * (int64_t)f], ib = faces[3 * (int64_t)f + 1], ic = faces[3 * (int64_t)f + 2];
    const float* col = colors + b * V * 3;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      out_colors[3 * i + c] = interp(u, v, w, col[3 * (int64_t)ia + c], col[3 * (int64_t)ib + c],
                                     col[3 * (int64_t)ic + c]);
    out_sdf[i] = interp(u, v, w, sdf[ia], sdf[ib], sdf[ic]);
  }
}

__global__ void interpolate_backward_kernel(const float* __restrict__ uv, const int32_t* __restrict__ index,
                                            const int32_t* __restrict__ faces, int64_t V, int S, int64_t BS,
                                            int64_t HW, const float* __restrict__ grad_sdf_out,
                                            const float* __restrict__ grad_colors_out,
                                            float* __restrict__ grad_sdf, float* __restrict__ grad_colors) {
  const int64_t total = BS * HW;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t f = index[i];
    if (f < 0) continue;
    const float gs = grad_sdf_out ? grad_sdf_out[i] : 0.f;
    const float g0 = grad_colors_out ? grad_colors_out[3 * i] : 0.f;
    const float g1 = grad_colors_out ? grad_colors_out[3 * i + 1] : 0.f;
    const float g2 = grad_colors_out ? grad_colors_out[3 * i + 2] : 0.f;
    if (gs == 0.f && g0 == 0.f && g1 == 0.f && g2 == 0.f) continue;
    const int64_t b = (i / HW) / S;
    const float u = uv[2 * i], v = uv[2 * i + 1];
    const float w = __fsub_rn(__fsub_rn(1.0f, u), v);
    const int32_t id[3] = {faces[3 * (int64_t)f], faces[3 * (int64_t)f + 1], faces[3 * (int64_t)f + 2]};
    const float wt[3] = {u, v, w};
    float* gc = grad_colors + b * V * 3;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (gs != 0.f) atomicAdd(grad_sdf + id[k], wt[k] * gs);
      atomicAdd(gc + 3 * (int64_t)id[k], wt[k] * g0);
      atomicAdd(gc + 3 * (int64_t)id[k] + 1, wt[k] * g1);
      atomicAdd(gc + 3 * (int64_t)id[k] + 2, wt[k] * g2);
    }
  }
}

// composite.slang:60-120: front-to-back over the masked shells of a pixel.
__global__ void shell_composite_forward_kernel(const float* __restrict__ sdf, const float* __restrict__ colors,
                                               const uint8_t* __restrict__ mask, int64_t P, int S,
                                               const float* __restrict__ sharpness, float* __restrict__ out_colors,
                                               float* __restrict__ out_T) {
  const float s = *sharpness;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < P; p += (int64_t)gridDim.x * blockDim.x) {
    float acc[3] = {0.f, 0.f, 0.f};
    float T = 1.0f;
    float e;
    float outer_cdf = sdf_to_cdf(1e10f, s, e);
    for (int l = 0; l < S; ++l) {
      if (!mask[p * S + l]) continue;
      const float inner = sdf[p * S + l];
      const float inner_cdf = sdf_to_cdf(inner, s, e);
      const float alpha = clamp01(alpha_raw(outer_cdf, inner_cdf));
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c] = over(acc[c], colors[(p * S + l) * 3 + c], T, alpha);
      T = __fmul_rn(T, __fsub_rn(1.0f, alpha));
      outer_cdf = inner_cdf;
    }
    out_colors[3 * p] = acc[0];
    out_colors[3 * p + 1] = acc[1];
    out_colors[3 * p + 2] = acc[2];
    out_T[p] = T;
  }
}

// Adds the CTA's sum of x to *out (one atomic).
__device__ __forceinline__ void block_sum_to(float x, float* __restrict__ out) {
  __shared__ float s_red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nw = (blockDim.x + 31) >> 5;
    float y = threadIdx.x < nw ? s_red[threadIdx.x] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    if (threadIdx.x == 0 && y != 0.f) atomicAdd(out, y);
  }
}

// composite.slang:122-218 (suffix trick, per-pixel sequential shells).
__global__ void shell_composite_backward_kernel(const float* __restrict__ sdf, const float* __restrict__ colors,
                                                const uint8_t* __restrict__ mask, int64_t P, int S,
                                                const float* __restrict__ sharpness,
                                                const float* __restrict__ out_colors, const float* __restrict__ out_T,
                                                const float* __restrict__ grad_colors_out,
                                                const float* __restrict__ grad_T_out, float* __restrict__ grad_sdf,
                                                float* __restrict__ grad_colors, float* __restrict__ grad_sharpness,
                                                int exact) {
  const float s = *sharpness;
  float d_sharp_total = 0.f;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < P; p += (int64_t)gridDim.x * blockDim.x) {
    const float final_rgb[3] = {out_colors[3 * p], out_colors[3 * p + 1], out_colors[3 * p + 2]};
    const float final_T = out_T[p];
    const float dL[3] = {grad_colors_out ? grad_colors_out[3 * p] : 0.f,
                         grad_colors_out ? grad_colors_out[3 * p + 1] : 0.f,
                         grad_colors_out ? grad_colors_out[3 * p + 2] : 0.f};
    const float dLT = grad_T_out ? grad_T_out[p] : 0.f;
    float acc[3] = {0.f, 0.f, 0.f};
    float T = 1.0f;
    float e_out;
    float outer_cdf = sdf_to_cdf(1e10f, s, e_out);
    float outer_sdf = 1e10f;
    bool first = true;
    int prev_shell = -1;
    float d_partial = 0.f;
    for (int l = 0; l < S; ++l) {
      if (!mask[p * S + l]) continue;
      const float inner = sdf[p * S + l];
      float e_in;
      const float inner_cdf = sdf_to_cdf(inner, s, e_in);
      const float raw = alpha_raw(outer_cdf, inner_cdf);
      const float alpha = clamp01(raw);
      const float weight = __fmul_rn(alpha, T);
      const float inv = __fdiv_rn(1.0f, __fadd_rn(__fsub_rn(1.0f, alpha), 1e-6f));
      float d_alpha = 0.f;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float col = colors[(p * S + l) * 3 + c];
        acc[c] = __fadd_rn(acc[c], __fmul_rn(weight, col));
        const float suffix = final_rgb[c] - acc[c];
        d_alpha += dL[c] * (T * col - suffix * inv);
        grad_colors[(p * S + l) * 3 + c] += weight * dL[c];
      }
      d_alpha += -dLT * final_T * inv;
      const float d_raw = (raw > 0.0f && raw < 1.0f) ? d_alpha : 0.0f;
      const float den = outer_cdf + 1e-5f;
      const float num = (outer_cdf - inner_cdf) + 1e-5f;
      const float d_num = d_raw / den;
      const float d_den = -d_raw * num / (den * den);
      const float d_oc = d_num + d_den;
      const float d_ic = -d_num;
      const float ki = inner_cdf * inner_cdf * e_in;
      const float ko = outer_cdf * outer_cdf * e_out;
      d_sharp_total += d_ic * ki * inner + d_oc * ko * outer_sdf;
      if (!first) {
        d_partial += d_oc * ko * s;
        const int slot = exact ? prev_shell : l - 1;
        grad_sdf[p * S + slot] += d_partial;
      }
      d_partial = d_ic * ki * s;
      T = __fmul_rn(T, __fsub_rn(1.0f, alpha));
      outer_cdf = inner_cdf;
      outer_sdf = inner;
      e_out = e_in;
      first = false;
      prev_shell = l;
    }
    if (!first) grad_sdf[p * S + (exact ? prev_shell : S - 1)] += d_partial;
  }
  block_sum_to(d_sharp_total, grad_sharpness);
}

// ---------------------------------------------------------------------------
// The explicit render's shading: interpolation and compositing of every shell
// of a pixel in one pass, and its adjoint, with the operations of the kernels
// above in their order. One thread per pixel; the per-shell samples stay in
// registers, where interpolate + composite write them per shell ([B, S, H, W],
// 16 B a sample), lay them out per pixel and read them again, and the adjoint
// does the same with their gradients.
//
// Bound by the scattered reads of the hit faces' vertices (forward) and the
// atomics on them (backward). 4 x 800^2, 8 shells: the kernels and
// layout copies of interpolate + composite took 0.5 ms forward and 0.6 ms
// backward; this 81 and 209 us.
// ---------------------------------------------------------------------------
struct ShellArgs {
  const float* uv;       // [B, S, H, W, 2]
  const int32_t* index;  // [B, S, H, W], -1 = miss
  const int32_t* faces;
  const float* sdf;     // [V]
  const float* colors;  // [B, V, 3]
  int64_t V, HW;
  int B, S;
  const float* sharpness;
  const float* background;  // [3], blended into the output image (NULL: no image)
};

// A pixel's hit on one shell: its vertices, weights and interpolated sample
// (interpolate.slang:22-76; w = 1 - u - v).
struct ShellHit {
  int32_t id[3];
  float wt[3];
  float sdf, rgb[3];
};

__device__ __forceinline__ ShellHit shell_hit(const ShellArgs& a, int64_t at, int32_t f, const float* __restrict__ col) {
  ShellHit h;
  const float2 uv = __ldg(reinterpret_cast<const float2*>(a.uv) + at);
#pragma unroll
  for (int q = 0; q < 3; ++q) h.id[q] = __ldg(a.faces + 3 * (int64_t)f + q);
  float s[3], c[3][3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    s[q] = __ldg(a.sdf + h.id[q]);
#pragma unroll
    for (int k = 0; k < 3; ++k) c[q][k] = __ldg(col + 3 * (int64_t)h.id[q] + k);
  }
  h.wt[0] = uv.x;
  h.wt[1] = uv.y;
  h.wt[2] = __fsub_rn(__fsub_rn(1.0f, uv.x), uv.y);
  h.sdf = interp(h.wt[0], h.wt[1], h.wt[2], s[0], s[1], s[2]);
#pragma unroll
  for (int k = 0; k < 3; ++k) h.rgb[k] = interp(h.wt[0], h.wt[1], h.wt[2], c[0][k], c[1][k], c[2][k]);
  return h;
}

constexpr int kShadeThreads = 128;

__global__ void __launch_bounds__(kShadeThreads)
    shade_shells_kernel(ShellArgs a, float* __restrict__ out_colors, float* __restrict__ out_T,
                        float* __restrict__ image) {
  const float s = *a.sharpness;
  const int64_t P = a.B * a.HW;
  float bg[3] = {0.f, 0.f, 0.f};
  if (image)
#pragma unroll
    for (int c = 0; c < 3; ++c) bg[c] = __ldg(a.background + c);
  float e;
  const float far_cdf = sdf_to_cdf(1e10f, s, e);
  for (int64_t p = blockIdx.x * (int64_t)kShadeThreads + threadIdx.x; p < P; p += (int64_t)gridDim.x * kShadeThreads) {
    const int64_t b = p / a.HW;
    const int64_t first = b * a.S * a.HW + (p - b * a.HW);
    const float* col = a.colors + b * a.V * 3;
    float acc[3] = {0.f, 0.f, 0.f};
    float T = 1.0f, outer_cdf = far_cdf;
    for (int l = 0; l < a.S; ++l) {
      const int64_t at = first + l * a.HW;
      const int32_t f = __ldg(a.index + at);
      if (f < 0) continue;
      const ShellHit h = shell_hit(a, at, f, col);
      const float inner_cdf = sdf_to_cdf(h.sdf, s, e);
      const float alpha = clamp01(alpha_raw(outer_cdf, inner_cdf));
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c] = over(acc[c], h.rgb[c], T, alpha);
      T = __fmul_rn(T, __fsub_rn(1.0f, alpha));
      outer_cdf = inner_cdf;
    }
    if (out_colors) {
#pragma unroll
      for (int c = 0; c < 3; ++c) out_colors[3 * p + c] = acc[c];
      out_T[p] = T;
    }
    if (image)
#pragma unroll
      for (int c = 0; c < 3; ++c) image[3 * p + c] = __fadd_rn(acc[c], __fmul_rn(bg[c], T));
  }
}

// The sample gradients of one hit, onto its face's vertices
// (interpolate_backward_kernel).
__device__ __forceinline__ void scatter_hit(const ShellHit& h, const float (&d_rgb)[3], float d_sdf,
                                            float4* __restrict__ rows) {
  if (d_sdf == 0.f && d_rgb[0] == 0.f && d_rgb[1] == 0.f && d_rgb[2] == 0.f) return;
#pragma unroll
  for (int q = 0; q < 3; ++q)
    red_add(rows + h.id[q], h.wt[q] * d_rgb[0], h.wt[q] * d_rgb[1], h.wt[q] * d_rgb[2], h.wt[q] * d_sdf);
}

// grad_out: d loss / d image when the background is blended in, else
// d loss / d out_colors (NULL: zero); grad_T: d loss / d out_T (NULL: zero);
// packed: [B, V] (r, g, b, signed distance) gradients.
__global__ void __launch_bounds__(kShadeThreads)
    shade_shells_backward_kernel(ShellArgs a, const float* __restrict__ out_colors, const float* __restrict__ out_T,
                                 const float* __restrict__ grad_out, const float* __restrict__ grad_T,
                                 float4* __restrict__ packed, float* __restrict__ grad_sharpness, int exact) {
  const float s = *a.sharpness;
  const int64_t P = a.B * a.HW;
  float bg[3] = {0.f, 0.f, 0.f};
  if (a.background)
#pragma unroll
    for (int c = 0; c < 3; ++c) bg[c] = __ldg(a.background + c);
  float e_far;
  const float far_cdf = sdf_to_cdf(1e10f, s, e_far);
  float d_sharp = 0.f;
  for (int64_t p = blockIdx.x * (int64_t)kShadeThreads + threadIdx.x; p < P; p += (int64_t)gridDim.x * kShadeThreads) {
    const int64_t b = p / a.HW;
    const int64_t first = b * a.S * a.HW + (p - b * a.HW);
    const float* col = a.colors + b * a.V * 3;
    float4* rows = packed + b * a.V;
    float dL[3] = {0.f, 0.f, 0.f}, final_rgb[3];
    float dLT = grad_T ? __ldg(grad_T + p) : 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      final_rgb[c] = __ldg(out_colors + 3 * p + c);
      if (grad_out) dL[c] = __ldg(grad_out + 3 * p + c);
      if (a.background) dLT += dL[c] * bg[c];
    }
    const float final_T = __ldg(out_T + p);
    float acc[3] = {0.f, 0.f, 0.f};
    float T = 1.0f, outer_cdf = far_cdf, outer_sdf = 1e10f, e_out = e_far;
    // The previous hit, whose gradient is complete once the next one is known:
    // its signed distance's goes to the slot before the next hit's shell
    // (S - 1 after the last), which is its own or, where the shells between
    // were missed, one without a sample (exact: always its own).
    ShellHit prev{};
    float prev_d[3] = {0.f, 0.f, 0.f}, d_partial = 0.f;
    int prev_shell = -1;
    for (int l = 0; l < a.S; ++l) {
      const int64_t at = first + l * a.HW;
      const int32_t f = __ldg(a.index + at);
      if (f < 0) continue;
      const ShellHit h = shell_hit(a, at, f, col);
      float e_in;
      const float inner_cdf = sdf_to_cdf(h.sdf, s, e_in);
      const float raw = alpha_raw(outer_cdf, inner_cdf);
      const float alpha = clamp01(raw);
      const float weight = __fmul_rn(alpha, T);
      const float inv = __fdiv_rn(1.0f, __fadd_rn(__fsub_rn(1.0f, alpha), 1e-6f));
      float d_alpha = 0.f, d_rgb[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        acc[c] = __fadd_rn(acc[c], __fmul_rn(weight, h.rgb[c]));
        const float suffix = final_rgb[c] - acc[c];
        d_alpha += dL[c] * (T * h.rgb[c] - suffix * inv);
        d_rgb[c] = weight * dL[c];
      }
      d_alpha += -dLT * final_T * inv;
      const float d_raw = (raw > 0.0f && raw < 1.0f) ? d_alpha : 0.0f;
      const float den = outer_cdf + 1e-5f;
      const float num = (outer_cdf - inner_cdf) + 1e-5f;
      const float d_num = d_raw / den;
      const float d_den = -d_raw * num / (den * den);
      const float d_oc = d_num + d_den;
      const float d_ic = -d_num;
      const float ki = inner_cdf * inner_cdf * e_in;
      const float ko = outer_cdf * outer_cdf * e_out;
      d_sharp += d_ic * ki * h.sdf + d_oc * ko * outer_sdf;
      if (prev_shell >= 0) {
        d_partial += d_oc * ko * s;
        scatter_hit(prev, prev_d, exact || prev_shell == l - 1 ? d_partial : 0.f, rows);
      }
      prev = h;
#pragma unroll
      for (int c = 0; c < 3; ++c) prev_d[c] = d_rgb[c];
      d_partial = d_ic * ki * s;
      T = __fmul_rn(T, __fsub_rn(1.0f, alpha));
      outer_cdf = inner_cdf;
      outer_sdf = h.sdf;
      e_out = e_in;
      prev_shell = l;
    }
    if (prev_shell >= 0)
      scatter_hit(prev, prev_d, exact || prev_shell == a.S - 1 ? d_partial : 0.f, rows);
  }
  block_sum_to(d_sharp, grad_sharpness);
}

}  // namespace
}  // namespace mt

using namespace mt;

extern "C" {

int mt_intersect(const float* xy, int64_t V, const int32_t* faces, const int32_t* sorted_triangles,
                 const int64_t* tile_boundaries, int32_t B, int32_t S, int32_t rows, int32_t cols, int32_t tile_h,
                 int32_t tile_w, int32_t H, int32_t W, float* out_uv, int32_t* out_index, mt_stream_t stream) {
  MT_REQUIRE(B >= 0 && S >= 1 && rows >= 0 && cols >= 0 && tile_h > 0 && tile_w > 0 && H >= 0 && W >= 0);
  MT_REQUIRE((int64_t)tile_h * tile_w <= 1024);
  MT_REQUIRE((int64_t)rows * tile_h >= H && (int64_t)cols * tile_w >= W);
  const int64_t blocks = (int64_t)B * S * rows * cols;
  if (blocks == 0 || H == 0 || W == 0) return MT_OK;
  MT_REQUIRE(xy && faces && tile_boundaries && out_uv && out_index);
  MT_REQUIRE(blocks < ((int64_t)1 << 31));
  const int bs = tile_h * tile_w;
  const size_t smem = intersect_smem(bs);
  auto launch = [&](auto kernel_c) -> int {
    constexpr auto kKernel = decltype(kernel_c)::value;
    // The list ranges' static shared memory counts towards the same limit.
    if (set_smem<kKernel>(smem + 1024) != MT_OK) return MT_ERR_CUDA;
    // As many CTAs as fit on the device at once.
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kKernel, bs, smem) != cudaSuccess) return MT_ERR_CUDA;
    const int64_t fit = (int64_t)kSmCount * (per_sm > 0 ? per_sm : 1);
    kKernel<<<(unsigned)(blocks < fit ? blocks : fit), bs, smem, as_stream(stream)>>>(
        xy, V, faces, sorted_triangles, tile_boundaries, blocks, S, rows, cols, tile_h, tile_w, H, W, out_uv,
        out_index);
    MT_CHECK_LAUNCH();
    return MT_OK;
  };
  return bs <= 256 ? launch(Constant<intersect_kernel<256>>{}) : launch(Constant<intersect_kernel<1024>>{});
}

int mt_interpolate(const float* uv, const int32_t* index, int32_t B, int32_t S, int32_t H, int32_t W,
                   const int32_t* faces, const float* signed_distances, const float* colors, int64_t V,
                   float* out_signed_distances, float* out_colors, mt_stream_t stream) {
  MT_REQUIRE(B >= 0 && S >= 1 && H >= 0 && W >= 0 && V >= 0);
  const int64_t total = (int64_t)B * S * H * W;
  if (total == 0) return MT_OK;
  MT_REQUIRE(uv && index && faces && signed_distances && colors && out_signed_distances && out_colors);
  interpolate_forward_kernel<<<grid_stride_blocks(total, 256), 256, 0, as_stream(stream)>>>(
      uv, index, faces, signed_distances, colors, V, S, (int64_t)B * S, (int64_t)H * W, out_signed_distances,
      out_colors);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_interpolate_backward(const float* uv, const int32_t* index, int32_t B, int32_t S, int32_t H, int32_t W,
                            const int32_t* faces, int64_t V, const float* grad_out_signed_distances,
                            const float* grad_out_colors, float* grad_signed_distances, float* grad_colors,
                            mt_stream_t stream) {
  MT_REQUIRE(B >= 0 && S >= 1 && H >= 0 && W >= 0 && V >= 0);
  const int64_t total = (int64_t)B * S * H * W;
  if (total == 0) return MT_OK;
  MT_REQUIRE(uv && index && faces && grad_signed_distances && grad_colors);
  interpolate_backward_kernel<<<grid_stride_blocks(total, 256), 256, 0, as_stream(stream)>>>(
      uv, index, faces, V, S, (int64_t)B * S, (int64_t)H * W, grad_out_signed_distances, grad_out_colors,
      grad_signed_distances, grad_colors);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_composite(const float* signed_distances, const float* colors, const uint8_t* mask, int64_t P, int32_t S,
                 const float* sharpness, float* out_colors, float* out_transmittances, mt_stream_t stream) {
  MT_REQUIRE(P >= 0 && S >= 0);
  if (P == 0) return MT_OK;
  MT_REQUIRE(sharpness && out_colors && out_transmittances);
  MT_REQUIRE(S == 0 || (signed_distances && colors && mask));
  shell_composite_forward_kernel<<<grid_stride_blocks(P, 256), 256, 0, as_stream(stream)>>>(
      signed_distances, colors, mask, P, S, sharpness, out_colors, out_transmittances);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_composite_backward(const float* signed_distances, const float* colors, const uint8_t* mask, int64_t P,
                          int32_t S, const float* sharpness, const float* out_colors,
                          const float* out_transmittances, const float* grad_out_colors,
                          const float* grad_out_transmittances, float* grad_signed_distances, float* grad_colors,
                          float* grad_sharpness, int32_t exact_adjoint, mt_stream_t stream) {
  MT_REQUIRE(P >= 0 && S >= 0);
  if (P == 0 || S == 0) return MT_OK;
  MT_REQUIRE(signed_distances && colors && mask && sharpness && out_colors && out_transmittances);
  MT_REQUIRE(grad_signed_distances && grad_colors && grad_sharpness);
  shell_composite_backward_kernel<<<grid_stride_blocks(P, 256), 256, 0, as_stream(stream)>>>(
      signed_distances, colors, mask, P, S, sharpness, out_colors, out_transmittances, grad_out_colors,
      grad_out_transmittances, grad_signed_distances, grad_colors, grad_sharpness, exact_adjoint ? 1 : 0);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_shade_shells(const float* uv, const int32_t* index, int32_t B, int32_t S, int32_t H, int32_t W,
                    const int32_t* faces, const float* signed_distances, const float* colors, int64_t V,
                    const float* sharpness, const float* background, float* out_colors, float* out_transmittances,
                    float* image, mt_stream_t stream) {
  MT_REQUIRE(B >= 0 && S >= 1 && H >= 0 && W >= 0 && V >= 0);
  const int64_t P = (int64_t)B * H * W;
  if (P == 0) return MT_OK;
  MT_REQUIRE(uv && index && faces && signed_distances && colors && sharpness);
  MT_REQUIRE((out_colors != nullptr) == (out_transmittances != nullptr) && (out_colors || image));
  MT_REQUIRE((image == nullptr) == (background == nullptr));
  MT_REQUIRE((reinterpret_cast<uintptr_t>(uv) & 7) == 0);
  const ShellArgs a{uv, index, faces, signed_distances, colors, V, (int64_t)H * W, B, S, sharpness, background};
  shade_shells_kernel<<<grid_stride_blocks(P, kShadeThreads, 64), kShadeThreads, 0, as_stream(stream)>>>(
      a, out_colors, out_transmittances, image);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_shade_shells_backward(const float* uv, const int32_t* index, int32_t B, int32_t S, int32_t H, int32_t W,
                             const int32_t* faces, const float* signed_distances, const float* colors, int64_t V,
                             const float* sharpness, const float* background, const float* out_colors,
                             const float* out_transmittances, const float* grad_out,
                             const float* grad_out_transmittances, float* packed_gradients, float* grad_sharpness,
                             int32_t exact_adjoint, mt_stream_t stream) {
  MT_REQUIRE(B >= 0 && S >= 1 && H >= 0 && W >= 0 && V >= 0);
  const int64_t P = (int64_t)B * H * W;
  if (P == 0) return MT_OK;
  MT_REQUIRE(uv && index && faces && signed_distances && colors && sharpness && out_colors && out_transmittances);
  MT_REQUIRE(packed_gradients && grad_sharpness && (reinterpret_cast<uintptr_t>(packed_gradients) & 15) == 0);
  MT_REQUIRE((reinterpret_cast<uintptr_t>(uv) & 7) == 0);
  const ShellArgs a{uv, index, faces, signed_distances, colors, V, (int64_t)H * W, B, S, sharpness, background};
  shade_shells_backward_kernel<<<grid_stride_blocks(P, kShadeThreads, 64), kShadeThreads, 0, as_stream(stream)>>>(
      a, out_colors, out_transmittances, grad_out, grad_out_transmittances,
      reinterpret_cast<float4*>(packed_gradients), grad_sharpness, exact_adjoint ? 1 : 0);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

}  // extern "C"

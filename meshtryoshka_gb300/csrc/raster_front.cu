// Rasterization front end for sm_103a: camera centres, vertex projection,
// spherical-harmonic colours (forward / backward), triangle tile bounds, key
// generation and tile delineation.
//
// Follows triangle_rasterization/project_vertices.slang, bound_triangles.slang,
// generate_keys.slang + keys.slang, delineate_tiles.slang and
// evaluate_spherical_harmonics.slang. Arithmetic follows the reference
// source's operations in their order, without contraction (explicit
// __fmul_rn / __fadd_rn, never fused by nvcc), so projected positions, tile
// bounds, key depths and colours equal the reference kernels evaluated
// operation by operation in IEEE-754 single precision.

#include "lookback.cuh"  // warp_sum, warp_inclusive_sum
#include "sh.cuh"

namespace mt {
namespace {

// ---------------------------------------------------------------------------
// Camera centres: inverse(extrinsics)[:, :3, 3]
// (triangle_rasterization/evaluate_spherical_harmonics.py:38), in fp64.
// ---------------------------------------------------------------------------
// One warp per camera: column 3 of the inverse is C[3][r] / det with
// det = sum_c m[0][c] C[0][c], so only seven cofactors are needed; lanes
// 0-3 compute C[0][c], lanes 4-6 C[3][r] (one 3x3 minor each).
__global__ void camera_positions_kernel(const float* __restrict__ ext, int B, float* __restrict__ out) {
  const int cam = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (cam >= B) return;  // whole warps exit together
  const float* E = ext + 16 * cam;
  double cof = 0.0;
  if (lane < 7) {
    const int skip_r = lane < 4 ? 0 : 3, skip_c = lane < 4 ? lane : lane - 4;
    int rs[3], cs[3], ri = 0, ci = 0;
    for (int k = 0; k < 4; ++k) {
      if (k != skip_r) rs[ri++] = k;
      if (k != skip_c) cs[ci++] = k;
    }
    auto m = [&](int r, int c) { return (double)E[4 * r + c]; };
    const double minor =
        m(rs[0], cs[0]) * (m(rs[1], cs[1]) * m(rs[2], cs[2]) - m(rs[1], cs[2]) * m(rs[2], cs[1])) -
        m(rs[0], cs[1]) * (m(rs[1], cs[0]) * m(rs[2], cs[2]) - m(rs[1], cs[2]) * m(rs[2], cs[0])) +
        m(rs[0], cs[2]) * (m(rs[1], cs[0]) * m(rs[2], cs[1]) - m(rs[1], cs[1]) * m(rs[2], cs[0]));
    cof = ((skip_r + skip_c) & 1) ? -minor : minor;
  }
  double det = 0.0;
#pragma unroll
  for (int c = 0; c < 4; ++c) det += (double)E[c] * __shfl_sync(0xffffffffu, cof, c);
  if (lane >= 4 && lane < 7) out[3 * cam + (lane - 4)] = (float)(cof / det);
}

// ---------------------------------------------------------------------------
// project_vertices.slang:51-92. cam = W2C [v, 1]; xy = (K cam).xy / cam.z.
// ---------------------------------------------------------------------------
// A CTA takes kEach vertices for each of its threads, so that a camera's 21
// values are read once for them (they were a quarter of the instructions).
// kPair: out_xy is 8-byte aligned. 14.7 M vertices and 4 cameras: 300 us with
// one vertex to a thread and two stores of a position, now 233 (the writes alone
// 130); 505,000 vertices 16, now 9.
constexpr int kProjectThreads = 256;

template <int kEach, bool kPair>
__global__ void __launch_bounds__(kProjectThreads)
    project_kernel(const float* __restrict__ verts, int64_t V, const float* __restrict__ ext,
                   const float* __restrict__ intr, int B, float* __restrict__ out_xy, float* __restrict__ out_depth) {
  for (int64_t base = blockIdx.x * (int64_t)(kEach * kProjectThreads) + threadIdx.x; base < V;
       base += (int64_t)gridDim.x * (kEach * kProjectThreads)) {
    float x[kEach], y[kEach], z[kEach];
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
      const int64_t v = min(base + j * kProjectThreads, V - 1);
      x[j] = __ldg(verts + 3 * v);
      y[j] = __ldg(verts + 3 * v + 1);
      z[j] = __ldg(verts + 3 * v + 2);
    }
    for (int b = 0; b < B; ++b) {
      float E[12], K[6];
#pragma unroll
      for (int i = 0; i < 12; ++i) E[i] = __ldg(ext + 16 * b + i);
#pragma unroll
      for (int i = 0; i < 6; ++i) K[i] = __ldg(intr + 9 * b + i);
#pragma unroll
      for (int j = 0; j < kEach; ++j) {
        const int64_t v = base + j * kProjectThreads;
        if (v >= V) break;
        // mul(W2C, float4(v, 1)) and mul(K, cam.xyz): row sums left to right.
        float cam[3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
          cam[r] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(E[4 * r], x[j]), __fmul_rn(E[4 * r + 1], y[j])),
                                       __fmul_rn(E[4 * r + 2], z[j])),
                             __fmul_rn(E[4 * r + 3], 1.0f));
        const float kx =
            __fadd_rn(__fadd_rn(__fmul_rn(K[0], cam[0]), __fmul_rn(K[1], cam[1])), __fmul_rn(K[2], cam[2]));
        const float ky =
            __fadd_rn(__fadd_rn(__fmul_rn(K[3], cam[0]), __fmul_rn(K[4], cam[1])), __fmul_rn(K[5], cam[2]));
        const int64_t o = (int64_t)b * V + v;
        const float px = __fdiv_rn(kx, cam[2]), py = __fdiv_rn(ky, cam[2]);
        if constexpr (kPair) {
          reinterpret_cast<float2*>(out_xy)[o] = make_float2(px, py);
        } else {
          out_xy[2 * o] = px;
          out_xy[2 * o + 1] = py;
        }
        out_depth[o] = cam[2];
      }
    }
  }
}

// The vertex's coefficients are read once into registers and serve every
// camera.
template <int kCoeff>
__device__ __forceinline__ void sh_forward_vertex(const float* __restrict__ verts, int64_t V,
                                                  const float* __restrict__ sh, const float* __restrict__ campos,
                                                  int B, int64_t v, float* __restrict__ out) {
  float coef[kCoeff][3];
#pragma unroll
  for (int k = 0; k < kCoeff; ++k) {
    const float* s = sh + ((int64_t)k * V + v) * 3;
    coef[k][0] = __ldg(s);
    coef[k][1] = __ldg(s + 1);
    coef[k][2] = __ldg(s + 2);
  }
  sh_colors<kCoeff>(verts, V, coef, campos, B, v, out);
}

__global__ void sh_forward_kernel(const float* __restrict__ verts, int64_t V, const float* __restrict__ sh,
                                  int n_coeff, const float* __restrict__ campos, int B, float* __restrict__ out) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x) {
    switch (n_coeff) {
      case 1: sh_forward_vertex<1>(verts, V, sh, campos, B, v, out); break;
      case 4: sh_forward_vertex<4>(verts, V, sh, campos, B, v, out); break;
      case 9: sh_forward_vertex<9>(verts, V, sh, campos, B, v, out); break;
      default: sh_forward_vertex<16>(verts, V, sh, campos, B, v, out); break;
    }
  }
}

// d sh_k = sum_b basis_k(dir_b) * d rgb_b * [rgb_b + 0.5 > 0]; the mask is
// read from the forward output (out > 0 exactly when the pre-clamp value is).
// Every row of the output is written (rows k >= n_coeff get zeros).
template <bool kPacked>
__global__ void sh_backward_kernel(const float* __restrict__ verts, int64_t V, int n_coeff, int C,
                                   const float* __restrict__ campos, int B, const float* __restrict__ colors,
                                   const float* __restrict__ dcolors, float* __restrict__ dsh) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x) {
    float acc[16][3];
    for (int k = 0; k < 16; ++k) acc[k][0] = acc[k][1] = acc[k][2] = 0.f;
    for (int b = 0; b < B; ++b) {
      const int64_t o = (int64_t)b * V + v;
      float g[3];
      colour_gradient<kPacked>(dcolors, o, g);
      bool any = false;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        g[c] = colors[3 * o + c] > 0.0f ? g[c] : 0.0f;
        any |= g[c] != 0.0f;
      }
      if (!any) continue;
      float x, y, z;
      view_dir(verts, v, campos + 3 * b, x, y, z);
      float basis[16];
      sh_basis(x, y, z, n_coeff, basis);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        if (k < n_coeff) {
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[k][c] += basis[k] * g[c];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      if (k < C) {
        float* d = dsh + ((int64_t)k * V + v) * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c) d[c] = acc[k][c];
      }
    }
    for (int k = 16; k < C; ++k) {
      float* d = dsh + ((int64_t)k * V + v) * 3;
      d[0] = d[1] = d[2] = 0.f;
    }
  }
}

// ---------------------------------------------------------------------------
// bound_triangles.slang:62-192: back-face and near-plane culling, tile AABB
// with min = int(x) / ts (truncation), max = int(ceil(x / ts)), clamped.
// ---------------------------------------------------------------------------
struct TileBounds {
  int r0, c0, r1, c1;
};

// ymax / tile as the reference divides it: for a power-of-two tile the
// product with the exact reciprocal is the same correctly rounded quotient.
__device__ __forceinline__ float div_by_tile(float x, int tile) {
  if ((tile & (tile - 1)) == 0) return __fmul_rn(x, __int_as_float((127 - (__ffs(tile) - 1)) << 23));
  return __fdiv_rn(x, (float)tile);
}

// max(v / tile, 0) with C's truncating division; for a power-of-two tile a
// shift (flooring) differs only for negative v, where both clamp to 0.
__device__ __forceinline__ int first_tile(int v, int tile) {
  if ((tile & (tile - 1)) == 0) return max(v >> (__ffs(tile) - 1), 0);
  return max(v / tile, 0);
}

// Tile rectangle of one projected triangle; mean_depth receives
// (ad + bd + cd) / 3 (keys.slang's key depth) when the face is not culled.
__device__ __forceinline__ TileBounds bounds_from_corners(float ax, float ay, float ad, float bx, float by, float bd,
                                                          float cx, float cy, float cd, int tile_h, int tile_w,
                                                          int rows, int cols, float near, float& mean_depth) {
  TileBounds t{0, 0, 0, 0};
  const float check = __fsub_rn(__fmul_rn(__fsub_rn(bx, ax), __fsub_rn(cy, ay)),
                                __fmul_rn(__fsub_rn(by, ay), __fsub_rn(cx, ax)));
  if (check < 0.0f) return t;
  if (fminf(fminf(ad, bd), cd) < near) return t;
  mean_depth = __fdiv_rn(__fadd_rn(__fadd_rn(ad, bd), cd), 3.0f);
  const float ymin = fminf(fminf(ay, by), cy), ymax = fmaxf(fmaxf(ay, by), cy);
  const float xmin = fminf(fminf(ax, bx), cx), xmax = fmaxf(fmaxf(ax, bx), cx);
  t.r0 = min(first_tile(f2i_rz(ymin), tile_h), rows);
  t.r1 = min(max(f2i_rz(ceilf(div_by_tile(ymax, tile_h))), 0), rows);
  t.c0 = min(first_tile(f2i_rz(xmin), tile_w), cols);
  t.c1 = min(max(f2i_rz(ceilf(div_by_tile(xmax, tile_w))), 0), cols);
  return t;
}

__device__ __forceinline__ bool face_in_range(int32_t ia, int32_t ib, int32_t ic, int64_t V) {
  return (uint64_t)ia < (uint64_t)V && (uint64_t)ib < (uint64_t)V && (uint64_t)ic < (uint64_t)V;
}

__device__ __forceinline__ TileBounds triangle_tile_bounds(const float* __restrict__ xy,
                                                           const float* __restrict__ depth, int64_t V,
                                                           const int32_t* __restrict__ faces, int64_t f, int b,
                                                           int tile_h, int tile_w, int rows, int cols, float near,
                                                           float& mean_depth) {
  const int64_t base = (int64_t)b * V;
  const int32_t ia = faces[3 * f], ib = faces[3 * f + 1], ic = faces[3 * f + 2];
  // A face that names a vertex outside [0, V) (only possible when an upstream
  // capacity overflowed) covers no tile.
  if (!face_in_range(ia, ib, ic, V)) return TileBounds{0, 0, 0, 0};
  return bounds_from_corners(xy[2 * (base + ia)], xy[2 * (base + ia) + 1], depth[base + ia], xy[2 * (base + ib)],
                             xy[2 * (base + ib) + 1], depth[base + ib], xy[2 * (base + ic)], xy[2 * (base + ic) + 1],
                             depth[base + ic], tile_h, tile_w, rows, cols, near, mean_depth);
}

// Rows f >= num_faces (a device value; all F when NULL) cover no tile.
// cameras: NULL (every camera has rows x cols tiles) or the ragged camera
// table [B, 6] whose first two columns give each camera's own grid.
__global__ void bound_kernel(const float* __restrict__ xy, const float* __restrict__ depth, int64_t V,
                             const int32_t* __restrict__ faces, int64_t F, const int32_t* __restrict__ num_faces,
                             int B, int tile_h, int tile_w, int rows, int cols, const int64_t* __restrict__ cameras,
                             float near, int32_t* __restrict__ out_min, int32_t* __restrict__ out_max,
                             int32_t* __restrict__ out_count) {
  const int64_t total = (int64_t)B * F;
  const int64_t live = num_faces ? min((int64_t)max(*num_faces, 0), F) : F;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int b = (int)(i / F);
    const int64_t f = i - (int64_t)b * F;
    const int rb = cameras ? (int)cameras[6 * b] : rows, cb = cameras ? (int)cameras[6 * b + 1] : cols;
    float mean;
    const TileBounds t = f < live ? triangle_tile_bounds(xy, depth, V, faces, f, b, tile_h, tile_w, rb, cb, near, mean)
                                  : TileBounds{0, 0, 0, 0};
    out_min[2 * i] = t.r0;
    out_min[2 * i + 1] = t.c0;
    out_max[2 * i] = t.r1;
    out_max[2 * i + 1] = t.c1;
    out_count[i] = (t.r1 - t.r0) * (t.c1 - t.c0);
  }
}

// ---------------------------------------------------------------------------
// generate_keys.slang:4-68 + keys.slang:6-22. One thread per (camera, face);
// keys land at the exclusive offset of (camera, face) in row-major tile order,
// so the unsorted order (and therefore the stable sort's tie order) is the
// reference's.
// ---------------------------------------------------------------------------
struct KeyLayout {
  int cam_off, cam_len, shell_off, shell_len, tile_off, tile_len, depth_off;
};

__device__ __forceinline__ uint64_t field_mask(int len) { return (uint64_t)((1u << len) - 1u); }

__global__ void keys_kernel(const float* __restrict__ depth, int64_t V, const int32_t* __restrict__ faces,
                            int64_t F, const int32_t* __restrict__ sfb, int S, const int32_t* __restrict__ tmin,
                            const int32_t* __restrict__ tmax, const int64_t* __restrict__ offsets, int B,
                            int grid_width, const int64_t* __restrict__ cameras, KeyLayout L, int64_t K,
                            uint64_t* __restrict__ out_keys, int32_t* __restrict__ out_tri) {
  const int64_t total = (int64_t)B * F;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int b = (int)(i / F);
    const int64_t f = i - (int64_t)b * F;
    const int r0 = tmin[2 * i], c0 = tmin[2 * i + 1], r1 = tmax[2 * i], c1 = tmax[2 * i + 1];
    if (r1 <= r0 || c1 <= c0) continue;
    uint32_t shell = 0;
    for (; shell < (uint32_t)S; ++shell)
      if (f < sfb[shell]) break;
    const int64_t base = (int64_t)b * V;
    const float da = depth[base + faces[3 * f]], db = depth[base + faces[3 * f + 1]],
                dc = depth[base + faces[3 * f + 2]];
    const float mean = __fdiv_rn(__fadd_rn(__fadd_rn(da, db), dc), 3.0f);
    const uint64_t fixed = (((uint64_t)b & field_mask(L.cam_len)) << L.cam_off) |
                           (((uint64_t)shell & field_mask(L.shell_len)) << L.shell_off) |
                           ((uint64_t)__float_as_uint(mean) << L.depth_off);
    int64_t k = (i == 0) ? 0 : offsets[i - 1];
    const int width = cameras ? (int)cameras[6 * b + 1] : grid_width;  // tiles per row of this camera
    for (int r = r0; r < r1; ++r) {
      for (int c = c0; c < c1; ++c) {
        if (k >= K) return;  // guarded: offsets and K always agree for valid inputs
        const uint32_t tile = (uint32_t)(r * width + c);
        out_keys[k] = fixed | (((uint64_t)tile & field_mask(L.tile_len)) << L.tile_off);
        out_tri[k] = (int32_t)f;
        ++k;
      }
    }
  }
}

// Shell of face f: the first boundary above f (keys.slang's shell field).
__device__ __forceinline__ uint32_t face_shell(const int32_t* __restrict__ sfb, int S, int64_t f) {
  uint32_t shell = 0;
  for (; shell < (uint32_t)S; ++shell)
    if (f < sfb[shell]) break;
  return shell;
}

// ---------------------------------------------------------------------------
// Tile bounds, key offsets and keys of a render. The keys and their order equal
// bound_kernel followed by an inclusive scan of the counts and keys_kernel:
// item i = (camera, face) in row-major order writes its keys at the sum of the
// counts of items < i.
//
// The B*F items are split into chunks of kFusedItems x kFusedThreads items,
// one CTA each, striped (item j * kFusedThreads + tid of the chunk) so that a
// warp's loads are adjacent. Three launches (four for many chunks), no CTA
// waits on another:
//   chunk_bounds_kernel  the tile rectangle (int4) and key depth of the items
//                        that touch a tile, in item order at the start of the
//                        chunk's records, with their places in the chunk; and
//                        the chunk's item and key counts;
//   chunk_scan_kernel    exclusive scan of the chunks' key counts, and the
//                        total: one CTA, or for many chunks one to each group
//                        of them, after chunk_group_kernel has summed each;
//   chunk_keys_kernel    reads its chunk's records back (coalesced), scans
//                        them and writes the keys.
// Most items touch no tile (back faces, faces outside the image), and a record
// for each of them was most of both kernels' traffic: 1003 and 769 us at 512^3,
// 16 shells, 4 cameras (96 M live faces x cameras), now 975 and 245.
// ---------------------------------------------------------------------------
constexpr int kFusedThreads = 256;
constexpr int kFusedItems = 4;
constexpr int kFusedSubTile = kFusedThreads * kFusedItems;
constexpr int kChunkScanThreads = 1024;
// Workspace: [0,256) status word (unused here: nothing waits), the chunks' key
// counts (int64 each) and item counts (int32 each), the groups' totals (int64
// each), the rectangle records (int4 per item), the key depths (float per item)
// and the places (uint16 per item); each region starts on a 256-byte boundary.
constexpr size_t kFusedHeader = 256;

__host__ __device__ inline size_t round256(size_t x) { return (x + 255) / 256 * 256; }

struct FusedArgs {
  const float* xy;
  const float* depth;
  int64_t V;
  const int32_t* faces;
  int64_t F;
  const int32_t* num_faces;
  int B, tile_h, tile_w, rows, cols;
  const int64_t* cameras;
  float near;
};

// The int32 count of bound_kernel, widened as the scan widens it.
__device__ __forceinline__ int64_t tile_count(const TileBounds& t) {
  return (int64_t)((t.r1 - t.r0) * (t.c1 - t.c0));
}

// Bounds (and key depth) of this thread's kFusedItems items of the sub-tile
// starting at item `first`, loads of all items issued together.
__device__ __forceinline__ void subtile_bounds(const FusedArgs& a, int64_t first, int64_t end, int64_t live,
                                               int (&cam)[kFusedItems], int64_t (&face)[kFusedItems],
                                               TileBounds (&t)[kFusedItems], float (&mean)[kFusedItems]) {
  {
    const int64_t i0 = first + threadIdx.x;
    // In 32 bits where the items allow: a 64-bit division takes 100 instructions.
    int b = (end >> 32) == 0 ? (int)((uint32_t)i0 / (uint32_t)a.F) : (int)(i0 / a.F);
    int64_t f = i0 - (int64_t)b * a.F;
#pragma unroll
    for (int j = 0; j < kFusedItems; ++j) {
      // Items at or past `end` (the chunk's end or B*F) get camera B.
      cam[j] = (i0 + (int64_t)j * kFusedThreads < end) ? b : a.B;
      face[j] = f;
      f += kFusedThreads;
      while (f >= a.F) {
        f -= a.F;
        ++b;
      }
    }
  }
  int32_t corner[kFusedItems][3];
#pragma unroll
  for (int j = 0; j < kFusedItems; ++j) {
    const bool ok = cam[j] < a.B && face[j] < live;
#pragma unroll
    for (int c = 0; c < 3; ++c) corner[j][c] = ok ? __ldg(a.faces + 3 * face[j] + c) : -1;
  }
  // Depths beside the positions: read only for faces with a rectangle, they
  // would wait for the positions (1051 us instead of 1002 at 512^3).
  float2 p[kFusedItems][3];
  float d[kFusedItems][3];
  bool ok[kFusedItems];
#pragma unroll
  for (int j = 0; j < kFusedItems; ++j) {
    ok[j] = face_in_range(corner[j][0], corner[j][1], corner[j][2], a.V);
    const int64_t base = (int64_t)cam[j] * a.V;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t v = base + (ok[j] ? corner[j][c] : 0);
      p[j][c] = ok[j] ? __ldg(reinterpret_cast<const float2*>(a.xy) + v) : make_float2(0.f, 0.f);
      d[j][c] = ok[j] ? __ldg(a.depth + v) : 0.f;
    }
  }
#pragma unroll
  for (int j = 0; j < kFusedItems; ++j) {
    t[j] = TileBounds{0, 0, 0, 0};
    mean[j] = 0.0f;
    if (ok[j]) {
      const int rb = a.cameras ? (int)a.cameras[6 * cam[j]] : a.rows;
      const int cb = a.cameras ? (int)a.cameras[6 * cam[j] + 1] : a.cols;
      t[j] = bounds_from_corners(p[j][0].x, p[j][0].y, d[j][0], p[j][1].x, p[j][1].y, d[j][1], p[j][2].x, p[j][2].y,
                                 d[j][2], a.tile_h, a.tile_w, rb, cb, a.near, mean[j]);
    }
  }
}

template <typename T>
__device__ __forceinline__ T block_sum(T x, T* s_warp) {
  x = warp_sum(x);
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = x;
  __syncthreads();
  T total = 0;
#pragma unroll
  for (int w = 0; w < kFusedThreads / 32; ++w) total += s_warp[w];
  return total;
}

struct ChunkRecords {
  int64_t* keys;    // per chunk: key count, then (scanned) its first key
  int32_t* items;   // per chunk: records
  int64_t* groups;  // per kScanGroup chunks: key count; NULL: one group
  int4* rect;       // per record (a chunk's start at its first item)
  float* depth;
  uint16_t* place;  // item's place in its chunk
};

__global__ void __launch_bounds__(kFusedThreads, 3) chunk_bounds_kernel(FusedArgs a, ChunkRecords rec) {
  constexpr int kWarps = kFusedThreads / 32;
  __shared__ int64_t s_warp[kWarps];
  __shared__ int s_live[kFusedItems * kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t items = (int64_t)a.B * a.F;
  const int64_t first = blockIdx.x * (int64_t)kFusedSubTile, end = min(first + kFusedSubTile, items);
  const int64_t live = a.num_faces ? min((int64_t)max(*a.num_faces, 0), a.F) : a.F;
  int cam[kFusedItems];
  int64_t face[kFusedItems];
  TileBounds t[kFusedItems];
  float mean[kFusedItems];
  subtile_bounds(a, first, end, live, cam, face, t, mean);
  int64_t sum = 0;
  uint32_t touching[kFusedItems];
#pragma unroll
  for (int j = 0; j < kFusedItems; ++j) {
    const int64_t count = tile_count(t[j]);
    sum += count;
    touching[j] = __ballot_sync(0xffffffffu, count != 0);
    if (lane == 0) s_live[j * kWarps + warp] = __popc(touching[j]);
  }
  const int64_t total = block_sum(sum, s_warp);  // its barrier also publishes s_live
  // The counts of all (item row, warp) pairs, one to a lane, scanned in every warp.
  static_assert(kFusedItems * kWarps == 32, "a lane to a pair");
  const int mine = s_live[lane], upto = warp_inclusive_sum(mine);
  const int all = __shfl_sync(0xffffffffu, upto, 31);
#pragma unroll
  for (int j = 0; j < kFusedItems; ++j) {
    const int before = __shfl_sync(0xffffffffu, upto - mine, j * kWarps + warp) + __popc(touching[j] & lanemask_lt());
    if ((touching[j] >> lane) & 1u) {
      rec.rect[first + before] = make_int4(t[j].r0, t[j].c0, t[j].r1, t[j].c1);
      rec.depth[first + before] = mean[j];
      rec.place[first + before] = (uint16_t)(j * kFusedThreads + threadIdx.x);
    }
  }
  if (threadIdx.x == 0) {
    rec.keys[blockIdx.x] = total;
    rec.items[blockIdx.x] = all;
  }
}

// Exclusive scan of the chunk counts in place, a CTA to each `group` consecutive
// ones; *out_count = total. Rounds of kScanGroup counts, each thread's four
// loaded together. Up to kOneCtaChunks chunks are one group (512^3's 117,000 in
// 29 rounds of one CTA took 117 us); of more, every kScanGroup are one, whose
// sum is known (`totals`), and each CTA adds up those of the groups before it.
constexpr int kScanPer = 4, kScanGroup = kScanPer * kChunkScanThreads;
constexpr int64_t kOneCtaChunks = 4 * kScanGroup;

// Sum of x over the CTA's kChunkScanThreads threads.
__device__ __forceinline__ int64_t scan_block_sum(int64_t x, int64_t* s_warp) {
  x = warp_sum(x);
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = x;
  __syncthreads();
  int64_t total = 0;
#pragma unroll
  for (int w = 0; w < kChunkScanThreads / 32; ++w) total += s_warp[w];
  __syncthreads();
  return total;
}

__global__ void __launch_bounds__(kChunkScanThreads)
    chunk_group_kernel(const int64_t* __restrict__ counts, int64_t chunks, int64_t* __restrict__ totals) {
  __shared__ int64_t s_warp[kChunkScanThreads / 32];
  int64_t mine = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int64_t c = blockIdx.x * (int64_t)kScanGroup + k * kChunkScanThreads + threadIdx.x;
    mine += c < chunks ? counts[c] : 0;
  }
  const int64_t total = scan_block_sum(mine, s_warp);
  if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kChunkScanThreads)
    chunk_scan_kernel(int64_t* __restrict__ counts, int64_t chunks, int64_t group,
                      const int64_t* __restrict__ totals, int64_t* __restrict__ out_count) {
  constexpr int kPer = kScanPer;
  __shared__ int64_t s_warp[kChunkScanThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t begin = blockIdx.x * group, end = min(begin + group, chunks);
  int64_t running = 0;
  if (totals) {
    for (int64_t g = tid; g < blockIdx.x; g += kChunkScanThreads) running += totals[g];
    running = scan_block_sum(running, s_warp);
  }
  for (int64_t base = begin; base < end; base += kScanGroup) {
    const int64_t c0 = base + (int64_t)tid * kPer;
    int64_t x[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) x[k] = c0 + k < end ? counts[c0 + k] : 0;
    int64_t mine = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) mine += x[k];
    const int64_t inc = warp_inclusive_sum(mine);
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    int64_t below = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kChunkScanThreads / 32; ++w) {
      const int64_t y = s_warp[w];
      all += y;
      below += (w < warp) ? y : 0;
    }
    int64_t run = running + below + inc - mine;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      if (c0 + k < end) counts[c0 + k] = run;
      run += x[k];
    }
    running += all;
    __syncthreads();
  }
  if (tid == 0 && blockIdx.x == gridDim.x - 1) *out_count = running;
}

// Each thread writes the keys of its records (in row-major tile order, at the
// item's exclusive offset: the chunk's offset + the CTA scan of the counts), as
// keys_kernel does.
__global__ void __launch_bounds__(kFusedThreads)
    chunk_keys_kernel(FusedArgs a, ChunkRecords rec, const int32_t* __restrict__ sfb, int S, KeyLayout L, int64_t K,
                      uint64_t* __restrict__ out_keys, int32_t* __restrict__ out_tri) {
  constexpr int kWarps = kFusedThreads / 32;
  __shared__ int64_t s_warp[2][kWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int many = rec.items[blockIdx.x];
  const int64_t first = blockIdx.x * (int64_t)kFusedSubTile;
  const int first_cam = (int)(first / a.F);
  const int64_t first_face = first - (int64_t)first_cam * a.F;
  int64_t base = rec.keys[blockIdx.x];
  int turn = 0;
  for (int p0 = 0; p0 < many; p0 += kFusedThreads, turn ^= 1) {
    const int64_t i = first + p0 + tid;
    const bool in = p0 + tid < many;
    const int4 r4 = in ? __ldcs(rec.rect + i) : make_int4(0, 0, 0, 0);
    const float depth = in ? __ldcs(rec.depth + i) : 0.0f;
    const int place = in ? (int)__ldcs(rec.place + i) : 0;
    const TileBounds tb{r4.x, r4.y, r4.z, r4.w};
    const int64_t count = tile_count(tb);
    const int64_t inc = warp_inclusive_sum(count);
    if (lane == 31) s_warp[turn][warp] = inc;
    __syncthreads();
    int64_t below = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const int64_t x = s_warp[turn][w];
      all += x;
      below += (w < warp) ? x : 0;
    }
    if (tb.r1 > tb.r0 && tb.c1 > tb.c0) {
      int64_t k = base + below + inc - count;
      int b = first_cam;
      int64_t f = first_face + place;
      while (f >= a.F) {
        f -= a.F;
        ++b;
      }
      const uint64_t fixed = (((uint64_t)b & field_mask(L.cam_len)) << L.cam_off) |
                             (((uint64_t)face_shell(sfb, S, f) & field_mask(L.shell_len)) << L.shell_off) |
                             ((uint64_t)__float_as_uint(depth) << L.depth_off);
      const int width = a.cameras ? (int)a.cameras[6 * b + 1] : a.cols;
      for (int r = tb.r0; r < tb.r1 && k < K; ++r) {
        for (int c = tb.c0; c < tb.c1; ++c) {
          if (k >= K || k < 0) break;  // past the capacity
          const uint32_t tile_index = (uint32_t)(r * width + c);
          out_keys[k] = fixed | (((uint64_t)tile_index & field_mask(L.tile_len)) << L.tile_off);
          out_tri[k] = (int32_t)f;
          ++k;
        }
      }
    }
    base += all;
  }
}

// ---------------------------------------------------------------------------
// delineate_tiles.slang:14-58: [start, end) per (camera, shell|0, tile) where
// the (camera, shell|0, tile) index changes between consecutive sorted keys.
// ---------------------------------------------------------------------------
__global__ void delineate_kernel(const uint64_t* __restrict__ keys, int64_t K_capacity,
                                 const int64_t* __restrict__ num_keys, KeyLayout L, int separate_shells, int B,
                                 int Sd, int64_t T, int64_t* __restrict__ out) {
  const int64_t K = num_keys ? min(max(*num_keys, (int64_t)0), K_capacity) : K_capacity;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < K; i += (int64_t)gridDim.x * blockDim.x) {
    auto index_of = [&](uint64_t key) -> int64_t {
      const int64_t cam = (int64_t)((key >> L.cam_off) & field_mask(L.cam_len));
      const int64_t sh = separate_shells ? (int64_t)((key >> L.shell_off) & field_mask(L.shell_len)) : 0;
      const int64_t tile = (int64_t)((key >> L.tile_off) & field_mask(L.tile_len));
      if (cam >= B || sh >= Sd || tile >= T) return -1;
      return (cam * Sd + sh) * T + tile;
    };
    const int64_t here = index_of(keys[i]);
    if (i > 0) {
      const int64_t prev = index_of(keys[i - 1]);
      if (here != prev) {
        if (prev >= 0) out[2 * prev + 1] = i;
        if (here >= 0) out[2 * here] = i;
      }
    }
    if (i == K - 1 && here >= 0) out[2 * here + 1] = K;
  }
}

inline bool layout_ok(const KeyLayout& L) {
  auto ok = [](int off, int len) { return off >= 0 && len >= 0 && len <= 31 && off + len <= 64; };
  return ok(L.cam_off, L.cam_len) && ok(L.shell_off, L.shell_len) && ok(L.tile_off, L.tile_len) &&
         L.depth_off >= 0 && L.depth_off + 32 <= 64;
}

}  // namespace
}  // namespace mt

using namespace mt;

template <bool kPacked>
static int sh_backward(const float* vertices, int64_t V, int32_t C, int32_t sh_degree,
                                             const float* camera_positions, int32_t B, const float* out_colors,
                                             const float* grad_colors, float* grad_spherical_harmonics,
                                             mt_stream_t stream) {
  MT_REQUIRE(V >= 0 && B >= 0 && sh_degree >= 0 && sh_degree <= 3);
  const int n = (sh_degree + 1) * (sh_degree + 1);
  MT_REQUIRE(C >= n);
  if (V == 0) return MT_OK;
  MT_REQUIRE(grad_spherical_harmonics);
  if (B == 0) {
    const size_t bytes = (size_t)C * (size_t)V * 3 * sizeof(float);
    return cudaMemsetAsync(grad_spherical_harmonics, 0, bytes, as_stream(stream)) == cudaSuccess ? MT_OK : MT_ERR_CUDA;
  }
  MT_REQUIRE(vertices && camera_positions && out_colors && grad_colors);
  MT_REQUIRE(!kPacked || (reinterpret_cast<uintptr_t>(grad_colors) & 15) == 0);
  sh_backward_kernel<kPacked><<<grid_stride_blocks(V, 128), 128, 0, as_stream(stream)>>>(
      vertices, V, n, C, camera_positions, B, out_colors, grad_colors, grad_spherical_harmonics);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

extern "C" {

int mt_camera_positions(const float* extrinsics, int32_t B, float* out, mt_stream_t stream) {
  MT_REQUIRE(B >= 0);
  if (B == 0) return MT_OK;
  MT_REQUIRE(extrinsics && out);
  camera_positions_kernel<<<grid_1d((int64_t)B * 32, 128), 128, 0, as_stream(stream)>>>(extrinsics, B, out);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_project_vertices(const float* vertices, int64_t V, const float* extrinsics, const float* intrinsics, int32_t B,
                        float* out_xy, float* out_depth, mt_stream_t stream) {
  MT_REQUIRE(V >= 0 && B >= 0);
  if (V == 0 || B == 0) return MT_OK;
  MT_REQUIRE(vertices && extrinsics && intrinsics && out_xy && out_depth);
  auto launch = [&](auto each, auto pair) {
    constexpr int kEach = decltype(each)::value;
    project_kernel<kEach, decltype(pair)::value>
        <<<grid_stride_blocks(V, kEach * kProjectThreads), kProjectThreads, 0, as_stream(stream)>>>(
            vertices, V, extrinsics, intrinsics, B, out_xy, out_depth);
  };
  // Four vertices to a thread where that leaves every SM two CTAs.
  const bool four = V >= (int64_t)2 * kSmCount * 4 * kProjectThreads;
  const bool pair = (reinterpret_cast<uintptr_t>(out_xy) & 7) == 0;
  if (four && pair) launch(std::integral_constant<int, 4>{}, std::true_type{});
  else if (four) launch(std::integral_constant<int, 4>{}, std::false_type{});
  else if (pair) launch(std::integral_constant<int, 1>{}, std::true_type{});
  else launch(std::integral_constant<int, 1>{}, std::false_type{});
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_evaluate_spherical_harmonics(const float* vertices, int64_t V, const float* spherical_harmonics, int32_t C,
                                    int32_t sh_degree, const float* camera_positions, int32_t B, float* out_colors,
                                    mt_stream_t stream) {
  MT_REQUIRE(V >= 0 && B >= 0 && sh_degree >= 0 && sh_degree <= 3);
  const int n = (sh_degree + 1) * (sh_degree + 1);
  MT_REQUIRE(C >= n);
  if (V == 0 || B == 0) return MT_OK;
  MT_REQUIRE(vertices && spherical_harmonics && camera_positions && out_colors);
  sh_forward_kernel<<<grid_stride_blocks(V, 256), 256, 0, as_stream(stream)>>>(vertices, V, spherical_harmonics, n,
                                                                              camera_positions, B, out_colors);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_evaluate_spherical_harmonics_backward(const float* vertices, int64_t V, int32_t C, int32_t sh_degree,
                                             const float* camera_positions, int32_t B, const float* out_colors,
                                             const float* grad_colors, float* grad_spherical_harmonics,
                                             mt_stream_t stream) {
  return sh_backward<false>(vertices, V, C, sh_degree, camera_positions, B, out_colors, grad_colors, grad_spherical_harmonics, stream);
}

int mt_evaluate_spherical_harmonics_packed_backward(const float* vertices, int64_t V, int32_t C, int32_t sh_degree,
                                             const float* camera_positions, int32_t B, const float* out_colors,
                                             const float* packed_gradients, float* grad_spherical_harmonics,
                                             mt_stream_t stream) {
  return sh_backward<true>(vertices, V, C, sh_degree, camera_positions, B, out_colors, packed_gradients, grad_spherical_harmonics, stream);
}

int mt_bound_triangles(const float* xy, const float* depth, int64_t V, const int32_t* faces, int64_t F,
                       const int32_t* num_faces, int32_t B, int32_t tile_h, int32_t tile_w, int32_t rows,
                       int32_t cols, const int64_t* cameras, float near_plane, int32_t* out_min, int32_t* out_max,
                       int32_t* out_count, mt_stream_t stream) {
  MT_REQUIRE(V >= 0 && F >= 0 && B >= 0 && tile_h > 0 && tile_w > 0 && rows >= 0 && cols >= 0);
  if (F == 0 || B == 0) return MT_OK;
  MT_REQUIRE(xy && depth && faces && out_min && out_max && out_count);
  bound_kernel<<<grid_stride_blocks((int64_t)B * F, 256), 256, 0, as_stream(stream)>>>(
      xy, depth, V, faces, F, num_faces, B, tile_h, tile_w, rows, cols, cameras, near_plane, out_min, out_max,
      out_count);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_generate_keys(const float* depth, int64_t V, const int32_t* faces, int64_t F,
                     const int32_t* shell_face_boundaries, int32_t S, const int32_t* tile_min,
                     const int32_t* tile_max, const int64_t* offsets, int32_t B, int32_t grid_width,
                     const int64_t* cameras, const int32_t* layout, int64_t K, int64_t* out_keys,
                     int32_t* out_triangles, mt_stream_t stream) {
  MT_REQUIRE(V >= 0 && F >= 0 && B >= 0 && S >= 0 && K >= 0 && layout);
  KeyLayout L{layout[0], layout[1], layout[2], layout[3], layout[4], layout[5], layout[6]};
  MT_REQUIRE(layout_ok(L));
  if (F == 0 || B == 0 || K == 0) return MT_OK;
  MT_REQUIRE(depth && faces && tile_min && tile_max && offsets && out_keys && out_triangles);
  MT_REQUIRE(S == 0 || shell_face_boundaries);
  keys_kernel<<<grid_stride_blocks((int64_t)B * F, 256), 256, 0, as_stream(stream)>>>(
      depth, V, faces, F, shell_face_boundaries, S, tile_min, tile_max, offsets, B, grid_width, cameras, L, K,
      reinterpret_cast<uint64_t*>(out_keys), out_triangles);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

static int64_t fused_chunks(int64_t items) { return (items + kFusedSubTile - 1) / kFusedSubTile; }

static size_t chunk_records(int64_t items, char* base, ChunkRecords* rec) {
  const int64_t chunks = fused_chunks(items);
  const int64_t groups = chunks > kOneCtaChunks ? (chunks + kScanGroup - 1) / kScanGroup : 0;
  size_t off = kFusedHeader;
  auto take = [&](size_t bytes) {
    char* p = base ? base + off : nullptr;
    off += round256(bytes);
    return p;
  };
  char* keys = take((size_t)chunks * sizeof(int64_t));
  char* counts = take((size_t)chunks * sizeof(int32_t));
  char* totals = take((size_t)groups * sizeof(int64_t));
  char* rect = take((size_t)items * sizeof(int4));
  char* depth = take((size_t)items * sizeof(float));
  char* place = take((size_t)items * sizeof(uint16_t));
  if (rec)
    *rec = ChunkRecords{reinterpret_cast<int64_t*>(keys),
                        reinterpret_cast<int32_t*>(counts),
                        groups ? reinterpret_cast<int64_t*>(totals) : nullptr,
                        reinterpret_cast<int4*>(rect),
                        reinterpret_cast<float*>(depth),
                        reinterpret_cast<uint16_t*>(place)};
  return off;
}

size_t mt_bound_and_generate_keys_workspace_bytes(int64_t items) {
  return chunk_records(items < 0 ? 0 : items, nullptr, nullptr);
}

int mt_bound_keys(const float* xy, const float* depth, int64_t V, const int32_t* faces, int64_t F,
                  const int32_t* num_faces, int32_t B, int32_t tile_h, int32_t tile_w, int32_t rows, int32_t cols,
                  const int64_t* cameras, float near_plane, int64_t* out_num_keys, void* workspace,
                  size_t workspace_bytes, mt_stream_t stream) {
  MT_REQUIRE(V >= 0 && F >= 0 && B >= 0 && tile_h > 0 && tile_w > 0 && rows >= 0 && cols >= 0);
  MT_REQUIRE(out_num_keys);
  const cudaStream_t s = as_stream(stream);
  const int64_t items = (int64_t)B * F;
  if (items == 0)
    return cudaMemsetAsync(out_num_keys, 0, sizeof(int64_t), s) == cudaSuccess ? MT_OK : MT_ERR_CUDA;
  MT_REQUIRE(xy && depth && faces && workspace);
  MT_REQUIRE((reinterpret_cast<uintptr_t>(xy) & 7) == 0);  // positions are read as float2
  MT_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 15) == 0);
  if (workspace_bytes < mt_bound_and_generate_keys_workspace_bytes(items)) return MT_ERR_WORKSPACE_TOO_SMALL;
  const int64_t chunks = fused_chunks(items);
  MT_REQUIRE(chunks < (int64_t)0x7fffffff);
  ChunkRecords rec;
  chunk_records(items, static_cast<char*>(workspace), &rec);
  const FusedArgs a{xy, depth, V, faces, F, num_faces, B, tile_h, tile_w, rows, cols, cameras, near_plane};
  chunk_bounds_kernel<<<(unsigned)chunks, kFusedThreads, 0, s>>>(a, rec);
  MT_CHECK_LAUNCH();
  const int64_t group = rec.groups ? kScanGroup : chunks;
  const unsigned groups = (unsigned)((chunks + group - 1) / group);
  if (rec.groups) {
    chunk_group_kernel<<<groups, kChunkScanThreads, 0, s>>>(rec.keys, chunks, rec.groups);
    MT_CHECK_LAUNCH();
  }
  chunk_scan_kernel<<<groups, kChunkScanThreads, 0, s>>>(rec.keys, chunks, group, rec.groups, out_num_keys);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_write_bounded_keys(int64_t F, const int32_t* shell_face_boundaries, int32_t S, int32_t B, int32_t cols,
                          const int64_t* cameras, const int32_t* layout, int64_t K, int64_t* out_keys,
                          int32_t* out_triangles, void* workspace, size_t workspace_bytes, mt_stream_t stream) {
  MT_REQUIRE(F >= 0 && B >= 0 && S >= 0 && K >= 0 && cols >= 0 && layout);
  KeyLayout L{layout[0], layout[1], layout[2], layout[3], layout[4], layout[5], layout[6]};
  MT_REQUIRE(layout_ok(L));
  const int64_t items = (int64_t)B * F;
  if (items == 0 || K == 0) return MT_OK;
  MT_REQUIRE(out_keys && out_triangles && workspace && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0);
  MT_REQUIRE(S == 0 || shell_face_boundaries);
  if (workspace_bytes < mt_bound_and_generate_keys_workspace_bytes(items)) return MT_ERR_WORKSPACE_TOO_SMALL;
  const int64_t chunks = fused_chunks(items);
  MT_REQUIRE(chunks < (int64_t)0x7fffffff);
  ChunkRecords rec;
  chunk_records(items, static_cast<char*>(workspace), &rec);
  FusedArgs a{};
  a.F = F;
  a.B = B;
  a.cols = cols;
  a.cameras = cameras;
  chunk_keys_kernel<<<(unsigned)chunks, kFusedThreads, 0, as_stream(stream)>>>(
      a, rec, shell_face_boundaries, S, L, K, reinterpret_cast<uint64_t*>(out_keys), out_triangles);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_bound_and_generate_keys(const float* xy, const float* depth, int64_t V, const int32_t* faces, int64_t F,
                               const int32_t* num_faces, const int32_t* shell_face_boundaries, int32_t S, int32_t B,
                               int32_t tile_h, int32_t tile_w, int32_t rows, int32_t cols, const int64_t* cameras,
                               float near_plane, const int32_t* layout, int64_t K, int64_t* out_keys,
                               int32_t* out_triangles, int64_t* out_num_keys, void* workspace, size_t workspace_bytes,
                               mt_stream_t stream) {
  MT_REQUIRE(V >= 0 && F >= 0 && B >= 0 && S >= 0 && K >= 0 && layout);
  KeyLayout L{layout[0], layout[1], layout[2], layout[3], layout[4], layout[5], layout[6]};
  MT_REQUIRE(layout_ok(L));
  MT_REQUIRE((int64_t)B * F == 0 || ((K == 0 || (out_keys && out_triangles)) && (S == 0 || shell_face_boundaries)));
  const int rc = mt_bound_keys(xy, depth, V, faces, F, num_faces, B, tile_h, tile_w, rows, cols, cameras, near_plane,
                               out_num_keys, workspace, workspace_bytes, stream);
  if (rc != MT_OK) return rc;
  return mt_write_bounded_keys(F, shell_face_boundaries, S, B, cols, cameras, layout, K, out_keys, out_triangles,
                               workspace, workspace_bytes, stream);
}

int mt_delineate_tiles(const int64_t* sorted_keys, int64_t K, const int64_t* num_keys, const int32_t* layout,
                       int32_t separate_shells, int32_t B, int32_t shell_dim, int64_t num_tiles,
                       int64_t* out_boundaries, mt_stream_t stream) {
  MT_REQUIRE(K >= 0 && B >= 0 && shell_dim >= 1 && num_tiles >= 0 && layout);
  KeyLayout L{layout[0], layout[1], layout[2], layout[3], layout[4], layout[5], layout[6]};
  MT_REQUIRE(layout_ok(L));
  const size_t bytes = (size_t)B * shell_dim * num_tiles * 2 * sizeof(int64_t);
  if (bytes == 0) return MT_OK;
  MT_REQUIRE(out_boundaries);
  if (cudaMemsetAsync(out_boundaries, 0, bytes, as_stream(stream)) != cudaSuccess) return MT_ERR_CUDA;
  if (K == 0) return MT_OK;
  MT_REQUIRE(sorted_keys);
  delineate_kernel<<<grid_stride_blocks(K, 256), 256, 0, as_stream(stream)>>>(
      reinterpret_cast<const uint64_t*>(sorted_keys), K, num_keys, L, separate_shells, B, shell_dim, num_tiles,
      out_boundaries);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

}  // extern "C"

// Coarse-to-fine subdivision, occupancy mesh and vertex de-duplication for
// sm_103a:
//   write_occupancy     triangle_extraction/write_occupancy.slang:1-20
//   upscale_occupancy   triangle_extraction/upscale_occupancy.slang:1-74
//   upscale_parameters  triangle_extraction/upscale_parameters.slang:1-198
//   get_occupancy_mesh  triangle_extraction/get_occupancy_mesh.slang:1-220
//   index_vertices      triangle_extraction/index_vertices.py:6-51 (keys,
//                       then the library's stable sort, then run heads)
//
// Packed occupancy: int32 [i, j, kp], bit b of word kp = voxel k = 32 kp + b.
// Floating-point results follow the reference source's operations in order
// (this unit is compiled without multiply-add contraction).

#include "lookback.cuh"  // warp_inclusive_sum
#include "mt_common.cuh"

namespace mt {
namespace {

constexpr int kThreads = 256;

// ---------------------------------------------------------------------------
// write_occupancy: set the bit of every triangle's voxel. Indices outside the
// grid are skipped (the reference writes them unchecked).
// ---------------------------------------------------------------------------
__global__ void write_occupancy_kernel(const int32_t* __restrict__ voxel_indices, int64_t n,
                                       int32_t* __restrict__ occupancy, int64_t words) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const int32_t v = voxel_indices[t];
    if (v < 0 || (int64_t)(v >> 5) >= words) continue;
    atomicOr(reinterpret_cast<unsigned int*>(occupancy) + (v >> 5), 1u << (v & 31));
  }
}

// ---------------------------------------------------------------------------
// upscale_occupancy: a new voxel (i, j, k) is occupied when any of its 8
// corners, mapped to the old grid by the unsigned integer arithmetic
//   old = ((new + side) * old_extent - side) / new_extent,
// lands in an occupied old voxel (optionally masked: old word & mask word).
//
// One thread per new word. The corner rows are (is, js) for the four
// (di, dj) sides, and since the new grid is at least as fine as the old one,
// the 32 bits x 2 sides of a new word map to old k in [ks_lo, ks_lo + 32]:
// at most two old words per row. So a word needs 8 loads (the reference
// samples 256), OR-ed across the four rows; the new bits follow from the runs
// of set old bits, of which a surface's band has one or two in a word.
// (Stepping both sides' old k along the 32 bits took every warp with a word of
// the band some 400 instructions: 78 us from 256^3 to 512^3; now 43 us.)
// ---------------------------------------------------------------------------
__global__ void upscale_occupancy_kernel(const int32_t* __restrict__ occ, const int32_t* __restrict__ mask,
                                         uint32_t I, uint32_t J, uint32_t KP, uint32_t I2, uint32_t J2,
                                         uint32_t KP2, int32_t* __restrict__ out) {
  const int64_t total = (int64_t)I2 * J2 * KP2;
  const uint32_t K = KP << 5, K2 = KP2 << 5;
  for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
    int i_, j_, kp_;
    word_position(w, (int)J2, (int)KP2, i_, j_, kp_);
    const uint32_t i = (uint32_t)i_, j = (uint32_t)j_, kp = (uint32_t)kp_;
    const uint32_t k_base = kp << 5;
    const uint32_t lo = ((k_base * K) / K2) >> 5;
    const bool has_hi = lo + 1 < KP;
    uint32_t a = 0, b = 0;
#pragma unroll
    for (uint32_t di = 0; di < 2; ++di) {
      const uint32_t is = ((i + di) * I - di) / I2;
#pragma unroll
      for (uint32_t dj = 0; dj < 2; ++dj) {
        const uint32_t js = ((j + dj) * J - dj) / J2;
        const int64_t row = ((int64_t)is * J + js) * KP;
        uint32_t wa = (uint32_t)__ldg(occ + row + lo);
        uint32_t wb = has_hi ? (uint32_t)__ldg(occ + row + lo + 1) : 0u;
        if (mask) {
          wa &= (uint32_t)__ldg(mask + row + lo);
          wb &= has_hi ? (uint32_t)__ldg(mask + row + lo + 1) : 0u;
        }
        a |= wa;
        b |= wb;
      }
    }
    uint32_t result = 0;
    // A run of old voxels [first, last] covers the new k with k1 >= first and
    // k0 <= last, where k0 = (k K) / K2 and k1 = ((k + 1) K - 1) / K2 are the
    // old k of its two sides: k from (first K2) / K to ((last + 1) K2 - 1) / K.
    for (uint64_t window = (uint64_t)b << 32 | a; window;) {
      const int at = __ffsll((long long)window) - 1;
      const int length = __ffsll((long long)~(window >> at)) - 1;  // -1: all 64 bits
      const int past = length < 0 ? 64 : at + length;
      window = past < 64 ? window >> past << past : 0ull;
      const uint32_t first = ((lo << 5) + at) * K2 / K, last = (((lo << 5) + past) * K2 - 1) / K;
      if (last < k_base || first > k_base + 31) continue;
      const uint32_t f = max(first, k_base) - k_base, l = min(last, k_base + 31) - k_base;
      result |= (0xffffffffu >> (31 - (l - f))) << f;
    }
    out[w] = (int32_t)result;
  }
}

// ---------------------------------------------------------------------------
// upscale_parameters: every new grid vertex samples the old vertices'
// signed distance and SH trilinearly, renormalising over the old vertices
// that exist. Vertex occupancy grids are [I+1, J+1, KP+1] words; offsets are
// the exclusive scan of their bit counts (one per word).
// ---------------------------------------------------------------------------
struct OldGrid {
  const int32_t* occ;      // old vertex occupancy
  const int32_t* offsets;  // old per-word vertex offsets
  const float* sdf;
  const float* sh;  // [C, sh_rows, 3]
  int64_t Vold, sh_rows;
  const int32_t* canonical;  // [Vold]: the row of sdf and sh that holds a vertex's values (NULL: its own)
  int I1, J1, KP1;  // old vertex occupancy dims
};

// The float `bytes` past a plane's start: 32 bits where a plane's bytes allow,
// so that a load adds one register to the plane's address.
template <typename Offset>
__device__ __forceinline__ float plane_load(const float* __restrict__ plane, Offset bytes) {
  return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(plane) + bytes));
}

// N planes of the flat channel that a lane holds: per plane, the sum over the
// present corners in corner order, times the normaliser. All 8 N loads are
// issued side by side (a branch around each corner's made them wait for one
// another). An absent corner reads a present one's row with weight zero: a
// zero added to a sum that starts at +0 changes nothing, as long as the row is
// finite. A sum that is not is formed again from the present corners alone.
template <int N, typename Offset>
__device__ __forceinline__ void upscale_planes(const float* __restrict__ src, int64_t src_plane, float* __restrict__ dst,
                                               int64_t dst_plane, uint32_t present, const Offset (&at)[8],
                                               const float (&wts)[8], float mult) {
  float x[N][8];
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int q = 0; q < 8; ++q) x[n][q] = plane_load(src + n * src_plane, at[q]);
  float acc[N];
  bool finite = true;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    acc[n] = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[n] += wts[q] * x[n][q];
    finite = finite && fabsf(acc[n]) < __int_as_float(0x7f800000);
  }
  if (!finite) {
#pragma unroll 1
    for (int n = 0; n < N; ++n) {
      float sum = 0.0f;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if ((present >> q) & 1u) sum += wts[q] * plane_load(src + n * src_plane, at[q]);
      dst[n * dst_plane] = sum * mult;
    }
    return;
  }
#pragma unroll
  for (int n = 0; n < N; ++n) dst[n * dst_plane] = acc[n] * mult;
}

// What the lanes of a warp share about the 32 vertices that they deal with.
struct DealtVertices {
  int32_t id[8][32];  // row of each corner's values, -1 = absent
  float wt[8][32], mult[32];
};
constexpr int kUpscaleWarps = 8, kUpscaleThreads = 32 * kUpscaleWarps;

// The vertices of the old grid's row (i, j) at k and k + 1, -1 where absent
// (read_vertex, upscale_parameters.slang:9-53; no index is negative here).
__device__ __forceinline__ void old_vertex_pair(const OldGrid& g, int i, int j, int k, int32_t& v0, int32_t& v1) {
  v0 = v1 = -1;
  const int kp = k >> 5, bit = k & 31;
  if ((unsigned)i >= (unsigned)g.I1 || (unsigned)j >= (unsigned)g.J1 || kp >= g.KP1) return;
  const int64_t word = ((int64_t)i * g.J1 + j) * g.KP1 + kp;
  const uint32_t chunk = (uint32_t)__ldg(g.occ + word);
  const uint32_t here = chunk >> bit;
  const int32_t base = __ldg(g.offsets + word);
  const int32_t at = base + __popc(chunk & ((1u << bit) - 1u));  // of the first vertex at or after bit
  if (here & 1u) v0 = at;
  if (bit < 31) {
    if (here & 2u) v1 = at + (int32_t)(here & 1u);
  } else if (kp + 1 < g.KP1 && ((uint32_t)__ldg(g.occ + word + 1) & 1u)) {
    v1 = __ldg(g.offsets + word + 1);
  }
}

// A CTA takes 256 consecutive words of the new vertex grid, one to a thread,
// and deals their vertices out to its warps 32 at a time: lane r of a batch
// takes the batch's r-th vertex, whose word is found in the running bit counts
// and whose bit by a popcount select. Offsets are an exclusive scan in word
// order, so that vertex is offset[first word] + r: every lane is busy and every
// [C, V, 3] row that a warp stores is contiguous.
//
// The SH sums go by the row's floats, not by vertices: a lane takes floats
// lane, lane + 32 and lane + 64 of the 96 that 32 vertices have in a plane
// (vertex and channel stay the same from plane to plane), so that a warp's
// load or store covers 128 consecutive bytes of new vertices. With a lane to
// a vertex every load and store strode over 12 B, and a branch around every
// corner made four loads wait for the next four: 687 us from 256^3 to 512^3
// (424 k to 2.93 M vertices, C = 16), and 119 us more for the copy of the
// canonical rows; now 465 us. Bound by its instructions (8 loads, two
// operations each, per output float).
template <typename Offset>
__global__ void __launch_bounds__(kUpscaleThreads, 3)
    upscale_parameters_kernel(OldGrid g, int C, const int32_t* __restrict__ new_occ,
                              const int32_t* __restrict__ new_offsets, int I1n, int J1n, int KP1n, int64_t Vnew,
                              float* __restrict__ new_sdf, float* __restrict__ new_sh) {
  __shared__ DealtVertices dealt[kUpscaleWarps];
  __shared__ uint32_t chunks[kUpscaleThreads];
  __shared__ int ends[kUpscaleThreads];  // inclusive running bit counts
  __shared__ int warp_counts[kUpscaleWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  DealtVertices& sh = dealt[warp];
  const int64_t total = (int64_t)I1n * J1n * KP1n;
  const int64_t base = blockIdx.x * (int64_t)kUpscaleThreads, mine = base + threadIdx.x;
  const uint32_t my_chunk = mine < total ? (uint32_t)__ldg(new_occ + mine) : 0u;
  const int incl = warp_inclusive_sum(__popc(my_chunk));
  if (lane == 31) warp_counts[warp] = incl;
  chunks[threadIdx.x] = my_chunk;
  __syncthreads();
  int before_warp = 0, span = 0;
#pragma unroll
  for (int w = 0; w < kUpscaleWarps; ++w) {
    before_warp += w < warp ? warp_counts[w] : 0;
    span += warp_counts[w];
  }
  if (span == 0) return;  // the whole CTA
  ends[threadIdx.x] = before_warp + incl;
  __syncthreads();
  // New grid position scale (upscale_parameters.slang:141-160).
  const float inv_i_max = 1.0f / (float)(I1n - 1);
  const float inv_j_max = 1.0f / (float)(J1n - 1);
  const float inv_k_max = 1.0f / (float)(32 * (KP1n - 1));
  // Old grid scale (sample_trilinear, :63-65).
  const float sx = (float)((g.KP1 - 1) * 32), sy = (float)(g.J1 - 1), sz = (float)(g.I1 - 1);
  const int64_t src_plane = 3 * g.sh_rows, dst_plane = 3 * Vnew;
  const int64_t first_vertex = __ldg(new_offsets + base);
  for (int start = 32 * warp; start < span; start += kUpscaleThreads) {
    const int r = start + lane;
    const int64_t vi = first_vertex + r;
    if (r < span && vi >= 0 && vi < Vnew) {
      int src = 0;  // the smallest word with ends[src] > r
#pragma unroll
      for (int step = kUpscaleThreads / 2; step > 0; step >>= 1)
        if (ends[src + step - 1] <= r) src += step;
      const int bit = select_bit(chunks[src], r - (src ? ends[src - 1] : 0));
      int i, j, kp;
      word_position(base + src, J1n, KP1n, i, j, kp);
      const int k = 32 * kp + bit;
      const float x = (float)k * inv_k_max, y = (float)j * inv_j_max, z = (float)i * inv_i_max;
      const float xu = x * sx, yu = y * sy, zu = z * sz;
      const int oi = (int)zu, oj = (int)yu, ok = (int)xu;
      // fmod(x, 1) of x >= 0, which the difference gives exactly.
      const float ti = zu - truncf(zu), tj = yu - truncf(yu), tk = xu - truncf(xu);
      int32_t ids[8];
#pragma unroll
      for (int q = 0; q < 8; q += 2) old_vertex_pair(g, oi + (q >> 2), oj + ((q >> 1) & 1), ok, ids[q], ids[q + 1]);
      float value[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (ids[q] >= g.Vold) ids[q] = -1;
        if (ids[q] >= 0 && g.canonical) ids[q] = __ldg(g.canonical + ids[q]);
        value[q] = ids[q] >= 0 ? __ldg(g.sdf + ids[q]) : 0.0f;
        sh.id[q][lane] = ids[q];
      }
      float den = 0.0f, d = 0.0f;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float wgt =
            ((q >> 2) == 0 ? 1.0f - ti : ti) * (((q >> 1) & 1) == 0 ? 1.0f - tj : tj) * ((q & 1) == 0 ? 1.0f - tk : tk);
        sh.wt[q][lane] = wgt;
        if (ids[q] >= 0) {
          d += wgt * value[q];
          den += wgt;
        }
      }
      const float mult = 1.0f / den;
      sh.mult[lane] = mult;
      new_sdf[vi] = d * mult;
    }
    __syncwarp();
    const int count = min(32, span - start);
#pragma unroll 1
    for (int f = lane; f < 3 * count; f += 32) {
      const int v = f / 3, ch = f - 3 * v;
      const int64_t row = first_vertex + start + v;
      if (row < 0 || row >= Vnew) continue;
      Offset at[8];
      float wts[8];
      uint32_t present = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int32_t id = sh.id[q][v];
        present |= (id >= 0 ? 1u : 0u) << q;
        at[q] = (Offset)12 * (Offset)id + (Offset)(4 * ch);
        wts[q] = sh.wt[q][v];
      }
      const float mult = sh.mult[v];
      float* dst = new_sh + 3 * row + ch;
      if (present == 0u) {
        for (int c = 0; c < C; ++c) dst[c * dst_plane] = 0.0f * mult;
        continue;
      }
      const Offset any = (Offset)12 * (Offset)sh.id[__ffs(present) - 1][v] + (Offset)(4 * ch);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (!((present >> q) & 1u)) {
          at[q] = any;
          wts[q] = 0.0f;
        }
      int c = 0;
#pragma unroll 1
      for (; c + 4 <= C; c += 4, dst += 4 * dst_plane)
        upscale_planes<4>(g.sh + c * src_plane, src_plane, dst, dst_plane, present, at, wts, mult);
#pragma unroll 1
      for (; c < C; ++c, dst += dst_plane)
        upscale_planes<1>(g.sh + c * src_plane, src_plane, dst, dst_plane, present, at, wts, mult);
    }
    __syncwarp();  // the next 32 vertices overwrite the shared ones
  }
}

// ---------------------------------------------------------------------------
// get_occupancy_mesh: two triangles per boundary face between occupied and
// free voxels; each (i, j, kp) entry of the [I+1, J+1, KP+1] grid owns the
// faces on its lower i, j and k sides.
// ---------------------------------------------------------------------------
struct Neighbourhood {
  uint32_t here, minus_i, minus_j;
  bool minus_k;
};

__device__ __forceinline__ Neighbourhood neighbourhood(const int32_t* __restrict__ occ, int I, int J, int KP, int i,
                                                       int j, int kp) {
  const bool il = i == I, jl = j == J, kl = kp == KP;
  auto at = [&](int a, int b, int c) { return (uint32_t)__ldg(occ + ((int64_t)a * J + b) * KP + c); };
  Neighbourhood n;
  n.here = (il || jl || kl) ? 0u : at(i, j, kp);
  n.minus_i = (jl || kl || i == 0) ? 0u : at(i - 1, j, kp);
  n.minus_j = (il || kl || j == 0) ? 0u : at(i, j - 1, kp);
  n.minus_k = (il || jl || kp == 0) ? false : ((at(i, j, kp - 1) & 0x80000000u) != 0);
  return n;
}

// Bits with a face on the lower k side: where a bit differs from the one
// before it (bit 0 against bit 31 of the previous word).
__device__ __forceinline__ uint32_t k_faces(const Neighbourhood& n) {
  return n.here ^ ((n.here << 1) | (n.minus_k ? 1u : 0u));
}

__global__ void count_mesh_triangles_kernel(const int32_t* __restrict__ occ, int I, int J, int KP,
                                            int32_t* __restrict__ counts) {
  const int64_t total = (int64_t)(I + 1) * (J + 1) * (KP + 1);
  for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
    const int kp = (int)(w % (KP + 1)), j = (int)((w / (KP + 1)) % (J + 1)), i = (int)(w / ((int64_t)(KP + 1) * (J + 1)));
    const Neighbourhood n = neighbourhood(occ, I, J, KP, i, j, kp);
    counts[w] = 2 * (__popc(n.here ^ n.minus_i) + __popc(n.here ^ n.minus_j) + __popc(k_faces(n)));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) counts[total] = 0;
}

// create_face (get_occupancy_mesh.slang:56-120): the face of `axis` at the
// entry's lower side, two triangles wound by `upper`, each corner written
// as (component 2, 1, 0) of its (i, j, k)-ordered coordinates.
__device__ __forceinline__ void write_face(int64_t index, int i, int j, int k, const int (&ijk_max)[3], int axis,
                                           bool upper, float* __restrict__ verts, float* __restrict__ tri_colors,
                                           const float* __restrict__ colors) {
  const int ijk[3] = {i, j, k};
  const int a0 = (axis + 1) % 3, a1 = (axis + 2) % 3;
  float v00[3], v01[3], v10[3], v11[3];
  const float plane = (float)ijk[axis] / (float)ijk_max[axis];
  v00[axis] = v01[axis] = v10[axis] = v11[axis] = plane;
  const float v0x = (float)ijk[a0] / (float)ijk_max[a0];
  const float v1x = (float)(ijk[a0] + 1) / (float)ijk_max[a0];
  const float vx0 = (float)ijk[a1] / (float)ijk_max[a1];
  const float vx1 = (float)(ijk[a1] + 1) / (float)ijk_max[a1];
  v00[a0] = v0x;
  v00[a1] = vx0;
  v01[a0] = v0x;
  v01[a1] = vx1;
  v10[a0] = v1x;
  v10[a1] = vx0;
  v11[a0] = v1x;
  v11[a1] = vx1;
  const float* col = colors + (axis * 2 + (upper ? 1 : 0)) * 3;
  const float* tris[2][3] = {{v00, upper ? v01 : v10, upper ? v10 : v01}, {v11, upper ? v10 : v01, upper ? v01 : v10}};
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    float* out = verts + (index + t) * 9;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      out[3 * c + 0] = tris[t][c][2];
      out[3 * c + 1] = tris[t][c][1];
      out[3 * c + 2] = tris[t][c][0];
    }
    float* oc = tri_colors + (index + t) * 3;
    oc[0] = col[0];
    oc[1] = col[1];
    oc[2] = col[2];
  }
}

__global__ void create_mesh_triangles_kernel(const int32_t* __restrict__ occ, int I, int J, int KP,
                                             const int32_t* __restrict__ offsets, int64_t T,
                                             const float* __restrict__ colors, float* __restrict__ verts,
                                             float* __restrict__ tri_colors) {
  const int64_t total = (int64_t)(I + 1) * (J + 1) * (KP + 1);
  const int ijk_max[3] = {I, J, KP * 32};
  for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
    const int kp = (int)(w % (KP + 1)), j = (int)((w / (KP + 1)) % (J + 1)), i = (int)(w / ((int64_t)(KP + 1) * (J + 1)));
    const Neighbourhood n = neighbourhood(occ, I, J, KP, i, j, kp);
    const uint32_t fi = n.here ^ n.minus_i, fj = n.here ^ n.minus_j, fk = k_faces(n);
    uint32_t any = fi | fj | fk;
    int64_t index = offsets[w];
    while (any) {
      const int bit = __ffs(any) - 1;
      any &= any - 1;
      const bool h = (n.here >> bit) & 1u;
      const int k = kp * 32 + bit;
      // Faces with normals along i, then j, then k (get_occupancy_mesh.slang:168-210).
      if (((fi >> bit) & 1u) && index + 2 <= T) {
        write_face(index, i, j, k, ijk_max, 0, h, verts, tri_colors, colors);
        index += 2;
      }
      if (((fj >> bit) & 1u) && index + 2 <= T) {
        write_face(index, i, j, k, ijk_max, 1, h, verts, tri_colors, colors);
        index += 2;
      }
      if (((fk >> bit) & 1u) && index + 2 <= T) {
        write_face(index, i, j, k, ijk_max, 2, h, verts, tri_colors, colors);
        index += 2;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// index_vertices (index_vertices.py:6-51).
//
// Quantization follows torch's CUDA kernels for round(points / tol): a
// division by a host scalar is a multiplication by its float reciprocal,
// then round half to even, then a truncating conversion to int64.
// ---------------------------------------------------------------------------
__global__ void quantize_points_kernel(const float* __restrict__ points, int64_t n, float inv_tol,
                                       int64_t* __restrict__ q, unsigned long long* __restrict__ max_abs) {
  unsigned long long m = 0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const float r = rintf(__fmul_rn(points[e], inv_tol));
    const int64_t v = (int64_t)r;
    q[e] = v;
    const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    m = a > m ? a : m;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, m, o);
    m = other > m ? other : m;
  }
  if ((threadIdx.x & 31) == 0 && m) atomicMax(max_abs, m);
}

// keys = (x << 2 shift) | (y << shift) | z with two's complement shifts,
// values = 0 .. V-1 (unless NULL).
__global__ void pack_point_keys_kernel(const int64_t* __restrict__ q, int64_t V, int shift,
                                       int64_t* __restrict__ keys, int32_t* __restrict__ values) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t x = (uint64_t)q[3 * v + 0], y = (uint64_t)q[3 * v + 1], z = (uint64_t)q[3 * v + 2];
    keys[v] = (int64_t)((x << (2 * shift)) | (y << shift) | z);
    if (values) values[v] = (int32_t)v;
  }
}

__global__ void iota_kernel(int64_t n, int32_t* __restrict__ values) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
    values[v] = (int32_t)v;
}

// Every sorted position p maps its original index to the original index at
// the start of its run of equal keys. The sort is stable over 0..n-1, so the
// run starts at the smallest original index: the first seen. The run start
// is the lower bound of the key (sorted in signed order) in [0, p].
__global__ void run_heads_kernel(const int64_t* __restrict__ sorted_keys, const int32_t* __restrict__ order,
                                 int64_t n, int32_t* __restrict__ out) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t key = sorted_keys[p];
    int64_t start = p;
    if (p > 0 && sorted_keys[p - 1] == key) {
      int64_t lo = 0, hi = p - 1;  // sorted_keys[hi] == key
      while (lo < hi) {
        const int64_t mid = lo + ((hi - lo) >> 1);
        if (sorted_keys[mid] < key) lo = mid + 1;
        else hi = mid;
      }
      start = lo;
    }
    const int32_t dst = order[p];
    if (dst >= 0 && dst < n) out[dst] = order[start];
  }
}

// ---------------------------------------------------------------------------
// First index of every key by an open-addressing table (linear probing, at most
// half full, so a probe meets its key or an empty slot): each key claims a slot
// and the slot keeps its least index; then every key looks its slot up. The
// same result as the stable sort followed by run heads, which moves every key
// eight times: 114 us for 424,000 points, this 30. Bound by the latency of
// the table's scattered reads and atomics.
//
// Table: [slots] keys, then [slots + 1] indices, all bits set where empty; the
// last index stands for the key whose bits are all set.
// ---------------------------------------------------------------------------
constexpr unsigned long long kEmptyKey = ~0ull;

// MurmurHash3's 64-bit finalizer (Appleby).
__device__ __forceinline__ uint64_t mix_key(uint64_t x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ull;
  return x ^ (x >> 33);
}

__global__ void claim_keys_kernel(const int64_t* __restrict__ keys, int64_t n, unsigned long long* table,
                                  uint32_t* first, uint64_t mask) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long key = (unsigned long long)__ldg(keys + v);
    uint64_t slot = mask + 1;
    if (key != kEmptyKey) {
      slot = mix_key(key) & mask;
      for (uint64_t probes = 0; probes <= mask; ++probes, slot = (slot + 1) & mask) {
        // Read first: a key that many points share is claimed by few.
        unsigned long long there = *(volatile unsigned long long*)(table + slot);
        if (there == kEmptyKey) there = atomicCAS(table + slot, kEmptyKey, key);
        if (there == kEmptyKey || there == key) break;
      }
    }
    if (*(volatile uint32_t*)(first + slot) > (uint32_t)v) atomicMin(first + slot, (uint32_t)v);
  }
}

__global__ void look_up_keys_kernel(const int64_t* __restrict__ keys, int64_t n,
                                    const unsigned long long* __restrict__ table, const uint32_t* __restrict__ first,
                                    uint64_t mask, int32_t* __restrict__ out) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long key = (unsigned long long)__ldg(keys + v);
    uint64_t slot = mask + 1;
    if (key != kEmptyKey) {
      slot = mix_key(key) & mask;
      for (uint64_t probes = 0; probes <= mask; ++probes, slot = (slot + 1) & mask)
        if (__ldg(table + slot) == key) break;
    }
    out[v] = (int32_t)__ldg(first + slot);
  }
}

int64_t key_slots(int64_t n) {
  int64_t slots = 64;
  while (slots < 2 * n) slots <<= 1;
  return slots;
}

}  // namespace
}  // namespace mt

using namespace mt;

extern "C" {

int mt_write_occupancy(const int32_t* voxel_indices, int64_t n, int32_t* occupancy, int64_t words,
                       mt_stream_t stream) {
  MT_REQUIRE(n >= 0 && words >= 0);
  if (n == 0 || words == 0) return MT_OK;
  MT_REQUIRE(voxel_indices && occupancy);
  write_occupancy_kernel<<<grid_stride_blocks(n, kThreads), kThreads, 0, as_stream(stream)>>>(voxel_indices, n,
                                                                                            occupancy, words);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_upscale_occupancy(const int32_t* occupancy, const int32_t* mask, int32_t I, int32_t J, int32_t KP,
                         int32_t I2, int32_t J2, int32_t KP2, int32_t* out, mt_stream_t stream) {
  MT_REQUIRE(I > 0 && J > 0 && KP > 0 && I2 >= I && J2 >= J && KP2 >= KP);
  // The reference's corner arithmetic is 32-bit unsigned: keep it exact.
  MT_REQUIRE((uint64_t)(I2 + 1) * (uint64_t)I <= 0xffffffffull && (uint64_t)(J2 + 1) * (uint64_t)J <= 0xffffffffull &&
             (uint64_t)(KP2 + 1) * 32ull * (uint64_t)KP * 32ull <= 0xffffffffull);
  MT_REQUIRE(occupancy && out);
  const int64_t total = (int64_t)I2 * J2 * KP2;
  upscale_occupancy_kernel<<<grid_stride_blocks(total, kThreads, 128), kThreads, 0, as_stream(stream)>>>(
      occupancy, mask, (uint32_t)I, (uint32_t)J, (uint32_t)KP, (uint32_t)I2, (uint32_t)J2, (uint32_t)KP2, out);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_upscale_canonical_parameters(const int32_t* old_vertex_occupancy, const int32_t* old_vertex_offsets,
                                    const float* old_signed_distances, const float* old_spherical_harmonics,
                                    const int32_t* canonical, int64_t sh_rows, int32_t C, int64_t Vold, int32_t I1,
                                    int32_t J1, int32_t KP1, const int32_t* new_vertex_occupancy,
                                    const int32_t* new_vertex_offsets, int32_t I1n, int32_t J1n, int32_t KP1n,
                                    int64_t Vnew, float* new_signed_distances, float* new_spherical_harmonics,
                                    mt_stream_t stream) {
  MT_REQUIRE(C >= 1 && Vold >= 0 && Vnew >= 0 && I1 >= 2 && J1 >= 2 && KP1 >= 2 && I1n >= 2 && J1n >= 2 &&
             KP1n >= 2);
  if (Vnew == 0) return MT_OK;
  MT_REQUIRE(old_vertex_occupancy && old_vertex_offsets && new_vertex_occupancy && new_vertex_offsets &&
             new_signed_distances && new_spherical_harmonics);
  MT_REQUIRE(Vold == 0 || (old_signed_distances && old_spherical_harmonics));
  MT_REQUIRE(sh_rows >= 0 && (canonical || sh_rows >= Vold));
  OldGrid g{old_vertex_occupancy, old_vertex_offsets, old_signed_distances, old_spherical_harmonics, Vold, sh_rows,
            canonical, I1, J1, KP1};
  const int64_t total = (int64_t)I1n * J1n * KP1n;
  const int64_t blocks64 = (total + kUpscaleThreads - 1) / kUpscaleThreads;  // a thread to a word
  MT_REQUIRE(blocks64 < ((int64_t)1 << 31));
  const unsigned blocks = (unsigned)blocks64;
  if (12 * sh_rows < ((int64_t)1 << 32))
    upscale_parameters_kernel<uint32_t><<<blocks, kUpscaleThreads, 0, as_stream(stream)>>>(
        g, C, new_vertex_occupancy, new_vertex_offsets, I1n, J1n, KP1n, Vnew, new_signed_distances,
        new_spherical_harmonics);
  else
    upscale_parameters_kernel<int64_t><<<blocks, kUpscaleThreads, 0, as_stream(stream)>>>(
        g, C, new_vertex_occupancy, new_vertex_offsets, I1n, J1n, KP1n, Vnew, new_signed_distances,
        new_spherical_harmonics);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_upscale_parameters(const int32_t* old_vertex_occupancy, const int32_t* old_vertex_offsets,
                          const float* old_signed_distances, const float* old_spherical_harmonics, int32_t C,
                          int64_t Vold, int32_t I1, int32_t J1, int32_t KP1, const int32_t* new_vertex_occupancy,
                          const int32_t* new_vertex_offsets, int32_t I1n, int32_t J1n, int32_t KP1n, int64_t Vnew,
                          float* new_signed_distances, float* new_spherical_harmonics, mt_stream_t stream) {
  return mt_upscale_canonical_parameters(old_vertex_occupancy, old_vertex_offsets, old_signed_distances,
                                         old_spherical_harmonics, nullptr, Vold, C, Vold, I1, J1, KP1,
                                         new_vertex_occupancy, new_vertex_offsets, I1n, J1n, KP1n, Vnew,
                                         new_signed_distances, new_spherical_harmonics, stream);
}

int mt_count_occupancy_mesh_triangles(const int32_t* occupancy, int32_t I, int32_t J, int32_t KP, int32_t* counts,
                                      mt_stream_t stream) {
  MT_REQUIRE(I >= 0 && J >= 0 && KP >= 0 && counts);
  MT_REQUIRE((I == 0 || J == 0 || KP == 0) || occupancy);
  const int64_t total = (int64_t)(I + 1) * (J + 1) * (KP + 1);
  count_mesh_triangles_kernel<<<grid_stride_blocks(total, kThreads), kThreads, 0, as_stream(stream)>>>(
      occupancy, I, J, KP, counts);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_create_occupancy_mesh_triangles(const int32_t* occupancy, int32_t I, int32_t J, int32_t KP,
                                       const int32_t* offsets, int64_t T, const float* colors, float* vertices,
                                       float* triangle_colors, mt_stream_t stream) {
  MT_REQUIRE(I >= 0 && J >= 0 && KP >= 0 && T >= 0);
  if (T == 0) return MT_OK;
  MT_REQUIRE(occupancy && offsets && colors && vertices && triangle_colors);
  const int64_t total = (int64_t)(I + 1) * (J + 1) * (KP + 1);
  create_mesh_triangles_kernel<<<grid_stride_blocks(total, 128), 128, 0, as_stream(stream)>>>(
      occupancy, I, J, KP, offsets, T, colors, vertices, triangle_colors);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_quantize_points(const float* points, int64_t V, float inv_tol, int64_t* quantized, uint64_t* max_abs,
                       mt_stream_t stream) {
  MT_REQUIRE(V >= 0 && max_abs);
  cudaStream_t s = as_stream(stream);
  if (cudaMemsetAsync(max_abs, 0, sizeof(uint64_t), s) != cudaSuccess) return MT_ERR_CUDA;
  if (V == 0) return MT_OK;
  MT_REQUIRE(points && quantized);
  quantize_points_kernel<<<grid_stride_blocks(3 * V, kThreads), kThreads, 0, s>>>(
      points, 3 * V, inv_tol, quantized, reinterpret_cast<unsigned long long*>(max_abs));
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_pack_point_keys(const int64_t* quantized, int64_t V, int32_t shift, int64_t* keys, int32_t* values,
                       mt_stream_t stream) {
  MT_REQUIRE(V >= 0 && V <= 0x7fffffffll && shift >= 0 && shift <= 21);
  if (V == 0) return MT_OK;
  MT_REQUIRE(quantized && keys);
  pack_point_keys_kernel<<<grid_stride_blocks(V, kThreads), kThreads, 0, as_stream(stream)>>>(quantized, V, shift,
                                                                                            keys, values);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_iota_i32(int64_t n, int32_t* values, mt_stream_t stream) {
  MT_REQUIRE(n >= 0 && n <= 0x7fffffffll);
  if (n == 0) return MT_OK;
  MT_REQUIRE(values);
  iota_kernel<<<grid_stride_blocks(n, kThreads), kThreads, 0, as_stream(stream)>>>(n, values);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

size_t mt_index_keys_workspace_bytes(int64_t n) {
  if (n <= 0) return 0;
  return (size_t)key_slots(n) * 12 + 16;
}

int mt_index_keys(const int64_t* keys, int64_t n, int32_t* out, void* workspace, size_t workspace_bytes,
                  mt_stream_t stream) {
  MT_REQUIRE(n >= 0 && n <= 0x7fffffff);
  if (n == 0) return MT_OK;
  MT_REQUIRE(keys && out && workspace && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0);
  const size_t bytes = mt_index_keys_workspace_bytes(n);
  if (workspace_bytes < bytes) return MT_ERR_WORKSPACE_TOO_SMALL;
  const int64_t slots = key_slots(n);
  unsigned long long* table = static_cast<unsigned long long*>(workspace);
  uint32_t* first = reinterpret_cast<uint32_t*>(table + slots);
  const cudaStream_t s = as_stream(stream);
  if (cudaMemsetAsync(workspace, 0xff, bytes, s) != cudaSuccess) return MT_ERR_CUDA;
  claim_keys_kernel<<<grid_stride_blocks(n, kThreads, 32), kThreads, 0, s>>>(keys, n, table, first, slots - 1);
  MT_CHECK_LAUNCH();
  look_up_keys_kernel<<<grid_stride_blocks(n, kThreads, 32), kThreads, 0, s>>>(keys, n, table, first, slots - 1, out);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_index_sorted_runs(const int64_t* sorted_keys, const int32_t* order, int64_t n, int32_t* out,
                         mt_stream_t stream) {
  MT_REQUIRE(n >= 0 && n <= 0x7fffffffll);
  if (n == 0) return MT_OK;
  MT_REQUIRE(sorted_keys && order && out);
  run_heads_kernel<<<grid_stride_blocks(n, kThreads), kThreads, 0, as_stream(stream)>>>(sorted_keys, order, n, out);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

}  // extern "C"

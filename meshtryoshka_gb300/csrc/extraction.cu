// Sparse-voxel extraction and per-step marching cubes for sm_103a.
//
// Voxel topology (extract_voxels) follows triangle_extraction/
// compute_vertex_occupancy.slang, count_occupancy.slang, create_voxels.slang
// and dilate_occupancy.slang; per-step tessellation follows
// count_triangle_vertices.slang, create_triangle_vertices.slang,
// count_triangle_faces.slang and create_triangle_faces.slang.
//
// Layout choices: every per-word kernel indexes the packed k axis fastest so
// a warp reads consecutive words; create_voxels deals the vertices of 32 words
// out to a warp's lanes, where the reference walks a word's bits in a loop; all
// [*, G] / [*, Nv] tables are read one row at a time so every row read is
// coalesced.
//
// For the captured training step the per-vertex SH rows can be skipped: the
// grid-SH colour kernels evaluate vertex colours straight from the grid
// coefficients (evaluate_spherical_harmonics.slang with the interpolation of
// create_triangle_vertices.slang) and send the SH gradient straight back to
// the grid through the per-grid-vertex contribution list, with the same bits
// as the row path.

#include <type_traits>

#include "lookback.cuh"  // warp_inclusive_sum
#include "mc_tables.h"
#include "mt_common.cuh"
#include "sh.cuh"

namespace mt {
namespace {

__constant__ uint8_t c_mc_count[256] = {MT_MC_CASE_COUNT_VALUES};
__constant__ uint64_t c_mc_edges[256] = {MT_MC_CASE_EDGES_VALUES};
__constant__ int8_t c_mc_owner[12] = {MT_MC_EDGE_OWNER_VALUES};
__constant__ uint8_t c_mc_axis[12] = {MT_MC_EDGE_AXIS_VALUES};

// ---------------------------------------------------------------------------
// compute_vertex_occupancy.slang:9-68, and where xcounts is given the voxel
// counts of count_occupancy.slang too.
//
// A warp takes 31 consecutive words of the vertex grid: a lane ORs the word's
// four voxel rows, and takes the bit before its first one from the lane below
// (lane 0 holds the word before). Bound by its index arithmetic: with both
// words of every row read per lane, and the voxels counted by a kernel of
// their own, 31 + 16 us at 512^3, now 27.
// ---------------------------------------------------------------------------
constexpr int kOccupancyWords = 31;

__global__ void vertex_occupancy_kernel(const int32_t* __restrict__ occ, int I, int J, int KP,
                                        int32_t* __restrict__ vocc, int32_t* __restrict__ vcounts,
                                        int32_t* __restrict__ xcounts) {
  const int64_t total = (int64_t)(I + 1) * (J + 1) * (KP + 1);
  const int lane = threadIdx.x & 31;
  const int64_t first_warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t slab = (int64_t)J * KP;
  for (int64_t base = first_warp * kOccupancyWords; base < total; base += warps * kOccupancyWords) {
    const int64_t w = base + lane - 1;
    uint32_t any = 0, own = 0;
    int i = 0, j = 0, kp = 0;
    if (w >= 0 && w < total) {
      word_position(w, J + 1, KP + 1, i, j, kp);
      if (kp < KP) {
        const int32_t* p = occ + i * slab + (int64_t)j * KP + kp;
        if (i < I && j < J) own = (uint32_t)__ldg(p);
        if (i < I && j > 0) any = (uint32_t)__ldg(p - KP);
        if (i > 0 && j < J) any |= (uint32_t)__ldg(p - slab);
        if (i > 0 && j > 0) any |= (uint32_t)__ldg(p - slab - KP);
        any |= own;
      }
    }
    const uint32_t before = __shfl_up_sync(0xffffffffu, any, 1);
    if (lane == 0 || w >= total) continue;
    const uint32_t result = any | (any << 1) | (kp > 0 ? before >> 31 : 0u);
    vocc[w] = (int32_t)result;
    vcounts[w] = __popc(result);
    if (xcounts) xcounts[w] = __popc(own);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    vcounts[total] = 0;
    if (xcounts) xcounts[total] = 0;
  }
}

// count_occupancy.slang:3-20 plus the zero fill of count_occupancy.py:30.
__global__ void count_occupancy_kernel(const int32_t* __restrict__ occ, int I, int J, int KP,
                                       int32_t* __restrict__ counts) {
  const int64_t total = (int64_t)(I + 1) * (J + 1) * (KP + 1);
  for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < total;
       w += (int64_t)gridDim.x * blockDim.x) {
    int i, j, kp;
    word_position(w, J + 1, KP + 1, i, j, kp);
    int c = 0;
    if (i < I && j < J && kp < KP) c = __popc((uint32_t)occ[((int64_t)i * J + j) * KP + kp]);
    counts[w] = c;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) counts[total] = 0;
}

// ---------------------------------------------------------------------------
// create_voxels.slang:3-276.
//
// A warp takes 32 consecutive words of the vertex grid. Each lane reads its
// own word, and where that holds a vertex the occupancy words and offsets of
// the four rows (i, j), (i, j + 1), (i + 1, j), (i + 1, j + 1), into the
// warp's shared memory; then the span's vertices are dealt out 32 at a time
// (lane r takes the r-th one). Offsets are exclusive scans in word order, so
// consecutive lanes write consecutive entries of every table.
//
// Bound by its writes (12 B a vertex, 16 B a lower corner, 48 B a voxel). A
// warp to each word, lane = bit, waited out the loads of one word after
// another, 460 words to a warp at 512^3 and nine in ten of them empty, and
// ran with the few lanes of the bits that a word has: 766 us at 512^3 (the
// large benchmark scene's band; extract_voxels 967 us). With this the call
// takes 310 us.
// ---------------------------------------------------------------------------
struct VoxelGrid {
  const int32_t* occ;   // [I, J, KP]
  const int32_t* xoff;  // [I+1, J+1, KP+1] voxel offsets
  const int32_t* vocc;  // [I+1, J+1, KP+1]
  const int32_t* voff;  // [I+1, J+1, KP+1] vertex offsets
  int I, J, KP;
  int64_t Nv;

  // Voxel occupancy word; 0 outside the voxel grid.
  __device__ __forceinline__ uint32_t vx(int i, int j, int kp) const {
    if (i >= I || j >= J || kp >= KP) return 0u;
    return (uint32_t)__ldg(occ + ((int64_t)i * J + j) * KP + kp);
  }
};

constexpr int kVoxelWarps = 8;  // warps per CTA: 21 KB of shared memory

// A span's words: the four rows' vertex and voxel occupancy and offsets, what
// bit 31 needs of the next words, and the word's position.
struct SpanWords {
  uint32_t vo[4][32], vx[4][32];
  int32_t voff[4][32], xoff[4][32];
  uint32_t last[32];  // bit 0: the vertex after bit 31 exists; bits 1..7: bit 31's x, y, z, xy, yz, xz, xyz neighbours are subvoxels
  int32_t i[32], j[32], kp[32];
};

// Per-neighbour-word state at a given bit: the reference's local_* arrays.
struct WordState {
  int32_t vidx, xidx, sidx;  // indices of the entry at this bit (-64 when out of range)
  uint32_t vo, so;           // vertex / subvoxel occupancy words
};

__device__ __forceinline__ WordState word_state(const SpanWords& q, int row, int word, bool outside, uint32_t below,
                                                int32_t Nv) {
  WordState s;
  s.vo = q.vo[row][word];
  const uint32_t vx = q.vx[row][word];
  s.so = s.vo & ~vx;
  const int32_t xo = q.xoff[row][word], vo = q.voff[row][word];
  s.vidx = outside ? -64 : vo + __popc(s.vo & below);
  s.xidx = outside ? -64 : xo + __popc(vx & below);
  s.sidx = outside ? -64 : Nv + (vo - xo) + __popc(s.so & below);
  return s;
}

__device__ __forceinline__ int32_t pick_diag(bool diag_sub, bool side_sub, const WordState& s) {
  // Neighbour one step along +x from a side neighbour (see create_voxels.slang:164-172).
  return diag_sub ? (side_sub ? s.sidx + 1 : s.sidx) : (side_sub ? s.xidx : s.xidx + 1);
}

// The neighbour test of bit 31 (create_voxels.slang:211-275).
__device__ __forceinline__ uint32_t last_bit_flags(const VoxelGrid& g, int i, int j, int kp, int64_t w) {
  const bool cx = kp < g.KP - 1, cy = j < g.J - 1, cz = i < g.I - 1;
  const uint32_t top = 1u << 31;
  uint32_t m = kp < g.KP && (__ldg(g.vocc + w + 1) & 1) ? 1u : 0u;
  m |= (cx ? (g.vx(i, j, kp + 1) & 1u) == 0u : true) ? 2u : 0u;
  m |= (cy ? (g.vx(i, j + 1, kp) & top) == 0u : true) ? 4u : 0u;
  m |= (cz ? (g.vx(i + 1, j, kp) & top) == 0u : true) ? 8u : 0u;
  m |= (cx && cy ? (g.vx(i, j + 1, kp + 1) & 1u) == 0u : true) ? 16u : 0u;
  m |= (cy && cz ? (g.vx(i + 1, j + 1, kp) & top) == 0u : true) ? 32u : 0u;
  m |= (cx && cz ? (g.vx(i + 1, j, kp + 1) & 1u) == 0u : true) ? 64u : 0u;
  m |= (cx && cy && cz ? (g.vx(i + 1, j + 1, kp + 1) & 1u) == 0u : true) ? 128u : 0u;
  return m;
}

__global__ void __launch_bounds__(32 * kVoxelWarps)
    create_voxels_kernel(VoxelGrid g, float* __restrict__ vertices, int32_t* __restrict__ neighbors,
                         int32_t* __restrict__ lower, int32_t* __restrict__ upper, int32_t* __restrict__ indices,
                         int64_t G) {
  __shared__ SpanWords spans[kVoxelWarps];
  SpanWords& q = spans[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int J1 = g.J + 1, KP1 = g.KP + 1;
  const int64_t total = (int64_t)(g.I + 1) * J1 * KP1;
  const int64_t mine = (blockIdx.x * (int64_t)kVoxelWarps + (threadIdx.x >> 5)) * 32 + lane;
  const uint32_t my_chunk = mine < total ? (uint32_t)__ldg(g.vocc + mine) : 0u;
  const int my_count = __popc(my_chunk);
  const int incl = warp_inclusive_sum(my_count);
  const int span = __shfl_sync(0xffffffffu, incl, 31);
  if (span == 0) return;  // the whole warp
  if (my_chunk != 0u) {
    int i, j, kp;
    word_position(mine, J1, KP1, i, j, kp);
#pragma unroll
    for (int row = 0; row < 4; ++row) {
      const int ri = i + (row >> 1), rj = j + (row & 1);
      const bool inside = ri <= g.I && rj <= g.J;
      const int64_t w = mine + (row >> 1) * ((int64_t)J1 * KP1) + (row & 1) * KP1;
      q.vo[row][lane] = row == 0 ? my_chunk : inside ? (uint32_t)__ldg(g.vocc + w) : 0u;
      q.vx[row][lane] = g.vx(ri, rj, kp);
      q.voff[row][lane] = inside ? __ldg(g.voff + w) : 0;
      q.xoff[row][lane] = inside ? __ldg(g.xoff + w) : 0;
    }
    q.last[lane] = (my_chunk >> 31) ? last_bit_flags(g, i, j, kp, mine) : 0u;
    q.i[lane] = i;
    q.j[lane] = j;
    q.kp[lane] = kp;
  }
  __syncwarp();

  const int64_t Nv = g.Nv;
  const float inv_i = 1.0f / (float)g.I;
  const float inv_j = 1.0f / (float)g.J;
  const float inv_k = 1.0f / (float)(32 * g.KP);
  const int32_t k_max = 32 * g.KP;
  for (int start = 0; start < span; start += 32) {
    const int r = start + lane;
    int before;
    const int word = dealt_word(incl, my_count, r, before);
    if (r >= span) continue;
    const uint32_t chunk = q.vo[0][word];
    const int pos = select_bit(chunk, r - before);
    const uint32_t bit = 1u << pos, below = bit - 1u;
    const int i = q.i[word], j = q.j[word], kp = q.kp[word];
    const int k = 32 * kp + pos;
    const bool no_j = j >= g.J, no_i = i >= g.I;
    const WordState s00 = word_state(q, 0, word, false, below, (int32_t)Nv);
    const WordState s01 = word_state(q, 1, word, no_j, below, (int32_t)Nv);
    const WordState s10 = word_state(q, 2, word, no_i, below, (int32_t)Nv);

    // Vertices (create_voxels.slang:37-53).
    float* v = vertices + (int64_t)s00.vidx * 3;
    v[0] = (float)k * inv_k;
    v[1] = (float)j * inv_j;
    v[2] = (float)i * inv_i;

    // Lower corners (create_voxels.slang:108-127, last bit fixed up at :201-206).
    const bool is_voxel = (s00.so & bit) == 0u;
    const int32_t chosen = is_voxel ? s00.xidx : s00.sidx;
    const uint32_t last = q.last[word];
    const bool x_valid = is_voxel || (pos < 31 ? ((chunk >> pos) >> 1) & 1u : last & 1u);
    const bool y_valid = is_voxel || (s01.vo & bit);
    const bool z_valid = is_voxel || (s10.vo & bit);
    lower[chosen] = s00.vidx;
    lower[G + chosen] = x_valid ? s00.vidx + 1 : -64;
    lower[2 * G + chosen] = y_valid ? s01.vidx : -64;
    lower[3 * G + chosen] = z_valid ? s10.vidx : -64;
    if (!is_voxel) continue;

    // Upper corners and linear index (create_voxels.slang:129-136).
    const WordState s11 = word_state(q, 3, word, no_i || no_j, below, (int32_t)Nv);
    const int32_t vi = s00.xidx;
    upper[vi] = s11.vidx + 1;
    upper[Nv + vi] = s11.vidx;
    upper[2 * Nv + vi] = s10.vidx + 1;
    upper[3 * Nv + vi] = s01.vidx + 1;
    indices[vi] = k_max * (g.J * i + j) + k;

    // Neighbours (create_voxels.slang:138-193 for bits 0..30, :211-275 for bit 31).
    bool x_sub, y_sub, z_sub, xy_sub, yz_sub, xz_sub, xyz_sub;
    if (pos < 31) {
      const uint32_t nb = bit << 1;
      x_sub = (s00.so & nb) != 0u;
      y_sub = (s01.so & bit) != 0u;
      z_sub = (s10.so & bit) != 0u;
      xy_sub = (s01.so & nb) != 0u;
      yz_sub = (s11.so & bit) != 0u;
      xz_sub = (s10.so & nb) != 0u;
      xyz_sub = (s11.so & nb) != 0u;
    } else {
      x_sub = last & 2u;
      y_sub = last & 4u;
      z_sub = last & 8u;
      xy_sub = last & 16u;
      yz_sub = last & 32u;
      xz_sub = last & 64u;
      xyz_sub = last & 128u;
    }
    neighbors[vi] = x_sub ? s00.sidx : s00.xidx + 1;
    neighbors[Nv + vi] = y_sub ? s01.sidx : s01.xidx;
    neighbors[2 * Nv + vi] = z_sub ? s10.sidx : s10.xidx;
    neighbors[3 * Nv + vi] = pick_diag(xy_sub, y_sub, s01);
    neighbors[4 * Nv + vi] = yz_sub ? s11.sidx : s11.xidx;
    neighbors[5 * Nv + vi] = pick_diag(xz_sub, z_sub, s10);
    neighbors[6 * Nv + vi] = pick_diag(xyz_sub, yz_sub, s11);
  }
}

// ---------------------------------------------------------------------------
// dilate_occupancy.slang:9-94 (box dilation, 0 < d < 32).
// ---------------------------------------------------------------------------
//
// A warp reads 32 consecutive words and writes the inner 30: each lane ORs its
// word over the box's rows, and takes the words before and after from the
// lanes beside it. Reading all three words per lane made 3 (2 d + 1)^2 loads
// a word: 52 us at 256^3, d = 4; now 22 us.
constexpr int kDilateWords = 30;

__global__ void dilate_kernel(const int32_t* __restrict__ occ, int I, int J, int KP, int d,
                              int32_t* __restrict__ out) {
  const int64_t total = (int64_t)I * J * KP;
  const int lane = threadIdx.x & 31;
  const int64_t first_warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = first_warp * kDilateWords; base < total; base += warps * kDilateWords) {
    const int64_t w = base + lane - 1;
    const bool there = w >= 0 && w < total;
    int i = 0, j = 0, kp = 0;
    uint32_t cur = 0;
    if (there) {
      word_position(w, J, KP, i, j, kp);
      const int i0 = max(i - d, 0), i1 = min(i + d, I - 1);
      const int j0 = max(j - d, 0), j1 = min(j + d, J - 1);
      for (int ii = i0; ii <= i1; ++ii) {
        const int32_t* row = occ + ((int64_t)ii * J + j0) * KP + kp;
#pragma unroll 4
        for (int jj = j0; jj <= j1; ++jj, row += KP) cur |= (uint32_t)__ldg(row);
      }
    }
    const uint32_t prev = __shfl_up_sync(0xffffffffu, cur, 1), next = __shfl_down_sync(0xffffffffu, cur, 1);
    if (!there || lane == 0 || lane > kDilateWords) continue;
    uint32_t result = cur;
    // Bits that spill in from the previous word (dilate_occupancy.slang:41-44).
    if (kp > 0) {
      uint32_t p = prev >> (32 - d);
      for (int b = 0; b < d; ++b) {
        result |= p;
        p >>= 1;
      }
    }
    uint32_t l = cur, r = cur;
    for (int b = 0; b < d; ++b) {
      r >>= 1;
      l <<= 1;
      result |= l | r;
    }
    if (kp < KP - 1) {
      uint32_t n = next << (32 - d);
      for (int b = 0; b < d; ++b) {
        result |= n;
        n <<= 1;
      }
    }
    out[w] = (int32_t)result;
  }
}

// ---------------------------------------------------------------------------
// count_triangle_vertices.slang:3-37
// ---------------------------------------------------------------------------
struct Corners4 {
  float d0, d[3];
  int32_t idx[3];  // lower_corners[1..3], may be negative
};

__device__ __forceinline__ Corners4 load_corners(const float* __restrict__ sdf, const int32_t* __restrict__ lower,
                                                 int64_t G, int64_t g) {
  Corners4 c;
  const int32_t i0 = __ldg(lower + g);
  c.d0 = __ldg(sdf + i0);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int32_t ia = __ldg(lower + (a + 1) * G + g);
    c.idx[a] = ia;
    c.d[a] = (ia >= 0) ? __ldg(sdf + ia) : c.d0;
  }
  return c;
}

// Bit a of the result: edge `a` of entry g crosses level set `iso`. The same
// predicate sizes the outputs (count) and places vertices (create), so the
// writes always stay inside the counted range.
__device__ __forceinline__ uint32_t crossing_mask(const Corners4& c, float iso) {
  const bool b0 = c.d0 < iso;
  return (uint32_t)(b0 != (c.d[0] < iso)) | ((uint32_t)(b0 != (c.d[1] < iso)) << 1) |
         ((uint32_t)(b0 != (c.d[2] < iso)) << 2);
}

__global__ void count_vertices_kernel(const float* __restrict__ sdf, const int32_t* __restrict__ lower, int64_t G,
                                      const float* __restrict__ level_sets, int S, int32_t* __restrict__ counts) {
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < G; g += (int64_t)gridDim.x * blockDim.x) {
    const Corners4 c = load_corners(sdf, lower, G, g);
    for (int s = 0; s < S; ++s) {
      const float iso = __ldg(level_sets + s);
      const bool b0 = c.d0 < iso;
      counts[(int64_t)s * G + g] = (b0 != (c.d[0] < iso)) + (b0 != (c.d[1] < iso)) + (b0 != (c.d[2] < iso));
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) counts[(int64_t)S * G] = 0;
}

// The crossings themselves, a byte each, for the scan that takes their numbers
// and the faces, which then find an edge's vertex without the types.
__global__ void count_crossings_kernel(const float* __restrict__ sdf, const int32_t* __restrict__ lower, int64_t G,
                                       const float* __restrict__ level_sets, int S, uint8_t* __restrict__ crossings) {
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < G; g += (int64_t)gridDim.x * blockDim.x) {
    const Corners4 c = load_corners(sdf, lower, G, g);
    for (int s = 0; s < S; ++s) crossings[(int64_t)s * G + g] = (uint8_t)crossing_mask(c, __ldg(level_sets + s));
  }
}

// create_triangle_vertices.slang:87-96: t is detached; positions / SH / sdf
// are linear in the corner values with weights (1 - t, t).
__device__ __forceinline__ float mc_weight(float d0, float d1, float iso) {
  if (d0 == d1) return 0.5f;
  const float t = (iso - d0) / (d1 - d0);
  return fminf(fmaxf(t, 0.0f), 1.0f);
}

// a + t * (b - a), rounded after each operation as the reference source
// writes it (create_triangle_vertices.slang:105-127).
__device__ __forceinline__ float lerp_ref(float a, float b, float t) {
  return __fadd_rn(a, __fmul_rn(t, __fsub_rn(b, a)));
}

// ---------------------------------------------------------------------------
// create_triangle_vertices.slang:145-199 (forward), in two passes.
//
// Pass 1, one thread per entry g: positions, signed distance and type of
// every vertex on g's crossing edges, plus the vertex's source record
// (origin corner, axis corner, t) in vertex order.
// Pass 2, one thread per (coefficient row k, vertex): the SH row k of the
// vertex from its two corners. Consecutive threads write consecutive
// vertices of one row, so the [C, V, 3] output is written coalesced.
// ---------------------------------------------------------------------------
constexpr int kShellsPerChunk = 21;

__device__ __forceinline__ uint64_t crossing_bits(const Corners4& c, const float* __restrict__ level_sets, int s0,
                                                  int s1) {
  uint64_t bits = 0;
  for (int s = s0; s < s1; ++s) bits |= (uint64_t)crossing_mask(c, __ldg(level_sets + s)) << (3 * (s - s0));
  return bits;
}

// One thread per entry: the crossings of its three edges with all shells (up
// to kShellsPerChunk at a time) as a bit each, then a turn per shell. Where
// vertices are few (1.4 to an entry at 512^3, 8 shells) a lane takes its own
// shells: 206 us, with the warp's lanes taking every shell that one of them
// crosses 284. Where they are many (2.2 at 16 shells) the lanes take them
// together, to write neighbouring vertices: 535 us, each its own 656. A loop over
// every (axis, shell) pair took 332 and 612, and 25 us at 256^3, 8 shells, now 15.
template <bool kTogether>
__global__ void create_vertices_kernel(const float* __restrict__ gv, const float* __restrict__ gsdf,
                                       const int32_t* __restrict__ lower, int64_t G,
                                       const float* __restrict__ level_sets, int S,
                                       const int32_t* __restrict__ voff, int64_t V, float* __restrict__ out_v,
                                       float* __restrict__ out_sdf, uint8_t* __restrict__ out_type,
                                       int32_t* __restrict__ sources) {
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < G; g += (int64_t)gridDim.x * blockDim.x) {
    const Corners4 c = load_corners(gsdf, lower, G, g);
    for (int s0 = 0; s0 < S; s0 += kShellsPerChunk) {
      const uint64_t crossings = crossing_bits(c, level_sets, s0, min(S, s0 + kShellsPerChunk));
      // Shells that the entry crosses, or with kTogether some lane of the warp
      // (bit 3 s).
      uint64_t shells = (crossings | (crossings >> 1) | (crossings >> 2)) & 0x1249249249249249ull;
      if constexpr (kTogether) {
        const unsigned warp = __activemask();
        shells = (uint64_t)__reduce_or_sync(warp, (uint32_t)(shells >> 32)) << 32 |
                 __reduce_or_sync(warp, (uint32_t)shells);
      }
      if (shells == 0) continue;
      const int32_t i0 = __ldg(lower + g);
      float v0x = 0.f, v0y = 0.f, v0z = 0.f;
      if (crossings != 0) {
        v0x = __ldg(gv + 3 * (int64_t)i0);
        v0y = __ldg(gv + 3 * (int64_t)i0 + 1);
        v0z = __ldg(gv + 3 * (int64_t)i0 + 2);
      }
      for (; shells; shells &= shells - 1) {
        const int at = __ffsll((long long)shells) - 1, sl = at / 3;
        uint32_t m = (uint32_t)(crossings >> at) & 7u;
        if (m == 0) continue;
        int64_t vi = (int64_t)__ldg(voff + (int64_t)(s0 + sl) * G + g);
        const float iso = __ldg(level_sets + s0 + sl);
        for (; m; m &= m - 1, ++vi) {
          if (vi >= V) break;  // beyond the caller's capacity (reported by the caller's count check)
          const int a = __ffs(m) - 1;
          const int32_t i1 = a == 0 ? c.idx[0] : a == 1 ? c.idx[1] : c.idx[2];
          const float d1 = a == 0 ? c.d[0] : a == 1 ? c.d[1] : c.d[2];
          const float v1x = __ldg(gv + 3 * (int64_t)i1), v1y = __ldg(gv + 3 * (int64_t)i1 + 1),
                      v1z = __ldg(gv + 3 * (int64_t)i1 + 2);
          const float t = mc_weight(c.d0, d1, iso);
          out_v[3 * vi + 0] = lerp_ref(v0x, v1x, t);
          out_v[3 * vi + 1] = lerp_ref(v0y, v1y, t);
          out_v[3 * vi + 2] = lerp_ref(v0z, v1z, t);
          out_sdf[vi] = lerp_ref(c.d0, d1, t);
          out_type[vi] = (uint8_t)a;
          sources[vi] = i0;
          sources[V + vi] = i1;
          sources[2 * V + vi] = __float_as_int(t);
        }
      }
    }
  }
}

// Rows have stride V (the buffer's capacity); only the first `count`
// vertices (device value, clamped to V; all V when count is NULL) are real.
//
// A CTA takes kRowTile consecutive grid entries, whose vertices are one run for
// each shell; its warps deal with 32 vertices of a run at a time, all planes,
// so the grid's rows come from memory once for all shells (in vertex order,
// shell after shell, they did for each: 3.7 GB instead of 1.25 at 352^3). A
// lane takes floats lane, lane + 32 and lane + 64 of the 96 that 32 vertices
// have in a plane (vertex and channel stay the same from plane to plane), so
// that a load or store covers 128 consecutive bytes. With a thread to a
// (plane, vertex) the sources were read again for every plane, as many bytes
// as the rows written, and every access strode over 12 B. 512^3, 8 shells,
// C = 16 (9.3 M vertices): 1240 us, now 765 (tiles of 512: 834; 768: 983).
constexpr int kRowTile = 256;
constexpr int kRowPlanes = 4;  // planes whose loads are issued side by side

template <typename Offset>
__device__ __forceinline__ const float* at_bytes(const float* p, Offset bytes) {
  return reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + bytes);
}

// Up to 32 consecutive vertices from v0, all planes.
template <typename Offset>
__device__ __forceinline__ void interpolate_rows(const float* __restrict__ gsh, int C, int64_t grid_plane,
                                                 const int32_t* __restrict__ sources, int64_t V, int64_t v0, int many,
                                                 int lane, float* __restrict__ out_sh) {
  const int64_t v = v0 + min(lane, many - 1);
  const int32_t i0 = __ldg(sources + v), i1 = __ldg(sources + V + v), tb = __ldg(sources + 2 * V + v);
  const int floats = 3 * many;
  const int64_t row_plane = 3 * V;
  Offset a0[3], a1[3];
  float t[3];
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const int f = 32 * p + lane, q = f / 3, ch = f - 3 * q;
    a0[p] = (Offset)12 * (Offset)__shfl_sync(0xffffffffu, i0, q) + (Offset)(4 * ch);
    a1[p] = (Offset)12 * (Offset)__shfl_sync(0xffffffffu, i1, q) + (Offset)(4 * ch);
    t[p] = __int_as_float(__shfl_sync(0xffffffffu, tb, q));
  }
  for (int k0 = 0; k0 < C; k0 += kRowPlanes) {
    float x0[kRowPlanes][3], x1[kRowPlanes][3];
#pragma unroll
    for (int j = 0; j < kRowPlanes; ++j) {
      if (k0 + j < C) {
        const float* plane = gsh + (k0 + j) * grid_plane;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          if (32 * p < floats) {
            x0[j][p] = __ldg(at_bytes(plane, a0[p]));
            x1[j][p] = __ldg(at_bytes(plane, a1[p]));
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kRowPlanes; ++j) {
      if (k0 + j < C) {
        float* dst = out_sh + (k0 + j) * row_plane + 3 * v0 + lane;
#pragma unroll
        for (int p = 0; p < 3; ++p)
          if (32 * p + lane < floats) __stcs(dst + 32 * p, lerp_ref(x0[j][p], x1[j][p], t[p]));
      }
    }
  }
}

template <typename Offset>
__global__ void __launch_bounds__(256, 4)
    interpolate_vertex_sh_kernel(const float* __restrict__ gsh, int C, int64_t G,
                                 const int32_t* __restrict__ sources, int64_t V, const int32_t* __restrict__ count,
                                 const int32_t* __restrict__ voff, int S, float* __restrict__ out_sh) {
  const int64_t n = count ? min((int64_t)max(*count, 0), V) : V;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t e0 = blockIdx.x * (int64_t)kRowTile, e1 = min(e0 + kRowTile, G);
  int turn = 0;  // batches so far, dealt to the warps in turn
  for (int s0 = 0; s0 < S; s0 += 32) {
    const int64_t row = (int64_t)(s0 + lane) * G;
    const int32_t first = s0 + lane < S ? __ldg(voff + row + e0) : 0;
    const int32_t last = s0 + lane < S ? __ldg(voff + row + e1) : 0;
    for (int j = 0; j < min(32, S - s0); ++j) {
      const int64_t b = __shfl_sync(0xffffffffu, first, j), e = min((int64_t)__shfl_sync(0xffffffffu, last, j), n);
      const int batches = (int)((max(e - b, (int64_t)0) + 31) >> 5);
      for (int i = (warp - turn) & 7; i < batches; i += 8)
        interpolate_rows<Offset>(gsh, C, 3 * G, sources, V, b + 32 * i, (int)min((int64_t)32, e - b - 32 * i), lane,
                                 out_sh);
      turn += batches;
    }
  }
}

// ---------------------------------------------------------------------------
// Live marching-cubes weight (not in the reference, which detaches t at
// create_triangle_vertices.slang:92-96). With t = (iso - d0) / (d1 - d0) live,
// a vertex's position and SH depend on its two corner SDFs through t:
//   dL/dt = g_pos . (p1 - p0) + sum_k g_sh_k . (sh1_k - sh0_k),
//   dt/dd0 = -(1 - t) / (d1 - d0),  dt/dd1 = -t / (d1 - d0),
// and its SDF, d0 + t (d1 - d0) = iso, does not depend on them at all. t is
// constant where the reference clamps it or sets it to 0.5 (d0 == d1), so
// only 0 < t < 1 contributes. One thread per vertex adds the two corner
// terms to the grid SDF gradient with atomics. Rows have stride V; only the
// first `count` vertices (device value; all V when NULL) are real.
// ---------------------------------------------------------------------------
__global__ void live_t_backward_kernel(const float* __restrict__ gv, const float* __restrict__ gsdf,
                                       const float* __restrict__ gsh, int C, int64_t G,
                                       const int32_t* __restrict__ sources, int64_t V,
                                       const int32_t* __restrict__ count, const float* __restrict__ grad_v,
                                       const float* __restrict__ grad_sh, float* __restrict__ grad_gsdf) {
  const int64_t n = count ? min((int64_t)max(*count, 0), V) : V;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i0 = __ldg(sources + v), i1 = __ldg(sources + V + v);
    const float t = __int_as_float(__ldg(sources + 2 * V + v));
    const float d0 = __ldg(gsdf + i0), d1 = __ldg(gsdf + i1);
    if (!(t > 0.0f && t < 1.0f) || d0 == d1) continue;
    float dldt = 0.0f;
    if (grad_v) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
        dldt += __ldg(grad_v + 3 * v + c) * (__ldg(gv + 3 * (int64_t)i1 + c) - __ldg(gv + 3 * (int64_t)i0 + c));
    }
    if (grad_sh) {
      for (int k = 0; k < C; ++k) {
        const float* g = grad_sh + ((int64_t)k * V + v) * 3;
        const float* p0 = gsh + ((int64_t)k * G + i0) * 3;
        const float* p1 = gsh + ((int64_t)k * G + i1) * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c) dldt += __ldg(g + c) * (__ldg(p1 + c) - __ldg(p0 + c));
      }
    }
    if (dldt == 0.0f) continue;
    const float q = dldt / (d1 - d0);
    atomicAdd(grad_gsdf + i0, -q * (1.0f - t));
    atomicAdd(grad_gsdf + i1, -q * t);
  }
}

// ---------------------------------------------------------------------------
// create_triangle_vertices.slang:201-291 (backward) as a gather. The detached
// weight t routes d(vertex) to the origin corner with (1 - t) and to the axis
// corner with t. Grid vertex x receives from the vertices of the one entry
// whose origin it is and from the vertices on axis a of the (at most three)
// entries whose axis-a corner it is; `inverse` [4, G] lists those entries.
// One thread per grid vertex writes all of x's gradients (zeros included),
// so no atomics and no zero-filled outputs are needed.
//
// Crossings are packed 3 bits per shell into 64-bit masks, shells taken in
// chunks of 21; the first chunk writes, later chunks add.
// ---------------------------------------------------------------------------
// `zero0` [G+1] and `zero1` [G] (either may be NULL) are cleared on the way,
// for the per-entry list passes that follow.
__global__ void invert_corners_kernel(const int32_t* __restrict__ lower, int64_t G, int32_t* __restrict__ inverse,
                                      int32_t* __restrict__ zero0 = nullptr, uint32_t* __restrict__ zero1 = nullptr) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < G; e += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int32_t x = __ldg(lower + r * G + e);
      if (x >= 0 && x < G) inverse[r * G + x] = (int32_t)e;
    }
    if (zero0) zero0[e] = 0;
    if (zero1) zero1[e] = 0u;
  }
  if (zero0 && blockIdx.x == 0 && threadIdx.x == 0) zero0[G] = 0;
}

// One contribution list of grid vertex x for the shells of one chunk: the
// vertex index and weight of every triangle vertex that x feeds.
struct GatherChunk {
  uint64_t own;       // crossings of x's own entry (3 bits per shell)
  uint64_t nb[3];     // crossings of the entry whose axis-a corner x is
  int64_t e, h[3];    // those entries (-1 = none)
  float d0, d1[3];    // own entry: origin and axis-corner signed distances
  float nd0[3], nd1[3];  // entry h[a]: origin and axis-a corner signed distances
};

__device__ __forceinline__ int64_t vertex_of(const int32_t* __restrict__ voff, int64_t G, int64_t entry, int s,
                                             uint64_t bits, int s0, int a) {
  const uint32_t m = (uint32_t)(bits >> (3 * (s - s0))) & 7u;
  return (int64_t)__ldg(voff + (int64_t)s * G + entry) + __popc(m & ((1u << a) - 1u));
}

// Calls f(vertex, weight) for each of x's contributions in this shell chunk:
// weight (1 - t) for the vertices of x's own entry, t for the axis-a vertices
// of the entries whose axis-a corner x is.
// Vertices at or past V (the buffers' capacity; only reached when the live
// count overflowed it) were never written and are skipped.
template <typename F>
__device__ __forceinline__ void for_each_contribution(const GatherChunk& q, const float* __restrict__ level_sets,
                                                      int s0, const int32_t* __restrict__ voff, int64_t G,
                                                      int64_t V, F&& f) {
  uint64_t bits = q.own;
  while (bits) {
    const int j = __ffsll((long long)bits) - 1;
    bits &= bits - 1;
    const int sl = j / 3, a = j - 3 * sl, s = s0 + sl;
    const int64_t vi = vertex_of(voff, G, q.e, s, q.own, s0, a);
    if (vi >= V) continue;
    f(vi, mc_weight(q.d0, q.d1[a], __ldg(level_sets + s)), true);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    uint64_t nbits = q.nb[a] & (0x1249249249249249ull << a);  // axis-a bits only
    while (nbits) {
      const int j = __ffsll((long long)nbits) - 1;
      nbits &= nbits - 1;
      const int s = s0 + j / 3;
      const int64_t vi = vertex_of(voff, G, q.h[a], s, q.nb[a], s0, a);
      if (vi >= V) continue;
      f(vi, mc_weight(q.nd0[a], q.nd1[a], __ldg(level_sets + s)), false);
    }
  }
}

// (1 - t) g, written g - t g as the reference's adjoint forms it, or t g.
__device__ __forceinline__ float weighted(float g, float t, bool origin) { return origin ? g - t * g : t * g; }

constexpr int kRowsPerPass = 16;  // SH coefficient rows accumulated in registers at once

__global__ void create_vertices_backward_kernel(const float* __restrict__ gsdf, int C,
                                                const int32_t* __restrict__ lower, int64_t G,
                                                const float* __restrict__ level_sets, int S,
                                                const int32_t* __restrict__ voff,
                                                const int32_t* __restrict__ inverse,
                                                const float* __restrict__ dv, const float* __restrict__ dsdf,
                                                const float* __restrict__ dsh, int64_t V, float* __restrict__ gdv,
                                                float* __restrict__ gdsdf, float* __restrict__ gdsh) {
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < G; x += (int64_t)gridDim.x * blockDim.x) {
    GatherChunk q;
    q.e = __ldg(inverse + x);
    Corners4 own{};
    if (q.e >= 0) own = load_corners(gsdf, lower, G, q.e);
    q.d0 = own.d0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      q.d1[a] = own.d[a];
      q.h[a] = __ldg(inverse + (int64_t)(a + 1) * G + x);
    }
    Corners4 nb[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (q.h[a] >= 0) {
        nb[a] = load_corners(gsdf, lower, G, q.h[a]);
        q.nd0[a] = nb[a].d0;
        q.nd1[a] = nb[a].d[a];
      }
    }
    const int chunks = S > 0 ? (S + kShellsPerChunk - 1) / kShellsPerChunk : 1;
    for (int chunk = 0; chunk < chunks; ++chunk) {
      const int s0 = chunk * kShellsPerChunk, s1 = min(S, s0 + kShellsPerChunk);
      q.own = q.e >= 0 ? crossing_bits(own, level_sets, s0, s1) : 0ull;
#pragma unroll
      for (int a = 0; a < 3; ++a) q.nb[a] = q.h[a] >= 0 ? crossing_bits(nb[a], level_sets, s0, s1) : 0ull;
      const bool first = chunk == 0;
      auto put = [&](float* dst, float value) { *dst = first ? value : *dst + value; };

      float d = 0.f, p[3] = {0.f, 0.f, 0.f};
      for_each_contribution(q, level_sets, s0, voff, G, V, [&](int64_t vi, float t, bool origin) {
        if (dsdf) d += weighted(__ldg(dsdf + vi), t, origin);
        if (dv) {
#pragma unroll
          for (int ch = 0; ch < 3; ++ch) p[ch] += weighted(__ldg(dv + 3 * vi + ch), t, origin);
        }
      });
      put(gdsdf + x, d);
      if (gdv) {
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) put(gdv + 3 * x + ch, p[ch]);
      }
      // SH rows in passes of 16: every contribution's 48 loads are independent.
      for (int k0 = 0; k0 < C; k0 += kRowsPerPass) {
        float r[kRowsPerPass][3];
#pragma unroll
        for (int kk = 0; kk < kRowsPerPass; ++kk) r[kk][0] = r[kk][1] = r[kk][2] = 0.f;
        if (dsh) {
          for_each_contribution(q, level_sets, s0, voff, G, V, [&](int64_t vi, float t, bool origin) {
#pragma unroll
            for (int kk = 0; kk < kRowsPerPass; ++kk) {
              if (k0 + kk < C) {
                const float* src = dsh + ((int64_t)(k0 + kk) * V + vi) * 3;
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) r[kk][ch] += weighted(__ldg(src + ch), t, origin);
              }
            }
          });
        }
#pragma unroll
        for (int kk = 0; kk < kRowsPerPass; ++kk) {
          if (k0 + kk < C) {
            float* dst = gdsh + ((int64_t)(k0 + kk) * G + x) * 3;
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) put(dst + ch, r[kk][ch]);
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The same backward as a contribution list and a gather (S <= 21 shells).
//
// entry_list_kernel (below) lists every contribution (vertex | origin flag
// << 31, t) of a grid vertex x, in the order in which
// create_vertices_backward_kernel enumerates them, at x's offset in a CSR list
// of at most 2V entries; vertex_grads_from_list_kernel and
// vertex_sh_gather_kernel sum the gradients over x's list in list order (the
// same sums, so the same bits).
// ---------------------------------------------------------------------------
template <int kRows, int kAhead>
__device__ __forceinline__ void gather_sh_rows(const float* __restrict__ dsh, int64_t row_plane, int32_t begin,
                                               int32_t end, int ch, const int2* __restrict__ list,
                                               float* __restrict__ dst, int64_t grid_plane) {
  float acc[kRows];
#pragma unroll
  for (int k = 0; k < kRows; ++k) acc[k] = 0.f;
  if (dsh) {
    for (int32_t p = begin; p < end; p += kAhead) {
      int2 e[kAhead];
#pragma unroll
      for (int j = 0; j < kAhead; ++j) e[j] = __ldg(list + min(p + j, end - 1));
      float x[kAhead][kRows];
#pragma unroll
      for (int j = 0; j < kAhead; ++j)
#pragma unroll
        for (int k = 0; k < kRows; ++k)
          x[j][k] = __ldg(dsh + 3 * (int64_t)(e[j].x & 0x7fffffff) + ch + k * row_plane);
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        if (p + j < end) {
#pragma unroll
          for (int k = 0; k < kRows; ++k) acc[k] += weighted(x[j][k], __int_as_float(e[j].y), e[j].x < 0);
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kRows; ++k) __stcs(dst + k * grid_plane, acc[k]);
}

// A thread to a float (grid vertex, channel) of the grid's rows: neighbouring
// threads read and write neighbouring floats, four rows at a time with four
// list entries ahead. Bound by the L1's line look-ups, one for each (list
// entry, row), as a list's vertices lie apart: a thread to a (row, grid
// vertex) made three of them and read the list again for every row; 16 rows at
// a time (one reading of the list) lose the lines that neighbouring lists
// share. 512^3, 8 shells, C = 16: 1178 us before, 1047 to 1111 with this (16 rows, one
// entry: 1553 us; 8 and 4: 1205).
constexpr int kGatherThreads = 192, kGatherRows = 4, kGatherAhead = 4;

__global__ void __launch_bounds__(kGatherThreads)
    vertex_sh_gather_kernel(const float* __restrict__ dsh, int C, int64_t V, int64_t G,
                            const int32_t* __restrict__ offsets, const int2* __restrict__ list,
                            float* __restrict__ gdsh) {
  const int64_t row_plane = 3 * V, grid_plane = 3 * G;
  const int64_t o = blockIdx.x * (int64_t)kGatherThreads + threadIdx.x;
  if (o >= grid_plane) return;
  const int64_t x = o / 3;
  const int ch = (int)(o - 3 * x);
  const int32_t begin = __ldg(offsets + x), end = __ldg(offsets + x + 1);
  int k = 0;
  for (; k + kGatherRows <= C; k += kGatherRows)
    gather_sh_rows<kGatherRows, kGatherAhead>(dsh ? dsh + k * row_plane : nullptr, row_plane, begin, end, ch, list,
                                              gdsh + k * grid_plane + o, grid_plane);
  for (; k < C; ++k)
    gather_sh_rows<1, kGatherAhead>(dsh ? dsh + k * row_plane : nullptr, row_plane, begin, end, ch, list,
                                    gdsh + k * grid_plane + o, grid_plane);
}

// The signed-distance and position gradients of the list.
__global__ void vertex_grads_from_list_kernel(const int32_t* __restrict__ offsets, const int2* __restrict__ list,
                                              int64_t G, const float* __restrict__ dv, const float* __restrict__ dsdf,
                                              float* __restrict__ gdv, float* __restrict__ gdsdf) {
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < G; x += (int64_t)gridDim.x * blockDim.x) {
    float d = 0.f, p[3] = {0.f, 0.f, 0.f};
    const int32_t end = __ldg(offsets + x + 1);
    for (int32_t q = __ldg(offsets + x); q < end; ++q) {
      const int2 e = __ldg(list + q);
      const int64_t vi = e.x & 0x7fffffff;
      const bool origin = e.x < 0;
      const float t = __int_as_float(e.y);
      if (dsdf) d += weighted(__ldg(dsdf + vi), t, origin);
      if (dv) {
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) p[ch] += weighted(__ldg(dv + 3 * vi + ch), t, origin);
      }
    }
    gdsdf[x] = d;
    if (gdv) {
#pragma unroll
      for (int ch = 0; ch < 3; ++ch) gdv[3 * x + ch] = p[ch];
    }
  }
}

// ---------------------------------------------------------------------------
// The contribution list, built per grid entry (mt_build_vertex_grad_list).
//
// Grid vertex x's list is four segments: the vertices of the entry whose
// origin x is, then the axis-0, axis-1 and axis-2 vertices of the entries
// whose axis-a corner x is, each in shell order (the order of
// for_each_contribution). Entry e owns segment r of x = lower[r][e] when the
// corner inverse names e there (so exactly the entries the per-vertex
// enumeration visits, also for inputs where two entries share a corner).
// Pass 1 adds each owned segment's length to x's count and stores it in byte
// r of x's segment word; pass 2 writes the segment at x's scanned offset plus
// the lengths of x's earlier segments. Each entry loads its own corners once
// (a pass per grid vertex loads four entries' corners for each: 318 + 411 us
// at 512^3, 8 shells; this 105 + 221, a turn per crossed shell; the count, which
// is its set bits where no vertex is past the capacity, 126 by turns).
// Counts and segment words start at zero (cleared by invert_corners_kernel).
// ---------------------------------------------------------------------------
template <bool kFill>
__global__ void entry_list_kernel(const float* __restrict__ gsdf, const int32_t* __restrict__ lower, int64_t G,
                                  const float* __restrict__ level_sets, int S, const int32_t* __restrict__ voff,
                                  const int32_t* __restrict__ inverse, int64_t V, int32_t* __restrict__ counts,
                                  uint32_t* __restrict__ segments, int2* __restrict__ list) {
  // No vertex past the capacity. Without level sets a caller may have no offsets.
  const bool fit = S == 0 || (int64_t)__ldg(voff + (int64_t)S * G) <= V;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < G; e += (int64_t)gridDim.x * blockDim.x) {
    const Corners4 c = load_corners(gsdf, lower, G, e);
    const uint64_t bits = crossing_bits(c, level_sets, 0, S);
    if (bits == 0) continue;
    // The shells that the entry crosses (bit 3 s), a turn each.
    const uint64_t shells = (bits | (bits >> 1) | (bits >> 2)) & 0x1249249249249249ull;
    int64_t x[4];
    x[0] = __ldg(lower + e);
#pragma unroll
    for (int a = 0; a < 3; ++a) x[a + 1] = c.idx[a];
    bool owns[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) owns[r] = x[r] >= 0 && x[r] < G && __ldg(inverse + r * G + x[r]) == (int32_t)e;
    if (!(owns[0] || owns[1] || owns[2] || owns[3])) continue;
    if (!kFill) {
      int n[4] = {__popcll(bits), __popcll(bits & 0x1249249249249249ull), __popcll(bits & 0x2492492492492492ull),
                  __popcll(bits & 0x4924924924924924ull)};
      if (!fit) n[0] = n[1] = n[2] = n[3] = 0;
      for (uint64_t left = fit ? 0ull : shells; left; left &= left - 1) {
        const int at = __ffsll((long long)left) - 1, s = at / 3;
        const uint32_t m = (uint32_t)(bits >> at) & 7u;
        const int64_t base = __ldg(voff + (int64_t)s * G + e);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (!((m >> a) & 1u) || base + __popc(m & ((1u << a) - 1u)) >= V) continue;
          ++n[0];
          ++n[a + 1];
        }
      }
      uint8_t* seg = reinterpret_cast<uint8_t*>(segments);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (owns[r] && n[r] > 0) {
          atomicAdd(counts + x[r], n[r]);
          seg[4 * x[r] + r] = (uint8_t)n[r];  // n[0] <= 3 * 21, n[a + 1] <= 21
        }
      }
    } else {
      const int64_t cap = 2 * V;
      int64_t pos[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        pos[r] = 0;
        if (owns[r]) {
          const uint32_t w = __ldg(segments + x[r]);
          uint32_t earlier = 0;
#pragma unroll
          for (int q = 0; q < r; ++q) earlier += (w >> (8 * q)) & 0xffu;
          pos[r] = (int64_t)__ldg(counts + x[r]) + earlier;  // counts = scanned offsets here
        }
      }
      for (uint64_t left = shells; left; left &= left - 1) {
        const int at = __ffsll((long long)left) - 1, s = at / 3;
        const uint32_t m = (uint32_t)(bits >> at) & 7u;
        const float iso = __ldg(level_sets + s);
        const int64_t base = __ldg(voff + (int64_t)s * G + e);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (!((m >> a) & 1u)) continue;
          const int64_t vi = base + __popc(m & ((1u << a) - 1u));
          if (vi >= V) continue;
          const int tb = __float_as_int(mc_weight(c.d0, c.d[a], iso));
          if (owns[0] && pos[0] < cap) list[pos[0]] = make_int2((int)vi | (int)0x80000000, tb);
          ++pos[0];
          if (owns[a + 1] && pos[a + 1] < cap) list[pos[a + 1]] = make_int2((int)vi, tb);
          ++pos[a + 1];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Grid SH -> vertex colours without per-vertex SH rows: the interpolation of
// create_triangle_vertices.slang:145-199 (coefficients of vertex v from its
// two grid corners with weight t) followed by
// evaluate_spherical_harmonics.slang:4-270 for every camera, the coefficients
// kept in registers. Same operations as interpolate_vertex_sh_kernel then
// sh_forward_kernel, so the same bits. Vertices at or past the live count are
// not touched.
// ---------------------------------------------------------------------------
// A CTA takes kColourTile consecutive grid entries and deals their vertices, a
// run for each shell, out to its threads, so that the grid's rows come from
// memory once for all shells. In vertex order, shell after shell, they were
// read again for each (7.3 GB at 352^3, 16 shells, instead of 1.5): 2.24 ms at
// 512^3, 16 shells, 4 cameras, now 1.19. Where they stay in the L2 anyway
// (kColourCached bytes) vertex order is as good: 55 us at 256^3, 8 shells
// (81 MB of rows), where the tiles' search makes 59. Interpolating by
// consecutive floats and turning them in shared memory, as the rows' kernel
// does, spent more on partial batches than it saved: 1.50 ms and 77 us.
//
// seen (where a caller gives it): a byte per vertex, zero for those that no key's
// triangle names, whose colours no compositing kernel reads and which are not
// written: with cameras inside a 512^3 scene of 16 shells 590 us (and 79 for the
// marks) instead of 1190.
constexpr int kColourTile = 256, kColourThreads = 128;
constexpr int kColourShells = 32;  // more shells: vertex order
constexpr int64_t kColourCached = (int64_t)100 << 20;

template <int kCoeff>
__device__ __forceinline__ void grid_sh_vertex(const float* __restrict__ gsh, int64_t G,
                                               const int32_t* __restrict__ sources, int64_t V,
                                               const float* __restrict__ verts, const float* __restrict__ campos,
                                               int B, int64_t v, float* __restrict__ out) {
  const int32_t i0 = __ldg(sources + v), i1 = __ldg(sources + V + v);
  const float t = __int_as_float(__ldg(sources + 2 * V + v));
  float coef[kCoeff][3];
#pragma unroll
  for (int k = 0; k < kCoeff; ++k) {
    const float* p0 = gsh + ((int64_t)k * G + i0) * 3;
    const float* p1 = gsh + ((int64_t)k * G + i1) * 3;
#pragma unroll
    for (int c = 0; c < 3; ++c) coef[k][c] = lerp_ref(__ldg(p0 + c), __ldg(p1 + c), t);
  }
  sh_colors<kCoeff>(verts, V, coef, campos, B, v, out);
}

// The vertices of the keys' triangles. Keys are in the order of their faces
// here (not yet sorted), so that neighbours' reads and writes lie together.
__global__ void mark_seen_kernel(const int32_t* __restrict__ triangles, int64_t K, const int64_t* __restrict__ count,
                                 const int32_t* __restrict__ faces, int64_t F, int64_t V, uint8_t* __restrict__ seen) {
  const int64_t n = count ? min(max(*count, (int64_t)0), K) : K;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const int32_t f = __ldg(triangles + k);
    if ((uint64_t)f >= (uint64_t)F || (k > 0 && __ldg(triangles + k - 1) == f)) continue;  // its first key marks
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int32_t v = __ldg(faces + 3 * (int64_t)f + c);
      if ((uint64_t)v < (uint64_t)V) seen[v] = 1;
    }
  }
}

template <int kCoeff>
__global__ void __launch_bounds__(kColourThreads)
    grid_sh_colors_kernel(const float* __restrict__ gsh, int64_t G, const int32_t* __restrict__ sources, int64_t V,
                          const int32_t* __restrict__ count, const int32_t* __restrict__ voff, int S,
                          const float* __restrict__ verts, const float* __restrict__ campos, int B,
                          const uint8_t* __restrict__ seen, float* __restrict__ out) {
  const int64_t n = count ? min((int64_t)max(*count, 0), V) : V;
  if (voff == nullptr) {  // vertex order: a CTA takes kColourThreads vertices
    const int64_t v = blockIdx.x * (int64_t)kColourThreads + threadIdx.x;
    if (v < n && (!seen || seen[v])) grid_sh_vertex<kCoeff>(gsh, G, sources, V, verts, campos, B, v, out);
    return;
  }
  __shared__ int ends[kColourShells];       // vertices of the tile up to and with shell s
  __shared__ int32_t starts[kColourShells];  // shell s's first vertex of the tile
  if (threadIdx.x < 32) {
    const int64_t e0 = blockIdx.x * (int64_t)kColourTile, e1 = min(e0 + kColourTile, G);
    const int s = threadIdx.x;
    const int64_t first = s < S ? __ldg(voff + (int64_t)s * G + e0) : 0;
    const int64_t last = s < S ? min((int64_t)__ldg(voff + (int64_t)s * G + e1), n) : 0;
    ends[s] = warp_inclusive_sum((int)max(last - first, (int64_t)0));
    starts[s] = (int32_t)first;
  }
  __syncthreads();
  const int total = ends[kColourShells - 1];
  for (int r = threadIdx.x; r < total; r += kColourThreads) {
    int s = 0;  // the first shell that ends past r
#pragma unroll
    for (int step = kColourShells / 2; step > 0; step >>= 1)
      if (ends[s + step - 1] <= r) s += step;
    const int64_t v = starts[s] + (int64_t)(r - (s > 0 ? ends[s - 1] : 0));
    if (!seen || seen[v]) grid_sh_vertex<kCoeff>(gsh, G, sources, V, verts, campos, B, v, out);
  }
}

// Backward: grid vertex x's SH gradient is sum over its list entries (v, t)
// of weighted(d sh_v), with d sh_v[k] = sum_b basis_k(dir_bv) d rgb_bv
// [rgb_bv > 0] formed on the fly (the sums of sh_backward_kernel, cameras in
// order, then of vertex_sh_gather_kernel, entries in list order: the same
// bits without the [C, V, 3] rows). One thread per (group of kRowsPerThread
// rows, grid vertex); consecutive threads write consecutive grid vertices of
// each row. Rows k >= n_coeff (up to C) are written as zeros.
// A CTA takes kShX consecutive grid vertices; their list entries are
// contiguous. In rounds of kShThreads entries, thread i forms entry i's
// weighted SH gradient (all rows: the per-vertex d sh_v of sh_backward_kernel,
// cameras in order, then weighted by the entry's (t, origin)) in shared
// memory, unless no camera sees the vertex (most of a large scene's: its
// entry adds nothing); then thread (row half h, grid vertex x) adds x's entries
// of the round to its 8 rows in list order. The sums stay in shared memory,
// which leaves registers for six CTAs to an SM, and are written by consecutive
// floats. The same sums in the same order as sh_backward_kernel +
// vertex_sh_gather_kernel. Bound by the latency of the scattered reads (list
// entry, then vertex, then colour): 2.60 ms at 512^3, 16 shells, 4 cameras with
// the sums in registers (two CTAs' worth of threads) and every entry added,
// now 1.92.
constexpr int kShThreads = 128;
constexpr int kShX = 64;
constexpr int kShStride = 49;  // 48 values per entry; odd stride spreads rows over banks
constexpr int kShCameras = 4;  // cameras whose gradients are loaded side by side

// False (nothing written) when no camera passes a gradient to the vertex.
template <bool kPacked>
__device__ __forceinline__ bool entry_sh_gradient(int2 e, int64_t V, const float* __restrict__ verts, int n_coeff,
                                                  const float* __restrict__ campos, int B,
                                                  const float* __restrict__ colors,
                                                  const float* __restrict__ dcolors, float* __restrict__ out) {
  const int64_t vi = e.x & 0x7fffffff;
  const bool origin = e.x < 0;
  const float t = __int_as_float(e.y);
  float d[16][3];
  bool seen = false;
  float px = 0.f, py = 0.f, pz = 0.f;
  for (int b0 = 0; b0 < B; b0 += kShCameras) {
    float g[kShCameras][3];
#pragma unroll
    for (int j = 0; j < kShCameras; ++j) {
      g[j][0] = g[j][1] = g[j][2] = 0.0f;
      if (b0 + j < B) colour_gradient<kPacked>(dcolors, (int64_t)(b0 + j) * V + vi, g[j]);
    }
#pragma unroll
    for (int j = 0; j < kShCameras; ++j) {
      if (g[j][0] == 0.0f && g[j][1] == 0.0f && g[j][2] == 0.0f) continue;  // also every camera past B
      const int64_t o = (int64_t)(b0 + j) * V + vi;
      bool any = false;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        g[j][c] = __ldg(colors + 3 * o + c) > 0.0f ? g[j][c] : 0.0f;
        any |= g[j][c] != 0.0f;
      }
      if (!any) continue;
      if (!seen) {
        seen = true;
        px = __ldg(verts + 3 * vi);
        py = __ldg(verts + 3 * vi + 1);
        pz = __ldg(verts + 3 * vi + 2);
#pragma unroll
        for (int k = 0; k < 16; ++k) d[k][0] = d[k][1] = d[k][2] = 0.f;
      }
      float dx, dy, dz;
      view_dir_at(px, py, pz, campos + 3 * (b0 + j), dx, dy, dz);
      float basis[16];
      sh_basis(dx, dy, dz, n_coeff, basis);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        if (k < n_coeff) {
#pragma unroll
          for (int c = 0; c < 3; ++c) d[k][c] += basis[k] * g[j][c];
        }
      }
    }
  }
  if (!seen) return false;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
#pragma unroll
    for (int c = 0; c < 3; ++c) out[3 * k + c] = weighted(d[k][c], t, origin);
  }
  return true;
}

template <bool kPacked>
__global__ void __launch_bounds__(kShThreads, 5)
    grid_sh_colors_backward_kernel(const int32_t* __restrict__ offsets, const int2* __restrict__ list, int64_t G,
                                   int64_t V, const float* __restrict__ verts, int C, int n_coeff,
                                   const float* __restrict__ campos, int B, const float* __restrict__ colors,
                                   const float* __restrict__ dcolors, float* __restrict__ gdsh) {
  __shared__ float s_grad[kShThreads * kShStride];
  __shared__ float s_sum[kShX * kShStride];
  __shared__ uint32_t s_seen[kShThreads / 32];
  const int tid = threadIdx.x;
  const int half = tid / kShX, xl = tid % kShX;  // rows 8*half .. 8*half+7 of grid vertex x0 + xl
  const int64_t x0 = (int64_t)blockIdx.x * kShX, x = x0 + xl;
  const int32_t e_begin = __ldg(offsets + x0), e_end = __ldg(offsets + min(x0 + kShX, G));
  const int32_t my_begin = x < G ? __ldg(offsets + x) : 0, my_end = x < G ? __ldg(offsets + x + 1) : 0;
  float* sum = s_sum + xl * kShStride + 24 * half;
#pragma unroll
  for (int j = 0; j < 24; ++j) sum[j] = 0.f;
  for (int32_t base = e_begin; base < e_end; base += kShThreads) {
    const bool seen = base + tid < e_end && entry_sh_gradient<kPacked>(__ldg(list + base + tid), V, verts, n_coeff, campos, B,
                                                                       colors, dcolors, s_grad + tid * kShStride);
    const uint32_t word = __ballot_sync(0xffffffffu, seen);
    if ((tid & 31) == 0) s_seen[tid >> 5] = word;
    __syncthreads();
    const int32_t lo = max(my_begin, base) - base, hi = min(my_end, base + kShThreads) - base;
    for (int32_t q = lo; q < hi; ++q) {
      if (!((s_seen[q >> 5] >> (q & 31)) & 1u)) continue;
      const float* src = s_grad + q * kShStride + 24 * half;
#pragma unroll
      for (int j = 0; j < 24; ++j) sum[j] += src[j];
    }
    __syncthreads();
  }
  __syncthreads();
  const int floats = 3 * (int)min((int64_t)kShX, G - x0);
  for (int f = tid; f < floats; f += kShThreads) {
    const int q = f / 3, c = f - 3 * q;
    for (int k = 0; k < min(C, 16); ++k)
      gdsh[(int64_t)k * 3 * G + 3 * x0 + f] = k < n_coeff ? s_sum[q * kShStride + 3 * k + c] : 0.f;
  }
}

// Two-pass form of the same backward (with scratch): pass 1, one thread per
// live vertex v, forms d sh_v (cameras in order, as sh_backward_kernel) once
// into a vertex-major array [V][16][3], for the vertices that a camera passes a
// gradient to (marked in `seen`; the others' rows are neither written nor
// read: most of a large scene's); pass 2, one thread per (8-row half h, grid
// vertex x), sums x's list entries of rows 8h .. 8h + 7 (96 contiguous bytes
// per entry) weighted, in list order. The same bits as the one-pass kernel,
// with each vertex's gradient formed once instead of once per entry. With
// every row written and read, and the results stored by threads 24 B apart,
// the two took 38 + 51 us at 256^3, 8 shells, 4 cameras and 0.92 + 1.16 ms at
// 512^3, 16 shells; now 43 + 46 us and 0.66 + 0.60 ms.
constexpr int kShGradThreads = 128;

template <bool kPacked>
__global__ void __launch_bounds__(kShGradThreads)
    vertex_sh_grad_kernel(const float* __restrict__ verts, int64_t V, const int32_t* __restrict__ count,
                          int n_coeff, const float* __restrict__ campos, int B, const float* __restrict__ colors,
                          const float* __restrict__ dcolors, float4* __restrict__ out,
                          uint8_t* __restrict__ seen) {
  // Each round, the CTA's kShGradThreads consecutive vertices form their
  // rows in shared memory, then write them as one contiguous block (full
  // 128-byte lines, where each thread's own 192-byte row would be written
  // 16 bytes at a time at a 192-byte stride).
  __shared__ float4 s_rows[kShGradThreads * 12];
  __shared__ uint32_t s_seen[kShGradThreads / 32];
  const int64_t n = count ? min((int64_t)max(*count, 0), V) : V;
  for (int64_t v0 = (int64_t)blockIdx.x * kShGradThreads; v0 < n; v0 += (int64_t)gridDim.x * kShGradThreads) {
    const int64_t v = v0 + threadIdx.x;
    bool any_camera = false;
    if (v < n) {
      const float px = __ldg(verts + 3 * v), py = __ldg(verts + 3 * v + 1), pz = __ldg(verts + 3 * v + 2);
      float d[16][3];
#pragma unroll
      for (int k = 0; k < 16; ++k) d[k][0] = d[k][1] = d[k][2] = 0.f;
      for (int b0 = 0; b0 < B; b0 += kShCameras) {
        float g[kShCameras][3];
#pragma unroll
        for (int j = 0; j < kShCameras; ++j) {
          g[j][0] = g[j][1] = g[j][2] = 0.0f;
          if (b0 + j < B) colour_gradient<kPacked>(dcolors, (int64_t)(b0 + j) * V + v, g[j]);
        }
#pragma unroll
        for (int j = 0; j < kShCameras; ++j) {
          if (g[j][0] == 0.0f && g[j][1] == 0.0f && g[j][2] == 0.0f) continue;  // also every camera past B
          const int64_t o = (int64_t)(b0 + j) * V + v;
          bool any = false;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            g[j][c] = __ldg(colors + 3 * o + c) > 0.0f ? g[j][c] : 0.0f;
            any |= g[j][c] != 0.0f;
          }
          if (!any) continue;
          any_camera = true;
          float dx, dy, dz;
          view_dir_at(px, py, pz, campos + 3 * (b0 + j), dx, dy, dz);
          float basis[16];
          sh_basis(dx, dy, dz, n_coeff, basis);
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            if (k < n_coeff) {
#pragma unroll
              for (int c = 0; c < 3; ++c) d[k][c] += basis[k] * g[j][c];
            }
          }
        }
      }
      seen[v] = any_camera ? 1 : 0;
      if (any_camera) {
        float4* row = s_rows + threadIdx.x * 12;
#pragma unroll
        for (int q = 0; q < 12; ++q) {
          const int j = 4 * q;
          row[q] = make_float4(d[j / 3][j % 3], d[(j + 1) / 3][(j + 1) % 3], d[(j + 2) / 3][(j + 2) % 3],
                               d[(j + 3) / 3][(j + 3) % 3]);
        }
      }
    }
    const uint32_t word = __ballot_sync(0xffffffffu, any_camera);
    if ((threadIdx.x & 31) == 0) s_seen[threadIdx.x >> 5] = word;
    __syncthreads();
    const int rows = (int)min((int64_t)kShGradThreads, n - v0);
    for (int i = threadIdx.x; i < rows * 12; i += kShGradThreads) {
      const int r = i / 12;
      if ((s_seen[r >> 5] >> (r & 31)) & 1u) out[v0 * 12 + i] = s_rows[i];
    }
    __syncthreads();  // the shared rows are written again by the next round
  }
}

constexpr int kShGatherThreads = 256, kShGatherAhead = 4;

__global__ void __launch_bounds__(kShGatherThreads)
    grid_sh_gather_kernel(const int32_t* __restrict__ offsets, const int2* __restrict__ list, int64_t G,
                          const float4* __restrict__ dsh, const uint8_t* __restrict__ seen, int C, int n_coeff,
                          float* __restrict__ gdsh) {
  // Adjacent threads take the two halves of one grid vertex, so a vertex's
  // 192-byte gradient row is read by neighbouring lanes together; the CTA's
  // sums are stored by consecutive floats.
  constexpr int kX = kShGatherThreads / 2;
  __shared__ float s_sum[kX * kShStride];
  const int half = threadIdx.x & 1, xl = threadIdx.x >> 1;
  const int64_t x0 = blockIdx.x * (int64_t)kX, x = x0 + xl;
  float acc[24];
#pragma unroll
  for (int j = 0; j < 24; ++j) acc[j] = 0.f;
  const int32_t end = x < G ? __ldg(offsets + x + 1) : 0;
  for (int32_t q0 = x < G ? __ldg(offsets + x) : 0; q0 < end; q0 += kShGatherAhead) {
    int2 e[kShGatherAhead];
    bool use[kShGatherAhead];
#pragma unroll
    for (int j = 0; j < kShGatherAhead; ++j) e[j] = __ldg(list + min(q0 + j, end - 1));
#pragma unroll
    for (int j = 0; j < kShGatherAhead; ++j) use[j] = q0 + j < end && __ldg(seen + (e[j].x & 0x7fffffff)) != 0;
#pragma unroll
    for (int j = 0; j < kShGatherAhead; ++j) {
      if (!use[j]) continue;
      const bool origin = e[j].x < 0;
      const float t = __int_as_float(e[j].y);
      const float4* src = dsh + (int64_t)(e[j].x & 0x7fffffff) * 12 + 6 * half;
      float4 val[6];
#pragma unroll
      for (int r = 0; r < 6; ++r) val[r] = __ldg(src + r);
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        acc[4 * r + 0] += weighted(val[r].x, t, origin);
        acc[4 * r + 1] += weighted(val[r].y, t, origin);
        acc[4 * r + 2] += weighted(val[r].z, t, origin);
        acc[4 * r + 3] += weighted(val[r].w, t, origin);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 24; ++j) s_sum[xl * kShStride + 24 * half + j] = acc[j];
  __syncthreads();
  const int floats = 3 * (int)min((int64_t)kX, G - x0);
  for (int f = threadIdx.x; f < floats; f += kShGatherThreads) {
    const int q = f / 3, c = f - 3 * q;
    for (int k = 0; k < min(C, 16); ++k)
      gdsh[(int64_t)k * 3 * G + 3 * x0 + f] = k < n_coeff ? s_sum[q * kShStride + 3 * k + c] : 0.f;
  }
}

size_t vertex_grad_bytes(int64_t G, int64_t V, int32_t** counts, int2** list, uint32_t** segments, void** scan_ws,
                         size_t* scan_bytes, char* base) {
  size_t off = 256;  // the workspace status word
  auto take = [&](size_t bytes) {
    char* q = base ? base + off : nullptr;
    off += (bytes + 255) & ~(size_t)255;
    return q;
  };
  char* c = take((size_t)(G + 1) * sizeof(int32_t));
  char* l = take((size_t)2 * (V > 0 ? V : 0) * sizeof(int2));
  char* seg = take((size_t)G * sizeof(uint32_t));
  const size_t sb = mt_scan_workspace_bytes(G + 1);
  char* sw = take(sb);
  if (counts) *counts = reinterpret_cast<int32_t*>(c);
  if (list) *list = reinterpret_cast<int2*>(l);
  if (segments) *segments = reinterpret_cast<uint32_t*>(seg);
  if (scan_ws) *scan_ws = sw;
  if (scan_bytes) *scan_bytes = sb;
  return off;
}

// ---------------------------------------------------------------------------
// count_triangle_faces.slang:15-50: cube code bit i <=> corner i >= iso with
// corner order (origin, +x, +xy, +y, +z, +xz, +xyz, +yz).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void load_cube(const float* __restrict__ sdf, const int32_t* __restrict__ lower, int64_t G,
                                          const int32_t* __restrict__ upper, int64_t Nv, int64_t v, float (&cube)[8]) {
  cube[0] = __ldg(sdf + __ldg(lower + v));
  cube[1] = __ldg(sdf + __ldg(lower + G + v));
  cube[2] = __ldg(sdf + __ldg(upper + 3 * Nv + v));
  cube[3] = __ldg(sdf + __ldg(lower + 2 * G + v));
  cube[4] = __ldg(sdf + __ldg(lower + 3 * G + v));
  cube[5] = __ldg(sdf + __ldg(upper + 2 * Nv + v));
  cube[6] = __ldg(sdf + __ldg(upper + v));
  cube[7] = __ldg(sdf + __ldg(upper + Nv + v));
}

// Count: int32_t (with the closing zero), or uint8_t for mt_exclusive_scan_bytes.
template <typename Count>
__global__ void count_faces_kernel(const float* __restrict__ sdf, const int32_t* __restrict__ lower, int64_t G,
                                   const int32_t* __restrict__ upper, int64_t Nv,
                                   const float* __restrict__ level_sets, int S, Count* __restrict__ counts,
                                   uint8_t* __restrict__ codes) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < Nv; v += (int64_t)gridDim.x * blockDim.x) {
    float cube[8];
    load_cube(sdf, lower, G, upper, Nv, v, cube);
    for (int s = 0; s < S; ++s) {
      const float iso = __ldg(level_sets + s);
      uint32_t code = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) code |= (uint32_t)(cube[q] >= iso) << q;
      codes[(int64_t)s * Nv + v] = (uint8_t)code;
      counts[(int64_t)s * Nv + v] = c_mc_count[code];
    }
  }
  if (sizeof(Count) == 4 && blockIdx.x == 0 && threadIdx.x == 0) counts[(int64_t)S * Nv] = 0;
}

// ---------------------------------------------------------------------------
// create_triangle_faces.slang:5-78. Edge id -> owning entry (self or upper
// neighbour) -> that entry's vertices at this level set -> the one whose
// type is the edge's axis. Triangles are written in reversed slot order.
// ---------------------------------------------------------------------------
// Writes only faces below F and searches only vertices below V (the
// buffers' capacities); with consistent offsets neither bound is reached.
//
// Work is dealt by triangle: a CTA reads kPer consecutive (shell, voxel) items
// (shell-major, the order of the slot offsets) for each of its threads, marks
// each of their triangles with its item in shared memory (at most 5 to an item;
// their slots are contiguous) and gives the triangles to its threads in turn,
// which have all of an item's look-ups once for three edges and the loads of the
// three side by side. Types are read where a caller has no crossings (an entry's
// up to three side by side). Bound by its instructions: dealt by slots, with a
// look-up of item, table and 64-bit addresses for each, 822 us at 512^3,
// 16 shells (24 M faces), 382 at 8 shells, 35 at 256^3, 8 shells; now 418, 203
// and 17 (with 4, 2 and 1 items to a thread 457, 570 and 626 at 16 shells). Grids
// that do not give every SM two CTAs of 8 items to a thread take one item to a
// thread: a 64^3 sphere's shell 5 us, with 8 items 9.
constexpr int kFaceThreads = 256;

template <bool kCrossings, int kPer>
__global__ void __launch_bounds__(kFaceThreads)
    create_faces_kernel(const int32_t* __restrict__ neighbors, const int32_t* __restrict__ indices, int64_t Nv,
                        int64_t G, int64_t V, const int32_t* __restrict__ voff, const uint8_t* __restrict__ types,
                        const uint8_t* __restrict__ codes, int S, const int32_t* __restrict__ foff, int64_t F,
                        int32_t* __restrict__ faces, int32_t* __restrict__ voxel_indices) {
  constexpr int kWarps = kFaceThreads / 32, kItems = kFaceThreads * kPer;
  __shared__ uint64_t s_edges[256];
  __shared__ uint8_t s_count[256];  // triangles
  __shared__ int8_t s_owner[12];
  __shared__ uint8_t s_axis[12];
  __shared__ int s_warp[kWarps];
  __shared__ uint8_t s_code[kItems];
  __shared__ uint16_t s_first[kItems];     // an item's first triangle in the CTA's
  __shared__ uint16_t s_item[kItems * 5];  // item of each triangle
  for (int i = threadIdx.x; i < 256; i += kFaceThreads) {
    s_edges[i] = c_mc_edges[i];
    s_count[i] = c_mc_count[i] / 3;
  }
  if (threadIdx.x < 12) {
    s_owner[threadIdx.x] = c_mc_owner[threadIdx.x];
    s_axis[threadIdx.x] = c_mc_axis[threadIdx.x];
  }
  const int64_t total = (int64_t)S * Nv;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t step = (int64_t)gridDim.x * kItems;
  const int64_t step_shells = step / Nv, step_voxels = step - step_shells * Nv;
  int64_t base = blockIdx.x * (int64_t)kItems;
  int64_t first_shell = base / Nv, first_voxel = base - first_shell * Nv;
  const int own = threadIdx.x * kPer;  // the thread's items are own .. own + kPer - 1
  uint32_t next[kPer];
  auto read = [&](int64_t from) {
#pragma unroll
    for (int k = 0; k < kPer; ++k) next[k] = from + own + k < total ? (uint32_t)__ldg(codes + from + own + k) : 0u;
  };
  read(base);
  int32_t next_slot = base < total ? __ldg(foff + base) : 0;
  __syncthreads();
  for (; base < total; base += step) {
    uint32_t code[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) code[k] = next[k];
    const int64_t first_tri = next_slot / 3;
    read(base + step);
    next_slot = base + step < total ? __ldg(foff + base + step) : 0;
    int n = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) n += s_count[code[k]];
    const int incl = warp_inclusive_sum(n);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();  // also: the last step's triangles are done
    int before = incl - n, span = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      before += w < warp ? s_warp[w] : 0;
      span += s_warp[w];
    }
    if (n > 0) {
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const int many = s_count[code[k]];
        s_code[own + k] = (uint8_t)code[k];
        s_first[own + k] = (uint16_t)before;
        for (int j = 0; j < many; ++j) s_item[before++] = (uint16_t)(own + k);
      }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < span; q += kFaceThreads) {
      const int item = s_item[q];
      int64_t v = first_voxel + item;
      int64_t row = first_shell * G;  // of the shell's vertex offsets
      while (v >= Nv) {  // at most kItems / Nv steps
        v -= Nv;
        row += G;
      }
      const uint32_t edges = (uint32_t)(s_edges[s_code[item]] >> (12 * (q - s_first[item])));
      int64_t at[3];  // each edge's entry, in the shell's row
      uint32_t axis[3], m[3];
      int32_t start[3];
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const int eid = (int)((edges >> (4 * e)) & 15u);
        const int owner = s_owner[eid];
        axis[e] = s_axis[eid];
        at[e] = row + ((owner < 0) ? v : (int64_t)__ldg(neighbors + (int64_t)owner * Nv + v));
      }
      const int32_t voxel = __ldg(indices + v);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        start[e] = __ldg(voff + at[e]);
        if constexpr (kCrossings) m[e] = (uint32_t)__ldg(types + at[e]);
      }
      const int64_t tri = first_tri + q;
      if ((uint64_t)tri >= (uint64_t)F) continue;
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        // The entry's vertex of the edge's axis (there is one); vertices past
        // the capacity were not written.
        int32_t target = -1;
        if constexpr (kCrossings) {
          const int32_t found = start[e] + __popc(m[e] & ((1u << axis[e]) - 1u));
          if (((m[e] >> axis[e]) & 1u) && found < V) target = found;
        } else {
          const int32_t count = __ldg(voff + at[e] + 1) - start[e];
          uint32_t type[3];
#pragma unroll
          for (int i = 0; i < 3; ++i)
            type[i] = i < count && (int64_t)start[e] + i < V ? (uint32_t)__ldg(types + start[e] + i) : 255u;
#pragma unroll
          for (int i = 2; i >= 0; --i)
            if (type[i] == axis[e]) target = start[e] + i;
        }
        faces[tri * 3 + 2 - e] = target;
      }
      voxel_indices[tri] = voxel;
    }
    first_shell += step_shells;
    first_voxel += step_voxels;
    if (first_voxel >= Nv) {
      first_voxel -= Nv;
      ++first_shell;
    }
  }
}

template <bool kCrossings>
int launch_create_faces(const int32_t* neighbors, const int32_t* indices, int64_t Nv, int64_t G, int64_t V,
                        const int32_t* voff, const uint8_t* types, const uint8_t* codes, int S, const int32_t* foff,
                        int64_t F, int32_t* faces, int32_t* voxel_indices, cudaStream_t stream) {
  const int64_t total = (int64_t)S * Nv;
  auto launch = [&](auto per) {
    constexpr int kPer = decltype(per)::value;
    const int64_t tiles = (total + kFaceThreads * kPer - 1) / (kFaceThreads * kPer);
    create_faces_kernel<kCrossings, kPer><<<grid_stride_blocks(tiles, 1), kFaceThreads, 0, stream>>>(
        neighbors, indices, Nv, G, V, voff, types, codes, S, foff, F, faces, voxel_indices);
  };
  if (total >= (int64_t)2 * kSmCount * 8 * kFaceThreads) launch(std::integral_constant<int, 8>{});
  else launch(std::integral_constant<int, 1>{});
  MT_CHECK_LAUNCH();
  return MT_OK;
}

// ---------------------------------------------------------------------------
// triangle_extraction/compute_sdf_regularizers.slang:18-128. Per voxel: the
// Eikonal terms of the trilinear SDF's gradient at the voxel centre (grid
// units) and a Laplacian curvature term at its +xyz corner. The operation
// order is the reference's (this unit is compiled without contraction).
// ---------------------------------------------------------------------------
struct VoxelCorners {
  int32_t i000, i001, i010, i100, i111, i110, i101, i011;  // grid vertex ids
  float d000, d001, d010, d100, d111, d110, d101, d011;
};

__device__ __forceinline__ VoxelCorners load_voxel_corners(const float* __restrict__ sdf,
                                                           const int32_t* __restrict__ lower, int64_t G,
                                                           const int32_t* __restrict__ upper, int64_t Nv, int64_t v) {
  VoxelCorners c;
  c.i000 = __ldg(lower + v);
  c.i001 = __ldg(lower + G + v);
  c.i010 = __ldg(lower + 2 * G + v);
  c.i100 = __ldg(lower + 3 * G + v);
  c.i111 = __ldg(upper + v);
  c.i110 = __ldg(upper + Nv + v);
  c.i101 = __ldg(upper + 2 * Nv + v);
  c.i011 = __ldg(upper + 3 * Nv + v);
  c.d000 = __ldg(sdf + c.i000);
  c.d001 = __ldg(sdf + c.i001);
  c.d010 = __ldg(sdf + c.i010);
  c.d100 = __ldg(sdf + c.i100);
  c.d111 = __ldg(sdf + c.i111);
  c.d110 = __ldg(sdf + c.i110);
  c.d101 = __ldg(sdf + c.i101);
  c.d011 = __ldg(sdf + c.i011);
  return c;
}

// Trilinear gradient at (0.5, 0.5, 0.5): weights (1 - t)(1 - t), t(1 - t), ...
// are all 0.25; the sums keep the reference's association.
__device__ __forceinline__ void centre_gradient(const VoxelCorners& c, float& dx, float& dy, float& dz) {
  const float t = 0.5f, t1 = 1.0f - t;
  const float w11 = t1 * t1, w01 = t * t1, w10 = t1 * t, w00 = t * t;
  dx = w11 * (c.d001 - c.d000) + w01 * (c.d011 - c.d010) + w10 * (c.d101 - c.d100) + w00 * (c.d111 - c.d110);
  dy = w11 * (c.d010 - c.d000) + w01 * (c.d011 - c.d001) + w10 * (c.d110 - c.d100) + w00 * (c.d111 - c.d101);
  dz = w11 * (c.d100 - c.d000) + w01 * (c.d101 - c.d001) + w10 * (c.d110 - c.d010) + w00 * (c.d111 - c.d011);
}

// stable_norm of compute_sdf_regularizers.slang:3-16.
__device__ __forceinline__ float stable_norm(float a, float b, float c) {
  const float scale = fmaxf(fmaxf(fabsf(a), fabsf(b)), fabsf(c));
  if (scale < 1e-10f) return 0.0f;
  const float inv = 1.0f / scale;
  const float sa = inv * a, sb = inv * b, sc = inv * c;
  return scale * sqrtf(sa * sa + sb * sb + sc * sc);
}

// Curvature sum: +yz, +xz, +xy corners, the present lower corners (+x, +y,
// +z) of the +xyz neighbour entry, minus (count) x the +xyz corner.
__device__ __forceinline__ float curvature_sum(const float* __restrict__ sdf, const VoxelCorners& c,
                                               const int32_t* __restrict__ lower, int64_t G, int32_t sub,
                                               int32_t (&extra)[3], int& counted) {
  float sum = c.d110 + c.d101 + c.d011;
  counted = 3;
#pragma unroll
  for (int i = 1; i < 4; ++i) {
    const int32_t corner = __ldg(lower + (int64_t)i * G + sub);
    extra[i - 1] = corner;
    if (corner >= 0) {
      sum += __ldg(sdf + corner);
      ++counted;
    }
  }
  return sum - (float)counted * c.d111;
}

__global__ void sdf_regularizers_kernel(const float* __restrict__ sdf, const int32_t* __restrict__ neighbors,
                                        const int32_t* __restrict__ lower, int64_t G,
                                        const int32_t* __restrict__ upper, int64_t Nv, int vx, int vy, int vz,
                                        float* __restrict__ eik_pos, float* __restrict__ eik_neg,
                                        float* __restrict__ curv) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < Nv; v += (int64_t)gridDim.x * blockDim.x) {
    const VoxelCorners c = load_voxel_corners(sdf, lower, G, upper, Nv, v);
    float dx, dy, dz;
    centre_gradient(c, dx, dy, dz);
    const float delta = stable_norm((float)vx * dx, (float)vy * dy, (float)vz * dz) - 1.0f;
    float pos = 0.0f, neg = 0.0f;
    if (delta < 0.0f) neg += delta * delta;
    if (delta > 0.0f) pos += delta * delta;
    eik_pos[v] = pos / 1.0f;
    eik_neg[v] = neg / 1.0f;
    int32_t extra[3];
    int counted;
    const float cs = curvature_sum(sdf, c, lower, G, __ldg(neighbors + 6 * Nv + v), extra, counted);
    curv[v] = cs * cs;
  }
}

// Adjoint (the reference differentiates the kernel automatically): with
// n = |(a, b, c)| and delta = n - 1, d delta / d a = a / n (0 when n is 0);
// each loss's gradient is scattered to the corners it reads.
__global__ void sdf_regularizers_backward_kernel(const float* __restrict__ sdf,
                                                 const int32_t* __restrict__ neighbors,
                                                 const int32_t* __restrict__ lower, int64_t G,
                                                 const int32_t* __restrict__ upper, int64_t Nv, int vx, int vy,
                                                 int vz, const float* __restrict__ g_pos,
                                                 const float* __restrict__ g_neg, const float* __restrict__ g_curv,
                                                 float* __restrict__ grad_sdf) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < Nv; v += (int64_t)gridDim.x * blockDim.x) {
    const VoxelCorners c = load_voxel_corners(sdf, lower, G, upper, Nv, v);
    float dx, dy, dz;
    centre_gradient(c, dx, dy, dz);
    const float a = (float)vx * dx, b = (float)vy * dy, cc = (float)vz * dz;
    const float n = stable_norm(a, b, cc);
    const float delta = n - 1.0f;
    float g_delta = 0.0f;
    if (g_pos && delta > 0.0f) g_delta += 2.0f * delta * g_pos[v];
    if (g_neg && delta < 0.0f) g_delta += 2.0f * delta * g_neg[v];
    float gd[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // 000 001 010 100 111 110 101 011
    if (g_delta != 0.0f && n > 0.0f) {
      const float gx = g_delta * a / n * (float)vx, gy = g_delta * b / n * (float)vy,
                  gz = g_delta * cc / n * (float)vz;
      const float w = 0.25f;
      // dx: +(001, 011, 101, 111), -(000, 010, 100, 110)
      gd[1] += w * gx; gd[7] += w * gx; gd[6] += w * gx; gd[4] += w * gx;
      gd[0] -= w * gx; gd[2] -= w * gx; gd[3] -= w * gx; gd[5] -= w * gx;
      // dy: +(010, 011, 110, 111), -(000, 001, 100, 101)
      gd[2] += w * gy; gd[7] += w * gy; gd[5] += w * gy; gd[4] += w * gy;
      gd[0] -= w * gy; gd[1] -= w * gy; gd[3] -= w * gy; gd[6] -= w * gy;
      // dz: +(100, 101, 110, 111), -(000, 001, 010, 011)
      gd[3] += w * gz; gd[6] += w * gz; gd[5] += w * gz; gd[4] += w * gz;
      gd[0] -= w * gz; gd[1] -= w * gz; gd[2] -= w * gz; gd[7] -= w * gz;
    }
    int32_t extra[3];
    int counted;
    const float cs = curvature_sum(sdf, c, lower, G, __ldg(neighbors + 6 * Nv + v), extra, counted);
    const float g_cs = g_curv ? 2.0f * cs * g_curv[v] : 0.0f;
    if (g_cs != 0.0f) {
      gd[5] += g_cs;
      gd[6] += g_cs;
      gd[7] += g_cs;
      gd[4] -= (float)counted * g_cs;
#pragma unroll
      for (int i = 0; i < 3; ++i)
        if (extra[i] >= 0) atomicAdd(grad_sdf + extra[i], g_cs);
    }
    const int32_t ids[8] = {c.i000, c.i001, c.i010, c.i100, c.i111, c.i110, c.i101, c.i011};
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (gd[q] != 0.0f) atomicAdd(grad_sdf + ids[q], gd[q]);
  }
}

// Last entry of every shell's block of an exclusive scan: the vertex and face
// boundaries of triangle_extraction/__init__.py:145-146 (faces / 3, floor),
// plus the face total of :131 (offsets are non-negative, so / is floor).
__global__ void shell_boundaries_kernel(const int32_t* __restrict__ voff, int64_t G,
                                        const int32_t* __restrict__ foff, int64_t Nv, int S,
                                        int32_t* __restrict__ vb, int32_t* __restrict__ fb,
                                        int32_t* __restrict__ num_faces) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < S) {
    vb[s] = G > 0 ? voff[(int64_t)(s + 1) * G] : 0;
    fb[s] = Nv > 0 ? foff[(int64_t)(s + 1) * Nv] / 3 : 0;
  }
  if (s == 0 && num_faces) *num_faces = foff[(int64_t)S * Nv] / 3;
}

__global__ void capacity_overflow_kernel(const int32_t* __restrict__ nv, int64_t cv, const int32_t* __restrict__ nf,
                                         int64_t cf, const int64_t* __restrict__ nk, int64_t ck,
                                         uint8_t* __restrict__ overflow) {
  bool over = false;
  if (nv) over |= (int64_t)*nv > cv;
  if (nf) over |= (int64_t)*nf > cf;
  if (nk) over |= *nk > ck;
  *overflow = over ? 1 : 0;
}

}  // namespace
}  // namespace mt

using namespace mt;

template <bool kPacked>
static int grid_sh_backward(const int32_t* list_offsets, const int32_t* list, int64_t G, int64_t V,
                               const float* vertices, int32_t C, int32_t sh_degree, const float* camera_positions,
                               int32_t B, const float* out_colors, const float* grad_colors,
                               float* grad_grid_spherical_harmonics, const int32_t* num_vertices, void* workspace,
                               size_t workspace_bytes, mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && V >= 0 && B >= 0 && sh_degree >= 0 && sh_degree <= 3);
  const int n = (sh_degree + 1) * (sh_degree + 1);
  MT_REQUIRE(C >= n);
  if (G == 0) return MT_OK;
  MT_REQUIRE(list_offsets && grad_grid_spherical_harmonics);
  // No cameras or vertices: every list sum is empty and the rows are zeros.
  const int Bn = V > 0 ? B : 0;
  MT_REQUIRE(Bn == 0 || (list && vertices && camera_positions && out_colors && grad_colors));
  MT_REQUIRE(!kPacked || (reinterpret_cast<uintptr_t>(grad_colors) & 15) == 0);
  cudaStream_t st = as_stream(stream);
  if (C > 16 && cudaMemsetAsync(grad_grid_spherical_harmonics + (size_t)16 * G * 3, 0,
                                (size_t)(C - 16) * G * 3 * sizeof(float), st) != cudaSuccess)
    return MT_ERR_CUDA;  // rows past degree 3's sixteen are zeros
  if (workspace && workspace_bytes >= mt_grid_sh_colors_backward_workspace_bytes(V) && Bn > 0) {
    float4* dsh = reinterpret_cast<float4*>(static_cast<char*>(workspace) + 256);
    MT_REQUIRE((reinterpret_cast<uintptr_t>(dsh) & 15) == 0);
    uint8_t* seen = reinterpret_cast<uint8_t*>(dsh + 12 * V);
    vertex_sh_grad_kernel<kPacked><<<grid_stride_blocks(V, kShGradThreads), kShGradThreads, 0, st>>>(
        vertices, V, num_vertices, n, camera_positions, Bn, out_colors, grad_colors, dsh, seen);
    MT_CHECK_LAUNCH();
    const int64_t blocks = (2 * G + kShGatherThreads - 1) / kShGatherThreads;
    MT_REQUIRE(blocks < ((int64_t)1 << 31));
    grid_sh_gather_kernel<<<(unsigned)blocks, kShGatherThreads, 0, st>>>(
        list_offsets, reinterpret_cast<const int2*>(list), G, dsh, seen, C, n, grad_grid_spherical_harmonics);
    MT_CHECK_LAUNCH();
    return MT_OK;
  }
  const int64_t xblocks = (G + kShX - 1) / kShX;
  MT_REQUIRE(xblocks < ((int64_t)1 << 31));
  grid_sh_colors_backward_kernel<kPacked><<<(unsigned)xblocks, kShThreads, 0, st>>>(
      list_offsets, reinterpret_cast<const int2*>(list), G, V, vertices, C, n, camera_positions, Bn, out_colors,
      grad_colors, grad_grid_spherical_harmonics);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

extern "C" {

int mt_count_grid(const int32_t* occupancy, int32_t I, int32_t J, int32_t KP, int32_t* vertex_occupancy,
                  int32_t* vertex_counts, int32_t* voxel_counts, mt_stream_t stream) {
  MT_REQUIRE(I >= 0 && J >= 0 && KP >= 0);
  MT_REQUIRE(vertex_occupancy && vertex_counts);
  MT_REQUIRE(occupancy || (int64_t)I * J * KP == 0);
  const int64_t total = (int64_t)(I + 1) * (J + 1) * (KP + 1);
  const int64_t lanes = (total + kOccupancyWords - 1) / kOccupancyWords * 32;
  vertex_occupancy_kernel<<<grid_stride_blocks(lanes, 256, 16), 256, 0, as_stream(stream)>>>(
      occupancy, I, J, KP, vertex_occupancy, vertex_counts, voxel_counts);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_compute_vertex_occupancy(const int32_t* occupancy, int32_t I, int32_t J, int32_t KP, int32_t* vertex_occupancy,
                                int32_t* vertex_counts, mt_stream_t stream) {
  return mt_count_grid(occupancy, I, J, KP, vertex_occupancy, vertex_counts, nullptr, stream);
}

int mt_count_occupancy(const int32_t* occupancy, int32_t I, int32_t J, int32_t KP, int32_t* voxel_counts,
                       mt_stream_t stream) {
  MT_REQUIRE(I >= 0 && J >= 0 && KP >= 0);
  MT_REQUIRE(voxel_counts);
  MT_REQUIRE(occupancy || (int64_t)I * J * KP == 0);
  const int64_t total = (int64_t)(I + 1) * (J + 1) * (KP + 1);
  count_occupancy_kernel<<<grid_stride_blocks(total, 256), 256, 0, as_stream(stream)>>>(occupancy, I, J, KP,
                                                                                       voxel_counts);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_create_voxels(const int32_t* occupancy, const int32_t* voxel_offsets, const int32_t* vertex_occupancy,
                     const int32_t* vertex_offsets, int32_t I, int32_t J, int32_t KP, int64_t num_voxels,
                     int64_t num_vertices, float* vertices, int32_t* neighbors, int32_t* lower_corners,
                     int32_t* upper_corners, int32_t* indices, mt_stream_t stream) {
  MT_REQUIRE(I >= 0 && J >= 0 && KP >= 0 && num_voxels >= 0 && num_vertices >= num_voxels);
  if (num_vertices == 0) return MT_OK;
  MT_REQUIRE(I > 0 && J > 0 && KP > 0);
  MT_REQUIRE(occupancy && voxel_offsets && vertex_occupancy && vertex_offsets && vertices && lower_corners);
  MT_REQUIRE(num_voxels == 0 || (neighbors && upper_corners && indices));
  MT_REQUIRE((int64_t)32 * KP * J * I < ((int64_t)1 << 31));
  VoxelGrid g{occupancy, voxel_offsets, vertex_occupancy, vertex_offsets, I, J, KP, num_voxels};
  const int64_t words = (int64_t)(I + 1) * (J + 1) * (KP + 1);
  const int threads = 32 * kVoxelWarps;  // a lane to a word; the words are below 2^29
  const unsigned blocks = (unsigned)((words + threads - 1) / threads);
  create_voxels_kernel<<<blocks, threads, 0, as_stream(stream)>>>(g, vertices, neighbors, lower_corners,
                                                                  upper_corners, indices, num_vertices);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_dilate_occupancy(const int32_t* occupancy, int32_t I, int32_t J, int32_t KP, int32_t dilation, int32_t* out,
                        mt_stream_t stream) {
  MT_REQUIRE(I >= 0 && J >= 0 && KP >= 0);
  MT_REQUIRE(dilation > 0 && dilation < 32);
  const int64_t total = (int64_t)I * J * KP;
  if (total == 0) return MT_OK;
  MT_REQUIRE(occupancy && out && occupancy != out);
  const int64_t lanes = (total + kDilateWords - 1) / kDilateWords * 32;
  dilate_kernel<<<grid_stride_blocks(lanes, 256, 128), 256, 0, as_stream(stream)>>>(occupancy, I, J, KP, dilation, out);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_count_triangle_vertices(const float* signed_distances, const int32_t* lower_corners, int64_t G,
                               const float* level_sets, int32_t S, int32_t* counts, mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && S >= 0 && counts);
  MT_REQUIRE(G == 0 || (signed_distances && lower_corners));
  MT_REQUIRE(S == 0 || level_sets);
  count_vertices_kernel<<<grid_stride_blocks(G, 256), 256, 0, as_stream(stream)>>>(signed_distances, lower_corners, G,
                                                                                  level_sets, S, counts);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_count_triangle_crossings(const float* signed_distances, const int32_t* lower_corners, int64_t G,
                                const float* level_sets, int32_t S, uint8_t* crossings, mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && S >= 0);
  if (G == 0 || S == 0) return MT_OK;
  MT_REQUIRE(signed_distances && lower_corners && level_sets && crossings);
  count_crossings_kernel<<<grid_stride_blocks(G, 256), 256, 0, as_stream(stream)>>>(signed_distances, lower_corners,
                                                                                   G, level_sets, S, crossings);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_create_triangle_vertices_live_t_backward(const float* grid_vertices, const float* grid_signed_distances,
                                                const float* grid_spherical_harmonics, int32_t C, int64_t G,
                                                const int32_t* vertex_sources, int64_t V, const int32_t* num_vertices,
                                                const float* grad_vertices, const float* grad_spherical_harmonics,
                                                float* grad_grid_signed_distances, mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && V >= 0 && C >= 1);
  if (V == 0 || G == 0 || (grad_vertices == nullptr && grad_spherical_harmonics == nullptr)) return MT_OK;
  MT_REQUIRE(grid_signed_distances && vertex_sources && grad_grid_signed_distances);
  MT_REQUIRE(grad_vertices == nullptr || grid_vertices != nullptr);
  MT_REQUIRE(grad_spherical_harmonics == nullptr || grid_spherical_harmonics != nullptr);
  live_t_backward_kernel<<<grid_stride_blocks(V, 256), 256, 0, as_stream(stream)>>>(
      grid_vertices, grid_signed_distances, grid_spherical_harmonics, C, G, vertex_sources, V, num_vertices,
      grad_vertices, grad_spherical_harmonics, grad_grid_signed_distances);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_create_triangle_vertices(const float* grid_vertices, const float* grid_signed_distances,
                                const float* grid_spherical_harmonics, int32_t C, const int32_t* lower_corners,
                                int64_t G, const float* level_sets, int32_t S, const int32_t* vertex_offsets,
                                int64_t V, const int32_t* num_vertices, float* vertices, float* signed_distances,
                                float* spherical_harmonics, uint8_t* vertex_types, int32_t* vertex_sources,
                                mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && S >= 0 && C >= 1 && V >= 0);
  if (G == 0 || S == 0 || V == 0) return MT_OK;
  MT_REQUIRE(grid_vertices && grid_signed_distances && lower_corners && level_sets && vertex_offsets && vertices &&
             signed_distances && vertex_types && vertex_sources);
  auto launch = [&](auto together) {
    create_vertices_kernel<decltype(together)::value><<<grid_stride_blocks(G, 128), 128, 0, as_stream(stream)>>>(
        grid_vertices, grid_signed_distances, lower_corners, G, level_sets, S, vertex_offsets, V, vertices,
        signed_distances, vertex_types, vertex_sources);
  };
  if (V > 2 * G) launch(std::true_type{});
  else launch(std::false_type{});
  MT_CHECK_LAUNCH();
  if (spherical_harmonics == nullptr) return MT_OK;  // rows left to mt_grid_sh_colors
  MT_REQUIRE(grid_spherical_harmonics);
  const int64_t blocks = (G + kRowTile - 1) / kRowTile;
  MT_REQUIRE(blocks < ((int64_t)1 << 31));
  if (12 * G < ((int64_t)1 << 32))
    interpolate_vertex_sh_kernel<uint32_t><<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(
        grid_spherical_harmonics, C, G, vertex_sources, V, num_vertices, vertex_offsets, S, spherical_harmonics);
  else
    interpolate_vertex_sh_kernel<int64_t><<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(
        grid_spherical_harmonics, C, G, vertex_sources, V, num_vertices, vertex_offsets, S, spherical_harmonics);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

size_t mt_create_triangle_vertices_backward_workspace_bytes(int64_t G, int64_t V) {
  if (G < 0 || V < 0) return 0;
  return vertex_grad_bytes(G, V, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
}

int mt_create_triangle_vertices_backward(const float* grid_signed_distances, int32_t C, const int32_t* lower_corners,
                                         int64_t G, const float* level_sets, int32_t S,
                                         const int32_t* vertex_offsets, const float* grad_vertices,
                                         const float* grad_signed_distances, const float* grad_spherical_harmonics,
                                         int64_t V, int32_t* corner_inverse, float* grad_grid_vertices,
                                         float* grad_grid_signed_distances, float* grad_grid_spherical_harmonics,
                                         void* workspace, size_t workspace_bytes, mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && S >= 0 && C >= 1 && V >= 0);
  if (G == 0) return MT_OK;
  MT_REQUIRE(grid_signed_distances && lower_corners && corner_inverse);
  MT_REQUIRE(grad_grid_signed_distances && grad_grid_spherical_harmonics);
  MT_REQUIRE(S == 0 || (level_sets && vertex_offsets));
  MT_REQUIRE(grad_vertices == nullptr || grad_grid_vertices != nullptr);
  cudaStream_t st = as_stream(stream);
  if (cudaMemsetAsync(corner_inverse, 0xff, (size_t)G * 4 * sizeof(int32_t), st) != cudaSuccess) return MT_ERR_CUDA;
  // With no level sets or no vertices, the gather writes zeros everywhere.
  const float* gv = V > 0 ? grad_vertices : nullptr;
  const float* gd = V > 0 ? grad_signed_distances : nullptr;
  const float* gs = V > 0 ? grad_spherical_harmonics : nullptr;
  const bool listed = S <= kShellsPerChunk && V < (int64_t)0x7fffffff && workspace &&
                      workspace_bytes >= mt_create_triangle_vertices_backward_workspace_bytes(G, V);
  int32_t* counts = nullptr;
  int2* list = nullptr;
  uint32_t* segments = nullptr;
  void* scan_ws = nullptr;
  size_t scan_bytes = 0;
  if (listed) vertex_grad_bytes(G, V, &counts, &list, &segments, &scan_ws, &scan_bytes, static_cast<char*>(workspace));
  invert_corners_kernel<<<grid_stride_blocks(G, 256), 256, 0, st>>>(lower_corners, G, corner_inverse, counts,
                                                                    segments);
  MT_CHECK_LAUNCH();
  if (!listed) {
    create_vertices_backward_kernel<<<grid_stride_blocks(G, 128), 128, 0, st>>>(
        grid_signed_distances, C, lower_corners, G, level_sets, S, vertex_offsets, corner_inverse, gv, gd, gs, V,
        grad_grid_vertices, grad_grid_signed_distances, grad_grid_spherical_harmonics);
    MT_CHECK_LAUNCH();
    return MT_OK;
  }
  entry_list_kernel<false><<<grid_stride_blocks(G, 256), 256, 0, st>>>(grid_signed_distances, lower_corners, G,
                                                                       level_sets, S, vertex_offsets, corner_inverse,
                                                                       V, counts, segments, nullptr);
  MT_CHECK_LAUNCH();
  const int rc = mt_exclusive_scan_i32(counts, G + 1, scan_ws, scan_bytes, stream);
  if (rc != MT_OK) return rc;
  entry_list_kernel<true><<<grid_stride_blocks(G, 256), 256, 0, st>>>(grid_signed_distances, lower_corners, G,
                                                                      level_sets, S, vertex_offsets, corner_inverse,
                                                                      V, counts, segments, list);
  MT_CHECK_LAUNCH();
  vertex_grads_from_list_kernel<<<grid_stride_blocks(G, 256), 256, 0, st>>>(counts, list, G, gv, gd,
                                                                            grad_grid_vertices,
                                                                            grad_grid_signed_distances);
  MT_CHECK_LAUNCH();
  const int64_t blocks = (3 * G + kGatherThreads - 1) / kGatherThreads;
  MT_REQUIRE(blocks < ((int64_t)1 << 31));
  vertex_sh_gather_kernel<<<(unsigned)blocks, kGatherThreads, 0, st>>>(gs, C, V, G, counts, list,
                                                                       grad_grid_spherical_harmonics);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_count_triangle_faces(const float* signed_distances, const int32_t* lower_corners, int64_t G,
                            const int32_t* upper_corners, int64_t Nv, const float* level_sets, int32_t S,
                            int32_t* face_counts, uint8_t* cell_codes, mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && Nv >= 0 && S >= 0 && face_counts);
  MT_REQUIRE(Nv == 0 || (signed_distances && lower_corners && upper_corners && cell_codes));
  MT_REQUIRE(S == 0 || level_sets);
  count_faces_kernel<<<grid_stride_blocks(Nv, 256), 256, 0, as_stream(stream)>>>(
      signed_distances, lower_corners, G, upper_corners, Nv, level_sets, S, face_counts, cell_codes);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_count_triangle_faces_bytes(const float* signed_distances, const int32_t* lower_corners, int64_t G,
                                  const int32_t* upper_corners, int64_t Nv, const float* level_sets, int32_t S,
                                  uint8_t* face_counts, uint8_t* cell_codes, mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && Nv >= 0 && S >= 0);
  MT_REQUIRE(Nv == 0 || (signed_distances && lower_corners && upper_corners && cell_codes));
  if (Nv == 0 || S == 0) return MT_OK;
  MT_REQUIRE(level_sets && face_counts);
  count_faces_kernel<<<grid_stride_blocks(Nv, 256), 256, 0, as_stream(stream)>>>(
      signed_distances, lower_corners, G, upper_corners, Nv, level_sets, S, face_counts, cell_codes);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_create_triangle_faces(const int32_t* neighbors, const int32_t* indices, int64_t Nv, int64_t G, int64_t V,
                             const int32_t* vertex_offsets, const uint8_t* vertex_types, const uint8_t* cell_codes,
                             int32_t S, const int32_t* face_offsets, int64_t F, int32_t* faces,
                             int32_t* voxel_indices, mt_stream_t stream) {
  MT_REQUIRE(Nv >= 0 && G >= 0 && V >= 0 && S >= 0 && F >= 0);
  if (Nv == 0 || S == 0 || F == 0) return MT_OK;
  MT_REQUIRE(neighbors && indices && vertex_offsets && vertex_types && cell_codes && face_offsets && faces &&
             voxel_indices);
  return launch_create_faces<false>(neighbors, indices, Nv, G, V, vertex_offsets, vertex_types, cell_codes, S, face_offsets,
                                    F, faces, voxel_indices, as_stream(stream));
}

int mt_create_triangle_faces_by_crossings(const int32_t* neighbors, const int32_t* indices, int64_t Nv, int64_t G,
                                          int64_t V, const int32_t* vertex_offsets, const uint8_t* crossings,
                                          const uint8_t* cell_codes, int32_t S, const int32_t* face_offsets, int64_t F,
                                          int32_t* faces, int32_t* voxel_indices, mt_stream_t stream) {
  MT_REQUIRE(Nv >= 0 && G >= 0 && V >= 0 && S >= 0 && F >= 0);
  if (Nv == 0 || S == 0 || F == 0) return MT_OK;
  MT_REQUIRE(neighbors && indices && vertex_offsets && crossings && cell_codes && face_offsets && faces &&
             voxel_indices);
  return launch_create_faces<true>(neighbors, indices, Nv, G, V, vertex_offsets, crossings, cell_codes, S, face_offsets,
                                    F, faces, voxel_indices, as_stream(stream));
}

int mt_compute_sdf_regularizers(const float* grid_signed_distances, const int32_t* voxel_neighbors,
                                const int32_t* voxel_lower_corners, int64_t G, const int32_t* voxel_upper_corners,
                                int64_t Nv, int32_t voxel_x, int32_t voxel_y, int32_t voxel_z,
                                float* eikonal_loss_pos, float* eikonal_loss_neg, float* curvature_loss,
                                mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && Nv >= 0);
  if (Nv == 0) return MT_OK;
  MT_REQUIRE(grid_signed_distances && voxel_neighbors && voxel_lower_corners && voxel_upper_corners &&
             eikonal_loss_pos && eikonal_loss_neg && curvature_loss);
  sdf_regularizers_kernel<<<grid_stride_blocks(Nv, 256), 256, 0, as_stream(stream)>>>(
      grid_signed_distances, voxel_neighbors, voxel_lower_corners, G, voxel_upper_corners, Nv, voxel_x, voxel_y,
      voxel_z, eikonal_loss_pos, eikonal_loss_neg, curvature_loss);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_compute_sdf_regularizers_backward(const float* grid_signed_distances, const int32_t* voxel_neighbors,
                                         const int32_t* voxel_lower_corners, int64_t G,
                                         const int32_t* voxel_upper_corners, int64_t Nv, int32_t voxel_x,
                                         int32_t voxel_y, int32_t voxel_z, const float* grad_eikonal_loss_pos,
                                         const float* grad_eikonal_loss_neg, const float* grad_curvature_loss,
                                         float* grad_grid_signed_distances, mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && Nv >= 0 && grad_grid_signed_distances);
  cudaStream_t st = as_stream(stream);
  if (G > 0 && cudaMemsetAsync(grad_grid_signed_distances, 0, (size_t)G * sizeof(float), st) != cudaSuccess)
    return MT_ERR_CUDA;
  if (Nv == 0) return MT_OK;
  MT_REQUIRE(grid_signed_distances && voxel_neighbors && voxel_lower_corners && voxel_upper_corners);
  sdf_regularizers_backward_kernel<<<grid_stride_blocks(Nv, 256), 256, 0, st>>>(
      grid_signed_distances, voxel_neighbors, voxel_lower_corners, G, voxel_upper_corners, Nv, voxel_x, voxel_y,
      voxel_z, grad_eikonal_loss_pos, grad_eikonal_loss_neg, grad_curvature_loss, grad_grid_signed_distances);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_shell_boundaries(const int32_t* vertex_offsets, int64_t G, const int32_t* face_offsets, int64_t Nv, int32_t S,
                        int32_t* vertex_boundaries, int32_t* face_boundaries, int32_t* num_faces,
                        mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && Nv >= 0 && S >= 0);
  if (S == 0 && !num_faces) return MT_OK;
  MT_REQUIRE(vertex_offsets && face_offsets);
  MT_REQUIRE(S == 0 || (vertex_boundaries && face_boundaries));
  shell_boundaries_kernel<<<grid_1d(S > 0 ? S : 1, 128), 128, 0, as_stream(stream)>>>(
      vertex_offsets, G, face_offsets, Nv, S, vertex_boundaries, face_boundaries, num_faces);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_capacity_overflow(const int32_t* num_vertices, int64_t vertex_capacity, const int32_t* num_faces,
                         int64_t face_capacity, const int64_t* num_keys, int64_t key_capacity, uint8_t* overflow,
                         mt_stream_t stream) {
  MT_REQUIRE(overflow);
  capacity_overflow_kernel<<<1, 1, 0, as_stream(stream)>>>(num_vertices, vertex_capacity, num_faces, face_capacity,
                                                          num_keys, key_capacity, overflow);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_vertex_grad_list_max_shells(void) { return kShellsPerChunk; }

// Workspace: status word, the segment words [G], the scan's scratch.
static size_t segment_bytes(int64_t G) { return ((size_t)G * sizeof(uint32_t) + 255) & ~(size_t)255; }

size_t mt_build_vertex_grad_list_workspace_bytes(int64_t G) {
  return 256 + segment_bytes(G) + mt_scan_workspace_bytes(G + 1);
}

int mt_build_vertex_grad_list(const float* grid_signed_distances, const int32_t* lower_corners, int64_t G,
                              const float* level_sets, int32_t S, const int32_t* vertex_offsets, int64_t V,
                              int32_t* corner_inverse, int32_t* list_offsets, int32_t* list, void* workspace,
                              size_t workspace_bytes, mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && S >= 0 && V >= 0);
  if (S > kShellsPerChunk || V >= (int64_t)0x7fffffff) return MT_ERR_TOO_LARGE;
  if (G == 0) return MT_OK;
  MT_REQUIRE(grid_signed_distances && lower_corners && corner_inverse && list_offsets && workspace);
  MT_REQUIRE(S == 0 || (level_sets && vertex_offsets));
  MT_REQUIRE(V == 0 || list);
  if (workspace_bytes < mt_build_vertex_grad_list_workspace_bytes(G)) return MT_ERR_WORKSPACE_TOO_SMALL;
  cudaStream_t st = as_stream(stream);
  char* ws = static_cast<char*>(workspace);
  uint32_t* segments = reinterpret_cast<uint32_t*>(ws + 256);
  const size_t scan_off = 256 + segment_bytes(G);
  if (cudaMemsetAsync(corner_inverse, 0xff, (size_t)G * 4 * sizeof(int32_t), st) != cudaSuccess) return MT_ERR_CUDA;
  invert_corners_kernel<<<grid_stride_blocks(G, 256), 256, 0, st>>>(lower_corners, G, corner_inverse, list_offsets,
                                                                    segments);
  MT_CHECK_LAUNCH();
  entry_list_kernel<false><<<grid_stride_blocks(G, 256), 256, 0, st>>>(
      grid_signed_distances, lower_corners, G, level_sets, S, vertex_offsets, corner_inverse, V, list_offsets,
      segments, nullptr);
  MT_CHECK_LAUNCH();
  const int rc = mt_exclusive_scan_i32(list_offsets, G + 1, ws + scan_off, workspace_bytes - scan_off, stream);
  if (rc != MT_OK) return rc;
  entry_list_kernel<true><<<grid_stride_blocks(G, 256), 256, 0, st>>>(
      grid_signed_distances, lower_corners, G, level_sets, S, vertex_offsets, corner_inverse, V, list_offsets,
      segments, reinterpret_cast<int2*>(list));
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_vertex_grads_from_list(const int32_t* list_offsets, const int32_t* list, int64_t G,
                              const float* grad_vertices, const float* grad_signed_distances,
                              float* grad_grid_vertices, float* grad_grid_signed_distances, mt_stream_t stream) {
  MT_REQUIRE(G >= 0);
  if (G == 0) return MT_OK;
  MT_REQUIRE(list_offsets && grad_grid_signed_distances);
  MT_REQUIRE(grad_vertices == nullptr || grad_grid_vertices != nullptr);
  vertex_grads_from_list_kernel<<<grid_stride_blocks(G, 256), 256, 0, as_stream(stream)>>>(
      list_offsets, reinterpret_cast<const int2*>(list), G, grad_vertices, grad_signed_distances, grad_grid_vertices,
      grad_grid_signed_distances);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_grid_sh_colors_of_seen(const float* grid_spherical_harmonics, int32_t C, int64_t G,
                              const int32_t* vertex_sources, int64_t V, const int32_t* num_vertices,
                              const int32_t* vertex_offsets, int32_t S, const float* vertices, int32_t sh_degree,
                              const float* camera_positions, int32_t B, const uint8_t* seen, float* out_colors,
                              mt_stream_t stream) {
  MT_REQUIRE(G >= 0 && V >= 0 && B >= 0 && S >= 0 && sh_degree >= 0 && sh_degree <= 3);
  const int n = (sh_degree + 1) * (sh_degree + 1);
  MT_REQUIRE(C >= n);
  if (V == 0 || B == 0) return MT_OK;
  MT_REQUIRE(grid_spherical_harmonics && vertex_sources && vertices && camera_positions && out_colors);
  const bool cached = 12 * G * n <= kColourCached;
  const int32_t* offsets = S <= kColourShells && !cached ? vertex_offsets : nullptr;
  const int64_t blocks = offsets ? (G + kColourTile - 1) / kColourTile : (V + kColourThreads - 1) / kColourThreads;
  MT_REQUIRE(blocks < ((int64_t)1 << 31));
  if (blocks == 0) return MT_OK;
  auto launch = [&](auto coeff) {
    grid_sh_colors_kernel<decltype(coeff)::value><<<(unsigned)blocks, kColourThreads, 0, as_stream(stream)>>>(
        grid_spherical_harmonics, G, vertex_sources, V, num_vertices, offsets, S, vertices, camera_positions, B, seen,
        out_colors);
  };
  switch (n) {
    case 1: launch(std::integral_constant<int, 1>{}); break;
    case 4: launch(std::integral_constant<int, 4>{}); break;
    case 9: launch(std::integral_constant<int, 9>{}); break;
    default: launch(std::integral_constant<int, 16>{}); break;
  }
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_mark_seen_vertices(const int32_t* triangles, int64_t K, const int64_t* num_keys, const int32_t* faces,
                          int64_t F, int64_t V, uint8_t* seen, mt_stream_t stream) {
  MT_REQUIRE(K >= 0 && F >= 0 && V >= 0);
  if (V == 0) return MT_OK;
  MT_REQUIRE(seen);
  if (cudaMemsetAsync(seen, 0, (size_t)V, as_stream(stream)) != cudaSuccess) return MT_ERR_CUDA;
  if (K == 0 || F == 0) return MT_OK;
  MT_REQUIRE(triangles && faces);
  mark_seen_kernel<<<grid_stride_blocks(K, 256), 256, 0, as_stream(stream)>>>(triangles, K, num_keys, faces, F, V,
                                                                             seen);
  MT_CHECK_LAUNCH();
  return MT_OK;
}

int mt_grid_sh_colors(const float* grid_spherical_harmonics, int32_t C, int64_t G, const int32_t* vertex_sources,
                      int64_t V, const int32_t* num_vertices, const float* vertices, int32_t sh_degree,
                      const float* camera_positions, int32_t B, float* out_colors, mt_stream_t stream) {
  return mt_grid_sh_colors_of_seen(grid_spherical_harmonics, C, G, vertex_sources, V, num_vertices, nullptr, 0,
                                   vertices, sh_degree, camera_positions, B, nullptr, out_colors, stream);
}

size_t mt_grid_sh_colors_backward_workspace_bytes(int64_t V) {
  // The rows [V][16][3], then a byte per vertex.
  return 256 + (size_t)(V > 0 ? V : 0) * (48 * sizeof(float) + 1);
}

int mt_grid_sh_colors_backward(const int32_t* list_offsets, const int32_t* list, int64_t G, int64_t V,
                               const float* vertices, int32_t C, int32_t sh_degree, const float* camera_positions,
                               int32_t B, const float* out_colors, const float* grad_colors,
                               float* grad_grid_spherical_harmonics, const int32_t* num_vertices, void* workspace,
                               size_t workspace_bytes, mt_stream_t stream) {
  return grid_sh_backward<false>(list_offsets, list, G, V, vertices, C, sh_degree, camera_positions, B, out_colors,
                                 grad_colors, grad_grid_spherical_harmonics, num_vertices, workspace,
                                 workspace_bytes, stream);
}

int mt_grid_sh_colors_packed_backward(const int32_t* list_offsets, const int32_t* list, int64_t G, int64_t V,
                                      const float* vertices, int32_t C, int32_t sh_degree, const float* camera_positions,
                                      int32_t B, const float* out_colors, const float* packed_gradients,
                                      float* grad_grid_spherical_harmonics, const int32_t* num_vertices, void* workspace,
                                      size_t workspace_bytes, mt_stream_t stream) {
  return grid_sh_backward<true>(list_offsets, list, G, V, vertices, C, sh_degree, camera_positions, B, out_colors,
                                packed_gradients, grad_grid_spherical_harmonics, num_vertices, workspace,
                                workspace_bytes, stream);
}

}  // extern "C"

// ct_accel.cu -- ct_build_accel: voxel brick maps from the caller's AABBs.
//
// Replaces the per-instance AABB BLAS + TLAS build of
// ACCEL_STRUCT_MNGR::build_blases / build_tlas (src/accel_struct_mngr.cpp:
// 1362-1504, 1854-1973).  The reference's AABBs are single voxels of a fixed
// grid (src/gvox/map_loader.cpp:264-272), so instead of a BVH over boxes each
// instance gets a dense grid of 8^3 bricks:
//
//   pass 1  per AABB: integer voxel coordinate, alignment check, per-instance
//           bounds (atomic min/max)                        -> host reads bounds
//   pass 2  per AABB: mark, at its brick, the bricks it lies in or touches
//           with its 26-neighbourhood, which are NEAR
//   pass 3  per brick cell: give NEAR bricks a mask slot and bricks with
//           voxels a primitive slot                       -> host reads counts
//   pass 4  per AABB: set the occupancy bit, keep the lowest primitive id
//           per voxel, record the voxel coordinate of the primitive
//   pass 5  rows of occupancy bits, then per cell and ray octant the cell
//           field the walks step by: the edge of the occupied-free cube from
//           the cell, by dilating the bits in shared memory (k_field)
//
// Device memory held by the result: two 4 B tables per brick cell, 64 B of
// occupancy mask per NEAR brick, 2 KiB of primitive ids per brick with
// voxels, 4 B per primitive, the cell field (4 B per cell), and one
// descriptor per instance.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>
#include "ct_accel.cuh"
#include "ct_range.h"

// Bounds as unsigned keys that only grow from 0, so that zeroed memory is
// their start: bound_key(v) is monotone in v, the minimum is kept as ~key.
struct InstBounds {
  uint32_t mn[3], mx[3];
  uint32_t inexact;   // any voxel whose centre cannot be recomputed exactly
  uint32_t misaligned;
};
__host__ __device__ inline uint32_t bound_key(int v) { return (uint32_t)v ^ 0x80000000u; }
__host__ __device__ inline int bound_value(uint32_t k) { return (int)(k ^ 0x80000000u); }

// The low 10 bits of a voxel's coordinates.  A grid has at most 1024 cells per
// axis, so these give the voxel's place in it exactly, and the passes after
// k_bounds read 4 bytes per voxel instead of its AABB.
__device__ __forceinline__ uint32_t pack_low(const int *c) {
  return ((uint32_t)c[0] & 1023u) | (((uint32_t)c[1] & 1023u) << 10) | (((uint32_t)c[2] & 1023u) << 20);
}

// An atomic maximum that most callers find done: same-address atomics queue up
// (8 per warp took 80 us for the 4.1 M voxels below), and a stale load costs one more.
__device__ __forceinline__ void raise(uint32_t *p, uint32_t v) {
  if (v > *(volatile uint32_t *)p) atomicMax(p, v);
}

// Per thread minima and maxima over a grid stride, then one reduction per
// warp.  Bounded by reading the AABBs: 46 us for 4.1 M voxels (98 MB),
// against 533 us with 6 atomics per voxel on one instance's 6 words.
// PAIRS: the AABBs are 8-byte aligned and read as 3 pairs; ie: 1 / e where
// that makes x * ie the same as x / e (e a power of two), else 0.  The ranges
// come from the caller's table unchecked (the host reads them back with the
// bounds, so that a build waits for the device once less): only their part
// inside the AABB table is read, of at most CT_MAX_PRIMITIVES entries, so that
// the stride cannot wrap either.
template <bool PAIRS>
__global__ void __launch_bounds__(256) k_bounds(const ct_instance *inst, const ct_aabb *aabb, uint32_t n_aabb, float e,
                                                float ie, InstBounds *B, uint32_t *low) {
  const uint32_t i = blockIdx.y;
  const uint32_t first = inst[i].first_primitive_index;
  const uint32_t count = ct_range_inside(first, inst[i].primitive_count, n_aabb);
  uint32_t mn[3] = {0u, 0u, 0u}, mx[3] = {0u, 0u, 0u}, inexact = 0u, misaligned = 0u;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
    const uint32_t gi = first + k;
    float b[6];
    if (PAIRS) {
      const float2 *p = (const float2 *)aabb + 3ull * gi;
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const float2 v = p[a];
        b[2 * a] = v.x;
        b[2 * a + 1] = v.y;
      }
    } else {
#pragma unroll
      for (int a = 0; a < 6; a++) b[a] = ((const float *)aabb)[6ull * gi + a];
    }
    int c[3];
    bool ok = true, exact = true;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float lo = b[a], hi = b[3 + a];
      const float v = ie != 0.0f ? lo * ie : lo / e, w = ie != 0.0f ? (hi - lo) * ie : (hi - lo) / e;
      const int iv = __float2int_rn(v);
      if (!(fabsf(v - (float)iv) <= 1e-3f) || !(fabsf(w - 1.0f) <= 1e-3f)) ok = false;
      if (!((float)iv * e == lo && (float)(iv + 1) * e == hi)) exact = false;
      c[a] = iv;
    }
    if (!ok) { misaligned |= 1u; continue; }
    if (!exact) inexact = 1u;
    low[gi] = pack_low(c);
    for (int a = 0; a < 3; a++) {
      mn[a] = max(mn[a], ~bound_key(c[a]));
      mx[a] = max(mx[a], bound_key(c[a]));
    }
  }
  const bool leader = (threadIdx.x & 31u) == 0u;
  for (int a = 0; a < 3; a++) {
    const uint32_t lo = __reduce_max_sync(0xFFFFFFFFu, mn[a]), hi = __reduce_max_sync(0xFFFFFFFFu, mx[a]);
    if (leader) {
      raise(&B[i].mn[a], lo);
      raise(&B[i].mx[a], hi);
    }
  }
  inexact = __reduce_or_sync(0xFFFFFFFFu, inexact);
  misaligned = __reduce_or_sync(0xFFFFFFFFu, misaligned);
  if (leader && inexact) atomicOr(&B[i].inexact, inexact);
  if (leader && misaligned) atomicOr(&B[i].misaligned, misaligned);
}

__device__ __forceinline__ bool voxel_local(uint32_t low, const DevGrid &g, int &x, int &y, int &z) {
  x = (int)((low - (uint32_t)g.gmin[0]) & 1023u);
  y = (int)(((low >> 10) - (uint32_t)g.gmin[1]) & 1023u);
  z = (int)(((low >> 20) - (uint32_t)g.gmin[2]) & 1023u);
  return x < g.bdim[0] * CT_BRICK && y < g.bdim[1] * CT_BRICK && z < g.bdim[2] * CT_BRICK;
}

// Bricks a voxel at local coordinate l of its brick touches along one axis, as
// bits for the offsets -1, 0, 1
__device__ __forceinline__ uint32_t touch_axis(int l) { return 2u | (l == 0 ? 1u : 0u) | (l == 7 ? 4u : 0u); }

// Per brick, the 27 bricks around it (bit (dz+1)*9 + (dy+1)*3 + (dx+1), itself
// bit 13) that its voxels lie in or touch.  Voxels of one brick follow one
// another, so most find their bits set: a load decides, and only the first few
// pay for the atomic (a stale load costs one more atomic, no bits).  35 us
// for 4.1 M voxels, against 65 us marking the neighbours' own words (up to 8
// loads a voxel) and 120 us with an atomic each.
__global__ void __launch_bounds__(256) k_mark(const DevGrid *grids, const uint32_t *low, uint32_t *marks) {
  const DevGrid &g = grids[blockIdx.y];
  const uint32_t n = g.primitive_count;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    int x, y, z;
    if (!voxel_local(low[g.first_primitive_index + k], g, x, y, z)) continue;
    const uint32_t tx = touch_axis(x & 7), ty = touch_axis(y & 7), tz = touch_axis(z & 7);
    const uint32_t row = ((ty & 1u) ? tx : 0u) | (tx << 3) | ((ty & 4u) ? tx << 6 : 0u);
    const uint32_t bits = ((tz & 1u) ? row : 0u) | (row << 9) | ((tz & 4u) ? row << 18 : 0u);
    uint32_t *p = &marks[g.table_offset + ((uint32_t)(z >> 3) * g.bdim[1] + (y >> 3)) * g.bdim[0] + (x >> 3)];
    if ((*(volatile uint32_t *)p & bits) != bits) atomicOr(p, bits);
  }
}

// counter[0]: mask slots (NEAR bricks), counter[1]: primitive slots (bricks with voxels)
__global__ void __launch_bounds__(256) k_assign_slots(const DevGrid *grids, const uint32_t *marks, uint32_t *table,
                                                      uint32_t *pslot, uint32_t *counter) {
  const DevGrid &g = grids[blockIdx.y];
  const int X = g.bdim[0], Y = g.bdim[1], Z = g.bdim[2];
  const uint32_t n = (uint32_t)X * Y * Z;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    const int x = (int)(c % X), y = (int)(c / X % Y), z = (int)(c / (X * Y));
    const uint32_t *m = marks + g.table_offset;
    bool near = false;
    for (int k = 0; k < 27; k++) {
      // the brick from which this one lies in direction k
      const int nx = x - (k % 3 - 1), ny = y - (k / 3 % 3 - 1), nz = z - (k / 9 - 1);
      if ((unsigned)nx < (unsigned)X && (unsigned)ny < (unsigned)Y && (unsigned)nz < (unsigned)Z)
        near = near || ((m[((uint32_t)nz * Y + ny) * X + nx] >> k) & 1u) != 0u;
    }
    const uint32_t at = g.table_offset + c;
    table[at] = near ? CT_NEAR_BIT | atomicAdd(&counter[0], 1u) : CT_EMPTY_SLOT;
    pslot[at] = ((m[c] >> 13) & 1u) ? atomicAdd(&counter[1], 1u) : CT_EMPTY_SLOT;
  }
}

// Occupancy bits, the lowest primitive of each voxel and each primitive's
// voxel.  Whole warps go through the loop together: the lanes whose voxels
// share an occupancy word (a row's voxels follow one another) set it with one
// atomic (29 us for 4.1 M voxels, against 55 us with an atomic each).
__global__ void __launch_bounds__(256) k_fill(const DevGrid *grids, const uint32_t *low, const uint32_t *table,
                                              const uint32_t *pslot, uint32_t *mask, uint32_t *prim, uint32_t *vcoord) {
  const DevGrid &g = grids[blockIdx.y];
  const uint32_t n = g.primitive_count;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const uint32_t k = base + threadIdx.x, gi = g.first_primitive_index + k;
    uint32_t word = 0xFFFFFFFFu, bit = 0u;
    int x, y, z;
    if (k < n && voxel_local(low[gi], g, x, y, z)) {
      const uint32_t cell = g.table_offset + ((uint32_t)(z >> 3) * g.bdim[1] + (y >> 3)) * g.bdim[0] + (x >> 3);
      const uint32_t slot = table[cell] & CT_EMPTY_SLOT;
      const uint32_t local = (uint32_t)(x & 7) + 8u * (uint32_t)(y & 7) + 64u * (uint32_t)(z & 7);
      word = slot * CT_MASK_WORDS + (local >> 5);
      bit = 1u << (local & 31u);
      atomicMin(&prim[pslot[cell] * 512u + local], k);
      vcoord[gi] = (uint32_t)x | ((uint32_t)y << 10) | ((uint32_t)z << 20);
    }
    const uint32_t same = __match_any_sync(0xFFFFFFFFu, word);
    const uint32_t bits = __reduce_or_sync(same, bit);
    if (bit && (threadIdx.x & 31u) == (uint32_t)__ffs(same) - 1u) atomicOr(&mask[word], bits);
  }
}

// The cell field (cell_field, ct_types.cuh): for every cell of a grid and
// every ray octant, the edge k of the largest cube without occupied cells
// that has the cell as its corner and extends in the octant's directions
// (cells beyond the grid count as empty: the walk clips every box to the
// grid), stored as the largest 4-bit code whose edge (ct_field_edge) is at
// most k.  The code of a cell is therefore the number of codes j = 1..15
// whose cube, of edge E_j, is empty.
//
// Occupancy is kept as bits, one row of cells along x per (y, z), and the
// cubes are tested by dilation, 32 cells of a row per word: D_j, the cells
// whose cube of edge E_j holds an occupied cell, is the union of D_(j-1) at
// the 8 corners {0, E_j - E_(j-1)}^3 (the smaller cubes cover the larger one
// as long as that step is at most E_(j-1)).
constexpr int kFieldCodes = 16;
__host__ __device__ constexpr int field_edge_of(int code) {
  const uint32_t t[4] = {CT_FIELD_EDGES0, CT_FIELD_EDGES1, CT_FIELD_EDGES2, CT_FIELD_EDGES3};
  return (int)((t[code >> 2] >> (8 * (code & 3))) & 255u);
}
constexpr int field_max_step() {
  int m = 0;
  for (int j = 2; j < kFieldCodes; j++) m = std::max(m, field_edge_of(j) - field_edge_of(j - 1));
  return m;
}
constexpr bool field_codes_ok() {
  if (field_edge_of(0) != 0 || field_edge_of(1) != 1) return false;
  for (int j = 2; j < kFieldCodes; j++) {
    const int d = field_edge_of(j) - field_edge_of(j - 1);
    if (d < 1 || d > field_edge_of(j - 1)) return false;
  }
  return field_edge_of(kFieldCodes - 1) <= 33;  // 32 cells and their cubes fit a 64-bit row
}
static_assert(field_codes_ok(), "cell field codes");

struct FieldGrid {
  uint32_t X, Y, Z;   // cells per axis
  uint32_t table_offset, bx, xw;  // bricks per axis x, occupancy words per row
  uint64_t row0;      // first occupancy word
  uint64_t word0;     // first word in cell_field
};

// occupancy rows from the brick table and the NEAR bricks' masks, whose byte
// y + 8z holds the brick's 8 cells of one row; counts the occupied cells
__global__ void __launch_bounds__(256) k_occ_rows(const FieldGrid *fg, const uint32_t *table, const uint8_t *mask,
                                                  uint32_t *rows, uint32_t *count) {
  const FieldGrid f = fg[blockIdx.y];
  const uint32_t n = f.xw * f.Y * f.Z;
  uint32_t voxels = 0;
  for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < n; w += gridDim.x * blockDim.x) {
    const uint32_t xw = w % f.xw, y = (w / f.xw) % f.Y, z = w / (f.xw * f.Y);
    const uint32_t *t = table + f.table_offset + ((z >> 3) * (f.Y >> 3) + (y >> 3)) * f.bx;
    uint32_t v = 0;
#pragma unroll
    for (uint32_t b = 0; b < 4; b++) {
      const uint32_t e = 4u * xw + b < f.bx ? t[4u * xw + b] : 0u;
      if (e & CT_NEAR_BIT)
        v |= (uint32_t)mask[(uint64_t)(e & CT_EMPTY_SLOT) * (4u * CT_MASK_WORDS) + (y & 7u) + 8u * (z & 7u)] << (8u * b);
    }
    rows[f.row0 + w] = v;
    voxels += (uint32_t)__popc(v);
  }
  voxels = __reduce_add_sync(0xFFFFFFFFu, voxels);
  if ((threadIdx.x & 31u) == 0u && voxels) atomicAdd(count, voxels);
}

// One block: 32 x 64 x 64 cells of one octant, in coordinates mirrored so
// that the octant's directions increase.  A row is 64 bits: the block's 32
// cells and the ones their cubes reach.  The tile and its margin (cubes reach
// E_15 - 1 cells past it, and a step reads that much zero padding) are
// dilated in shared memory, 15 levels from one buffer to the other; each
// level adds one bit to the bit-sliced codes of the thread's 4 output rows.
// Bounded by shared-memory reads (2.5 rows read, 1 written per row and level)
// and the margin (2.1 rows worked on per row kept): 161 us on the 256^3
// terrain (9.5 M cells, 8 octants), 183 us with a thread per row (4 read),
// 8.5 ms with one byte per cell in HBM and 16 sweeps per octant.  512 threads
// with longer strips (fewer reads, half the warps) made the build 5% slower.
constexpr int kFieldTile = 64;
constexpr int kFieldSpan = kFieldTile + CT_FIELD_MAX_EDGE - 1;  // rows per axis with the margin
constexpr int kFieldPad = field_max_step();  // empty rows a step may read past the margin
constexpr int kFieldThreads = 1024;
constexpr int kFieldStrip = (kFieldSpan + kFieldThreads / kFieldSpan - 1) / (kFieldThreads / kFieldSpan);  // rows per thread
constexpr int kFieldPadZ = kFieldPad + kFieldStrip;  // a strip's last rows may lie past the margin
constexpr uint32_t kFieldSmem = 2u * (kFieldSpan + kFieldPad) * (kFieldSpan + kFieldPadZ) * sizeof(uint64_t);
static_assert(kFieldSmem <= 227 * 1024, "shared memory per block");
constexpr int kFieldOut = kFieldTile * kFieldTile / kFieldThreads;  // output rows per thread

// 64 cells of a row from cell `at` (any sign; cells outside the row are empty)
__device__ __forceinline__ uint64_t row_bits(const uint32_t *row, int xw, int at) {
  const int w = at >> 5, sh = at & 31;
  uint32_t v[3];
#pragma unroll
  for (int i = 0; i < 3; i++) v[i] = w + i >= 0 && w + i < xw ? row[w + i] : 0u;
  return (uint64_t)__funnelshift_r(v[0], v[1], sh) | ((uint64_t)__funnelshift_r(v[1], v[2], sh) << 32);
}
// the low 8 bits of v, bit i moved to bit 4i
__device__ __forceinline__ uint32_t spread_nibbles(uint32_t v) {
  v = (v | (v << 12)) & 0x000F000Fu;
  v = (v | (v << 6)) & 0x03030303u;
  return (v | (v << 3)) & 0x11111111u;
}

// A block's tile: rows along y and z inside the grid (with the margin, and of
// the tile itself) and the pitch of a z plane.
struct FieldTile {
  int ny, nz, oy, oz, py;
};
// Level J on: one more code for the cells whose cube of edge E_J is empty,
// then the dilation to E_(J+1).  A thread works on a strip of rows along z, so
// that it reads a row's pair along y once for both ends of the step along z.
template <int J>
__device__ __forceinline__ void field_levels(const FieldTile &T, uint64_t *src, uint64_t *dst,
                                             uint32_t (&c)[kFieldOut][4]) {
  const int tid = (int)threadIdx.x;
#pragma unroll
  for (int k = 0; k < kFieldOut; k++) {
    const int o = tid + k * kFieldThreads, ly = o % kFieldTile, lz = o / kFieldTile;
    if (ly < T.oy && lz < T.oz) {
      uint32_t carry = ~(uint32_t)src[lz * T.py + ly];
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const uint32_t t = c[k][b] & carry;
        c[k][b] ^= carry;
        carry = t;
      }
    }
  }
  if constexpr (J + 1 < kFieldCodes) {
    constexpr int d = field_edge_of(J + 1) - field_edge_of(J);
    constexpr int need = CT_FIELD_MAX_EDGE - field_edge_of(J + 1);  // rows past the tile the later levels still read
    const int rows_y = min(T.ny, kFieldTile + need), rows_z = min(T.nz, kFieldTile + need);
    const int ly = tid % kFieldSpan, z0 = tid / kFieldSpan * kFieldStrip;
    if (ly < rows_y && z0 < rows_z) {
      const uint64_t *r = src + z0 * T.py + ly;
      uint64_t *w = dst + z0 * T.py + ly;
      uint64_t a[kFieldStrip + d];
#pragma unroll
      for (int i = 0; i < kFieldStrip + d; i++) a[i] = r[i * T.py] | r[i * T.py + d];
#pragma unroll
      for (int i = 0; i < kFieldStrip; i++) {
        const uint64_t v = a[i] | a[i + d];
        if (z0 + i < rows_z) w[i * T.py] = v | (v >> d);
      }
    }
    __syncthreads();
    field_levels<J + 1>(T, dst, src, c);
  }
}

__global__ void __launch_bounds__(kFieldThreads) k_field(const FieldGrid *fg, const uint32_t *rows, uint32_t *field) {
  extern __shared__ uint64_t s_rows[];
  const FieldGrid f = fg[blockIdx.z];
  const uint32_t octant = blockIdx.y;
  const uint32_t ty_n = (f.Y + kFieldTile - 1) / kFieldTile, tz_n = (f.Z + kFieldTile - 1) / kFieldTile;
  if (blockIdx.x >= f.xw * ty_n * tz_n) return;
  const int x0 = 32 * (int)(blockIdx.x % f.xw), y0 = kFieldTile * (int)(blockIdx.x / f.xw % ty_n),
            z0 = kFieldTile * (int)(blockIdx.x / (f.xw * ty_n));
  const bool mx = octant & 1u, my = octant & 2u, mz = octant & 4u;
  // rows of the tile and its margin inside the grid; the others stay empty
  FieldTile T;
  T.ny = min(kFieldSpan, (int)f.Y - y0);
  T.nz = min(kFieldSpan, (int)f.Z - z0);
  T.oy = min(kFieldTile, T.ny);
  T.oz = min(kFieldTile, T.nz);
  T.py = T.ny + kFieldPad;
  const int oy = T.oy, oz = T.oz;
  const uint32_t tid = threadIdx.x;
  const int plane = T.py * (T.nz + kFieldPadZ);
  uint64_t *src = s_rows, *dst = s_rows + plane;
  for (int i = (int)tid; i < 2 * plane; i += kFieldThreads) s_rows[i] = 0ull;
  __syncthreads();
  for (int i = (int)tid; i < T.ny * T.nz; i += kFieldThreads) {
    const int ly = i % T.ny, lz = i / T.ny;
    const int y = my ? (int)f.Y - 1 - (y0 + ly) : y0 + ly, z = mz ? (int)f.Z - 1 - (z0 + lz) : z0 + lz;
    const uint32_t *row = rows + f.row0 + ((uint64_t)z * f.Y + y) * f.xw;
    src[lz * T.py + ly] = mx ? __brevll(row_bits(row, (int)f.xw, (int)f.X - 64 - x0)) : row_bits(row, (int)f.xw, x0);
  }
  __syncthreads();
  uint32_t c[kFieldOut][4];
#pragma unroll
  for (int k = 0; k < kFieldOut; k++) {
    c[k][0] = c[k][1] = c[k][2] = c[k][3] = 0u;
  }
  field_levels<1>(T, src, dst, c);
#pragma unroll
  for (int k = 0; k < kFieldOut; k++) {
    const int o = (int)tid + k * kFieldThreads, ly = o % kFieldTile, lz = o / kFieldTile;
    if (ly >= oy || lz >= oz) continue;
    const int y = my ? (int)f.Y - 1 - (y0 + ly) : y0 + ly, z = mz ? (int)f.Z - 1 - (z0 + lz) : z0 + lz;
    uint32_t *out = field + f.word0 + (((uint64_t)octant * f.Z + z) * f.Y + y) * f.bx;
#pragma unroll
    for (int g = 0; g < 4; g++) {
      // cells x0 + 8g .. + 7 in the block's direction, one word of the row
      const int xb = (x0 >> 3) + g;
      if (xb >= (int)f.bx) break;
      uint32_t v = 0;
#pragma unroll
      for (int b = 0; b < 4; b++) {
        uint32_t byte = (c[k][b] >> (8 * g)) & 255u;
        if (mx) byte = __brev(byte) >> 24;
        v |= spread_nibbles(byte) << b;
      }
      out[mx ? (int)f.bx - 1 - xb : xb] = v;
    }
  }
}

// Builds the cell field of every grid (see k_field) from the brick masks,
// with one bit per cell of scratch, and counts the occupied cells.
static cudaError_t build_cell_field(ct_accel *acc, const std::vector<FieldGrid> &hf, FieldGrid *d_fg, uint32_t *rows,
                                    uint32_t *d_count, cudaStream_t stream) {
  const uint32_t n_inst = (uint32_t)hf.size();
  uint64_t max_words = 0, max_tiles = 0;
  for (const FieldGrid &f : hf) {
    max_words = std::max<uint64_t>(max_words, (uint64_t)f.xw * f.Y * f.Z);
    max_tiles = std::max<uint64_t>(max_tiles, (uint64_t)f.xw * ((f.Y + kFieldTile - 1) / kFieldTile) *
                                                  ((f.Z + kFieldTile - 1) / kFieldTile));
  }
  cudaError_t e = cudaFuncSetAttribute(k_field, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFieldSmem);
  if (e != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(d_fg, hf.data(), sizeof(FieldGrid) * n_inst, cudaMemcpyHostToDevice, stream)) != cudaSuccess)
    return e;
  const uint64_t want = (max_words + 255) / 256;
  k_occ_rows<<<dim3((uint32_t)std::min<uint64_t>(want, 8192), n_inst), 256, 0, stream>>>(
      d_fg, acc->d_table, (const uint8_t *)acc->d_mask, rows, d_count);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  k_field<<<dim3((uint32_t)max_tiles, 8, n_inst), kFieldThreads, kFieldSmem, stream>>>(d_fg, rows, acc->d_field);
  return cudaGetLastError();
}

static ct_status cuda_fail(cudaError_t e) {
  ct_set_cuda_error(e);
  return CT_ERR_CUDA;
}

#define CT_TRY(x)                              \
  do {                                         \
    cudaError_t _e = (x);                      \
    if (_e != cudaSuccess) { st = cuda_fail(_e); goto fail; } \
  } while (0)

// Device memory of the structures, from one pool per device, so that a scene
// that is rebuilt after every edit reuses the memory of the structure it
// replaced instead of mapping and unmapping it (the 17 cudaMalloc / cudaFree
// of a build and its release took 2.7 ms on the 256^3 terrain).  A structure's
// blocks go back to the pool when it is freed; the pool keeps them as long as
// all it holds, for live structures too, is at most kPoolKeep, and gives the
// rest back to the driver (a scene above that maps its memory anew on every
// rebuild).  ct_release_memory gives back what no structure uses.
//
// The structures' grids are small cudaMalloc blocks (see ~ct_accel).  The
// pool's device keeps another one, so that the driver's slab they lie in stays
// mapped: 1 us for the cudaMalloc and 3 us for the cudaFree of 512 bytes,
// against 2.2 and 0.9 ms with the slab mapped and unmapped each time.
constexpr uint64_t kPoolKeep = 256ull << 20;
static std::mutex g_pool_mu;
static std::vector<cudaMemPool_t> g_pools;

static cudaError_t device_pool(int dev, cudaMemPool_t *out) {
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if ((size_t)dev >= g_pools.size()) g_pools.resize((size_t)dev + 1, nullptr);
  if (!g_pools[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = kPoolKeep;
    if ((e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return e;
    }
    void *slab = nullptr;
    if ((e = cudaMalloc(&slab, 256)) != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return e;
    }
    g_pools[dev] = pool;
  }
  *out = g_pools[dev];
  return cudaSuccess;
}

// Pieces of one allocation, 256-byte aligned.
struct Arena {
  char *base = nullptr;
  uint64_t bytes = 0;
  uint64_t add(uint64_t n) {
    const uint64_t at = bytes;
    bytes += (n + 255u) & ~255ull;
    return at;
  }
  cudaError_t alloc(cudaMemPool_t pool, cudaStream_t s) {
    return cudaMallocFromPoolAsync((void **)&base, bytes ? bytes : 256, pool, s);
  }
  template <class T>
  T *at(uint64_t off) const { return (T *)(base + off); }
};

// Work on any stream may still read the structure.  cudaFree of the grids,
// memory of their own, waits for the device; the blocks, for which cudaFree
// does not wait, go back to the pool behind it.  (cudaDeviceSynchronize would
// break every capture that is under way, also the thread-local and relaxed
// ones of other threads, which cudaFree leaves alone.)
ct_accel::~ct_accel() {
  int cur = 0;
  const bool other = cudaGetDevice(&cur) == cudaSuccess && cur != device;
  if (other) cudaSetDevice(device);
  cudaFree(d_grids);
  for (void *b : block) cudaFree(b);
  cudaFree(ws_ptr);
  if (other) cudaSetDevice(cur);
}

extern "C" ct_status ct_build_accel(const ct_scene_desc *scene, ct_accel **out, ct_stream stream_) {
  if (!scene || !out) return CT_ERR_INVALID_ARG;
  *out = nullptr;
  cudaStream_t stream = (cudaStream_t)stream_;
  if (scene->instance_count == 0 || scene->instance_address == 0 || scene->aabb_address == 0) return CT_ERR_INVALID_ARG;
  if (!(scene->voxel_extent > 0.0f) || !isfinite(scene->voxel_extent)) return CT_ERR_INVALID_ARG;
  if (scene->instance_count > CT_MAX_INSTANCES || scene->aabb_count > CT_MAX_PRIMITIVES) return CT_ERR_CAPACITY;
  if ((scene->instance_address & 3u) || (scene->aabb_address & 3u)) return CT_ERR_INVALID_ARG;

  ct_status st = CT_OK;
  const uint32_t n_inst = scene->instance_count;
  const float e = scene->voxel_extent;
  const ct_instance *d_inst = (const ct_instance *)(uintptr_t)scene->instance_address;
  const ct_aabb *d_aabb = (const ct_aabb *)(uintptr_t)scene->aabb_address;
  std::vector<ct_instance> h_inst(n_inst);
  std::vector<InstBounds> h_b(n_inst);
  std::vector<FieldGrid> hf(n_inst);
  cudaMemPool_t pool = nullptr;
  Arena scratch, marks, tables, bricks;
  uint64_t o_fg, o_b, o_counter, o_low, o_marks, o_rows, o_table, o_pslot, o_vcoord, o_field, o_mask, o_prim;
  InstBounds *d_b = nullptr;
  uint32_t *d_low = nullptr;      // per AABB: low bits of its coordinates
  uint32_t *d_counter = nullptr;  // [0] mask slots, [1] primitive slots, [2] voxels
  ct_accel *acc = new (std::nothrow) ct_accel();
  if (!acc) return CT_ERR_CAPACITY;
  uint64_t total_cells = 0, max_cells = 0, max_prims = 0, field_words = 0, row_words = 0;
  uint32_t n_slots = 0, n_pslots = 0;
  uint32_t counts[3] = {0, 0, 0};
  uint32_t per_inst = 0;  // blocks per instance of the passes over AABBs

  CT_TRY(cudaGetDevice(&acc->device));
  CT_TRY(device_pool(acc->device, &pool));
  o_b = scratch.add(sizeof(InstBounds) * n_inst);
  o_counter = scratch.add(sizeof(counts));
  o_low = scratch.add(sizeof(uint32_t) * (uint64_t)scene->aabb_count);
  CT_TRY(scratch.alloc(pool, stream));
  d_b = scratch.at<InstBounds>(o_b);
  d_counter = scratch.at<uint32_t>(o_counter);
  d_low = scratch.at<uint32_t>(o_low);
  CT_TRY(cudaMemsetAsync(scratch.base, 0, o_low, stream));
  // the instances' primitive counts are on the device: a grid for the whole
  // table, spread over the instances
  per_inst = std::max(1u, std::min((scene->aabb_count + 255u) / 256u, std::max(1u, 2048u / n_inst)));
  {
    // x / e is x * (1 / e) exactly when e is a power of two of moderate size
    int exponent = 0;
    const float ie = frexpf(e, &exponent) == 0.5f && e > 1e-30f && e < 1e30f ? 1.0f / e : 0.0f;
    const dim3 grid(per_inst, n_inst);
    if (scene->aabb_address & 7u)
      k_bounds<false><<<grid, 256, 0, stream>>>(d_inst, d_aabb, scene->aabb_count, e, ie, d_b, d_low);
    else
      k_bounds<true><<<grid, 256, 0, stream>>>(d_inst, d_aabb, scene->aabb_count, e, ie, d_b, d_low);
  }
  CT_TRY(cudaGetLastError());
  CT_TRY(cudaMalloc(&acc->d_grids, sizeof(DevGrid) * n_inst));  // while the bounds are computed
  CT_TRY(cudaMemcpyAsync(h_inst.data(), d_inst, sizeof(ct_instance) * n_inst, cudaMemcpyDeviceToHost, stream));
  CT_TRY(cudaMemcpyAsync(h_b.data(), d_b, sizeof(InstBounds) * n_inst, cudaMemcpyDeviceToHost, stream));
  CT_TRY(cudaStreamSynchronize(stream));
  for (uint32_t i = 0; i < n_inst; i++) {
    if (ct_range_outside(h_inst[i].first_primitive_index, h_inst[i].primitive_count, scene->aabb_count)) {
      st = CT_ERR_INVALID_ARG;
      goto fail;
    }
    max_prims = h_inst[i].primitive_count > max_prims ? h_inst[i].primitive_count : max_prims;
  }
  acc->h_grids.resize(n_inst);
  acc->info.grid_exact = 1;
  for (uint32_t i = 0; i < n_inst; i++) {
    if (h_b[i].misaligned) { st = CT_ERR_NOT_GRID_ALIGNED; goto fail; }
    DevGrid &g = acc->h_grids[i];
    memset(&g, 0, sizeof(g));
    m4 T = load_m4(h_inst[i].transform);
    g.world2obj_inst = ct_inverse(T);
    m4 Tt = T;
    Tt.c[0].w = 0.f; Tt.c[1].w = 0.f; Tt.c[2].w = 0.f; Tt.c[3].w = 1.f;
    g.obj2world_tlas = Tt;
    g.world2obj_tlas = ct_inverse(Tt);
    g.first_primitive_index = h_inst[i].first_primitive_index;
    g.primitive_count = h_inst[i].primitive_count;
    g.grid_exact = h_b[i].inexact ? 0u : 1u;
    if (!g.grid_exact) acc->info.grid_exact = 0;
    int mn[3], mx[3];
    for (int a = 0; a < 3; a++) {
      if (h_inst[i].primitive_count == 0) { mn[a] = 0; mx[a] = 0; }
      else { mn[a] = bound_value(~h_b[i].mn[a]); mx[a] = bound_value(h_b[i].mx[a]); }
      // one empty voxel of margin on every side, brick aligned
      int lo = mn[a] - 1, hi = mx[a] + 1;
      int glo = (lo >= 0) ? (lo / CT_BRICK) * CT_BRICK : -((-lo + CT_BRICK - 1) / CT_BRICK) * CT_BRICK;
      g.gmin[a] = glo;
      g.bdim[a] = (hi - glo) / CT_BRICK + 1;
      if (g.bdim[a] * CT_BRICK > 1024) { st = CT_ERR_CAPACITY; goto fail; }  // 10-bit voxel coordinates
    }
    g.table_offset = (uint32_t)total_cells;
    total_cells += (uint64_t)g.bdim[0] * g.bdim[1] * g.bdim[2];
    max_cells = std::max(max_cells, (uint64_t)g.bdim[0] * g.bdim[1] * g.bdim[2]);
    if (total_cells > 0x7FFFFFFFull) { st = CT_ERR_CAPACITY; goto fail; }
    if (i == 0)
      for (int a = 0; a < 3; a++) { acc->info.grid_min[a] = mn[a]; acc->info.grid_dim[a] = mx[a] - mn[a] + 1; }
    // the cell field: 8 octants of one word per 8 cells, rows of occupancy bits
    FieldGrid &f = hf[i];
    f.X = (uint32_t)g.bdim[0] * CT_BRICK;
    f.Y = (uint32_t)g.bdim[1] * CT_BRICK;
    f.Z = (uint32_t)g.bdim[2] * CT_BRICK;
    f.table_offset = g.table_offset;
    f.bx = (uint32_t)g.bdim[0];
    f.xw = (f.X + 31u) / 32u;
    f.row0 = row_words;
    f.word0 = g.field_offset = field_words;
    row_words += (uint64_t)f.xw * f.Y * f.Z;
    field_words += (uint64_t)f.X * f.Y * f.Z;
  }
  // what the grids' sizes decide, in one block; what the brick counts decide follows
  o_table = tables.add(sizeof(uint32_t) * total_cells);
  o_pslot = tables.add(sizeof(uint32_t) * total_cells);
  o_vcoord = tables.add(sizeof(uint32_t) * (uint64_t)scene->aabb_count);
  o_field = tables.add(sizeof(uint32_t) * field_words);
  CT_TRY(tables.alloc(pool, stream));
  acc->block[0] = tables.base;
  acc->d_table = tables.at<uint32_t>(o_table);
  acc->d_pslot = tables.at<uint32_t>(o_pslot);
  acc->d_vcoord = tables.at<uint32_t>(o_vcoord);
  acc->d_field = tables.at<uint32_t>(o_field);
  CT_TRY(cudaMemcpyAsync(acc->d_grids, acc->h_grids.data(), sizeof(DevGrid) * n_inst, cudaMemcpyHostToDevice, stream));
  acc->n_primitives = scene->aabb_count;
  CT_TRY(cudaMemsetAsync(acc->d_vcoord, 0xFF, sizeof(uint32_t) * (uint64_t)scene->aabb_count, stream));
  {
    dim3 grid((uint32_t)((max_prims + 255) / 256 < 4096 ? (max_prims + 255) / 256 : 4096), n_inst);
    if (grid.x == 0) grid.x = 1;
    o_marks = marks.add(sizeof(uint32_t) * total_cells);
    CT_TRY(marks.alloc(pool, stream));
    CT_TRY(cudaMemsetAsync(marks.base, 0, marks.bytes, stream));
    k_mark<<<grid, 256, 0, stream>>>(acc->d_grids, d_low, marks.at<uint32_t>(o_marks));
    CT_TRY(cudaGetLastError());
    const uint64_t cb = (max_cells + 255) / 256;
    k_assign_slots<<<dim3((uint32_t)std::min<uint64_t>(cb, 8192), n_inst), 256, 0, stream>>>(
        acc->d_grids, marks.at<uint32_t>(o_marks), acc->d_table, acc->d_pslot, d_counter);
    CT_TRY(cudaGetLastError());
    CT_TRY(cudaFreeAsync(marks.base, stream));
    marks.base = nullptr;
    CT_TRY(cudaMemcpyAsync(counts, d_counter, sizeof(counts), cudaMemcpyDeviceToHost, stream));
    CT_TRY(cudaStreamSynchronize(stream));
    n_slots = counts[0];
    n_pslots = counts[1];
    const uint64_t ns = n_slots ? n_slots : 1, nps = n_pslots ? n_pslots : 1;
    o_mask = bricks.add(sizeof(uint32_t) * CT_MASK_WORDS * ns);
    o_prim = bricks.add(sizeof(uint32_t) * 512ull * nps);
    CT_TRY(bricks.alloc(pool, stream));
    acc->block[1] = bricks.base;
    acc->d_mask = bricks.at<uint32_t>(o_mask);
    acc->d_prim = bricks.at<uint32_t>(o_prim);
    CT_TRY(cudaMemsetAsync(acc->d_mask, 0, sizeof(uint32_t) * CT_MASK_WORDS * ns, stream));
    CT_TRY(cudaMemsetAsync(acc->d_prim, 0xFF, sizeof(uint32_t) * 512ull * nps, stream));
    k_fill<<<grid, 256, 0, stream>>>(acc->d_grids, d_low, acc->d_table, acc->d_pslot, acc->d_mask,
                                     acc->d_prim, acc->d_vcoord);
    CT_TRY(cudaGetLastError());
    // the field's scratch follows the bounds' (its block is free again once
    // the kernels above are through with it)
    CT_TRY(cudaFreeAsync(scratch.base, stream));
    scratch = Arena();
    o_counter = scratch.add(sizeof(uint32_t));
    o_fg = scratch.add(sizeof(FieldGrid) * n_inst);
    o_rows = scratch.add(sizeof(uint32_t) * row_words);
    CT_TRY(scratch.alloc(pool, stream));
    d_counter = scratch.at<uint32_t>(o_counter);
    CT_TRY(cudaMemsetAsync(d_counter, 0, sizeof(uint32_t), stream));
    CT_TRY(build_cell_field(acc, hf, scratch.at<FieldGrid>(o_fg), scratch.at<uint32_t>(o_rows), d_counter, stream));
    CT_TRY(cudaMemcpyAsync(&acc->info.voxel_count, d_counter, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
  }
  acc->dev.grids = acc->d_grids;
  acc->dev.n_grids = n_inst;
  acc->dev.extent = e;
  acc->dev.brick_table = acc->d_table;
  acc->dev.brick_mask = acc->d_mask;
  acc->dev.brick_pslot = acc->d_pslot;
  acc->dev.brick_prim = acc->d_prim;
  acc->dev.cell_field = acc->d_field;
  acc->dev.voxel_coord = acc->d_vcoord;
  acc->dev.aabbs = d_aabb;
  acc->dev.max_steps = CT_DDA_MAX_STEPS;
  acc->info.instance_count = n_inst;
  acc->info.brick_count = n_pslots;
  acc->info.device_bytes = sizeof(DevGrid) * n_inst + 8ull * total_cells + 2048ull * total_cells + 64ull * n_slots +
                           2048ull * n_pslots +
                           4ull * scene->aabb_count;
  CT_TRY(cudaFreeAsync(scratch.base, stream));
  scratch.base = nullptr;
  CT_TRY(cudaStreamSynchronize(stream));  // also lands info.voxel_count
  *out = acc;
  return CT_OK;
fail:
  if (scratch.base) cudaFreeAsync(scratch.base, stream);
  if (marks.base) cudaFreeAsync(marks.base, stream);
  delete acc;
  return st;
}

extern "C" ct_status ct_accel_free(ct_accel *acc) {
  if (!acc) return CT_ERR_INVALID_ARG;
  delete acc;
  return CT_OK;
}

extern "C" ct_status ct_release_memory(void) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e);
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if ((size_t)dev >= g_pools.size() || !g_pools[dev]) return CT_OK;  // nothing was built here
  e = cudaMemPoolTrimTo(g_pools[dev], 0);
  return e == cudaSuccess ? CT_OK : cuda_fail(e);
}

extern "C" ct_status ct_accel_get_info(const ct_accel *acc, ct_accel_info *out) {
  if (!acc || !out) return CT_ERR_INVALID_ARG;
  *out = acc->info;
  return CT_OK;
}

// one octant of a grid's cell field, decoded to an edge per cell (the walk's
// cell_field lookup, cell by cell)
__global__ void k_field_unpack(const uint32_t *field, uint64_t word0, uint32_t octant, uint32_t X, uint32_t Y,
                               uint32_t Z, uint8_t *out) {
  const uint64_t n = (uint64_t)X * Y * Z;
  for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < n; c += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = (uint32_t)(c % X), y = (uint32_t)((c / X) % Y), z = (uint32_t)(c / ((uint64_t)X * Y));
    const uint64_t w = word0 + (((uint64_t)octant * Z + z) * Y + y) * (X / 8u) + (x >> 3);
    out[c] = (uint8_t)ct_field_edge((field[w] >> ((x & 7u) * 4u)) & 15u);
  }
}

extern "C" ct_status ct_accel_field(const ct_accel *acc, uint32_t instance, uint32_t octant, uint8_t *edges,
                                    int32_t grid_min[3], uint32_t cells[3], ct_stream stream) {
  if (!acc || !grid_min || !cells || octant >= 8u || instance >= acc->h_grids.size()) return CT_ERR_INVALID_ARG;
  const DevGrid &g = acc->h_grids[instance];
  const uint32_t X = (uint32_t)g.bdim[0] * CT_BRICK, Y = (uint32_t)g.bdim[1] * CT_BRICK,
                 Z = (uint32_t)g.bdim[2] * CT_BRICK;
  for (int a = 0; a < 3; a++) grid_min[a] = g.gmin[a];
  cells[0] = X;
  cells[1] = Y;
  cells[2] = Z;
  if (!edges) return CT_OK;
  const uint64_t n = (uint64_t)X * Y * Z;
  if (n == 0) return CT_OK;
  const uint64_t want = (n + 255) / 256;
  k_field_unpack<<<(uint32_t)(want < 8192 ? want : 8192), 256, 0, (cudaStream_t)stream>>>(
      acc->d_field, g.field_offset, octant, X, Y, Z, edges);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CT_OK : cuda_fail(e);
}

// ct_device.cuh -- device-side scene access, voxel traversal and the
// direct-lighting building blocks shared by the frame kernels.  Included by
// exactly one translation unit (ct_kernels.cu), which owns the device
// status word.
//
// Semantics follow cube-tracing's shaders (file:line given per function);
// the data layout, traversal and thread mapping are this library's own.
#pragma once
#include <cstdint>
#include "ct_types.cuh"
#include "ct_fpmath.h"

// device error word: [0] status, [1] detail, [2] pixel
__device__ uint32_t g_ct_error[4];
__device__ __forceinline__ void ct_latch_error(uint32_t status, uint32_t detail, uint32_t pixel) {
  if (atomicCAS(&g_ct_error[0], 0u, status) == 0u) {
    g_ct_error[1] = detail;
    g_ct_error[2] = pixel;
  }
}

// Work counters (flushed to ct_params.counters_address when
// CT_PARAM_COUNT_RAYS is set): rays by kind, 8^3 bricks the walks entered,
// voxel box tests, light candidates evaluated, neighbour records read by
// spatial reuse, temporal reuse records read, shaded (hit) pixels.
struct RayStats {
  uint32_t primary, shadow, bounce, bricks, voxel_tests, candidates, neighbours, temporal, hits, bounce_hits,
      walker_bricks;
};

// ---------------------------------------------------------------------------
// per-frame view of the caller's buffers (WORLD / RESTIR / Status tables).
// From `instances` on the members are WORLD's and RESTIR's addresses and then
// Status's words from frame_number to max_depth, in those tables' order, which
// load_frame_view copies word by word.
struct FrameView {
  float4 *swapchain;
  const float4 *previous_swapchain;
  float4 *taa_frame;
  uint32_t W, H;
  ct_light_config light_config;
  uint32_t _pad0;
  // WORLD
  const ct_instance *instances;
  const ct_instance *instances_prev;
  const ct_primitive *primitives;
  const ct_primitive *primitives_prev;
  const ct_aabb *aabbs;
  const ct_aabb *aabbs_prev;
  const uint32_t *remap_p;    // WORLD.remapped_primitive_address (CT_REMAP_BIT)
  const uint32_t *remap_l;    // WORLD.remapped_cube_light_address
  const ct_material *materials;
  const ct_light *point_lights;
  const ct_light *cube_lights;
  const ct_light *env_lights;
  // RESTIR
  ct_reservoir *prev_reservoir;
  ct_reservoir *int_reservoir;
  ct_reservoir *cur_reservoir;
  ct_di_info *prev_di;
  ct_di_info *di;
  ct_velocity *velocity;
  ct_path_reservoir *out_path_reservoir;
  ct_path_reservoir *temporal_path_reservoir;
  float *indirect_color;
  // Status
  uint32_t frame_number, _pad1;
  uint64_t num_accumulated_frames;
  uint32_t pixel[2];
  uint32_t is_active, _pad2;
  uint64_t light_config_address;
  uint32_t obj_count;
  float time;
  uint32_t is_afternoon, max_depth;
};

__device__ __forceinline__ f3 ld3(const float *p) { return f3{p[0], p[1], p[2]}; }
__device__ __forceinline__ void st3(float *p, f3 v) { p[0] = v.x; p[1] = v.y; p[2] = v.z; }

struct Material {
  uint32_t type;
  f3 diffuse, specular, emission;
  float roughness, ior;
};
__device__ __forceinline__ Material load_material(const FrameView &F, uint32_t idx) {
  const ct_material &m = F.materials[idx];
  Material r;
  r.type = m.type;
  r.diffuse = ld3(m.diffuse);
  r.specular = ld3(m.specular);
  r.emission = ld3(m.emission);
  r.roughness = m.roughness;
  r.ior = m.ior;
  return r;
}

struct Light {
  f3 position, emissive;
  uint32_t inst, prim;
  float size;
  uint32_t type;
};
__device__ __forceinline__ Light load_light(const ct_light *buf, uint32_t idx) {
  const ct_light &l = buf[idx];
  Light r;
  r.position = ld3(l.position);
  r.emissive = ld3(l.emissive);
  r.inst = l.instance_info.instance_id;
  r.prim = l.instance_info.primitive_id;
  r.size = l.size;
  r.type = l.type;
  return r;
}
// light_get_by_type (light.glsl:47-64); unknown types give an empty light
__device__ __forceinline__ Light light_get_by_type(const FrameView &F, uint32_t type, uint32_t idx) {
  if (type == CT_LIGHT_POINT) return load_light(F.point_lights, idx);
  if (type == CT_LIGHT_ENV_MAP) return load_light(F.env_lights, idx);
  if (type == CT_LIGHT_CUBE) return load_light(F.cube_lights, idx);
  Light l = {};
  l.type = CT_LIGHT_NONE;
  return l;
}

// ---------------------------------------------------------------------------
// sky / environment (mat.glsl:111-202, light.glsl:71-76)
__device__ __forceinline__ f3 bg_mix(f3 dir, f3 a, f3 b) {
  f3 u = normalize(dir);
  float t = 0.5f * (u.y + 1.0f);
  return gmix(a, b, t);
}
__device__ __forceinline__ f3 bg_day(f3 d) { return bg_mix(d, mk3(1.0f, 1.0f, 1.0f), mk3(0.5f, 0.7f, 1.0f)); }
__device__ __forceinline__ f3 bg_night(f3 d) { return bg_mix(d, mk3(0.2f, 0.2f, 0.3f), mk3(0.2f, 0.2f, 0.5f)); }
__device__ __forceinline__ f3 bg_sunset(f3 d) { return bg_mix(d, mk3(0.8f, 0.4f, 0.0f), mk3(1.0f, 0.4f, 0.0f)); }
__device__ __forceinline__ f3 bg_sunrise(f3 d) { return bg_mix(d, mk3(0.7f, 0.35f, 0.0f), mk3(0.8f, 0.4f, 0.0f)); }
__device__ __forceinline__ f3 sky_color(float t, uint32_t is_afternoon, f3 dir) {
  const float night_duration = 0.5f, sunrise_duration = 0.10f, full_daylight_transition = 0.10f,
              full_night_transition = 0.10f;
  const float sunrise_end = night_duration + sunrise_duration;
  const float sunrise_to_daylight = sunrise_end + full_daylight_transition;
  const float zenith_transition = 1.0f - sunrise_to_daylight;
  const float daylight_end = 1.0f - zenith_transition;
  const float sunset_start = 1.0f - zenith_transition - sunrise_duration;
  const float sunset_end = 1.0f - zenith_transition - sunrise_duration - full_night_transition;
  if (is_afternoon) {
    if (t < night_duration) return bg_night(dir);
    if (t < sunrise_end) return gmix(bg_night(dir), bg_sunrise(dir), t);
    if (t < sunrise_to_daylight) return gmix(bg_sunrise(dir), bg_sunset(dir), t);
    return gmix(bg_sunset(dir), bg_day(dir), t);
  }
  if (t > daylight_end) return gmix(bg_sunrise(dir), bg_day(dir), t);
  if (t > sunset_start) return gmix(bg_sunset(dir), bg_sunrise(dir), t);
  if (t > sunset_end) return gmix(bg_night(dir), bg_sunset(dir), t);
  return bg_night(dir);
}

// ---------------------------------------------------------------------------
// voxel lookup
__device__ __forceinline__ uint32_t table_entry(const DevAccel &A, const DevGrid &g, int bx, int by, int bz) {
  if ((unsigned)bx >= (unsigned)g.bdim[0] || (unsigned)by >= (unsigned)g.bdim[1] || (unsigned)bz >= (unsigned)g.bdim[2])
    return CT_EMPTY_SLOT;
  return __ldg(&A.brick_table[g.table_offset + ((uint32_t)bz * g.bdim[1] + by) * g.bdim[0] + bx]);
}
// primitive id (instance relative) of grid-local voxel (x,y,z), or -1
__device__ __forceinline__ uint32_t cell_index(const DevGrid &g, int bx, int by, int bz) {
  return g.table_offset + ((uint32_t)bz * g.bdim[1] + by) * g.bdim[0] + bx;
}
__device__ __forceinline__ int32_t voxel_prim(const DevAccel &A, const DevGrid &g, int x, int y, int z) {
  const int bx = x >> 3, by = y >> 3, bz = z >> 3;
  uint32_t e = table_entry(A, g, bx, by, bz);
  if (!(e & CT_NEAR_BIT)) return -1;
  uint32_t slot = e & CT_EMPTY_SLOT;
  uint32_t local = (uint32_t)(x & 7) + 8u * (uint32_t)(y & 7) + 64u * (uint32_t)(z & 7);
  uint32_t w = __ldg(&A.brick_mask[slot * CT_MASK_WORDS + (local >> 5)]);
  if (!((w >> (local & 31u)) & 1u)) return -1;
  uint32_t ps = __ldg(&A.brick_pslot[cell_index(g, bx, by, bz)]);
  return (int32_t)__ldg(&A.brick_prim[ps * 512u + local]);
}

// voxel centre in object space: (AABB.minimum + AABB.maximum) * 0.5
// (primitives.glsl:369, 397, 439, 524)
__device__ __forceinline__ f3 voxel_center(const DevAccel &A, const DevGrid &g, int x, int y, int z, uint32_t prim) {
  if (g.grid_exact) {
    float e = A.extent;
    f3 mn = f3{(float)(x + g.gmin[0]) * e, (float)(y + g.gmin[1]) * e, (float)(z + g.gmin[2]) * e};
    f3 mx = f3{(float)(x + g.gmin[0] + 1) * e, (float)(y + g.gmin[1] + 1) * e, (float)(z + g.gmin[2] + 1) * e};
    return (mn + mx) * 0.5f;
  }
  const ct_aabb &b = A.aabbs[g.first_primitive_index + prim];
  return (ld3(b.minimum) + ld3(b.maximum)) * 0.5f;
}

// primitive id of a voxel known to be occupied (its field code is 0)
__device__ __forceinline__ uint32_t voxel_prim_occupied(const DevAccel &A, const DevGrid &g, int x, int y, int z) {
  const uint32_t local = (uint32_t)(x & 7) + 8u * (uint32_t)(y & 7) + 64u * (uint32_t)(z & 7);
  return __ldg(&A.brick_prim[__ldg(&A.brick_pslot[cell_index(g, x >> 3, y >> 3, z >> 3)]) * 512u + local]);
}

// ---------------------------------------------------------------------------
// The walk over one instance's cell field, offering every voxel whose box the
// ray passes within `eps` voxels of.  The box test (and therefore which voxel
// is hit and at what distance) is rounding-sensitive near voxel edges;
// visiting this superset of candidates makes the result depend only on the
// box test itself, never on the traversal order or on how the walk rounds.
//
// Every step leaves one axis-aligned box of cells through its exit face: the
// cube without occupied cells that the field gives for the ray's octant, with
// the current cell as its corner, taken when the ray stays clear of the
// cube's side faces (so that no voxel beside the cube comes within eps of the
// ray inside it), or a single cell: an occupied one, or the current one when
// the ray passes near a side face of its cube.  A single cell's voxel is
// tested, and its neighbours when the ray passes within eps of their faces.
//
// What bounds the walks is instruction issue, so a step is built from few and
// full-rate instructions:
//  * the ray is mirrored, axis by axis, so that no component of its direction
//    is negative: every box then begins at the current cell, the far faces
//    are the exit candidates and the near ones lie behind the ray;
//  * cells are floats holding whole numbers; adding 2^23 turns one into an
//    index (and, rounding down, a position into its cell), which takes the
//    place of the conversions between integers and floats that run at an
//    eighth of the rate (12 of them a step before);
//  * the distances to the box's lower faces are carried from the step that
//    entered it, the entry face's as a large number, so that the near-face
//    screen is two minima and a compare.
// On the 1080p terrain frame the shadow walker went from 4.80 to 3.04 ms with
// this step, the bounce walker from 1.20 to 0.73 ms and the primary rays from
// 0.98 to 0.78 ms.
#define CT_WALK_FAR 1e30f
#define CT_WALK_MAGIC 8388608.0f  // 2^23

// A ray in grid-local voxel units, mirrored.
//   o.w  margin of the near-face screen, 2 eps + 1e-3
//   d.w  the stop test's allowance per |1/d| of the exit axis
//   inv  1 / d (infinity for an axis the ray does not move along);
//        inv.w (bits) 28 when x is mirrored, else 0
//   g    cells per axis; g.w (bits) first word of the octant's field, less
//        the magic numbers of the cell indices
//   st   word strides of the field along x (+-1 per 8 cells), y and z,
//        negative on mirrored axes; st.w (bits) t at which the ray leaves
//        the grid or its range
struct __align__(16) WalkRay {
  float4 o, d, inv, g;
  int4 st;
};

struct WalkState {
  float cx, cy, cz;  // current cell
  float qx, qy, qz;  // ray's distance past the cell's lower faces where it entered; CT_WALK_FAR for the entry face
  float t;           // where it entered
  float ie;          // |1/d| of the entry axis (-infinity: the walk began in this cell)
  int steps;
  int bkey;          // brick of the current cell (work counters)
};

// one box: its far faces, where and on which axis the ray leaves it
struct WalkBox {
  float hx, hy, hz;
  float t, px, py, pz;
  float ib;  // |1/d| of the exit axis
  int ax;
};

enum { WALK_MORE = 0, WALK_DONE = 1, WALK_LIMIT = 2, WALK_TEST_OWN = 3, WALK_TEST_NEAR = 4 };

__device__ __forceinline__ float walk_eps(const WalkRay &R) { return (R.o.w - 1e-3f) * 0.5f; }

// false: the ray does not overlap the grid within [tmin, tmax].  `ird`: the
// caller's safe_inverse(d_obj), whose reciprocals are the walk's where the
// voxel edge is 1.
__device__ __forceinline__ bool walk_init(const DevAccel &A, const DevGrid &g, f3 o_obj, f3 d_obj, f3 ird, float tmin,
                                          float tmax, WalkRay &R, WalkState &s) {
  const float e = A.extent;
  float o[3], d[3], inv[3];
  // x / e is x * (1 / e) exactly when e is a power of two (the usual voxel
  // edges 1 and 2^-5), and one multiply is far cheaper than an IEEE division
  if ((__float_as_uint(e) & 0x007FFFFFu) == 0u && e > 1e-30f && e < 1e30f) {
    const float ie = 1.0f / e;
    o[0] = o_obj.x * ie; o[1] = o_obj.y * ie; o[2] = o_obj.z * ie;
    d[0] = d_obj.x * ie; d[1] = d_obj.y * ie; d[2] = d_obj.z * ie;
  } else {
    o[0] = o_obj.x / e; o[1] = o_obj.y / e; o[2] = o_obj.z / e;
    d[0] = d_obj.x / e; d[1] = d_obj.y / e; d[2] = d_obj.z / e;
  }
  if (e == 1.0f) {
    inv[0] = ird.x; inv[1] = ird.y; inv[2] = ird.z;
  } else {
    inv[0] = 1.f / d[0]; inv[1] = 1.f / d[1]; inv[2] = 1.f / d[2];
  }
  const int cells[3] = {g.bdim[0] * CT_BRICK, g.bdim[1] * CT_BRICK, g.bdim[2] * CT_BRICK};
  float t0 = tmin, t1 = tmax, L = 0.f;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float G = (float)cells[a], gm = (float)g.gmin[a];
    o[a] = o[a] - gm;
    if (d[a] == 0.f) {
      if (o[a] < 0.f || o[a] > G) return false;
      inv[a] = INFINITY;
    } else {
      const float ta = (0.f - o[a]) * inv[a], tb = (G - o[a]) * inv[a];
      t0 = fmaxf(t0, fminf(ta, tb));
      t1 = fminf(t1, fmaxf(ta, tb));
    }
  }
  if (!(t0 <= t1)) return false;
  // rounding allowance of the box test (see the comment above)
  uint32_t oct = 0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float w = o[a] + (float)g.gmin[a];
    L = fmaxf(L, fmaxf(fabsf(w), fabsf(w + d[a] * t1)));
    if (d[a] < 0.f) {
      oct |= 1u << a;
      o[a] = (float)cells[a] - o[a];
      d[a] = -d[a];
    }
    inv[a] = fabsf(inv[a]);
  }
  const float eps = 2e-4f + 4e-6f * L;
  float c[3], q[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float p = __fmaf_rn(d[a], t0, o[a]);
    c[a] = fmaxf(0.f, fminf(floorf(p), (float)(cells[a] - 1)));
    q[a] = p - c[a];
  }
  const uint32_t Y = (uint32_t)cells[1], Z = (uint32_t)cells[2], bx = (uint32_t)g.bdim[0];
  const int sy = (oct & 2u) ? -(int)bx : (int)bx, sz = (oct & 4u) ? -(int)(bx * Y) : (int)(bx * Y);
  uint32_t base = oct * Z * Y * bx;
  if (oct & 1u) base += bx - 1u;
  if (oct & 2u) base += (Y - 1u) * bx;
  if (oct & 4u) base += (Z - 1u) * Y * bx;
  base -= 0x4B000000u * ((uint32_t)sy + (uint32_t)sz);
  R.o = make_float4(o[0], o[1], o[2], 2.0f * eps + 1e-3f);
  // see walk_advance
  R.d = make_float4(d[0], d[1], d[2], (eps - 2e-4f) * 0.25f + 1e-6f);
  R.inv = make_float4(inv[0], inv[1], inv[2], __uint_as_float((oct & 1u) ? 28u : 0u));
  R.g = make_float4((float)cells[0], (float)cells[1], (float)cells[2], __uint_as_float(base));
  R.st = make_int4((oct & 1u) ? -1 : 1, sy, sz, __float_as_int(t1));
  s.cx = c[0]; s.cy = c[1]; s.cz = c[2];
  s.qx = q[0]; s.qy = q[1]; s.qz = q[2];
  s.t = t0;
  s.ie = -INFINITY;
  s.bkey = -1;
  // the walk's cap: CT_DDA_MAX_STEPS counts from here, so a smaller
  // A.max_steps (a test's) ends the walk after that many cells
  s.steps = CT_DDA_MAX_STEPS - (int)A.max_steps;
  return true;
}

// The t past which the walk's boxes hold nothing that matters, for a stop
// distance `stop`: a box further than its allowance past it cannot beat it.
// Capped below infinity so that a walk whose box the ray never leaves (no
// direction) ends.
__device__ __forceinline__ float walk_limit(const WalkRay &R, float stop) {
  return fminf(fminf(stop + 1e-5f * fabsf(stop) + 1e-6f, __int_as_float(R.st.w)), CT_WALK_FAR);
}

// bits of a cell's whole-number float in the low mantissa
__device__ __forceinline__ uint32_t walk_bits(float c) { return __float_as_uint(c + CT_WALK_MAGIC); }

// the field's edge at the current cell, as a float
__device__ __forceinline__ float walk_field(const uint32_t *field, const WalkRay &R, const WalkState &s) {
  const uint32_t xb = walk_bits(s.cx);
  const uint32_t w = __float_as_uint(R.g.w) + (uint32_t)R.st.x * ((xb & 1023u) >> 3) +
                     (uint32_t)R.st.y * walk_bits(s.cy) + (uint32_t)R.st.z * walk_bits(s.cz);
  const uint32_t code = (__ldg(field + w) >> (((xb << 2) & 28u) ^ __float_as_uint(R.inv.w))) & 15u;
  const bool lo = code < 8u;
  const uint32_t b =
      __byte_perm(lo ? CT_FIELD_EDGES0 : CT_FIELD_EDGES2, lo ? CT_FIELD_EDGES1 : CT_FIELD_EDGES3, code & 7u);
  return __uint_as_float(__byte_perm(b, 0x4B000000u, 0x7440u)) - CT_WALK_MAGIC;  // byte 0 of b
}

// the box of `k` cells per axis from the current cell, clipped to the grid
__device__ __forceinline__ WalkBox walk_box(const WalkRay &R, const WalkState &s, float k) {
  WalkBox b;
  b.hx = fminf(s.cx + k, R.g.x);
  b.hy = fminf(s.cy + k, R.g.y);
  b.hz = fminf(s.cz + k, R.g.z);
  // 0 * infinity (on a face the ray does not move towards) is no exit
  const float tx = (b.hx - R.o.x) * R.inv.x, ty = (b.hy - R.o.y) * R.inv.y, tz = (b.hz - R.o.z) * R.inv.z;
  b.t = fminf(fminf(tx, ty), fminf(tz, INFINITY));
  b.ax = tx == b.t ? 0 : (ty == b.t ? 1 : 2);
  b.ib = b.ax == 0 ? R.inv.x : (b.ax == 1 ? R.inv.y : R.inv.z);
  b.px = __fmaf_rn(R.d.x, b.t, R.o.x);
  b.py = __fmaf_rn(R.d.y, b.t, R.o.y);
  b.pz = __fmaf_rn(R.d.z, b.t, R.o.z);
  return b;
}

// Screen on a box: false only when the ray stays well clear (2 eps + 1e-3
// voxels) of every face of the box other than its entry and exit faces, and
// crosses the box too far from the entry/exit edge to pass near it.  The ray
// does not cross those other faces' planes inside the box and moves away
// from the lower ones, so it is nearest to them where it enters, and to the
// upper ones where it leaves.  A voxel outside the box that the ray passes
// within eps of, while inside the box, lies beyond one of these faces: none
// when this is false.
__device__ __forceinline__ bool walk_near(const WalkRay &R, const WalkState &s, const WalkBox &b) {
  const float ex = b.ax == 0 ? CT_WALK_FAR : b.hx - b.px, ey = b.ax == 1 ? CT_WALK_FAR : b.hy - b.py,
              ez = b.ax == 2 ? CT_WALK_FAR : b.hz - b.pz;
  const float q = fminf(fminf(s.qx, s.qy), s.qz), h = fminf(fminf(ex, ey), ez);
  // eps + margin = 1.5 margin - 5e-4
  return fminf(q, h) < R.o.w || !(b.t - s.t > __fmaf_rn(1.5f, R.o.w, -5e-4f) * (s.ie + b.ib));
}

// Moves on to the cell behind the box's exit face; false when the walk ends.
//
// The next box begins at b.t, computed in grid-local coordinates whose
// rounding (a few ulps of the coordinate scale L, with eps = 2e-4 + 4e-6 L) is
// amplified by |1/d| on the exit axis: a voxel behind that face has box-test
// distance at least b.t - 1e-6 L |1/d|.  The walk ends only when that bound
// (R.d.w holds the allowance) lies past the limit, so that a voxel on the
// same face plane as the best hit (an exact tie) is still seen.
__device__ __forceinline__ bool walk_advance(const WalkRay &R, WalkState &s, const WalkBox &b, float lim) {
  if (b.t - fminf(R.d.w * b.ib, CT_WALK_FAR) > lim) return false;
  // the ray's cell clamped to the box; rounding down to a whole number by the
  // magic addition (positions are within [-1, 1025])
  const float fx = __fadd_rd(b.px, CT_WALK_MAGIC) - CT_WALK_MAGIC, fy = __fadd_rd(b.py, CT_WALK_MAGIC) - CT_WALK_MAGIC,
              fz = __fadd_rd(b.pz, CT_WALK_MAGIC) - CT_WALK_MAGIC;
  s.cx = b.ax == 0 ? b.hx : fmaxf(s.cx, fminf(fx, b.hx - 1.0f));
  s.cy = b.ax == 1 ? b.hy : fmaxf(s.cy, fminf(fy, b.hy - 1.0f));
  s.cz = b.ax == 2 ? b.hz : fmaxf(s.cz, fminf(fz, b.hz - 1.0f));
  s.qx = b.ax == 0 ? CT_WALK_FAR : b.px - s.cx;
  s.qy = b.ax == 1 ? CT_WALK_FAR : b.py - s.cy;
  s.qz = b.ax == 2 ? CT_WALK_FAR : b.pz - s.cz;
  s.t = b.t;
  s.ie = b.ib;
  return s.cx < R.g.x && s.cy < R.g.y && s.cz < R.g.z;
}

// One step.  WALK_TEST_OWN / WALK_TEST_NEAR: the walk stands in a single cell
// whose voxel (and near neighbours) / near neighbours are to be tested before
// it moves on (box: that cell).
template <bool COUNT>
__device__ __forceinline__ int walk_step(const uint32_t *field, const WalkRay &R, WalkState &s, float lim,
                                         RayStats &rs, WalkBox &b) {
  if (++s.steps > CT_DDA_MAX_STEPS) return WALK_LIMIT;
  if (COUNT) {
    // bricks per axis < 128; a mirrored grid's bricks are its bricks
    const int key = (int)(((walk_bits(s.cx) >> 3) & 127u) | (((walk_bits(s.cy) >> 3) & 127u) << 7) |
                          (((walk_bits(s.cz) >> 3) & 127u) << 14));
    if (key != s.bkey) {
      rs.bricks++;
      s.bkey = key;
    }
  }
  const float k = walk_field(field, R, s);
  b = walk_box(R, s, fmaxf(k, 1.0f));
  if (k == 0.0f) return WALK_TEST_OWN;
  if (walk_near(R, s, b)) {
    // the cell alone: a test only when the ray passes near one of its faces
    b = walk_box(R, s, 1.0f);
    if (walk_near(R, s, b)) return WALK_TEST_NEAR;
  }
  return walk_advance(R, s, b, lim) ? WALK_MORE : WALK_DONE;
}

// the grid's cell of a mirrored one
__device__ __forceinline__ int3 walk_cell(const WalkRay &R, int x, int y, int z) {
  return make_int3(R.st.x < 0 ? (int)R.g.x - 1 - x : x, R.st.y < 0 ? (int)R.g.y - 1 - y : y,
                   R.st.z < 0 ? (int)R.g.z - 1 - z : z);
}

// t interval over which the ray lies within eps of the plane coordinate c on
// axis a, clipped to [t0, t1]
__device__ __forceinline__ void near_interval(float o, float d, float inv, float c, float eps, float t0, float t1,
                                              float &lo, float &hi) {
  if (d == 0.f) {
    if (fabsf(o - c) < eps) { lo = t0; hi = t1; } else { lo = 1.f; hi = 0.f; }
    return;
  }
  float ta = (c - eps - o) * inv, tb = (c + eps - o) * inv;
  lo = fmaxf(fminf(ta, tb), t0);
  hi = fminf(fmaxf(ta, tb), t1);
}

// Neighbours of the (mirrored) cell c that the ray passes within eps of while
// it crosses c (t in [t_in, t_out]), except the previous and the next cell of
// the walk, as a mask over the 3x3x3 block (bit (dz+1)*9 + (dy+1)*3 +
// (dx+1)).  Axis 3: none.
__device__ __forceinline__ uint32_t walk_neighbour_mask(float4 ro, float4 rd, float4 ri, float c0, float c1, float c2,
                                                     float t_in, float t_out, int entry_axis, int exit_axis) {
  const float c[3] = {c0, c1, c2};
  const float o[3] = {ro.x, ro.y, ro.z}, d[3] = {rd.x, rd.y, rd.z}, inv[3] = {ri.x, ri.y, ri.z};
  const float eps = (ro.w - 1e-3f) * 0.5f;
  // near-face intervals: [axis][0 = lower face, 1 = upper face]
  float lo[3][2], hi[3][2];
  bool any_other = false;
#pragma unroll
  for (int a = 0; a < 3; a++) {
#pragma unroll
    for (int f = 0; f < 2; f++) {
      near_interval(o[a], d[a], inv[a], c[a] + (float)f, eps, t_in, t_out, lo[a][f], hi[a][f]);
      const bool is_entry = a == entry_axis && f == 0, is_exit = a == exit_axis && f == 1;
      if (!is_entry && !is_exit && lo[a][f] <= hi[a][f]) any_other = true;
    }
  }
  if (!any_other) {
    // only the corner between the entry and exit faces can be near
    if (entry_axis > 2 || entry_axis == exit_axis) return 0u;
    float l = t_in, h = t_out;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (a == entry_axis) { l = fmaxf(l, lo[a][0]); h = fminf(h, hi[a][0]); }
      if (a == exit_axis) { l = fmaxf(l, lo[a][1]); h = fminf(h, hi[a][1]); }
    }
    if (l > h) return 0u;
    const int w[3] = {1, 3, 9};
    int bit = 13;
#pragma unroll
    for (int a = 0; a < 3; a++) bit += (a == exit_axis ? w[a] : 0) - (a == entry_axis ? w[a] : 0);
    return 1u << bit;
  }
  // general case: every neighbour whose touching faces are all near at a
  // common time, except the previous and the next cell of the walk
  uint32_t mask = 0u;
  for (int dz = -1; dz <= 1; dz++)
    for (int dy = -1; dy <= 1; dy++)
      for (int dx = -1; dx <= 1; dx++) {
        const int dd[3] = {dx, dy, dz};
        if (dx == 0 && dy == 0 && dz == 0) continue;
        const int nz = (dx != 0) + (dy != 0) + (dz != 0);
        if (nz == 1) {
          const int a = dx != 0 ? 0 : (dy != 0 ? 1 : 2);
          if (a == entry_axis && dd[a] < 0) continue;
          if (a == exit_axis && dd[a] > 0) continue;
        }
        float l = t_in, h = t_out;
#pragma unroll
        for (int a = 0; a < 3; a++) {
          if (dd[a] == 0) continue;
          const int f = dd[a] > 0 ? 1 : 0;
          l = fmaxf(l, lo[a][f]);
          h = fminf(h, hi[a][f]);
        }
        if (l > h) continue;
        mask |= 1u << ((dz + 1) * 9 + (dy + 1) * 3 + (dx + 1));
      }
  return mask;
}
// The same out of line, for the shadow walker: its walk, step and test phases
// are one kernel (698 us a frame at 1277x719, 711 with the mask inline).  A
// closest-hit walk has the one use and takes it inline: against a call, primary
// rays at 1080p 593 -> 548 us, the path tracer's 512x512 x 8 samples 2.36 -> 2.27 ms.
__device__ __noinline__ uint32_t walk_neighbour_mask_call(float4 ro, float4 rd, float4 ri, float c0, float c1, float c2,
                                                          float t_in, float t_out, int entry_axis, int exit_axis) {
  return walk_neighbour_mask(ro, rd, ri, c0, c1, c2, t_in, t_out, entry_axis, exit_axis);
}
// the axis of the face the walk entered the cell through (3: it began there)
__device__ __forceinline__ int walk_entry(const WalkState &s) {
  return s.qx >= CT_WALK_FAR ? 0 : (s.qy >= CT_WALK_FAR ? 1 : (s.qz >= CT_WALK_FAR ? 2 : 3));
}

// Visitor interface of the walks that test in place:
//   bool visit(int x, int y, int z, uint32_t prim)   returns true to stop
//   float stop_t()                                    boxes entered later are skipped
//   uint32_t tests                                    voxels offered
//
// The tests of the single cell a walk stands in (box b), then the step out of
// it; `st` is what walk_step returned.
template <class V>
__device__ __forceinline__ int walk_test(const DevAccel &A, const DevGrid &g, const WalkRay &R, WalkState &s,
                                         const WalkBox &b, int st, float &lim, V &vis) {
  const int cx = (int)(walk_bits(s.cx) & 1023u), cy = (int)(walk_bits(s.cy) & 1023u),
            cz = (int)(walk_bits(s.cz) & 1023u);
  bool near = true;
  if (st == WALK_TEST_OWN) {
    const int3 c = walk_cell(R, cx, cy, cz);
    vis.tests++;
    if (vis.visit(c.x, c.y, c.z, voxel_prim_occupied(A, g, c.x, c.y, c.z))) return WALK_DONE;
    near = walk_near(R, s, b);
  }
  if (near) {
    for (uint32_t m = walk_neighbour_mask(R.o, R.d, R.inv, s.cx, s.cy, s.cz, s.t, b.t, walk_entry(s), b.ax); m;
         m &= m - 1u) {
      const int nb = __ffs(m) - 1;
      const int3 c = walk_cell(R, cx + nb % 3 - 1, cy + (nb / 3) % 3 - 1, cz + nb / 9 - 1);
      const int32_t pr = voxel_prim(A, g, c.x, c.y, c.z);
      if (pr < 0) continue;
      vis.tests++;
      if (vis.visit(c.x, c.y, c.z, (uint32_t)pr)) return WALK_DONE;
    }
  }
  lim = walk_limit(R, vis.stop_t());
  return walk_advance(R, s, b, lim) ? WALK_MORE : WALK_DONE;
}

// Runs the walk for at most `rounds` rounds of up to `inner` steps and the
// tests of the cell they end in.  The lanes of a warp leave the steps
// together, so that the tests (long, and needed by most walks once) run side
// by side instead of one lane at a time: with the tests inside the step loop
// 5.9 of 32 lanes were active per instruction in the path tracer (512x512,
// 8 samples of depth 3 in a 128^3 grid at 25%, forward: 4.8 -> 1.9 ms).
template <bool COUNT, class V>
__device__ __forceinline__ int walk_run(const DevAccel &A, const DevGrid &g, const WalkRay &R, WalkState &s, V &vis,
                                        RayStats &rs, int rounds, int inner) {
  const uint32_t *field = A.cell_field + g.field_offset;
  float lim = walk_limit(R, vis.stop_t());
  for (int it = 0; it < rounds; it++) {
    int st = WALK_MORE;
    WalkBox b;
#pragma unroll 1
    for (int k = 0; k < inner && st == WALK_MORE; k++) st = walk_step<COUNT>(field, R, s, lim, rs, b);
    if (st >= WALK_TEST_OWN) st = walk_test(A, g, R, s, b, st, lim, vis);
    if (st != WALK_MORE) return st;
  }
  return WALK_MORE;
}

// Steps per round of a walk that runs to its end in place: 8 (primary rays
// 0.757 ms per 1080p frame against 0.776 ms at 4 and 0.800 ms at 2).
#ifndef CT_WALK_INNER
#define CT_WALK_INNER 8
#endif
// Returns false if the walk hit its step cap (error latched by the caller).
template <class V>
__device__ __forceinline__ bool walk_traverse(const DevAccel &A, const DevGrid &g, f3 o_obj, f3 d_obj, f3 ird,
                                              float tmin, float tmax, V &vis, RayStats &rs) {
  WalkRay R;
  WalkState s;
  if (!walk_init(A, g, o_obj, d_obj, ird, tmin, tmax, R, s)) return true;
  return walk_run<true>(A, g, R, s, vis, rs, CT_DDA_MAX_STEPS + 1, CT_WALK_INNER) != WALK_LIMIT;
}

// ---------------------------------------------------------------------------
// Hit rules
//
// closest hit by box-test distance, ties -> lowest global primitive index.
struct HitRecord {
  bool hit;
  float t;
  uint32_t inst, prim, gprim;
};
__device__ __forceinline__ bool hit_better(float t, uint32_t g, const HitRecord &b) {
  return !b.hit || t < b.t || (t == b.t && g < b.gprim);
}

// Closest hit.  PRIMARY: intersection shader semantics (rint.glsl:10-43 with
// is_hit_from_ray_providing_model, primitives.glsl:357-382): object-space ray
// from the instance's TLAS transform, oriented box test (division), hits
// reported for t > 0.  Otherwise ray-query semantics (bounce.glsl:85-119):
// candidates are tested with is_hit_from_ray (primitives.glsl:412-453):
// object-space ray from the inverse of INSTANCE.transform, non-oriented box
// test (multiplication by safeInverse(direction)), hits for t >= 0.  Rays may
// start inside a box; hits lie within [0, tmax].
// a walk's object-space ray and the reciprocal direction the box test takes
struct ObjRay {
  f3 ro, rd, ird;
};
template <bool PRIMARY>
struct ClosestVisitor {
  const DevAccel &A; const DevGrid &g;
  const ObjRay &R;
  f3 radius, inv_radius;
  float tmax;
  uint32_t inst;
  HitRecord &best;
  uint32_t tests;
  __device__ float stop_t() const { return best.hit ? best.t : tmax; }
  __device__ bool visit(int x, int y, int z, uint32_t prim) {
    f3 c = voxel_center(A, g, x, y, z, prim);
    BoxHit h = box_test(c, radius, inv_radius, R.ro, R.rd, true, PRIMARY, R.ird);
    if (!h.hit) return false;
    const float t = h.t;
    if (PRIMARY ? !(t > 0.f) : !(t >= 0.f)) return false;
    if (!(t <= (best.hit ? best.t : tmax))) return false;
    uint32_t gp = g.first_primitive_index + prim;
    if (hit_better(t, gp, best)) { best.hit = true; best.t = t; best.inst = inst; best.prim = prim; best.gprim = gp; }
    return false;
  }
};

// Visibility with ray-query semantics (light.glsl:106-137): the first hit in
// (t, primitive) order with t in [0, tmax] decides; it blocks unless it is
// the light's own voxel.
struct VisibilityVisitor {
  const DevAccel &A; const DevGrid &g;
  f3 ro, rd, ird;  // object space
  f3 radius, inv_radius;
  float tmax;
  uint32_t inst;
  // decisive key of the target
  float target_t; uint32_t target_g; bool has_target; uint32_t target_inst, target_prim;
  bool blocked;
  uint32_t tests;
  __device__ float stop_t() const { return fminf(tmax, target_t); }
  __device__ bool visit(int x, int y, int z, uint32_t prim) {
    if (has_target && inst == target_inst && prim == target_prim) return false;
    BoxHit h = box_test(voxel_center(A, g, x, y, z, prim), radius, inv_radius, ro, rd, false, false, ird);
    if (!h.hit) return false;
    const float t = h.t;
    if (!(t >= 0.f && t <= tmax)) return false;
    const uint32_t gp = g.first_primitive_index + prim;
    blocked = t < target_t || (t == target_t && gp < target_g);
    return blocked;
  }
};

__device__ __forceinline__ f3 half_extent_v(const DevAccel &A) { float h = A.extent * 0.5f; return f3{h, h, h}; }

// A closest hit as a resumable walk over every instance in turn, so that a
// warp can refill lanes whose ray is done.  PRIMARY: a camera ray (traceRayEXT
// with the RIS_SELECTION hit group); otherwise intersect()'s bounce ray
// (bounce.glsl:9-125), whose origin compute_ray_origin(origin, direction)
// moves.  The walk's ray and the object-space one the box tests read lie in
// memory the caller places (shared memory in the walkers).
struct ClosestRay {
  WalkRay &r;
  ObjRay &obj;
};
struct ClosestWalk {
  uint32_t inst;     // instance being walked
  WalkState s;
  HitRecord best;
};
// The first instance from w.inst on whose grid the ray overlaps; false when
// none is left.  `ray(o, d)` gives the world-space ray, which the walk does
// not keep (the walkers are register bound).
template <bool PRIMARY, class RayFn>
__device__ __forceinline__ bool closest_walk_instance(const DevAccel &A, ClosestWalk &w, float tmax, const RayFn &ray,
                                                      const ClosestRay &R) {
  for (; w.inst < A.n_grids; w.inst++) {
    const DevGrid &g = A.grids[w.inst];
    f3 o, d;
    ray(o, d);
    const m4 &m = PRIMARY ? g.world2obj_tlas : g.world2obj_inst;
    const f3 ro = xyz(mul(m, mk4(PRIMARY ? o : compute_ray_origin(o, d), 1.0f)));
    const f3 rd = xyz(mul(m, mk4(d, 0.0f)));
    const f3 ird = safe_inverse(rd);
    WalkRay r;
    if (walk_init(A, g, ro, rd, ird, 0.f, w.best.hit ? w.best.t : tmax, r, w.s)) {
      R.r = r;
      R.obj.ro = ro;
      R.obj.rd = rd;
      R.obj.ird = ird;
      return true;
    }
  }
  return false;
}
// true when the ray is already decided (no instance to walk)
template <bool PRIMARY, class RayFn>
__device__ __forceinline__ bool closest_walk_begin(const DevAccel &A, ClosestWalk &w, float tmax, const RayFn &ray,
                                                   const ClosestRay &R) {
  w.best = HitRecord{false, 0.f, 0u, 0u, 0u};
  w.inst = 0;
  return !closest_walk_instance<PRIMARY>(A, w, tmax, ray, R);
}
// The walk through the current instance: WALK_MORE, or how it ended.
template <bool PRIMARY, bool COUNT>
__device__ __forceinline__ int closest_walk_run(const DevAccel &A, ClosestWalk &w, float tmax, int rounds, int inner,
                                                uint32_t pixel, RayStats &rs, const ClosestRay &R) {
  const f3 radius = half_extent_v(A), inv_radius = safe_inverse(radius);
  const DevGrid &g = A.grids[w.inst];
  ClosestVisitor<PRIMARY> v{A, g, R.obj, radius, inv_radius, tmax, w.inst, w.best, 0u};
  const int st = walk_run<COUNT>(A, g, R.r, w.s, v, rs, rounds, inner);
  rs.voxel_tests += v.tests;
  if (st == WALK_LIMIT) ct_latch_error(CT_ERR_ITER_LIMIT, PRIMARY ? 1 : 4, pixel);
  return st;
}
template <bool PRIMARY, bool COUNT, class RayFn>
__device__ __forceinline__ int closest_walk_advance(const DevAccel &A, ClosestWalk &w, float tmax, int rounds,
                                                    int inner, uint32_t pixel, RayStats &rs, const RayFn &ray,
                                                    const ClosestRay &R) {
  if (closest_walk_run<PRIMARY, COUNT>(A, w, tmax, rounds, inner, pixel, rs, R) == WALK_MORE) return WALK_MORE;
  w.inst++;
  return closest_walk_instance<PRIMARY>(A, w, tmax, ray, R) ? WALK_MORE : WALK_DONE;
}
// The whole walk in place; false: no hit.  One set-up serves every instance:
// a second copy of it is instruction fetch, which stalls the path tracer most
// (one sample to depth 8 at 1277 x 719: 585 us with two copies, 568 us with
// one).  The refilling walkers keep two: with one, a lane waits a phase for
// its set-up (a 1080p frame's extension rays 742 -> 890 us).
template <bool PRIMARY>
__device__ __forceinline__ bool closest_walk(const DevAccel &A, ClosestWalk &w, f3 origin, f3 dir, float tmax,
                                             uint32_t pixel, RayStats &rs) {
  WalkRay r;
  ObjRay obj;
  const ClosestRay R{r, obj};
  const auto ray = [&](f3 &o, f3 &d) { o = origin; d = dir; };
  w.best = HitRecord{false, 0.f, 0u, 0u, 0u};
  for (w.inst = 0; closest_walk_instance<PRIMARY>(A, w, tmax, ray, R); w.inst++)
    closest_walk_run<PRIMARY, true>(A, w, tmax, 1 << 20, CT_WALK_INNER, pixel, rs, R);
  return w.best.hit;
}

// closest hit of a camera ray in place
__device__ HitRecord trace_primary(const DevAccel &A, f3 o, f3 d, float tmax, uint32_t pixel, RayStats &rs) {
  HitRecord best = {false, 0.f, 0u, 0u, 0u};
  const f3 radius = half_extent_v(A), inv_radius = safe_inverse(radius);
  for (uint32_t i = 0; i < A.n_grids; i++) {
    const DevGrid &g = A.grids[i];
    ObjRay R;
    R.ro = xyz(mul(g.world2obj_tlas, mk4(o, 1.0f)));
    R.rd = xyz(mul(g.world2obj_tlas, mk4(d, 0.0f)));
    R.ird = safe_inverse(R.rd);
    ClosestVisitor<true> v{A, g, R, radius, inv_radius, tmax, i, best, 0u};
    if (!walk_traverse(A, g, R.ro, R.rd, R.ird, 0.f, best.hit ? best.t : tmax, v, rs))
      ct_latch_error(CT_ERR_ITER_LIMIT, 1, pixel);
    rs.voxel_tests += v.tests;
  }
  return best;
}

// is_vertex_visible (light.glsl:82-142) under the visibility rule above.
__device__ bool vertex_visible(const DevAccel &A, f3 o, f3 d, float distance, uint32_t t_inst, uint32_t t_prim,
                               bool check_instance, uint32_t pixel, RayStats &rs) {
  const f3 radius = half_extent_v(A), inv_radius = safe_inverse(radius);
  // key of the target voxel (the decisive order is (t, global primitive))
  float target_t = INFINITY;
  uint32_t target_g = 0xFFFFFFFFu;
  bool has_target = check_instance && t_inst < A.n_grids;
  if (has_target) {
    const DevGrid &g = A.grids[t_inst];
    if (t_prim < g.primitive_count) {
      uint32_t gp = g.first_primitive_index + t_prim;
      uint32_t pk = __ldg(&A.voxel_coord[gp]);
      int x = (int)(pk & 0x3FFu), y = (int)((pk >> 10) & 0x3FFu), z = (int)((pk >> 20) & 0x3FFu);
      f3 ro = xyz(mul(g.world2obj_inst, mk4(o, 1.0f)));
      f3 rd = xyz(mul(g.world2obj_inst, mk4(d, 0.0f)));
      f3 c = voxel_center(A, g, x, y, z, t_prim);
      BoxHit h = box_test(c, radius, inv_radius, ro, rd, false, false, safe_inverse(rd));
      if (h.hit && h.t >= 0.f && h.t <= distance) { target_t = h.t; target_g = gp; }
    }
  }
  for (uint32_t i = 0; i < A.n_grids; i++) {
    const DevGrid &g = A.grids[i];
    f3 ro = xyz(mul(g.world2obj_inst, mk4(o, 1.0f)));
    f3 rd = xyz(mul(g.world2obj_inst, mk4(d, 0.0f)));
    const f3 ird = safe_inverse(rd);
    VisibilityVisitor v{A, g, ro, rd, ird, radius, inv_radius, distance, i, target_t, target_g, has_target, t_inst,
                        t_prim, false, 0u};
    float tlim = fminf(distance, target_t);
    if (!walk_traverse(A, g, ro, rd, ird, 0.f, tlim, v, rs)) ct_latch_error(CT_ERR_ITER_LIMIT, 2, pixel);
    rs.voxel_tests += v.tests;
    if (v.blocked) return false;
  }
  return true;
}

// is_vertex_visible with previous_frame set (light.glsl:82-142 over
// p.tlas_previous), for temporal reuse after a scene edit.  Candidates come
// from the previous scene's brick map `A`: a primitive is a candidate when
// its voxel box in that scene passes the query's box test with t in
// [0, distance] -- the boxes a BVH over the previous AABBs reports.  The
// intersection shader then tests the CURRENT AABB of the same (instance,
// primitive) id: is_hit_from_ray (primitives.glsl:412-453) reads
// WORLD.aabb_address and, with previous_frame set, the current INSTANCE.
// The first candidate in (t, primitive) order decides, as in vertex_visible.
// Needs exact voxel grids in `A` (the previous boxes are recomputed from
// their integer coordinates).
struct PrevQueryVisitor {
  const DevAccel &A; const DevGrid &g;
  const ct_aabb *aabbs;
  uint32_t cur_first;
  f3 ro, rd, inv_rd;
  f3 radius, inv_radius;
  float tmax;
  uint32_t inst;
  float target_t; uint32_t target_g; bool has_target; uint32_t target_inst, target_prim;
  bool blocked;
  uint32_t tests;
  __device__ float stop_t() const { return tmax; }
  __device__ bool visit(int x, int y, int z, uint32_t prim) {
    if (has_target && inst == target_inst && prim == target_prim) return false;
    const BoxHit h0 = box_test(voxel_center(A, g, x, y, z, prim), radius, inv_radius, ro, rd, false, false, inv_rd);
    if (!h0.hit || !(h0.t >= 0.f && h0.t <= tmax)) return false;
    const ct_aabb &b = aabbs[cur_first + prim];
    const BoxHit h = box_test((ld3(b.minimum) + ld3(b.maximum)) * 0.5f, radius, inv_radius, ro, rd, false, false, inv_rd);
    if (!h.hit || !(h.t >= 0.f && h.t <= tmax)) return false;
    const uint32_t gp = g.first_primitive_index + prim;
    if (h.t < target_t || (h.t == target_t && gp < target_g)) {
      blocked = true;
      return true;
    }
    return false;
  }
};

__device__ bool vertex_visible_prev(const DevAccel &A, const FrameView &F, f3 o, f3 d, float distance,
                                    uint32_t t_inst, uint32_t t_prim, bool check_instance, uint32_t pixel,
                                    RayStats &rs) {
  const f3 radius = half_extent_v(A), inv_radius = safe_inverse(radius);
  for (uint32_t i = 0; i < A.n_grids; i++)
    if (!A.grids[i].grid_exact) {
      ct_latch_error(CT_ERR_UNSUPPORTED, 41, pixel);
      return true;
    }
  float target_t = INFINITY;
  uint32_t target_g = 0xFFFFFFFFu;
  const bool has_target = check_instance && t_inst < A.n_grids;
  if (has_target) {
    const DevGrid &g = A.grids[t_inst];
    if (t_prim < g.primitive_count) {
      const uint32_t gp = g.first_primitive_index + t_prim;
      const uint32_t pk = __ldg(&A.voxel_coord[gp]);
      const int x = (int)(pk & 0x3FFu), y = (int)((pk >> 10) & 0x3FFu), z = (int)((pk >> 20) & 0x3FFu);
      const f3 ro = xyz(mul(g.world2obj_inst, mk4(o, 1.0f)));
      const f3 rd = xyz(mul(g.world2obj_inst, mk4(d, 0.0f)));
      const f3 inv_rd = safe_inverse(rd);
      const BoxHit h0 = box_test(voxel_center(A, g, x, y, z, t_prim), radius, inv_radius, ro, rd, false, false, inv_rd);
      if (h0.hit && h0.t >= 0.f && h0.t <= distance) {
        const ct_aabb &b = F.aabbs[F.instances[t_inst].first_primitive_index + t_prim];
        const BoxHit h =
            box_test((ld3(b.minimum) + ld3(b.maximum)) * 0.5f, radius, inv_radius, ro, rd, false, false, inv_rd);
        if (h.hit && h.t >= 0.f && h.t <= distance) { target_t = h.t; target_g = gp; }
      }
    }
  }
  for (uint32_t i = 0; i < A.n_grids; i++) {
    const DevGrid &g = A.grids[i];
    const f3 ro = xyz(mul(g.world2obj_inst, mk4(o, 1.0f)));
    const f3 rd = xyz(mul(g.world2obj_inst, mk4(d, 0.0f)));
    PrevQueryVisitor v{A, g, F.aabbs, F.instances[i].first_primitive_index, ro, rd, safe_inverse(rd), radius,
                       inv_radius, distance, i, target_t, target_g, has_target, t_inst, t_prim, false, 0u};
    if (!walk_traverse(A, g, ro, rd, safe_inverse(rd), 0.f, distance, v, rs)) ct_latch_error(CT_ERR_ITER_LIMIT, 3, pixel);
    rs.voxel_tests += v.tests;
    if (v.blocked) return false;
  }
  return true;
}

// ---------------------------------------------------------------------------
// vertex_visible split for k_trace_shadow into a stepping phase and a testing
// phase.  A visibility query's decision does not depend on the order in which
// candidates are tested: the stop distance is fixed (min(distance, target
// t)), and the ray is blocked when ANY candidate voxel other than the target
// passes the box test with t in [0, distance] and a key below the target's.
// So a lane may step on past a cell with tests to make (its own voxel and the
// neighbours the ray passes within eps of, exactly the candidates walk_run
// offers) and leave them to a job that the warp tests later, 32 jobs at a
// time, one per lane.  The stepping phase keeps only the cheap part (the
// field's word and the near-face screen, which rule out nearly all cells);
// the box tests and neighbour masks, rare and long, run with full warps
// instead of one lane at a time.  A lane may enumerate a few cells past its
// first blocker; the decision is the same.

// a lane's ray as both phases read it, kept in shared memory
struct ShadowRay {
  WalkRay r;              // as walk_init made it
  f3 ro, rd, ird;         // object space, and safe_inverse(rd) as the box test takes it
  float tmax;             // the query distance
  float target_t;         // key of the target voxel (INFINITY: none)
  uint32_t target_g;
  uint32_t target_inst;   // 0xFFFFFFFF when the query does not check an instance
  uint32_t target_prim;
  uint32_t inst;          // instance being walked
};

// is_vertex_visible's set-up (light.glsl:82-105): the query, and the target
// voxel's key by its own box test.  True: `obj` is the object-space ray of
// instance 0, where the walk begins (the target's, usually).
__device__ __forceinline__ bool shadow_ray_target(const DevAccel &A, ShadowRay &R, ObjRay &obj, f3 o, f3 d,
                                                  float distance, uint32_t t_inst, uint32_t t_prim,
                                                  bool check_instance) {
  R.tmax = distance;
  R.target_t = INFINITY;
  R.target_g = 0xFFFFFFFFu;
  const bool has_target = check_instance && t_inst < A.n_grids;
  R.target_inst = has_target ? t_inst : 0xFFFFFFFFu;
  R.target_prim = t_prim;
  if (!has_target) return false;
  const DevGrid &g = A.grids[t_inst];
  if (t_prim >= g.primitive_count) return false;
  const f3 radius = half_extent_v(A), inv_radius = safe_inverse(radius);
  const uint32_t gp = g.first_primitive_index + t_prim;
  const uint32_t pk = __ldg(&A.voxel_coord[gp]);
  const int x = (int)(pk & 0x3FFu), y = (int)((pk >> 10) & 0x3FFu), z = (int)((pk >> 20) & 0x3FFu);
  obj.ro = xyz(mul(g.world2obj_inst, mk4(o, 1.0f)));
  obj.rd = xyz(mul(g.world2obj_inst, mk4(d, 0.0f)));
  obj.ird = safe_inverse(obj.rd);
  const BoxHit h =
      box_test(voxel_center(A, g, x, y, z, t_prim), radius, inv_radius, obj.ro, obj.rd, false, false, obj.ird);
  if (h.hit && h.t >= 0.f && h.t <= distance) { R.target_t = h.t; R.target_g = gp; }
  return t_inst == 0u;
}

// The first instance from `inst` on whose grid the ray overlaps; false when
// none is left.  `known`: `obj` is the object-space ray of instance `inst`.
__device__ __forceinline__ bool shadow_ray_next(const DevAccel &A, ShadowRay &R, ObjRay obj, WalkState &s,
                                                uint32_t inst, f3 o, f3 d, bool known) {
#pragma unroll 1
  for (; inst < A.n_grids; inst++, known = false) {
    const DevGrid &g = A.grids[inst];
    if (!known) {
      obj.ro = xyz(mul(g.world2obj_inst, mk4(o, 1.0f)));
      obj.rd = xyz(mul(g.world2obj_inst, mk4(d, 0.0f)));
      obj.ird = safe_inverse(obj.rd);
    }
    WalkRay r;
    if (walk_init(A, g, obj.ro, obj.rd, obj.ird, 0.f, fminf(R.tmax, R.target_t), r, s)) {
      R.r = r;
      R.ro = obj.ro;
      R.rd = obj.rd;
      R.ird = obj.ird;
      R.inst = inst;
      return true;
    }
  }
  return false;
}

// VisibilityVisitor::visit on the stored ray: true when voxel
// (x, y, z) = primitive `prim` of the instance blocks the ray
__device__ __forceinline__ bool shadow_blocks(const DevAccel &A, const DevGrid &g, const ShadowRay &R, int x, int y,
                                              int z, uint32_t prim) {
  if (R.inst == R.target_inst && prim == R.target_prim) return false;
  const f3 radius = half_extent_v(A), inv_radius = safe_inverse(radius);
  const BoxHit h = box_test(voxel_center(A, g, x, y, z, prim), radius, inv_radius, R.ro, R.rd, false, false, R.ird);
  if (!h.hit) return false;
  const float t = h.t;
  if (!(t >= 0.f && t <= R.tmax)) return false;
  const uint32_t gp = g.first_primitive_index + prim;
  return t < R.target_t || (t == R.target_t && gp < R.target_g);
}

// A cell's job: the (mirrored) cell crossed over [t_in, t_out], entered
// across axis `entry` (3: the walk began in it) and left across `exit`, with
// its own voxel to test or its near neighbours alone.
// Packed: x = cx | cy << 10 | cz << 20 | entry << 30, y = lane | exit << 5 | own << 7 | near << 8.
__device__ __forceinline__ uint4 shadow_job(const WalkRay &R, const WalkState &s, const WalkBox &b, bool own,
                                            uint32_t lane) {
  const uint32_t near = !own || walk_near(R, s, b) ? 1u : 0u;
  return make_uint4((walk_bits(s.cx) & 1023u) | ((walk_bits(s.cy) & 1023u) << 10) |
                        ((walk_bits(s.cz) & 1023u) << 20) | ((uint32_t)walk_entry(s) << 30),
                    lane | ((uint32_t)b.ax << 5) | (own ? 128u : 0u) | (near << 8), __float_as_uint(s.t),
                    __float_as_uint(b.t));
}
__device__ __forceinline__ uint32_t shadow_job_lane(uint4 j) { return j.y & 31u; }

// The tests of one job, those walk_run makes in a single cell: the cell's own
// voxel, then the neighbours the ray passes within eps of.
__device__ __forceinline__ bool shadow_job_blocked(const DevAccel &A, const ShadowRay &R, uint4 j, uint32_t &tests) {
  const DevGrid &g = A.grids[R.inst];
  const int cx = (int)(j.x & 0x3FFu), cy = (int)((j.x >> 10) & 0x3FFu), cz = (int)((j.x >> 20) & 0x3FFu);
  if (j.y & 128u) {
    const int3 c = walk_cell(R.r, cx, cy, cz);
    tests++;
    if (shadow_blocks(A, g, R, c.x, c.y, c.z, voxel_prim_occupied(A, g, c.x, c.y, c.z))) return true;
  }
  if (!(j.y & 256u)) return false;
  for (uint32_t m = walk_neighbour_mask_call(R.r.o, R.r.d, R.r.inv, (float)cx, (float)cy, (float)cz, __uint_as_float(j.z),
                                        __uint_as_float(j.w), (int)(j.x >> 30), (int)((j.y >> 5) & 3u));
       m; m &= m - 1u) {
    const int k = __ffs(m) - 1;
    const int3 c = walk_cell(R.r, cx + k % 3 - 1, cy + (k / 3) % 3 - 1, cz + k / 9 - 1);
    const int32_t pr = voxel_prim(A, g, c.x, c.y, c.z);
    if (pr < 0) continue;
    tests++;
    if (shadow_blocks(A, g, R, c.x, c.y, c.z, (uint32_t)pr)) return true;
  }
  return false;
}

// One step of the walk without its visits: leaves the current box; a single
// cell with a test to make sets `job` (its tests are the caller's).
// WALK_MORE, WALK_DONE (left the grid or passed the limit) or WALK_LIMIT.
template <bool COUNT>
__device__ __forceinline__ int shadow_step(const uint32_t *field, const WalkRay &R, WalkState &s, float lim,
                                           uint32_t lane, RayStats &rs, bool &job, uint4 &jb) {
  WalkBox b;
  const int st = walk_step<COUNT>(field, R, s, lim, rs, b);
  job = st >= WALK_TEST_OWN;
  if (!job) return st;
  jb = shadow_job(R, s, b, st == WALK_TEST_OWN, lane);
  return walk_advance(R, s, b, lim) ? WALK_MORE : WALK_DONE;
}

// ---------------------------------------------------------------------------
// Unit axis vectors (one component +-1, the others +-0) are what voxel faces
// give for normals.  normalize() returns them unchanged, bit for bit (the
// length is exactly 1 and x/1 == x, signed zeros included), so the helpers
// below skip the square root and the divisions for them.
__device__ __forceinline__ bool is_unit_axis(f3 v) {
  const float ax = fabsf(v.x), ay = fabsf(v.y), az = fabsf(v.z);
  return (ax == 1.0f && ay == 0.0f && az == 0.0f) || (ax == 0.0f && ay == 1.0f && az == 0.0f) ||
         (ax == 0.0f && ay == 0.0f && az == 1.0f);
}
__device__ __forceinline__ f3 normalize_n(f3 v) { return is_unit_axis(v) ? v : normalize(v); }

// materials (mat.glsl:24-88, light.glsl:200-229)
__device__ __forceinline__ void orthonormal_basis(f3 n, f3 &t1, f3 &t2) {
  if (fabsf(n.x) > fabsf(n.y)) t1 = normalize_n(f3{-n.z, 0.0f, n.x});
  else t1 = normalize_n(f3{0.0f, n.z, -n.y});
  t2 = normalize_n(cross(n, t1));
}
// z component of to_local(n, v) = dot(v, normalize(n)) (mat.glsl:58-64); the
// other two components are dot(u,w) and dot(v2,w) of the basis and unused by
// the Lambertian lobe.
__device__ __forceinline__ float local_z(f3 n, f3 v) { return dot(v, normalize_n(n)); }

__device__ __forceinline__ f3 evaluate_material(const Material &m, f3 n, f3 wo, f3 wi) {
  switch (m.type & 0xFFu) {
    case 1u: {  // metal (mat.glsl:30-36)
      f3 half_dir = normalize(wi + wo);
      float r = gmin(m.roughness, 1.0f);
      float p = ct_powf(1.0f - dot(wi, half_dir), 5.0f);
      f3 fres = mk3(r) + (mk3(1.0f) - mk3(r)) * p;
      f3 diff = (mk3(1.0f) - fres) * (mk3(1.0f) - m.specular);
      f3 spec = fres * m.specular;
      return (diff + spec) * 0.31830988618379067153776752674503f;
    }
    case 2u: {  // dielectric (mat.glsl:38-50)
      float p = ct_powf(1.0f - dot(wi, wo), 5.0f);
      f3 fres = mk3(m.roughness) + (mk3(1.0f) - mk3(m.roughness)) * p;
      f3 diff = (mk3(1.0f) - fres) * (m.diffuse * 0.31830988618379067153776752674503f);
      return diff + fres;
    }
    case 3u:  // constant medium (mat.glsl:53-55)
      return m.diffuse * 0.079577471545947667884441881686255f;
    default: {
      float wo_z = local_z(n, wo), wi_z = local_z(n, wi);
      if (gmin(wo_z, wi_z) < 1e-6f) return mk3(0.f);
      return m.diffuse * 0.31830988618379067153776752674503f * wi_z;
    }
  }
}
__device__ __forceinline__ float sample_material_pdf(const Material &m, f3 n, f3 wo, f3 wi) {
  switch (m.type & 0xFFu) {
    case 1u: case 2u: return 6.283185307179586476925286766559f;
    case 3u: return 12.566370614359172953850573533118f;
    default: {
      float wo_z = local_z(n, wo), wi_z = local_z(n, wi);
      if (gmin(wo_z, wi_z) < 1e-6f) return 0.f;
      return 0.31830988618379067153776752674503f * wi_z;
    }
  }
}
// The same out of line, for the reconnection shift, which needs it four times
// (temporal and spatial shifts of a 1080p frame 987 -> 960 us).
__device__ __noinline__ float sample_material_pdf_call(const Material &m, f3 n, f3 wo, f3 wi) {
  return sample_material_pdf(m, n, wo, wi);
}

// ---------------------------------------------------------------------------
// light sampling (light.glsl:160-164, 295-435; prng.glsl:64-173)
__device__ __forceinline__ float geom_fact_sa(f3 P, f3 Ps, f3 ns) {
  f3 dir = normalize(Ps - P);
  float dist2 = dot(Ps - P, Ps - P);
  return fabsf(dot(ns, dir)) / dist2;
}
__device__ __forceinline__ f3 random_cube_normal(uint32_t &seed) {
  uint32_t face = gmin(urnd_interval(seed, 0u, 6u), 5u);
  switch (face) {
    case 0: return f3{-1.f, 0.f, 0.f};
    case 1: return f3{1.f, 0.f, 0.f};
    case 2: return f3{0.f, -1.f, 0.f};
    case 3: return f3{0.f, 1.f, 0.f};
    case 4: return f3{0.f, 0.f, -1.f};
    default: return f3{0.f, 0.f, 1.f};
  }
}
__device__ __forceinline__ f3 random_quad(f3 n, f3 p, f2 s, uint32_t &seed) {
  float u = rnd(seed);
  float v = rnd(seed);
  f2 q = f2{u, v} * s;
  f3 xa, ya;
  orthonormal_basis(n, xa, ya);
  return p + xa * q.x + ya * q.y;
}
__device__ __forceinline__ f3 random_unit_vector(uint32_t &seed, uint32_t pixel) {
  f3 p = f3{0.f, 0.f, 0.f};
  // not unrolled: the copies cost more instruction fetch than they save
  // (spatial_sample 1.235 -> 1.195 ms, first candidates 766 -> 753 us at 1080p)
#pragma unroll 1
  for (int i = 0; i < CT_SAMPLER_MAX_TRIES; i++) {
    float a = -1.0f + rnd(seed) * (1.0f - -1.0f);
    float b = -1.0f + rnd(seed) * (1.0f - -1.0f);
    float c = -1.0f + rnd(seed) * (1.0f - -1.0f);
    p = f3{a, b, c};
    if (p.x * p.x + p.y * p.y + p.z * p.z >= 1.0f) {
      if (i == CT_SAMPLER_MAX_TRIES - 1) ct_latch_error(CT_ERR_ITER_LIMIT, 3, pixel);
      continue;
    }
    break;
  }
  return normalize(p);
}

// The tries of a cube light's sampling loop for a shading point whose normal n
// is a unit axis, by signs alone.  A try draws a face and two quad coordinates
// and succeeds when the face looks at P and the point lies in front of P's
// plane.  With axis vectors both tests are the sign of one difference of
// coordinates:
//   * whether a face looks at P depends on the face alone, and so does the
//     second test for the two faces parallel to P's plane: one bit per face,
//     worked out once per light;
//   * for the other faces the second test needs the point's coordinate along
//     n, which is the light's plus or minus one of the two draws
//     (orthonormal_basis of the face's normal).
// Each quantity is computed as the full sample computes it, so the outcome of
// every try is the same.  A try costs a third of the full sample's
// instructions (RIS 1.32 -> 0.86 ms, spatial re-evaluation 1.40 -> 1.23 ms per
// 1080p terrain frame).
struct CubeTries {
  uint32_t ok, free_, use_u, neg;  // one bit per face, in random_cube_normal's order
  float pos, half_quad, p, sn;     // along n: the light's position, P; sign of n
  __device__ __forceinline__ CubeTries(f3 P, f3 n, const Light &l) {
    const float lp[3] = {l.position.x, l.position.y, l.position.z}, pp[3] = {P.x, P.y, P.z};
    const float half_extent = l.size * 0.5f;
    const int b = n.x != 0.f ? 0 : (n.y != 0.f ? 1 : 2);
    sn = b == 0 ? n.x : (b == 1 ? n.y : n.z);
    ok = 0u;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float vm = pp[a] - (lp[a] + -1.f * half_extent), vp = pp[a] - (lp[a] + 1.f * half_extent);
      bool m = vm * -1.f > 0.f, q = vp * 1.f > 0.f;
      if (a == b) {
        m = m && vm * sn < 0.f;
        q = q && vp * sn < 0.f;
        pos = lp[a];
        p = pp[a];
      }
      ok |= (m ? 1u : 0u) << (2 * a) | (q ? 2u : 0u) << (2 * a);
    }
    free_ = 3u << (2 * b);
    use_u = b == 0 ? 0u : (b == 1 ? 0x30u : 0x0Fu);
    neg = b == 0 ? 0x3Cu : (b == 1 ? 0x13u : 0x09u);
    half_quad = l.size * 0.5f;
  }
  // one try: advances the stream by its three draws
  __device__ __forceinline__ bool operator()(uint32_t &seed) const {
    const uint32_t r = lcg(seed), u = lcg(seed), v = lcg(seed);
    // floor of the rounded product rnd * 6, which differs from the exact one
    // for a single value of the 24 bits
    const uint32_t bit = 1u << (((r * 6u) >> 24) + (r == 13981013u ? 1u : 0u));
    if (!(ok & bit)) return false;
    if (free_ & bit) return true;
    const float q = ((float)((use_u & bit) ? u : v) / (float)0x01000000) * half_quad;
    const float at = (neg & bit) ? pos - q : pos + q;
    return (p - at) * sn < 0.f;
  }
};

struct LightSample {
  bool vis;
  f3 l_pos, l_nor, Le;
  float G;
  bool g_set;
};

// sample_lights: chooses a point on `l` as seen from the shading point, its
// pdf update, and (when `visibility`) asks the visibility provider `vp` about
// the shadow ray; `slot` names the call site so that a later pass can find
// the answer (see VisCapture / VisRead).
template <class VP>
__device__ LightSample sample_lights(const FrameView &F, f3 P, f3 n, uint32_t hit_inst, uint32_t hit_prim, Light l,
                                     float &pdf, uint32_t &seed, bool calc_pdf, bool visibility, uint32_t pixel,
                                     VP &vp, uint32_t slot) {
  LightSample s;
  s.g_set = false;
  s.G = 0.f;
  s.l_pos = mk3(0.f);
  s.l_nor = mk3(0.f);
  if (l.inst == hit_inst && l.prim == hit_prim) { s.vis = false; s.Le = mk3(0.f); return s; }
  bool vis = true, check_instance = false;
  float distance = -1.0f;
  f3 l_wi = mk3(0.f), l_pos = mk3(0.f), l_nor = mk3(0.f);
  if (l.type == CT_LIGHT_CUBE) {
    const float half_extent = l.size * 0.5f;
    const f2 quad = f2{l.size, l.size};
    uint32_t i = 0;
    const f3 c = l.position - P;
    const bool fast = is_unit_axis(n) && fabsf(c.x) + fabsf(c.y) + fabsf(c.z) < INFINITY;
    // A try succeeds only for a point in front of the shading point's plane
    // (dot(P - l_pos, n) < 0).  When the whole cube lies behind that plane,
    // by a margin far above the rounding of l_pos, all 11 tries fail and the
    // first 10 only advance the RNG (3 draws each: a face, two quad
    // coordinates): jump over their 30 draws and run the last try, which
    // leaves l_pos, l_nor and the seed exactly as the full loop does.
    {
      const float reach = dot(c, n) + half_extent * (fabsf(n.x) + fabsf(n.y) + fabsf(n.z));
      const float scale = fmaxf(fmaxf(fmaxf(fabsf(P.x), fabsf(P.y)), fmaxf(fabsf(P.z), fabsf(l.position.x))),
                                fmaxf(fmaxf(fabsf(l.position.y), fabsf(l.position.z)), l.size));
      if (reach < -1e-5f * scale) {
        seed = lcg_jump<30>(seed);
        i = 10;
      }
    }
    if (fast) {
      const CubeTries tries(P, n, l);
      uint32_t before;  // the stream before the deciding try, drawn again in full
      do {
        before = seed;
        vis = tries(seed);
      } while (!vis && i++ < 10);
      l_nor = random_cube_normal(before);
      l_pos = l.position + l_nor * half_extent;
      l_pos = random_quad(l_nor, l_pos, quad * 0.5f, before);
    } else {
      do {
        vis = true;
        l_nor = random_cube_normal(seed);
        l_pos = l.position + l_nor * half_extent;
        l_pos = random_quad(l_nor, l_pos, quad * 0.5f, seed);
        l_wi = normalize(P - l_pos);
        vis = vis && (dot(l_wi, l_nor) > 0.0f);
        vis = vis && (dot(l_wi, n) < 0.0f);
      } while (!vis && i++ < 10);
    }
    if (fast) l_wi = normalize(P - l_pos);
    l_pos = offset_twice(l_pos, l_nor);
    distance = length(P - l_pos);
    if (calc_pdf) {
      float area = quad.x * quad.y * 6.0f;
      pdf = pdf / area;
    }
    check_instance = true;
    s.G = geom_fact_sa(P, l_pos, l_nor);
    s.g_set = true;
  } else if (l.type == CT_LIGHT_POINT) {
    l_pos = l.position;
    l_nor = normalize(P - l_pos);
    distance = length(P - l_pos);
    l_wi = l_nor;
    s.G = geom_fact_sa(P, l_pos, l_nor);
    s.g_set = true;
  } else if (l.type == CT_LIGHT_ENV_MAP) {
    f3 u = random_unit_vector(seed, pixel);
    f3 l_dir = dot(u, n) > 0.0f ? u : -u;
    l_pos = P + (l_dir * 1e9f);
    l_nor = normalize(P - l_pos);
    distance = length(P - l_pos);
    l_wi = l_nor;
    l.emissive = l.emissive * sky_color(F.time, F.is_afternoon, l_dir);
    if (calc_pdf) pdf = pdf / 0.079577471545947667884441881686255f;
    s.G = 1.0f;
    s.g_set = true;
  }
  f3 l_v = -l_wi;
  if (visibility && vis) vis = vis && vp(P, l_v, distance, l.inst, l.prim, check_instance, slot);
  s.vis = vis;
  s.l_pos = l_pos;
  s.l_nor = l_nor;
  s.Le = vis ? l.emissive : mk3(0.f);
  return s;
}

// calculate_sampled_light (light.glsl:401-435).  `scatter_dir` is the
// HIT_INFO_INPUT.scatter_dir the shader updates in place; `G` stays 0 when the
// sampler returns before computing it (the shader leaves it unset).
template <class VP>
__device__ f3 calculate_sampled_light(const FrameView &F, f3 ray_dir, f3 P, f3 n, uint32_t hit_inst, uint32_t hit_prim,
                                      const Material &mat, const Light &light, float pdf, float &pdf_out, float &G,
                                      uint32_t &seed, bool calc_pdf, bool use_pdf, bool use_visibility,
                                      f3 &scatter_dir, uint32_t pixel, VP &vp, uint32_t slot) {
  f3 surface_normal = normalize_n(n);
  f3 wo = -normalize(ray_dir);
  pdf_out = pdf;
  G = 0.f;
  f3 result = mk3(0.f);
  if (all_le_zero(light.emissive)) return result;
  LightSample s = sample_lights(F, P, n, hit_inst, hit_prim, light, pdf_out, seed, calc_pdf, use_visibility, pixel, vp,
                                slot);
  if (s.g_set) G = s.G;
  if (s.vis) {
    f3 wi = normalize(s.l_pos - P);
    f3 brdf = evaluate_material(mat, surface_normal, wo, wi);
    scatter_dir = wi;
    if (use_pdf) result = brdf * s.Le * G / pdf_out;
    else result = brdf * s.Le * G;
  }
  return result;
}

// ---------------------------------------------------------------------------
// reservoirs (reservoir.glsl:17-126)
struct Reservoir {
  uint32_t Y, l_type, seed;
  float W_y, W_sum, M;
  f3 F;
};
__device__ __forceinline__ Reservoir reservoir_empty() {
  Reservoir r;
  r.W_y = 0.f; r.seed = 0; r.W_sum = 0.f; r.M = 0.f; r.Y = 0xFFFFFFFFu; r.l_type = CT_LIGHT_NONE; r.F = mk3(0.f);
  return r;
}
__device__ __forceinline__ Reservoir load_reservoir(const ct_reservoir *b, uint32_t i) {
  const ct_reservoir &s = b[i];
  Reservoir r;
  r.Y = s.Y; r.l_type = s.l_type; r.seed = s.seed; r.W_y = s.W_y; r.W_sum = s.W_sum; r.M = s.M; r.F = ld3(s.F);
  return r;
}
__device__ __forceinline__ void store_reservoir(ct_reservoir *b, uint32_t i, const Reservoir &r) {
  ct_reservoir &s = b[i];
  s.Y = r.Y; s.l_type = r.l_type; s.seed = r.seed; s.W_y = r.W_y; s.W_sum = r.W_sum; s.M = r.M; st3(s.F, r.F);
}
__device__ __forceinline__ bool update_reservoir(Reservoir &r, uint32_t X, uint32_t l_type, uint32_t random_seed, f3 Fv,
                                                 float w, float c, uint32_t &seed) {
  if (w < 0.0f || isnan(w) || isinf(w)) return false;
  r.M += c;
  r.W_sum += w;
  if (rnd(seed) < (w / r.W_sum)) {
    r.Y = X; r.l_type = l_type; r.seed = random_seed; r.F = Fv;
    return true;
  }
  return false;
}
__device__ __forceinline__ bool reservoir_valid(const Reservoir &r) {
  return r.M > 0.0f && r.Y != 0xFFFFFFFFu && r.l_type != CT_LIGHT_NONE;
}

// shading point of a DI info record, as every pass reconstructs it
struct Shade {
  f3 P;          // compute_ray_origin(position, normal) applied twice
  f3 n;
  float distance;
  uint32_t inst, prim, mat_index;
};

// reservoir_get_radiance (reservoir.glsl:98-112): re-evaluates the reservoir's
// sample, replaying its stored light seed, with a shadow ray.
template <class VP>
__device__ f3 reservoir_get_radiance(const FrameView &F, const Reservoir &r, f3 ray_dir, const Shade &s,
                                     const Material &mat, uint32_t pixel, VP &vp, uint32_t slot) {
  if (!reservoir_valid(r)) return mk3(0.f);
  Light light = light_get_by_type(F, r.l_type, r.Y);
  uint32_t seed = r.seed;
  float pdf_out, G;
  f3 scatter = mk3(0.f);
  return calculate_sampled_light(F, ray_dir, s.P, s.n, s.inst, s.prim, mat, light, 1.0f, pdf_out, G, seed, false,
                                 false, true, scatter, pixel, vp, slot);
}

// ---------------------------------------------------------------------------
// Visibility providers.  The shading passes run twice over a pixel: the
// generating pass records every shadow ray the shader would trace (VisCapture,
// into a compacted queue traced by k_trace_shadow), the resolving pass
// replays the same deterministic light samples and reads the answers back
// (VisRead).  A call site traces at most one ray and owns one fixed slot.
#define CT_VIS_SLOTS 16u  // per pixel: 2 per spatial neighbour; stage 0 uses 0..2

struct RayQueue {
  float4 *a;        // origin.xyz, distance
  float4 *b;        // direction.xyz, result slot (bits)
  uint2 *c;         // target (instance | check flag << 31, primitive)
  uint32_t *count;
  uint32_t capacity;
};

struct VisNever {  // for samplers called with visibility off
  __device__ bool operator()(f3, f3, float, uint32_t, uint32_t, bool, uint32_t) { return true; }
};

// Exclusive prefix of `n` over the block plus one atomicAdd on `counter`;
// returns this thread's first position.  Blocks are whole warps.
__device__ __forceinline__ uint32_t block_reserve(uint32_t n, uint32_t *counter) {
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t block_base;
  const uint32_t tid = threadIdx.y * blockDim.x + threadIdx.x;
  const uint32_t lane = tid & 31u, wid = tid >> 5;
  const uint32_t nwarps = (blockDim.x * blockDim.y + 31u) >> 5;
  uint32_t incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= (uint32_t)o) incl += v;
  }
  if (lane == 31u) warp_sum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    uint32_t w = lane < nwarps ? warp_sum[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, wi, o);
      if (lane >= (uint32_t)o) wi += v;
    }
    if (lane < nwarps) warp_sum[lane] = wi - w;
    if (lane == nwarps - 1u) block_base = wi ? atomicAdd(counter, wi) : 0u;
  }
  __syncthreads();
  return block_base + warp_sum[wid] + incl - n;
}

struct VisRead {
  const uint8_t *vis;
  uint32_t base;
  __device__ bool operator()(f3, f3, float, uint32_t, uint32_t, bool, uint32_t slot) { return vis[base + slot] != 0; }
};

__device__ __forceinline__ Shade shade_from_di(const ct_di_info &d) {
  Shade s;
  f3 pos = ld3(d.position);
  s.n = ld3(d.normal);
  s.P = offset_twice(pos, s.n);
  s.distance = d.distance;
  s.inst = d.instance_hit.instance_id;
  s.prim = d.instance_hit.primitive_id;
  s.mat_index = d.mat_index;
  return s;
}

#define CT_HLF_MAX 6.5504e+4f
#define CT_HLF_MIN 1.175494351e-38f

// The dielectric scatter callable's first step (rcall_scatter.glsl:20-30): a
// normal that faces along the ray is turned and the point pushed through the
// face.  The callable works on the caller's hit record (sample_material,
// light.glsl:231-260, takes it inout).
__device__ __forceinline__ bool dielectric_face(f3 &hit, f3 &nrm, f3 ray_dir) {
  if (!(dot(ray_dir, nrm) > 0.0f)) return false;
  nrm = -nrm;
  hit = hit - nrm * CT_HLF_MIN * 2.0f;
  return true;
}

// The shading point the rest of the first pass sees after RIS.  The BRDF
// candidates (restir_resampling.glsl:193-230) hand the pass's hit record to
// sample_material, so on a dielectric hit from behind its face the record
// leaves RIS turned: the RIS visibility pass and TEMPORAL_REUSE that follow
// in the same invocation (rgen.glsl:255-262) work on the turned record, while
// the DI record and everything after the first pass keep the hit as found.
// Only the first candidate can turn it (the turned normal faces the ray).
__device__ __forceinline__ void turn_after_ris(const FrameView &F, Shade &S, f3 ray_dir) {
  if (!(F.is_active & CT_RIS_BRDF_BIT) || F.light_config.brdf_count == 0u) return;
  if ((F.materials[S.mat_index].type & 0xFFu) != 2u) return;
  dielectric_face(S.P, S.n, ray_dir);
}

// ct_nrc.cu -- the neural radiance cache's fully fused MLP on the fifth-
// generation tensor cores (ct_nrc_encode / ct_nrc_infer /
// ct_nrc_infer_encoded, include/ct.h).  No counterpart in the reference,
// whose path tracer has no cache.
//
// Network: 256 inputs (the encoding below, zero padded) -> 5 hidden layers
// of 64 with ReLU -> 16 outputs, of which the first three are RGB radiance.
// Weights are bf16, row-major (output, input); products accumulate in fp32
// in tensor memory; each hidden activation is rounded to bf16 before the
// next layer reads it.
//
// One CTA of 512 threads per SM: four warpgroups, each walking its own tiles
// of 128 queries with two 16 KB buffers, 128 tensor-memory columns and two
// mbarriers of its own.  The weights (66 KB) are shared; with the buffers the
// CTA holds 194 KB.  Per tile:
//  * every thread encodes its query (row = thread), K-major in
//    128-byte-swizzled atoms of 8 rows x 64 bf16, one block of 64 of the 256
//    inputs at a time in one buffer, while the MMAs of the previous tile's
//    layers run on the other;
//  * one thread of the warpgroup issues tcgen05.mma (M 128, N 64, K 16 per
//    instruction, bf16 inputs, fp32 accumulator) and commits to the buffer's
//    mbarrier;
//  * every warp reads its 32 TMEM lanes (tcgen05.ld 32x32b), rounds to bf16,
//    applies ReLU and writes the next layer's input;
//  * the last layer (N 16) writes RGB to global memory.
// What bounds it is instruction issue: the encoding's 48 sincospi and 128
// exponentials and the epilogues are some 3500 instructions per query against
// 68 kFLOP of MMAs, at 4 warps per scheduler (issue 62% active): 2.07 M queries
// take 359 us (3060 and 333 us with the bins below 2^-126 flushed to 0, which
// the weights can bring to the output).  Whole 64 KB tiles let only two
// warpgroups in (issue 44%, 573 us).  With flushed bins, encoding a tile before
// its layers instead of during the previous tile's took 353 us against 341, one
// barrier for a layer and a block 357 us.
// Warpgroups synchronise on their own named barriers.  Operands are staged
// with ordinary 16-byte shared stores (no TMA).  Every wait is bounded
// (about one second); a warpgroup that gives up latches an error in the
// library's NRC status word and stops; the CTA frees its tensor memory and
// returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>
#include "ct.h"
#include "ct_profile.cuh"

namespace ct_nrc {

constexpr int kTile = 128;
constexpr int kIn = CT_NRC_INPUT_DIMS;     // 256
constexpr int kWidth = CT_NRC_WIDTH;       // 64
constexpr int kOut = CT_NRC_OUTPUT_DIMS;   // 16
constexpr int kHidden = CT_NRC_HIDDEN_LAYERS;  // 5
constexpr int kGroups = 4;                    // warpgroups per CTA, one tile each
constexpr int kThreads = kTile * kGroups;     // 512
constexpr int kTmemCols = 128 * kGroups;      // two tiles' 64 accumulator columns per warpgroup
constexpr int kBlockK = 64;                   // inputs per buffer
static_assert(kIn == 4 * kBlockK, "blocks of the first layer");

// shared memory regions, each 1024-byte aligned (128-byte swizzle atoms)
constexpr uint32_t kBufBytes = kTile * kBlockK * 2;         // 16 KB
constexpr uint32_t kSmemA = 0;                              // two buffers per warpgroup
constexpr uint32_t kSmemW0 = kSmemA + kGroups * 2 * kBufBytes;  // 4 K-blocks of [64 x 64] = 32 KB
constexpr uint32_t kSmemWh = kSmemW0 + 4 * 8192;            // 4 hidden layers of [64 x 64] = 32 KB
constexpr uint32_t kSmemW5 = kSmemWh + 4 * 8192;            // [16 x 64] = 2 KB
constexpr uint32_t kSmemBar = kSmemW5 + 2048;               // two mbarriers (8 B) per warpgroup
constexpr uint32_t kSmemFail = kSmemBar + 16 * kGroups;     // a word per warpgroup: a wait ran out
constexpr uint32_t kSmemTmem = kSmemFail + 4 * kGroups;     // TMEM address
constexpr uint32_t kSmemBytes = kSmemTmem + 16 + 1024;      // + slack to align the base to 1024
static_assert(kSmemBytes <= 227 * 1024, "shared memory per CTA");

// weight offsets in the packed bf16 buffer (elements)
constexpr uint32_t kW0 = 0;
constexpr uint32_t kWh = kW0 + kWidth * kIn;
constexpr uint32_t kW5 = kWh + 4 * kWidth * kWidth;
static_assert(kW5 + kOut * kWidth == CT_NRC_WEIGHT_COUNT, "weight packing");

__device__ uint32_t g_nrc_status;  // 0: ok; else the first failure (detail code)

// byte offset of 16-byte chunk `chunk` (8 bf16) of row `row` in a K-major
// region of 64-element rows, 128-byte swizzled: 8-row atoms of 1024 B, the
// chunk index XORed with the row within the atom
__device__ __forceinline__ uint32_t sw128(uint32_t row, uint32_t chunk) {
  return (row >> 3) * 1024u + (row & 7u) * 128u + (((chunk ^ (row & 7u)) & 7u) << 4);
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 B apart (stride byte offset), version 1 (sm_100)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;            // leading byte offset: unused with a 128-byte swizzle (16 B)
  d |= (uint64_t)(1024u >> 4) << 32;  // stride byte offset
  d |= (uint64_t)1u << 46;            // descriptor version
  d |= (uint64_t)2u << 61;            // 128-byte swizzle
  return d;
}

// instruction descriptor, kind::f16: bf16 A and B (K-major), fp32 D, M x N
__host__ __device__ constexpr uint32_t instr_desc(uint32_t m, uint32_t n) {
  return (1u << 4)            // D format: f32
         | (1u << 7)          // A format: bf16
         | (1u << 10)         // B format: bf16
         | ((n >> 3) << 17)   // N / 8
         | ((m >> 4) << 24);  // M / 16
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool try_bar(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// waits for the mbarrier phase `parity`, for at most about one second; the
// clock is read only by waits that the first try does not end
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity) {
  if (try_bar(bar, parity)) return true;
  const uint64_t t0 = now_ns();
  while (now_ns() - t0 <= 1000000000ull)
    if (try_bar(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 fp32 columns of this thread's TMEM lane; tmem_wait before they are read
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// the loaded registers pass through the wait, so that no use moves before it
__device__ __forceinline__ void tmem_wait16(uint32_t *r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// ---------------------------------------------------------------------------
// The input encoding, 256 values per query:
//   [0, 96)    position q = clamp((p - bbox_min) / bbox_extent, 0, 1): for
//              axis c and band k < 16, t = (q_c * 2^k) mod 2,
//              sin(pi t) at 32c + 2k and cos(pi t) at 32c + 2k + 1;
//   [96, 160)  direction: one-blob of u0 = atan2(w.z, w.x) / 2pi + 1/2 and
//              u1 = w.y / 2 + 1/2, 32 bins each, bin i = exp(-((u - (i +
//              1/2) / 32) * 32)^2 / 2);
//   [160, 224) the normal, the same way;
//   [224, 227) albedo; [227, 256) zero.
// Bin i of a one-blob with u32 = 32 u: exp(-d^2 / 2), d = u32 - (i + 1/2), as
// 2^(d^2 * (-log2(e) / 2)), subnormal results kept.
__device__ __forceinline__ float blob_bin(float u32, int i) {
  const float d = u32 - ((float)i + 0.5f), x = (d * d) * -0.72134752044448170368f;
  float r;
  asm("ex2.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ uint4 pack8(const float *v) {
  return make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
}

// The encoding in 16-byte chunks of 8 values: chunk 4c + j holds bands 4j ..
// 4j + 3 of axis c, chunks 12 + 8v + j (j < 4) the first angle's bins 8j .. 8j
// + 7 of vector v, chunks 12 + 8v + 4 + j the second angle's, chunk 28 the
// albedo and chunks 29-31 zeros.  sincospi reduces its argument itself, so a
// band's phase is q_c 2^k, an exact product, as it stands.
//
// encode_block<KB> emits (emit(chunk, v)) the 8 chunks of block KB.
template <class Emit>
__device__ __forceinline__ void encode_axis(float p, float bmin, float bext, int chunk, Emit &&emit) {
  const float x = fminf(fmaxf((p - bmin) / bext, 0.0f), 1.0f);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    float v[8];
#pragma unroll
    for (int b = 0; b < 4; b++) sincospif(x * (float)(1u << (4 * j + b)), &v[2 * b], &v[2 * b + 1]);
    emit(chunk + j, pack8(v));
  }
}
template <class Emit>
__device__ __forceinline__ void encode_blob(float u, int chunk, Emit &&emit) {
  const float u32 = u * 32.0f;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = blob_bin(u32, 8 * j + i);
    emit(chunk + j, pack8(v));
  }
}
__device__ __forceinline__ float azimuth(const float *w) {
  return atan2f(w[2], w[0]) * (0.5f / 3.14159265358979323846f) + 0.5f;
}
__device__ __forceinline__ float elevation(const float *w) { return w[1] * 0.5f + 0.5f; }
template <int KB, class Emit>
__device__ __forceinline__ void encode_block(const ct_nrc_query &q, const float *bmin, const float *bext, Emit &&emit) {
  if (KB == 0) {
    encode_axis(q.position[0], bmin[0], bext[0], 0, emit);
    encode_axis(q.position[1], bmin[1], bext[1], 4, emit);
  } else if (KB == 1) {
    encode_axis(q.position[2], bmin[2], bext[2], 8, emit);
    encode_blob(azimuth(q.direction), 12, emit);
  } else if (KB == 2) {
    encode_blob(elevation(q.direction), 16, emit);
    encode_blob(azimuth(q.normal), 20, emit);
  } else {
    encode_blob(elevation(q.normal), 24, emit);
    const float v[8] = {q.albedo[0], q.albedo[1], q.albedo[2], 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    emit(28, pack8(v));
#pragma unroll
    for (int ch = 29; ch < 32; ch++) emit(ch, make_uint4(0u, 0u, 0u, 0u));
  }
}

// A warp encodes 32 queries, block by block through its own shared memory, so
// that the rows (512 B each) leave in whole 128-byte lines: a thread storing
// its own row sends each 16-byte chunk to a sector of its own.
constexpr int kEncodeThreads = 128;
__global__ void __launch_bounds__(kEncodeThreads) k_nrc_encode(const ct_nrc_query *q, uint32_t n, float3 bmin,
                                                               float3 bext, __nv_bfloat16 *out) {
  __shared__ uint4 s_rows[kEncodeThreads / 32][32][9];  // 8 chunks a row, padded against bank conflicts
  const uint32_t lane = threadIdx.x & 31u, first = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u;
  uint4(*rows)[9] = s_rows[threadIdx.x >> 5];
  if (first >= n) return;  // whole warps
  const float mn[3] = {bmin.x, bmin.y, bmin.z}, ex[3] = {bext.x, bext.y, bext.z};
  const ct_nrc_query qq = q[min(first + lane, n - 1u)];
  const auto store = [&](int kb) {
    __syncwarp();
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) {
      const uint32_t r = i * 4u + (lane >> 3), ch = lane & 7u;
      if (first + r < n) reinterpret_cast<uint4 *>(out + (uint64_t)(first + r) * kIn)[kb * 8 + ch] = rows[r][ch];
    }
    __syncwarp();
  };
  const auto put = [&](int ch, uint4 v) { rows[lane][ch & 7] = v; };
  encode_block<0>(qq, mn, ex, put);
  store(0);
  encode_block<1>(qq, mn, ex, put);
  store(1);
  encode_block<2>(qq, mn, ex, put);
  store(2);
  encode_block<3>(qq, mn, ex, put);
  store(3);
}

// The encoding in single precision, for the training of the fp32 network
// (float[n][256]): the values, and bit for bit the roundings, of the torch
// expressions in cube_tracing/nrc.py (encode), which took some 45 launches.
// One thread per 4 consecutive values, so that a warp stores 512 contiguous
// bytes of a row; the warps of a row's two halves take one kind of value each.
__device__ __forceinline__ float4 encode_f32_freq(float p, float bmin, float bext, int band) {
  float x = (p - bmin) / bext;
  if (!isnan(x)) x = fminf(fmaxf(x, 0.0f), 1.0f);  // torch's clamp keeps a NaN
  float v[4];
#pragma unroll
  for (int b = 0; b < 2; b++) {
    const float t = fmodf(x * (float)(1u << (band + b)), 2.0f);
    const float a = 3.14159265358979323846f * t;
    v[2 * b] = sinf(a);
    v[2 * b + 1] = cosf(a);
  }
  return make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ float4 encode_f32_blob(float u, int bin) {
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float d = (u - ((float)(bin + i) + 0.5f) / 32.0f) * 32.0f;
    v[i] = expf(-0.5f * d * d);
  }
  return make_float4(v[0], v[1], v[2], v[3]);
}
__global__ void __launch_bounds__(256) k_nrc_encode_f32(const ct_nrc_query *q, uint32_t n, float3 bmin, float3 bext,
                                                        float4 *out) {
  const uint64_t at = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t i = (uint32_t)(at >> 6), c = (uint32_t)(at & 63u);  // row, group of 4 values
  if (i >= n) return;
  const ct_nrc_query &r = q[i];
  float4 v;
  if (c < 24u) {
    const uint32_t a = c >> 3;  // axis: 8 groups of 2 bands
    const float mn = a == 0 ? bmin.x : (a == 1 ? bmin.y : bmin.z), ex = a == 0 ? bext.x : (a == 1 ? bext.y : bext.z);
    v = encode_f32_freq(r.position[a], mn, ex, 2 * (int)(c & 7u));
  } else if (c < 56u) {
    const uint32_t k = (c - 24u) >> 3;  // direction's two angles, then the normal's: 8 groups of 4 bins
    const float *w = k < 2u ? r.direction : r.normal;
    const float u = (k & 1u) ? w[1] * 0.5f + 0.5f : atan2f(w[2], w[0]) * (0.5f / 3.14159265358979323846f) + 0.5f;
    v = encode_f32_blob(u, 4 * (int)((c - 24u) & 7u));
  } else {
    v = c == 56u ? make_float4(r.albedo[0], r.albedo[1], r.albedo[2], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  out[at] = v;
}

// The training loss's elementwise part and its gradient: per row and channel
//   rel = (pred - target)^2 / (pred^2 + 0.01),   terms = rel w,
//   grad = (((1 / total) w) / (pred^2 + 0.01)) (2 (pred - target))
// in the operation order of the torch expressions and their autograd (15
// launches): the caller sums `terms` and divides by `total`.  pred and grad
// are rows of 16 (the network's outputs; channels 3 to 15 have no gradient).
__global__ void __launch_bounds__(256) k_nrc_loss(const float *pred, const float *target, const float *weight,
                                                  const float *total, uint32_t n, float *terms, float4 *grad) {
  const uint64_t at = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t i = (uint32_t)(at >> 2);  // a row's four groups of 4 outputs
  if (i >= n) return;
  float g[4] = {0.f, 0.f, 0.f, 0.f};
  if ((at & 3u) == 0u) {
    const float w = weight[i], s = (1.0f / *total) * w;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float p = pred[16ull * i + c], d = p - target[3ull * i + c], den = p * p + 0.01f;
      terms[3ull * i + c] = (d * d) / den * w;
      g[c] = s / den * (2.0f * d);
    }
  }
  grad[at] = make_float4(g[0], g[1], g[2], g[3]);
}

// warpgroup g's named barrier (ids 1 to kGroups; 0 is __syncthreads)
__device__ __forceinline__ void group_sync(uint32_t g) { asm volatile("bar.sync %0, 128;" ::"r"(g + 1u) : "memory"); }

// a block of an MLP layer: D[128 x N] (+)= A[128 x 64] * W[N x 64]^T
__device__ __forceinline__ void block_mma(uint32_t tmem, uint32_t a_base, uint32_t w_base, uint32_t idesc,
                                          bool accumulate, uint32_t bar) {
  fence_after();
  for (int j = 0; j < 4; j++)
    mma(tmem, smem_desc(a_base + j * 32), smem_desc(w_base + j * 32), idesc, (accumulate || j != 0) ? 1u : 0u);
  commit(bar);
}

template <bool ENCODE>
__global__ void __launch_bounds__(kThreads, 1) k_nrc_mlp(const ct_nrc_query *q, const __nv_bfloat16 *encoded,
                                                         uint32_t n, float3 bmin, float3 bext,
                                                         const __nv_bfloat16 *weights, float *rgb) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t base = smem_u32(smem);
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t g = tid >> 7, row = tid & (kTile - 1);  // warpgroup, and this thread's row of its tile
  uint32_t *tmem_slot = (uint32_t *)(smem + kSmemTmem);
  volatile uint32_t *fail = (volatile uint32_t *)(smem + kSmemFail) + g;

  // weights into their swizzled regions (16-byte chunks)
  for (uint32_t i = tid; i < (uint32_t)(kWidth * (kIn / 8)); i += kThreads) {  // W0: 64 rows x 32 chunks
    const uint32_t r = i / 32u, ch = i % 32u;
    const uint4 v = *reinterpret_cast<const uint4 *>(weights + kW0 + r * kIn + ch * 8u);
    *reinterpret_cast<uint4 *>(smem + kSmemW0 + (ch >> 3) * 8192u + sw128(r, ch & 7u)) = v;
  }
  for (uint32_t i = tid; i < 4u * kWidth * 8u; i += kThreads) {  // W1..W4: 4 x 64 rows x 8 chunks
    const uint32_t l = i / 512u, r = (i / 8u) % 64u, ch = i % 8u;
    const uint4 v = *reinterpret_cast<const uint4 *>(weights + kWh + l * 4096u + r * 64u + ch * 8u);
    *reinterpret_cast<uint4 *>(smem + kSmemWh + l * 8192u + sw128(r, ch)) = v;
  }
  for (uint32_t i = tid; i < (uint32_t)kOut * 8u; i += kThreads) {  // W5: 16 rows x 8 chunks
    const uint32_t r = i / 8u, ch = i % 8u;
    const uint4 v = *reinterpret_cast<const uint4 *>(weights + kW5 + r * 64u + ch * 8u);
    *reinterpret_cast<uint4 *>(smem + kSmemW5 + sw128(r, ch)) = v;
  }
  if (tid == 0) {
    for (uint32_t k = 0; k < 2u * kGroups; k++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(base + kSmemBar + 8u * k) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (row == 0) *fail = 0u;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_async_smem();
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem = tmem_base + 128u * g;              // this warpgroup's accumulator columns, two tiles'
  const uint32_t lane_bits = ((warp & 3u) * 32u) << 16;    // a warp reads TMEM lanes 32 (warp % 4) + 0..31
  const uint32_t bar0 = base + kSmemBar + 16u * g, bar1 = bar0 + 8u;
  const uint32_t buf0 = kSmemA + g * 2u * kBufBytes, buf1 = buf0 + kBufBytes;
  const float mn[3] = {bmin.x, bmin.y, bmin.z}, ex[3] = {bext.x, bext.y, bext.z};
  uint32_t par0 = 0, par1 = 0;  // phase each mbarrier is in
  // a wait that ran out shows at the warpgroup's next barrier
  const auto wait0 = [&]() {
    if (!wait_bar(bar0, par0)) *fail = 1u;
    par0 ^= 1u;
    __syncwarp();  // tcgen05.ld is a warp's
  };
  const auto wait1 = [&]() {
    if (!wait_bar(bar1, par1)) *fail = 1u;
    par1 ^= 1u;
    __syncwarp();
  };
  // the warpgroup's writes to its buffers are complete and visible to the
  // MMAs; false when it has given up
  const auto ready = [&]() {
    fence_async_smem();
    fence_before();
    group_sync(g);
    return *fail == 0u;
  };
  const uint32_t tiles = (n + kTile - 1) / kTile;
  // tiles in turn over the CTAs' first warpgroups, then their second ones, ...:
  // a few tiles spread over the SMs.  A warpgroup runs the hidden layers of
  // tile `cur` (activations in buffer 0) and the first layer of tile `next`
  // (a block of inputs at a time in buffer 1) in turn, so that it encodes while
  // a layer's MMAs run.  The two tiles' accumulators alternate.
  const uint32_t stride = gridDim.x * kGroups;
  uint32_t cur = 0, next = g * gridDim.x + blockIdx.x;
  uint32_t acc = 0;  // columns of tile `cur`: 64 acc
  bool have = false, ok = true;
  ct_nrc_query qq;
  while (ok && (have || next < tiles)) {
    const bool feed = next < tiles;
    const uint32_t t_cur = tmem + 64u * acc, t_next = tmem + 64u * (acc ^ 1u);
    // rows past the end repeat the last query; their results are not stored
    if (ENCODE && feed) qq = q[min(next * kTile + row, n - 1u)];
    const auto fill = [&](auto kb_c) {
      constexpr int kb = decltype(kb_c)::value;
      if (ENCODE) {
        encode_block<kb>(qq, mn, ex, [&](int ch, uint4 v) {
          *reinterpret_cast<uint4 *>(smem + buf1 + sw128(row, (uint32_t)ch & 7u)) = v;
        });
      } else {
        // 8 threads per row: whole 128-byte lines of the encoded rows
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) {
          const uint32_t r = i * 16u + (row >> 3), ch = row & 7u, at = next * kTile + r;
          uint4 v = make_uint4(0, 0, 0, 0);
          if (at < n) v = *reinterpret_cast<const uint4 *>(encoded + (uint64_t)at * kIn + kb * kBlockK + ch * 8u);
          *reinterpret_cast<uint4 *>(smem + buf1 + sw128(r, ch)) = v;
        }
      }
    };
    // hidden layer (or output) `layer` of cur: the accumulator, rounded to
    // bf16, then ReLU (which commutes), into buffer 0, and the layer's MMAs
    const auto layer_begin = [&](int layer) {
      fence_after();
#pragma unroll
      for (uint32_t c0 = 0; c0 < (uint32_t)kWidth; c0 += 32) {
        uint32_t r[32];
        tmem_ld16(t_cur + lane_bits + c0, r);
        tmem_ld16(t_cur + lane_bits + c0 + 16, r + 16);
        tmem_wait16(r);
        tmem_wait16(r + 16);
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
          uint32_t h[4];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(r[k + 2 * j]), __uint_as_float(r[k + 2 * j + 1]));
            const __nv_bfloat162 m = __hmax2(v, __nv_bfloat162(__ushort_as_bfloat16(0), __ushort_as_bfloat16(0)));
            h[j] = *reinterpret_cast<const uint32_t *>(&m);
          }
          *reinterpret_cast<uint4 *>(smem + buf0 + sw128(row, (c0 + k) >> 3)) = make_uint4(h[0], h[1], h[2], h[3]);
        }
      }
      if (!ready()) return false;
      if (row == 0) {
        const bool last = layer == kHidden;
        block_mma(t_cur, base + buf0, base + (last ? kSmemW5 : kSmemWh + (layer - 1) * 8192u),
                  last ? instr_desc(128, kOut) : instr_desc(128, kWidth), false, bar0);
      }
      return true;
    };
    // block kb of next's inputs and its MMAs
    const auto feed_block = [&](auto kb_c) {
      constexpr int kb = decltype(kb_c)::value;
      if (kb > 0) wait1();
      fill(kb_c);
      if (!ready()) return false;
      if (row == 0)
        block_mma(t_next, base + buf1, base + kSmemW0 + kb * 8192u, instr_desc(128, kWidth), kb != 0, bar1);
      return true;
    };
    const auto step = [&](int layer, auto kb_c) {
      if (ok && have) ok = layer_begin(layer);
      if (ok && feed) ok = feed_block(kb_c);
      if (ok && have) wait0();
    };
    step(1, std::integral_constant<int, 0>{});
    step(2, std::integral_constant<int, 1>{});
    step(3, std::integral_constant<int, 2>{});
    step(4, std::integral_constant<int, 3>{});
    if (ok && have) {
      ok = layer_begin(kHidden);
      if (ok) wait0();
    }
    if (ok && have) {
      fence_after();
      uint32_t r[16];
      tmem_ld16(t_cur + lane_bits, r);
      tmem_wait16(r);
      const uint32_t qi = cur * kTile + row;
      if (qi < n) {
        rgb[3ull * qi] = __uint_as_float(r[0]);
        rgb[3ull * qi + 1] = __uint_as_float(r[1]);
        rgb[3ull * qi + 2] = __uint_as_float(r[2]);
      }
      // the next barrier orders these tensor-memory reads before the MMAs that
      // overwrite the columns
    }
    if (ok && feed) wait1();
    have = feed;
    cur = next;
    next += stride;
    acc ^= 1u;
  }
  // every tensor-memory read of this CTA is complete (tcgen05.wait::ld), and
  // every thread's word about its last wait is written
  fence_before();
  __syncthreads();
  if (row == 0 && *fail != 0u) atomicCAS(&g_nrc_status, 0u, 1u);
  if (warp == 0) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

}  // namespace ct_nrc

static ct_status nrc_status(cudaError_t e) {
  if (e == cudaSuccess) return CT_OK;
  return CT_ERR_CUDA;
}

static ct_status check_net(const ct_nrc_net *net) {
  if (!net || !net->weights_address || (net->weights_address & 15u)) return CT_ERR_INVALID_ARG;
  for (int c = 0; c < 3; c++)
    if (!(net->bbox_extent[c] > 0.0f) || !isfinite(net->bbox_min[c]) || !isfinite(net->bbox_extent[c]))
      return CT_ERR_INVALID_ARG;
  return CT_OK;
}

static int nrc_grid(uint32_t n) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    sms = v > 0 ? v : 148;
  }
  const uint32_t tiles = (uint32_t)(((uint64_t)n + ct_nrc::kTile - 1) / ct_nrc::kTile);
  return (int)(tiles < (uint32_t)sms ? tiles : (uint32_t)sms);
}

static cudaError_t launch_mlp(bool encode, const ct_nrc_net *net, const ct_nrc_query *q, const void *encoded,
                              uint32_t n, float *rgb, cudaStream_t s) {
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(ct_nrc::k_nrc_mlp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)ct_nrc::kSmemBytes);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ct_nrc::k_nrc_mlp<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)ct_nrc::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const float3 bmin = make_float3(net->bbox_min[0], net->bbox_min[1], net->bbox_min[2]);
  const float3 bext = make_float3(net->bbox_extent[0], net->bbox_extent[1], net->bbox_extent[2]);
  const __nv_bfloat16 *w = (const __nv_bfloat16 *)(uintptr_t)net->weights_address;
  const int grid = nrc_grid(n);
  if (encode)
    CT_TIMED(CT_K_NRC_MLP, s,
             ct_nrc::k_nrc_mlp<true><<<grid, ct_nrc::kThreads, ct_nrc::kSmemBytes, s>>>(q, nullptr, n, bmin, bext, w, rgb));
  else
    CT_TIMED(CT_K_NRC_MLP, s,
             ct_nrc::k_nrc_mlp<false><<<grid, ct_nrc::kThreads, ct_nrc::kSmemBytes, s>>>(
                 nullptr, (const __nv_bfloat16 *)encoded, n, bmin, bext, w, rgb));
  return cudaGetLastError();
}

extern "C" ct_status ct_nrc_encode(const ct_nrc_net *net, const ct_nrc_query *queries, uint32_t n, void *encoded,
                                   ct_stream stream) {
  ct_status st = check_net(net);
  if (st != CT_OK) return st;
  if (n == 0) return CT_OK;
  if (!queries || !encoded || ((uintptr_t)encoded & 15u)) return CT_ERR_INVALID_ARG;
  const float3 bmin = make_float3(net->bbox_min[0], net->bbox_min[1], net->bbox_min[2]);
  const float3 bext = make_float3(net->bbox_extent[0], net->bbox_extent[1], net->bbox_extent[2]);
  cudaStream_t s = (cudaStream_t)stream;
  CT_TIMED(CT_K_NRC_ENCODE, s,
           ct_nrc::k_nrc_encode<<<(n + ct_nrc::kEncodeThreads - 1) / ct_nrc::kEncodeThreads, ct_nrc::kEncodeThreads, 0, s>>>(queries, n, bmin, bext, (__nv_bfloat16 *)encoded));
  return nrc_status(cudaGetLastError());
}

extern "C" ct_status ct_nrc_encode_f32(const ct_nrc_net *net, const ct_nrc_query *queries, uint32_t n, float *encoded,
                                       ct_stream stream) {
  ct_status st = check_net(net);
  if (st != CT_OK) return st;
  if (n == 0) return CT_OK;
  if (!queries || !encoded || ((uintptr_t)encoded & 15u)) return CT_ERR_INVALID_ARG;
  if (n > 1u << 24) return CT_ERR_CAPACITY;
  const float3 bmin = make_float3(net->bbox_min[0], net->bbox_min[1], net->bbox_min[2]);
  const float3 bext = make_float3(net->bbox_extent[0], net->bbox_extent[1], net->bbox_extent[2]);
  cudaStream_t s = (cudaStream_t)stream;
  CT_TIMED(CT_K_NRC_ENCODE, s, ct_nrc::k_nrc_encode_f32<<<(n + 3u) / 4u, 256, 0, s>>>(queries, n, bmin, bext, (float4 *)encoded));
  return nrc_status(cudaGetLastError());
}

extern "C" ct_status ct_nrc_loss(const float *pred, const float *target, const float *weight, const float *total,
                                 uint32_t n, float *terms, float *grad, ct_stream stream) {
  if (n == 0) return CT_OK;
  if (!pred || !target || !weight || !total || !terms || !grad || ((uintptr_t)grad & 15u)) return CT_ERR_INVALID_ARG;
  if (n > 1u << 24) return CT_ERR_CAPACITY;
  cudaStream_t s = (cudaStream_t)stream;
  CT_TIMED(CT_K_NRC_LOSS, s, ct_nrc::k_nrc_loss<<<(n + 63u) / 64u, 256, 0, s>>>(pred, target, weight, total, n, terms, (float4 *)grad));
  return nrc_status(cudaGetLastError());
}

extern "C" ct_status ct_nrc_infer(const ct_nrc_net *net, const ct_nrc_query *queries, uint32_t n, float *rgb,
                                  ct_stream stream) {
  ct_status st = check_net(net);
  if (st != CT_OK) return st;
  if (n == 0) return CT_OK;
  if (!queries || !rgb) return CT_ERR_INVALID_ARG;
  return nrc_status(launch_mlp(true, net, queries, nullptr, n, rgb, (cudaStream_t)stream));
}

extern "C" ct_status ct_nrc_infer_encoded(const ct_nrc_net *net, const void *encoded, uint32_t n, float *rgb,
                                          ct_stream stream) {
  ct_status st = check_net(net);
  if (st != CT_OK) return st;
  if (n == 0) return CT_OK;
  if (!encoded || !rgb || ((uintptr_t)encoded & 15u)) return CT_ERR_INVALID_ARG;
  return nrc_status(launch_mlp(false, net, nullptr, encoded, n, rgb, (cudaStream_t)stream));
}

extern "C" ct_status ct_nrc_status(int reset, uint32_t *out) {
  if (!out) return CT_ERR_INVALID_ARG;
  cudaError_t e = cudaMemcpyFromSymbol(out, ct_nrc::g_nrc_status, sizeof(uint32_t));
  if (e == cudaSuccess && reset) {
    const uint32_t zero = 0;
    e = cudaMemcpyToSymbol(ct_nrc::g_nrc_status, &zero, sizeof(uint32_t));
  }
  return nrc_status(e);
}

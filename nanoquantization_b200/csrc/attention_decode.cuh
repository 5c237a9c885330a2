// Attention of one decode step (one token per sequence) over a paged cache, heads of 128, 16-bit types: head norms, rotary
// embedding and the K/V store of the step's token, scores, softmax (plain, capped, with a sink) or sigmoid weights, and the
// weighted values, in one launch.
//
// Bound by reading the visible keys and values once.  A thread-block cluster takes one (sequence, key/value head, group of up
// to eight query heads) and splits the keys over its CTAs; inside a CTA every warp takes tiles of 16 keys on its own, through
// a ring of its own that it fills with cp.async, so that nothing but the end waits for another warp.
//
//   scores   S[key, head] = K q: mma m16n8k16 with the keys as rows and the query heads as its eight columns, so that a small
//            group of heads wastes columns and not rows;
//   weights  a lane holds two heads' weights of two keys; packed to 16 bits and transposed in registers (movmatrix) they are
//            the second operand of the next product;
//   values   O[dim, head] = V^T p: V through a transposing ldmatrix, 16 dimensions per mma.
//
// A lane's maxima, sums and accumulators all belong to the same two heads.  The warps meet in shared memory, the CTAs of a
// cluster in distributed shared memory, always in the same order.
//
// 48 sequences of about 1140 keys, 32 heads over 8, bfloat16 (223 MB, 35 us at the copy rate): 41 us, where flash_attn's paged
// kernel with a launch for QK-norm and K/V store takes 71.  One sequence of 2048 keys: 9.1 us, 14.1.  The one place found where those
// are ahead: 64 sequences of 100 keys, 64 heads over 8 (512 CTAs where 444 are resident): 16.4 us, 15.3.
#pragma once
#include <cooperative_groups.h>
#include "common.cuh"

namespace nqb200 {
namespace attdec {

namespace cg = cooperative_groups;

constexpr int kDim = 128, kWarps = 4, kThreads = 32 * kWarps, kTile = 16, kHeads = 8;
constexpr int kTileBytes = 2 * kTile * kDim * 2;              // keys, then values
__host__ __device__ constexpr int ring_bytes(int stages) { return kWarps * stages * kTileBytes; }
constexpr int kOS = kDim + 4;                                 // stride of a head's partial sums
constexpr int kShare = kDim + 4;                              // floats of a head's share: sums, maximum, sum of weights
constexpr float kLog2e = 1.4426950408889634f;

enum Mode { kSoftmax = 0, kCapped = 1, kSigmoid = 2 };

template <typename T> struct Args {
  const T* proj; int64_t stride;                   // the step's projections, a row per sequence
  int64_t q_off, k_off, v_off;                     // elements; head h of q at q_off + 128 h
  T *k_cache, *v_cache;                            // [rows, kv_heads, 128]
  const int32_t* table; int table_width, block_size;
  const int32_t* last; int last_shift;             // the step's token stands at last[b] + last_shift
  const int64_t* rows;                             // its cache row, or null: from the table
  int heads, kv_heads, head_groups, chunk;         // chunk 0: every earlier key is visible
  T* out; int64_t out_stride, out_col;
  float scale, softcap, out_scale;
  const float *sink, *temp, *bias;                 // per query head, or null
  // rotation by angles position * inv_freq, in float, of the first `rot` dimensions, with norms where q_norm is given
  int rot, interleaved;
  const float *inv_freq, *q_norm, *k_norm;
  float eps;
  // or (cos_sin given) by a [position, cos | sin] table after norms with 16-bit weights, rounded where 16-bit tensors would stand
  const float* cos_sin; const int64_t* positions;
  const T *q_weight, *k_weight;
  float* shares; int parts;                        // a sequence over several clusters (parts > 1, plain softmax): their shares
};

struct Fixed {                                     // behind the ring
  alignas(16) uint16_t q[kHeads][kDim + 8];
  alignas(16) uint16_t knew[kDim];
  float m[kWarps][kHeads], l[kWarps][kHeads];
  float cm[kHeads], cl[kHeads];                    // of the CTA, read by the cluster
  float out[kHeads][kDim];
};
__host__ __device__ constexpr int smem_bytes(int stages) { return ring_bytes(stages) + (int)sizeof(Fixed); }

template <typename T> struct Traits;
template <> struct Traits<__half> { static constexpr bool kBf16 = false; };
template <> struct Traits<__nv_bfloat16> { static constexpr bool kBf16 = true; };

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool ok) {
  const int n = ok ? 16 : 0;                       // zeros where there is nothing to read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n));
}
template <bool BF16>
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ uint32_t transpose8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ float exp2_fast(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float recip_fast(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

// The step's own query heads (into fx.q, zeros beyond R) and key (into fx.knew): a head per warp at a time, a lane holds
// elements 4 lane .. 4 lane + 3 and gets their partners in the rotation by shuffles.
constexpr int kNew = (kHeads + kWarps) / kWarps;              // heads and key per warp at most
template <typename T>
__device__ __forceinline__ void request_new(const Args<T>& a, uint2 (&raw)[kNew], const T* row, int h0, int R, int kvh, bool newest) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < kNew; ++i) {
    const int r = warp + i * kWarps;
    raw[i] = make_uint2(0u, 0u);
    if (r < R || (newest && r == kHeads))
      raw[i] = reinterpret_cast<const uint2*>(r < kHeads ? row + a.q_off + (int64_t)(h0 + r) * kDim : row + a.k_off + (int64_t)kvh * kDim)[lane];
  }
}
template <typename T>
__device__ __forceinline__ void rotate_new(const Args<T>& a, Fixed& fx, const uint2 (&raws)[kNew], int b, int pos, int R, bool newest) {
  constexpr bool BF16 = Traits<T>::kBf16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool tabled = a.cos_sin != nullptr;
  const int rot = tabled ? kDim : a.rot, half = rot / 2;
  float c[4], s[4];                                // of this lane's elements; s with the sign of the partner's term
  int mate[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int i = 4 * lane + e;
    const bool swap = !tabled && a.interleaved, first = swap ? (i & 1) == 0 : i < half;
    const int f = swap ? i >> 1 : first ? i : i - half;
    c[e] = 1.f;
    s[e] = 0.f;
    mate[e] = i;
    if (i < rot) {
      mate[e] = swap ? i ^ 1 : first ? i + half : i - half;
      if (tabled) {
        const float* cs = a.cos_sin + a.positions[b] * kDim;   // [cos(64) | sin(64)]
        c[e] = cs[f];
        s[e] = cs[half + f];
      } else {
        sincosf((float)pos * a.inv_freq[f], &s[e], &c[e]);
      }
      if (first) s[e] = -s[e];
    }
  }
#pragma unroll
  for (int i = 0; i < kNew; ++i) {
    const int r = warp + i * kWarps;
    if (r >= kHeads + (newest ? 1 : 0)) break;
    uint2* dst = reinterpret_cast<uint2*>(r < kHeads ? fx.q[r] : fx.knew) + lane;
    if (r >= R && r < kHeads) {
      *dst = make_uint2(0u, 0u);
      continue;
    }
    const uint2 raw = raws[i];
    float v[4] = {raw16_to_float<BF16>((uint16_t)(raw.x & 0xFFFF)), raw16_to_float<BF16>((uint16_t)(raw.x >> 16)),
                  raw16_to_float<BF16>((uint16_t)(raw.y & 0xFFFF)), raw16_to_float<BF16>((uint16_t)(raw.y >> 16))};
    if (tabled || a.q_norm) {
      float ss = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
      if (tabled) {
        const float inv = rsqrtf(ss / (float)kDim + a.eps);
        const uint16_t* w = reinterpret_cast<const uint16_t*>(r < kHeads ? a.q_weight : a.k_weight) + 4 * lane;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          v[e] = raw16_to_float<BF16>(float_to_raw16<BF16>(raw16_to_float<BF16>(float_to_raw16<BF16>(v[e] * inv)) * raw16_to_float<BF16>(w[e])));
      } else {
        const float inv = 1.f / sqrtf(ss / (float)kDim + a.eps);
        const float* w = (r < kHeads ? a.q_norm : a.k_norm) + 4 * lane;
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = v[e] * inv * w[e];
      }
    }
    uint32_t y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float other = 0.f;
      if (tabled) {                                // half a head away: the same element of the lane 16 on
        other = __shfl_xor_sync(0xFFFFFFFFu, v[e], 16);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float t = __shfl_sync(0xFFFFFFFFu, v[k], mate[e] >> 2);
          if (k == (mate[e] & 3)) other = t;
        }
      }
      y[e] = float_to_raw16<BF16>(4 * lane + e < rot ? v[e] * c[e] + other * s[e] : v[e]);   // an infinity passes as it is
    }
    *dst = make_uint2(y[0] | (y[1] << 16), y[2] | (y[3] << 16));
  }
}

// STAGES: tiles of a warp's ring.  Two (one under way while one is used) leave room for three CTAs per SM; a grid of no more
// than two, or one, per SM takes three, or four, so that as much is under way.  64 CTAs of 256 keys: 10.9 us with two, 9.4
// with four; 256 CTAs of 950 keys: 34 us with two, 29 with three; 384 CTAs of 1300 keys: 59 us with three, 49 with two.
template <typename T, int MODE, int STAGES>
__global__ void __launch_bounds__(kThreads, STAGES == 2 ? 3 : STAGES == 3 ? 2 : 1) attention_decode_kernel(const __grid_constant__ Args<T> a) {
  constexpr bool BF16 = Traits<T>::kBf16;
  constexpr int kStages = STAGES, kRing = ring_bytes(STAGES);
  extern __shared__ __align__(128) uint8_t smem[];
  Fixed& fx = *reinterpret_cast<Fixed*>(smem + kRing);
  grid_launch_dependents();
  grid_dependency_wait();
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, csize = gridDim.x / a.parts, rank = blockIdx.x % csize;
  const int unit = blockIdx.y, b = blockIdx.z;
  const int per_kv = a.heads / a.kv_heads, kvh = unit / a.head_groups, hg = unit % a.head_groups;
  const int h0 = kvh * per_kv + hg * kHeads, R = min(kHeads, per_kv - hg * kHeads);
  const int pos = a.last[b] + a.last_shift;
  const int lo = a.chunk > 0 ? pos / a.chunk * a.chunk : 0;
  // a position below 0: a row without a sequence, which has no tile to read and none to store, and gets zeros
  const int tiles = pos < 0 ? 0 : (pos - lo) / kTile + 1, per = (tiles + (int)gridDim.x - 1) / (int)gridDim.x;
  const int t0 = min((int)blockIdx.x * per, tiles), t1 = min(t0 + per, tiles);
  const bool newest = t1 == tiles && t0 < t1;      // this CTA has the tile with the step's own key
  const T* row = a.proj + (int64_t)b * a.stride;
  uint8_t* ring = smem + warp * (kStages * kTileBytes);
  const uint32_t ring_a = smem_addr(ring);
  const int32_t* table = a.table + (int64_t)b * a.table_width;

  // 16-byte piece c of key k of a tile at k * 256 + ((c ^ (k & 7)) * 16): ldmatrix finds eight keys' pieces in different banks
  auto load = [&](int t, int stage) {
    if (t < t1) {
      const int p0 = lo + t * kTile, mine = min(p0 + (lane & 15), pos), blk = mine / a.block_size;
      const int at = table[blk] * a.block_size + (mine - blk * a.block_size);
      const int c = lane & 15;
#pragma unroll
      for (int i = 0; i < kTile / 2; ++i) {
        const int k = 2 * i + (lane >> 4);
        const int64_t src = ((int64_t)__shfl_sync(0xFFFFFFFFu, at, k) * a.kv_heads + kvh) * kDim + c * 8;
        const uint32_t dst = ring_a + stage * kTileBytes + k * 256 + ((c ^ (k & 7)) << 4);
        const bool ok = p0 + k < pos;
        copy16(dst, a.k_cache + src, ok);
        copy16(dst + kTile * 256, a.v_cache + src, ok);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // requested ahead of the table's entries, so that the two trips to memory are one
  uint2 raws[kNew];
  if (pos >= 0) request_new<T>(a, raws, row, h0, R, kvh, newest);
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) load(t0 + warp + s * kWarps, s);

  if (pos >= 0) rotate_new<T>(a, fx, raws, b, pos, R, newest);
  __syncthreads();

  const int g = lane >> 2, t4 = lane & 3;
  uint32_t qf[8][2];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    qf[k][0] = *reinterpret_cast<const uint32_t*>(&fx.q[g][16 * k + 2 * t4]);
    qf[k][1] = *reinterpret_cast<const uint32_t*>(&fx.q[g][16 * k + 8 + 2 * t4]);
  }
  // of this lane's two heads, 2 t4 and 2 t4 + 1
  float factor[2], shift[2], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = 2 * t4 + u;
    factor[u] = a.scale * (a.temp && r < R ? a.temp[h0 + r] : 1.f);
    shift[u] = a.bias && r < R ? a.bias[h0 + r] : 0.f;
    if (MODE == kSoftmax) { factor[u] *= kLog2e; shift[u] *= kLog2e; }
  }
  const float inv_cap = MODE == kCapped ? 1.f / a.softcap : 0.f;
  float O[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) O[i][e] = 0.f;
  // lane's row and piece for ldmatrix: keys as stored, and values transposed
  const int krow = lane & 15, kpiece = lane >> 4, vrow = (lane & 7) + ((lane >> 4) << 3), vpiece = (lane >> 3) & 1;

  int stage = 0;
  for (int t = t0 + warp; t < t1; t += kWarps) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncwarp();                                  // the tile is there for every lane, the one before it is no longer read
    const int ahead = stage == 0 ? kStages - 1 : stage - 1;
    load(t + (kStages - 1) * kWarps, ahead);
    const uint32_t kt = ring_a + stage * kTileBytes, vt = kt + kTile * 256;
    const int p0 = lo + t * kTile;
    if (t == tiles - 1) {                          // the step's own key and value: into the tile, and into the cache
      const int k = pos - p0, c = lane & 15;
      const bool is_v = lane >= 16;
      const uint4 v = is_v ? *reinterpret_cast<const uint4*>(row + a.v_off + (int64_t)kvh * kDim + c * 8) : *reinterpret_cast<const uint4*>(fx.knew + c * 8);
      *reinterpret_cast<uint4*>(ring + stage * kTileBytes + (is_v ? kTile * 256 : 0) + k * 256 + ((c ^ (k & 7)) << 4)) = v;
      if (hg == 0) {
        const int blk = pos / a.block_size;
        const int64_t at = a.rows ? a.rows[b] : (int64_t)table[blk] * a.block_size + (pos - blk * a.block_size);
        *reinterpret_cast<uint4*>((is_v ? a.v_cache : a.k_cache) + (at * a.kv_heads + kvh) * kDim + c * 8) = v;
      }
      __syncwarp();
    }
    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      uint32_t kf[4];
      ldsm4(kf, kt + krow * 256 + (((2 * k + kpiece) ^ (krow & 7)) << 4));
      mma<BF16>(c, kf, qf[k][0], qf[k][1]);
    }
    float x[4];
    const bool in[2] = {p0 + g <= pos, p0 + g + 8 <= pos};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float s = c[e] * factor[e & 1] + shift[e & 1];
      // tanh as 1 - 2 / (1 + e^2y)
      if (MODE == kCapped) s = (a.softcap * kLog2e) * (1.f - 2.f * recip_fast(1.f + exp2_fast(s * inv_cap * (2.f * kLog2e))));
      if (MODE == kSigmoid) x[e] = in[e >> 1] ? recip_fast(1.f + exp2_fast(s * -kLog2e)) : 0.f;
      else x[e] = in[e >> 1] ? s : -INFINITY;
    }
    if (MODE != kSigmoid) {
      float top[2] = {fmaxf(x[0], x[2]), fmaxf(x[1], x[3])};
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        top[0] = fmaxf(top[0], __shfl_xor_sync(0xFFFFFFFFu, top[0], o));
        top[1] = fmaxf(top[1], __shfl_xor_sync(0xFFFFFFFFu, top[1], o));
      }
      if (__any_sync(0xFFFFFFFFu, top[0] > m[0] || top[1] > m[1])) {
        float corr[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float n = fmaxf(m[u], top[u]);
          corr[u] = m[u] == n ? 1.f : exp2_fast(m[u] - n);   // 0 ahead of the first tile
          m[u] = n;
          l[u] *= corr[u];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) { O[i][0] *= corr[0]; O[i][1] *= corr[1]; O[i][2] *= corr[0]; O[i][3] *= corr[1]; }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x[e] = m[e & 1] == -INFINITY ? (isnan(x[e]) ? x[e] : 0.f) : exp2_fast(x[e] - m[e & 1]);   // no finite score so far: no weight
        l[e & 1] += x[e];
      }
    }
    const uint32_t p_lo = transpose8((uint32_t)float_to_raw16<BF16>(x[0]) | ((uint32_t)float_to_raw16<BF16>(x[1]) << 16));
    const uint32_t p_hi = transpose8((uint32_t)float_to_raw16<BF16>(x[2]) | ((uint32_t)float_to_raw16<BF16>(x[3]) << 16));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t vf[4];
      ldsm4t(vf, vt + vrow * 256 + (((2 * i + vpiece) ^ (vrow & 7)) << 4));
      mma<BF16>(O[i], vf, p_lo, p_hi);
    }
    stage = stage + 1 == kStages ? 0 : stage + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();

  // the warps' shares over their rings
  float* po = reinterpret_cast<float*>(ring);      // [head][kOS]
#pragma unroll
  for (int i = 0; i < 8; ++i) {
#pragma unroll
    for (int e = 0; e < 4; ++e) po[(2 * t4 + (e & 1)) * kOS + 16 * i + g + 8 * (e >> 1)] = O[i][e];
  }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    l[0] += __shfl_xor_sync(0xFFFFFFFFu, l[0], o);
    l[1] += __shfl_xor_sync(0xFFFFFFFFu, l[1], o);
  }
  if (lane < 4) {
#pragma unroll
    for (int u = 0; u < 2; ++u) { fx.m[warp][2 * lane + u] = m[u]; fx.l[warp][2 * lane + u] = l[u]; }
  }
  __syncthreads();
  T* out = a.out + (int64_t)b * a.out_stride + a.out_col;
  const auto finish = [&](int r, int d, float o, float sum, float top) {   // top in units of log 2
    if (MODE == kSoftmax && a.parts > 1) {
      float* share = a.shares + (((int64_t)b * a.heads + h0 + r) * a.parts + blockIdx.x / csize) * kShare;
      share[d] = o;
      if (d == 0) { share[kDim] = top; share[kDim + 1] = sum; }
      return;
    }
    if (MODE != kSigmoid) {
      if (a.sink) sum += exp2_fast(a.sink[h0 + r] * kLog2e - top);
      o = pos < 0 ? 0.f : o / sum;
    }
    reinterpret_cast<uint16_t*>(out)[(int64_t)(h0 + r) * kDim + d] = float_to_raw16<BF16>(o * a.out_scale);
  };
  for (int r = 0; r < R; ++r) {
    float top = -INFINITY, o = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) top = fmaxf(top, fx.m[w][r]);
    // the sink takes part in the maximum, or its weight could overflow
    if (MODE != kSigmoid && a.sink) top = fmaxf(top, a.sink[h0 + r] * kLog2e);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = MODE == kSigmoid || fx.m[w][r] == top ? 1.f : exp2_fast(fx.m[w][r] - top);   // 0: a warp without keys
      o += f * reinterpret_cast<const float*>(smem + w * (kStages * kTileBytes))[r * kOS + tid];
      sum += f * fx.l[w][r];
    }
    if (csize == 1) {
      finish(r, tid, o, sum, top);
    } else {
      fx.out[r][tid] = o;
      if (tid == 0) { fx.cm[r] = top; fx.cl[r] = sum; }
    }
  }
  if (csize == 1) return;
  cl.sync();
  for (int e = rank * kThreads + tid; e < R * kDim; e += csize * kThreads) {
    const int r = e / kDim, d = e % kDim;
    float pm[8], pl[8], po8[8], top = -INFINITY, o = 0.f, sum = 0.f;   // all of the cluster's shares at once
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const Fixed* s = cl.map_shared_rank(&fx, k < csize ? k : 0);
      pm[k] = k < csize ? s->cm[r] : -INFINITY;
      pl[k] = s->cl[r];
      po8[k] = s->out[r][d];
      top = fmaxf(top, pm[k]);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float f = k >= csize ? 0.f : MODE == kSigmoid || pm[k] == top ? 1.f : exp2_fast(pm[k] - top);
      o += f * po8[k];
      sum += f * pl[k];
    }
    finish(r, d, o, sum, top);
  }
  cl.sync();                                       // peers may still read this CTA's shared memory
}

// The shares of a sequence's clusters, a CTA per (query head, sequence), in the clusters' order.
template <typename T>
__global__ void __launch_bounds__(kThreads) attention_shares_kernel(const float* __restrict__ shares, T* __restrict__ out, int64_t out_stride, int parts, const int32_t* last,
                                                                    int last_shift) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int64_t head = (int64_t)blockIdx.y * gridDim.x + blockIdx.x;
  const float* s = shares + head * parts * kShare;
  float top = -INFINITY, sum = 0.f, o = 0.f;
  for (int p = 0; p < parts; ++p) top = fmaxf(top, s[p * kShare + kDim]);
#pragma unroll 4
  for (int p = 0; p < parts; ++p) {
    const float m = s[p * kShare + kDim], f = m == top ? 1.f : exp2f(m - top);
    o += f * s[p * kShare + threadIdx.x];
    sum += f * s[p * kShare + kDim + 1];
  }
  o = last[blockIdx.y] + last_shift < 0 ? 0.f : o / sum;   // as above: a row without a sequence
  reinterpret_cast<uint16_t*>(out)[blockIdx.y * out_stride + (int64_t)blockIdx.x * kDim + threadIdx.x] = float_to_raw16<Traits<T>::kBf16>(o);
}

static inline bool supported(int64_t heads, int64_t kv_heads, int64_t dim, int64_t vdim) {
  return dim == kDim && vdim == kDim && kv_heads > 0 && heads > 0 && heads % kv_heads == 0 && kv_heads <= 4096 && heads <= 65535;
}

// PLAIN: the caller has neither capped scores nor sigmoid weights, and their kernels are not built.
template <typename T, int STAGES, bool PLAIN>
static inline int launch_stages(const Args<T>& a, int csize, int64_t batch, bool sigmoid, cudaStream_t st) {
  constexpr int smem = smem_bytes(STAGES);
  const auto kernel = PLAIN ? attention_decode_kernel<T, kSoftmax, STAGES>
                      : sigmoid        ? attention_decode_kernel<T, PLAIN ? kSoftmax : kSigmoid, STAGES>
                      : a.softcap > 0.f ? attention_decode_kernel<T, PLAIN ? kSoftmax : kCapped, STAGES>
                                        : attention_decode_kernel<T, kSoftmax, STAGES>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) { cudaGetLastError(); return NQB200_ERR_LAUNCH; }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(csize * a.parts), (unsigned)(a.kv_heads * a.head_groups), (unsigned)batch);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)csize;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, kernel, a) != cudaSuccess) { cudaGetLastError(); return NQB200_ERR_LAUNCH; }
  return NQB200_OK;
}

// How a step is split.  Clusters of 1, 2, 4, 8 CTAs that a B200 holds at once (cudaOccupancyMaxActiveClusters; clusters do not
// cross the chip's processing clusters, so that 15 and not 18 of eight fit), with a ring of 4, 3, 2 tiles per warp:
constexpr int kResident[4][3] = {{148, 296, 444}, {74, 148, 222}, {33, 71, 104}, {15, 33, 48}};
constexpr int kMostParts = 16;
struct Split { int csize, stages, parts; };
// `keys`: the most that a sequence of the step may see.  A CTA for every 64 keys (a tile per warp) as long as all clusters are
// resident, and as long a ring as leaves them so.  2 sequences of 16384 keys, 8 key/value heads: 60 us where the 16 clusters of
// eight did not fit at once (ring of 4), 34 so.
// Where clusters of eight leave the chip unfilled and a CTA would get 1024 keys or more, and `shares` may be used, a sequence goes
// over several of them, down to 256 keys a CTA (1024 where 16 clusters have an SM per CTA already), and a second kernel adds their
// shares (about 3 us).  One sequence of 32768 keys, 8 key/value heads: 52 us over one cluster each, 28.8 over four; 1 key/value
// head: 52 over one, 15.0 over sixteen; at 8192 keys 17.7 and 14.2, 18.2 and 11.5; at 4096 keys 12.0 and 12.0, 12.5 and 9.9.  16 clusters
// of 1024 keys a CTA: 21.4 us, 25.9 when split in two.
static inline Split split(int64_t units, int64_t keys, bool shares) {
  Split s = {1, 2, 1};
  int row = 0;
  while (row < 3 && units <= kResident[row + 1][2] && keys > (int64_t)s.csize * kWarps * kTile) { s.csize *= 2; ++row; }
  if (shares && row == 3 && keys >= 8 * 1024) {
    const int64_t least = units > kResident[3][0] ? 1024 : 256;
    while (s.parts < kMostParts && units * s.parts * 2 <= kResident[3][1] && keys >= 8 * s.parts * 2 * least) s.parts *= 2;
  }
  while (s.stages < 4 && units * s.parts <= kResident[row][3 - s.stages]) ++s.stages;
  // few keys, and as many turns with two CTAs per SM as with three: 512 of 100 keys 15.3 and 15.7 us, of 300 23.4 and 24.4
  const auto turns = [&](int per_sm) { return (units + kNumSMs * per_sm - 1) / (kNumSMs * per_sm); };
  if (s.stages == 2 && s.csize == 1 && keys <= 512 && turns(2) == turns(3)) s.stages = 3;
  return s;
}
static inline int head_groups(int heads, int kv_heads) { return (heads / kv_heads + kHeads - 1) / kHeads; }
static inline int64_t share_floats(int64_t batch, int heads, int parts) { return parts > 1 ? batch * heads * parts * kShare : 0; }

template <bool PLAIN, typename T>
static inline int launch(Args<T>& a, int64_t batch, int64_t keys, bool sigmoid, cudaStream_t st) {
  a.head_groups = head_groups(a.heads, a.kv_heads);
  const Split s = split((int64_t)a.kv_heads * a.head_groups * batch, keys, a.shares != nullptr);
  a.parts = s.parts;
  const int rc = s.stages == 4   ? launch_stages<T, 4, PLAIN>(a, s.csize, batch, sigmoid, st)
                 : s.stages == 3 ? launch_stages<T, 3, PLAIN>(a, s.csize, batch, sigmoid, st)
                                 : launch_stages<T, 2, PLAIN>(a, s.csize, batch, sigmoid, st);
  if (rc != NQB200_OK || s.parts == 1) return rc;
  return launch_overlapped(attention_shares_kernel<T>, dim3((unsigned)a.heads, (unsigned)batch), dim3(kThreads), 0, st, (const float*)a.shares, a.out + a.out_col,
                           a.out_stride, s.parts, a.last, a.last_shift);
}

}  // namespace attdec
}  // namespace nqb200

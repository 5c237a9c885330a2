// The elementwise steps either side of the linears in a Qwen3 block, one kernel
// each instead of the 5-10 small launches PyTorch needs: residual add + RMSNorm,
// per-head QK-norm + rotary embedding, SiLU(gate) * up.  At decode these launches
// cost as much as the GEMVs.  Roundings follow the reference modules exactly
// (nanoquantization/layers/norm.py:18-32, layers/rope.py:24-45,
// models/qwen3_quantized.py:150,213-214): fp32 inside, one rounding to the
// 16-bit type wherever the reference materialises a 16-bit tensor.
#include "common.cuh"

namespace nqb200 {

template <bool BF16> __device__ __forceinline__ float rnd16(float v) { return raw16_to_float<BF16>(float_to_raw16<BF16>(v)); }

// One CTA per token.  h = x (+ residual), rounded; residual_out = h; out = (round16(h * rsqrt(mean(h^2)+eps))) * w.
template <bool BF16>
__global__ void __launch_bounds__(256) add_rmsnorm_kernel(const uint16_t* __restrict__ x, const uint16_t* residual,
                                                          const uint16_t* __restrict__ weight, uint16_t* __restrict__ out,
                                                          uint16_t* residual_out, int H, float eps) {
  extern __shared__ float hbuf[];  // H floats
  __shared__ float red[8];
  grid_launch_dependents();  // the next kernel's weight fetch may start now
  grid_dependency_wait();    // x and residual come from the kernel ahead
  const size_t row = (size_t)blockIdx.x * H;
  float ss = 0.f;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float h = raw16_to_float<BF16>(x[row + i]);
    if (residual) h = rnd16<BF16>(h + raw16_to_float<BF16>(residual[row + i]));
    if (residual_out) residual_out[row + i] = float_to_raw16<BF16>(h);
    hbuf[i] = h;
    ss += h * h;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) tot += red[w];
  const float inv = rsqrtf(tot / (float)H + eps);
  for (int i = threadIdx.x; i < H; i += blockDim.x)
    out[row + i] = float_to_raw16<BF16>(rnd16<BF16>(hbuf[i] * inv) * raw16_to_float<BF16>(weight[i]));
}

// Eight 16-bit values held as four words.
template <bool BF16> __device__ __forceinline__ void unpack8(const uint4& r, float (&v)[8]) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[2 * k] = raw16_to_float<BF16>((uint16_t)(w[k] & 0xFFFF));
    v[2 * k + 1] = raw16_to_float<BF16>((uint16_t)(w[k] >> 16));
  }
}
template <bool BF16> __device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = (uint32_t)float_to_raw16<BF16>(v[2 * k]) | ((uint32_t)float_to_raw16<BF16>(v[2 * k + 1]) << 16);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// The same for rows of whole 16-byte pieces.  Bound by memory (8 bytes per element) for prompts and by latency for a few
// tokens, so a row is spread over as many threads as it has pieces, up to 512, every load of the row is under way at
// once, and the row stays in registers between the sum and the use.
// H = 4096, bfloat16, with residual: 3000 rows 46 us element by element, 24 us so (4.1 TB/s); 48 rows 13.5 and 2.4 us;
// 1 row 14.5 and 2.7 us.
template <bool BF16, int PIECES>
__global__ void __launch_bounds__(512) add_rmsnorm_vec_kernel(const uint16_t* __restrict__ x, const uint16_t* residual,
                                                              const uint16_t* __restrict__ weight, uint16_t* __restrict__ out,
                                                              uint16_t* residual_out, int H, float eps) {
  __shared__ float red[16];
  grid_launch_dependents();
  const int n8 = H >> 3, tid = threadIdx.x, threads = blockDim.x;
  const size_t row = (size_t)blockIdx.x * n8;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 w[PIECES], a[PIECES], r[PIECES];
  grid_dependency_wait();
#pragma unroll
  for (int j = 0; j < PIECES; ++j) {
    const int c = tid + j * threads;
    a[j] = c < n8 ? reinterpret_cast<const uint4*>(x)[row + c] : zero;
    r[j] = residual && c < n8 ? reinterpret_cast<const uint4*>(residual)[row + c] : zero;
    w[j] = c < n8 ? reinterpret_cast<const uint4*>(weight)[c] : zero;
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < PIECES; ++j) {
    float h[8];
    unpack8<BF16>(a[j], h);
    if (residual) {
      float o[8];
      unpack8<BF16>(r[j], o);
#pragma unroll
      for (int e = 0; e < 8; ++e) h[e] = rnd16<BF16>(h[e] + o[e]);
      a[j] = pack8<BF16>(h);
    }
    const int c = tid + j * threads;
    if (residual_out && c < n8) reinterpret_cast<uint4*>(residual_out)[row + c] = a[j];
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += h[e] * h[e];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int q = 0; q < (threads >> 5); ++q) tot += red[q];
  const float inv = rsqrtf(tot / (float)H + eps);
#pragma unroll
  for (int j = 0; j < PIECES; ++j) {
    float h[8], g[8];
    unpack8<BF16>(a[j], h);
    unpack8<BF16>(w[j], g);
#pragma unroll
    for (int e = 0; e < 8; ++e) h[e] = rnd16<BF16>(h[e] * inv) * g[e];
    const int c = tid + j * threads;
    if (c < n8) reinterpret_cast<uint4*>(out)[row + c] = pack8<BF16>(h);
  }
}

// One warp per (token, head) of q and k inside a fused [T, (Hq + 2*Hkv) * D] buffer, D = 128, in place:
// RMSNorm over the head (weight qw / kw), then the half-split rotation with the fp32 cos|sin table row
// of the token's position.  v is untouched.  With a paged cache given ([slots, Hkv, D] for k and for v,
// slot_of[t] = the token's slot), the rotated k and the v of every token are also stored there by
// the warps that hold them, which saves the two scatter launches that would follow.
template <bool BF16>
__global__ void __launch_bounds__(256) qknorm_rope_kernel(uint16_t* __restrict__ qkv, const uint16_t* __restrict__ qw,
                                                          const uint16_t* __restrict__ kw, const float* __restrict__ cos_sin,
                                                          const int64_t* __restrict__ positions, int T, int Hq, int Hkv,
                                                          int row_stride, float eps, const int64_t* __restrict__ slot_of,
                                                          uint16_t* __restrict__ k_cache, uint16_t* __restrict__ v_cache) {
  constexpr int D = 128;
  grid_launch_dependents();
  grid_dependency_wait();
  const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int heads = Hq + Hkv + (slot_of ? Hkv : 0);  // with a cache, the v heads get a warp each too
  if (gw >= T * heads) return;
  const int t = gw / heads, hd = gw % heads;
  uint16_t* p = qkv + (size_t)t * row_stride + (size_t)hd * D;  // q heads first, then k heads, then v heads
  if (hd >= Hq + Hkv) {
    // a v head: 256 bytes to its slot
    uint16_t* dst = v_cache + ((size_t)slot_of[t] * Hkv + (hd - Hq - Hkv)) * D;
    reinterpret_cast<uint2*>(dst)[lane] = reinterpret_cast<const uint2*>(p)[lane];
    return;
  }
  const uint16_t* w = hd < Hq ? qw : kw;
  // lane owns elements lane, lane+32, lane+64, lane+96: (lane, lane+64) and (lane+32, lane+96) are rotation pairs
  float v[4];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) { v[j] = raw16_to_float<BF16>(p[lane + 32 * j]); ss += v[j] * v[j]; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
  const float inv = rsqrtf(ss / (float)D + eps);
#pragma unroll
  for (int j = 0; j < 4; ++j)
    v[j] = rnd16<BF16>(rnd16<BF16>(v[j] * inv) * raw16_to_float<BF16>(w[lane + 32 * j]));
  const float* cs = cos_sin + (size_t)positions[t] * D;  // [cos(64) | sin(64)]
  uint16_t* kdst = (slot_of && hd >= Hq) ? k_cache + ((size_t)slot_of[t] * Hkv + (hd - Hq)) * D : nullptr;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int i = lane + 32 * j;
    const float c = cs[i], s = cs[64 + i];
    const float a = v[j], b = v[j + 2];
    const uint16_t lo = float_to_raw16<BF16>(a * c - b * s), hi = float_to_raw16<BF16>(a * s + b * c);
    p[i] = lo;
    p[i + 64] = hi;
    if (kdst) { kdst[i] = lo; kdst[i + 64] = hi; }
  }
}

// The same for buffers whose rows start on 8-byte boundaries: half a warp per (token, head).
template <bool BF16>
__global__ void __launch_bounds__(256) qknorm_rope_vec_kernel(uint16_t* __restrict__ qkv, const uint16_t* __restrict__ qw,
                                                              const uint16_t* __restrict__ kw, const float* __restrict__ cos_sin,
                                                              const int64_t* __restrict__ positions, int T, int Hq, int Hkv,
                                                              int row_stride, float eps, const int64_t* __restrict__ slot_of,
                                                              uint16_t* __restrict__ k_cache, uint16_t* __restrict__ v_cache) {
  constexpr int D = 128;
  grid_launch_dependents();
  grid_dependency_wait();
  // 16 lanes per head, two heads per warp: lane l of a head owns elements 4l..4l+3 and their partners 64 places on, so
  // that every access is 8 bytes wide and a head's 256 bytes are two of them.  3000 tokens of
  // 32 + 8 + 8 heads, with the cache: 29 us with 2-byte accesses, 21 us so.
  const int lane = threadIdx.x & 15;
  const int heads = Hq + Hkv + (slot_of ? Hkv : 0);  // with a cache, the v heads get their lanes too
  const int at = blockIdx.x * (blockDim.x >> 4) + (threadIdx.x >> 4);
  const bool in = at < T * heads;                     // the other head of the warp may still be inside: no early return
  const int t = in ? at / heads : 0, hd = in ? at - t * heads : 0;
  uint2* p = reinterpret_cast<uint2*>(qkv + (size_t)t * row_stride + (size_t)hd * D);  // q heads, then k heads, then v heads
  uint2 lo = p[lane], hi = p[lane + 16];
  const bool is_v = hd >= Hq + Hkv;
  uint2* dst = nullptr;   // the cache row, for k and v
  if (slot_of && hd >= Hq) {
    const size_t row = (size_t)slot_of[t] * Hkv;
    dst = reinterpret_cast<uint2*>(is_v ? v_cache + (row + (hd - Hq - Hkv)) * D : k_cache + (row + (hd - Hq)) * D);
  }
  float a[4], b[4];
  const uint32_t lw[2] = {lo.x, lo.y}, hw[2] = {hi.x, hi.y};
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    a[e] = raw16_to_float<BF16>((uint16_t)(lw[e >> 1] >> (16 * (e & 1))));
    b[e] = raw16_to_float<BF16>((uint16_t)(hw[e >> 1] >> (16 * (e & 1))));
    ss += a[e] * a[e] + b[e] * b[e];
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
  if (!is_v) {
    const float inv = rsqrtf(ss / (float)D + eps);
    const uint2* w = reinterpret_cast<const uint2*>(hd < Hq ? qw : kw);
    const uint2 wl = w[lane], wh = w[lane + 16];
    const uint32_t wlw[2] = {wl.x, wl.y}, whw[2] = {wh.x, wh.y};
    const float4* cs = reinterpret_cast<const float4*>(cos_sin + (size_t)positions[t] * D);  // [cos(64) | sin(64)]
    const float4 cv = cs[lane], sv = cs[lane + 16];
    const float c[4] = {cv.x, cv.y, cv.z, cv.w}, s[4] = {sv.x, sv.y, sv.z, sv.w};
    uint32_t ol[2] = {0u, 0u}, oh[2] = {0u, 0u};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float u = rnd16<BF16>(rnd16<BF16>(a[e] * inv) * raw16_to_float<BF16>((uint16_t)(wlw[e >> 1] >> (16 * (e & 1)))));
      const float v = rnd16<BF16>(rnd16<BF16>(b[e] * inv) * raw16_to_float<BF16>((uint16_t)(whw[e >> 1] >> (16 * (e & 1)))));
      ol[e >> 1] |= (uint32_t)float_to_raw16<BF16>(u * c[e] - v * s[e]) << (16 * (e & 1));
      oh[e >> 1] |= (uint32_t)float_to_raw16<BF16>(u * s[e] + v * c[e]) << (16 * (e & 1));
    }
    lo = make_uint2(ol[0], ol[1]);
    hi = make_uint2(oh[0], oh[1]);
    if (in) { p[lane] = lo; p[lane + 16] = hi; }
  }
  if (in && dst) { dst[lane] = lo; dst[lane + 16] = hi; }
}

// out[t, i] = round16(silu(gate)) * up, gate = gate_up[t, i], up = gate_up[t, I + i]
template <bool BF16>
__global__ void __launch_bounds__(256) silu_mul_kernel(const uint16_t* __restrict__ gate_up, uint16_t* __restrict__ out,
                                                       int64_t T, int I) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int64_t total = T * (int64_t)I;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = idx / I;
    const int i = (int)(idx - t * I);
    const float g = raw16_to_float<BF16>(gate_up[t * 2 * I + i]);
    const float u = raw16_to_float<BF16>(gate_up[t * 2 * I + I + i]);
    const float s = rnd16<BF16>(g / (1.f + expf(-g)));
    out[idx] = float_to_raw16<BF16>(s * u);
  }
}

// The same, in pieces of E values (whole words of 4, 8 or 16 bytes), P pieces per thread under way at once; pieces are numbered
// through all rows, so that no thread idles at a row's end.  The exponential and the
// division of a call's last values are what a small call waits for, so that pieces are short where there are few of them; large calls
// are bound by memory (6 bytes per result) and take 16 bytes at a time.  bfloat16, us by pieces of 1, 2, 4, 8 values and of two times 8:
// 17 x 3072 1.53, 1.23, 1.36, 1.59, 2.17; 300 x 3072 4.91, 2.86, 2.76, 3.31, 3.55; 1000 x 4096 15.5, 10.1, 7.85, 7.10, 7.82; 4000 x 12288
// 152, 101, 73.6, 61.7, 58.7 (5.0 TB/s).
template <int E> struct Piece;
template <> struct Piece<2> { using type = uint32_t; };
template <> struct Piece<4> { using type = uint2; };
template <> struct Piece<8> { using type = uint4; };
template <bool BF16, int E, int P>
__global__ void __launch_bounds__(256) silu_mul_vec_kernel(const uint16_t* __restrict__ gate_up, uint16_t* __restrict__ out, uint32_t pieces, uint32_t per_row) {
  using W = typename Piece<E>::type;
  union Values { W w; uint16_t v[E]; };
  grid_launch_dependents();
  grid_dependency_wait();
  const uint32_t first = blockIdx.x * (256u * P) + threadIdx.x;
  Values g[P], u[P];
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const uint32_t at = first + 256u * j;
    if (at < pieces) {
      const W* row = reinterpret_cast<const W*>(gate_up) + at + (size_t)(at / per_row) * per_row;
      g[j].w = row[0];
      u[j].w = row[per_row];
    }
  }
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const uint32_t at = first + 256u * j;
    if (at >= pieces) break;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float a = raw16_to_float<BF16>(g[j].v[e]);
      g[j].v[e] = float_to_raw16<BF16>(rnd16<BF16>(a / (1.f + expf(-a))) * raw16_to_float<BF16>(u[j].v[e]));
    }
    reinterpret_cast<W*>(out)[at] = g[j].w;
  }
}

}  // namespace nqb200

using namespace nqb200;

extern "C" int nqb200_add_rmsnorm(const void* x, const void* residual, const void* weight, void* out, void* residual_out,
                                  int64_t T, int64_t H, float eps, int dtype, void* stream) {
  if (T < 0 || H <= 0 || H > 65536) return NQB200_ERR_BAD_SHAPE;
  if (dtype != NQB200_F16 && dtype != NQB200_BF16) return NQB200_ERR_BAD_DTYPE;
  if (T == 0) return NQB200_OK;
  if (!x || !weight || !out) return NQB200_ERR_NULL_POINTER;
  cudaStream_t st = (cudaStream_t)stream;
  // whole 16-byte pieces, at most three per thread: ragged rows go element by element
  if (H % 8 == 0 && H <= 3 * 512 * 8 && aligned16(x) && aligned16(weight) && aligned16(out) && aligned16(residual) && aligned16(residual_out)) {
    const int n8 = (int)H / 8, threads = n8 >= 512 ? 512 : (n8 + 31) / 32 * 32, pieces = (n8 + threads - 1) / threads;
#define NQB200_NORM(P)                                                                                                              \
  return launch_overlapped(dtype == NQB200_BF16 ? add_rmsnorm_vec_kernel<true, P> : add_rmsnorm_vec_kernel<false, P>, dim3((unsigned)T), \
                           dim3((unsigned)threads), 0, st, (const uint16_t*)x, (const uint16_t*)residual, (const uint16_t*)weight,    \
                           (uint16_t*)out, (uint16_t*)residual_out, (int)H, eps)
    if (pieces == 1) NQB200_NORM(1);
    if (pieces == 2) NQB200_NORM(2);
    NQB200_NORM(3);
#undef NQB200_NORM
  }
  const size_t smem = (size_t)H * sizeof(float);
  return launch_overlapped(dtype == NQB200_BF16 ? add_rmsnorm_kernel<true> : add_rmsnorm_kernel<false>, dim3((unsigned)T), dim3(256), smem, st,
                           (const uint16_t*)x, (const uint16_t*)residual, (const uint16_t*)weight, (uint16_t*)out,
                           (uint16_t*)residual_out, (int)H, eps);
}

static int qknorm_rope_launch(void* qkv, const void* q_weight, const void* k_weight, const float* cos_sin,
                              const int64_t* positions, const int64_t* slots, void* k_cache, void* v_cache, int64_t T,
                              int64_t num_q_heads, int64_t num_kv_heads, int64_t head_dim, int64_t row_stride, float eps,
                              int dtype, void* stream) {
  if (T < 0 || num_q_heads <= 0 || num_kv_heads <= 0 || head_dim != 128) return NQB200_ERR_BAD_SHAPE;
  if (dtype != NQB200_F16 && dtype != NQB200_BF16) return NQB200_ERR_BAD_DTYPE;
  if (T == 0) return NQB200_OK;
  if (!qkv || !q_weight || !k_weight || !cos_sin || !positions) return NQB200_ERR_NULL_POINTER;
  if (slots && (!k_cache || !v_cache)) return NQB200_ERR_NULL_POINTER;
  const int64_t heads = T * (num_q_heads + num_kv_heads + (slots ? num_kv_heads : 0));
  cudaStream_t st = (cudaStream_t)stream;
  // below about 4096 heads a lane's eight elements take longer than the traffic they save: 1 token of 32 + 8 + 8 heads 1.58 us with
  // a warp per head, 1.71 with half of one; 100 tokens 2.39 and 2.30, of 16 + 8 + 8 2.09 and 2.09; 1000 tokens 10.1 and 8.0
  const auto on8 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7u) == 0; };
  const bool vec = on8(qkv) && row_stride % 4 == 0 && on8(q_weight) && on8(k_weight) && aligned16(cos_sin) && on8(k_cache) && on8(v_cache) &&
                   heads <= INT32_MAX - 16 && heads >= 4096;
  const auto kernel = vec ? (dtype == NQB200_BF16 ? qknorm_rope_vec_kernel<true> : qknorm_rope_vec_kernel<false>)
                          : (dtype == NQB200_BF16 ? qknorm_rope_kernel<true> : qknorm_rope_kernel<false>);
  const int64_t per_block = vec ? 16 : 8;
  return launch_overlapped(kernel, dim3((unsigned)((heads + per_block - 1) / per_block)), dim3(256), 0, st,
                           (uint16_t*)qkv, (const uint16_t*)q_weight, (const uint16_t*)k_weight, cos_sin, positions, (int)T,
                           (int)num_q_heads, (int)num_kv_heads, (int)row_stride, eps, slots, (uint16_t*)k_cache, (uint16_t*)v_cache);
}

extern "C" int nqb200_qknorm_rope(void* qkv, const void* q_weight, const void* k_weight, const float* cos_sin,
                                  const int64_t* positions, int64_t T, int64_t num_q_heads, int64_t num_kv_heads,
                                  int64_t head_dim, int64_t row_stride, float eps, int dtype, void* stream) {
  return qknorm_rope_launch(qkv, q_weight, k_weight, cos_sin, positions, nullptr, nullptr, nullptr, T, num_q_heads, num_kv_heads,
                            head_dim, row_stride, eps, dtype, stream);
}

extern "C" int nqb200_qknorm_rope_kv(void* qkv, const void* q_weight, const void* k_weight, const float* cos_sin,
                                     const int64_t* positions, const int64_t* slots, void* k_cache, void* v_cache, int64_t T,
                                     int64_t num_q_heads, int64_t num_kv_heads, int64_t head_dim, int64_t row_stride, float eps,
                                     int dtype, void* stream) {
  if (!slots) return NQB200_ERR_NULL_POINTER;
  return qknorm_rope_launch(qkv, q_weight, k_weight, cos_sin, positions, slots, k_cache, v_cache, T, num_q_heads, num_kv_heads,
                            head_dim, row_stride, eps, dtype, stream);
}

extern "C" int nqb200_silu_mul(const void* gate_up, void* out, int64_t T, int64_t I, int dtype, void* stream) {
  if (T < 0 || I <= 0 || I > INT32_MAX) return NQB200_ERR_BAD_SHAPE;
  if (dtype != NQB200_F16 && dtype != NQB200_BF16) return NQB200_ERR_BAD_DTYPE;
  if (T == 0) return NQB200_OK;
  if (!gate_up || !out) return NQB200_ERR_NULL_POINTER;
  // where the piece grows: the times at the kernel cross between 0.3 and 0.4, 1.3 and 3, 8 and 16 million values
  const auto whole = [&](int e) {
    return I % e == 0 && ((reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(out)) & (2 * e - 1)) == 0 && T <= INT32_MAX / (I / e);
  };
#define NQB200_SILU(E, P)                                                                                                             \
  return launch_overlapped(dtype == NQB200_BF16 ? silu_mul_vec_kernel<true, E, P> : silu_mul_vec_kernel<false, E, P>,                    \
                           dim3((unsigned)((T * (I / E) + 256 * P - 1) / (256 * P))), dim3(256), 0, (cudaStream_t)stream,                \
                           (const uint16_t*)gate_up, (uint16_t*)out, (uint32_t)(T * (I / E)), (uint32_t)(I / E))
  if (whole(8) && T >= 12000000 / I) NQB200_SILU(8, 2);
  if (whole(8) && T >= 2400000 / I) NQB200_SILU(8, 1);
  if (whole(4) && T >= 320000 / I) NQB200_SILU(4, 1);
  if (whole(2)) NQB200_SILU(2, 1);
#undef NQB200_SILU
  const int64_t total = T * I;
  const int64_t want = (total + 255) / 256;
  const unsigned blocks = (unsigned)(want < (int64_t)kNumSMs * 16 ? want : (int64_t)kNumSMs * 16);
  cudaStream_t st = (cudaStream_t)stream;
  return launch_overlapped(dtype == NQB200_BF16 ? silu_mul_kernel<true> : silu_mul_kernel<false>, dim3(blocks), dim3(256), 0, st,
                           (const uint16_t*)gate_up, (uint16_t*)out, T, (int)I);
}

// Chunk-masked attention of prompts on the 5th-generation tensor cores (head sizes 64 and 128, cache pages of a
// multiple of 128 tokens); what it computes is stated at nqb200_chunk_attention.
//
// One CTA takes 256 queries of one head as two tiles of 128 and walks over key tiles of 128, each in two halves of 64.
//   warp 0        TMA: Q once, then two-stage rings of K tiles and of V tiles, straight from the pages.
//   warps 1, 2    one lane of each issues tcgen05.mma for a query tile: S = Q K^T of a half (both operands in shared memory)
//                 and O += P V (P in tensor memory, V in shared memory as it lies there: the operand's rows are keys).
//   warps 4-19    softmax: four warps for each half of each query tile, a thread per row and half.
// Tensor memory holds S of both tiles (two halves of 64 columns each) and O of both; P overwrites the first half of its own S.
// So four chains S -> weights -> O += P V -> next S run beside each other, and a scheduler has a warp of each.  What bounds it:
// per 256 x 128 scores the tensor pipe needs 2560 cycles (S 48 per MMA of N = 64, which shared memory sets, O 64), the
// exponentials 2048, and about 4500 pass, because the chains meet at the pipes.  8192 tokens of 32 heads of 128, us, in turns against
// whole tiles with one softmax thread per row and one polling issuer: chunks of 4096 645 -> 400, one chunk 1093 -> 673, scores beyond
// the cap 2673 -> 1590, no cap 932 -> 589, sigmoid weights 963 -> 624.  An own warp for S beside the two for O, polling instead of
// suspended softmax waits and query tiles started apart gained nothing.
//
// The weights are 2^(score - m).  m is the largest score of the tile that a row begins in, or the sink, and follows the largest score
// when it falls behind by more than kLag in log2 units; O and the sums are then rescaled: no weight is above 2^kLag, whatever the
// scores do, and after a row's first tiles it hardly ever happens.  (With 7 the error to float64 is for every kind of scores measured at most
// what whole tiles with a lag of 8 had; smaller lags take off up to 5 % more of it and cost 2 to 3 % each where scores spread by 6 log2 units.)
// A half finds out by itself that its scores ask for no move, from the largest magnitude, which the choice below needs as well; that
// the other half has not moved it learns from what that one hands on, in the order of the products, and does not wait for the other's
// scores: 955 -> 671 us with a cap of 120, against halves that compare their maxima in every tile.  Of the 673 the hand-over takes 65.
// (A reference that never moves, which a cap of 50 allows, needs neither, but its weights reach 2^100 and more values overflow, and the
// largest weight of a row is rounded where it could be a power of two: up to 11 % more error.)  The cap is monotonic, so the
// maximum is taken over raw scores.
// For scores well inside the cap tanh is its Taylor series, which costs fused multiply-adds on register pairs only: three terms
// up to a tenth of the cap, where what they leave out (0.054 y^6) is below float's rounding, five terms beyond; up to
// twice the cap it is the seventh convergent of Lambert's continued fraction (one reciprocal more per score); a warp
// whose half tile has a larger score, or needs a mask, takes the general path, of which there is one with and one without a cap (as one,
// the cap's exponential and reciprocal are computed either way: 128 tokens without a cap 9.7 us instead of 8.3, 600 19.4 instead of 17.7).
//
// The sum that a row is divided by takes the weights in float32, before the product's rounding to bf16.
//
// Sigmoid weights (nqb200_attention.sigmoid) need no maximum and no sum: a weight is 1 / (1 + 2^x), two weights share one
// reciprocal, 1 / a = b / (a b), with x clamped to 60 so that a b stays finite (weights below 2^-60 are 2^-60).
//
// Every wait is bounded; on expiry NQB200_ERR_WAIT_TIMEOUT goes to the status word, all roles drain and tensor memory is
// released.
#include "mixers.cuh"
#include "tma_utils.cuh"
#include "umma_utils.cuh"
#include <type_traits>

namespace nqb200 {
namespace att {

constexpr int kTile = 128, kThreads = 640;
constexpr uint32_t kColS = 0, kColO = 256, kTmemCols = 512;
constexpr float kLog2e = 1.4426950408889634f, kLag = 7.f, kSeriesRange = 0.4f, kShortRange = 0.1f, kFractionRange = 2.f;

struct Params {
  nqb200_batch bt;
  bf16* out; int64_t out_stride;
  int heads, kv_heads, chunk;
  float scale, softcap, out_scale;
  // a raw score s in log2 units: top tanh(ysc s), or s ysc_top without a cap; and tanh's series in s, with the powers of ysc and top in them
  float ysc, top, ysc_top, c3, c5, c7, c9;
  int folded;          // none of the coefficients leaves the range of normal numbers
  const float* sink;
  const float* temp; const float* bias;      // of sigmoid weights
  int* status;
};

// The issuers' waits poll: a suspended warp is woken late, and the tensor pipe has nothing queued meanwhile.
__device__ __forceinline__ bool poll_bar_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  const uint32_t b = smem_u32(bar);
  unsigned long long t0 = 0;
  for (uint32_t polls = 0;;) {
    if (__all_sync(0xFFFFFFFFu, mbar_test_wait(b, parity))) return true;
    if ((++polls & 255u) == 0) {
      const unsigned long long t = global_timer_ns();
      if (!t0) t0 = t;
      const bool late = t - t0 > kWaitLimitNs;
      if (late) {
        *abort_flag = 1;
        if (status) atomicExch(status, NQB200_ERR_WAIT_TIMEOUT);
      }
      if (__any_sync(0xFFFFFFFFu, late || *abort_flag != 0)) return false;
    }
  }
}

// D[tmem] (+)= A[smem descriptor] * B[smem descriptor]; the descriptors' high halves are the same.
__device__ __forceinline__ void umma_ss_lohi(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n .reg .b64 a, b;\n setp.ne.b32 p, %5, 0;\n mov.b64 a, {%1, %3};\n mov.b64 b, {%2, %3};\n"
               " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n}"
               ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate) : "memory");
}
// Operand whose rows in shared memory run along k (the contraction), 64 columns = 128 swizzled bytes a row: 8-row groups
// 1024 bytes apart along k, further blocks of 64 columns `block_bytes` apart.
__device__ __forceinline__ uint64_t smem_desc_mn(uint32_t addr, uint32_t block_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(block_bytes >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
               "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
                 "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                 "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
               "%24,%25,%26,%27,%28,%29,%30,%31,%32};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
                 "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
                 "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
// pairs of floats in one 64-bit register
__device__ __forceinline__ uint64_t pair2(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void unpair2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) { float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ float max3_abs(float a, float b, float c) { float r; asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ float ex2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

template <int D, int V, bool SIGMOID>
__global__ void __launch_bounds__(kThreads, 1)
attention_umma_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                      const Params p) {
  constexpr uint32_t kQBytes = kTile * D * 2, kKBytes = kTile * D * 2, kVBytes = kTile * V * 2, kBox = kTile * 128;
  constexpr uint32_t kOffK = 2 * kQBytes, kOffV = kOffK + 2 * kKBytes;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_q, bar_kfull[2], bar_kfree[2], bar_vfull[2], bar_vfree[2], bar_s[2][2], bar_p[2][2], bar_pv[2][2], bar_o[2], bar_x[2][4], bar_m[2][2][4], bar_drain;
  __shared__ float s_x[2][2][2][kTile], s_m[2][2][kTile];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort_i;
  volatile int* s_abort = &s_abort_i;
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = warp_index(), lane = threadIdx.x & 31;

  grid_launch_dependents();
  grid_dependency_wait();
  const int b = blockIdx.z, h = blockIdx.y, kvh = h / (p.heads / p.kv_heads);
  const int t0 = p.bt.cu[b], n = p.bt.cu[b + 1] - t0, pos0 = p.bt.pos0[b];
  const int i0 = (int)(gridDim.x - 1 - blockIdx.x) * 2 * kTile;     // long rows first
  if (i0 >= n) return;
  const int first = pos0 + i0, lo_first = p.chunk > 0 ? first / p.chunk * p.chunk : 0, kstart = lo_first / kTile * kTile;
  int nq[2];
#pragma unroll
  for (int q = 0; q < 2; ++q)
    nq[q] = __shfl_sync(0xFFFFFFFFu, i0 + q * kTile < n ? (pos0 + min(i0 + (q + 1) * kTile, n) - 1 - kstart) / kTile + 1 : 0, 0);
  const int nmax = max(nq[0], nq[1]);

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar_q), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_kfull[s]), 1); mbar_init(smem_u32(&bar_kfree[s]), 2);
      mbar_init(smem_u32(&bar_vfull[s]), 1); mbar_init(smem_u32(&bar_vfree[s]), 2);
      mbar_init(smem_u32(&bar_s[s][0]), 1); mbar_init(smem_u32(&bar_s[s][1]), 1); mbar_init(smem_u32(&bar_p[s][0]), 4); mbar_init(smem_u32(&bar_p[s][1]), 4);
      mbar_init(smem_u32(&bar_pv[s][0]), 1); mbar_init(smem_u32(&bar_pv[s][1]), 1); mbar_init(smem_u32(&bar_o[s]), 1);
    }
    for (int s = 0; s < 8; ++s) {
      mbar_init(smem_u32(&bar_x[s >> 2][s & 3]), 2);
      mbar_init(smem_u32(&bar_m[s >> 2][0][s & 3]), 32); mbar_init(smem_u32(&bar_m[s >> 2][1][s & 3]), 32);
    }
    mbar_init(smem_u32(&bar_drain), 2);
    s_abort_i = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(smem_u32(&s_tmem), kTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;

  // of the 96 registers a thread that 640 threads can have: 32 x 128 + 112 x 512 = 96 x 640
  if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;"); else asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA
    const bool el = elect_one();
    const int tiles_q = nq[1] > 0 ? 2 : 1;
    if (el) {
      prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v);
      mbar_expect_tx(smem_u32(&bar_q), (uint32_t)tiles_q * kQBytes);
      for (int q = 0; q < tiles_q; ++q)
        for (int c = 0; c < D / 64; ++c) tma_load_2d(smem + q * kQBytes + c * kBox, &tm_q, h * D + c * 64, t0 + i0 + q * kTile, smem_u32(&bar_q));
    }
    __syncwarp();
    int issued = 0;
    for (int j = 0; j < nmax; ++j, ++issued) {
      const int s = j & 1, pos = kstart + j * kTile;
      if (j >= 2 && !wait_bar_warp(&bar_kfree[s], ((j >> 1) - 1) & 1, s_abort, p.status)) break;
      const int row = __shfl_sync(0xFFFFFFFFu, (int)kv_row(p.bt, b, pos), 0);    // the tile lies in one page
      if (el) {
        mbar_expect_tx(smem_u32(&bar_kfull[s]), kKBytes);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_load_2d(smem + kOffK + s * kKBytes + c * kBox, &tm_k, kvh * D + c * 64, row, smem_u32(&bar_kfull[s]));
      }
      if (j >= 2 && !wait_bar_warp(&bar_vfree[s], ((j >> 1) - 1) & 1, s_abort, p.status)) {
        mbar_wait(smem_u32(&bar_kfull[s]), (j >> 1) & 1);
        break;
      }
      if (el) {
        mbar_expect_tx(smem_u32(&bar_vfull[s]), kVBytes);
#pragma unroll
        for (int c = 0; c < V / 64; ++c) tma_load_2d(smem + kOffV + s * kVBytes + c * kBox, &tm_v, kvh * V + c * 64, row, smem_u32(&bar_vfull[s]));
      }
    }
    // do not leave while a copy may still be landing
    mbar_wait(smem_u32(&bar_q), 0);
    for (int j = issued > 2 ? issued - 2 : 0; j < issued; ++j) {
      mbar_wait(smem_u32(&bar_kfull[j & 1]), (j >> 1) & 1);
      mbar_wait(smem_u32(&bar_vfull[j & 1]), (j >> 1) & 1);
    }
  } else if (warp < 3) {
    // ------------------------------------------------------------------ MMA
    // A warp per query tile, of which one lane issues (elect_one).  A half's S may overwrite its weights once their product has
    // completed.  A ring stage is handed back by both warps, by its only user twice.
    const int q = warp - 1;
    const bool el = elect_one();
    const uint32_t idesc_s = umma_idesc(1, 128, kTile / 2);
    const uint32_t idesc_o = umma_idesc(1, 128, V) | (1u << 16);   // B's rows run along k
    const uint64_t dq = umma_smem_desc_sw128(smem + q * kQBytes), dk = umma_smem_desc_sw128(smem + kOffK), dv = smem_desc_mn(smem + kOffV, kBox);
    const uint32_t k_hi = (uint32_t)(dq >> 32), v_hi = (uint32_t)(dv >> 32), q_lo = (uint32_t)dq, k_lo = (uint32_t)dk, v_lo = (uint32_t)dv;
    const uint32_t tS = tmem + kColS + q * 128, tO = tmem + kColO + q * 128;
    const int mine = nq[q], others = nq[q ^ 1];
    bool ok = mine > 0 && poll_bar_warp(&bar_q, 0, s_abort, p.status);
    for (int j = 0; ok && j <= mine; ++j) {
      const int i = j - 1, s = j & 1, so = s ^ 1;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (j > 0) {      // O += P V of the tile before
          if (half == 0) ok = poll_bar_warp(&bar_vfull[so], (i >> 1) & 1, s_abort, p.status);
          ok = ok && poll_bar_warp(&bar_p[q][half], so, s_abort, p.status);
          if (!ok) break;
          tc_fence_after();
          if (el) {
#pragma unroll
            for (int ks = 0; ks < kTile / 32; ++ks)
              umma_ts_lohi(tO, tS + half * 64 + ks * 8, v_lo + so * (kVBytes >> 4) + half * (8192 >> 4) + ks * (2048 >> 4), v_hi, idesc_o,
                           (i > 0 || half > 0 || ks > 0) ? 1u : 0u);
            umma_commit(smem_u32(j == mine && half == 1 ? &bar_o[q] : &bar_pv[q][half]));
            if (half == 1) {
              umma_commit(smem_u32(&bar_vfree[so]));
              if (i >= others) umma_commit(smem_u32(&bar_vfree[so]));
            }
          }
        }
        if (j < mine) {
          if (j > 0) ok = poll_bar_warp(&bar_pv[q][half], so, s_abort, p.status);   // the weights have been read: their place takes the next scores
          if (half == 0) ok = ok && poll_bar_warp(&bar_kfull[s], (j >> 1) & 1, s_abort, p.status);
          if (!ok) break;
          tc_fence_after();
          if (el) {
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks)
              umma_ss_lohi(tS + half * 64, q_lo + (ks >> 2) * (kBox >> 4) + (ks & 3) * 2,
                           k_lo + s * (kKBytes >> 4) + half * (8192 >> 4) + (ks >> 2) * (kBox >> 4) + (ks & 3) * 2, k_hi, idesc_s, ks > 0 ? 1u : 0u);
            umma_commit(smem_u32(&bar_s[q][half]));
            if (half == 1) {
              umma_commit(smem_u32(&bar_kfree[s]));
              if (j >= others) umma_commit(smem_u32(&bar_kfree[s]));
            }
          }
        }
      }
    }
    // everything issued has completed before tensor memory may be released
    if (el) umma_commit(smem_u32(&bar_drain));
    mbar_wait(smem_u32(&bar_drain), 0);
  } else if (warp >= 4) {
    // -------------------------------------------------------------- softmax
    const int q = (warp - 4) >> 3, half = ((warp - 4) >> 2) & 1, quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lanes = (uint32_t)(32 * quarter) << 16, tS = tmem + lanes + kColS + q * 128 + half * 64, tO = tmem + lanes + kColO + q * 128;
    const int i = i0 + q * kTile + row, pos = pos0 + i, wfirst = pos - lane, wlast = wfirst + 31;
    const int lo = p.chunk > 0 ? pos / p.chunk * p.chunk : 0, lo_last = p.chunk > 0 ? wlast / p.chunk * p.chunk : 0;
    const bool capped = p.softcap > 0.f;
    auto score = [&](float s) {   // in log2 units
      const float y = s * p.ysc;
      return p.top * (capped ? tanh_fast(y) : y);
    };
    auto done = [&]() {           // this half of the weights is in tensor memory
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_p[q][half]));
    };
    int exchanges = 0;
    auto exchange = [&](float mine, float& other) {   // with the thread that has the row's other half
      const int x = exchanges & 1;
      s_x[q][half][x][row] = mine;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_x[q][quarter]));
      const bool got = wait_bar_warp(&bar_x[q][quarter], x, s_abort, p.status);
      tc_fence_after();
      other = s_x[q][half ^ 1][x][row];
      ++exchanges;
      return got;
    };
    const float sg_scale = -p.scale * (p.temp ? p.temp[h] : 1.f) * kLog2e, sg_shift = p.bias ? -p.bias[h] * kLog2e : 0.f;
    const float sink = p.sink ? p.sink[h] * kLog2e : -INFINITY;
    float m = sink;
    uint64_t lsum = pair2(0.f, 0.f);
    // A row's reference goes from half to half in the order of their products: 0 and 1 of the first tile, 0 and 1 of the next, and so on,
    // except in the tiles where rows begin (the first, and the one of the last row's chunk), where both agree on it.
    const int second = (lo_last - kstart) / kTile;
    auto pass = [&](float mine) {    // (every lane arrives: a branch for one of them cost 2 % of the kernel)
      s_m[q][half][row] = mine;
      mbar_arrive(smem_u32(&bar_m[q][half][quarter]));
    };
    auto take = [&](int n) {       // what the other half passed on, its n-th
      if (!wait_bar_warp(&bar_m[q][half ^ 1][quarter], (n - 1) & 1, s_abort, p.status)) return false;
      const float got = s_m[q][half ^ 1][row];
      if (__any_sync(0xFFFFFFFFu, got != m)) {
        const float f = got != m ? ex2(m - got) : 1.f;
        lsum = mul2(lsum, pair2(f, f));
        m = got;
      }
      return true;
    };
    auto catch_up = [&](int j, bool joint) {      // with what came before this half of tile j
      const int n = j - 1 - (second > 0 && j > second ? 1 : 0);      // tiles before it in which it was passed on
      if (half == 1) return joint || take(n + 1);
      return j == 0 || j == 1 || j - 1 == second || take(n);
    };
    // top tanh(y) by its series, TERMS powers of y^2 beyond the first (0: no cap)
    auto weights = [&](auto terms, const uint32_t (&r)[2][32], uint64_t nm2) {
      constexpr int TERMS = decltype(terms)::value;
      const uint64_t k1 = pair2(p.ysc_top, p.ysc_top), k3 = pair2(p.c3, p.c3), k5 = pair2(p.c5, p.c5), k7 = pair2(p.c7, p.c7), k9 = pair2(p.c9, p.c9);
      uint64_t ls[2] = {lsum, 0};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t w[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const uint64_t t = pair2(__uint_as_float(r[c][2 * e]), __uint_as_float(r[c][2 * e + 1]));
          uint64_t f = k1;
          if (TERMS) {
            const uint64_t t2 = mul2(t, t);
            f = TERMS == 4 ? fma2(fma2(k9, t2, k7), t2, k5) : k5;
            f = fma2(fma2(f, t2, k3), t2, k1);
          }
          float x0, x1;
          unpair2(fma2(t, f, nm2), x0, x1);
          x0 = ex2(x0);
          x1 = ex2(x1);
          w[e] = pack_bf16(x0, x1);
          ls[e & 1] = add2(ls[e & 1], pair2(x0, x1));
        }
        tmem_st16(tS + c * 16, w);
      }
      lsum = add2(ls[0], ls[1]);
    };
    bool ok = true;
    for (int j = 0; j < nq[q]; ++j) {
      // where rows of this warp begin both halves agree on a reference, the largest score of the two
      const bool joint = j == 0 || j == second;
      ok = (SIGMOID || catch_up(j, joint)) && wait_bar_warp(&bar_s[q][half], j & 1, s_abort, p.status);
      if (!ok) break;
      tc_fence_after();
      const int key0 = kstart + j * kTile + half * 64;
      const bool masked = key0 + 63 > wfirst || key0 < lo_last;     // for any row of the warp
      uint32_t r[2][32];     // the row's scores, all of this half
#pragma unroll
      for (int c = 0; c < 2; ++c) tmem_ld32(tS + c * 32, r[c]);
      tc_wait_ld();
      if constexpr (SIGMOID) {
        const uint64_t sg_scale2 = pair2(sg_scale, sg_scale), sg_shift2 = pair2(sg_shift, sg_shift), one2 = pair2(1.f, 1.f);
        auto sigmoid2 = [&](uint32_t s0, uint32_t s1, float& w0, float& w1) {
          float x0, x1;
          unpair2(fma2(pair2(__uint_as_float(s0), __uint_as_float(s1)), sg_scale2, sg_shift2), x0, x1);
          float d0, d1;
          unpair2(add2(pair2(ex2(fminf(x0, 60.f)), ex2(fminf(x1, 60.f))), one2), d0, d1);
          const float r = rcp_fast(d0 * d1);
          w0 = r * d1;
          w1 = r * d0;
        };
        if (!masked) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t w[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              float x0, x1;
              sigmoid2(r[c][2 * e], r[c][2 * e + 1], x0, x1);
              w[e] = pack_bf16(x0, x1);
            }
            tmem_st16(tS + c * 16, w);
          }
        } else {
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t v[16], w[8];
            tmem_ld_32x32b_x16(tS + c * 16, v);
            tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int key = key0 + c * 16 + 2 * e;
              float x0, x1;
              sigmoid2(v[2 * e], v[2 * e + 1], x0, x1);
              w[e] = pack_bf16(key <= pos && key >= lo ? x0 : 0.f, key + 1 <= pos && key + 1 >= lo ? x1 : 0.f);
            }
            tmem_st8(tS + c * 8, w);      // lies behind what has been read of S
          }
        }
        done();
        continue;
      }
      float ab = 0.f, mx = -INFINITY;     // the largest magnitude and, where it is asked for, the largest score
      if (!masked) {
        float hi[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int e = 0; e < 32; e += 2) hi[(e >> 1) & 3] = max3_abs(hi[(e >> 1) & 3], __uint_as_float(r[c][e]), __uint_as_float(r[c][e + 1]));
        ab = fmaxf(fmaxf(hi[0], hi[1]), fmaxf(hi[2], hi[3]));
      }
      const float lag = m + kLag;
      // (|score| <= |y top|: at most this, so that most tiles need neither the cap nor the sign)
      if (joint || masked || !__all_sync(0xFFFFFFFFu, ab * p.ysc_top <= lag)) {
        if (!masked) {
          float hi[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int e = 0; e < 32; e += 2) hi[(e >> 1) & 3] = max3(hi[(e >> 1) & 3], __uint_as_float(r[c][e]), __uint_as_float(r[c][e + 1]));
          mx = fmaxf(fmaxf(hi[0], hi[1]), fmaxf(hi[2], hi[3]));
        } else {
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              const int key = key0 + c * 32 + e;
              mx = (key <= pos && key >= lo) ? fmaxf(mx, __uint_as_float(r[c][e])) : mx;
            }
        }
        if (joint) {
          float mo;
          if (!(ok = exchange(mx, mo))) break;
          mx = fmaxf(mx, mo);
        }
        mx = mx == -INFINITY ? mx : score(mx);
      }
      const bool move = mx > lag;      // also from -inf
      if (!joint) pass(move ? mx : m);
      if (j == 0) {
        m = fmaxf(m, mx);
        lsum = pair2(p.sink && half == 0 ? ex2(sink - m) : 0.f, 0.f);
      } else if (__any_sync(0xFFFFFFFFu, move)) {
        const float f = move ? ex2(m - mx) : 1.f;
        lsum = mul2(lsum, pair2(f, f));
        m = move ? mx : m;
        if (half == 0 || !joint) {
          // O has the products of all halves before this one, and no other until this one's weights are reported
          if (!(ok = wait_bar_warp(&bar_pv[q][half ^ 1], (j - 1 + half) & 1, s_abort, p.status))) break;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < V / 32; ++c) {
            tmem_ld32(tO + c * 32, r[0]);
            tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 32; ++e) r[0][e] = __float_as_uint(__uint_as_float(r[0][e]) * f);
            tmem_st32(tO + c * 32, r[0]);
          }
          tc_wait_st();
          tmem_ld32(tS, r[0]);      // the scores again
          tc_wait_ld();
        }
      }
      const float mu = m == -INFINITY ? 0.f : m;
      const uint64_t ysc2 = pair2(p.ysc, p.ysc), nm2 = pair2(-mu, -mu), k1 = pair2(p.top, p.top);
      auto within = [&](float y) { return __all_sync(0xFFFFFFFFu, ab * p.ysc <= y); };      // for every score of the warp's
      const int range = masked ? 2 : !capped || (p.folded && within(kSeriesRange)) ? 0 : within(kFractionRange) ? 1 : 2;
      if (range == 1) {
        // tanh y = y (10395 + 1260 y^2 + 21 y^4) / (10395 + 4725 y^2 + 210 y^4 + y^6)
        const uint64_t n0 = pair2(10395.f, 10395.f), n1 = pair2(1260.f, 1260.f), n2 = pair2(21.f, 21.f), d1 = pair2(4725.f, 4725.f), d2 = pair2(210.f, 210.f);
        uint64_t ls[2] = {lsum, 0};
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t w[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const uint64_t y = mul2(pair2(__uint_as_float(r[c][2 * e]), __uint_as_float(r[c][2 * e + 1])), ysc2), y2 = mul2(y, y);
            const uint64_t num = mul2(mul2(y, k1), fma2(fma2(n2, y2, n1), y2, n0)), den = fma2(fma2(add2(y2, d2), y2, d1), y2, n0);
            float a, c2, x0, x1;
            unpair2(den, a, c2);
            unpair2(fma2(num, pair2(rcp_fast(a), rcp_fast(c2)), nm2), x0, x1);
            x0 = ex2(x0);
            x1 = ex2(x1);
            w[e] = pack_bf16(x0, x1);
            ls[e & 1] = add2(ls[e & 1], pair2(x0, x1));
          }
          tmem_st16(tS + c * 16, w);
        }
        lsum = add2(ls[0], ls[1]);
      } else if (range == 0) {
        if (!capped) weights(std::integral_constant<int, 0>(), r, nm2);
        else if (within(kShortRange)) weights(std::integral_constant<int, 2>(), r, nm2);
        else weights(std::integral_constant<int, 4>(), r, nm2);
      } else {
        // from tensor memory again, a piece at a time: compact code for the few tiles at the edges
        auto general = [&](auto cap) {
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t v[16], w[8];
            tmem_ld_32x32b_x16(tS + c * 16, v);
            tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              float x[2];
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int key = key0 + c * 16 + 2 * e + u;
                const float s = __uint_as_float(v[2 * e + u]) * p.ysc;
                x[u] = (key <= pos && key >= lo) ? ex2(p.top * (decltype(cap)::value ? tanh_fast(s) : s) - mu) : 0.f;
              }
              w[e] = pack_bf16(x[0], x[1]);
              lsum = add2(lsum, pair2(x[0], x[1]));
            }
            tmem_st8(tS + c * 8, w);      // lies behind what has been read of S
          }
        };
        if (capped) general(std::true_type()); else general(std::false_type());
      }
      done();
    }
    if (ok && nq[q] > 0) {
      ok = (SIGMOID || catch_up(nq[q], true)) && wait_bar_warp(&bar_o[q], 0, s_abort, p.status);
      float f = p.out_scale;
      if (ok && !SIGMOID) {
        float a, c2, other;
        unpair2(lsum, a, c2);
        const float l = a + c2;
        ok = exchange(l, other);
        f /= l + other;
      }
      if (ok) {
        tc_fence_after();
        bf16* dst = p.out + (size_t)(t0 + i) * p.out_stride + (size_t)h * V + half * (V / 2);
#pragma unroll
        for (int c = 0; c < V / 64; ++c) {
          uint32_t r[32];
          tmem_ld32(tO + half * (V / 2) + c * 32, r);
          tc_wait_ld();
          if (i < n) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              uint4 v;
              v.x = pack_bf16(__uint_as_float(r[8 * e]) * f, __uint_as_float(r[8 * e + 1]) * f);
              v.y = pack_bf16(__uint_as_float(r[8 * e + 2]) * f, __uint_as_float(r[8 * e + 3]) * f);
              v.z = pack_bf16(__uint_as_float(r[8 * e + 4]) * f, __uint_as_float(r[8 * e + 5]) * f);
              v.w = pack_bf16(__uint_as_float(r[8 * e + 6]) * f, __uint_as_float(r[8 * e + 7]) * f);
              *reinterpret_cast<uint4*>(dst + c * 32 + e * 8) = v;
            }
          }
          __syncwarp();
        }
        tc_fence_before();
      }
    }
  }
  // all roles meet here, also after a give-up, so that tensor memory is always released
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, kTmemCols); }
}

static bool encode_rows(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t row_bytes) {
  PFN_cuTensorMapEncodeTiled enc = tensor_map_encoder();
  if (!enc) return false;
  cuuint64_t dims[2] = {cols, rows}, strides[1] = {row_bytes};
  cuuint32_t box[2] = {64, (cuuint32_t)kTile}, estr[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D, int V, bool SIGMOID>
static int launch_t(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const Params& p, cudaStream_t st) {
  // at least 120 KB, whatever the sizes: one CTA per SM, because a CTA takes all of the SM's tensor memory
  const size_t need = (size_t)kTile * (2 * D + 2 * D + 2 * V) * 2 + 1024, smem = need > 120 * 1024 ? need : 120 * 1024;
  if (cudaFuncSetAttribute(attention_umma_kernel<D, V, SIGMOID>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    return NQB200_ERR_LAUNCH;
  }
  const dim3 grid((unsigned)((p.bt.max_len + 2 * kTile - 1) / (2 * kTile)), (unsigned)p.heads, (unsigned)p.bt.batch);
  return launch_overlapped(attention_umma_kernel<D, V, SIGMOID>, grid, dim3(kThreads), smem, st, q, k, v, p);
}
template <int D, int V>
static int launch(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const Params& p, bool sigmoid, cudaStream_t st) {
  return sigmoid ? launch_t<D, V, true>(q, k, v, p, st) : launch_t<D, V, false>(q, k, v, p, st);
}

}  // namespace att

// From 128 tokens and, with chunks, 512 positions a chunk: below, tiles of 128 x 256 are mostly mask.
bool attention_umma_supports(const void* q, int64_t q_stride, const void* k_cache, const void* v_cache, const void* out, int64_t out_stride,
                             int64_t cache_rows, const nqb200_attention* a, const nqb200_batch* b) {
  return (a->dim == 64 || a->dim == 128) && (a->vdim == 64 || a->vdim == 128) && b->block_size % att::kTile == 0 && cache_rows > 0 &&
         cache_rows % b->block_size == 0 && b->max_len >= att::kTile && (a->chunk <= 0 || a->chunk >= 512) && a->scale > 0.f && q_stride % 8 == 0 &&
         out_stride % 8 == 0 && aligned16(q) && aligned16(k_cache) && aligned16(v_cache) && aligned16(out);
}
int attention_umma(const void* q, int64_t q_stride, const void* k_cache, const void* v_cache, void* out, int64_t out_stride, int64_t cache_rows,
                   const nqb200_attention* a, const nqb200_batch* b, int* status, cudaStream_t st) {
  CUtensorMap tq, tk, tv;
  if (!att::encode_rows(&tq, q, b->tokens, (uint64_t)a->heads * a->dim, (uint64_t)q_stride * 2) ||
      !att::encode_rows(&tk, k_cache, cache_rows, (uint64_t)a->kv_heads * a->dim, (uint64_t)a->kv_heads * a->dim * 2) ||
      !att::encode_rows(&tv, v_cache, cache_rows, (uint64_t)a->kv_heads * a->vdim, (uint64_t)a->kv_heads * a->vdim * 2))
    return NQB200_ERR_LAUNCH;
  att::Params p = {};
  p.bt = *b; p.out = (bf16*)out; p.out_stride = out_stride; p.heads = a->heads; p.kv_heads = a->kv_heads; p.chunk = a->chunk;
  p.scale = a->scale; p.softcap = a->softcap; p.out_scale = a->out_scale; p.sink = a->sink; p.temp = a->temp; p.bias = a->bias;
  p.status = status;
  p.ysc = p.softcap > 0.f ? p.scale / p.softcap : p.scale;
  p.top = p.softcap > 0.f ? p.softcap * att::kLog2e : att::kLog2e;
  p.ysc_top = p.top * p.ysc;
  const float z = p.ysc * p.ysc;
  p.c3 = -p.ysc_top / 3.f * z; p.c5 = p.ysc_top * (2.f / 15.f) * z * z; p.c7 = -p.ysc_top * (17.f / 315.f) * z * z * z;
  p.c9 = p.ysc_top * (62.f / 2835.f) * z * z * z * z;
  p.folded = p.ysc >= 1.f / 4096.f && p.ysc <= 4096.f;
  if (a->dim == 64) return a->vdim == 64 ? att::launch<64, 64>(tq, tk, tv, p, a->sigmoid, st) : att::launch<64, 128>(tq, tk, tv, p, a->sigmoid, st);
  return a->vdim == 64 ? att::launch<128, 64>(tq, tk, tv, p, a->sigmoid, st) : att::launch<128, 128>(tq, tk, tv, p, a->sigmoid, st);
}

}  // namespace nqb200

// Linears of a decode batch or a short prompt on the 5th-generation tensor cores: W4A16 GEMM for more than 16 tokens, group
// size 128.  (Long prompts take the two-SM kernel, gemm_umma_pair.cu, except where that one's rule leaves small layers here.)
//
//   D[n, tok] (TMEM, fp32) = sum_k W[k, n] (TMEM, 16-bit) * x[tok, k] (smem)
//
// Measured in chains of calls (bf16, microseconds): 4096 x 24576 34.9 -> 25.2 at 48 tokens and 38.2 -> 34.7 at 128, 12288 x 4096
// 19.7 -> 17.1 at 48, against the form before this one (issuing threads of their own, whole tiles or an even
// split of K, the epilogue's stores two bytes wide); 1.21 in the mean over 91 calls of 17 to 400 tokens, before the prefetch at
// warp 0.  A unit takes 0.71 us at 17 tokens, 0.73 at 48 and 0.87 at 128, where memory needs 0.39.  No pipe is full (ncu,
// 48 tokens of 4096 x 24576: issue slots 53 % of active cycles, ALU 35, FMA 33, tensor 21, DRAM 25): it is the chain from weights to
// MMAs with its fill and drain.  Two blocks per SM, each half as large, reach the same rate.  Clusters that add their parts through distributed shared memory instead of a second kernel were
// slower (48 tokens, 4096 x 6144 13.1, 4096 x 24576 29.0): fewer of them fit, and the exchange took 2 us.
//
// The weights are the 128-row A operand, dequantised to their true 16-bit values (q - z) * s -- the integer difference first,
// then one multiply, which is the reference's rounding -- straight from registers into tensor memory; the tokens are the MMA's
// N, up to 128 per tile, read from shared memory as TMA wrote them.
//
// Work: a unit is one 128-k group of one output tile of 256 columns (two A blocks) x all tokens of a token tile.  CTA c, one
// per SM, takes a contiguous range of units: whole tiles, or an equal share (a tile that a boundary cuts leaves as fp32
// segments, which a second kernel adds in CTA order, so that results do not depend on timing).
//
//   warp 0        TMA of the packed weights: 128 x 128 bytes per unit.  Before the wait for the kernel ahead on the stream the
//                 first ones are brought into the L2 cache, which is all that may be done then: that kernel may have written them.
//                 Up to 64 tokens a tile the whole ring, beyond it four units: 42 calls of 17 to 128 tokens in chains take 0.98 of the
//                 time that copies into shared memory at that point took (1.006 without any, 0.994 with two, 0.986 with four).  The whole
//                 ring also beyond 64 would keep a call's first copies waiting on an idle stream: 100 tokens of 4096 -> 12288 20.0 -> 20.3 us.
//   warp 2        TMA of the activations: one box of both 64-k halves per unit.
//   warp 1        MMA issuer: per half unit and k-step two MMAs (one per A block) of M 128, N tokens, K 16.
//   warps 3-18    dequantisers, two sets of 8 taking alternate units; a slot of the A operand holds half a unit.  Scales and
//                 zero-points come from global memory, a unit ahead.
//   warps 19-26   epilogue: accumulator (two of them up to 64 tokens) -> bias -> 16 bits -> out, or the fp32 segment.
//
// Every wait is bounded; on expiry the kernel records NQB200_ERR_WAIT_TIMEOUT in the workspace status word (when a workspace
// is given), all roles drain, and tensor memory is released.
#include "umma_w4.cuh"
#include <mutex>

namespace nqb200 {
namespace pre {

constexpr int kTileN = 256, kTileT = 128, kUnitK = 128;
constexpr int kDequantWarps = 16, kEpiWarps = 8, kFirstDequant = 3, kFirstEpi = kFirstDequant + kDequantWarps;
constexpr int kThreads = (kFirstEpi + kEpiWarps) * 32;
constexpr int kWStageBytes = 16384;
constexpr int kMaxW = 8, kMaxX = 4, kMaxA = 6;
constexpr int kAhead = 4;        // units whose weights are brought into L2 ahead of the dependency wait, beyond 64 tokens a tile
constexpr int kSmemBudget = 220 * 1024;
constexpr int kTmemCols = 512;

struct Params {
  const uint16_t* sc; const uint32_t* qz;
  const void* bias; int bias_dtype; uint16_t* out;
  int M, N, G;
  int ntt, nt;                  // token tiles, tokens of each (a multiple of 16: the MMA's N)
  long long U;                  // units: column tiles x token tiles x G
  int ctas, whole;              // whole: ranges end on tile boundaries
  int sw, sx, sa, nd;           // stages of the weight ring and of the activation ring, A slots, accumulators
  float* slots;                 // [2 ctas][nt / 4][256 lanes][4 tokens] fp32: segments of cut tiles
  int* status;                  // may be null
};

// CTA c's units: [range_begin(c), range_begin(c + 1))
__host__ __device__ __forceinline__ long long range_begin(long long c, long long U, long long C, int G, int whole) {
  return whole ? c * (U / G) / C * G : c * U / C;
}
// which CTA an equal share gives unit u to
__host__ __device__ __forceinline__ int cta_of_unit(long long u, long long U, long long C) { return (int)(((u + 1) * C - 1) / U); }

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

// A ring position that advances without a division.
struct Ring {
  int i = 0, n; uint32_t ph = 0;
  __device__ explicit Ring(int n_) : n(n_) {}
  __device__ void next() { if (++i == n) { i = 0; ph ^= 1u; } }
};
// Where a role stands in its CTA's range: the tile and the group, advancing by single units.
struct Place {
  int tn, tt, g;
  __device__ Place(long long u, const Params& p) {
    const long long item = u / p.G;
    g = (int)(u - item * p.G); tn = (int)(item / p.ntt); tt = (int)(item - (long long)tn * p.ntt);
  }
  __device__ void next(const Params& p) { if (++g == p.G) { g = 0; if (++tt == p.ntt) { tt = 0; ++tn; } } }
};

// A warp's share of a tile that an accumulator holds: the 32 columns of lane quarter q of A block `blk`.  The whole tile leaves with bias in 16 bits, part of one (another CTA has the rest) as an fp32 segment.  `read` is called
// when the accumulator has been read.
template <bool BF16, typename F>
__device__ __forceinline__ void store_tile(const Params& p, int tn, int tt, bool full, int which, uint32_t src, int q, int blk, F&& read) {
  const int lane = threadIdx.x & 31, odd = lane & 1, at = 128 * blk + 32 * q + lane;
  const int n = tn * kTileN + 128 * blk + column_of_lane(32 * q + lane), tok0 = tt * p.nt;   // lanes l, l + 1 (l even): columns n, n + 1
  const float bv = (full && p.bias && n < p.N) ? bias_to_float(p.bias, p.bias_dtype, n) : 0.f;
  const int tokens = (n & ~31) < p.N ? p.M - tok0 : 0;       // whole warps: N is a multiple of 32
  uint16_t* out = p.out + (size_t)tok0 * p.N + (n & ~1);
  float4* part = reinterpret_cast<float4*>(p.slots) + (size_t)(2 * blockIdx.x + which) * p.nt * 64 + at;
  for (int c0 = 0; c0 < p.nt; c0 += 16) {
    uint32_t v[16];
    tmem_ld_32x32b_x16(src + c0, v);
    tc_wait_ld();
    if (c0 + 16 >= p.nt) read();
    if (full) {
#pragma unroll
      for (int t = 0; t < 8; t += 2) {        // two neighbours exchange: each stores two columns of eight tokens
        const uint32_t lo = (uint32_t)float_to_raw16<BF16>(__uint_as_float(v[t]) + bv) | ((uint32_t)float_to_raw16<BF16>(__uint_as_float(v[t + 1]) + bv) << 16);
        const uint32_t hi = (uint32_t)float_to_raw16<BF16>(__uint_as_float(v[t + 8]) + bv) | ((uint32_t)float_to_raw16<BF16>(__uint_as_float(v[t + 9]) + bv) << 16);
        const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
        const uint32_t left = odd ? got : lo, right = odd ? hi : got;
        const int tok = c0 + t + 8 * odd;
        uint16_t* dst = out + (size_t)tok * p.N;
        if (tok < tokens) *reinterpret_cast<uint32_t*>(dst) = __byte_perm(left, right, 0x5410);
        if (tok + 1 < tokens) *reinterpret_cast<uint32_t*>(dst + p.N) = __byte_perm(left, right, 0x7632);
      }
    } else {
#pragma unroll
      for (int c = 0; c < 16; c += 4)
        __stcg(part + (size_t)((c0 + c) / 4) * 256,
               make_float4(__uint_as_float(v[c]), __uint_as_float(v[c + 1]), __uint_as_float(v[c + 2]), __uint_as_float(v[c + 3])));
    }
  }
}

template <bool BF16>
__global__ void __launch_bounds__(kThreads, 1)
umma_prefill_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const Params p) {
  constexpr uint32_t LO = 0x000F000Fu, HI = 0x00F000F0u;
  constexpr uint32_t MAGIC = BF16 ? 0x43004300u : 0x64006400u;  // 128.0 / 1024.0 in both halves
  constexpr uint32_t SIXTEENTH = 0x2C002C00u;                   // 1/16 in both halves (fp16)

  extern __shared__ uint8_t smem_raw[];
  // wfull / wfree: a unit's weights landed / its 8 dequantiser warps have read them (a wait on a phase's parity is only right
  // for a waiter that has seen the phase before, and the two sets take alternate units: the "landed" barriers are counted per
  // unit modulo twice the ring, so that each belongs to one set).  xfull / xfree: its activations.  afull / afree: the A slot
  // of half a unit filled / the half's MMAs have completed (twice the slots, for the same reason).  dfull / dempty: accumulator.
  __shared__ __align__(8) uint64_t bar_wfull[2 * kMaxW], bar_wfree[kMaxW], bar_xfull[kMaxX], bar_xfree[kMaxX], bar_afull[kMaxA],
      bar_afree[2 * kMaxA], bar_dfull[2], bar_dempty[2], bar_drain;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort_i;

  volatile int* s_abort = &s_abort_i;
  int* status = p.status;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const long long u_begin = range_begin(blockIdx.x, p.U, p.ctas, p.G, p.whole);
  const int nunits = (int)(range_begin(blockIdx.x + 1, p.U, p.ctas, p.G, p.whole) - u_begin);
  const int x_bytes = p.nt * 256, col_a = kTmemCols - 64 * p.sa;
  const uint32_t x_base = smem_base, w_base = smem_base + p.sx * x_bytes;

  grid_launch_dependents();
  Place at(u_begin, p);
  if (warp == 0) {
    const bool el = elect_one();
    if (el) {
      for (int s = 0; s < p.sw; ++s) {
        mbar_init(smem_u32(&bar_wfull[s]), 1); mbar_init(smem_u32(&bar_wfull[p.sw + s]), 1); mbar_init(smem_u32(&bar_wfree[s]), kDequantWarps / 2);
      }
      for (int s = 0; s < p.sx; ++s) { mbar_init(smem_u32(&bar_xfull[s]), 1); mbar_init(smem_u32(&bar_xfree[s]), 1); }
      for (int s = 0; s < p.sa; ++s) {
        mbar_init(smem_u32(&bar_afull[s]), kDequantWarps / 2); mbar_init(smem_u32(&bar_afree[s]), 1); mbar_init(smem_u32(&bar_afree[p.sa + s]), 1);
      }
      for (int d = 0; d < 2; ++d) { mbar_init(smem_u32(&bar_dfull[d]), 1); mbar_init(smem_u32(&bar_dempty[d]), kEpiWarps); }
      mbar_init(smem_u32(&bar_drain), 1);
      s_abort_i = 0;
      mbar_fence_init();
      prefetch_tmap(&tm_w);
    }
    __syncwarp();
    Place ahead = at;
    for (int i = 0; i < (p.nt <= 64 ? p.sw : kAhead) && i < nunits; ++i) {
      if (el) tma_prefetch_2d(&tm_w, ahead.tn * 32, ahead.g * kUnitK);
      ahead.next(p);
    }
    __syncwarp();
  }
  grid_dependency_wait();  // the activations come from the kernel ahead on the stream
  // Tensor memory is taken after the wait: a kernel ahead that needs it has then given it back.
  if (warp == 1) { tmem_alloc(smem_u32(&s_tmem), kTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;

  if (warp == 0) {
    // ------------------------------------------------- producer of the packed weights
    const bool el = elect_one();
    Ring rw(p.sw), rl(2 * p.sw);     // rw.ph: parity of the phase after the one in which the stage was last given back
    int i = 0;
    for (; i < nunits; ++i) {
      if (i >= p.sw && !wait_bar_warp(&bar_wfree[rw.i], rw.ph ^ 1u, s_abort, status)) break;
      const uint32_t bar = smem_u32(&bar_wfull[rl.i]);
      if (el) {
        mbar_expect_tx(bar, kWStageBytes);
        tma_load_2d(w_base + rw.i * kWStageBytes, &tm_w, at.tn * 32, at.g * kUnitK, bar);
      }
      rw.next(); rl.next(); at.next(p);
    }
    // do not leave while a copy of ours may still be landing in this CTA's shared memory
    for (int j = i > p.sw ? i - p.sw : 0; j < i; ++j) mbar_wait(smem_u32(&bar_wfull[j % (2 * p.sw)]), (j / (2 * p.sw)) & 1);
  } else if (warp == 2) {
    // ------------------------------------------------- producer of the activations
    const bool el = elect_one();
    if (el) prefetch_tmap(&tm_x);
    __syncwarp();
    Ring rx(p.sx);
    int i = 0;
    for (; i < nunits; ++i) {
      if (i >= p.sx && !wait_bar_warp(&bar_xfree[rx.i], rx.ph ^ 1u, s_abort, status)) break;
      const uint32_t bar = smem_u32(&bar_xfull[rx.i]);
      if (el) {
        mbar_expect_tx(bar, (uint32_t)x_bytes);
        tma_load_3d(x_base + rx.i * x_bytes, &tm_x, 0, at.tt * p.nt, 2 * at.g, bar);
      }
      rx.next(); at.next(p);
    }
    for (int j = i > p.sx ? i - p.sx : 0; j < i; ++j) mbar_wait(smem_u32(&bar_xfull[j % p.sx]), (j / p.sx) & 1);
  } else if (warp == 1) {
    // ------------------------------------------------- MMA issuer
    const bool el = elect_one();
    const uint32_t idesc = umma_idesc(BF16 ? 1 : 0, 128, p.nt);
    const uint64_t desc0 = umma_smem_desc_sw128(x_base);
    const uint32_t desc_hi = (uint32_t)(desc0 >> 32), desc_lo0 = (uint32_t)desc0, half = (uint32_t)(p.nt * 128) >> 4;
    Ring rx(p.sx), ra(p.sa), rf(2 * p.sa), rd(p.nd);
    bool ok = true, first = true;
    for (int i = 0; ok && i < nunits; ++i) {
      const bool last = at.g == p.G - 1 || i == nunits - 1;
      if (first) ok = wait_bar_warp(&bar_dempty[rd.i], rd.ph ^ 1u, s_abort, status);   // the epilogue drained it (a fresh one is drained)
      ok = ok && wait_bar_warp(&bar_xfull[rx.i], rx.ph, s_abort, status);
      const uint32_t d = tmem + rd.i * 2 * p.nt;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ok = ok && wait_bar_warp(&bar_afull[ra.i], ra.ph, s_abort, status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t lo = desc_lo0 + (uint32_t)(rx.i * x_bytes >> 4) + h * half, a = tmem + col_a + ra.i * 64;
        const uint32_t acc0 = (!first || h > 0) ? 1u : 0u;
        if (el) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            umma_ts_lohi(d, a + ks * 8, lo + ks * 2, desc_hi, idesc, ks > 0 ? 1u : acc0);
            umma_ts_lohi(d + p.nt, a + 32 + ks * 8, lo + ks * 2, desc_hi, idesc, ks > 0 ? 1u : acc0);
          }
          umma_commit(smem_u32(&bar_afree[rf.i]));
          if (h == 1) {
            umma_commit(smem_u32(&bar_xfree[rx.i]));
            if (last) umma_commit(smem_u32(&bar_dfull[rd.i]));
          }
        }
        ra.next(); rf.next();
      }
      rx.next();
      if (last) rd.next();
      first = last;
      at.next(p);
    }
    // everything issued has completed before tensor memory may be released
    if (el) umma_commit(smem_u32(&bar_drain));
    mbar_wait(smem_u32(&bar_drain), 0);
  } else if (warp < kFirstEpi) {
    // ------------------------------------------------- dequantisers
    const int dw = warp - kFirstDequant;
    const int q = warp & 3, b = (dw >> 2) & 1, set = dw >> 3;
    const int g = lane >> 2;
    const bool el = elect_one();
    const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16) + col_a + 32 * b;
    // ldmatrix.x4: lanes 8j..8j+7 address rows 8j..8j+7 of two k-steps; 16-byte chunk c of row r sits at chunk c ^ (r & 7)
    const uint32_t ld_off = (uint32_t)lane * 128u + ((uint32_t)((4 * b + q) ^ (lane & 7)) << 4);
    const uint32_t pick = (g & 1) ? 0x3232u : 0x1010u;
    // this thread's eight columns (one word): its scales and zero-points come from global memory, a unit of its set ahead
    const int n_in = 128 * b + 32 * q + 8 * (g >> 1);
    uint4 sv = make_uint4(0u, 0u, 0u, 0u);
    uint32_t zw = 0u;
    auto fetch = [&]() {
      const int n0 = at.tn * kTileN + n_in;
      if (n0 < p.N) {
        sv = __ldg(reinterpret_cast<const uint4*>(p.sc + (size_t)at.g * p.N + n0));
        zw = __ldg(p.qz + (size_t)at.g * (p.N / 8) + n0 / 8);
      }
    };
    if (set) at.next(p);
    if (set < nunits) fetch();
    // rf: the half unit whose MMAs free this one's A slot (of the first ones: the phase before the first, which is over)
    Ring rw(p.sw), rl(2 * p.sw), ra(p.sa), rf(2 * p.sa);
    rf.i = p.sa; rf.ph = 1u;
    if (set) { rw.next(); rl.next(); ra.next(); ra.next(); rf.next(); rf.next(); }
    uint32_t lo_mask, hi_mask, magic;
    asm volatile("mov.u32 %0, %1;" : "=r"(lo_mask) : "n"(LO));
    asm volatile("mov.u32 %0, %1;" : "=r"(hi_mask) : "n"(HI));
    asm volatile("mov.u32 %0, %1;" : "=r"(magic) : "n"(MAGIC));
    bool ok = true;
    for (int i = set; ok && i < nunits; i += 2) {
      // per column of this thread's four (every second one of its word): the scale, and what to remove, in both halves
      uint32_t sc2[4], zm2[4];
      {
        const uint32_t swd[4] = {sv.x, sv.y, sv.z, sv.w}, zz = __byte_perm(zw, 0, pick);
#pragma unroll
        for (int pp = 0; pp < 4; ++pp) {
          sc2[pp] = __byte_perm(swd[pp], 0, pick);
          // fp16: odd nibbles arrive as 1024 + 16 q; fma by 1/16 with -(64 + z) gives q - z exactly
          if (!BF16 && (pp & 1)) zm2[pp] = ((zz >> (4 * pp - 4)) & HI) | 0xD400D400u;
          else zm2[pp] = ((zz >> (4 * pp)) & LO) | MAGIC;     // 1024 + z (128 + z)
        }
      }
      at.next(p); at.next(p);
      if (i + 2 < nunits) fetch();
      ok = wait_bar_warp(&bar_wfull[rl.i], rl.ph, s_abort, status);
      const uint32_t st = w_base + rw.i * kWStageBytes + ld_off;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t R[8];
        ldmatrix_x4_trans(R[0], R[1], R[2], R[3], st + h * 8192u);
        ldmatrix_x4_trans(R[4], R[5], R[6], R[7], st + h * 8192u + 4096u);
        ok = wait_bar_warp(&bar_afree[rf.i], rf.ph, s_abort, status) && ok;
        tc_fence_after();
        const uint32_t acol = lane_base + ra.i * 64;
#pragma unroll
        for (int ph = 0; ph < 2; ++ph) {
#pragma unroll
          for (int kp = 0; kp < 2; ++kp) {     // two k-steps per store
            uint32_t a[8];
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              const uint32_t R0 = R[4 * kp + 2 * kk], R1 = R[4 * kp + 2 * kk + 1];
              uint32_t a0, a1, a2, a3;
              if (BF16) {
                a0 = and_or(R0 >> (8 * ph), lo_mask, magic); a1 = and_or(R0 >> (8 * ph + 4), lo_mask, magic);
                a2 = and_or(R1 >> (8 * ph), lo_mask, magic); a3 = and_or(R1 >> (8 * ph + 4), lo_mask, magic);
                a1 = sub2<true>(a1, zm2[2 * ph + 1]); a3 = sub2<true>(a3, zm2[2 * ph + 1]);
              } else {
                const uint32_t l = R0 >> (8 * ph), hh = R1 >> (8 * ph);
                a0 = and_or(l, lo_mask, magic); a1 = and_or(l, hi_mask, magic); a2 = and_or(hh, lo_mask, magic); a3 = and_or(hh, hi_mask, magic);
                a1 = fma2_f16(a1, SIXTEENTH, zm2[2 * ph + 1]); a3 = fma2_f16(a3, SIXTEENTH, zm2[2 * ph + 1]);
              }
              a[4 * kk] = mul2<BF16>(sub2<BF16>(a0, zm2[2 * ph]), sc2[2 * ph]);
              a[4 * kk + 1] = mul2<BF16>(a1, sc2[2 * ph + 1]);
              a[4 * kk + 2] = mul2<BF16>(sub2<BF16>(a2, zm2[2 * ph]), sc2[2 * ph]);
              a[4 * kk + 3] = mul2<BF16>(a3, sc2[2 * ph + 1]);
            }
            tmem_st_16x128b_x4(acol + ((uint32_t)(16 * ph) << 16) + 16 * kp, a);
          }
        }
        if (h == 1) {
          __syncwarp();
          if (el) mbar_arrive(smem_u32(&bar_wfree[rw.i]));   // this warp has read what it needs of the packed tile
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (el) mbar_arrive(smem_u32(&bar_afull[ra.i]));
        ra.next(); rf.next();
      }
      // the other set's unit lies between
      rw.next(); rw.next(); rl.next(); rl.next(); ra.next(); ra.next(); rf.next(); rf.next();
    }
  } else {
    // ------------------------------------------------- epilogue
    const int q = warp & 3, blk = (warp - kFirstEpi) >> 2;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16) + blk * p.nt;
    Ring rd(p.nd);
    int left = nunits, seg = 0;
    while (left > 0) {
      const int len = min(p.G - at.g, left);
      left -= len;
      if (!wait_bar_warp(&bar_dfull[rd.i], rd.ph, s_abort, status)) break;
      tc_fence_after();
      store_tile<BF16>(p, at.tn, at.tt, len == p.G, seg > 0, lane_base + rd.i * 2 * p.nt, q, blk, [&]() {
        tc_fence_before();      // it may be overwritten
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_dempty[rd.i]));
      });
      rd.next();
      ++seg;
      at.g = p.G - 1;
      at.next(p);
    }
  }

  // all roles meet here, also after a give-up, so that tensor memory is always released
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, kTmemCols); }
}

// out[tok, n] of the tiles that more than one CTA worked on: their segments in CTA order, + bias.  A thread adds one column of QUADS x
// four tokens, and two neighbours write two columns of half of these each; blockIdx.x is the tile.  Bound by how many loads are under
// way: eight a thread, of one quad where a tile has many segments and of two where it has up to five (4096 x 12288, 128 tokens, three
// parts: 22.2 -> 21.4 us a call).
constexpr int kFixThreads = 256;
template <bool BF16, int QUADS>
__global__ void __launch_bounds__(kFixThreads) umma_prefill_fixup_kernel(const Params p) {
  grid_launch_dependents();
  constexpr int kAhead = 8 / QUADS;
  const long long u0 = (long long)blockIdx.x * p.G;
  const int c0 = cta_of_unit(u0, p.U, p.ctas), c1 = cta_of_unit(u0 + p.G - 1, p.U, p.ctas);
  if (c0 == c1) return;
  const int tn = (int)(blockIdx.x / (unsigned)p.ntt), tt = (int)(blockIdx.x % (unsigned)p.ntt);
  const int l = threadIdx.x, quad = blockIdx.y * QUADS, tok = tt * p.nt + quad * 4;
  const int n = tn * kTileN + (l & 128) + column_of_lane(l & 127);   // lanes l, l + 1 (l even): columns n, n + 1
  if (tok >= p.M || (n & ~31) >= p.N) return;                        // whole warps: N is a multiple of 32
  // the tile is a CTA's second segment where that CTA's range begins before it
  const bool second = range_begin(c0, p.U, p.ctas, p.G, 0) < u0;
  const size_t seg = (size_t)p.nt * 64;
  const float4* src = reinterpret_cast<const float4*>(p.slots) + (2 * (size_t)c0 + 2) * seg + (size_t)quad * 256 + l;
  const float4* own = src - (second ? seg : 2 * seg);
  grid_dependency_wait();
  float4 s[QUADS];
#pragma unroll
  for (int j = 0; j < QUADS; ++j) s[j] = __ldcg(own + j * 256);      // the tile's tokens are a multiple of 16: quads come in pairs
  for (int c = c0 + 1; c <= c1; c += kAhead, src += 2 * kAhead * seg) {
    float4 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)      // all under way before the first is added, also where fewer are left (the rest are zeros)
      asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n mov.f32 %2, 0f00000000;\n mov.f32 %3, 0f00000000;\n"
                   " @p ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];\n}" : "=f"(v[k].x), "=f"(v[k].y), "=f"(v[k].z), "=f"(v[k].w)
                   : "l"(src + (size_t)(2 * (k / QUADS)) * seg + (k % QUADS) * 256), "r"((int)(c + k / QUADS <= c1)) : "memory");
#pragma unroll
    for (int k = 0; k < 8; ++k) { float4& t = s[k % QUADS]; t.x += v[k].x; t.y += v[k].y; t.z += v[k].z; t.w += v[k].w; }
  }
  const float b = p.bias ? bias_to_float(p.bias, p.bias_dtype, n) : 0.f;
#pragma unroll
  for (int j = 0; j < QUADS; ++j) {
    const uint32_t lo = (uint32_t)float_to_raw16<BF16>(s[j].x + b) | ((uint32_t)float_to_raw16<BF16>(s[j].y + b) << 16);   // tokens 0, 1
    const uint32_t hi = (uint32_t)float_to_raw16<BF16>(s[j].z + b) | ((uint32_t)float_to_raw16<BF16>(s[j].w + b) << 16);   // tokens 2, 3
    const uint32_t got = __shfl_xor_sync(0xffffffffu, (l & 1) ? lo : hi, 1);
    const uint32_t left = (l & 1) ? got : lo, right = (l & 1) ? hi : got;      // of columns n & ~1 and n | 1, this thread's two tokens
    const int t0 = tok + 4 * j + ((l & 1) ? 2 : 0);
    uint16_t* dst = p.out + (size_t)t0 * p.N + (n & ~1);
    if (t0 < p.M) *reinterpret_cast<uint32_t*>(dst) = __byte_perm(left, right, 0x5410);
    if (t0 + 1 < p.M) *reinterpret_cast<uint32_t*>(dst + p.N) = __byte_perm(left, right, 0x7632);
  }
}

// x[M][K] as [K / 64][M][64]: a box of both 64-k halves of a group, each [tokens][128 bytes] with the 128-byte swizzle
static bool encode_k_halves(CUtensorMap* m, CUtensorMapDataType dt, const void* x, int M, int K, int nt) {
  PFN_cuTensorMapEncodeTiled enc = tensor_map_encoder();
  if (!enc) return false;
  cuuint64_t dims[3] = {64, (cuuint64_t)M, (cuuint64_t)(K / 64)};
  cuuint64_t strides[2] = {(cuuint64_t)K * 2, 128};
  cuuint32_t box[3] = {64, (cuuint32_t)nt, 2}, estr[3] = {1, 1, 1};
  return enc(m, dt, 3, const_cast<void*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct Plan { int ntn, ntt, nt, G, ctas, whole, sw, sx, sa, nd, smem; long long U; bool fixup; };
static Plan make_plan(int64_t M, int64_t N, int64_t K) {
  Plan pl;
  pl.G = (int)(K / kUnitK);
  pl.ntt = (int)((M + kTileT - 1) / kTileT);      // as few token tiles as hold M, all alike
  pl.nt = (int)(((M + pl.ntt - 1) / pl.ntt + 15) / 16 * 16);
  pl.ntn = (int)((N + kTileN - 1) / kTileN);
  const long long items = (long long)pl.ntn * pl.ntt;
  pl.U = items * pl.G;
  // tensor memory: two accumulators of two blocks up to 64 tokens, one beyond, the rest (at most six slots) for the A operand
  pl.nd = pl.nt <= 64 ? 2 : 1;
  pl.sa = (kTmemCols - pl.nd * 2 * pl.nt) / 64;
  if (pl.sa > kMaxA) pl.sa = kMaxA;
  const int x_bytes = pl.nt * 256;
  pl.sx = pl.nt <= 64 ? 4 : 3;
  pl.sw = (kSmemBudget - 1024 - pl.sx * x_bytes) / kWStageBytes;
  if (pl.sw > kMaxW) pl.sw = kMaxW;
  pl.smem = pl.sx * x_bytes + pl.sw * kWStageBytes + 1024;
  // Whole tiles, an equal share for every SM, or every tile in equally many parts (then a CTA leaves one segment instead of
  // two): whichever this model expects to end first.  Microseconds, from chains of calls with 17 to 400 tokens of 14 shapes: a
  // unit takes 0.71 at 17 tokens, 0.73 at 48, 0.87 at 128, a seventh more in parts; 4 to 6 go before and behind the units (2.8 from
  // the end of the kernel ahead to the first MMA); the second kernel has segments to read, eight at a time; a chain of calls of
  // more than about 100 CTAs each overlaps less.  48 tokens, 4096 x 24576: whole tiles 28.3, shares 27.2; 4096 x 6144: six parts
  // 12.5, shares of 148 12.6, whole tiles 26.9; 3072 x 3072: eight parts 7.9, six 8.4, twelve 10.5.
  const double unit = 0.66 + 0.0017 * pl.nt;
  auto t_shares = [&](long long ctas, long long segments, long long per_tile, double base, double slower) {
    return base + (ctas > 100 ? 0.7 : 0.0) + slower * unit * (double)((pl.U + ctas - 1) / ctas) + 0.45 * (double)((per_tile + 6) / 8) + (double)segments * pl.nt / 5000.0;
  };
  const long long waves = (items + kNumSMs - 1) / kNumSMs, all = pl.U < kNumSMs ? pl.U : kNumSMs;
  double best = 3.0 + 0.017 * pl.nt + (double)waves * pl.G * unit + (pl.nd == 1 ? 1.5 * (double)(waves - 1) : 0.0);
  pl.whole = 1;
  pl.ctas = (int)(items < kNumSMs ? items : (long long)kNumSMs);
  const double t_all = t_shares(all, 2 * all, (all + items - 1) / items + 1, 6.0, 1.05);
  if (t_all < best) { best = t_all; pl.whole = 0; pl.ctas = (int)all; }
  for (long long parts = 2; parts <= pl.G && parts * items <= kNumSMs; ++parts) {
    const double t = t_shares(parts * items, parts * items, parts, 5.2, 1.15);
    if (t < best) { best = t; pl.whole = 0; pl.ctas = (int)(parts * items); }
  }
  pl.fixup = false;
  if (!pl.whole)
    for (int c = 1; c < pl.ctas && !pl.fixup; ++c) pl.fixup = range_begin(c, pl.U, pl.ctas, pl.G, 0) % pl.G != 0;
  return pl;
}
static size_t slot_bytes(const Plan& pl) { return pl.fixup ? (size_t)2 * pl.ctas * pl.nt * 256 * sizeof(float) : 0; }

template <bool BF16>
static int launch_t(const CUtensorMap& tw, const CUtensorMap& tx, const Params& sp, const Plan& pl, cudaStream_t st) {
  // The shared-memory attribute belongs to the device that is current when it is set: one flag per device.
  static std::mutex mu;
  static bool configured[kMaxDevices] = {false};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) { cudaGetLastError(); return NQB200_ERR_UNSUPPORTED_DEVICE; }
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!configured[dev]) {
      if (cudaFuncSetAttribute(umma_prefill_kernel<BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget) != cudaSuccess) {
        cudaGetLastError();
        return NQB200_ERR_LAUNCH;
      }
      configured[dev] = true;
    }
  }
  const int rc = launch_overlapped(umma_prefill_kernel<BF16>, dim3(pl.ctas), dim3(kThreads), pl.smem, st, tw, tx, sp);
  if (rc != NQB200_OK || !pl.fixup) return rc;
  const bool few = pl.ctas <= 4ll * pl.ntn * pl.ntt;     // a tile then has five segments at most
  const dim3 grid((unsigned)(pl.ntn * pl.ntt), pl.nt / (few ? 8 : 4));
  return few ? launch_overlapped(umma_prefill_fixup_kernel<BF16, 2>, grid, dim3(kFixThreads), 0, st, sp)
             : launch_overlapped(umma_prefill_fixup_kernel<BF16, 1>, grid, dim3(kFixThreads), 0, st, sp);
}

}  // namespace pre

bool umma_prefill_supports(int64_t M, int64_t N, int64_t K, int64_t g) {
  return M > 16 && g == 128 && K % 128 == 0 && N % 32 == 0;
}

// Another cost model's estimate of this kernel, made for an earlier form of it: the two-SM kernel's rule was fitted against
// these numbers, and only against these.
double umma_prefill_estimate_us(int64_t M, int64_t N, int64_t K) {
  const long long tiles = ((N + pre::kTileN - 1) / pre::kTileN) * ((M + pre::kTileT - 1) / pre::kTileT);
  const int G = (int)(K / 128);
  const int nt = M >= pre::kTileT ? pre::kTileT : (int)((M + 15) / 16) * 16;
  const double t_group = 1.2 * nt / 128.0 > 0.7 ? 1.2 * nt / 128.0 : 0.7;
  double best_us = 1e30, unsplit_us = 0.0;
  for (int ks = 1; ks <= 16 && ks <= G; ++ks) {
    const long long waves = (tiles * ks + kNumSMs - 1) / kNumSMs;
    double us = (double)waves * ((double)((G + ks - 1) / ks) * t_group + 1.5);
    if (ks > 1) us += 3.0 + (double)ks * (double)M * (double)N * 8.0 / 6.0e6;
    if (ks == 1) unsplit_us = us;
    if (us < best_us - 1e-9) best_us = us;
  }
  return best_us < 0.92 * unsplit_us ? best_us : unsplit_us;
}

int umma_prefill_launches(int64_t M, int64_t N, int64_t K) { return pre::make_plan(M, N, K).fixup ? 2 : 1; }

size_t umma_prefill_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  return (size_t)kCounterBytes + pre::slot_bytes(pre::make_plan(M, N, K));
}

int launch_umma_prefill(const GemmArgs& a) {
  using namespace pre;
  const Plan pl = make_plan(a.M, a.N, a.K);
  Params sp;
  sp.sc = (const uint16_t*)a.sc; sp.qz = a.qz;
  sp.bias = a.bias; sp.bias_dtype = a.bias_dtype; sp.out = (uint16_t*)a.out;
  sp.M = a.M; sp.N = a.N; sp.G = pl.G; sp.ntt = pl.ntt; sp.nt = pl.nt; sp.U = pl.U; sp.ctas = pl.ctas; sp.whole = pl.whole;
  sp.sw = pl.sw; sp.sx = pl.sx; sp.sa = pl.sa; sp.nd = pl.nd;
  sp.status = (a.ws && a.ws_bytes >= (size_t)kCounterBytes) ? (int*)a.ws + (kCounterBytes / 4 - 1) : nullptr;
  sp.slots = nullptr;
  if (pl.fixup) {
    if (!a.ws || a.ws_bytes < (size_t)kCounterBytes + slot_bytes(pl)) return NQB200_ERR_WORKSPACE;
    if (!aligned16(a.ws)) return NQB200_ERR_MISALIGNED;
    sp.slots = (float*)((char*)a.ws + kCounterBytes);
  }
  alignas(64) CUtensorMap tw, tx;
  const CUtensorMapDataType xdt = a.dtype == NQB200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  bool ok = encode_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, a.qw, a.K, a.N / 8, kUnitK, 32, CU_TENSOR_MAP_SWIZZLE_128B);
  ok = ok && encode_k_halves(&tx, xdt, a.x, a.M, a.K, pl.nt);
  if (!ok) return NQB200_ERR_LAUNCH;
  return a.dtype == NQB200_BF16 ? launch_t<true>(tw, tx, sp, pl, a.stream) : launch_t<false>(tw, tx, sp, pl, a.stream);
}

}  // namespace nqb200

// Attention of fp32 tensors on the tensor cores, calls of more than one round of tiles with head dims 33 to 64 (f32_sm100.cu has the others,
// and the operator's reference): one CTA takes two tiles of 128 query rows of a head, so that every key and value block that
// it fetches serves 256 rows.  With one tile to a CTA the blocks' way from L2 into shared memory set the time: 2 x 4096 tokens,
// 8 heads of 40 took 284 us without any product and 305 with them.
//
// Q and K are three bf16 numbers per element and a score six of their products, as there.  The weights and V are two
// fp16 numbers each, a value rounded to fp16 and the rest rounded to fp16, which is 22 bits and a sign: P V is the weights' second part
// times V's first, and their first part times [V's first part | V's second part], three products where bf16 parts take six, and
// 32 KB of V a block instead of 48, without which two tiles and their blocks do not fit.
// fp16's range is kept by powers of two: 2^14 in the weights (at most 1), and in each block of 128 rows of V the
// one that brings its largest magnitude to 2^14 .. 2^15; it is taken out again when the block's O is added up.  An element
// below 2^-16 of its block's largest loses bits; split_pair_kernel counts them, and where a block has 16 or more (an outlying
// row or column: of numbers from one distribution it is one in ten thousand) the pair kernel does nothing but make V's bf16 parts, and
// f32_tcgen05_kernel behind it, which otherwise returns at once, computes the call.
//
// The tensor core cuts its sums off instead of rounding them.  The products of fp16 parts have 22 bits, so that every step
// of a sum loses some, where those of bf16 parts have 16 and lose next to none: O comes out short by 2.2e-7 to 2.5e-7 of itself (N(0,1)
// tensors).  kPutBack, a factor in the power of two that is taken out, makes up for the mean of it.
//
// Error against 64 bits (2-norm, relative; N(0,1), one tile to a CTA / here): 1024 tokens, heads of 40 2.18e-7 / 1.98e-7, of 64
// 2.04e-7 / 1.96e-7; 4096 tokens 2.58e-7 / 2.35e-7 and 2.41e-7 / 2.31e-7; queries six times as large, 1024 tokens, heads of 64 3.69e-7 / 3.76e-7.
// Measured, us in short bursts (one tile to a CTA / here): 2 x 4096 tokens, 8 heads of 40 310 / 222, 10 heads of 64 438 / 376; for
// seconds, when the power cap holds the clock at 1.7 GHz, 336 / 235 and 475 / 397.  What bounds it: at head dim 64 the products, 24 MMAs
// of Q K^T that read both operands from shared memory at its full rate (64 cycles each) and 16 of P V to a block and tile; at 40, where those
// are 18 and shorter ones, the chain from a tile's scores through its softmax to its next scores.
//
// f32_pair_kernel: persistent over (batch, head, 256 query rows); 12 warps:
//   warp 0      TMA producer: Q of both tiles per item, K blocks through two slots, V blocks through one
//   warp 1      MMA issuer (the whole warp, one lane issues), per block: P V of tile 0, Q K^T of tile 0 and the next block, the same of
//               tile 1; a tile's softmax runs under the other tile's products
//   warp 2      TMEM allocation / release
//   warps 4-7   softmax of tile 0, one thread per query row: scores -> weights -> two fp16 parts in the columns that the scores
//               came in, then the block's O from TMEM into the row's fp32 accumulators
//   warps 8-11  the same for tile 1
#include <math.h>

#include "sm100_ptx.cuh"
#include "f32_split.cuh"


namespace dt {
namespace {

constexpr int kBM = 128, kBN = 128;
constexpr int kThreads = 384;
constexpr int kRegsLow = 80, kRegsHigh = 208;  // 128 * low + 256 * high <= 384 threads * 168 at launch
constexpr int kPlane = 128 * 128;              // bytes of one part of 128 rows: 64 columns of 16 bits
constexpr int kQTile = 3 * kPlane;
// Beside Q there is room for eight parts: three places of two and two of one.  V(j) takes the place of two j mod 3 and K(j), three
// parts, the place of two j + 1 mod 3 and the place of one j mod 2.  So V(j) can be fetched as soon as both tiles' scores of block j - 1
// are there, and K(j) when P V of block j - 2 is done.  (K in two places of three and V in one of its own: V's way from L2, 1500
// cycles and more, stood between two blocks, 2 x 4096 tokens, 10 heads of 64 372 us.)
constexpr int kRing = 8;
constexpr int kSmemBytes = 2 * kQTile + kRing * kPlane + 256 + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory");
// TMEM columns: S of the two tiles, then their O (2 D columns each).  The weights of 32 keys take the columns of their scores:
// 16 of first parts, 16 of second parts.
constexpr uint32_t kColO = 256;
constexpr float kWeightScale = 16384.f;
#ifndef X_PUT
#define X_PUT 2
#endif
constexpr float kPutBack = 1.f + X_PUT * 1.1920929e-7f;
constexpr int kSplitThreads = 256;
constexpr int kSplitIt = 4;  // rounds over 128 rows: 256 threads take at least 32 rows of up to 64 columns at a time

struct PairBars {
  uint64_t q_full, q_empty;
  uint64_t s_full[2], p_half[2][2], o_full[2];  // [tile], [tile][half of the keys]
  uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2];  // blocks in turn
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(PairBars) <= 256, "barrier area");

struct PairArgs {
  float* o;
  float* lse;
  int64_t o_sb, o_ss, o_sh;
  unsigned int* status;
  const uint32_t* flags;  // [n_flags]: bit 0, V does not fit two fp16 parts; bit 1, a number does not fit three bf16 parts
  int n_flags;
  uint32_t *done, *no_parts;  // written for the kernels behind this one: it has computed the call; the CUDA cores have to
  const float* v_undo;    // [B, Hkv, n_kb]: what takes the power of two out of a block's O
  int n_kb;
  int Sq, Sk, Hq, Hkv, D;
  int n_qp, n_items;
  float scale_log2;
};

struct PairSplitTensor {
  const float* src;
  uint4* dst;  // Q, K: [B, S, H, 3, D] bf16; V: [B, S, H, 2, D] fp16
  int64_t sb, ss, sh;
  int S, H, n_blk;
  unsigned begin, end;  // its blocks of 128 rows of a head in the launch's numbering
};
struct PairSplitArgs {
  PairSplitTensor t[3];
  float* v_undo;
  unsigned n_units;
  int per_row;  // D / 8
  uint32_t* flags;
};

// Bound: HBM / L2 writes (4 bytes read and 6 or 4 written per element).  A CTA takes 128 rows of a head at a time and keeps them in
// registers, V's between finding their largest magnitude and writing the parts.
__global__ void __launch_bounds__(kSplitThreads, 4) split_pair_kernel(const __grid_constant__ PairSplitArgs a) {
  __shared__ uint32_t s_max[kSplitThreads / 32];
  __shared__ int s_lossy;
  ptx::wait_for_previous();
  ptx::let_next_start();
  const int ch = threadIdx.x % a.per_row, r0 = threadIdx.x / a.per_row, r_step = kSplitThreads / a.per_row;
  uint32_t bad = 0;
  for (unsigned u = blockIdx.x; u < a.n_units; u += gridDim.x) {
    const int which = u < a.t[0].end ? 0 : u < a.t[1].end ? 1 : 2;
    const PairSplitTensor& t = a.t[which];
    const unsigned unit = u - t.begin, h = unit % t.H, bb = unit / t.H, blk = bb % t.n_blk, b = bb / t.n_blk;
    const int rows = r0 < r_step ? min(kBM, t.S - (int)blk * kBM) : 0;
    const float* src = t.src + b * t.sb + (int64_t)(blk * kBM) * t.ss + h * t.sh + ch * 8;
    float x[kSplitIt][8];
#pragma unroll
    for (int i = 0; i < kSplitIt; ++i) {
      const int r = r0 + i * r_step;
      float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
      if (r < rows) {
        lo = __ldg(reinterpret_cast<const float4*>(src + r * t.ss));
        hi = __ldg(reinterpret_cast<const float4*>(src + r * t.ss) + 1);
      }
      x[i][0] = lo.x; x[i][1] = lo.y; x[i][2] = lo.z; x[i][3] = lo.w;
      x[i][4] = hi.x; x[i][5] = hi.y; x[i][6] = hi.z; x[i][7] = hi.w;
    }
    const size_t row0 = (size_t)(b * t.S + blk * kBM) * t.H + h;
    if (which < 2) {
#pragma unroll
      for (int i = 0; i < kSplitIt; ++i) {
        const int r = r0 + i * r_step;
        if (r >= rows) break;
        uint4 w[3];
        bad |= 2u * f32_three_parts(x[i], w);
        uint4* dst = t.dst + (row0 + (size_t)r * t.H) * 3 * a.per_row + ch;
#pragma unroll
        for (int p = 0; p < 3; ++p) dst[p * a.per_row] = w[p];
      }
      continue;
    }
    uint32_t mx = 0;
#pragma unroll
    for (int i = 0; i < kSplitIt; ++i)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        bad |= 2u * f32_out_of_range(x[i][e]);
        mx = max(mx, __float_as_uint(x[i][e]) & 0x7fffffffu);  // (NaN compares above everything)
      }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (threadIdx.x == 0) s_lossy = 0;
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSplitThreads / 32; ++i) mx = max(mx, s_max[i]);
    const bool fits = mx < 0x5c800000u && mx >= 0x0d800000u;  // 2^-100 <= the largest magnitude < 2^58
    if (!fits && mx != 0) bad |= 1u;
    const int e = fits ? (int)(mx >> 23) - 127 : 0;  // 2^e <= the largest magnitude < 2^(e + 1)
    const float up = __uint_as_float((uint32_t)(127 + 14 - e) << 23);
    if (threadIdx.x == 0) a.v_undo[(size_t)(b * t.H + h) * t.n_blk + blk] = __uint_as_float((uint32_t)(127 - 14 + e) << 23) * kPutBack;
    int lossy = 0;
#pragma unroll
    for (int i = 0; i < kSplitIt; ++i) {
      const int r = r0 + i * r_step;
      uint32_t w[2][4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float x0 = x[i][2 * k] * up, x1 = x[i][2 * k + 1] * up;
        lossy += (x0 != 0.f && fabsf(x0) < 0.25f) + (x1 != 0.f && fabsf(x1) < 0.25f);  // its rest is below fp16's normal numbers
        w[0][k] = ptx::cvt_pack_f16(x0, x1);
        float h0, h1;
        ptx::unpack_f16(w[0][k], h0, h1);
        w[1][k] = ptx::cvt_pack_f16(x0 - h0, x1 - h1);
      }
      if (r < rows) {
        uint4* dst = t.dst + (row0 + (size_t)r * t.H) * 2 * a.per_row + ch;
        dst[0] = make_uint4(w[0][0], w[0][1], w[0][2], w[0][3]);
        dst[a.per_row] = make_uint4(w[1][0], w[1][1], w[1][2], w[1][3]);
      }
    }
    if (lossy) atomicAdd(&s_lossy, lossy);
    __syncthreads();
    if (s_lossy >= 16) bad |= 1u;
    __syncthreads();  // (s_lossy and s_max are written again)
  }
  const int no16 = __syncthreads_or((int)(bad & 1u)), no_parts = __syncthreads_or((int)(bad & 2u));
  if (threadIdx.x == 0) a.flags[blockIdx.x] = (no16 ? 1u : 0u) | (no_parts ? 2u : 0u);
}

__device__ constexpr int kProdA[6] = {2, 0, 1, 1, 0, 0};  // the small products first (f32_sm100.cu)
__device__ constexpr int kProdB[6] = {0, 2, 1, 0, 1, 0};

// NPV: the head dim, rounded up to a multiple of 16
template <int NPV>
__global__ void __launch_bounds__(kThreads, 1)
f32_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const PairArgs a, const __grid_constant__ F32SplitArgs v_parts) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  constexpr int kRingAt = 2 * kQTile;
  PairBars* bars = reinterpret_cast<PairBars*>(base_ptr + kRingAt + kRing * kPlane);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_full, 1);
    ptx::mbar_init(&bars->q_empty, 1);
    for (int t = 0; t < 2; ++t) {
      ptx::mbar_init(&bars->s_full[t], 1);
      ptx::mbar_init(&bars->p_half[t][0], 4);  // one arrival per softmax warp
      ptx::mbar_init(&bars->p_half[t][1], 4);
      ptx::mbar_init(&bars->o_full[t], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&bars->k_full[i], 1);
      ptx::mbar_init(&bars->k_empty[i], 1);
      ptx::mbar_init(&bars->v_full[i], 1);
      ptx::mbar_init(&bars->v_empty[i], 1);
    }
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  ptx::wait_for_previous();
  uint32_t bad = 0;
  for (int i = threadIdx.x; i < a.n_flags; i += kThreads) bad |= a.flags[i];
  const int no_parts = __syncthreads_or((int)(bad & 2u)), no16 = __syncthreads_or((int)(bad & 1u));
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *a.done = no16 && !no_parts ? 0u : 1u;
    *a.no_parts = no_parts ? 1u : 0u;
  }
  if (no_parts || no16) {  // the whole grid alike, before anything was allocated
    if (!no_parts) f32_split_planes(v_parts, blockIdx.x * kThreads + threadIdx.x, gridDim.x * kThreads);
    return;
  }
  if (warp == 2) {
    ptx::tmem_alloc(&bars->tmem_base, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile int* abort_flag = &bars->abort_flag;
  const int nkv = (a.Sk + kBN - 1) / kBN, G = a.Hq / a.Hkv;
  auto tiles_of = [&](int qp) { return qp * 2 * kBM + kBM < a.Sq ? 2 : 1; };

  if (warp < 4) {
    ptx::setmaxnreg_dec<kRegsLow>();
    if (warp == 0) {
      // =========================== TMA producer ===========================
      if (lane == 0) {
        ptx::prefetch_tensormap(&map_q);
        ptx::prefetch_tensormap(&map_k);
        ptx::prefetch_tensormap(&map_v);
        const int v_boxes = (2 * a.D + 63) >> 6;
        int n_item = 0;
        uint32_t n_k = 0, n_v = 0;  // blocks fetched so far, over all items
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t par) -> bool {
          if (ptx::mbar_wait(bar, par, abort_flag)) return true;
          atomicCAS(a.status, 0u, 2u);
          *abort_flag = 1;
          ok = false;
          return false;
        };
        for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x, ++n_item) {
          const int qp = item % a.n_qp, bh = item / a.n_qp, h = bh % a.Hq, b = bh / a.Hq, kvh = h / G, tiles = tiles_of(qp);
          auto load_k = [&](int j) -> bool {
            const uint32_t n = n_k++;
            uint64_t* bar = &bars->k_full[n & 1];
            if (n >= 2 && !wait(&bars->v_empty[n & 1], ((n - 2) >> 1) & 1)) return false;  // V(n - 2), and K(n - 2) before it
            ptx::mbar_arrive_expect_tx(bar, (uint32_t)(3 * kPlane));
            for (int p = 0; p < 3; ++p)
              ptx::tma_load_4d(base_ptr + kRingAt + (p < 2 ? (n + 1) % 3 * 2 + p : 6 + (n & 1)) * kPlane, &map_k, bar, 0, kvh * 3 + p, j * kBN, b);
            return true;
          };
          auto load_v = [&](int j) -> bool {
            const uint32_t n = n_v++;
            uint64_t* bar = &bars->v_full[n & 1];
            if (n >= 1 && !wait(&bars->k_empty[(n - 1) & 1], ((n - 1) >> 1) & 1)) return false;
            ptx::mbar_arrive_expect_tx(bar, (uint32_t)(v_boxes * kPlane));
            for (int c = 0; c < v_boxes; ++c)
              ptx::tma_load_4d(base_ptr + kRingAt + (n % 3 * 2 + c) * kPlane, &map_v, bar, c * 64, kvh, j * kBN, b);
            return true;
          };
          if (!load_k(0)) break;
          if (n_item > 0 && !wait(&bars->q_empty, (n_item - 1) & 1)) break;
          ptx::mbar_arrive_expect_tx(&bars->q_full, (uint32_t)(tiles * kQTile));
          for (int t = 0; t < tiles; ++t)
            for (int p = 0; p < 3; ++p)
              ptx::tma_load_4d(base_ptr + t * kQTile + p * kPlane, &map_q, &bars->q_full, 0, h * 3 + p, (qp * 2 + t) * kBM, b);
          for (int j = 0; j < nkv && ok; ++j) ok = load_v(j) && (j + 1 >= nkv || load_k(j + 1));
        }
      }
    } else if (warp == 1) {
      // =========================== MMA issuer (the whole warp, one lane issues) ===========================
      const bool on = ptx::elect_one();
      constexpr uint32_t idesc_qk = ptx::make_idesc_f16(1, kBM, kBN, 0, 0);
      const uint32_t idesc_pv = ptx::make_idesc_f16(0, kBM, 2 * a.D, 0, 1);
      constexpr uint32_t idesc_lo = ptx::make_idesc_f16(0, kBM, NPV, 0, 1);
      const uint64_t q_desc = ptx::make_smem_desc_sw128(base, 16, 1024);
      const uint64_t k_desc = ptx::make_smem_desc_sw128(base + kRingAt, 16, 1024);
      const uint64_t v_desc = ptx::make_smem_desc_sw128(base + kRingAt, kPlane, 1024);
      int n_item = 0;
      uint32_t n_k = 0, n_v = 0, p_par[2] = {0u, 0u};
      int k_at = 1, v_at = 0;  // their places of two
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity, unsigned code) -> bool {
        if (__all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag))) return true;
        if (on) atomicCAS(a.status, 0u, code);
        *abort_flag = 1;
        ok = false;
        return false;
      };
      for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x, ++n_item) {
        const int tiles = tiles_of(item % a.n_qp);
        if (!wait(&bars->q_full, n_item & 1, 1u)) break;
        auto qk = [&](int t) {
          const uint64_t qd = q_desc + (uint64_t)(t * (kQTile >> 4));
          const uint64_t kd = k_desc + (uint64_t)(k_at * (2 * kPlane >> 4)), kd2 = k_desc + (uint64_t)((6 + (n_k & 1)) * (kPlane >> 4));
#pragma unroll
          for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int ks = 0; ks < NPV / 16; ++ks)
              ptx::mma_ss_on(on, tmem + t * kBN, qd + (uint64_t)((kProdA[i] * kPlane + ks * 32) >> 4),
                             (kProdB[i] == 2 ? kd2 : kd) + (uint64_t)(((kProdB[i] & 1) * kPlane + ks * 32) >> 4), idesc_qk, (i | ks) ? 1u : 0u);
          ptx::tc_commit_on(on, &bars->s_full[t]);
        };
        auto k_done = [&](bool last) {
          ptx::tc_commit_on(on, &bars->k_empty[n_k & 1]);
          if (last) ptx::tc_commit_on(on, &bars->q_empty);
          ++n_k;
          if (++k_at == 3) k_at = 0;
        };
        if (!wait(&bars->k_full[n_k & 1], (n_k >> 1) & 1, 1u)) break;
        ptx::tc_fence_after();
        for (int t = 0; t < tiles; ++t) qk(t);
        k_done(nkv == 1);
        for (int j = 0; j < nkv && ok; ++j) {
          const bool more = j + 1 < nkv;
          const int steps = (min(kBN, a.Sk - j * kBN) + 15) >> 4, first = steps > 4 ? 4 : 0;
          if (!wait(&bars->v_full[n_v & 1], (n_v >> 1) & 1, 1u)) break;
          const uint64_t vd = v_desc + (uint64_t)(v_at * (2 * kPlane >> 4));
          for (int t = 0; t < tiles && ok; ++t) {
            const uint32_t p = tmem + t * kBN, o = tmem + kColO + t * 128;
            // the second 64 keys are handed over first; their weights' second parts, those of the first 64, then the first parts
            auto pv = [&](int half, int part) {
              const uint32_t from = p + half * 64 + part * 16;
              if (steps == 8) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  ptx::mma_ts_on(on, o, from + (i >> 1) * 32 + (i & 1) * 8, vd + (uint64_t)((half * 4 + i) * (2048 >> 4)),
                                 part == 1 && !(half == 1 && i == 0) ? idesc_lo : idesc_pv, part == 1 && half == 1 && i == 0 ? 0u : 1u);
              } else {
#pragma unroll 1
                for (int ks = half * 4; ks < min(half * 4 + 4, steps); ++ks)
                  ptx::mma_ts_on(on, o, p + (ks >> 1) * 32 + (ks & 1) * 8 + part * 16, vd + (uint64_t)(ks * (2048 >> 4)),
                                 part == 1 && ks != first ? idesc_lo : idesc_pv, part == 1 && ks == first ? 0u : 1u);
              }
            };
            if (!wait(&bars->p_half[t][1], p_par[t], 4u)) break;
            ptx::tc_fence_after();
            pv(1, 1);
            if (!wait(&bars->p_half[t][0], p_par[t], 4u)) break;
            p_par[t] ^= 1u;
            ptx::tc_fence_after();
            pv(0, 1);
            pv(1, 0);
            pv(0, 0);
            ptx::tc_commit_on(on, &bars->o_full[t]);
            if (t == tiles - 1) ptx::tc_commit_on(on, &bars->v_empty[n_v & 1]);
            if (more) {
              if (t == 0) {
                if (!wait(&bars->k_full[n_k & 1], (n_k >> 1) & 1, 1u)) break;
                ptx::tc_fence_after();
              }
              qk(t);  // over the weights that the P V above has read
              if (t == tiles - 1) k_done(j + 2 == nkv);
            }
          }
          ++n_v;
          if (++v_at == 3) v_at = 0;
        }
      }
    }
  } else {
    ptx::setmaxnreg_inc<kRegsHigh>();
    // =========================== softmax / accumulation / store ===========================
    const int t = (warp - 4) >> 2;
    const int row_in_tile = ((warp & 3) << 5) + lane;
    const uint32_t tl = tmem + ((uint32_t)((warp & 3) << 5) << 16), t_s = tl + t * kBN, t_o = tl + kColO + t * 128;
    const float sl2 = a.scale_log2;
    const uint64_t scale2 = ptx::pack_f32x2(sl2, sl2), weight2 = ptx::pack_f32x2(kWeightScale, kWeightScale);
    const uint64_t minus2 = ptx::pack_f32x2(-1.f, -1.f);
    uint32_t par = 0;  // of this tile's S and O, over all items
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity, unsigned code) -> bool {
      if (__all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag))) return true;
      atomicCAS(a.status, 0u, code);
      *abort_flag = 1;
      ok = false;
      return false;
    };
    for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x) {
      const int qp = item % a.n_qp, bh = item / a.n_qp, h = bh % a.Hq, b = bh / a.Hq;
      if (t >= tiles_of(qp)) continue;
      const int row = (qp * 2 + t) * kBM + row_in_tile;
      const float* v_undo = a.v_undo + (size_t)(b * a.Hkv + h / G) * a.n_kb;
      float m = -INFINITY, l = 0.f;
      uint64_t acc[NPV / 2];  // the row's output, two columns each
#pragma unroll
      for (int i = 0; i < NPV / 2; ++i) acc[i] = 0ull;
      for (int j = 0; j < nkv; ++j, par ^= 1u) {
        const float undo = __ldg(v_undo + j);  // (asked for early)
        if (!wait(&bars->s_full[t], par, 3u)) break;
        ptx::tc_fence_after();
        const int left = a.Sk - j * kBN;
        auto fetch = [&](int c, uint32_t(&s)[32]) { ptx::tmem_ld32(t_s + c * 32, s); };
        auto hide = [&](int c, uint32_t(&s)[32]) {
          if (left < kBN) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i >= left) s[i] = 0xff800000u;  // -inf
          }
        };
        auto top = [&](const uint32_t(&s)[32]) {
          float x[2] = {__uint_as_float(s[0]), __uint_as_float(s[1])};
#pragma unroll
          for (int i = 2; i < 30; i += 4) {
            x[0] = ptx::max3(x[0], __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
            x[1] = ptx::max3(x[1], __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
          }
          return fmaxf(ptx::max3(x[0], __uint_as_float(s[30]), __uint_as_float(s[31])), x[1]);
        };
        uint32_t s0[32], s1[32];
        fetch(0, s0);
        fetch(1, s1);
        ptx::tc_wait_ld();
        hide(0, s0);
        hide(1, s1);
        float mx = fmaxf(top(s0), top(s1));
        fetch(2, s0);
        fetch(3, s1);
        ptx::tc_wait_ld();
        hide(2, s0);
        hide(3, s1);
        mx = fmaxf(mx, fmaxf(top(s0), top(s1)));  // finite: every block has a key
        const float m_new = fmaxf(m, mx * sl2);
        if (__any_sync(0xffffffffu, m_new != m)) {
          const float alpha = fast_exp2(m - m_new);
          const uint64_t alpha2 = ptx::pack_f32x2(alpha, alpha);
#pragma unroll
          for (int i = 0; i < NPV / 2; ++i) acc[i] = ptx::mul_f32x2(acc[i], alpha2);
          l *= alpha;
          m = m_new;
        }
        const uint64_t neg_m2 = ptx::pack_f32x2(-m, -m);
        uint64_t lsum[2] = {0ull, 0ull};
        auto weights = [&](int c, const uint32_t(&s)[32]) {
          uint32_t w[2][16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const uint64_t x2 = ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1])), scale2, neg_m2);
            float x0, x1, h0, h1;
            ptx::unpack_f32x2(x2, x0, x1);
            const uint64_t p2 = ptx::mul_f32x2(ptx::pack_f32x2(fast_exp2(x0), fast_exp2(x1)), weight2);
            lsum[i & 1] = ptx::add_f32x2(lsum[i & 1], p2);
            ptx::unpack_f32x2(p2, x0, x1);
            w[0][i] = ptx::cvt_pack_f16(x0, x1);
            ptx::unpack_f16(w[0][i], h0, h1);
            ptx::unpack_f32x2(ptx::fma_f32x2(ptx::pack_f32x2(h0, h1), minus2, p2), x0, x1);
            w[1][i] = ptx::cvt_pack_f16(x0, x1);
          }
          ptx::tmem_st16(t_s + c * 32, w[0]);
          ptx::tmem_st16(t_s + c * 32 + 16, w[1]);
        };
        auto hand_over = [&](int half) {
          ptx::tc_wait_st();
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&bars->p_half[t][half]);
        };
        weights(2, s0);
        fetch(0, s0);
        weights(3, s1);
        fetch(1, s1);
        hand_over(1);
        ptx::tc_wait_ld();
        hide(0, s0);
        hide(1, s1);
        weights(0, s0);
        weights(1, s1);
        hand_over(0);
        float l0, l1;
        ptx::unpack_f32x2(ptx::add_f32x2(lsum[0], lsum[1]), l0, l1);
        l += l0 + l1;
        // the block's O joins the row's accumulators
        if (!wait(&bars->o_full[t], par, 5u)) break;
        ptx::tc_fence_after();
        const uint64_t undo2 = ptx::pack_f32x2(undo, undo);
#pragma unroll
        for (int c = 0; c < NPV / 16; ++c) {
          uint32_t first[16], second[16];
          ptx::tmem_ld16(t_o + c * 16, first);
          ptx::tmem_ld16(t_o + a.D + c * 16, second);  // (what columns from D on hold is not stored)
          ptx::tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 8; ++i)
            acc[c * 8 + i] = ptx::fma_f32x2(
                ptx::add_f32x2(ptx::pack_f32x2(__uint_as_float(first[2 * i]), __uint_as_float(first[2 * i + 1])),
                               ptx::pack_f32x2(__uint_as_float(second[2 * i]), __uint_as_float(second[2 * i + 1]))),
                undo2, acc[c * 8 + i]);
        }
      }
      if (!ok) break;
      const float inv = 1.f / l;  // l >= the weight of the row's maximum
      float* orow = a.o + b * a.o_sb + (int64_t)row * a.o_ss + h * a.o_sh;
      if (row < a.Sq) {
#pragma unroll
        for (int c = 0; c < NPV / 4; ++c) {
          float x, y, z, w;
          ptx::unpack_f32x2(acc[2 * c], x, y);
          ptx::unpack_f32x2(acc[2 * c + 1], z, w);
          if (c * 4 < a.D) *reinterpret_cast<float4*>(orow + c * 4) = make_float4(x * inv, y * inv, z * inv, w * inv);
        }
        if (a.lse) a.lse[((int64_t)b * a.Hq + h) * a.Sq + row] = m * kLn2 + logf(l * (1.f / kWeightScale));
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

template <int NPV>
int launch_t(const dt_sdpa_params& p, const F32PairScratch& w, cudaStream_t stream) {
  PairSplitArgs sp{};
  sp.per_row = p.D / 8;
  sp.flags = w.flags;
  const dt_tensor4* src[3] = {&p.q, &p.k, &p.v};
  CUtensorMap maps[3];
  for (int i = 0; i < 3; ++i) {
    const int S = i ? p.Sk : p.Sq, H = i ? p.Hkv : p.Hq, parts = i < 2 ? 3 : 2;
    PairSplitTensor& t = sp.t[i];
    t.src = static_cast<const float*>(src[i]->ptr);
    t.dst = reinterpret_cast<uint4*>(w.planes[i]);
    t.sb = src[i]->stride_b; t.ss = src[i]->stride_s; t.sh = src[i]->stride_h;
    t.S = S; t.H = H;
    t.n_blk = (S + kBM - 1) / kBM;
    t.begin = sp.n_units;
    sp.n_units += (unsigned)((size_t)p.B * H * t.n_blk);
    t.end = sp.n_units;
    // Q and K: the parts as one more factor of the head axis, [B, S, 3 H, D]; V: side by side, [B, S, H, 2 D]
    const int heads = i < 2 ? 3 * H : H, width = i < 2 ? p.D : 2 * p.D;
    const dt_tensor4 view{w.planes[i], (int64_t)S * H * parts * p.D, (int64_t)H * parts * p.D, width};
    if (!make_bshd_tensor_map(&maps[i], view, p.B, S, heads, width, i < 2 ? DT_BF16 : DT_F16, kBM)) return DT_UNSUPPORTED;
  }
  PairArgs a{};
  a.status = device_status_word();
  if (!a.status) return DT_CUDA;
  // the powers of two behind V's parts, in the room that bf16 parts would take
  sp.v_undo = reinterpret_cast<float*>(w.planes[2] + (size_t)p.B * p.Sk * p.Hkv * p.D * 4);
  a.v_undo = sp.v_undo;
  a.n_kb = sp.t[2].n_blk;
  a.flags = w.flags;
  a.n_flags = w.n_flags;
  a.done = w.done;
  a.no_parts = w.no_parts;
  a.o = static_cast<float*>(p.o.ptr);
  a.lse = p.lse;
  a.o_sb = p.o.stride_b; a.o_ss = p.o.stride_s; a.o_sh = p.o.stride_h;
  a.Sq = p.Sq; a.Sk = p.Sk; a.Hq = p.Hq; a.Hkv = p.Hkv; a.D = p.D;
  a.n_qp = (p.Sq + 2 * kBM - 1) / (2 * kBM);
  a.n_items = a.n_qp * p.Hq * p.B;
  a.scale_log2 = p.scale * kLog2e;
  auto kern = f32_pair_kernel<NPV>;
  DT_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
  DT_CUDA_TRY(launch_behind(split_pair_kernel, dim3(w.n_flags), dim3(kSplitThreads), 0, stream, 1, sp));
  const int n_sm = device_sm_count();
  kern<<<a.n_items < n_sm ? a.n_items : n_sm, kThreads, kSmemBytes, stream>>>(maps[0], maps[1], maps[2], a, *w.v_parts);
  DT_CUDA_TRY(cudaGetLastError());
  return DT_OK;
}

}  // namespace

// Two tiles to a CTA where that pays: a block of two takes about 1.42 times as long as a block of one, and there are about half as many rounds
// over the SMs; what a call of few blocks gains does not make up for the launch more.  Single tiles / pairs, us in a graph: 1100 tokens,
// 10 heads of 40, 2 images (2 rounds or 1) 55.4 / 45.9; 2000 tokens (3 or 2) 125.3 / 117.8; 8 images, 8 heads: 640 tokens (3 or 2, 5 blocks)
// 55.3 / 56.9, 768 tokens 67.6 / 62.2, 1100 tokens (4 or 3) 111.9 / 118.4; one image, 2000 tokens, 8 heads (128 tiles, one round) 48 / 59.
// Below 512 keys the error is a few per cent larger than with bf16 parts, and above smaller (heads of 64, 128 keys: 1.70e-7 / 1.77e-7).
bool f32_pair_pays(const dt_sdpa_params& p) {
  if (p.D <= 32 || p.D > 64 || p.Sk < 512) return false;
  const double heads = (double)p.B * p.Hq, sms = device_sm_count(), blocks = (p.Sk + kBN - 1) / kBN;
  const double singles = ceil(heads * ((p.Sq + kBM - 1) / kBM) / sms), pairs = ceil(heads * ((p.Sq + 2 * kBM - 1) / (2 * kBM)) / sms);
  return (100 * singles - 142 * pairs) * blocks >= 100;
}

unsigned f32_pair_units(const dt_sdpa_params& p) {
  return (unsigned)p.B * ((unsigned)p.Hq * ((p.Sq + kBM - 1) / kBM) + 2u * p.Hkv * ((p.Sk + kBM - 1) / kBM));
}

int launch_f32_pair(const dt_sdpa_params& p, const F32PairScratch& w, cudaStream_t stream) {
  return p.D <= 48 ? launch_t<48>(p, w, stream) : launch_t<64>(p, w, stream);
}

}  // namespace dt

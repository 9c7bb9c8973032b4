// Flash-attention forward for sm_100a: TMA-staged Q/K/V tiles, tcgen05.mma with TMEM accumulators,
// warp-specialised online softmax.  Serves the diffusion shapes of the reference
// (Libraries/SwiftDiffusion/Sources/Models/Flux1.swift:224-232 joint attention, Wan.swift:95-131 video
// self-attention, UNetXL.swift:67-185 cross-attention) and the masked text encoders (an additive mask as 4th
// input, alone or with isCausal: Llama.swift:70-73, CLIPTextModel.swift:46-51): fp16/bf16 I/O, fp32 accumulation,
// head dim up to 256, grouped KV heads, optional bottom-right causal rule, BSHD strided views.
//
// One CTA = one (batch, head, pair of 128-row query tiles); at head dim 256 (AuraFlow.swift:358, Gemma3.swift:148,
// Qwen3_5.swift:59-82) one tile, because TMEM holds S and O of only one.  12 warps:
//   warp 0      TMA producer: Q tiles once, then K(j), V(j) blocks of 128 keys through a ring of slots
//   warp 1      MMA issuer (one elected lane): S_t = Q_t K(j)^T  (operands in shared memory) and
//               O_t += P_t V(j) (P read from TMEM, V from shared memory), interleaved over the two tiles so
//               that the tensor pipe works on one tile while the other tile's softmax runs
//   warp 2      TMEM allocation / release
//   warps 4-7   softmax of tile 0: one thread per query row; reads its S row from TMEM, keeps the running
//               max / sum, rescales O in TMEM only when the max grew by more than 2^8 (the final 1/l
//               normalisation makes the result independent of that choice), writes P as 16-bit back to
//               TMEM over the S columns, and at the end normalises O and stores it
//   warps 8-11  the same for tile 1 (at head dim 256 nothing)
// TMEM (512 columns x 128 lanes, fp32): S0 [0,128) S1 [128,256) O0 [256,256+D) O1 [256+D,256+2D).
// Every mbarrier wait is bounded; a wait that runs out stores a code into the device status word and the
// CTA unwinds (TMEM is released on that path too).
#include <stdlib.h>

#include <type_traits>

#include "sm100_ptx.cuh"

namespace dt {
namespace {

constexpr int kBM = 128;       // query rows per tile
constexpr int kBN = 128;       // keys per block
constexpr int kThreads = 384;
constexpr int kHalfBytes = 128 * 128;  // [128 rows][64 x 16-bit] = 16 KB, one TMA box
constexpr float kRescaleThreshold = 8.f;
constexpr int kMaxExtraOutputs = 7;
// every kPolyPeriod-th pair of exponentials is evaluated with the polynomial instead of MUFU.EX2 (1 of 16 pairs with
// period 16), where fewer instructions have been worth more than relief of the special-function unit
// (measured on B200, Flux shape, TFLOP/s: period 1 (all polynomial) 996, 2: 1066, 3: 1123, 4: 1140, 6: 1157, 8: 1149,
// 16: 1160, none: 1147; with the softmax and the MMA warps free-running, never waiting for each other, the same order; since whole blocks
// have a path without branches the joint attention takes 222.6 / 217.6 / 219.5 / 218.2 us with 4 / 8 / 16 / none)
#ifndef DT_POLY_PERIOD
#define DT_POLY_PERIOD 16
#endif
constexpr int kPolyPeriod = DT_POLY_PERIOD;

template <int D, bool kMask = false>
struct Cfg {
  // Query tiles per work item.  TMEM (512 columns) holds S (128 columns) and O (D columns) of two tiles up to
  // D = 128; at D = 256 it holds one tile, whose softmax is run by the first softmax warpgroup alone (the second
  // one idles), and the columns of the second tile's S hold a second S buffer of the same tile: the tensor pipe runs
  // P V(j-1) and Q K(j+1)^T while the softmax works on block j (per key block that tile has twice the tensor-core
  // work of a D = 128 tile under the same softmax, so one warpgroup keeps up).
  static constexpr int kTiles = D == 256 ? 1 : 2;
  static constexpr int kSoftmaxWarps = 4 * kTiles;
  // Registers of a loading or issuing and of a softmax thread.  With 208 the softmax loop spilt up to 37 (80 / 208 -> 56 / 224: joint attention
  // 218.3 -> 216.1 us, 2 x 4096 tokens, 20 heads of 64 260.8 -> 254.6).  With one tile warps 8 to 11 have nothing to do and need none of theirs: an
  // issuer that walks its loop with one lane spills at 56 (96 to 192 bytes at head dim 256, 0 to 12 with 80; cut calls of 64 spill 64
  // bytes, but with 72 / 216 they were 0.7 % slower), and the masked softmax still spilt at 224.  Before / now, us: chunk of 1777 x 5873
  // 120.5 -> 117.6, 8192 tokens, 12 heads 631.6 -> 625.5, masks of 1501 and 2766 tokens, 16 / 8 heads 50.8 -> 49.1 and 117.9 -> 117.0.
  static constexpr int kRegsLow = kTiles == 1 ? 80 : 56, kRegsHigh = kTiles == 1 ? 240 : 224, kRegsIdle = 24;
  static_assert(128 * (kRegsLow + kTiles * kRegsHigh + (2 - kTiles) * kRegsIdle) <= kThreads * 168, "more registers than the CTA is launched with");
  static constexpr int kHalves = D / 64;
  static constexpr int kTileBytes = kHalves * kHalfBytes;  // one Q tile / one K block / one V block
  // the masked variant gives 32 KB of the K/V ring to the second mask staging buffers (D = 256: two 64 KB slots,
  // one K and one V block in flight, and the mask buffers fit beside them)
  static constexpr int kSlots = D == 256 ? 2 : (D == 128 ? 4 : 8) - (kMask ? 32 * 1024 / kTileBytes : 0);
  static constexpr int kMaskBytes = kMask ? kSoftmaxWarps * 32 * 128 : 0;  // per softmax warp: 32 rows x 64 keys x 16-bit (one half block)
  static constexpr int kStageBytes = kSoftmaxWarps * 32 * 128;  // per softmax warp: 32 rows x 64 x 16-bit of O for the TMA store
  static constexpr int kQBufs = D == 64 ? 2 : 1;        // Q buffers: with D = 64 there is room to load the next item's Q early
  static constexpr int kQBytes = kQBufs * kTiles * kTileBytes;
  static constexpr int kRingBytes = kSlots * kTileBytes;
  static constexpr int kBarBytes = 512;
  static constexpr int kSmemBytes = kQBytes + kRingBytes + kStageBytes + kMaskBytes + kBarBytes + 1024;
  static constexpr uint32_t kTmemCols = 512;
  static constexpr uint32_t kColS0 = 0, kColS1 = 128, kColO0 = 256, kColO1 = 256 + D;  // (tile 1's columns: only with kTiles == 2)
  static constexpr uint32_t kColP0 = 384, kColP1 = 448;  // kAhead: the weights have columns of their own
};
static_assert(Cfg<256, true>::kSmemBytes <= 227 * 1024, "shared memory of the widest variant");

struct PrefillArgs {
  void* o;
  float* lse;
#ifdef DT_BRINGUP
  float* dbg;   // optional [2][128][128] fp32 dump of the first S block of CTA (0,0,0), or timeline stamps
  int options;  // bit 1: timeline probe of CTA 0 into dbg
#endif
  int64_t o_sb, o_ss, o_sh;
  unsigned int* status;
  int Sq, Sk, Hq, Hkv;
  float scale_log2;
  int is_causal;
  int window;         // sliding window W (0 = off): row i sees keys j > i + (Sk - Sq) - W
  const void* sinks;  // [Hq] attention sinks in the tensors' type, or null
  // additive mask [B or 1, Hq or 1, Sq, Sk] in the tensors' type (kernel variant kMask only): element strides,
  // 0 on a broadcast axis; rows are 16-byte aligned (base and strides multiples of 8 elements)
  const void* mask;
  int64_t m_sb, m_sh, m_sq;
  // one byte per (32 query rows x 64 keys) patch of the mask: non-zero when the patch holds a non-zero entry;
  // [mask batches][mask heads][n_rg row groups][n_kh key halves, padded to an even count]
  const unsigned char* mask_flags;
  int n_rg, n_kh;
  uint32_t* not_finite;  // kSplit: set when some O is an infinity or NaN, for the kernel behind
  float scale;  // the plain scale (scale_log2 = scale * log2(e)); the masked variant adds the mask in this domain
  int item_rows;          // query rows of a work item: a pair of tiles, or one tile where pairs would leave SMs idle
  int n_qpairs, n_items;  // work items = (batch, head, item_rows query rows)
  // Items in whole rounds over the grid: n_slots of them, of which the causal order may leave some empty.  The items from
  // n_slots on (fewer than one round) are pairs of tiles taken tile by tile; n_places counts those tiles too.
  int n_slots;
  int n_places;
  // The cut kernel: an item's K/V blocks are cut into n_splits runs, whose shares of the result go to `part`;
  // cut_combine_kernel puts them together.
  int n_splits;           // (times an item's K/V blocks below 2^31)
  float* part;            // [n_items * n_splits][kBM / 32][D + 2][32]: weights' maximum, their sum, O
  // variable-length batch (both null otherwise): packed rows, sequence s owns query rows [off_q[s], off_q[s+1])
  // and key rows [off_k[s], off_k[s+1]); the item's batch index is then the sequence
  const int32_t* off_q;
  const int32_t* off_k;
  // head-sharded mode: the same O tile is also stored into these views (other GPUs' output buffers, same
  // strides as o) with ordinary 16-byte stores
  void* extra_o[kMaxExtraOutputs];
  int n_extra;
  int d_real;  // the tensors' head dim (<= the kernel's D): TMA zero-fills the columns beyond it on load and clips them on store
  int cut_lets_next;  // the cut kernel: cut_combine_kernel may be brought in while it runs
};

struct Barriers {
  uint64_t q_full[2];
  uint64_t q_empty[2];
  uint64_t s_full[2];
  uint64_t o_full[2];  // all P*V of an item done: O may be read (separate from s_full so no barrier runs two phases ahead)
  uint64_t p_half[2][2];  // [tile][first / second 64 keys of P written]
  uint64_t kv_full[8];
  uint64_t kv_empty[8];
  // One tile per item, kAhead: completes once per P V of the tile.  Waited for before O is rescaled, where S being there does not say
  // that the previous block's P V has run.
  uint64_t pv_done[2];
  uint32_t tmem_base;
  int abort_flag;
};

template <typename T>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  if constexpr (std::is_same<T, __half>::value) {
    __half2 t = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
  } else {
    __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
  }
}

// S = Q K^T for one 128-row tile: both operands K-major with 128-byte swizzle, D/16 steps of k = 16.
// Descriptor start addresses advance by 32 B per step inside a 64-element half and by 16 KB to the next half.
template <int D>
__device__ __forceinline__ void issue_qk(bool on, uint32_t s_tmem, uint64_t q_desc, uint64_t k_desc, uint32_t idesc) {
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    const uint64_t o = (uint64_t)(((ks >> 2) * kHalfBytes + (ks & 3) * 32) >> 4);
    ptx::mma_ss_on(on, s_tmem, q_desc + o, k_desc + o, idesc, ks > 0 ? 1u : 0u);
  }
}

// O (+)= P V for one tile: P from TMEM (two 16-bit keys per 32-bit column, 8 columns per step), V is
// [key][d] = MN-major; one step consumes 16 keys = 2 KB of each 64-wide half.
__device__ __forceinline__ void issue_pv(bool on, uint32_t o_tmem, uint32_t p_tmem, uint64_t v_desc, uint32_t idesc,
                                         uint32_t accumulate, int k_begin, int k_end) {
  if (k_end - k_begin == 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int kk = k_begin + i;
      ptx::mma_ts_on(on, o_tmem, p_tmem + kk * 8, v_desc + (uint64_t)(kk * (2048 >> 4)), idesc, (kk > 0) ? 1u : accumulate);
    }
  } else {
#pragma unroll 1
    for (int kk = k_begin; kk < k_end; ++kk)
      ptx::mma_ts_on(on, o_tmem, p_tmem + kk * 8, v_desc + (uint64_t)(kk * (2048 >> 4)), idesc, (kk > 0) ? 1u : accumulate);
  }
}

// The same for the weights of the kSplit variant: their high parts and, 64 columns further, what those leave over.
template <bool kSplit>
__device__ __forceinline__ void issue_pv_parts(bool on, uint32_t o_tmem, uint32_t p_tmem, uint64_t v_desc, uint32_t idesc,
                                               uint32_t accumulate, int k_begin, int k_end) {
  issue_pv(on, o_tmem, p_tmem, v_desc, idesc, accumulate, k_begin, k_end);
  if constexpr (kSplit) {
#pragma unroll 1
    for (int kk = k_begin; kk < k_end; ++kk)
      ptx::mma_ts_on(on, o_tmem, p_tmem + 64 + kk * 8, v_desc + (uint64_t)(kk * (2048 >> 4)), idesc, 1u);
  }
}

// Experiment builds (-DDT_PREFILL_OPTIONS=bits, never the product): bit 3 = the softmax warps skip the exponentials;
// bit 4 = nobody waits for S or P (free-running softmax and MMA: garbage results, the pure throughput of each
// side); bit 5 = the softmax warps skip the row maximum; bit 6 (with bit 4) = the softmax warps do nothing per block.  Bring-up builds: a.options bit 1 = timeline probe of CTA 0.
#ifndef DT_PREFILL_OPTIONS
#define DT_PREFILL_OPTIONS 0
#endif
#define DT_OPT(bit) ((DT_PREFILL_OPTIONS & (bit)) != 0)
#ifdef DT_BRINGUP
__device__ __forceinline__ void stamp(const PrefillArgs& a, int slot) {
  if ((a.options & 2) && a.dbg != nullptr && blockIdx.x == 0 && slot < 4096)
    reinterpret_cast<unsigned long long*>(a.dbg)[slot] = ptx::globaltimer_ns();
}
#else
__device__ __forceinline__ void stamp(const PrefillArgs&, int) {}
#endif

// First of an item's n K/V blocks that belongs to its run c
__device__ __forceinline__ int cut_at(const PrefillArgs& a, int n, int c) { return n * c / a.n_splits; }

// K/V blocks from key 0 to the last one that the query rows below `end` may see (not for variable lengths)
__device__ __forceinline__ int blocks_to(const PrefillArgs& a, int end) {
  int nkv = (a.Sk + kBN - 1) / kBN;
  if (a.is_causal) {
    const long long lim = (long long)min(a.Sq, end) + (a.Sk - a.Sq);
    nkv = max(1, min(nkv, (int)((max(0LL, min((long long)a.Sk, lim)) + kBN - 1) / kBN)));
  }
  return nkv;
}

// (query tile (pair), batch x head) at a place of the processing order: query rows fastest, so that CTAs running at the
// same time share one head's K/V in L2; under the causal rule heaviest first (all heads' last rows, then the ones before,
// ...), because an item's work grows with its query position.
__device__ __forceinline__ void place_of(const PrefillArgs& a, int order, int& qt, int& bh) {
  if (a.is_causal) {
    const int nbh = a.n_items / a.n_qpairs, level = order / nbh;
    bh = order - level * nbh;
    qt = a.n_qpairs - 1 - level;
  } else {
    bh = order / a.n_qpairs;
    qt = order - bh * a.n_qpairs;
  }
}

// Run c's share of 32 rows (one softmax warp's).
template <int D>
__device__ __forceinline__ float* share_of(const PrefillArgs& a, int run, int unit) {
  return a.part + ((size_t)run * (kBM / 32) + unit) * (size_t)((D + 2) * 32);
}

// Puts the shares of cut items together, added in the order of the keys: one block per 32 rows of an item and 64 columns.
// (As the last step of the attention kernel itself, by the warp that arrives last, it took longer than the cut saved: 256
// columns from three shares are a chain of two dozen L2 round trips for one warp.)
// Bound: the latency of L2; a thread keeps eight shares' loads in flight.
template <typename T, int D>
__global__ void __launch_bounds__(256) cut_combine_kernel(const PrefillArgs a) {
  __shared__ __align__(16) uint16_t rows[32][64 + 8];
  ptx::wait_for_previous();
  ptx::let_next_start();
  const int item = blockIdx.x / (kBM / 32), unit = blockIdx.x - item * (kBM / 32), col0 = blockIdx.y * 64;
  const int r = threadIdx.x & 31, cg = threadIdx.x >> 5;  // two groups of four columns per thread: cg and cg + 8
  int qt, bh;
  place_of(a, item, qt, bh);
  const int h = bh % a.Hq, b = bh / a.Hq, row0 = qt * kBM + unit * 32, row = row0 + r;
  if (row0 >= a.Sq) return;
  const int n = blocks_to(a, (qt + 1) * kBM);
  // with fewer blocks than runs some of them are empty: run i of the others
  const int n_shares = min(n, a.n_splits);
  auto at = [&](int i) { return share_of<D>(a, item * a.n_splits + (n < a.n_splits ? ((i + 1) * a.n_splits - 1) / n : i), unit); };
  float m = -INFINITY;
#pragma unroll 8
  for (int i = 0; i < n_shares; ++i) m = fmaxf(m, __ldg(at(i) + r));
  float l = 0.f;
  float4 acc[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll 8
  for (int i = 0; i < n_shares; ++i) {
    const float* sh = at(i);
    const float mc = __ldg(sh + r), lc = __ldg(sh + 32 + r);
    float4 x[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) x[g] = __ldg(reinterpret_cast<const float4*>(sh + 64) + (col0 / 4 + cg + 8 * g) * 32 + r);
    // A share that saw no key counts nothing, but it is not left out: a row whose scores are all NaN has no maximum either
    // (a maximum ignores NaN), and its NaN sum and O must reach the result as they do in a call that is not cut.
    const float f = mc == -INFINITY ? 0.f : fast_exp2(mc - m);
    l = fmaf(f, lc, l);
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      acc[g].x = fmaf(f, x[g].x, acc[g].x);
      acc[g].y = fmaf(f, x[g].y, acc[g].y);
      acc[g].z = fmaf(f, x[g].z, acc[g].z);
      acc[g].w = fmaf(f, x[g].w, acc[g].w);
    }
  }
  if (a.sinks) {  // as in the attention kernel's epilogue
    const float sl = to_float(reinterpret_cast<const T*>(a.sinks)[h]) * kLog2e;
    if (m == -INFINITY) {
      m = sl;
      l = 1.f;
    } else {
      l += fast_exp2(sl - m);
    }
  }
  const float inv = (l > 0.f && m != -INFINITY) ? 1.f / l : 0.f;
  if (a.lse && cg == 0 && col0 == 0 && row < a.Sq)
    a.lse[((int64_t)b * a.Hq + h) * a.Sq + row] = (l > 0.f && m != -INFINITY) ? m * kLn2 + logf(l) : -INFINITY;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    uint2 pk;
    pk.x = pack_pair<T>(acc[g].x * inv, acc[g].y * inv);
    pk.y = pack_pair<T>(acc[g].z * inv, acc[g].w * inv);
    *reinterpret_cast<uint2*>(&rows[r][(cg + 8 * g) * 4]) = pk;
  }
  __syncthreads();
  T* obase = reinterpret_cast<T*>(a.o) + (int64_t)b * a.o_sb + (int64_t)h * a.o_sh + col0;
  const int rr = threadIdx.x >> 3, ch = threadIdx.x & 7;
  if (row0 + rr < a.Sq && col0 + ch * 8 < a.d_real)
    *reinterpret_cast<uint4*>(obase + (int64_t)(row0 + rr) * a.o_ss + ch * 8) = *reinterpret_cast<const uint4*>(&rows[rr][ch * 8]);
}

// Pre-pass of the masked variant: which (32 rows x 64 keys) patches of the additive mask hold anything but zeros.
// A padding mask is zero almost everywhere, and the attention kernel skips the patches flagged zero altogether.
// One warp per patch, 8 lanes on a row's 128 contiguous bytes; entries beyond Sq / Sk are never read.
__global__ void __launch_bounds__(256) mask_flags_kernel(const unsigned short* __restrict__ mask, int64_t m_sb, int64_t m_sh,
                                                         int64_t m_sq, int Hm, int Sq, int Sk, int n_rg, int n_kh,
                                                         int is_causal, unsigned char* __restrict__ flags) {
  ptx::wait_for_previous();
  ptx::let_next_start();
  const int lane = threadIdx.x & 31;
  const int kh = blockIdx.x * 8 + (threadIdx.x >> 5), rg = blockIdx.y, bh = blockIdx.z;
  if (kh >= n_kh) return;
  const int mb = bh / Hm, mh = bh - mb * Hm;
  const unsigned short* base = mask + mb * m_sb + mh * m_sh;
  const int key = kh * 64 + (lane & 7) * 8;
  uint32_t any = 0u;
  // under the causal rule the attention kernel never visits a patch that lies wholly beyond its rows' last visible key
  const bool visited = !is_causal || (long long)kh * 64 <= (long long)rg * 32 + 31 + (Sk - Sq);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = rg * 32 + i * 4 + (lane >> 3);
    if (!visited || row >= Sq || key >= Sk) continue;
    const unsigned short* src = base + (int64_t)row * m_sq + key;
    if (key + 8 <= Sk) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
      any |= v.x | v.y | v.z | v.w;
    } else {
      for (int e = 0; key + e < Sk; ++e) any |= src[e];
    }
  }
  const bool nz = __any_sync(0xffffffffu, any != 0u);
  if (lane == 0) flags[((int64_t)bh * n_rg + rg) * n_kh + kh] = nz ? 1 : 0;
}

// Pre-pass for masks whose rows do not start on 16 bytes (a dense [S, S] mask of an odd S): the same flags, and the
// flagged patches copied to rows of `ld` entries, a multiple of 8 (patches of zeros are never read, so they are not
// written either).  One warp per patch, two entries of a row per lane, the whole patch in 32 registers.
__global__ void __launch_bounds__(256) mask_repack_kernel(const unsigned short* __restrict__ mask, int64_t m_sb, int64_t m_sh,
                                                          int64_t m_sq, int Hm, int Sq, int Sk, int n_rg, int n_kh,
                                                          int is_causal, unsigned char* __restrict__ flags,
                                                          unsigned short* __restrict__ copy, int ld,
                                                          uint32_t* __restrict__ not_finite) {
  ptx::wait_for_previous();
  ptx::let_next_start();
  const int lane = threadIdx.x & 31;
  const int kh = blockIdx.x * 8 + (threadIdx.x >> 5), rg = blockIdx.y, bh = blockIdx.z;
  if (threadIdx.x == 0 && blockIdx.x == 0 && rg == 0 && bh == 0) *not_finite = 0u;
  if (kh >= n_kh) return;
  const int mb = bh / Hm, mh = bh - mb * Hm;
  const unsigned short* base = mask + mb * m_sb + mh * m_sh;
  const int k0 = kh * 64 + lane, k1 = k0 + 32;
  uint32_t v[32], any = 0u;
  const bool visited = !is_causal || (long long)kh * 64 <= (long long)rg * 32 + 31 + (Sk - Sq);
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int row = rg * 32 + i;
    const unsigned short* src = base + (int64_t)row * m_sq;
    v[i] = 0u;
    if (visited && row < Sq) {
      if (k0 < Sk) v[i] = __ldg(src + k0);
      if (k1 < Sk) v[i] |= (uint32_t)__ldg(src + k1) << 16;
    }
    any |= v[i];
  }
  const bool nz = __any_sync(0xffffffffu, any != 0u);
  if (lane == 0) flags[((int64_t)bh * n_rg + rg) * n_kh + kh] = nz ? 1 : 0;
  if (!nz) return;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int row = rg * 32 + i;
    if (row >= Sq) break;
    unsigned short* dst = copy + ((int64_t)bh * Sq + row) * ld;
    if (k0 < Sk) dst[k0] = (unsigned short)v[i];
    if (k1 < Sk) dst[k1] = (unsigned short)(v[i] >> 16);
  }
}

// 16-bit pair -> two floats (the mask is stored in the tensors' type)
template <typename T>
__device__ __forceinline__ float2 unpack_pair(uint32_t x) {
  if constexpr (std::is_same<T, __half>::value) return __half22float2(*reinterpret_cast<const __half2*>(&x));
  else return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x));
}

// kForm: see launch_t
template <typename T, int D, bool kMask, bool kSplit, bool kCut, int kForm>
__global__ void __launch_bounds__(kThreads, 1)
prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o,
                       const PrefillArgs a) {
  using C = Cfg<D, kMask>;
  constexpr int kBf16 = std::is_same<T, __half>::value ? 0 : 1;
  constexpr bool kLong = kForm > 0, kMayEarly = kForm > 1;
  constexpr bool kAhead = kLong && D == 64 && !kMask;  // columns for P beside S and O: see launch_t
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t q_smem = base;
  const uint32_t ring_smem = base + C::kQBytes;
  const uint32_t stage_smem = base + C::kQBytes + C::kRingBytes;
  // masked variant: [second mask staging buffers] between the O staging rows and the barriers
  const uint32_t mask_smem = stage_smem + C::kStageBytes;
  Barriers* bars = reinterpret_cast<Barriers*>(base_ptr + C::kQBytes + C::kRingBytes + C::kStageBytes + C::kMaskBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = a.Hq / a.Hkv;

  // Work items (batch, head, item_rows query rows).  The CTA is persistent: it takes items blockIdx.x, + gridDim.x, ...
  struct Item {
    int b, h, kvh, q0, nkv, j0;  // K/V blocks j0 .. j0 + nkv - 1; nkv == 0: nothing to do (q0 beyond the sequence)
    int sq, sk, off;             // rows of this (batch item | sequence); causal: key j visible to query i iff j <= i + off
    int qrow, krow;              // first packed row of the sequence (0 unless variable-length)
    bool two;
  };
  auto item_at = [&](int order, int tile) {  // tile: one of the pair's tiles, or -1 for the whole item
    Item it;
    int qt, bh;
    place_of(a, order, qt, bh);
    it.h = bh % a.Hq;
    it.b = bh / a.Hq;
    it.kvh = it.h / G;
    it.q0 = qt * a.item_rows + max(tile, 0) * kBM;
    it.sq = a.Sq;
    it.sk = a.Sk;
    it.qrow = it.krow = 0;
    if (a.off_q) {
      it.qrow = a.off_q[it.b];
      it.krow = a.off_k[it.b];
      it.sq = a.off_q[it.b + 1] - it.qrow;
      it.sk = a.off_k[it.b + 1] - it.krow;
      it.b = 0;
    }
    it.off = it.sk - it.sq;
    it.two = C::kTiles == 2 && tile < 0 && a.item_rows > kBM && it.q0 + kBM < it.sq;
    it.j0 = 0;
    if (it.q0 >= it.sq) {  // a pair without a second tile, or a sequence shorter than the longest one
      it.nkv = 0;
      return it;
    }
    int nkv = max(1, (it.sk + kBN - 1) / kBN);  // a sequence without keys still runs one (fully masked) block
    if (a.is_causal) nkv = blocks_to(a, it.q0 + (it.two ? 2 : 1) * kBM);  // (never together with variable lengths)
    if (a.window > 0) {  // blocks entirely below the first row's window are never visited
      const long long lo = (long long)it.q0 + it.off - a.window + 1;
      it.j0 = (int)min((long long)(nkv - 1), max(0LL, lo) / kBN);
    }
    it.nkv = nkv - it.j0;
    return it;
  };
  // Whole items, then single tiles: place `item` of the CTAs' turns.  Under the causal rule the turns go forwards over the CTAs in even
  // rounds and backwards in odd ones, so that every CTA's items add up to about the same number of K/V blocks.
  auto decode_item = [&](int item) {
    int order = item;
    if (a.is_causal) {
      const int round = item / (int)gridDim.x;
      int pos = item - round * (int)gridDim.x;
      if (round & 1) pos = (int)gridDim.x - 1 - pos;
      order = round * (int)gridDim.x + pos;
    }
    int tile = -1;
    if constexpr (C::kTiles == 2) {
      if (order >= a.n_slots) {  // single tiles (under the causal rule in a round that goes forwards)
        tile = (order - a.n_slots) & 1;
        order = a.n_slots + ((order - a.n_slots) >> 1);
      }
    }
    if (order >= a.n_items) {  // a slot of the last, incomplete round without an item
      return Item{};
    }
    return item_at(order, tile);
  };
  // This CTA's work in turn: its whole items and then a single tile, or (cut) runs of items' blocks.  A kernel of its own
  // for cut calls, because what they need costs the others up to 1 us at the start and 2 % in the loops of the 256-wide variant.
  auto next_work = [&](int& next, Item& w) -> bool {
    if constexpr (kCut) {
      while (next < a.n_items * a.n_splits) {
        const int order = next / a.n_splits, c = next - order * a.n_splits;
        next += gridDim.x;
        w = item_at(order, -1);
        const int n = w.nkv;
        w.j0 = cut_at(a, n, c);
        w.nkv = cut_at(a, n, c + 1) - w.j0;
        if (w.nkv > 0) return true;  // (empty: an item with fewer blocks than runs)
      }
      return false;
    } else {
      while (next < a.n_places) {
        w = decode_item(next);
        next += gridDim.x;
        if (w.nkv > 0) return true;
      }
      return false;
    }
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&bars->q_full[i], 1);
      ptx::mbar_init(&bars->q_empty[i], 1);
    }
    for (int t = 0; t < 2; ++t) {
      ptx::mbar_init(&bars->s_full[t], 1);
      ptx::mbar_init(&bars->o_full[t], 1);
      ptx::mbar_init(&bars->p_half[t][0], 4);  // one arrival per softmax warp
      ptx::mbar_init(&bars->p_half[t][1], 4);
    }
    for (int i = 0; i < C::kSlots; ++i) {
      ptx::mbar_init(&bars->kv_full[i], 1);
      ptx::mbar_init(&bars->kv_empty[i], 1);
    }
    for (int t = 0; t < 2; ++t) ptx::mbar_init(&bars->pv_done[t], 1);
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 2) {
    ptx::tmem_alloc(&bars->tmem_base, C::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile int* abort_flag = &bars->abort_flag;
  ptx::wait_for_previous();
  // (Calls of several rounds do not overlap their neighbours: 32 / 8 heads of 128 under an unaligned mask, 1001 tokens 47.4 -> 45.7 us
  // with it, but 1501 tokens 62.1 -> 65.0 and 2047 tokens 76.5 -> 82.4.)
  if (kCut ? a.cut_lets_next != 0 : a.n_items <= (int)gridDim.x) ptx::let_next_start();

  // Register budget: the data-movement warpgroup gives registers back, the softmax warpgroups take them.
  // (Each setmaxnreg must dominate the code it governs, hence the nesting.)
  if (warp < 4) {
    ptx::setmaxnreg_dec<C::kRegsLow>();
    if (warp == 0) {
      // =========================== TMA producer ===========================
      if (lane == 0) {
        ptx::prefetch_tensormap(&map_q);
        ptx::prefetch_tensormap(&map_k);
        ptx::prefetch_tensormap(&map_v);
        ptx::prefetch_tensormap(&map_o);
        int ring_it = 0;  // K/V ring position, continues across items
        int n_item = 0;
        bool ok = true;
        auto load_kv = [&](const Item& w, int j, bool is_v) {
          const int slot = ring_it % C::kSlots, use = ring_it / C::kSlots;
          if (use > 0 && !ptx::mbar_wait(&bars->kv_empty[slot], (use - 1) & 1, abort_flag)) {
            atomicCAS(a.status, 0u, 2u);
            *abort_flag = 1;
            return false;
          }
          ptx::mbar_arrive_expect_tx(&bars->kv_full[slot], (uint32_t)C::kTileBytes);
#pragma unroll
          for (int hf = 0; hf < C::kHalves; ++hf)
            ptx::tma_load_4d(base_ptr + C::kQBytes + slot * C::kTileBytes + hf * kHalfBytes, is_v ? &map_v : &map_k,
                             &bars->kv_full[slot], hf * 64, w.kvh, w.krow + (w.j0 + j) * kBN, w.b);
          ++ring_it;
          return true;
        };
        int walk = blockIdx.x;
        Item w, nx;
        bool more_work = next_work(walk, nx);
        for (; more_work && ok; ++n_item) {
          w = nx;
          // first K/V block of this item may be fetched while the previous item still owns the Q buffers
          // (one tile per item: the MMA warp consumes K(0), K(1), V(0), K(2), V(1), ..., and the ring follows that order)
          if constexpr (C::kTiles == 1) ok = load_kv(w, 0, false) && (w.nkv == 1 || load_kv(w, 1, false));
          else ok = load_kv(w, 0, false) && load_kv(w, 0, true);
          if (!ok) break;
          const int qb = n_item % C::kQBufs, quse = n_item / C::kQBufs;
          if (quse > 0 && !ptx::mbar_wait(&bars->q_empty[qb], (quse - 1) & 1, abort_flag)) {
            atomicCAS(a.status, 0u, 2u);
            *abort_flag = 1;
            break;
          }
          stamp(a, 16 * n_item + 0);
          ptx::mbar_arrive_expect_tx(&bars->q_full[qb], (uint32_t)((w.two ? 2 : 1) * C::kTileBytes));
          for (int t = 0; t < (w.two ? 2 : 1); ++t)
#pragma unroll
            for (int hf = 0; hf < C::kHalves; ++hf)
              ptx::tma_load_4d(base_ptr + (qb * C::kTiles + t) * C::kTileBytes + hf * kHalfBytes, &map_q, &bars->q_full[qb], hf * 64,
                               w.h, w.qrow + w.q0 + t * kBM, w.b);
          // The Q tiles of the NEXT item are pulled into L2 now: their rows are 256-byte pieces a whole
          // token stride apart (slow to gather from HBM), and the real load sits on the critical path
          // between two items.
          more_work = next_work(walk, nx);  // (behind this item's own first loads: finding it takes a few hundred cycles)
          if (more_work) {
            for (int t = 0; t < (nx.two ? 2 : 1); ++t)
#pragma unroll
              for (int hf = 0; hf < C::kHalves; ++hf)
                ptx::tma_prefetch_l2_4d(&map_q, hf * 64, nx.h, nx.qrow + nx.q0 + t * kBM, nx.b);
          }
          if constexpr (C::kTiles == 1) {
            for (int j = 0; j < w.nkv && ok; ++j) ok = load_kv(w, j, true) && (j + 2 >= w.nkv || load_kv(w, j + 2, false));
          } else {
            for (int j = 1; j < w.nkv && ok; ++j) ok = load_kv(w, j, false) && load_kv(w, j, true);
          }
        }
      }
    } else if (warp == 1) {
      // =========================== MMA issuer ===========================
      // The lane that issues is the elected one, which keeps the operands in uniform registers: behind "lane == 0" each MMA took at
      // least 45 cycles to issue, where one of N = 64 with its rows in TMEM runs for 32 (one elected lane or the whole warp in step:
      // 10).  Two text prompts of 77 tokens, 4 images of 9216 tokens, 20 heads of 64: 118.0 -> 108.5 us; 300 tokens, 10 heads 8.8 -> 8.6;
      // window of 300, 5000 tokens, 16 / 4 heads 47.0 -> 44.4.  The whole warp walks the loop at head dims 64 and 128 (a window of 300,
      // 2100 tokens, heads of 64: 19.7 us, one lane 20.2; 4096 tokens, 20 heads of 64: 273.6 and 277.3), one lane in cut calls of 64
      // (8 heads, 128 x 16000: 25.6, the warp 26.4) and at 256, where the two are alike.
      constexpr bool kWarpIssue = D == 128 || (D == 64 && !kCut);
      if (kWarpIssue || ptx::elect_one()) {
        const bool on = kWarpIssue ? ptx::elect_one() : true;
        constexpr uint32_t idesc_qk = ptx::make_idesc_f16(kBf16, kBM, kBN, 0, 0);
        constexpr uint32_t idesc_pv = ptx::make_idesc_f16(kBf16, kBM, D, 0, 1);
        // Descriptors differ only in the 14-bit start-address field, so stepping through a tile is one add.
        const uint64_t desc_k_major = ptx::make_smem_desc_sw128(0, 16, 1024);            // Q, K
        const uint64_t desc_mn_major = ptx::make_smem_desc_sw128(0, kHalfBytes, 1024);   // V
        const uint64_t qd_base = desc_k_major | (uint64_t)((q_smem & 0x3FFFFu) >> 4);
        const uint64_t ring_k = desc_k_major | (uint64_t)((ring_smem & 0x3FFFFu) >> 4);
        const uint64_t ring_v = desc_mn_major | (uint64_t)((ring_smem & 0x3FFFFu) >> 4);
        const uint32_t s0 = tmem + C::kColS0, s1 = tmem + C::kColS1, o0 = tmem + C::kColO0, o1 = tmem + C::kColO1;
        int slot = 0, par = 0;     // ring position of the next K/V block to consume
        uint32_t pph0 = 0, pph1 = 0;  // phases of the P hand-off barriers, per tile
        int n_item = 0;
        bool ok = true;
        auto fail = [&](unsigned code) {
          if (on) atomicCAS(a.status, 0u, code);
          *abort_flag = 1;
          ok = false;
        };
        auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
          const bool done = ptx::mbar_wait(bar, parity, abort_flag);
          return kWarpIssue ? __all_sync(0xffffffffu, done) : done;
        };
        auto advance = [&]() {
          if (++slot == C::kSlots) { slot = 0; par ^= 1; }
        };
        int walk = blockIdx.x;
        Item w;
        for (; ok && next_work(walk, w); ++n_item) {
          const int ntile = w.two ? 2 : 1;
          const int qb = n_item % C::kQBufs;
          const uint64_t qd0 = qd_base + (uint64_t)(qb * C::kTiles * (C::kTileBytes >> 4));
          const uint64_t qd1 = qd0 + (uint64_t)(C::kTileBytes >> 4);
          if constexpr (C::kTiles == 1) {
            // One tile per item (D = 256): S is double-buffered in TMEM (the columns a second tile would use), so that
            // Q K(j+1)^T and P V(j-1) run while the softmax works on block j.  Order on the tensor pipe:
            // QK(0) QK(1) | PV(0) QK(2) | PV(1) QK(3) | ...
            if (!wait(&bars->q_full[qb], (n_item / C::kQBufs) & 1)) {
              fail(1u);
              break;
            }
            auto qk = [&](int i) -> bool {  // S[i & 1] = Q K(i)^T from the ring's next slot
              if (!wait(&bars->kv_full[slot], par)) {
                fail(1u);
                return false;
              }
              ptx::tc_fence_after();
              issue_qk<D>(on, (i & 1) ? s1 : s0, qd0, ring_k + (uint64_t)(slot * (C::kTileBytes >> 4)), idesc_qk);
              ptx::tc_commit_on(on, &bars->s_full[i & 1]);
              ptx::tc_commit_on(on, &bars->kv_empty[slot]);
              if (i == w.nkv - 1) ptx::tc_commit_on(on, &bars->q_empty[qb]);  // Q is no longer needed: the next item may load its own
              advance();
              return true;
            };
            if (!qk(0) || (w.nkv > 1 && !qk(1))) break;
            for (int j = 0; j < w.nkv && ok; ++j) {
              const int b = j & 1;
              const uint32_t sb = b ? s1 : s0;
              uint32_t& pph = b ? pph1 : pph0;
              const int valid = max(16, min(kBN, w.sk - (w.j0 + j) * kBN));
              const int ksteps = (valid + 15) >> 4;
              const int k_mid = min(ksteps, 4);
              if (!wait(&bars->kv_full[slot], par)) {  // V(j)
                fail(1u);
                break;
              }
              const int slot_v = slot;
              const uint64_t vd = ring_v + (uint64_t)(slot_v * (C::kTileBytes >> 4));
              advance();
              if (!wait(&bars->p_half[b][0], pph)) { fail(4u); break; }
              ptx::tc_fence_after();
              issue_pv_parts<kSplit>(on, o0, sb, vd, idesc_pv, j > 0 ? 1u : 0u, 0, k_mid);
              if (!wait(&bars->p_half[b][1], pph)) { fail(4u); break; }
              pph ^= 1;
              ptx::tc_fence_after();
              issue_pv_parts<kSplit>(on, o0, sb, vd, idesc_pv, 1u, k_mid, ksteps);
              ptx::tc_commit_on(on, &bars->kv_empty[slot_v]);
              ptx::tc_commit_on(on, &bars->pv_done[0]);
              if (j + 2 < w.nkv && !qk(j + 2)) break;  // overwrites the S / P columns the P V above has just read
              if (j + 1 == w.nkv) ptx::tc_commit_on(on, &bars->o_full[0]);
            }
            continue;
          }
          // ---- S_t(0) = Q_t K(0)^T ----
          if (on) stamp(a, 16 * n_item + 5);
          if (!wait(&bars->q_full[qb], (n_item / C::kQBufs) & 1)) {
            fail(1u);
            break;
          }
          if (on) stamp(a, 16 * n_item + 6);
          if (!wait(&bars->kv_full[slot], par)) {
            fail(1u);
            break;
          }
          if (on) stamp(a, 16 * n_item + 1);
          ptx::tc_fence_after();
          {
            const uint64_t kd = ring_k + (uint64_t)(slot * (C::kTileBytes >> 4));
            issue_qk<D>(on, s0, qd0, kd, idesc_qk);
            ptx::tc_commit_on(on, &bars->s_full[0]);
            if (ntile == 2) {
              issue_qk<D>(on, s1, qd1, kd, idesc_qk);
              ptx::tc_commit_on(on, &bars->s_full[1]);
            }
            ptx::tc_commit_on(on, &bars->kv_empty[slot]);
            if (w.nkv == 1) ptx::tc_commit_on(on, &bars->q_empty[qb]);  // Q is no longer needed: the next item may load its own
            advance();
          }
          for (int j = 0; j < w.nkv && ok; ++j) {
            const int slot_v = slot, par_v = par;
            advance();
            const int slot_k = slot, par_k = par;
            const bool more = j + 1 < w.nkv;
            if (more) advance();
            const int valid = max(16, min(kBN, w.sk - (w.j0 + j) * kBN));  // at least one 16-key step (P = 0 there if sk = 0)
            const int ksteps = (valid + 15) >> 4;
            const int k_mid = min(ksteps, 4);
            if (!wait(&bars->kv_full[slot_v], par_v) ||
                (more && !wait(&bars->kv_full[slot_k], par_k))) {
              fail(1u);
              break;
            }
            const uint64_t vd = ring_v + (uint64_t)(slot_v * (C::kTileBytes >> 4));
            const uint64_t kd = ring_k + (uint64_t)(slot_k * (C::kTileBytes >> 4));
            const bool last_qk = more && (j + 2 == w.nkv);  // the QK issued in this iteration is the item's last
            if constexpr (kAhead) {
#pragma unroll
              for (int t = 0; t < 2; ++t) {
                if (t == 1 && ntile == 1) break;
                uint32_t& pph = t ? pph1 : pph0;
                const uint32_t o_t = t ? o1 : o0, p_t = tmem + (t ? C::kColP1 : C::kColP0);
                const bool last_tile = t == ntile - 1;
                if (!wait(&bars->p_half[t][0], pph)) { fail(4u); break; }
                ptx::tc_fence_after();
                issue_pv(on, o_t, p_t, vd, idesc_pv, j > 0 ? 1u : 0u, 0, k_mid);
                if (more) {
                  issue_qk<D>(on, t ? s1 : s0, t ? qd1 : qd0, kd, idesc_qk);
                  ptx::tc_commit_on(on, &bars->s_full[t]);
                  if (last_tile) {
                    ptx::tc_commit_on(on, &bars->kv_empty[slot_k]);
                    if (last_qk) ptx::tc_commit_on(on, &bars->q_empty[qb]);
                  }
                }
                if (!wait(&bars->p_half[t][1], pph)) { fail(4u); break; }
                pph ^= 1;
                ptx::tc_fence_after();
                issue_pv(on, o_t, p_t, vd, idesc_pv, 1u, k_mid, ksteps);
                ptx::tc_commit_on(on, &bars->pv_done[t]);
                if (!more) ptx::tc_commit_on(on, &bars->o_full[t]);
                if (last_tile) ptx::tc_commit_on(on, &bars->kv_empty[slot_v]);
              }
              continue;
            }
            // ---- tile 0 ----  (P arrives in two halves of 64 keys so P*V starts while the softmax still runs)
            if (!DT_OPT(16) && !wait(&bars->p_half[0][0], pph0)) { fail(4u); break; }
            if (j == 0 && on) stamp(a, 16 * n_item + 2);
            ptx::tc_fence_after();
            issue_pv_parts<kSplit>(on, o0, s0, vd, idesc_pv, j > 0 ? 1u : 0u, 0, k_mid);
            if (!DT_OPT(16) && !wait(&bars->p_half[0][1], pph0)) { fail(4u); break; }
            pph0 ^= 1;
            ptx::tc_fence_after();
            issue_pv_parts<kSplit>(on, o0, s0, vd, idesc_pv, 1u, k_mid, ksteps);
            if (ntile == 1) ptx::tc_commit_on(on, &bars->kv_empty[slot_v]);
            if (more) issue_qk<D>(on, s0, qd0, kd, idesc_qk);
            ptx::tc_commit_on(on, more ? &bars->s_full[0] : &bars->o_full[0]);  // next S ready, or (last block) O complete
            if (!more && on) stamp(a, 16 * n_item + 3);
            if (more && ntile == 1) {
              ptx::tc_commit_on(on, &bars->kv_empty[slot_k]);
              if (last_qk) ptx::tc_commit_on(on, &bars->q_empty[qb]);
            }
            // ---- tile 1 ----
            if (ntile == 2) {
              if (!DT_OPT(16) && !wait(&bars->p_half[1][0], pph1)) { fail(4u); break; }
              ptx::tc_fence_after();
              issue_pv_parts<kSplit>(on, o1, s1, vd, idesc_pv, j > 0 ? 1u : 0u, 0, k_mid);
              if (!DT_OPT(16) && !wait(&bars->p_half[1][1], pph1)) { fail(4u); break; }
              pph1 ^= 1;
              ptx::tc_fence_after();
              issue_pv_parts<kSplit>(on, o1, s1, vd, idesc_pv, 1u, k_mid, ksteps);
              ptx::tc_commit_on(on, &bars->kv_empty[slot_v]);
              if (more) issue_qk<D>(on, s1, qd1, kd, idesc_qk);
              ptx::tc_commit_on(on, more ? &bars->s_full[1] : &bars->o_full[1]);
              if (more) {
                ptx::tc_commit_on(on, &bars->kv_empty[slot_k]);
                if (last_qk) ptx::tc_commit_on(on, &bars->q_empty[qb]);
              }
            }
          }
        }
      }
    }
  } else if (C::kTiles == 1 && warp >= 8) {
    ptx::setmaxnreg_dec<C::kRegsIdle>();  // (no second tile)
  } else {
    ptx::setmaxnreg_inc<C::kRegsHigh>();
    // =========================== softmax / correction / epilogue ===========================
    const int t = (warp - 4) >> 2;  // tile
    const int row_in_tile = ((warp & 3) << 5) + lane;
    const uint32_t lane_addr = (uint32_t)((warp & 3) << 5) << 16;
    uint32_t t_s = tmem + (t ? C::kColS1 : C::kColS0) + lane_addr;  // (one tile per item: S alternates between the two)
    const uint32_t t_o = tmem + (t ? C::kColO1 : C::kColO0) + lane_addr;
    uint32_t sph = 0, sph_b = 0, oph = 0;  // phases of s_full[] / o_full[t], continue across items
    bool ok = true;
#ifdef DT_BRINGUP
    bool first_dump = true;
#endif
    int n_item = 0;
    uint32_t n_blocks = 0;  // K/V blocks this warpgroup has handed over so far, over all items (one tile per item)
    const bool probe = (warp == 4 && lane == 0);
    const uint32_t t_p = tmem + (t ? C::kColP1 : C::kColP0) + lane_addr;  // (kAhead)
    // The P V of this tile's previous block has run.
    auto wait_pv = [&](uint32_t n_blocks) -> bool {
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->pv_done[C::kTiles == 1 ? 0 : t], (n_blocks - 1) & 1u, abort_flag))) {
        atomicCAS(a.status, 0u, 7u);
        *abort_flag = 1;
        return false;
      }
      ptx::tc_fence_after();
      return true;
    };

    int walk = blockIdx.x;
    Item w;
    while (ok && next_work(walk, w)) {
      if (t == 1 && !w.two) continue;  // this item has no second tile: neither side touches tile 1's barriers
      const int row = w.q0 + t * kBM + row_in_tile;
      const long long vis = a.is_causal ? (long long)row + w.off : (long long)w.sk;  // last visible key
      const long long lo = a.window > 0 ? (long long)row + w.off - a.window + 1 : 0;  // first visible key
      // Blocks below j_seen lie wholly at or before this row's last key, those from j_near on wholly at or behind its first one: worked out
      // once, and a block's test is two comparisons (kLong; 2 images, 4096 tokens, 20 heads of 64 254.8 -> 251.0 us).
      const int j_seen = (int)max(0LL, (min((long long)w.sk - 1, vis) + 1) / kBN - w.j0);
      const int j_near = (int)max(0LL, (lo + kBN - 1) / kBN - w.j0);
      float m_used = -INFINITY, l = 0.f;
      // masked variant: this warp's row of patch flags (null when its 32 rows lie beyond Sq: nothing to add there)
      const unsigned char* patch_flags = nullptr;
      if constexpr (kMask) {
        const int rg = (w.q0 + t * kBM + ((warp & 3) << 5)) >> 5;
        if (rg < a.n_rg) {
          const int64_t mb = a.m_sb ? w.b : 0, mh = a.m_sh ? w.h : 0;
          const int64_t hm = a.m_sh ? a.Hq : 1;
          patch_flags = a.mask_flags + ((mb * hm + mh) * a.n_rg + rg) * a.n_kh;
        }
      }
      // flags of block jj: bit 0 = its first 64 keys carry mask values, bit 1 = its second 64 keys
      auto block_flags = [&](int jj) -> uint32_t {
        if (!kMask || patch_flags == nullptr || jj >= w.nkv) return 0u;
        const uint32_t f = __ldg(reinterpret_cast<const unsigned short*>(patch_flags + 2 * (w.j0 + jj)));
        return ((f & 0xffu) ? 1u : 0u) | ((f >> 8) ? 2u : 0u);
      };
      uint32_t flags_cur = block_flags(0);

      for (int j = 0; j < (DT_OPT(64) ? 0 : w.nkv); ++j) {  // (experiment bit 6: no softmax work at all)
        const uint32_t flags_next = block_flags(j + 1);  // asked for early, used when the next block's mask is requested
        // Masked variant: the warp's 32 rows x 128 mask values of a block travel global -> shared memory with
        // asynchronous 16-byte copies, 8 lanes on one row's 128 contiguous bytes (whole cache lines; a lane fetching its
        // own row's 256 bytes would touch 32 lines per instruction and that made the L1 the bottleneck), in two halves
        // of 64 keys with a staging buffer each: the first one in this warp's O staging rows (idle until the epilogue), the
        // second one in the area taken from the K/V ring.  A block's halves are requested one block ahead; rows beyond Sq
        // and keys beyond Sk are zero-filled, never read.
        auto mask_prefetch = [&](int jj, int half, uint32_t flags) {
          if constexpr (kMask) {
            if (jj < w.nkv && ((flags >> half) & 1u)) {  // patches without mask values are not even fetched
              const int keyh = (w.j0 + jj) * kBN + half * 64;
              const uint32_t buf = (half ? mask_smem : stage_smem) + (uint32_t)(warp - 4) * (32 * 128);
              const T* mbase = reinterpret_cast<const T*>(a.mask) + (int64_t)w.b * a.m_sb + (int64_t)w.h * a.m_sh + keyh;
              const int ch = lane & 7;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int r = i * 4 + (lane >> 3);  // row within the warp's 32
                const int grow = w.q0 + t * kBM + ((warp & 3) << 5) + r;
                const int left = grow < w.sq ? w.sk - (keyh + ch * 8) : 0;  // mask entries from this chunk's first key on
                const int nbytes = left >= 8 ? 16 : (left > 0 ? left * 2 : 0);
                ptx::cp_async_16(buf + (uint32_t)r * 128 + (((uint32_t)ch ^ ((uint32_t)r & 7u)) << 4),
                                 nbytes ? (const void*)(mbase + (int64_t)grow * a.m_sq + ch * 8) : (const void*)a.mask, nbytes);
              }
            }
            ptx::cp_async_commit();  // always a group, possibly empty, so that the wait counts stay regular
          }
        };
        if constexpr (kMask) {
          if (j == 0) {
            // the O staging rows double as the first mask buffer: the previous item's TMA store must have read them
            if (lane == 0) ptx::bulk_wait_read_all();
            __syncwarp();
            mask_prefetch(0, 0, flags_cur);
            mask_prefetch(0, 1, flags_cur);
          }
        }
        // S buffer of this block: the tile's own, or (one tile per item) the two buffers in turn
        const int sb = C::kTiles == 1 ? (j & 1) : t;
        if constexpr (C::kTiles == 1) t_s = tmem + (sb ? C::kColS1 : C::kColS0) + lane_addr;
        uint32_t& sph_cur = (C::kTiles == 1 && sb) ? sph_b : sph;
        if (!DT_OPT(16) && !__all_sync(0xffffffffu, ptx::mbar_wait(&bars->s_full[sb], sph_cur, abort_flag))) {
          atomicCAS(a.status, 0u, 3u);
          *abort_flag = 1;
          ok = false;
          break;
        }
        sph_cur ^= 1;
        if (probe && j == 0) stamp(a, 16 * n_item + 8);
        ptx::tc_fence_after();
        uint32_t s[4][32];
        const float sl2 = a.scale_log2;
        float half_scale[2] = {sl2, sl2};  // from a half's scores to log2 units
        if constexpr (kMask) {
          // scores in two halves of 64 keys; each half gets mask / scale added once its mask values have landed (the
          // scores stay in the unscaled domain of the unmasked kernel).  A half whose mask values are all zero for the
          // whole warp -- most of a padding mask -- is left as it is.
          // kSplit: the half goes to log2 units and gets mask * log2(e), as in the CUDA-core kernel that these calls come from:
          // mask / scale overflows for entries that do not overflow there (-1e38 in a fully masked row), or scales below 2^-128.
          const uint64_t inv2 = ptx::pack_f32x2(kSplit ? kLog2e : 1.f / a.scale, kSplit ? kLog2e : 1.f / a.scale);
          const uint64_t to_log2 = ptx::pack_f32x2(sl2, sl2);
          auto add_mask_half = [&](int half) {
            if (!((flags_cur >> half) & 1u)) return;  // the same answer for the whole warp
            const uint32_t buf = (half ? mask_smem : stage_smem) + (uint32_t)(warp - 4) * (32 * 128) + (uint32_t)lane * 128;
            uint4 mk[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) mk[q] = ptx::ld_shared_v4(buf + ((((uint32_t)q) ^ ((uint32_t)lane & 7u)) << 4));
            uint32_t any = 0u;
#pragma unroll
            for (int q = 0; q < 8; ++q) any |= mk[q].x | mk[q].y | mk[q].z | mk[q].w;
            if (__any_sync(0xffffffffu, any != 0u)) {
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                const uint32_t mw[4] = {mk[q].x, mk[q].y, mk[q].z, mk[q].w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const float2 mf = unpack_pair<T>(mw[u]);
                  const int c = half * 2 + (q >> 2), i = (q & 3) * 8 + u * 2;
                  uint64_t s2 = ptx::pack_f32x2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
                  if constexpr (kSplit) s2 = ptx::mul_f32x2(s2, to_log2);
                  const uint64_t r2 = ptx::fma_f32x2(ptx::pack_f32x2(mf.x, mf.y), inv2, s2);
                  float r0, r1;
                  ptx::unpack_f32x2(r2, r0, r1);
                  s[c][i] = __float_as_uint(r0);
                  s[c][i + 1] = __float_as_uint(r1);
                }
              }
              if constexpr (kSplit) half_scale[half] = 1.f;
            }
            __syncwarp();  // every lane has read its row: the buffer may be refilled
          };
          ptx::tmem_ld32(t_s + 0, s[0]);
          ptx::tmem_ld32(t_s + 32, s[1]);
          ptx::cp_async_wait<1>();  // this block's first half has landed (its second half may still be on its way)
          __syncwarp();
          ptx::tc_wait_ld();
          add_mask_half(0);
          mask_prefetch(j + 1, 0, flags_next);
          ptx::tmem_ld32(t_s + 64, s[2]);
          ptx::tmem_ld32(t_s + 96, s[3]);
          ptx::cp_async_wait<1>();  // this block's second half (the group behind it is the next block's first half)
          __syncwarp();
          ptx::tc_wait_ld();
          add_mask_half(1);
          mask_prefetch(j + 1, 1, flags_next);
          flags_cur = flags_next;
        } else {
          ptx::tmem_ld32(t_s + 0, s[0]);
          ptx::tmem_ld32(t_s + 32, s[1]);
          ptx::tmem_ld32(t_s + 64, s[2]);
          ptx::tmem_ld32(t_s + 96, s[3]);
          ptx::tc_wait_ld();
        }
        if (probe && j == 0) stamp(a, 16 * n_item + 4);

#ifdef DT_BRINGUP
        if (a.dbg != nullptr && !(a.options & 2) && first_dump && j == 0 && blockIdx.x == 0) {
          float* dst = a.dbg + ((size_t)t * kBM + row_in_tile) * kBN;
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) dst[c * 32 + i] = __uint_as_float(s[c][i]);
        }
        first_dump = false;
#endif

        const int key0 = (w.j0 + j) * kBN;
        const bool need_mask = kLong ? j >= j_seen || j < j_near
                                     : (key0 + kBN > w.sk) || (a.is_causal && (long long)(key0 + kBN - 1) > vis) || (long long)key0 < lo;
        // chunks of 32 keys that lie entirely beyond Sk are skipped (short K/V such as 77 text tokens)
        const int nch = kLong && j + 1 < w.nkv ? 4 : max(1, (min(kBN, w.sk - key0) + 31) >> 5);  // at least the chunk the MMA warp always reads
        // bounds relative to this block as 32-bit values, so that each element costs one compare against a
        // constant: columns hi_rel+1 .. 127 and 0 .. lo_rel-1 are hidden
        auto hide = [&](int c_begin, int c_end) {
          const long long lim = min((long long)w.sk - 1, vis);  // keys <= lim visible
          const int hi_rel = (int)max(-1LL, min(lim - key0, (long long)(kBN - 1)));
          const int lo_rel = (int)max(0LL, min(lo - key0, (long long)kBN));
          if (lo_rel == 0) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              if (c < c_begin || c >= c_end || c >= nch || (c + 1) * 32 - 1 <= hi_rel) continue;  // chunk never read, or entirely visible
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (c * 32 + i > hi_rel) s[c][i] = 0xff800000u;  // -inf
            }
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              if (c < c_begin || c >= c_end || c >= nch) continue;
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (c * 32 + i > hi_rel || c * 32 + i < lo_rel) s[c][i] = 0xff800000u;  // -inf
            }
          }
        };
        if (need_mask) hide(0, 4);
        if (probe && j == 0) stamp(a, 16 * n_item + 12);
        // kLong: whole blocks take a path without a branch per chunk of 32 keys, so that the chunks' instructions interleave; with the branches
        // a chunk's chain of maxima ended before the next began (630 cycles of a warp's 2650 for a block, now 400).
        auto block = [&](auto path) -> bool {
        constexpr bool kWhole = decltype(path)::value > 0, kEarly = decltype(path)::value > 1;
        uint64_t lsum[4][2];
#pragma unroll
        for (int c = 0; c < 4; ++c) lsum[c][0] = lsum[c][1] = 0ull;
        uint32_t rest[16];  // (kSplit)
        // p = exp2(s * scale_log2 - m) of scores 2i and 2i+1 of chunk c: packed fp32x2 multiply-add, packed row sums in two
        // accumulators per chunk, packed conversion to the 16-bit P the second MMA reads from TMEM
        auto weigh = [&](int c, int i, uint64_t scale2, uint64_t neg_m2) {
          const uint64_t x2 = ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(s[c][2 * i]), __uint_as_float(s[c][2 * i + 1])),
                                             scale2, neg_m2);
          float p0, p1;
          if (DT_OPT(8)) {  // bring-up: no exponentials
            ptx::unpack_f32x2(x2, p0, p1);
          } else if ((i % kPolyPeriod) == kPolyPeriod - 1) {  // a share of the exponentials runs on the FMA pipes
            ptx::exp2_poly_x2(x2, p0, p1);
          } else {
            float x0, x1;
            ptx::unpack_f32x2(x2, x0, x1);
            p0 = fast_exp2(x0);
            p1 = fast_exp2(x1);
          }
          lsum[c][i & 1] = ptx::add_f32x2(lsum[c][i & 1], ptx::pack_f32x2(p0, p1));
          // the packed pair goes into the register score i of this chunk came in (scores 2i and 2i+1 are used up)
          if constexpr (kSplit) {  // weights of 16 bits and more: the rounded one and the rest of it
            const uint32_t hi = pack_pair<T>(p0, p1);
            const float2 f = unpack_pair<T>(hi);
            s[c][i] = hi;
            rest[i] = pack_pair<T>(p0 - f.x, p1 - f.y);
          } else if constexpr (kBf16 != 0) ptx::cvt_pack_bf16_into(s[c][i], p0, p1);
          else ptx::cvt_pack_f16_into(s[c][i], p0, p1);
        };
        // row max: four independent chains of 3-input max (one per 32-column chunk)
        float mxc[4];
        if constexpr (kEarly) {
          // Between blocks the reference maximum hardly ever moves, so the first half's exponentials (bound by the special-function unit) do
          // not wait for the block's maximum, which is found beside them; where it does move they are taken again.  (2 x 4096 tokens, 20
          // heads of 64 246.6 -> 236.4 us, 2304 tokens, 10 heads 57.4 -> 55.4.  At 128, where the products take twice as long, the two tiles' warps
          // get in each other's way: joint attention 233 -> 237 us; at 256 119.5 -> 125.2 for a chunk of 1777 x 5873.)  Not for an item's first
          // block, which has no maximum yet.
          const uint64_t scale2 = ptx::pack_f32x2(sl2, sl2);
          const float neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
          const uint64_t neg_m2 = ptx::pack_f32x2(neg_m, neg_m);
#pragma unroll
          for (int c = 0; c < 4; ++c) mxc[c] = -INFINITY;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
#pragma unroll
            for (int c = 0; c < 4; ++c) mxc[c] = ptx::max3(mxc[c], __uint_as_float(s[c][2 * i]), __uint_as_float(s[c][2 * i + 1]));
            weigh(0, i, scale2, neg_m2);
            weigh(1, i, scale2, neg_m2);
          }
        } else if constexpr (kWhole) {
#pragma unroll
          for (int c = 0; c < 4; ++c) mxc[c] = ptx::max3(__uint_as_float(s[c][0]), __uint_as_float(s[c][1]), __uint_as_float(s[c][2]));
#pragma unroll
          for (int i = 3; i < 31; i += 2)
#pragma unroll
            for (int c = 0; c < 4; ++c) mxc[c] = ptx::max3(mxc[c], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
#pragma unroll
          for (int c = 0; c < 4; ++c) mxc[c] = fmaxf(mxc[c], __uint_as_float(s[c][31]));
        } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c >= nch) {
            mxc[c] = -INFINITY;
            continue;
          }
          mxc[c] = ptx::max3(__uint_as_float(s[c][0]), __uint_as_float(s[c][1]), __uint_as_float(s[c][2]));
#pragma unroll
          for (int i = 3; i < 31; i += 2) mxc[c] = ptx::max3(mxc[c], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
          mxc[c] = fmaxf(mxc[c], __uint_as_float(s[c][31]));
        }
        }
        // (scale > 0 is a precondition of this kernel)
        float mx = kSplit ? fmaxf(fmaxf(mxc[0], mxc[1]) * half_scale[0], fmaxf(mxc[2], mxc[3]) * half_scale[1])
                          : fmaxf(fmaxf(mxc[0], mxc[1]), fmaxf(mxc[2], mxc[3])) * sl2;
        if (DT_OPT(32)) mx = __uint_as_float(s[0][0]) * sl2;  // bring-up: no row maximum
        const float m_cand = fmaxf(m_used, mx);
        // Lazy rescale: keep the old reference max unless the new one is larger by more than the threshold.
        const bool grow = (m_cand - m_used > kRescaleThreshold) || (m_used == -INFINITY && m_cand != -INFINITY);
        if (__any_sync(0xffffffffu, grow)) {
          const float m_new = grow ? m_cand : m_used;
          const float alpha = (m_new == -INFINITY) ? 1.f : fast_exp2(m_used - m_new);
          l *= alpha;
          m_used = m_new;
          if (j > 0) {
            if constexpr (C::kTiles == 1 || kAhead) {
              // With S double-buffered, or P not in its place, this block's scores arrive before the previous block's P V has run: O may only
              // be touched once that one has retired.  (It cannot be more than one phase behind: the P V of this block
              // waits for the P written below.)
              if (!wait_pv(n_blocks)) return false;
            }
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
              uint32_t ov[32];
              ptx::tmem_ld32(t_o + c * 32, ov);
              ptx::tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
              ptx::tmem_st32(t_o + c * 32, ov);
            }
          }
          if constexpr (kEarly) {
            ptx::tmem_ld32(t_s + 0, s[0]);
            ptx::tmem_ld32(t_s + 32, s[1]);
            ptx::tc_wait_ld();
            if (need_mask) hide(0, 2);
            const uint64_t scale2 = ptx::pack_f32x2(sl2, sl2);
            const float neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
            const uint64_t neg_m2 = ptx::pack_f32x2(neg_m, neg_m);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              lsum[c][0] = lsum[c][1] = 0ull;
#pragma unroll
              for (int i = 0; i < 16; ++i) weigh(c, i, scale2, neg_m2);
            }
          }
        }
        if (probe && j == 0) stamp(a, 16 * n_item + 13);
        const float neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
        const uint64_t neg_m2 = ptx::pack_f32x2(neg_m, neg_m);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint64_t scale2 = ptx::pack_f32x2(half_scale[c >> 1], half_scale[c >> 1]);
          if (kWhole || c < nch) {
          if (!kEarly || c > 1) {
#pragma unroll
            for (int i = 0; i < 16; ++i) weigh(c, i, scale2, neg_m2);
          }
          if constexpr (kAhead) {
            // the previous block's last MMAs read these columns (the first half's are free: the commit that announced S stood behind
            // the MMAs that read them)
            if (c == 2 && n_blocks > 0 && !wait_pv(n_blocks)) return false;
          }
          ptx::tmem_st16((kAhead ? t_p : t_s) + c * 16, s[c]);
          if constexpr (kSplit) ptx::tmem_st16(t_s + 64 + c * 16, rest);
          }
          if (c == 1 || c == 3) {  // 64 keys of P are in TMEM: let the MMA warp start on them
            ptx::tc_wait_st();
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&bars->p_half[sb][c >> 1]);
            if (probe && j == 0) stamp(a, 16 * n_item + 14 + (c >> 1));
          }
        }
        {
          float a0, a1, b0, b1;
#pragma unroll
          for (int c = 0; c < 4; ++c) lsum[c][0] = ptx::add_f32x2(lsum[c][0], lsum[c][1]);
          ptx::unpack_f32x2(ptx::add_f32x2(lsum[0][0], lsum[1][0]), a0, a1);
          ptx::unpack_f32x2(ptx::add_f32x2(lsum[2][0], lsum[3][0]), b0, b1);
          l += (a0 + a1) + (b0 + b1);
        }
        return true;
        };
        if (kMayEarly && nch == 4 && j > 0) ok = block(std::integral_constant<int, kMayEarly ? 2 : 0>{});
        else if (kLong && nch == 4) ok = block(std::integral_constant<int, kLong ? 1 : 0>{});
        else ok = block(std::integral_constant<int, 0>{});
        if (!ok) break;
        ++n_blocks;
      }
      if (!ok) break;
      if (probe) stamp(a, 16 * n_item + 9);

      // ---- epilogue: O / l -> global (the MMA warp already works on the next item's first S meanwhile) ----
      if (!DT_OPT(16) && !__all_sync(0xffffffffu, ptx::mbar_wait(&bars->o_full[t], oph, abort_flag))) {
        atomicCAS(a.status, 0u, 5u);
        *abort_flag = 1;
        ok = false;
        break;
      }
      oph ^= 1;
      if (probe) stamp(a, 16 * n_item + 10);
      ptx::tc_fence_after();
      if constexpr (kCut) {  // the run's share: (maximum, sum, O)
        float* mine = share_of<D>(a, walk - (int)gridDim.x, warp & 3);
        __stcg(mine + lane, m_used);
        __stcg(mine + 32 + lane, l);
#pragma unroll 1
        for (int c = 0; c < D / 16; ++c) {
          uint32_t ov[16];
          ptx::tmem_ld16(t_o + c * 16, ov);
          ptx::tc_wait_ld();
          if constexpr (kSplit) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (!(__uint_as_float(ov[i]) * 0.f == 0.f)) *a.not_finite = 1u;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)  // [D / 4][32 rows][4]: a warp writes 512 consecutive bytes
            __stcg(reinterpret_cast<float4*>(mine + 64) + (c * 4 + i) * 32 + lane,
                   make_float4(__uint_as_float(ov[4 * i]), __uint_as_float(ov[4 * i + 1]), __uint_as_float(ov[4 * i + 2]),
                               __uint_as_float(ov[4 * i + 3])));
        }
        ptx::tc_fence_before();
        ++n_item;
        continue;
      }
      if (a.sinks && row < w.sq) {
        // attention sink: one more score without a value row joins the denominator (l and O are relative to m_used)
        const float sl = to_float(reinterpret_cast<const T*>(a.sinks)[w.h]) * kLog2e;
        if (m_used == -INFINITY) {
          m_used = sl;
          l = 1.f;
        } else {
          l += fast_exp2(sl - m_used);
        }
      }
      uint64_t probe = 0ull;  // kSplit: O * 0 added up, NaN where an O is not finite
      // a row that never saw a visible key (m_used still -inf) yields zeros, whatever the masked entries summed to
      const float inv = (l > 0.f && m_used != -INFINITY) ? 1.f / l : 0.f;
      // O goes out through shared memory and a TMA store per warp (32 rows x 64 columns): whole 128-byte
      // row pieces reach L2, instead of 16-byte pieces scattered over 32 rows per instruction.
      {
        const uint32_t my_stage = stage_smem + (uint32_t)(warp - 4) * (32 * 128);
        const int wrow0 = w.q0 + t * kBM + ((warp & 3) << 5);
        // The tensor map clips at the end of the tensor, not at the end of a packed sequence: with variable
        // lengths a warp whose 32 rows reach past its sequence stores row by row instead.
        const bool tma_ok = a.off_q ? (wrow0 + 32 <= w.sq) : (wrow0 < w.sq);
        const bool guarded_main = a.off_q != nullptr && wrow0 < w.sq && !tma_ok;
#pragma unroll
        for (int hf = 0; hf < D / 64; ++hf) {
          // the previous TMA store of this warp (last half, or the previous item) must have read the staging rows
          // before they are overwritten: waited for here, as late as possible, not right after issuing it
          if (lane == 0) ptx::bulk_wait_read_all();
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t ov[32];
            ptx::tmem_ld32(t_o + hf * 64 + c * 32, ov);
            ptx::tc_wait_ld();
            if constexpr (kSplit) {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                probe = ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(ov[2 * i]), __uint_as_float(ov[2 * i + 1])), 0ull, probe);
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint4 pk;
              pk.x = pack_pair<T>(__uint_as_float(ov[v * 8 + 0]) * inv, __uint_as_float(ov[v * 8 + 1]) * inv);
              pk.y = pack_pair<T>(__uint_as_float(ov[v * 8 + 2]) * inv, __uint_as_float(ov[v * 8 + 3]) * inv);
              pk.z = pack_pair<T>(__uint_as_float(ov[v * 8 + 4]) * inv, __uint_as_float(ov[v * 8 + 5]) * inv);
              pk.w = pack_pair<T>(__uint_as_float(ov[v * 8 + 6]) * inv, __uint_as_float(ov[v * 8 + 7]) * inv);
              // 128-byte swizzle: 16-byte chunk q of row r lives at chunk q ^ (r & 7)
              const uint32_t q = (uint32_t)(c * 4 + v);
              const uint32_t addr = my_stage + (uint32_t)lane * 128 + ((q ^ ((uint32_t)lane & 7u)) << 4);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(pk.x), "r"(pk.y), "r"(pk.z), "r"(pk.w)
                           : "memory");
            }
          }
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && tma_ok && hf * 64 < a.d_real) {  // (a half made of padding columns only is not stored)
            ptx::tma_store_4d(&map_o, my_stage, hf * 64, w.h, w.qrow + wrow0, w.b);
            ptx::bulk_commit_group();
          }
          if (a.n_extra > 0 || guarded_main) {
            // copies of the tile for the other GPUs (and the row-guarded store of a sequence's last rows):
            // 8 lanes write one row's 128 bytes, 4 rows per instruction
            const int64_t row_off = (int64_t)w.b * a.o_sb + (int64_t)w.h * a.o_sh + hf * 64 + (int64_t)w.qrow * a.o_ss;
#pragma unroll 1
            for (int e = guarded_main ? -1 : 0; e < a.n_extra; ++e) {
              T* dst = reinterpret_cast<T*>(e < 0 ? a.o : a.extra_o[e]) + row_off;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int r = i * 4 + (lane >> 3), ch = lane & 7;
                uint4 val;
                const uint32_t addr = my_stage + (uint32_t)r * 128 + (((uint32_t)ch ^ ((uint32_t)r & 7u)) << 4);
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(val.x), "=r"(val.y), "=r"(val.z), "=r"(val.w) : "r"(addr));
                if (wrow0 + r < w.sq && hf * 64 + ch * 8 < a.d_real) *reinterpret_cast<uint4*>(dst + (int64_t)(wrow0 + r) * a.o_ss + ch * 8) = val;
              }
            }
          }
          __syncwarp();
        }
      }
      if constexpr (kSplit) {
        float p0, p1;
        ptx::unpack_f32x2(probe, p0, p1);
        if (!(p0 + p1 == 0.f)) *a.not_finite = 1u;
      }
      if (a.lse && row < w.sq)
        a.lse[((int64_t)w.b * a.Hq + w.h) * a.Sq + w.qrow + row] =
            (l > 0.f && m_used != -INFINITY) ? m_used * kLn2 + logf(l) : -INFINITY;
      // the next item's first P*V overwrites O: order this thread's TMEM reads before its later arrivals
      ptx::tc_fence_before();
      if (probe) stamp(a, 16 * n_item + 11);
      ++n_item;
    }
  }

  // =========================== teardown ===========================
  if (warp >= 4 && lane == 0) ptx::bulk_wait_read_all();  // staging rows read; the global writes complete with the kernel
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, C::kTmemCols);
  }
}

#ifdef DT_BRINGUP
int g_options = 0;
float* g_dbg = nullptr;
#endif

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// How a call's work is laid out over the SMs.
struct Plan {
  int item_rows, n_q, n_items;
  int n_whole;           // items taken whole, in full rounds
  int n_single;          // the items behind them as single tiles (0: they are whole too)
  int n_splits;          // runs per item of a cut call (0: not cut)
};

long long blocks_of_item(const dt_sdpa_params& p, int item_rows, int qt) {
  const long long all = (p.Sk + kBN - 1) / kBN;
  if (!p.is_causal) return all;
  const long long end = (long long)(qt + 1) * item_rows < p.Sq ? (long long)(qt + 1) * item_rows : p.Sq;
  long long lim = end + (p.Sk - p.Sq);
  if (lim > p.Sk) lim = p.Sk;
  const long long n = (lim + kBN - 1) / kBN;
  return n < 1 ? 1 : n;
}

Plan make_plan(const dt_sdpa_params& p, int tiles) {
  Plan r{};
  const int sms = device_sm_count();
  const bool varlen = p.seq_offsets_q != nullptr;
  const int rows = varlen ? p.max_seq_q : p.Sq, bh = p.Hq * (varlen ? p.n_seq : p.B);
  // One tile per item where even that does not fill the SMs once: a pair of tiles on one SM takes about 1.5 times as long
  // as one tile, and half of the SMs would have nothing to do.
  const long long singles = (long long)((rows + kBM - 1) / kBM) * bh;
  r.item_rows = tiles == 2 && singles > sms ? 2 * kBM : kBM;
  r.n_q = (rows + r.item_rows - 1) / r.item_rows;
  r.n_items = r.n_whole = r.n_q * bh;
  if (varlen) return r;
  const int rest = r.n_items % sms;
  // For the same reason a last round of pairs that fills less than half of the SMs is taken tile by tile (2 images, 4096
  // tokens, 20 heads of 64: 4.3 rounds, 302 -> 293 us).  The rows' results do not depend on it.  Under the causal rule the last
  // round holds the lightest pairs, and behind an odd number of rounds its order gives them to the CTAs with the least work:
  // twice as many tiles reach CTAs that have more (32 / 8 heads of 128, 1280 and 1536 tokens: 29.6 and 33.6 us in pairs, 34.4
  // and 41.7 us by tiles; of 64, 4096 tokens: 125 and 133 us).  So there only behind an even number, and for enough pairs (32 / 8
  // heads of 64: 56 pairs at 2816 tokens 72.5 us in pairs, 70.0 by tiles; 24 pairs at 2400 tokens 56.7 and 60.1 us).
  const bool tiles_pay = !p.is_causal || (r.n_items / sms % 2 == 0 && 3 * rest >= sms);
  if (r.item_rows > kBM && r.n_items > sms && rest > 0 && 2 * rest <= sms && tiles_pay) {
    r.n_whole = r.n_items - rest;
    r.n_single = 2 * rest;
    return r;
  }
  // A call that leaves half of the SMs without any item (a short chunk of queries behind a long prefix): every item's K/V blocks
  // cut into equal runs, when that saves at least kCutGain blocks' time.  A run lies in one
  // item: with runs of equal length over all SMs, whatever items they fell into, there were up to twice as many shares to write
  // and read (400 x 1536, 16 / 4 heads of 256: 24.3 us uncut, 32.2 us so, 22.4 us by items).  Measured against the uncut call (Sq x
  // Sk, time uncut / cut, saving 4 blocks): 24 heads of 64, 128 x 1024 causal: 18.2 / 14.7 us; 6 heads of 256, 128 x 1024: 18.5 /
  // 17.6 us, but 16 heads (64 items, two runs each) 400 x 1024: 19.4 / 19.6, causal 19.9 / 20.6 us.  Runs of at least 4 blocks: of
  // 2 the shares of a long item take longer to add (2 heads of 64, 8192 keys: 23.6 against 19.1 us; 1280 keys 11.7 against 14.9 us).
  const int kCutGain = tiles == 1 && 3 * r.n_items > sms ? 5 : 4;
  constexpr int kMinRun = 4;
  if (2 * r.n_items > sms || p.sliding_window > 0) return r;
  const long long longest = blocks_of_item(p, r.item_rows, r.n_q - 1);  // (the last rows see the most)
  // How many: one run per SM, or, where the items divide the SMs badly, up to four shorter ones (52 heads of 128, 128 x 16000: 2
  // runs each, one per CTA, 111 us; 5 each, up to two per CTA, 102; 50 heads of 64: 108 and 95).  In quarters of a block's time a
  // run's own start and end are about kRunCost, a share to add kShareCost (6 or 20 and 2 in their place: within 1 %).
  constexpr int kRunCost = 12, kShareCost = 1;
  long long splits = 0, saved = 0, best = 0;
  for (long long n = 2; n <= longest / kMinRun && r.n_items * n <= 4 * sms && longest * n < (1LL << 31); ++n) {
    const long long rounds = (r.n_items * n + sms - 1) / sms, per = (longest + n - 1) / n;
    const long long cost = rounds * (4 * per + kRunCost) + n * kShareCost;
    if (splits == 0 || cost < best) {
      splits = n;
      best = cost;
      saved = longest - rounds * per;
    }
  }
  if (splits == 0 || saved < kCutGain) return r;
  r.n_splits = (int)splits;
  return r;
}
size_t split_bytes(const Plan& plan, int D) {  // (a cut call's items are single tiles)
  return (size_t)plan.n_items * plan.n_splits * (kBM / 32) * (D + 2) * 32 * sizeof(float);
}

bool mask_rows_aligned(const dt_sdpa_params& p) {
  return !(reinterpret_cast<uintptr_t>(p.mask) % 16 || p.mask_stride_b % 8 || p.mask_stride_h % 8 || p.mask_stride_q % 8);
}
// The first 4 KB of a workspace hold the split-KV ticket counters, which every call leaves zero: the flags start behind.
constexpr size_t kTicketBytes = 4096;
size_t mask_flag_bytes(const dt_sdpa_params& p) {
  const size_t Bm = p.mask_stride_b ? p.B : 1, Hm = p.mask_stride_h ? p.Hq : 1;
  const size_t n_rg = (p.Sq + 31) / 32, n_kh = ((p.Sk + 63) / 64 + 1) & ~(size_t)1;
  return kTicketBytes + (Bm * Hm * n_rg * n_kh + 255) / 256 * 256;
}
int repacked_row(const dt_sdpa_params& p) { return (p.Sk + 7) / 8 * 8; }
size_t prefill_repack_bytes_needed(const dt_sdpa_params& p) {  // the flags, the word that says "not finite" and the copy
  const size_t Bm = p.mask_stride_b ? p.B : 1, Hm = p.mask_stride_h ? p.Hq : 1;
  return mask_flag_bytes(p) + 256 + Bm * Hm * p.Sq * (size_t)repacked_row(p) * 2;
}
size_t cut_bytes(const dt_sdpa_params& p) {
  const int D = p.D > 128 ? 256 : p.D > 64 ? 128 : 64, tiles = D == 256 ? 1 : 2;
  return split_bytes(make_plan(p, tiles), D);
}

template <typename T, int D, bool kMask, bool kSplit = false>
int launch_t(const dt_sdpa_params& p, cudaStream_t stream, void* const* extra, int n_extra, void* workspace,
             size_t workspace_bytes) {
  using C = Cfg<D, kMask>;
  // Head dim 64: P beside S and O, and each block's Q K^T ahead of the end of the one before.  Two tiles of head dim 64 leave 128 TMEM
  // columns, so P does not have to overwrite S: the next block's Q K^T is issued as soon as the first half of P says that S has been
  // read, and runs under the second half of the softmax, which used to wait for it (a quarter of a block's 3600 cycles).  2 images, 4096
  // tokens, heads of 64: 20 heads 290.2 -> 275.7 us, 10 heads 175.3 -> 163.1; 8 heads of 40: 124.3 -> 119.5; 300 tokens, 10 heads: 8.8 -> 8.3.
  // Not where the second block is the last and holds 32 keys at most (two text prompts), the call has several rounds and every head ends in a
  // lone tile: nothing stands beside that tile's softmax, its products are short, and it has a hand-over more.  Time without / with
  // it, mean and worst over 12 such calls (777 to 4641 rows, 8 to 20 heads, 2 and 4 images): 129 keys 0.985 and 0.955, 154 keys 0.982 and
  // 0.950 (4 images, 4641 rows, 10 heads: 37.5 / 39.5 us), 160 keys 0.985 and 0.946; 176 keys 1.012 and 0.989, 260 keys 1.011 and 1.003, 520
  // keys 1.037 and 1.026.  Pairs of tiles only (28 calls): 154 keys 0.999 and 0.991, 176 keys 1.023 and 1.010.  Nor for a single block, where
  // nothing is ahead of anything: 100 keys, 48 calls, 0.993 and 0.975.  (The masked variant has not been built with it.)
  // And for all widths: a softmax without branches inside whole blocks (kLong), where items have more than three blocks or end in more than 32
  // keys.  us in a graph before / with it: joint attention, 4608 tokens, 24 heads of 128 229 / 216; 2 images, 4096 tokens, 20 heads of 64 275 /
  // 255; 16384 x 512, 40 heads of 128 210 / 201; causal, 5000 tokens, 16 / 4 heads of 128 103.6 / 98.6, of 256 165.9 / 164.9; 4096 tokens
  // under a padding mask 332 / 319.  Two paths in turn cost shorter items more: 4096 x 257, 40 heads of 128 44.9 / 45.6; 160 keys, 4 images
  // of 4641 rows, 10 heads of 64 36.3 / 37.4; and masks with two parts per weight (kSplit), whose registers are full: 1501 tokens 107.8 / 110.3.
  constexpr bool kMayLong = !kSplit;
  // At head dim 64 a third path (kMayEarly) for calls of eight blocks and more without a window; as code in the way of shorter ones and of
  // windows, whose edges move the maximum, it costs (window of 300, 5000 tokens 42.6 / 47.6 us).  Without / with it over 13 lengths of self-attention
  // at 5 counts of heads, causal calls and 4096 rows of cross-attention: 400 keys 0.972 to 0.978, 512 0.968 to 0.998, 640 0.990 to 1.015, 768
  // 0.989 to 1.014, 896 0.997 to 1.018, 1024 1.000 to 1.022, 1536 1.008 to 1.026, 3072 1.020 to 1.035; sequences of different lengths are not
  // moved (0.996 to 1.004).
  constexpr int kEarlyKeys = 1024;
  constexpr int kAheadKeys = kBN + 32;
  CUtensorMap mq, mk, mv, mo;
  if (!make_bshd_tensor_map(&mq, p.q, p.B, p.Sq, p.Hq, p.D, p.dtype, kBM)) return DT_UNSUPPORTED;
  if (!make_bshd_tensor_map(&mk, p.k, p.B, p.Sk, p.Hkv, p.D, p.dtype, kBN)) return DT_UNSUPPORTED;
  if (!make_bshd_tensor_map(&mv, p.v, p.B, p.Sk, p.Hkv, p.D, p.dtype, kBN)) return DT_UNSUPPORTED;
  if (!make_bshd_tensor_map(&mo, p.o, p.B, p.Sq, p.Hq, p.D, p.dtype, 32)) return DT_UNSUPPORTED;
  PrefillArgs a{};
  a.o = p.o.ptr;
  a.lse = p.lse;
#ifdef DT_BRINGUP
  a.dbg = g_dbg;
  a.options = g_options;
#endif
  a.o_sb = p.o.stride_b; a.o_ss = p.o.stride_s; a.o_sh = p.o.stride_h;
  a.status = device_status_word();
  if (!a.status) return DT_CUDA;
  a.Sq = p.Sq; a.Sk = p.Sk; a.Hq = p.Hq; a.Hkv = p.Hkv;
  a.scale_log2 = p.scale * kLog2e;
  a.scale = p.scale;
  a.mask = p.mask;
  a.m_sb = p.mask_stride_b; a.m_sh = p.mask_stride_h; a.m_sq = p.mask_stride_q;
  if (kMask) {
    if (!workspace || workspace_bytes < (kSplit ? prefill_repack_bytes_needed(p) : mask_flag_bytes(p))) return DT_WORKSPACE;
    const int Bm = p.mask_stride_b ? p.B : 1, Hm = p.mask_stride_h ? p.Hq : 1;
    a.n_rg = (p.Sq + 31) / 32;
    a.n_kh = ((p.Sk + 63) / 64 + 1) & ~1;
    unsigned char* flags = static_cast<unsigned char*>(workspace) + kTicketBytes;
    a.mask_flags = flags;
    dim3 fgrid((a.n_kh + 7) / 8, a.n_rg, Bm * Hm);
    if (fgrid.y > 65535 || fgrid.z > 65535) return DT_UNSUPPORTED;
    if (kSplit) {
      const int ld = repacked_row(p);
      a.not_finite = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(workspace) + mask_flag_bytes(p));
      unsigned short* copy = reinterpret_cast<unsigned short*>(reinterpret_cast<uint8_t*>(a.not_finite) + 256);
      DT_CUDA_TRY(launch_behind(mask_repack_kernel, fgrid, dim3(256), 0, stream, 1, static_cast<const unsigned short*>(p.mask),
                                p.mask_stride_b, p.mask_stride_h, p.mask_stride_q, Hm, p.Sq, p.Sk, a.n_rg, a.n_kh, p.is_causal,
                                flags, copy, ld, a.not_finite));
      a.mask = copy;
      a.m_sq = ld;
      a.m_sh = Hm > 1 ? (int64_t)p.Sq * ld : 0;
      a.m_sb = Bm > 1 ? (int64_t)Hm * p.Sq * ld : 0;
    } else
    DT_CUDA_TRY(launch_behind(mask_flags_kernel, fgrid, dim3(256), 0, stream, 1, static_cast<const unsigned short*>(p.mask),
                              p.mask_stride_b, p.mask_stride_h, p.mask_stride_q, Hm, p.Sq, p.Sk, a.n_rg, a.n_kh, p.is_causal, flags));
  }
  a.is_causal = p.is_causal;
  a.window = p.sliding_window;
  a.sinks = p.sinks;
  if (n_extra < 0 || n_extra > kMaxExtraOutputs) return DT_BAD_ARG;
  a.n_extra = n_extra;
  a.d_real = p.D;
  for (int i = 0; i < n_extra; ++i) a.extra_o[i] = extra[i];
  a.off_q = p.seq_offsets_q;
  a.off_k = p.seq_offsets_k;
  const Plan plan = make_plan(p, C::kTiles);
  a.item_rows = plan.item_rows;
  a.n_qpairs = plan.n_q;
  a.n_items = plan.n_items;
  const int n_sm = device_sm_count();
  const size_t split_at = kMask ? (kSplit ? prefill_repack_bytes_needed(p) : mask_flag_bytes(p)) : kTicketBytes;
  if (plan.n_splits > 0 && n_extra == 0 && workspace && reinterpret_cast<uintptr_t>(workspace) % 16 == 0 &&
      workspace_bytes >= align256(split_at) + split_bytes(plan, D)) {
    a.n_splits = plan.n_splits;
    a.part = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + align256(split_at));
    auto kern = prefill_tcgen05_kernel<T, D, kMask, kSplit, true, kMayLong ? 1 : 0>;  // (its runs have at least four blocks)
    DT_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
    const int runs = plan.n_items * plan.n_splits;
    // The kernel that adds the shares comes in early only where a third of the SMs has no run: otherwise its CTAs crowd onto the few that
    // are free.  Launched behind the runs / early / by this rule, us: 8 heads of 256, 128 x 16000 (144 runs) 32.0 / 34.1 / 30.4, 256 x 5000
    // (128) 22.1 / 23.5 / 21.9; 4 heads of 256, 256 x 12000 (128) 27.6 / 29.7 / 26.6; not early / early: 400 x 3000 (96) 20.3 / 19.1; 16 heads
    // of 256, 128 x 2000 (64) 19.2 / 17.6.  (The first figure has ordinary launches on both sides.)
    a.cut_lets_next = 3 * runs <= 2 * n_sm;
    DT_CUDA_TRY(launch_behind(kern, dim3(runs < n_sm ? runs : n_sm), dim3(kThreads), C::kSmemBytes, stream, 1, mq, mk, mv, mo, a));
    DT_CUDA_TRY(launch_behind(cut_combine_kernel<T, D>, dim3(plan.n_items * (kBM / 32), (p.D + 63) / 64), dim3(256), 0, stream, 1, a));
    return DT_OK;
  }
  auto kern = prefill_tcgen05_kernel<T, D, kMask, kSplit, false, 0>;
  if constexpr (kMayLong) {
    const bool lone_ends = p.seq_offsets_q == nullptr && plan.item_rows > kBM && plan.n_items > n_sm && (p.Sq + kBM - 1) / kBM % 2 == 1;
    const int keys = p.seq_offsets_q ? p.max_seq_k : p.Sk;
    const bool is_long = D == 64 && !kMask ? keys > (lone_ends ? kAheadKeys : kBN) : keys > 3 * kBN || (keys > kBN && (keys - 1) % kBN >= 32);
    if (is_long) kern = prefill_tcgen05_kernel<T, D, kMask, kSplit, false, 1>;
    if constexpr (D == 64 && !kMask) {
      if (is_long && keys >= kEarlyKeys && p.sliding_window == 0) kern = prefill_tcgen05_kernel<T, D, kMask, kSplit, false, 2>;
    }
  }
  DT_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
  const int ctas = a.n_items < n_sm ? a.n_items : n_sm;  // one persistent CTA per SM
  a.n_slots = plan.n_single > 0 ? plan.n_whole : (a.n_items + ctas - 1) / ctas * ctas;
  a.n_places = a.n_slots + plan.n_single;
  if (a.n_items <= n_sm) {
    DT_CUDA_TRY(launch_behind(kern, dim3(ctas), dim3(kThreads), C::kSmemBytes, stream, 1, mq, mk, mv, mo, a));
  } else {
    kern<<<ctas, kThreads, C::kSmemBytes, stream>>>(mq, mk, mv, mo, a);
    DT_CUDA_TRY(cudaGetLastError());
  }
  return DT_OK;
}

}  // namespace

bool prefill_supported(const dt_sdpa_params& p) {
  // variable-length batches: the plain operator only (per-sequence lengths are on the device, so the causal and
  // window cases, which need sq <= sk per sequence, stay on the generic kernel)
  if (p.seq_offsets_q && (p.is_causal || p.sliding_window > 0 || p.n_seq > 65535)) return false;
  if (p.sliding_window > 0 && p.Sq > p.Sk) return false;  // rows that may see no key: generic kernel
  if (p.dtype != DT_F16 && p.dtype != DT_BF16) return false;
  if (p.D < 8 || p.D > 256 || p.D % 8) return false;  // head dims below 64 / 128 / 256 run zero-padded (SD1.5: 40, 80, 160)
  if (p.mask && !mask_rows_aligned(p)) return false;  // each row's entries are read with 16-byte loads
  if (!(p.scale > 0.f)) return false;
  if (p.Hq % p.Hkv) return false;
  if (p.Hq > 65535 || p.B > 65535) return false;
  if (p.is_causal && p.Sq > p.Sk) return false;  // rows without any visible key: left to the generic kernel
  auto ok = [](const dt_tensor4& t) {
    return (reinterpret_cast<uintptr_t>(t.ptr) % 16 == 0) && t.stride_b % 8 == 0 && t.stride_s % 8 == 0 &&
           t.stride_h % 8 == 0;
  };
  return ok(p.q) && ok(p.k) && ok(p.v) && ok(p.o);
}

// The masked variant needs its flags; the scratch of cut items is optional (without it, or with less, nothing is cut).
size_t prefill_workspace_bytes(const dt_sdpa_params& p) {
  const size_t cut = cut_bytes(p);
  if (cut) return align256(p.mask ? mask_flag_bytes(p) : kTicketBytes) + cut;
  return p.mask ? mask_flag_bytes(p) : 0;
}

// Masks whose rows are not 16-byte aligned: copied to aligned rows first.  The calls come from the CUDA-core kernel, whose
// weights are fp32, so this variant multiplies V with two 16-bit parts of every weight: 333 tokens, 32 / 8 heads of 128,
// causal and padding mask, bf16: 117 us there, 27 us here, error against 64 bits 1.6e-3 (the rounding of the result) in both.  A mask per head of a long
// sequence would need a copy as large as itself: up to 256 MB.
bool prefill_repack_supported(const dt_sdpa_params& p) {
  if (!p.mask || mask_rows_aligned(p) || (p.flags & DT_FLAG_FORCE_GENERIC)) return false;
  dt_sdpa_params plain = p;
  plain.mask = nullptr;
  // Up to one 64-key tile the CUDA-core kernel takes a single step (41 tokens, 32 heads: 18.2 us there, 19.2 us here), and with
  // heads up to 64 and a block of its own for every CTA two steps cost less than three launches and scratch: 77 tokens, 12 heads of
  // 64: 23.2 us on the device there and 19.6 here, but one call after another 23 and 33 (129 tokens: 33 and 21 on the device).
  if (p.Sk <= 64 || !prefill_supported(plain) || (p.Sq + 31) / 32 > 65535) return false;
  if (p.Sk <= 128 && p.D <= 64 && (double)((p.Sq + 63) / 64) * p.Hq * p.B <= device_sm_count()) return false;
  const size_t Bm = p.mask_stride_b ? p.B : 1, Hm = p.mask_stride_h ? p.Hq : 1;
  return Bm * Hm <= 65535 && Bm * Hm * p.Sq * (size_t)repacked_row(p) * 2 <= ((size_t)256 << 20);
}

size_t prefill_repack_workspace_bytes(const dt_sdpa_params& p) {
  const size_t cut = cut_bytes(p);
  return cut ? align256(prefill_repack_bytes_needed(p)) + cut : prefill_repack_bytes_needed(p);
}

// An infinity in V is 0 * inf = NaN to the second part of a weight that has none, and a NaN in V reaches the rows of other tiles
// than on the CUDA cores.  Either makes every O of the tiles that see its key an infinity or NaN, as NaN scores do: where one came
// out, the CUDA-core kernel behind, which otherwise returns at once, computes the call (encoder of 333 tokens 24 -> 27 us; looking V
// over in the first pass, a few dozen blocks, took 15 us).
int launch_prefill_repack(const dt_sdpa_params& p, cudaStream_t stream, void* workspace, size_t workspace_bytes) {
#define DT_REPACK_GO(T, DD) launch_t<T, DD, true, true>(p, stream, nullptr, 0, workspace, workspace_bytes)
#define DT_REPACK_BY_D(T) (p.D > 128 ? DT_REPACK_GO(T, 256) : p.D > 64 ? DT_REPACK_GO(T, 128) : DT_REPACK_GO(T, 64))
  const int st = p.dtype == DT_F16 ? DT_REPACK_BY_D(__half) : DT_REPACK_BY_D(__nv_bfloat16);
#undef DT_REPACK_BY_D
#undef DT_REPACK_GO
  if (st != DT_OK) return st;
  return launch_generic(p, stream, reinterpret_cast<const uint32_t*>(static_cast<uint8_t*>(workspace) + mask_flag_bytes(p)));
}

int launch_prefill(const dt_sdpa_params& p, cudaStream_t stream, void* const* extra_outputs, int n_extra, void* workspace,
                   size_t workspace_bytes) {
#define DT_PREFILL_GO(T, DD, M) launch_t<T, DD, M>(p, stream, extra_outputs, n_extra, workspace, workspace_bytes)
#define DT_PREFILL_BY_D(T, M) (p.D > 128 ? DT_PREFILL_GO(T, 256, M) : p.D > 64 ? DT_PREFILL_GO(T, 128, M) : DT_PREFILL_GO(T, 64, M))
  if (p.mask) return p.dtype == DT_F16 ? DT_PREFILL_BY_D(__half, true) : DT_PREFILL_BY_D(__nv_bfloat16, true);
  return p.dtype == DT_F16 ? DT_PREFILL_BY_D(__half, false) : DT_PREFILL_BY_D(__nv_bfloat16, false);
#undef DT_PREFILL_BY_D
#undef DT_PREFILL_GO
}

}  // namespace dt

#ifdef DT_BRINGUP
// Bring-up builds only: kernel probe bits and the buffer the probes write to.
extern "C" int dt_internal_set_prefill_options(int options) {
  dt::g_options = options;
  return 0;
}
extern "C" int dt_internal_set_prefill_dump(float* device_buffer) {
  dt::g_dbg = device_buffer;
  return 0;
}
#endif

// Sparse indexed attention (the operator of sparse_indexed.cu) of many tokens on tcgen05: 16-bit tensors, 64 query heads
// per KV head (or a multiple), head dim 256 or 512, values = keys -- the reference's prompt shape
// (Libraries/SwiftLLM/Sources/Models/DeepSeek4.swift:521-545).
//
// One CTA = one (token, KV head, 64 query heads) at a time, persistent over them.  A token's keys -- its window of raw
// rows, then its selected rows -- are gathered kTK at a time into a ring of shared-memory tiles in the swizzled layout that
// both products read: S = Q K^T takes the tile as [keys][dims] (M = 64 heads, N = kTK keys), O^T = K^T P^T takes the same
// bytes as [dims][keys] (M = 128 dims, N = 64 heads, D / 128 of them).  The transposed second product runs the tensor core
// at full height where [64 heads] x [256 dims] would use half of it, and its accumulator is 256 columns of TMEM, which
// leaves room for two S buffers of two accumulators each (neighbouring MMAs on one accumulator wait for each other: a chain
// of M = 64, N = 48 MMAs took 66 cycles each, twice its share of the pipe).  10 warps:
//   warps 0-3   softmax, one thread per head (the 64 rows of S are lanes 0-15 of the four TMEM quarters); P goes to shared
//               memory in two 16-bit parts per weight; O^T is rescaled only when a head's maximum grew by more than 2^8; at
//               the end O^T / l is stored, two neighbouring dims per 4-byte store
//   warps 4-7   gather: TMA loads of four named rows x 64 dims; entries that name no row read zeros; entries behind a
//               token's last valid one are left out (a prompt's first tokens have few)
//   warp 8      MMA issuer: QK(0) QK(1) | PV(0) QK(2) | PV(1) QK(3) | ...
//   warp 9      TMEM allocation, TMA of the next token's queries
// Why two parts: a weight of 16 bits relative to a maximum that is older than the tile makes the result's error against 64 bits
// 4 % larger than relative to the running maximum (2.07e-3 -> 2.15e-3 in bf16 for N(0,1) scores; 20 % where few keys carry the
// weight), and rescaling O^T for every growth costs more than the second part's products (659 and 608 us where one part and the
// older maximum take 514).  With two parts the error is the rounding of the result, 1.66e-3.
// Measured (prompt of 4096 tokens, 64 heads of 512, 128 + up to 512 keys each): 2110 us with warp-level MMAs, 608 us here
// (451 TFLOP/s of visible work).  Bound: the tensor pipe's operand reads from shared memory and the softmax warps' chain.  The
// products of one accumulator follow one another: with the accumulators in turn the call took 660 us.
// What set the time on the way: the gather.  With asynchronous 16-byte copies of four warps it moved 11 bytes per cycle
// (1775 us), with all the TMA loads issued by one warp, 68 cycles each, 7 (1446 us).
// Every mbarrier wait is bounded.  The softmax warps also meet at a named barrier once per tile; a wait that ran out is part
// of what they vote on there, so that all four leave together.
#include <type_traits>

#include "sm100_ptx.cuh"

namespace dt {
namespace {

constexpr int kThreads = 320;
constexpr int kHeads = 64;
constexpr int kTK = 48;      // keys per tile
constexpr int kBufs = 3;     // tiles in the ring
constexpr int kMaxD = 512;
constexpr int kSub = kTK * 128;                     // 64 dims of a tile: [kTK keys][128 bytes]
constexpr int kTileBytes = (kMaxD / 64) * kSub;
constexpr int kQSub = kHeads * 128;
constexpr int kQBytes = (kMaxD / 64) * kQSub;
constexpr int kPBytes = kHeads * 128;               // [64 heads][up to 64 keys], one part of the weights
constexpr int kSmemBytes = kQBytes + kBufs * kTileBytes + 2 * kPBytes + 1024 + 1024;
constexpr uint32_t kColS = 256;                     // S buffers behind the 256 columns of O^T
constexpr float kRescaleThreshold = 8.f;
static_assert(kSmemBytes <= 227 * 1024, "shared memory");
static_assert(kTK % 16 == 0 && kTK <= 64 && kSub % 1024 == 0, "tile");

struct Bars {
  uint64_t q_full, q_empty;
  uint64_t kv_full[kBufs], kv_empty[kBufs];
  uint64_t s_full[2];
  // One phase per tile: its weights are in shared memory; its P V has run.  The softmax warps wait for every tile's P V in
  // turn: a phase left out would let the next wait's parity be that of an older one.
  uint64_t p_full, pv_done;
  uint32_t tmem_base;
  int abort_flag;
  uint32_t valid[kBufs][4];  // bit 4 k + i of word w: row 4 (w + 4 k) + i of the tile holds a key
  uint32_t last[kBufs];      // the tile is its token's last
  float alpha[kHeads];       // rescale factors of the current tile
  float inv[kHeads];         // 1 / l of a finished token (its own array: a slower warp may still be rescaling)
};
static_assert(sizeof(Bars) <= 1024, "barrier area");

struct Args {
  void* o;
  const int32_t* selected;
  const void* sinks;
  float* lse;
  unsigned int* status;
  int64_t o_sb, o_ss, o_sh, sel_sb, sel_sq;
  int raw_rows_b, comp_rows_b;  // rows of the maps from one batch item to the next
  int raw_cols_h, comp_cols_h;  // columns from one KV head to the next
  int B, Sq, Hq, Hkv, D, Sr, Sc, n_sel;
  int groups, n_items;  // 64-head groups per KV head; tokens x KV heads x groups
  float scale_log2;
  int is_causal, window;
};

struct Item {
  int b, i, kvh, h0;
  int first, n_raw;
};

__device__ __forceinline__ Item decode_item(const Args& a, int item) {
  Item w;
  const int hg = item % (a.Hkv * a.groups), tok = item / (a.Hkv * a.groups);
  w.kvh = hg / a.groups;
  w.h0 = hg * kHeads;
  w.b = tok / a.Sq;
  w.i = a.Sq - 1 - (tok - w.b * a.Sq);  // the longest key lists (a prompt's last tokens) first
  const long long last = a.is_causal ? (long long)w.i + (a.Sr - a.Sq) : (long long)a.Sr - 1;
  const long long last_c = min(last, (long long)a.Sr - 1);
  const long long first = a.window > 0 ? max(0LL, (long long)w.i + (a.Sr - a.Sq) - a.window + 1) : 0LL;
  w.first = (int)first;
  w.n_raw = last_c >= first ? (int)(last_c - first + 1) : 0;
  return w;
}

// two floats -> 16-bit pair and back
template <typename T>
__device__ __forceinline__ uint32_t pack_pair(uint64_t x2) {
  float lo, hi;
  ptx::unpack_f32x2(x2, lo, hi);
  return std::is_same<T, __half>::value ? ptx::cvt_pack_f16(lo, hi) : ptx::cvt_pack_bf16(lo, hi);
}
template <typename T>
__device__ __forceinline__ uint64_t unpack_pair(uint32_t x) {
  if constexpr (std::is_same<T, __half>::value) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&x));
    return ptx::pack_f32x2(f.x, f.y);
  } else {
    return ptx::pack_f32x2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u));
  }
}

// OR of a predicate over the 128 softmax threads, the same answer for all of them.
__device__ __forceinline__ bool vote_any(bool x) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"((uint32_t)x) : "memory");
  return r != 0;
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
sparse_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_raw,
                      const __grid_constant__ CUtensorMap map_comp, const Args a) {
  constexpr int kBf16 = std::is_same<T, __half>::value ? 0 : 1;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t ring = base + kQBytes, pbuf = ring + kBufs * kTileBytes;
  Bars* bars = reinterpret_cast<Bars*>(base_ptr + kQBytes + kBufs * kTileBytes + 2 * kPBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_full, 1);
    ptx::mbar_init(&bars->q_empty, 1);
    for (int i = 0; i < kBufs; ++i) {
      ptx::mbar_init(&bars->kv_full[i], 4);  // one arrival per gather warp (and the bytes)
      ptx::mbar_init(&bars->kv_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) ptx::mbar_init(&bars->s_full[i], 1);
    ptx::mbar_init(&bars->p_full, 4);  // one arrival per softmax warp
    ptx::mbar_init(&bars->pv_done, 1);
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 9) {
    ptx::tmem_alloc(&bars->tmem_base, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile int* abort_flag = &bars->abort_flag;
  const int subs = a.D / 64;
  auto report = [&](unsigned code) {
    atomicCAS(a.status, 0u, code);
    *abort_flag = 1;
  };

  if (warp >= 4 && warp < 8) {
    // =========================== gather ===========================
    constexpr int kGroups = kTK / 16;  // groups of four rows per warp: w, w + 4, ...; lane 4 k + i looks up row i of the k-th
    const int gw = warp - 4;
    const bool on = ptx::elect_one();
    if (lane == 0) {
      ptx::prefetch_tensormap(&map_raw);
      ptx::prefetch_tensormap(&map_comp);
    }
    int buf = 0;
    uint32_t par = 1;  // parity of kv_empty: the first round over the ring passes at once
    bool ok = true;
    for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x) {
      const Item w = decode_item(a, item);
      const int32_t* sel = a.selected + w.b * a.sel_sb + (int64_t)w.i * a.sel_sq;
      int n_sel = a.Sc > 0 ? a.n_sel : 0;
      while (n_sel > 0) {  // up to the last entry that names a row
        const int at = n_sel - 1 - lane, idx = at >= 0 ? __ldg(sel + at) : -1;
        const uint32_t have = __ballot_sync(0xffffffffu, idx >= 0 && idx < a.Sc);
        if (have) {
          n_sel -= __ffs(have) - 1;
          break;
        }
        n_sel = max(0, n_sel - 32);
      }
      const int raw4 = (w.n_raw + 3) & ~3;  // raw rows first, rounded up so that a lane's four rows are of one tensor
      const int n_tiles = max(1, (raw4 + n_sel + kTK - 1) / kTK);  // a token without keys still runs one (fully hidden) tile
      for (int tile = 0; tile < n_tiles; ++tile) {
        int row = -1;  // -1: no key
        if (lane < 4 * kGroups) {
          const int key = tile * kTK + 4 * (gw + 4 * (lane >> 2)) + (lane & 3);
          if (key < raw4) {
            if (key < w.n_raw) row = w.first + key + w.b * a.raw_rows_b;
          } else if (key - raw4 < n_sel) {
            const int idx = __ldg(sel + key - raw4);
            if (idx >= 0 && idx < a.Sc) row = idx + w.b * a.comp_rows_b;
          }
        }
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->kv_empty[buf], par, abort_flag))) {
          if (lane == 0) report(2u);
          ok = false;
          break;
        }
        const uint32_t have = __ballot_sync(0xffffffffu, row >= 0);
        if (lane == 0) {
          bars->valid[buf][gw] = have;
          if (gw == 0) bars->last[buf] = tile == n_tiles - 1;
          ptx::mbar_arrive_expect_tx(&bars->kv_full[buf], (uint32_t)(subs * kGroups * 512));
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kGroups; ++k) {
          const bool raw = tile * kTK + 4 * (gw + 4 * k) < raw4;
          const CUtensorMap* map = raw ? &map_raw : &map_comp;
          const int col = w.kvh * (raw ? a.raw_cols_h : a.comp_cols_h);
          const int r0 = __shfl_sync(0xffffffffu, row, 4 * k), r1 = __shfl_sync(0xffffffffu, row, 4 * k + 1);
          const int r2 = __shfl_sync(0xffffffffu, row, 4 * k + 2), r3 = __shfl_sync(0xffffffffu, row, 4 * k + 3);
          const uint32_t dst = ring + buf * kTileBytes + (gw + 4 * k) * 512;
          if (on) {
#pragma unroll 4
            for (int s = 0; s < subs; ++s) ptx::tma_gather4_2d(dst + s * kSub, map, &bars->kv_full[buf], col + s * 64, r0, r1, r2, r3);
          }
        }
        __syncwarp();
        if (++buf == kBufs) { buf = 0; par ^= 1; }
      }
    }
  } else if (warp == 8) {
    // =========================== MMA issuer (the whole warp, one lane issues) ===========================
    const bool on = ptx::elect_one();
    constexpr uint32_t idesc_qk = ptx::make_idesc_f16(kBf16, kHeads, kTK, 0, 0);
    constexpr uint32_t idesc_pv = ptx::make_idesc_f16(kBf16, 128, kHeads, 1, 0);
    const uint64_t q_desc = ptx::make_smem_desc_sw128(base, 16, 1024);
    const uint64_t k_desc = ptx::make_smem_desc_sw128(ring, 16, 1024);    // [keys][dims]
    const uint64_t vt_desc = ptx::make_smem_desc_sw128(ring, kSub, 1024); // the same bytes as [dims][keys]
    const uint64_t p_desc = ptx::make_smem_desc_sw128(pbuf, 16, 1024);
    int kbuf = 0, vbuf = 0, n_item = 0;  // ring positions of the next Q K^T and the next P V
    uint32_t kpar = 0, gq = 0, gv = 0;   // tiles of Q K^T and of P V so far
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity, unsigned code) -> bool {
      if (__all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag))) return true;
      if (on) report(code);
      ok = false;
      return false;
    };
    for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x, ++n_item) {
      if (!wait(&bars->q_full, n_item & 1, 1u)) break;
      bool last_qk = false;  // the newest Q K^T was the token's last
      auto qk = [&]() -> bool {
        if (!wait(&bars->kv_full[kbuf], kpar, 1u)) return false;
        ptx::tc_fence_after();
        last_qk = bars->last[kbuf] != 0;
        const uint32_t s0 = tmem + kColS + (gq & 1u) * 128;
        const uint64_t kd = k_desc + (uint64_t)(kbuf * (kTileBytes >> 4));
#pragma unroll
        for (int s = 0; s < kMaxD / 64; ++s)
          if (s < subs) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              ptx::mma_ss_on(on, s0 + (ks & 1) * 64, q_desc + (uint64_t)((s * kQSub + ks * 32) >> 4),
                             kd + (uint64_t)((s * kSub + ks * 32) >> 4), idesc_qk, (s > 0 || ks > 1) ? 1u : 0u);
          }
        ptx::tc_commit_on(on, &bars->s_full[gq & 1u]);
        if (last_qk) ptx::tc_commit_on(on, &bars->q_empty);
        ++gq;
        if (++kbuf == kBufs) { kbuf = 0; kpar ^= 1; }
        return true;
      };
      if (!qk() || (!last_qk && !qk())) break;
      for (uint32_t t = 0; ok; ++t) {
        if (!wait(&bars->p_full, gv & 1u, 4u)) break;
        ptx::tc_fence_after();
        const uint64_t vd = vt_desc + (uint64_t)(vbuf * (kTileBytes >> 4));
#pragma unroll
        for (int mt = 0; mt < kMaxD / 128; ++mt)
#pragma unroll
          for (int ks = 0; ks < kTK / 16; ++ks)
#pragma unroll
            for (int part = 0; part < 2; ++part)  // the weights' high parts and what those leave over
              if (2 * mt < subs)
                ptx::mma_ss_on(on, tmem + mt * kHeads, vd + (uint64_t)((mt * 2 * kSub + ks * 2048) >> 4),
                               p_desc + (uint64_t)((part * kPBytes + ks * 32) >> 4), idesc_pv, (t > 0 || part > 0 || ks > 0) ? 1u : 0u);
        ptx::tc_commit_on(on, &bars->kv_empty[vbuf]);
        ptx::tc_commit_on(on, &bars->pv_done);
        ++gv;
        if (++vbuf == kBufs) vbuf = 0;
        if (!last_qk) {
          if (!qk()) break;
        } else if (gv == gq) {
          break;  // the token's last tile
        }
      }
    }
  } else if (warp == 9) {
    // =========================== queries ===========================
    if (lane == 0) {
      ptx::prefetch_tensormap(&map_q);
      int n_item = 0;
      for (int item = blockIdx.x; item < a.n_items; item += gridDim.x, ++n_item) {
        const Item w = decode_item(a, item);
        if (n_item > 0 && !ptx::mbar_wait(&bars->q_empty, (n_item - 1) & 1, abort_flag)) { report(2u); break; }
        ptx::mbar_arrive_expect_tx(&bars->q_full, (uint32_t)(subs * kQSub));
        for (int s = 0; s < subs; ++s) ptx::tma_load_4d(base_ptr + s * kQSub, &map_q, &bars->q_full, s * 64, w.i, w.h0, w.b);
      }
    }
  } else {
    // =========================== softmax / rescale / store (warps 0-3) ===========================
    const uint32_t tl = tmem + ((uint32_t)(warp << 5) << 16);
    const int head = warp * 16 + (lane & 15);  // lanes 16-31 carry no rows of S
    const bool mine = lane < 16;
    const float sl2 = a.scale_log2;
    uint32_t g = 0;
    int kbuf = 0;
    uint32_t kpar = 0;
    bool ok = true, lost = false;  // lost: a wait for P V ran out, part of what the next vote is about
    for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x) {
      const Item w = decode_item(a, item);
      float m = -INFINITY, l = 0.f;
      bool last = false;
      for (int t = 0; !last; ++t, ++g) {
        const uint32_t sb = g & 1u;
        bool failed = !__all_sync(0xffffffffu, ptx::mbar_wait(&bars->s_full[sb], (g >> 1) & 1u, abort_flag) &&
                                                   ptx::mbar_wait(&bars->kv_full[kbuf], kpar, abort_flag)) || lost;
        ptx::tc_fence_after();
        uint32_t s[kTK], s_odd[kTK];
#pragma unroll
        for (int c = 0; c < kTK / 16; ++c) {
          ptx::tmem_ld16(tl + kColS + sb * 128 + c * 16, s + c * 16);
          ptx::tmem_ld16(tl + kColS + sb * 128 + 64 + c * 16, s_odd + c * 16);
        }
        last = bars->last[kbuf] != 0;
        uint32_t valid[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) valid[i] = bars->valid[kbuf][i];
        if (++kbuf == kBufs) { kbuf = 0; kpar ^= 1; }
        ptx::tc_wait_ld();
#pragma unroll
        for (int r = 0; r < kTK; ++r) s[r] = __float_as_uint(__uint_as_float(s[r]) + __uint_as_float(s_odd[r]));
        const bool full = (valid[0] & valid[1] & valid[2] & valid[3]) == (1u << (kTK / 4)) - 1u;
        if (!full) {
#pragma unroll
          for (int r = 0; r < kTK; ++r)
            if (!((valid[(r >> 2) & 3] >> (((r >> 4) << 2) | (r & 3))) & 1u)) s[r] = 0xff800000u;  // -inf
        }
        float mx = __uint_as_float(s[0]), mx1 = __uint_as_float(s[1]);
#pragma unroll
        for (int r = 2; r < kTK; r += 4) {
          mx = ptx::max3(mx, __uint_as_float(s[r]), __uint_as_float(s[r + 1]));
          if (r + 3 < kTK) mx1 = ptx::max3(mx1, __uint_as_float(s[r + 2]), __uint_as_float(s[r + 3]));
        }
        const float m_cand = fmaxf(m, fmaxf(mx, mx1) * sl2);  // scale > 0
        const bool grow = mine && ((m_cand - m > kRescaleThreshold) || (m == -INFINITY && m_cand != -INFINITY));
        if (vote_any(grow || failed)) {
          if (vote_any(failed)) {
            if (failed) report(3u);
            ok = false;
            break;
          }
          const float m_new = grow ? m_cand : m;
          const float alpha = m_new == -INFINITY ? 1.f : fast_exp2(m - m_new);
          l *= alpha;
          m = m_new;
          if (t > 0) {
            // every thread holds dims, not heads, of O^T: the heads' factors go through shared memory
            if (mine) bars->alpha[head] = alpha;
            const bool late = !__all_sync(0xffffffffu, ptx::mbar_wait(&bars->pv_done, (g - 1) & 1u, abort_flag));
            if (vote_any(late)) {  // (also orders the factors' writes before the reads below)
              if (late) report(7u);
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            for (int c = 0; c < subs * 2; ++c) {  // 16 columns at a time
              uint32_t ov[16];
              ptx::tmem_ld16(tl + c * 16, ov);
              ptx::tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * bars->alpha[(c & 3) * 16 + i]);
              ptx::tmem_st16(tl + c * 16, ov);
            }
            ptx::tc_wait_st();
          }
        }
        const float neg_m = m == -INFINITY ? 0.f : -m;
        const uint64_t neg_m2 = ptx::pack_f32x2(neg_m, neg_m), scale2 = ptx::pack_f32x2(sl2, sl2);
        uint64_t lsum = 0ull;
        uint32_t pw[kTK / 2], rest[kTK / 2];
#pragma unroll
        for (int i = 0; i < kTK / 2; ++i) {
          const uint64_t x2 = ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1])), scale2, neg_m2);
          float x0, x1;
          ptx::unpack_f32x2(x2, x0, x1);
          const uint64_t p2 = ptx::pack_f32x2(fast_exp2(x0), fast_exp2(x1));
          lsum = ptx::add_f32x2(lsum, p2);
          pw[i] = pack_pair<T>(p2);
          rest[i] = pack_pair<T>(ptx::fma_f32x2(unpack_pair<T>(pw[i]), ptx::pack_f32x2(-1.f, -1.f), p2));
        }
        float s0, s1;
        ptx::unpack_f32x2(lsum, s0, s1);
        l += s0 + s1;
        // the previous tile's P V has read its weights (it ran behind this tile's Q K^T: usually over by now)
        if (g > 0) lost = !__all_sync(0xffffffffu, ptx::mbar_wait(&bars->pv_done, (g - 1) & 1u, abort_flag));
        if (mine && !lost) {
          const uint32_t prow = pbuf + (uint32_t)head * 128;
#pragma unroll
          for (int q = 0; q < kTK / 8; ++q) {
            const uint32_t at = prow + (uint32_t)((q ^ (head & 7)) << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(pw[4 * q]), "r"(pw[4 * q + 1]), "r"(pw[4 * q + 2]),
                         "r"(pw[4 * q + 3])
                         : "memory");
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + kPBytes), "r"(rest[4 * q]), "r"(rest[4 * q + 1]),
                         "r"(rest[4 * q + 2]), "r"(rest[4 * q + 3])
                         : "memory");
          }
        }
        ptx::fence_proxy_async_smem();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->p_full);
      }
      if (!ok) break;

      // ---- O^T / l -> global ----
      float m_f = m, inv = l > 0.f ? 1.f / l : 0.f;
      if (a.sinks) {  // one more score column without a value row
        const float sl = to_float(reinterpret_cast<const T*>(a.sinks)[w.h0 + head]) * kLog2e;
        m_f = fmaxf(m, sl);
        const float alpha = exp2f(m - m_f);
        l = l * alpha + exp2f(sl - m_f);
        inv = l > 0.f ? alpha / l : 0.f;
      }
      if (mine) bars->inv[head] = inv;
      if (a.lse && mine) a.lse[((int64_t)w.b * a.Hq + w.h0 + head) * a.Sq + w.i] = l > 0.f ? m_f * kLn2 + logf(l) : -INFINITY;
      const bool late = !__all_sync(0xffffffffu, ptx::mbar_wait(&bars->pv_done, (g - 1) & 1u, abort_flag)) || lost;
      if (vote_any(late)) {
        if (late) report(5u);
        ok = false;
        break;
      }
      ptx::tc_fence_after();
      T* obase = reinterpret_cast<T*>(a.o) + w.b * a.o_sb + (int64_t)w.i * a.o_ss + (int64_t)w.h0 * a.o_sh;
      const int odd = lane & 1;
      for (int mt = 0; mt < subs / 2; ++mt) {
        T* ocol = obase + mt * 128 + (warp << 5) + (lane & ~1) + odd * a.o_sh;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t ov[32];
          ptx::tmem_ld32(tl + mt * kHeads + c * 32, ov);
          ptx::tc_wait_ld();
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const float v0 = __uint_as_float(ov[2 * k]) * bars->inv[c * 32 + 2 * k];
            const float v1 = __uint_as_float(ov[2 * k + 1]) * bars->inv[c * 32 + 2 * k + 1];
            // the even lane keeps head 2 k of both dims, the odd one head 2 k + 1
            const float other = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
            const float lo = odd ? other : v0, hi = odd ? v1 : other;
            *reinterpret_cast<uint32_t*>(ocol + (int64_t)(c * 32 + 2 * k) * a.o_sh) = kBf16 ? ptx::cvt_pack_bf16(lo, hi) : ptx::cvt_pack_f16(lo, hi);
          }
        }
      }
      ptx::tc_fence_before();  // the next token's first P V overwrites O^T: its hand-off comes after these reads
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

int64_t row_stride(const dt_tensor4& t, int rows, const dt_sparse_indexed_params& p) {  // (a lone row may carry any stride)
  return rows > 1 ? t.stride_s : (int64_t)(p.Hkv - 1) * t.stride_h + p.D;
}

bool key_map_fits(const dt_tensor4& t, int rows, const dt_sparse_indexed_params& p) {
  const int64_t rs = row_stride(t, rows, p), cols = (int64_t)(p.Hkv - 1) * t.stride_h + p.D;
  if (rs <= 0 || rs % 8 || (p.Hkv > 1 && t.stride_h < 0) || cols >= (1LL << 31) || rs >= (1LL << 39)) return false;
  return p.B == 1 || (t.stride_b >= 0 && t.stride_b % rs == 0 && (p.B - 1) * (t.stride_b / rs) + rows < (1LL << 31));
}

bool key_map(CUtensorMap* map, const dt_tensor4& t, const dt_sparse_indexed_params& p, int rows, int& rows_b, int& cols_h) {
  const int64_t rs = row_stride(t, rows, p);
  rows_b = p.B > 1 ? (int)(t.stride_b / rs) : 0;
  cols_h = p.Hkv > 1 ? (int)t.stride_h : 0;
  return make_rows_tensor_map(map, t.ptr, (int64_t)(p.B - 1) * rows_b + rows, (int64_t)(p.Hkv - 1) * cols_h + p.D, rs, p.dtype);
}

template <typename T>
int launch_t(const dt_sparse_indexed_params& p, cudaStream_t stream) {
  Args a{};
  a.o = p.o.ptr;
  a.selected = p.selected; a.sinks = p.sinks; a.lse = p.lse;
  a.o_sb = p.o.stride_b; a.o_ss = p.o.stride_s; a.o_sh = p.o.stride_h;
  a.sel_sb = p.selected_stride_b; a.sel_sq = p.selected_stride_q;
  a.B = p.B; a.Sq = p.Sq; a.Hq = p.Hq; a.Hkv = p.Hkv; a.D = p.D; a.Sr = p.Sr; a.Sc = p.Sc; a.n_sel = p.n_selected;
  a.groups = p.Hq / p.Hkv / kHeads;
  a.n_items = p.B * p.Sq * p.Hkv * a.groups;
  a.scale_log2 = p.scale * kLog2e;
  a.is_causal = p.is_causal;
  a.window = p.sliding_window;
  a.status = device_status_word();
  if (!a.status) return DT_CUDA;
  // a box of 64 heads of one token: the map's token and head axes change places
  const dt_tensor4 view{p.q.ptr, p.q.stride_b, p.q.stride_h, p.q.stride_s};
  CUtensorMap mq;
  if (!make_bshd_tensor_map(&mq, view, p.B, p.Hq, p.Sq, p.D, p.dtype, kHeads)) return DT_UNSUPPORTED;
  // keys as rows of a 2-D map: batch items a whole number of rows apart, KV heads as more columns of a row
  CUtensorMap mr, mc;
  const bool raw = p.Sr > 0, comp = p.Sc > 0 && p.n_selected > 0;
  if (raw && !key_map(&mr, p.k_raw, p, p.Sr, a.raw_rows_b, a.raw_cols_h)) return DT_UNSUPPORTED;
  if (comp && !key_map(&mc, p.k_comp, p, p.Sc, a.comp_rows_b, a.comp_cols_h)) return DT_UNSUPPORTED;
  if (!raw) mr = mc;  // (no group of four names a row of the missing one)
  if (!comp) {
    mc = mr;
    a.n_sel = 0;
  }
  auto kern = sparse_tcgen05_kernel<T>;
  DT_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
  const int n_sm = device_sm_count();
  kern<<<a.n_items < n_sm ? a.n_items : n_sm, kThreads, kSmemBytes, stream>>>(mq, mr, mc, a);
  DT_CUDA_TRY(cudaGetLastError());
  return DT_OK;
}

}  // namespace

bool sparse_tcgen05_supported(const dt_sparse_indexed_params& p, bool same_kv) {
  if (p.D % 256 || p.D > kMaxD || !same_kv || !(p.scale > 0.f) || (p.Hq / p.Hkv) % kHeads) return false;
  const bool raw = p.Sr > 0, comp = p.Sc > 0 && p.n_selected > 0;
  if ((!raw && !comp) || (raw && !key_map_fits(p.k_raw, p.Sr, p)) || (comp && !key_map_fits(p.k_comp, p.Sc, p))) return false;
  // Few tokens leave SMs idle here, and the warp-level kernel spreads a token's keys over a cluster of CTAs, up to about 300 of
  // them (four per token and 64 heads for 16 tokens, two for 19).  Tokens x 64 heads, 640 keys each, there and here: head dim
  // 512: 8: 21.5 us and (like 16) 27, 16: 30.8 and 27.2, 18: 55 and 27.1, 64: 76 and 27; 4096 keys: 16: 134 and 135 us, 18: 248 and
  // 135.  Head dim 256: 16: 19.9 and 20.5, 18: 21.5 and 20.5, 20: 34.1 and 20.5; 4096 keys: 16: 82 and 95, 18: 91 and 95, 20: 156 and 95.
  const long long items = (long long)p.B * p.Sq * p.Hq / kHeads;
  return items >= (p.D == 256 ? 19 : 16) && items < (1LL << 30);
}

int launch_sparse_tcgen05(const dt_sparse_indexed_params& p, cudaStream_t stream) {
  return p.dtype == DT_F16 ? launch_t<__half>(p, stream) : launch_t<__nv_bfloat16>(p, stream);
}

}  // namespace dt

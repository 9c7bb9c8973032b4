// Attention of fp32 tensors on the tensor cores (the reference's upcastAttention,
// Libraries/SwiftDiffusion/Sources/Models/UNet.swift:217-265: fp32 scores, softmax over the keys, P*V).
//
// An fp32 number is the exact sum of three bf16 numbers: itself rounded to bf16, the rest rounded to bf16, and what that
// leaves.  A product x*y is then formed from the six partial products x_a*y_b with a + b <= 2; the dropped ones are below
// 2^-23 of it at worst, with either sign, and about 2^-26 on average: less than one fp32 rounding.  Q, K and V are split once per
// call by split_planes_kernel into a workspace.  The weights P are split in registers on their way into TMEM, their parts cut
// off instead of rounded, which takes an instruction less per part: there the dropped products are below 2^-22 at worst, of V's
// parts' signs.  (With the inputs' parts cut off as well all dropped products had the sign of the product and were up to 2^-21
// of it: scores of numbers like 1 + 2^-7 - 2^-23 came out short by that much.)
//
// The tensor core adds into fp32 accumulators without rounding to nearest, so long sums are kept off it: a block's scores
// take the small partial products first, and O is accumulated over ONE block of keys in TMEM and added to fp32 registers
// from there, rounded to nearest.
//
// f32_tcgen05_kernel: one CTA = one (batch, head, 128 query rows) at a time, persistent over the work items.  12 warps:
//   warp 0      TMA producer: Q planes per item, then K and V planes of kBN keys through a ring in the order
//               K(0) K(1) V(0) K(2) V(1) ...
//   warp 1      MMA issuer: S = Q K^T (6 * D/16 products per block, both operands in shared memory), O_blk = P V
//               (P in TMEM), ordered QK(0) QK(1) | PV(0) QK(2) | PV(1) QK(3) | ... over two S buffers
//   warp 2      TMEM allocation / release
//   warps 4-7   softmax of the first half of every block's keys, one thread per query row: scores -> weights -> three
//               bf16 planes over the S columns, then the previous block's O from TMEM into the row's fp32 accumulators
//   warps 8-11  the same for the second half, with a maximum, a sum and an O of their own; the two are put together when
//               the item ends
// The halves need nothing from each other while an item runs, so a scheduler has two warps to choose from, and a thread
// with 64 scores has registers left to work on several at a time (one warpgroup for all 128 spent 100 cycles on each pair
// of weights, the latency of the chain, and the call took 700 us).
// Measured (SD1.5 upcast self-attention: 2 images, 4096 tokens, 8 heads of 40): 3309 us on the CUDA cores (fp32 multiply-
// adds, 13 TFLOP/s), 299 us here in short bursts, 343 to 355 us one call after another for a second, when the power cap holds
// the clock at 1.8 instead of 1.97 GHz; error against 64 bits 1.2e-6 there, 2.6e-7 here (2-norm, relative).
// Per 128 x 128 scores at D = 40 the tensor pipe has 18 N=128 MMAs for Q K^T and 48 N=48 MMAs for P V.
// Every mbarrier wait is bounded, as in the half-precision kernel.
//
// Inputs that hold an infinity, a NaN, a magnitude of 2^58 and above (a score of 128 such products may leave the fp32
// range) or one below 2^-110 other than zero (its parts leave the bf16 range) are not for this kernel: split_planes_kernel reports them, f32_tcgen05_kernel then does nothing and the CUDA-core
// kernel behind it in the stream, which otherwise returns at once, computes the call.
#include "sm100_ptx.cuh"

namespace dt {
namespace {

constexpr int kBM = 128;
constexpr int kThreads = 384;
constexpr int kRegsLow = 80, kRegsHigh = 208;  // 128 * low + 256 * high <= 384 threads * 168 at launch
constexpr int kSplitThreads = 256;
constexpr int kSplitCtas = 1184;  // 8 per SM: the flag words in front of the planes are this many

// Head dims up to NPV (a multiple of 16, the N of the P V products); up to 64 a plane of a row is one 128-byte swizzle
// row, above it is two and the key block is halved to fit the same ring.
template <int NPV>
struct F32Cfg {
  static constexpr int kHalves = NPV > 64 ? 2 : 1;
  static constexpr int kBN = NPV > 64 ? 64 : 128;
  static constexpr int kQPlane = kHalves * kBM * 128;   // bytes of one plane of the Q tile
  static constexpr int kKvHalf = kBN * 128;
  static constexpr int kKvPlane = kHalves * kKvHalf;    // 16 KB either way
  static constexpr int kQBytes = 3 * kQPlane;
  static constexpr int kSlotBytes = 3 * kKvPlane;
  static constexpr int kSlots = NPV > 64 ? 2 : 3;
  static constexpr int kSmemBytes = kQBytes + kSlots * kSlotBytes + 256 + 2 * kBM * 4 + 1024;
  static constexpr int kHN = kBN / 2;                   // keys of a softmax warpgroup's half
  // TMEM columns of a buffer: S, whose halves the first two planes of the halves' P overwrite, and behind it the third
  static constexpr uint32_t kBufCols = kBN + kHN;
  static constexpr uint32_t kColO = 2 * kBufCols;       // two of NPV columns
  static_assert(kColO + 2 * NPV <= 512, "TMEM columns");
  static_assert(kSmemBytes <= 227 * 1024, "shared memory");
};

struct F32Bars {
  uint64_t q_full, q_empty;
  uint64_t s_full[2], p_full[2][2];  // [buffer], [half][buffer]
  uint64_t o_full[2];                // [half] completes once per block's P V
  uint64_t x_full, x_empty;          // the second half's O, maximum and sum of a finished item: there / read
  uint64_t kv_full[3], kv_empty[3];
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(F32Bars) <= 256, "barrier area");

struct F32Args {
  float* o;
  float* lse;
  int64_t o_sb, o_ss, o_sh;
  unsigned int* status;
  const uint32_t* flags;  // [kSplitCtas] non-zero: some input cannot be split
  uint32_t* any_flag;     // their union, written for the kernel behind this one
  int n_flags;
  int Sq, Sk, Hq, Hkv, D;
  int n_qt, n_items;
  float scale_log2;
};

struct SplitTensor {
  const float* src;
  uint4* dst;  // [B, S, H, 3, D] bf16
  int64_t sb, ss, sh;
  int S, H;
  unsigned begin, end;  // its 8-element pieces in the launch's numbering
};
struct SplitArgs {
  SplitTensor t[3];
  unsigned n_pieces;
  int per_row;  // D / 8
  uint32_t* flags;
};

// The bits of 2^58 (larger numbers, infinities and NaN all compare above them) and of 2^-110 (the last of a smaller number's
// 24 bits is below the smallest bf16, 2^-133; zero is fine).
__device__ __forceinline__ uint32_t out_of_range(float x) {
  const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
  return u != 0u && u - 0x08800000u >= 0x5c800000u - 0x08800000u ? 1u : 0u;
}

// Bound: HBM / L2 writes (10 bytes moved per element in, 4 read and 6 written).  One 8-element piece per thread and step:
// two 16-byte loads, three 16-byte stores.
__global__ void __launch_bounds__(kSplitThreads) split_planes_kernel(const SplitArgs a) {
  ptx::wait_for_previous();
  ptx::let_next_start();
  uint32_t bad = 0;
  for (unsigned g = blockIdx.x * kSplitThreads + threadIdx.x; g < a.n_pieces; g += gridDim.x * kSplitThreads) {
    const SplitTensor& t = g < a.t[0].end ? a.t[0] : g < a.t[1].end ? a.t[1] : a.t[2];
    const unsigned piece = g - t.begin;
    const unsigned row = piece / a.per_row, ch = piece - row * a.per_row;
    const unsigned tok = row / t.H, h = row - tok * t.H;
    const unsigned b = tok / t.S, s = tok - b * t.S;
    const float4* src = reinterpret_cast<const float4*>(t.src + b * t.sb + s * t.ss + h * t.sh + ch * 8);
    const float4 lo = __ldg(src), hi = __ldg(src + 1);
    const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint32_t w[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float x0 = x[2 * i], x1 = x[2 * i + 1];
      bad |= out_of_range(x0) | out_of_range(x1);
      // x = a + r, r = b + t: a and b to the nearest bf16 (both differences are exact)
      const uint32_t a0 = (__float_as_uint(x0) + 0x8000u) & 0xffff0000u, a1 = (__float_as_uint(x1) + 0x8000u) & 0xffff0000u;
      const float r0 = x0 - __uint_as_float(a0), r1 = x1 - __uint_as_float(a1);
      const uint32_t b0 = (__float_as_uint(r0) + 0x8000u) & 0xffff0000u, b1 = (__float_as_uint(r1) + 0x8000u) & 0xffff0000u;
      const float t0 = r0 - __uint_as_float(b0), t1 = r1 - __uint_as_float(b1);
      w[0][i] = __byte_perm(a0, a1, 0x7632);
      w[1][i] = __byte_perm(b0, b1, 0x7632);
      w[2][i] = __byte_perm(__float_as_uint(t0), __float_as_uint(t1), 0x7632);
    }
    uint4* dst = t.dst + (size_t)row * 3 * a.per_row + ch;
#pragma unroll
    for (int p = 0; p < 3; ++p) dst[p * a.per_row] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
  }
  const int any = __syncthreads_or((int)bad);
  if (threadIdx.x == 0) a.flags[blockIdx.x] = any ? 1u : 0u;
}

// The partial products in the order they are added: the small ones first.  (row operand's plane, column operand's plane)
__device__ constexpr int kProdA[6] = {2, 0, 1, 1, 0, 0};
__device__ constexpr int kProdB[6] = {0, 2, 1, 0, 1, 0};

template <int NPV>
__global__ void __launch_bounds__(kThreads, 1)
f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const F32Args a) {
  using C = F32Cfg<NPV>;
  constexpr int kBN = C::kBN;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t ring_smem = base + C::kQBytes;
  F32Bars* bars = reinterpret_cast<F32Bars*>(base_ptr + C::kQBytes + C::kSlots * C::kSlotBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  float* xch = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 256);  // [2][kBM]: the second half's maximum, sum

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_full, 1);
    ptx::mbar_init(&bars->q_empty, 1);
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&bars->s_full[i], 1);
      ptx::mbar_init(&bars->p_full[0][i], 4);  // one arrival per softmax warp
      ptx::mbar_init(&bars->p_full[1][i], 4);
      ptx::mbar_init(&bars->o_full[i], 1);
    }
    ptx::mbar_init(&bars->x_full, 4);
    ptx::mbar_init(&bars->x_empty, 4);
    for (int i = 0; i < C::kSlots; ++i) {
      ptx::mbar_init(&bars->kv_full[i], 1);
      ptx::mbar_init(&bars->kv_empty[i], 1);
    }
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  ptx::wait_for_previous();
  uint32_t bad = 0;
  for (int i = threadIdx.x; i < a.n_flags; i += kThreads) bad |= a.flags[i];
  const int skip = __syncthreads_or((int)bad);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.any_flag = skip ? 1u : 0u;
  if (skip) return;  // the whole grid alike, before anything was allocated
  if (warp == 2) {
    ptx::tmem_alloc(&bars->tmem_base, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile int* abort_flag = &bars->abort_flag;
  if (a.n_items <= (int)gridDim.x) ptx::let_next_start();  // (as in the half-precision kernel)
  const int nkv = (a.Sk + kBN - 1) / kBN, G = a.Hq / a.Hkv;
  const int dsteps = (a.D + 15) >> 4;  // k-steps of Q K^T (columns beyond D are zeros in both operands)

  if (warp < 4) {
    ptx::setmaxnreg_dec<kRegsLow>();
    if (warp == 0) {
      // =========================== TMA producer ===========================
      if (lane == 0) {
        ptx::prefetch_tensormap(&map_q);
        ptx::prefetch_tensormap(&map_k);
        ptx::prefetch_tensormap(&map_v);
        const int halves = (a.D + 63) >> 6;  // 64-column halves of a plane that exist
        int slot = 0, n_item = 0;
        uint32_t par = 1;  // parity of kv_empty: the first round over the ring passes at once
        bool ok = true;
        auto fail = [&]() {
          atomicCAS(a.status, 0u, 2u);
          *abort_flag = 1;
          ok = false;
          return false;
        };
        for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x, ++n_item) {
          const int qt = item % a.n_qt, bh = item / a.n_qt, h = bh % a.Hq, b = bh / a.Hq, kvh = h / G;
          auto load_kv = [&](const CUtensorMap* map, int j) -> bool {
            if (!ptx::mbar_wait(&bars->kv_empty[slot], par, abort_flag)) return fail();
            ptx::mbar_arrive_expect_tx(&bars->kv_full[slot], (uint32_t)(3 * halves * C::kKvHalf));
            for (int p = 0; p < 3; ++p)
              for (int hf = 0; hf < halves; ++hf)
                ptx::tma_load_4d(base_ptr + C::kQBytes + slot * C::kSlotBytes + p * C::kKvPlane + hf * C::kKvHalf, map,
                                 &bars->kv_full[slot], hf * 64, kvh * 3 + p, j * kBN, b);
            if (++slot == C::kSlots) { slot = 0; par ^= 1; }
            return true;
          };
          if (!load_kv(&map_k, 0)) break;
          if (n_item > 0 && !ptx::mbar_wait(&bars->q_empty, (n_item - 1) & 1, abort_flag)) { fail(); break; }
          ptx::mbar_arrive_expect_tx(&bars->q_full, (uint32_t)(3 * halves * kBM * 128));
          for (int p = 0; p < 3; ++p)
            for (int hf = 0; hf < halves; ++hf)
              ptx::tma_load_4d(base_ptr + p * C::kQPlane + hf * kBM * 128, &map_q, &bars->q_full, hf * 64, h * 3 + p, qt * kBM, b);
          if (nkv > 1 && !load_kv(&map_k, 1)) break;
          for (int j = 0; j < nkv && ok; ++j) ok = load_kv(&map_v, j) && (j + 2 >= nkv || load_kv(&map_k, j + 2));
        }
      }
    } else if (warp == 1) {
      // =========================== MMA issuer (the whole warp, one lane issues) ===========================
      const bool on = ptx::elect_one();
      constexpr uint32_t idesc_qk = ptx::make_idesc_f16(1, kBM, kBN, 0, 0);
      constexpr uint32_t idesc_pv = ptx::make_idesc_f16(1, kBM, NPV, 0, 1);
      const uint64_t q_desc = ptx::make_smem_desc_sw128(base, 16, 1024);
      const uint64_t k_desc = ptx::make_smem_desc_sw128(ring_smem, 16, 1024);
      const uint64_t v_desc = ptx::make_smem_desc_sw128(ring_smem, C::kKvHalf, 1024);
      int slot = 0, n_item = 0;
      uint32_t par = 0, g = 0;  // g: key blocks handed to the tensor pipe before this item; block g + j uses S buffer (g + j) & 1
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity, unsigned code) -> bool {
        if (__all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag))) return true;
        if (on) atomicCAS(a.status, 0u, code);
        *abort_flag = 1;
        ok = false;
        return false;
      };
      auto advance = [&]() {
        if (++slot == C::kSlots) { slot = 0; par ^= 1; }
      };
      for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x, ++n_item) {
        if (!wait(&bars->q_full, n_item & 1, 1u)) break;
        auto qk = [&](int j) -> bool {
          if (!wait(&bars->kv_full[slot], par, 1u)) return false;
          ptx::tc_fence_after();
          const uint32_t buf = (g + (uint32_t)j) & 1u;
          const uint64_t kd = k_desc + (uint64_t)(slot * (C::kSlotBytes >> 4));
#pragma unroll
          for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int ks = 0; ks < (NPV + 15) / 16; ++ks)
              if (ks < dsteps)
                ptx::mma_ss_on(on, tmem + buf * C::kBufCols,
                               q_desc + (uint64_t)((kProdA[i] * C::kQPlane + (ks >> 2) * (kBM * 128) + (ks & 3) * 32) >> 4),
                               kd + (uint64_t)((kProdB[i] * C::kKvPlane + (ks >> 2) * C::kKvHalf + (ks & 3) * 32) >> 4), idesc_qk,
                               (i | ks) ? 1u : 0u);
          ptx::tc_commit_on(on, &bars->s_full[buf]);
          ptx::tc_commit_on(on, &bars->kv_empty[slot]);
          if (j == nkv - 1) ptx::tc_commit_on(on, &bars->q_empty);
          advance();
          return true;
        };
        if (!qk(0) || (nkv > 1 && !qk(1))) break;
        for (int j = 0; j < nkv && ok; ++j) {
          const uint32_t gj = g + (uint32_t)j, buf = gj & 1u;
          const int left = a.Sk - j * kBN;
          if (!wait(&bars->kv_full[slot], par, 1u)) break;
          // both halves, then their MMAs in turn: neighbours in the pipe do not wait for each other's accumulator
          if (!wait(&bars->p_full[0][buf], (gj >> 1) & 1u, 4u) || !wait(&bars->p_full[1][buf], (gj >> 1) & 1u, 4u)) break;
          ptx::tc_fence_after();
          const uint32_t pb = tmem + buf * C::kBufCols;
          const uint64_t vd = v_desc + (uint64_t)(slot * (C::kSlotBytes >> 4));
          const int steps0 = min(C::kHN, left + 15) >> 4, steps1 = min(C::kHN, max(left - C::kHN, 1) + 15) >> 4;  // (P is zero beyond the keys)
#pragma unroll
          for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int ks = 0; ks < C::kHN / 16; ++ks)
#pragma unroll
              for (int hf = 0; hf < 2; ++hf)
                if (ks < (hf ? steps1 : steps0))
                  ptx::mma_ts_on(on, tmem + C::kColO + hf * NPV,
                                 pb + (kProdA[i] < 2 ? hf * C::kHN + kProdA[i] * (C::kHN / 2) : kBN + hf * (C::kHN / 2)) + ks * 8,
                                 vd + (uint64_t)((kProdB[i] * C::kKvPlane + (hf * (C::kHN / 16) + ks) * 2048) >> 4), idesc_pv,
                                 (i | ks) ? 1u : 0u);
          ptx::tc_commit_on(on, &bars->kv_empty[slot]);
          ptx::tc_commit_on(on, &bars->o_full[0]);
          ptx::tc_commit_on(on, &bars->o_full[1]);
          advance();
          if (j + 2 < nkv && !qk(j + 2)) break;  // into the columns the P V above has just read
        }
        g += (uint32_t)nkv;
      }
    }
  } else {
    ptx::setmaxnreg_inc<kRegsHigh>();
    // =========================== softmax / accumulation / store ===========================
    const int hf = (warp - 4) >> 2;  // which half of a block's keys
    const int row_in_tile = ((warp & 3) << 5) + lane;
    const uint32_t tl = tmem + ((uint32_t)((warp & 3) << 5) << 16), t_o = tl + C::kColO + hf * NPV;
    const float sl2 = a.scale_log2;
    const uint64_t scale2 = ptx::pack_f32x2(sl2, sl2);
    uint32_t g = 0;  // key blocks seen so far
    int n_item = 0;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity, unsigned code) -> bool {
      if (__all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag))) return true;
      atomicCAS(a.status, 0u, code);
      *abort_flag = 1;
      ok = false;
      return false;
    };
    for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x, ++n_item) {
      const int qt = item % a.n_qt, bh = item / a.n_qt, h = bh % a.Hq, b = bh / a.Hq;
      const int row = qt * kBM + row_in_tile;
      float m = -INFINITY, l = 0.f;
      uint64_t acc[NPV / 2];  // the row's output over this half of the keys, two columns each
#pragma unroll
      for (int i = 0; i < NPV / 2; ++i) acc[i] = 0ull;
      // a block's O (its P V has run) joins the row's accumulators
      auto add_block = [&](uint32_t block) -> bool {
        if (!wait(&bars->o_full[hf], block & 1u, 5u)) return false;
        ptx::tc_fence_after();
#pragma unroll
        for (int c = 0; c < NPV / 16; ++c) {
          uint32_t ov[16];
          ptx::tmem_ld16(t_o + c * 16, ov);
          ptx::tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 8; ++i)
            acc[c * 8 + i] = ptx::add_f32x2(acc[c * 8 + i], ptx::pack_f32x2(__uint_as_float(ov[2 * i]), __uint_as_float(ov[2 * i + 1])));
        }
        return true;
      };
      for (int j = 0; j < nkv; ++j, ++g) {
        const uint32_t buf = g & 1u, ts = tl + buf * C::kBufCols;
        if (!wait(&bars->s_full[buf], (g >> 1) & 1u, 3u)) break;
        ptx::tc_fence_after();
        uint32_t s[C::kHN / 32][32];
#pragma unroll
        for (int c = 0; c < C::kHN / 32; ++c) ptx::tmem_ld32(ts + hf * C::kHN + c * 32, s[c]);
        ptx::tc_wait_ld();
        const int left = a.Sk - j * kBN - hf * C::kHN;  // keys of this half of the block (none, or fewer: the last block's)
        if (left < C::kHN) {
#pragma unroll
          for (int c = 0; c < C::kHN / 32; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i >= left) s[c][i] = 0xff800000u;  // -inf
        }
        float mx = -INFINITY;
        {
          float mxc[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) mxc[e] = __uint_as_float(s[0][e]);
#pragma unroll
          for (int i = 4; i < C::kHN; i += 8)  // four chains of 3-input maxima
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int x = i + e, y = i + 4 + e;
              mxc[e] = y < C::kHN ? ptx::max3(mxc[e], __uint_as_float(s[x >> 5][x & 31]), __uint_as_float(s[y >> 5][y & 31]))
                                  : fmaxf(mxc[e], __uint_as_float(s[x >> 5][x & 31]));
            }
          mx = fmaxf(fmaxf(mxc[0], mxc[1]), fmaxf(mxc[2], mxc[3]));
        }
        const float m_new = fmaxf(m, mx * sl2);  // -inf while this half has seen no key at all; scale > 0
        const float alpha = m_new == -INFINITY ? 1.f : fast_exp2(m - m_new);
        const float neg_m = m_new == -INFINITY ? 0.f : -m_new;
        const uint64_t neg_m2 = ptx::pack_f32x2(neg_m, neg_m);
        uint64_t lsum[2] = {0ull, 0ull};
#pragma unroll
        for (int c = 0; c < C::kHN / 32; ++c) {
          uint32_t w[3][16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const uint64_t x2 = ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(s[c][2 * i]), __uint_as_float(s[c][2 * i + 1])),
                                               scale2, neg_m2);
            float x0, x1;
            ptx::unpack_f32x2(x2, x0, x1);
            const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
            lsum[i & 1] = ptx::add_f32x2(lsum[i & 1], ptx::pack_f32x2(p0, p1));
            // three planes, cut off and not rounded
            const float r0 = p0 - __uint_as_float(__float_as_uint(p0) & 0xffff0000u);
            const float r1 = p1 - __uint_as_float(__float_as_uint(p1) & 0xffff0000u);
            const float t0 = r0 - __uint_as_float(__float_as_uint(r0) & 0xffff0000u);
            const float t1 = r1 - __uint_as_float(__float_as_uint(r1) & 0xffff0000u);
            w[0][i] = __byte_perm(__float_as_uint(p0), __float_as_uint(p1), 0x7632);
            w[1][i] = __byte_perm(__float_as_uint(r0), __float_as_uint(r1), 0x7632);
            w[2][i] = __byte_perm(__float_as_uint(t0), __float_as_uint(t1), 0x7632);
          }
          ptx::tmem_st16(ts + hf * C::kHN + c * 16, w[0]);
          ptx::tmem_st16(ts + hf * C::kHN + C::kHN / 2 + c * 16, w[1]);
          ptx::tmem_st16(ts + kBN + hf * (C::kHN / 2) + c * 16, w[2]);
        }
        ptx::tc_wait_st();
        if (j > 0) {
          if (!add_block(g - 1)) break;
        } else if (hf == 1 && n_item > 0 && !wait(&bars->x_empty, (n_item - 1) & 1, 6u)) {
          break;  // (the other warpgroup still reads the previous item's O of this half)
        }
        if (__any_sync(0xffffffffu, m_new != m)) {
          const uint64_t alpha2 = ptx::pack_f32x2(alpha, alpha);
#pragma unroll
          for (int i = 0; i < NPV / 2; ++i) acc[i] = ptx::fma_f32x2(acc[i], alpha2, 0ull);
          l *= alpha;
          m = m_new;
        }
        // the weights are in TMEM and the O columns are free: P V of this block may run
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->p_full[hf][buf]);
        float s0, s1;
        ptx::unpack_f32x2(ptx::add_f32x2(lsum[0], lsum[1]), s0, s1);
        l += s0 + s1;
      }
      if (!ok || !add_block(g - 1)) break;
      if (hf == 1) {
        // this half's result to the other warpgroup: O through this half's TMEM columns, the rest through shared memory
#pragma unroll
        for (int c = 0; c < NPV / 16; ++c) {
          uint32_t ov[16];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float x, y;
            ptx::unpack_f32x2(acc[c * 8 + i], x, y);
            ov[2 * i] = __float_as_uint(x);
            ov[2 * i + 1] = __float_as_uint(y);
          }
          ptx::tmem_st16(t_o + c * 16, ov);
        }
        ptx::tc_wait_st();
        ptx::tc_fence_before();
        xch[row_in_tile] = m;
        xch[kBM + row_in_tile] = l;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->x_full);
        continue;
      }
      if (!wait(&bars->x_full, n_item & 1, 6u)) break;
      ptx::tc_fence_after();
      const float m1 = xch[row_in_tile], l1 = xch[kBM + row_in_tile];
      const float m_all = fmaxf(m, m1);  // finite: the first half of the first block holds a key
      const float f0 = fast_exp2(m - m_all), f1 = m1 == -INFINITY ? 0.f : fast_exp2(m1 - m_all);
      l = l * f0 + l1 * f1;
      const float inv = 1.f / l;  // l >= the weight of the row's maximum, 1
      float* orow = a.o + b * a.o_sb + (int64_t)row * a.o_ss + h * a.o_sh;
#pragma unroll
      for (int c = 0; c < NPV / 16; ++c) {
        uint32_t ov[16];
        ptx::tmem_ld16(t_o + NPV + c * 16, ov);
        ptx::tc_wait_ld();
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          float x, y, z, w;
          ptx::unpack_f32x2(acc[c * 8 + v * 2], x, y);
          ptx::unpack_f32x2(acc[c * 8 + v * 2 + 1], z, w);
          const float4 o4 = make_float4((x * f0 + __uint_as_float(ov[4 * v]) * f1) * inv, (y * f0 + __uint_as_float(ov[4 * v + 1]) * f1) * inv,
                                        (z * f0 + __uint_as_float(ov[4 * v + 2]) * f1) * inv, (w * f0 + __uint_as_float(ov[4 * v + 3]) * f1) * inv);
          if (row < a.Sq && c * 16 + v * 4 < a.D) *reinterpret_cast<float4*>(orow + c * 16 + v * 4) = o4;
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->x_empty);
      if (a.lse && row < a.Sq) a.lse[((int64_t)b * a.Hq + h) * a.Sq + row] = m_all * kLn2 + logf(l);
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

size_t plane_bytes(const dt_sdpa_params& p, int S, int H) {
  return ((size_t)p.B * S * H * p.D * 6 + 255) / 256 * 256;
}
// The first 4 KB of a workspace hold the split-KV ticket counters and stay as they are; then the flag words, their union
// and the planes.
constexpr size_t kTicketBytes = 4096, kFlagBytes = (kSplitCtas + 64) * 4;

template <int NPV>
int launch_t(const dt_sdpa_params& p, void* workspace, cudaStream_t stream) {
  using C = F32Cfg<NPV>;
  uint8_t* planes = static_cast<uint8_t*>(workspace) + kTicketBytes + kFlagBytes;
  uint32_t* flags = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(workspace) + kTicketBytes);
  F32Args a{};
  a.status = device_status_word();
  if (!a.status) return DT_CUDA;

  SplitArgs sp{};
  sp.per_row = p.D / 8;
  sp.flags = flags;
  const dt_tensor4* src[3] = {&p.q, &p.k, &p.v};
  CUtensorMap maps[3];
  for (int i = 0; i < 3; ++i) {
    const int S = i ? p.Sk : p.Sq, H = i ? p.Hkv : p.Hq;
    SplitTensor& t = sp.t[i];
    t.src = static_cast<const float*>(src[i]->ptr);
    t.dst = reinterpret_cast<uint4*>(planes);
    t.sb = src[i]->stride_b; t.ss = src[i]->stride_s; t.sh = src[i]->stride_h;
    t.S = S; t.H = H;
    t.begin = sp.n_pieces;
    sp.n_pieces += (unsigned)((size_t)p.B * S * H * sp.per_row);
    t.end = sp.n_pieces;
    // the planes as one more factor of the head axis: [B, S, 3 H, D]
    const dt_tensor4 view{planes, (int64_t)S * H * 3 * p.D, (int64_t)H * 3 * p.D, p.D};
    if (!make_bshd_tensor_map(&maps[i], view, p.B, S, 3 * H, p.D, DT_BF16, i ? C::kBN : kBM)) return DT_UNSUPPORTED;
    planes += plane_bytes(p, S, H);
  }
  const unsigned need = (sp.n_pieces + kSplitThreads - 1) / kSplitThreads;
  const unsigned split_ctas = need < (unsigned)kSplitCtas ? need : (unsigned)kSplitCtas;
  a.flags = flags;
  a.any_flag = flags + kSplitCtas;
  a.n_flags = (int)split_ctas;
  a.o = static_cast<float*>(p.o.ptr);
  a.lse = p.lse;
  a.o_sb = p.o.stride_b; a.o_ss = p.o.stride_s; a.o_sh = p.o.stride_h;
  a.Sq = p.Sq; a.Sk = p.Sk; a.Hq = p.Hq; a.Hkv = p.Hkv; a.D = p.D;
  a.n_qt = (p.Sq + kBM - 1) / kBM;
  a.n_items = a.n_qt * p.Hq * p.B;
  a.scale_log2 = p.scale * kLog2e;
  auto kern = f32_tcgen05_kernel<NPV>;
  DT_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
  const int n_sm = device_sm_count();
  DT_CUDA_TRY(launch_behind(split_planes_kernel, dim3(split_ctas), dim3(kSplitThreads), 0, stream, 1, sp));
  // CTAs that come in while the splitting pass runs out land where there is room, not spread over the SM pairs and dies as those of an ordinary
  // launch are.  Long calls lose more by that than the hidden launch gives: those of several rounds, and those of one round that leaves
  // a tenth to half of the SMs empty.  Us in a graph, ordinary launches before and after / overlapped / this rule: 2 x 6144 tokens, 10 heads of
  // 40 894 / 933 / 874, 10 heads of 64 856 / 900 / 860 (cool GPU); one image, 5200 tokens, 8 heads of 64 318 / 327 / 319; 2500 tokens, 5 heads of
  // 64 (100 items) 59.5 / 62.2 / 58.8, of 40 54.7 / 56.4 / 53.6.  Shorter calls gain (2 x 1800 tokens, 8 heads of 40, called from Python:
  // ordinary 86.7, overlapped 84.1), and so do all of head dims 65 to 80 (2 x 4100 tokens, 10 heads of 80: 740 / 706, ordinary 727).
  const bool uneven = a.n_items <= n_sm && 2 * a.n_items > n_sm && 10 * a.n_items <= 9 * n_sm && p.Sk > 1536;
  const bool rounds = a.n_items > n_sm && p.Sk > 2048;
  const int ctas = a.n_items < n_sm ? a.n_items : n_sm;
  if (NPV == 80 || !(uneven || rounds)) {
    DT_CUDA_TRY(launch_behind(kern, dim3(ctas), dim3(kThreads), C::kSmemBytes, stream, 1, maps[0], maps[1], maps[2], a));
  } else {
    kern<<<ctas, kThreads, C::kSmemBytes, stream>>>(maps[0], maps[1], maps[2], a);
    DT_CUDA_TRY(cudaGetLastError());
  }
  return launch_generic(p, stream, a.any_flag);  // returns at once unless the inputs could not be split
}

}  // namespace

// The plain operator on fp32 views whose rows are read and written 16 bytes at a time.  Above a head dim of 128 the row's
// accumulators no longer fit the registers; masks, windows, sinks, the causal rule and variable lengths stay on the
// CUDA-core kernel.
bool f32_mma_supported(const dt_sdpa_params& p) {
  if (p.dtype != DT_F32 || p.D % 8 || p.D > 128) return false;
  if (p.mask || p.is_causal || p.sliding_window > 0 || p.sinks || p.seq_offsets_q) return false;
  // (a score is below 2^123: times 2^4 it stays finite, and so does every difference from a maximum)
  if ((p.flags & DT_FLAG_FORCE_GENERIC) || !(p.scale > 0.f) || p.scale * kLog2e > 16.f) return false;
  // (128 x 128, one head of 40: 25.8 us on the CUDA cores, 13.3 here; 128 x 141, 8 heads 33.8 and 15.3: no size from a tile on is slower)
  if (p.Sq < kBM || p.Sk < kBM) return false;
  if (p.Hq > 65535 || p.B > 65535) return false;
  auto ok = [](const dt_tensor4& t) {
    return reinterpret_cast<uintptr_t>(t.ptr) % 16 == 0 && t.stride_b % 4 == 0 && t.stride_s % 4 == 0 && t.stride_h % 4 == 0;
  };
  if (!ok(p.q) || !ok(p.k) || !ok(p.v) || !ok(p.o)) return false;
  // 32-bit piece numbers and work items
  return ((double)p.B * p.Sq * p.Hq + 2.0 * p.B * p.Sk * p.Hkv) * (p.D / 8) < 2e9 && (double)p.B * p.Hq * (p.Sq / kBM + 1) < 2e9;
}

size_t f32_mma_workspace_bytes(const dt_sdpa_params& p) {
  return kTicketBytes + kFlagBytes + plane_bytes(p, p.Sq, p.Hq) + 2 * plane_bytes(p, p.Sk, p.Hkv);
}

int launch_f32_mma(const dt_sdpa_params& p, void* workspace, cudaStream_t stream) {
  if (p.D <= 48) return launch_t<48>(p, workspace, stream);
  if (p.D <= 64) return launch_t<64>(p, workspace, stream);
  if (p.D <= 80) return launch_t<80>(p, workspace, stream);
  return launch_t<128>(p, workspace, stream);
}

}  // namespace dt

// Numbers of 32 bits as sums of 16-bit ones: what the two fp32 attention kernels (f32_sm100.cu, f32_pair_sm100.cu) share.
#pragma once

#include "common.cuh"

namespace dt {

struct F32SplitTensor {
  const float* src;
  uint4* dst;  // [B, S, H, 3, D] bf16
  int64_t sb, ss, sh;
  int S, H;
  unsigned begin, end;  // its 8-element pieces in the launch's numbering
};
struct F32SplitArgs {
  F32SplitTensor t[3];
  unsigned n_pieces;
  int per_row;  // D / 8
  uint32_t* flags;
};

// The bits of 2^58 (larger numbers, infinities and NaN all compare above them) and of 2^-110 (the last of a smaller number's
// 24 bits is below the smallest bf16, 2^-133; zero is fine).
__device__ __forceinline__ uint32_t f32_out_of_range(float x) {
  const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
  return u != 0u && u - 0x08800000u >= 0x5c800000u - 0x08800000u ? 1u : 0u;
}

// x = a + r, r = b + t: a and b to the nearest bf16 (both differences are exact).  Returns whether a number cannot be split.
__device__ __forceinline__ uint32_t f32_three_parts(const float (&x)[8], uint4 (&out)[3]) {
  uint32_t w[3][4], bad = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float x0 = x[2 * i], x1 = x[2 * i + 1];
    bad |= f32_out_of_range(x0) | f32_out_of_range(x1);
    const uint32_t a0 = (__float_as_uint(x0) + 0x8000u) & 0xffff0000u, a1 = (__float_as_uint(x1) + 0x8000u) & 0xffff0000u;
    const float r0 = x0 - __uint_as_float(a0), r1 = x1 - __uint_as_float(a1);
    const uint32_t b0 = (__float_as_uint(r0) + 0x8000u) & 0xffff0000u, b1 = (__float_as_uint(r1) + 0x8000u) & 0xffff0000u;
    const float t0 = r0 - __uint_as_float(b0), t1 = r1 - __uint_as_float(b1);
    w[0][i] = __byte_perm(a0, a1, 0x7632);
    w[1][i] = __byte_perm(b0, b1, 0x7632);
    w[2][i] = __byte_perm(__float_as_uint(t0), __float_as_uint(t1), 0x7632);
  }
#pragma unroll
  for (int p = 0; p < 3; ++p) out[p] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
  return bad;
}

// Pieces first, first + step, ... of the launch: two 16-byte loads, three 16-byte stores each.  Returns whether one of them holds a
// number that cannot be split.
__device__ __forceinline__ uint32_t f32_split_planes(const F32SplitArgs& a, unsigned first, unsigned step) {
  uint32_t bad = 0;
  for (unsigned g = first; g < a.n_pieces; g += step) {
    const F32SplitTensor& t = g < a.t[0].end ? a.t[0] : g < a.t[1].end ? a.t[1] : a.t[2];
    const unsigned piece = g - t.begin;
    const unsigned row = piece / a.per_row, ch = piece - row * a.per_row;
    const unsigned tok = row / t.H, h = row - tok * t.H;
    const unsigned b = tok / t.S, s = tok - b * t.S;
    const float4* src = reinterpret_cast<const float4*>(t.src + b * t.sb + s * t.ss + h * t.sh + ch * 8);
    const float4 lo = __ldg(src), hi = __ldg(src + 1);
    const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint4 w[3];
    bad |= f32_three_parts(x, w);
    uint4* dst = t.dst + (size_t)row * 3 * a.per_row + ch;
#pragma unroll
    for (int p = 0; p < 3; ++p) dst[p * a.per_row] = w[p];
  }
  return bad;
}

// Where f32_sm100.cu lets f32_pair_sm100.cu compute a call: the room of Q's, K's and V's parts (6 bytes an element), a flag word per CTA of
// its splitting pass, and what splits V into bf16 parts should they be needed after all.
struct F32PairScratch {
  uint8_t* planes[3];
  uint32_t* flags;
  int n_flags;
  uint32_t *done, *no_parts;  // written: not zero where f32_sm100.cu's kernel has nothing to do; where the CUDA cores have the call
  const F32SplitArgs* v_parts;
};
bool f32_pair_pays(const dt_sdpa_params& p);
unsigned f32_pair_units(const dt_sdpa_params& p);
int launch_f32_pair(const dt_sdpa_params& p, const F32PairScratch& w, cudaStream_t stream);

}  // namespace dt

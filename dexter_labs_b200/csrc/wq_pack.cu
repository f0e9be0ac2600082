// The two ends of a packed weight's life: packing a dense weight (load time) and the dense
// weight back from its packed form.  Both are single passes bound by HBM; their arithmetic is the
// reference's (python/dexter/quant.py:75-133, python/dexter/ops/reference/gemm.py:51-73) bit for bit.
#include "wq_common.cuh"

namespace dx {

// ------------------------------------------------------------------ dequantise
// W[k,n] bf16 with the same bit-pattern arithmetic as the GEMM kernels.
//
// Bound by HBM: 2 bytes written and bits/8 read per weight (int4 3072 x 14336: 19.5 us, 5.7 TB/s, where one
// thread per weight with its own divisions took 180 us).  A thread converts 8 columns of 8
// packed rows: eight 8-byte loads in flight, scales and zero points fetched once for all of them,
// 16-byte stores, consecutive lanes on consecutive columns (256 B read and 512 B written per row
// and warp).  Eight rows because every group and plane boundary is a multiple of 8 (the rule
// below) and so scales never change inside a thread.
//
// int8: deq8 of two weights at a time, both differences and the product one instruction for the two.  (3072 x 14336 with
// zero points: 21.0 us; 21.7 with deq8.)
__device__ __forceinline__ uint32_t deq8_pair(uint32_t word, uint32_t high, uint32_t zero2, uint32_t scale2) {
  const uint32_t q0 = prmt(word, 0x4B000000u, 0x7650u + 2 * high), q1 = prmt(word, 0x4B000000u, 0x7651u + 2 * high);
  float lo, hi;
  asm("{\n\t.reg .b64 v, b, z, s;\n\tmov.b64 v, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 z, {%5, %6};\n\t"
      "mov.b64 s, {%7, %8};\n\tadd.rn.f32x2 v, v, b;\n\tadd.rn.f32x2 v, v, z;\n\tmul.rn.f32x2 v, v, s;\n\t"
      "mov.b64 {%0, %1}, v;\n\t}\n"
      : "=f"(lo), "=f"(hi)
      : "r"(q0), "r"(q1), "f"(-8388608.0f), "f"(-bf16lo_f32(zero2)), "f"(-bf16hi_f32(zero2)), "f"(bf16lo_f32(scale2)),
        "f"(bf16hi_f32(scale2)));
  return cvt_bf16x2(hi, lo);
}
template <int BITS, bool RELAID>
__global__ void __launch_bounds__(128)
wq_dequant_kernel(const uint8_t* __restrict__ qw, const __nv_bfloat16* __restrict__ scales,
                  const __nv_bfloat16* __restrict__ zeros, __nv_bfloat16* __restrict__ out, int N, int K,
                  int group) {
  const int n8 = N >> 3;
  const int rows = BITS == 4 ? K >> 1 : K;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int rc = idx / n8;
  if (rc >= (rows >> 3)) return;
  const int n = (idx - rc * n8) << 3;
  const int r0 = rc << 3;
  uint2 w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    w[i] = __ldcs(reinterpret_cast<const uint2*>(qw + static_cast<long long>(r0 + i) * N + n));
  constexpr int PLANES = BITS == 4 ? 2 : 1;
#pragma unroll
  for (int pl = 0; pl < PLANES; ++pl) {
    const int k0 = r0 + pl * rows;
    const long long so = static_cast<long long>(k0 / group) * N + n;
    const uint4 sv = __ldg(reinterpret_cast<const uint4*>(scales + so));
    const uint32_t s[4] = {sv.x, sv.y, sv.z, sv.w};
    uint32_t z[4];
    if (zeros != nullptr) {
      const uint4 zv = __ldg(reinterpret_cast<const uint4*>(zeros + so));
      z[0] = zv.x; z[1] = zv.y; z[2] = zv.z; z[3] = zv.w;
    } else {
      z[0] = z[1] = z[2] = z[3] = BITS == 4 ? 0x43084308u : 0x43004300u;  // 136 and 128: the midpoints
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t v[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {  // column pairs
        if (BITS == 4) {
          uint32_t pair;  // the two nibbles at bits 0 and 16
          if (RELAID) {   // row parity picks the half word, the plane the row of the pair
            const uint32_t word = h < 2 ? w[(i & ~1) | pl].x : w[(i & ~1) | pl].y;
            const uint32_t q = word >> (16 * (i & 1) + 8 * (h & 1));
            pair = (q & 0xFu) | ((q & 0xF0u) << 12);
          } else {
            const uint32_t word = h < 2 ? w[i].x : w[i].y;
            pair = prmt(word >> (4 * pl), 0u, (h & 1) ? 0x4342u : 0x4140u);
          }
          v[h] = deq4(pair, z[h], s[h]);
        } else {
          const uint32_t word = h < 2 ? w[i].x : w[i].y;
          v[h] = deq8_pair(word, h & 1, z[h], s[h]);
        }
      }
      __stcs(reinterpret_cast<uint4*>(out + static_cast<long long>(k0 + i) * N + n),
             make_uint4(v[0], v[1], v[2], v[3]));
    }
  }
}

// Any shape (output widths that are no multiple of 8, odd groups).  Rows start on any byte there, so lanes
// take single columns: consecutive lanes on consecutive bytes and bf16s, four columns 32 apart per
// lane, scales kept in registers from row to row.  (Eight consecutive columns per thread with scales
// looked up per weight: 72 us for int4 3072 x 14335.)
constexpr int kDequantRows = 16;  // packed rows per warp
template <int BITS>
__global__ void __launch_bounds__(256)
wq_dequant_cols_kernel(const uint8_t* __restrict__ qw, const __nv_bfloat16* __restrict__ scales,
                       const __nv_bfloat16* __restrict__ zeros, __nv_bfloat16* __restrict__ out, int N, int K,
                       int group, int relaid) {
  constexpr int PLANES = BITS == 4 ? 2 : 1;
  const int rows = BITS == 4 ? K >> 1 : K;
  const int r0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * kDequantRows;
  const int r1 = r0 + kDequantRows < rows ? r0 + kDequantRows : rows;
  const int n = blockIdx.x * 128 + (threadIdx.x & 31);
  if (r0 >= rows) return;
  uint32_t s[PLANES][4], z[PLANES][4];
  float z8[4];
  int left[PLANES];  // rows until the plane's next group
  auto load = [&](int pl, int gi) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (n + 32 * j >= N) continue;
      const long long so = static_cast<long long>(gi) * N + n + 32 * j;
      s[pl][j] = __bfloat16_as_ushort(scales[so]);
      if (BITS == 4) z[pl][j] = zeros ? __bfloat16_as_ushort(zeros[so]) : 0x4308u;
      else z8[j] = zeros ? __bfloat162float(zeros[so]) : 128.0f;
    }
  };
#pragma unroll
  for (int pl = 0; pl < PLANES; ++pl) {
#pragma unroll
    for (int j = 0; j < 4; ++j) s[pl][j] = z[pl][j] = 0u;
    const int k = r0 + pl * rows, gi = k / group;
    left[pl] = group - (k - gi * group);
    load(pl, gi);
  }
#pragma unroll 4
  for (int r = r0; r < r1; ++r) {
    uint32_t q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      q[j] = n + 32 * j >= N ? 0u
             : BITS == 4 && relaid ? fetch_q4(qw, N, rows, r, n + 32 * j, 1) | (fetch_q4(qw, N, rows, r + rows, n + 32 * j, 1) << 4)
                                   : qw[static_cast<long long>(r) * N + n + 32 * j];
#pragma unroll
    for (int pl = 0; pl < PLANES; ++pl) {
      if (left[pl]-- == 0) {
        load(pl, (r + pl * rows) / group);
        left[pl] = group - 1;
      }
      __nv_bfloat16* dst = out + (static_cast<long long>(r) + static_cast<long long>(pl) * rows) * N + n;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (n + 32 * j >= N) continue;
        const uint32_t v = BITS == 4 ? deq4(q[j] >> (4 * pl), z[pl][j], s[pl][j])
                                     : cvt_bf16x2(0.0f, deq8(q[j], 0, z8[j], __uint_as_float(s[pl][j] << 16)));
        dst[32 * j] = __ushort_as_bfloat16(static_cast<unsigned short>(v & 0xFFFFu));
      }
    }
  }
}

template <int BITS>
static int launch_dequant(const void* qweight, const void* scales, const void* zeros, void* out, int N, int K,
                          int group, int relaid, cudaStream_t stream) {
  const uint8_t* q = static_cast<const uint8_t*>(qweight);
  const __nv_bfloat16* s = static_cast<const __nv_bfloat16*>(scales);
  const __nv_bfloat16* z = static_cast<const __nv_bfloat16*>(zeros);
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  const int rows = BITS == 4 ? K / 2 : K;
  // Whole 8 x 8 blocks with one scale row each, and every vector access on its alignment.
  const uintptr_t p16 = reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(o);
  const long long chunks = static_cast<long long>(N >> 3) * (rows >> 3);
  if (N % 8 == 0 && rows % 8 == 0 && group % 8 == 0 && p16 % 16 == 0 && reinterpret_cast<uintptr_t>(q) % 8 == 0 &&
      chunks + 128 < (1ll << 31)) {
    const unsigned grid = static_cast<unsigned>((chunks + 127) / 128);
    if (BITS == 4 && relaid)
      wq_dequant_kernel<BITS, BITS == 4><<<grid, 128, 0, stream>>>(q, s, z, o, N, K, group);
    else
      wq_dequant_kernel<BITS, false><<<grid, 128, 0, stream>>>(q, s, z, o, N, K, group);
  } else {
    const dim3 grid((N + 127) / 128, (rows + 8 * kDequantRows - 1) / (8 * kDequantRows));
    if (grid.y > 65535) return DXB_ERR_SHAPE;
    wq_dequant_cols_kernel<BITS><<<grid, 256, 0, stream>>>(q, s, z, o, N, K, group, relaid);
  }
  return cudaGetLastError() == cudaSuccess ? DXB_OK : DXB_ERR_CUDA;
}

// -------------------------------------------------------------------- quantise
// Packs a dense bf16 weight [N, K] (nn.Linear style): per group of `group` consecutive k and per
// output n an fp32 scale (and zero point), codes round(w / scale + shift) clamped to the grid, the
// codes transposed to [K, N] (int8) or [K/2, N] (int4, row i low and row i + K/2 high nibble).
//
// 2 bytes read and bits/8 written per weight, once each; bound by instruction issue (int4 14336 x 3072:
// 35 us, 931 us as element-wise passes; the copy alone would
// take 17 us).  One CTA packs 64 outputs x
// two spans of 128 k (for int4 the two spans share their packed rows: k and k + K/2).  A half warp
// reads one output's span with one 16-byte load per lane (256 B runs), finds the group's extremes
// by shuffles in packed bf16, codes its 8 values in registers, and four outputs make the 32-bit
// words of the transposed tile, which goes through shared memory (swizzled: no bank conflicts) to
// leave as 64-byte rows.
//
// Arithmetic, in the order of the framework's tensor expressions on this device (so the bytes
// are those of that chain of element-wise passes): all fp32; division by a constant is
// multiplication by its rounded reciprocal, division by the scale is an exact division; rounding
// to nearest even.  The codes get there without dividing: a product with the reciprocal of
// the scale is within 1.2e-5 (int8: 1.1e-4) of the quotient's own rounded sum, so only values closer than
// that to a rounding boundary, and groups that the grid does not cover, take the division.
struct QuantGrid {
  float levels, inv_levels, mid;
  bool symmetric;
};
template <int BITS>
__device__ __forceinline__ QuantGrid quant_grid(bool symmetric) {
  constexpr float levels = BITS == 4 ? 15.0f : 255.0f;
  return QuantGrid{levels, 1.0f / levels, BITS == 4 ? 8.0f : 128.0f, symmetric};
}
// A clamp that lets NaN through, as the tensor library's does.
__device__ __forceinline__ float clamp_nan(float v, float lo, float hi) {
  return v != v ? v : fminf(fmaxf(v, lo), hi);
}
// Scale and shift of a group from its extremes (symmetric: hi = largest magnitude).
__device__ __forceinline__ void quant_scale(const QuantGrid& g, float lo, float hi, float& scale, float& shift) {
  if (g.symmetric) {
    const float peak = hi != hi ? hi : fmaxf(hi, 1e-8f);
    scale = __fmul_rn(__fmul_rn(2.0f, peak), g.inv_levels);
    shift = g.mid;
  } else {
    const float s = __fmul_rn(__fsub_rn(hi, lo), g.inv_levels);
    scale = s != s ? s : fmaxf(s, 1e-8f);
    shift = clamp_nan(rintf(__fdiv_rn(-lo, scale)), 0.0f, g.levels);
  }
}
// Packed-bf16 max / min that let NaN through.
__device__ __forceinline__ uint32_t max2_nan(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t min2_nan(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("min.NaN.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ float max_halves(uint32_t v) {
  return __uint_as_float(max2_nan(v, prmt(v, v, 0x1032u)) << 16);
}
__device__ __forceinline__ float min_halves(uint32_t v) {
  return __uint_as_float(min2_nan(v, prmt(v, v, 0x1032u)) << 16);
}

__device__ __forceinline__ float rcp_approx(float v) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
// One value's code by exact division.
__device__ __forceinline__ uint32_t quant_code(const QuantGrid& g, float w, float scale, float shift) {
  const float r = rintf(__fadd_rn(__fdiv_rn(w, scale), shift));
  return static_cast<uint32_t>(static_cast<uint8_t>(clamp_nan(r, 0.0f, g.levels)));
}
// Codes of a lane's 8 values, eight bytes in k order, from ONE multiply-add per value: with 192.5 (int8:
// 768.5) added, the sum's mantissa is a fixed-point number whose bits 16.. are the rounded code (int8
// after a shift by two) and whose low 16 bits say how far above a rounding boundary it lies.  The
// constant carries a margin as well, so values within the margin of a boundary are those with less than
// twice the margin there.  (Rounding by adding and subtracting 1.5 * 2^23 and taking the distance as a
// difference took three instructions more per value: 40 us for int4 14336 x 3072, 39 so.  Two multiply-adds per
// instruction, a minimum of three without sorting the halves first, and 16-byte stores: 37.5 -> 35.0, int8 43.7 -> 39.0.)
// `inside`: every value's sum lies on the grid or so little beside it that it is within the margin.
// PEAKS: `inv` went through quant_peaks, so that a group's extremes are no such case.
template <int BITS, bool PEAKS>
struct QuantFixed {
  static constexpr uint32_t kMargin = PEAKS ? 18 : BITS == 4 ? 2 : 16;  // in 2^-16
  static constexpr float kBase = (BITS == 4 ? 192.5f : 768.5f) + kMargin / 65536.0f;  // exact, as is shift + kBase
};
// Both values of a bf16 pair times `inv` plus `base`, in one instruction.
__device__ __forceinline__ void fma_pair(uint32_t x, float inv, float base, uint32_t& lo, uint32_t& hi) {
  asm("{\n\t.reg .b64 v, m, a;\n\tmov.b64 v, {%2, %3};\n\tmov.b64 m, {%4, %4};\n\tmov.b64 a, {%5, %5};\n\t"
      "fma.rn.f32x2 v, v, m, a;\n\tmov.b64 {%0, %1}, v;\n\t}\n"
      : "=r"(lo), "=r"(hi)
      : "r"(x << 16), "r"(x & 0xFFFF0000u), "f"(inv), "f"(base));
}
template <int BITS, bool PEAKS>
__device__ __forceinline__ uint2 quant_code8(const QuantGrid& g, const uint32_t (&x)[4], float scale, float inv,
                                             float shift, bool inside) {
  constexpr uint32_t kNear = 2 * QuantFixed<BITS, PEAKS>::kMargin;
  const float base = shift + QuantFixed<BITS, PEAKS>::kBase;
  uint32_t u[8], nearest = 0xFFFFFFFFu;
#pragma unroll
  for (int j = 0; j < 8; j += 2) fma_pair(x[j >> 1], inv, base, u[j], u[j + 1]);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (BITS == 8) u[j] <<= 2;
    if (j & 1) nearest = __vimin3_u16x2(nearest, u[j - 1], u[j]);  // of the low halves; the upper ones' is not used
  }
  if (!inside || (nearest & 0xFFFFu) < kNear) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (!inside || (u[j] & 0xFFFFu) < kNear)
        u[j] = quant_code(g, (j & 1) ? bf16hi_f32(x[j >> 1]) : bf16lo_f32(x[j >> 1]), scale, shift) << 16;
  }
  uint2 v = make_uint2(prmt(prmt(u[0], u[1], 0x0062u), prmt(u[2], u[3], 0x0062u), 0x5410u),
                       prmt(prmt(u[4], u[5], 0x0062u), prmt(u[6], u[7], 0x0062u), 0x5410u));
  if (PEAKS) {  // 16 -> 15 (bytes are 64 + code so far)
    v.x -= (v.x >> 4) & 0x01010101u;
    v.y -= (v.y >> 4) & 0x01010101u;
  }
  if (BITS == 4) {
    v.x &= 0x0F0F0F0Fu;
    v.y &= 0x0F0F0F0Fu;
  }
  return v;
}
// On the symmetric int4 grid the largest magnitude of every group falls on a rounding boundary: +-7.5 + 8,
// which sent a lane of every group to the division (53 us for 14336 x 3072, 41 so; 43 on the other grid).  The
// negative one's code (0 or 1) is found once per group, exactly, and the reciprocal is moved by 4e-5 so
// that both extremes land clearly on their codes' side (the positive one on 15 or 16, see above).
// Their distance from the boundary is then 3e-4; sums near any OTHER boundary move by at most 6.5 / 7.5
// of that, 2.6e-4, so a margin of 18 * 2^-16 = 2.75e-4 tells the two apart (all errors of computation:
// 1.2e-5).  int8 has its second boundary too close to the first for this (126.5 / 127.5).
__device__ __forceinline__ float quant_peaks(const QuantGrid& g, float peak, float scale, float inv, float shift) {
  return inv * (quant_code(g, -peak, scale, shift) == 0 ? 1.00004f : 0.99996f);
}
// Sums of extremes that miss the grid by rounding errors only are within the margin of a boundary.
template <int BITS>
__device__ __forceinline__ bool quant_inside(const QuantGrid& g, float lo, float hi, float inv, float shift) {
  constexpr float slack = BITS == 4 ? 1.5e-5f : 1.2e-4f;
  return __fmaf_rn(lo, inv, shift) >= -0.5f - slack && __fmaf_rn(hi, inv, shift) <= g.levels + 0.5f + slack;  // false for NaN
}
// The zero point as it is stored: int4 kernels build 128 + q, so their zero points carry the 128.
template <int BITS>
__device__ __forceinline__ __nv_bfloat16 stored_zero(float shift) {
  return __float2bfloat16_rn(BITS == 4 ? __fadd_rn(shift, 128.0f) : shift);
}
// Extremes of groups that no span covers (one scale per output channel, or odd group sizes):
// one warp per (output, group) reads the group's run of k; scale and shift go to fp32 scratch for
// the coding pass and to the packed weight.
template <int BITS>
__global__ void __launch_bounds__(256, 4)
wq_quant_stats_kernel(const __nv_bfloat16* __restrict__ w, float* __restrict__ scale32, float* __restrict__ shift32,
                      __nv_bfloat16* __restrict__ scales, __nv_bfloat16* __restrict__ zeros, int N, int K, int group,
                      int symmetric) {
  const QuantGrid g = quant_grid<BITS>(symmetric != 0);
  const int lane = threadIdx.x & 31;
  const int groups = K / group;
  const long long job = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (job >= static_cast<long long>(N) * groups) return;
  const int n = static_cast<int>(job / groups), gi = static_cast<int>(job - static_cast<long long>(n) * groups);
  const uint4* src = reinterpret_cast<const uint4*>(w + static_cast<long long>(n) * K + static_cast<long long>(gi) * group);
  uint32_t hi = 0xFF80FF80u, lo = 0x7F807F80u;  // -inf, +inf
#pragma unroll 4
  for (int i = lane; i < (group >> 3); i += 32) {
    const uint4 v = __ldg(src + i);
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (symmetric) {
        hi = max2_nan(hi, x[j] & 0x7FFF7FFFu);
      } else {
        hi = max2_nan(hi, x[j]);
        lo = min2_nan(lo, x[j]);
      }
    }
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    hi = max2_nan(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    if (!symmetric) lo = min2_nan(lo, __shfl_xor_sync(0xffffffffu, lo, d));
  }
  if (lane == 0) {
    float scale, shift;
    quant_scale(g, min_halves(lo), max_halves(hi), scale, shift);
    const long long o = static_cast<long long>(gi) * N + n;
    scale32[o] = scale;
    shift32[o] = shift;
    scales[o] = __float2bfloat16_rn(scale);
    if (zeros != nullptr) zeros[o] = stored_zero<BITS>(shift);
  }
}

// Outputs per CTA.  (128: a 14336 x 3072 weight is 2.3 rounds of CTAs on the chip and takes three.)
constexpr int kQuantOuts = 64;

// LPG: lanes per group (group = 8 * LPG: 32, 64 or 128, extremes found here), or 0: scales and
// shifts come from the pass above.
template <int BITS, int LPG, bool SYM>
__global__ void __launch_bounds__(256, 4)
wq_quant_pack_kernel(const __nv_bfloat16* __restrict__ w, const float* __restrict__ scale32,
                     const float* __restrict__ shift32, uint8_t* __restrict__ q, __nv_bfloat16* __restrict__ scales,
                     __nv_bfloat16* __restrict__ zeros, int N, int K, int group) {
  constexpr int kPlanes = BITS == 4 ? 1 : 2;  // spans that have packed rows of their own
  // [span][row][word of 4 outputs], words rotated by row / 8; the second span half a bank row on
  __shared__ uint32_t tile[kPlanes * (128 * 16 + 16)];
  auto cell = [&](int pl, int row, int wd) -> uint32_t& {
    return tile[pl * (128 * 16 + 16) + row * 16 + ((wd + (row >> 3)) & 15)];
  };
  const QuantGrid g = quant_grid<BITS>(SYM);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = lane >> 4, l = lane & 15;
  const int rows = BITS == 4 ? K >> 1 : K;      // packed rows
  const int row0 = blockIdx.x * (BITS == 4 ? 128 : 256);  // spans first: neighbouring CTAs read on in the same rows
  const int n0 = blockIdx.y * kQuantOuts;
  // this lane's 8 consecutive k
  const int k = (BITS == 4 ? half * rows + row0 : row0 + half * 128) + 8 * l;
  const bool k_ok = BITS == 4 ? row0 + 8 * l < rows : k < rows;
  const int gi = k_ok ? k / group : 0;
#pragma unroll 1
  for (int quad = warp; quad < kQuantOuts / 4; quad += 8) {
    uint4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int n = n0 + 4 * quad + i;
      v[i] = k_ok && n < N ? __ldcs(reinterpret_cast<const uint4*>(w + static_cast<long long>(n) * K + k))
                           : make_uint4(0u, 0u, 0u, 0u);
    }
    uint2 code[4];  // [output] its 8 codes
    if (LPG > 0) {
      // Extremes of the four outputs' groups: the first two butterfly steps halve the number of
      // outputs a lane carries, so it ends with those of ONE group (output `own`), computes that
      // group's scale and shift once, and hands them to the other lanes of the group.
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t x[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
        if (SYM) {
          hi[i] = max2_nan(max2_nan(x[0] & 0x7FFF7FFFu, x[1] & 0x7FFF7FFFu), max2_nan(x[2] & 0x7FFF7FFFu, x[3] & 0x7FFF7FFFu));
        } else {
          hi[i] = max2_nan(max2_nan(x[0], x[1]), max2_nan(x[2], x[3]));
          lo[i] = min2_nan(min2_nan(x[0], x[1]), min2_nan(x[2], x[3]));
        }
      }
      constexpr int D1 = LPG > 0 ? LPG / 2 : 1, D2 = LPG > 0 ? LPG / 4 : 1;
      const bool up1 = (l & D1) != 0, up2 = (l & D2) != 0;
      const int own = (up1 ? 2 : 0) + (up2 ? 1 : 0);
      uint32_t h2[2], l2[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        h2[i] = max2_nan(up1 ? hi[2 + i] : hi[i], __shfl_xor_sync(0xffffffffu, up1 ? hi[i] : hi[2 + i], D1));
        if (!SYM) l2[i] = min2_nan(up1 ? lo[2 + i] : lo[i], __shfl_xor_sync(0xffffffffu, up1 ? lo[i] : lo[2 + i], D1));
      }
      uint32_t h1 = max2_nan(up2 ? h2[1] : h2[0], __shfl_xor_sync(0xffffffffu, up2 ? h2[0] : h2[1], D2)), l1 = 0u;
      if (!SYM) l1 = min2_nan(up2 ? l2[1] : l2[0], __shfl_xor_sync(0xffffffffu, up2 ? l2[0] : l2[1], D2));
#pragma unroll
      for (int d = LPG / 8; d >= 1; d >>= 1) {
        h1 = max2_nan(h1, __shfl_xor_sync(0xffffffffu, h1, d));
        if (!SYM) l1 = min2_nan(l1, __shfl_xor_sync(0xffffffffu, l1, d));
      }
      const float hi_f = max_halves(h1), lo_f = SYM ? -hi_f : min_halves(l1);
      float scale, shift;
      quant_scale(g, lo_f, hi_f, scale, shift);
      float inv = rcp_approx(scale);
      const int inside = quant_inside<BITS>(g, lo_f, hi_f, inv, shift) ? 1 : 0;
      constexpr bool kPeaks = BITS == 4 && SYM;
      if (kPeaks) inv = quant_peaks(g, hi_f, scale, inv, shift);
      const int n_own = n0 + 4 * quad + own;
      if ((l & (D2 - 1)) == 0 && k_ok && n_own < N) {
        const long long o = static_cast<long long>(gi) * N + n_own;
        scales[o] = __float2bfloat16_rn(scale);
        if (zeros != nullptr) zeros[o] = stored_zero<BITS>(shift);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int from = (i >> 1) * D1 + (i & 1) * D2;  // a lane of this group that owns output i
        const uint32_t x[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
        const float sc = __shfl_sync(0xffffffffu, scale, from, LPG > 0 ? LPG : 32);
        const float iv = __shfl_sync(0xffffffffu, inv, from, LPG > 0 ? LPG : 32);
        const float sh = __shfl_sync(0xffffffffu, shift, from, LPG > 0 ? LPG : 32);
        const bool in = __shfl_sync(0xffffffffu, inside, from, LPG > 0 ? LPG : 32) != 0;
        code[i] = quant_code8<BITS, kPeaks>(g, x, sc, iv, sh, in);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int n = n0 + 4 * quad + i;
        const uint32_t x[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
        const long long o = static_cast<long long>(gi) * N + (n < N ? n : 0);
        const float scale = __ldg(scale32 + o), shift = __ldg(shift32 + o), inv = rcp_approx(scale);
        const float hi = max_halves(max2_nan(max2_nan(x[0], x[1]), max2_nan(x[2], x[3])));
        const float lo = min_halves(min2_nan(min2_nan(x[0], x[1]), min2_nan(x[2], x[3])));
        code[i] = quant_code8<BITS, false>(g, x, scale, inv, shift, quant_inside<BITS>(g, lo, hi, inv, shift));
      }
    }
    // 4 x 8 bytes -> the words of 8 rows (four outputs each)
    uint32_t word[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t a = h ? code[0].y : code[0].x, b = h ? code[1].y : code[1].x;
      const uint32_t c = h ? code[2].y : code[2].x, e = h ? code[3].y : code[3].x;
      const uint32_t ab0 = prmt(a, b, 0x5140u), ab1 = prmt(a, b, 0x7362u);
      const uint32_t ce0 = prmt(c, e, 0x5140u), ce1 = prmt(c, e, 0x7362u);
      word[4 * h] = prmt(ab0, ce0, 0x5410u);
      word[4 * h + 1] = prmt(ab0, ce0, 0x7632u);
      word[4 * h + 2] = prmt(ab1, ce1, 0x5410u);
      word[4 * h + 3] = prmt(ab1, ce1, 0x7632u);
    }
    if (BITS == 4) {
      // The half warps hold the low and the high nibbles of the same rows: each takes the even or
      // the odd rows of the pair.
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const uint32_t mine = half ? word[j + 1] : word[j];
        const uint32_t other = __shfl_xor_sync(0xffffffffu, half ? word[j] : word[j + 1], 16);
        const uint32_t packed = half ? (other | (mine << 4)) : (mine | (other << 4));
        cell(0, 8 * l + j + half, quad) = packed;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) cell(kPlanes - 1 ? half : 0, 8 * l + j, quad) = word[j];
    }
  }
  __syncthreads();
  if (N % 16 == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0) {
    // Whole 16-byte chunks of a row, four lanes a row.
    const int n = n0 + 16 * (lane & 3);
    uint8_t* dst = q + static_cast<long long>(row0 + (threadIdx.x >> 2)) * N + n;
#pragma unroll
    for (int i = 0; i < 2 * kPlanes; ++i) {
      const int r = (threadIdx.x >> 2) + 64 * i, wd = 4 * (lane & 3);
      const int pl = r >> 7, rr = r & 127;
      if (row0 + r < rows && n < N)
        *reinterpret_cast<uint4*>(dst) = make_uint4(cell(pl, rr, wd), cell(pl, rr, wd + 1), cell(pl, rr, wd + 2), cell(pl, rr, wd + 3));
      dst += 64ll * N;
    }
    return;
  }
  const bool words = N % 4 == 0 && (reinterpret_cast<uintptr_t>(q) & 3) == 0;
#pragma unroll 4
  for (int i = 2 * warp + half; i < kPlanes * 128; i += 16) {  // a half warp per row
    const int row = row0 + i;
    const uint32_t v = cell(i >> 7, i & 127, l);
    const int n = n0 + 4 * l;
    uint8_t* dst = q + static_cast<long long>(row) * N + n;
    if (words) {
      if (row < rows && n < N) *reinterpret_cast<uint32_t*>(dst) = v;
    } else {
      // rows that start on odd bytes: consecutive lanes store consecutive bytes
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int col = 16 * b + l;
        const uint32_t wv = __shfl_sync(0xffffffffu, v, 4 * b + (l >> 2), 16);
        if (row < rows && n0 + col < N)
          q[static_cast<long long>(row) * N + n0 + col] = static_cast<uint8_t>(wv >> (8 * (l & 3)));
      }
    }
  }
}

template <int BITS>
static int launch_quantize(const void* weight, void* qweight, void* scales, void* zeros, void* scratch, int N, int K,
                           int group, int symmetric, cudaStream_t stream) {
  const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(weight);
  uint8_t* q = static_cast<uint8_t*>(qweight);
  __nv_bfloat16* s = static_cast<__nv_bfloat16*>(scales);
  __nv_bfloat16* z = static_cast<__nv_bfloat16*>(zeros);
  const int rows = BITS == 4 ? K / 2 : K;
  const int span = BITS == 4 ? 128 : 256;
  const dim3 grid((rows + span - 1) / span, (N + kQuantOuts - 1) / kQuantOuts);
  if (grid.y > 65535) return DXB_ERR_UNSUPPORTED;
  if (dxb_quantize_scratch_bytes(N, K, group, BITS) == 0) {
    auto kernel = group == 128 ? (symmetric ? wq_quant_pack_kernel<BITS, 16, true> : wq_quant_pack_kernel<BITS, 16, false>)
                  : group == 64 ? (symmetric ? wq_quant_pack_kernel<BITS, 8, true> : wq_quant_pack_kernel<BITS, 8, false>)
                                : (symmetric ? wq_quant_pack_kernel<BITS, 4, true> : wq_quant_pack_kernel<BITS, 4, false>);
    kernel<<<grid, 256, 0, stream>>>(w, nullptr, nullptr, q, s, z, N, K, group);
  } else {
    const long long cells = static_cast<long long>(K / group) * N;
    float* scale32 = static_cast<float*>(scratch);
    wq_quant_stats_kernel<BITS><<<static_cast<unsigned>((cells + 7) / 8), 256, 0, stream>>>(
        w, scale32, scale32 + cells, s, z, N, K, group, symmetric);
    wq_quant_pack_kernel<BITS, 0, false><<<grid, 256, 0, stream>>>(w, scale32, scale32 + cells, q, s, z, N, K, group);
  }
  return cudaGetLastError() == cudaSuccess ? DXB_OK : DXB_ERR_CUDA;
}

}  // namespace dx

extern "C" {

// Groups of 32, 64 or 128 that the spans of the packing kernel cover whole (for int4 both
// halves of K in spans of 128) are done in one pass and need no scratch.
size_t dxb_quantize_scratch_bytes(int N, int K, int group_size, int bits) {
  if (N <= 0 || K <= 0 || group_size <= 0) return 0;
  const int rows = bits == 4 ? K / 2 : K;
  if ((group_size == 32 || group_size == 64 || group_size == 128) && rows % group_size == 0) return 0;
  return static_cast<size_t>(K / group_size) * N * 2 * sizeof(float);
}

int dxb_quantize(const void* weight, void* qweight, void* scales, void* zeros, void* scratch, int N, int K,
                 int group_size, int bits, int symmetric, void* cuda_stream) {
  using namespace dx;
  if (bits != 4 && bits != 8) return DXB_ERR_BITS;
  if (!weight || !qweight || !scales || (!symmetric && !zeros)) return DXB_ERR_NULL;
  if (N <= 0 || K <= 0 || group_size <= 0 || K % group_size) return DXB_ERR_SHAPE;
  // lanes take 8 consecutive k of one group with one aligned load
  if (K % (bits == 4 ? 16 : 8) || group_size % 8 || reinterpret_cast<uintptr_t>(weight) % 16) return DXB_ERR_UNSUPPORTED;
  if (dxb_quantize_scratch_bytes(N, K, group_size, bits) && !scratch) return DXB_ERR_WORKSPACE;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  void* z = symmetric ? nullptr : zeros;
  return bits == 4 ? launch_quantize<4>(weight, qweight, scales, z, scratch, N, K, group_size, symmetric ? 1 : 0, stream)
                   : launch_quantize<8>(weight, qweight, scales, z, scratch, N, K, group_size, symmetric ? 1 : 0, stream);
}

int dxb_dequantize_ex(const void* qweight, const void* scales, const void* zeros, void* w_out, int N,
                      int K, int group_size, int bits, int weight_layout, void* cuda_stream) {
  using namespace dx;
  if (bits != 4 && bits != 8) return DXB_ERR_BITS;
  if (!qweight || !scales || !w_out) return DXB_ERR_NULL;
  if (N <= 0 || K <= 0 || group_size <= 0 || K % group_size || (bits == 4 && K % 2))
    return DXB_ERR_SHAPE;
  if (weight_layout != DXB_LAYOUT_DEXTER && (weight_layout != DXB_LAYOUT_B200 || bits != 4 || K % 4 || N % 4))
    return DXB_ERR_UNSUPPORTED;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  return bits == 4 ? launch_dequant<4>(qweight, scales, zeros, w_out, N, K, group_size,
                                       weight_layout == DXB_LAYOUT_B200, stream)
                   : launch_dequant<8>(qweight, scales, zeros, w_out, N, K, group_size, 0, stream);
}

int dxb_dequantize(const void* qweight, const void* scales, const void* zeros, void* w_out, int N,
                   int K, int group_size, int bits, void* cuda_stream) {
  return dxb_dequantize_ex(qweight, scales, zeros, w_out, N, K, group_size, bits, DXB_LAYOUT_DEXTER, cuda_stream);
}

}  // extern "C"

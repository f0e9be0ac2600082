// GEMM for few tokens, and for the shapes the tcgen05 kernel cannot take (output widths that are no
// multiple of 16, groups of 32): weights straight from HBM into registers and through mma.sync.
//
// With up to 16 tokens a launch is a read of the weights, and what it costs beyond that is fixed:
// the tcgen05 pipeline sets up TMEM, barriers and rings, and hands every unit over three times, about
// 4 us in all around a read of 1 to 3 us.  Here a warp loads packed words, converts them in registers
// and multiplies at once; there is nothing to set up and one hand-over at the end.  The tensor work
// is far below what mma.sync delivers: at 16 tokens a weight byte carries 64 flops.
//
// CTA = 32 * CPW output columns x all K of up to 8 * MT tokens; its warps take interleaved steps of 32
// packed rows and add up through shared memory.  Each warp keeps a ring of steps of its own in
// shared memory, filled by cp.async (no registers and no barriers: a warp only waits for its own
// copies), so that weights, scales and activations of the next kStages - 1 steps are on their way.  (With the
// ring in registers, activations and scales only fit one step ahead and every step waited for
// L2: 9.2 us for one token x 3072 x 9216, 20 us for 14336 x 3072.)
// A lane owns packed rows 8c .. 8c+7 of a step and 4 * CPW columns (c = lane % 4, g = lane / 4): its
// activations are one 16-byte read per token and plane, and since a matrix product does not care how
// k is numbered, rows (8c + 4h .. 8c + 4h + 3) serve as the k indices {2c, 2c+1, 2c+8, 2c+9} of the
// h-th m16n8k16 product.  Columns are the products' m, tokens their n.  Few tiles and long K: a
// cluster shares a tile's steps and adds through distributed shared memory.
#pragma once
#include <type_traits>

#include "wq_common.cuh"

namespace dx {

struct SmallParams {
  const __nv_bfloat16* x;
  const uint8_t* qw;
  const __nv_bfloat16* scales;
  const __nv_bfloat16* zeros;
  const __nv_bfloat16* bias;
  __nv_bfloat16* out;
  long long ldx, ldo;
  int M, N, K, group;
  int rows;      // packed rows
  int steps;     // rows / 32
  int tiles_n;   // column tiles
  int tiles;     // column tiles x token blocks; tile t: token block t / tiles_n
  int cluster;   // CTAs that share a tile's K
  int epilogue;
  int group_shift;  // log2(group / 32) where that is a power of two, else -1
  int ring_bytes;   // all warps' rings (the sums lie over them afterwards)
};

// kSmallW4Sym: repacked and on the symmetric grid (no zero points).  Its sums and those of kSmallW8 come divided by
// kSymAcc.
enum : int { kSmallW4 = 0, kSmallW4Relaid = 1, kSmallW8 = 2, kSmallW4Sym = 3 };

__device__ __forceinline__ void mma_m16n8k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Copies of 16 or 4 bytes of which `bytes` exist (the rest becomes zero).
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global.L2::128B [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global.L2::128B [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
  return v;
}

// How the rows of packed weights and scales lie in memory:
//   kRows16       all chunks of 16 bytes whole and aligned
//   kRows8        widths that are a multiple of 8 only: packed rows in chunks of 8 bytes, scale rows as before
//   kRowsShifted  any width: the aligned 16-byte chunks that cover a row are copied (three instead of two, five of a
//                 scale row instead of four) and the words are put together from them.  The shift of a
//                 packed row is the same in every step (32 rows are a multiple of 16 bytes), so its addresses are
//                 set up once as in the other cases.
//   kRowsWords    tensors that do not start on 16 bytes: words of four bytes, nine copies a lane and step
// us with words / as it is now: int4 50 tokens 1536 x 1000 6.8 / 4.2 (shifted 5.2), 1536 x 1001 6.8 / 5.2, 8 tokens 2048 x
// 1990 4.3 / 3.8; int8 120 tokens 512 x 1003 6.35 / 4.8.
enum : int { kRows16 = 0, kRows8 = 1, kRowsShifted = 2, kRowsWords = 3 };

// One step of one warp's ring.  Packed rows are stored in the order r -> (r % 8) * 4 + r / 8, so that the
// four rows a warp reads with one instruction lie side by side (no bank conflicts).  Words: rows start
// on any byte, so 36 bytes from the aligned address before are kept (and 68 of the scale rows).
template <int KIND, int ROWS, int CPW, int MT>
struct SmallStage {
  static constexpr int kPlanes = KIND == kSmallW8 ? 1 : 2;
  static constexpr int kRow = ROWS == kRowsWords ? 36 : ROWS == kRowsShifted ? 48 : 32 * CPW;  // bytes of a packed row
  static constexpr int kScaleRow = ROWS == kRowsWords ? 68 : ROWS == kRowsShifted ? 80 : 64 * CPW;
  static constexpr int kX = 32 * kRow;                    // activations: [plane][token][32 k]
  static constexpr int kS = kX + kPlanes * MT * 512;      // scales [plane], then zero points [plane]
  static constexpr int kBytes = (kS + 2 * kPlanes * kScaleRow + 15) / 16 * 16;
  // (sixteen rings of four shifted steps with two planes and two token tiles are more than a CTA may have)
  static constexpr int kStages = CPW == 2 || (ROWS == kRowsShifted && kPlanes * MT == 4) ? 3 : 4;
};

template <int KIND, int ROWS, int CPW, int MT>
__global__ void __launch_bounds__(CPW == 1 ? 512 : 256, CPW == 1 ? 1 : 2) wq_gemm_small(const SmallParams p) {
  constexpr bool RAGGED = ROWS == kRowsWords, SHIFTED = ROWS == kRowsShifted;
  using St = SmallStage<KIND, ROWS, CPW, MT>;
  constexpr bool W4 = KIND != kSmallW8;
  constexpr int PLANES = St::kPlanes;
  constexpr int STAGES = St::kStages;
  constexpr int BN = 32 * CPW;
  constexpr int TOK = 8 * MT;
  constexpr int kRedRow = BN + 1;
  extern __shared__ __align__(16) uint8_t small_smem[];
  float* red = reinterpret_cast<float*>(small_smem);  // [warps][TOK][BN + 1], over the rings
  float* recv = reinterpret_cast<float*>(small_smem + p.ring_bytes);  // cluster: one slot per other CTA
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int c = lane & 3, g = lane >> 2;
  const int crank = p.cluster > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  const int stride = warps * p.cluster;  // steps between two of this warp
  const bool has_zero = KIND != kSmallW4Sym && p.zeros != nullptr;
  const uint32_t ring = smem_u32(small_smem) + warp * STAGES * St::kBytes;
  pdl_launch_dependents();
  if (p.cluster > 1) cluster_arrive_relaxed();  // "this CTA runs", before anyone writes to its shared memory
  bool waited = false;

  const int tile_first = static_cast<int>(blockIdx.x) / p.cluster;
  const int tile_step = static_cast<int>(gridDim.x) / p.cluster;
  for (int tile = tile_first; tile < p.tiles; tile += tile_step) {
    const int tblock = tile / p.tiles_n;
    const int n0 = (tile - tblock * p.tiles_n) * BN;
    const int m0 = tblock * TOK;
    const int toks = p.M - m0 < TOK ? p.M - m0 : TOK;
    const int first = crank * warps + warp;
    const int count = first < p.steps ? (p.steps - first + stride - 1) / stride : 0;

    // ---- copies of one step.  What a lane copies stays the same from step to step, so its addresses
    // are set up once and advanced: the conversion keeps the integer pipe busy enough (with
    // addresses computed per copy that pipe was 92 % busy and the launch half as fast).
    // A lane beyond the last column or token copies 0 bytes, which writes zeros.
    constexpr int CB = ROWS == kRows8 ? 8 : 16;  // bytes of a chunk
    constexpr int CH = St::kRow / CB;            // chunks per packed row
    const uint8_t* w_src[CH];
    uint32_t w_dst[CH];
    uint32_t w_have = 0;
    const uint8_t* s_src = nullptr;
    uint32_t s_dst = 0, s_have = 0;
    int s_first = 0;
    uintptr_t s_end = 0;
    const uintptr_t w_end = reinterpret_cast<uintptr_t>(p.qw) + static_cast<uintptr_t>(p.rows) * p.N;
    // A chunk as far as the tensor goes (beyond it zeros).
    auto copy_upto = [&](uint32_t dst, const uint8_t* src, const void* inside, uintptr_t end) {
      const long long room = static_cast<long long>(end - reinterpret_cast<uintptr_t>(src));
      cp_async16(dst, room > 0 ? src : inside, room >= 16 ? 16u : room > 0 ? static_cast<uint32_t>(room) : 0u);
    };
    const __nv_bfloat16* x_src[MT];
    uint32_t x_have[MT];
    const long long w_advance = 32ll * stride * p.N;
    if (!RAGGED) {
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const int q = lane + 32 * j, r = q / CH, h = q % CH;
        if (SHIFTED) {
          w_src[j] = reinterpret_cast<const uint8_t*>(
                         reinterpret_cast<uintptr_t>(p.qw + (32ll * first + r) * p.N + n0) & ~uintptr_t(15)) + 16 * h;
        } else {
          const int n = n0 + CB * h;  // h depends on the lane only: 32 is a multiple of CH
          w_have = n < p.N ? CB : 0u;
          w_src[j] = p.qw + (32ll * first + r) * p.N + (n < p.N ? n : 0);
        }
        w_dst[j] = ((r & 7) * 4 + (r >> 3)) * St::kRow + CB * h;
      }
      constexpr int SCH = St::kScaleRow / 16;
      const int rs = lane / SCH, h = lane % SCH;
      const int pl = PLANES == 2 ? rs & 1 : 0;
      const int n = n0 + 8 * h;
      const bool ok = rs < PLANES * (has_zero ? 2 : 1);
      const __nv_bfloat16* base = rs >= PLANES && has_zero ? p.zeros : p.scales;
      s_src = reinterpret_cast<const uint8_t*>(base + (SHIFTED || n < p.N ? n : 0));
      s_end = reinterpret_cast<uintptr_t>(base + static_cast<long long>(p.K / p.group) * p.N);
      s_dst = St::kS + (ok ? rs : 0) * St::kScaleRow + 16 * h;
      s_have = ok ? (SHIFTED || n < p.N ? 16u : 0u) : 0xFFFFFFFFu;  // all ones: nothing to copy
      s_first = pl * p.steps;
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const int t = 8 * mt + g;  // 8 tokens x 4 chunks of 16 bytes
      x_have[mt] = t < toks ? 16u : 0u;
      x_src[mt] = p.x + static_cast<long long>(t < toks ? m0 + t : 0) * p.ldx + 32 * first + 8 * c;
    }
    const uint32_t x_dst = St::kX + g * 64 + 16 * c;
    int w_step = first;  // the step that copy_w takes next (copy_x is always called in the same order)
    auto copy_w = [&](uint32_t slot_addr) {
      if (!RAGGED) {
#pragma unroll
        for (int j = 0; j < CH; ++j) {
          if (SHIFTED) copy_upto(slot_addr + w_dst[j], w_src[j], p.qw, w_end);
          else if (CB == 8) cp_async8(slot_addr + w_dst[j], w_src[j], w_have);
          else cp_async16(slot_addr + w_dst[j], w_src[j], w_have);
          w_src[j] += w_advance;
        }
        if (s_have != 0xFFFFFFFFu) {
          const int s32 = w_step + s_first;
          const int grp = p.group_shift >= 0 ? s32 >> p.group_shift : s32 / (p.group >> 5);
          const uint8_t* src = s_src + static_cast<long long>(grp) * (2 * p.N);
          if (SHIFTED)  // (s_src is 16 * h past the row's first column: rounded down, 16 * h past its first chunk)
            copy_upto(slot_addr + s_dst, reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(src) & ~uintptr_t(15)),
                      p.scales, s_end);
          else
            cp_async16(slot_addr + s_dst, src, s_have);
        }
      } else {
        const long long row0 = 32ll * w_step;
        const uintptr_t end = reinterpret_cast<uintptr_t>(p.qw) + static_cast<uintptr_t>(p.rows) * p.N;
#pragma unroll 3
        for (int j = 0; j < 9; ++j) {
          const int q = lane + 32 * j, r = q / 9, h = q - 9 * r;
          const uintptr_t a = ((reinterpret_cast<uintptr_t>(p.qw) + (row0 + r) * p.N + n0) & ~uintptr_t(3)) + 4 * h;
          const uint32_t have = a >= end ? 0u : end - a < 4 ? static_cast<uint32_t>(end - a) : 4u;
          cp_async4(slot_addr + ((r & 7) * 4 + (r >> 3)) * St::kRow + 4 * h, have ? reinterpret_cast<const void*>(a) : p.qw, have);
        }
        const int words = PLANES * (has_zero ? 2 : 1) * 17;
        const uintptr_t elems = static_cast<uintptr_t>(p.K / p.group) * p.N;
        for (int q = lane; q < words; q += 32) {
          const int rs = q / 17, h = q - 17 * rs;
          const int pl = PLANES == 2 ? rs & 1 : 0;
          const uintptr_t base = reinterpret_cast<uintptr_t>(rs >= PLANES ? p.zeros : p.scales);
          const uintptr_t s_end = base + 2 * elems;
          const uintptr_t a = ((base + 2 * (static_cast<uintptr_t>((w_step + pl * p.steps) / (p.group >> 5)) * p.N + n0)) &
                               ~uintptr_t(3)) + 4 * h;
          const uint32_t have = a >= s_end ? 0u : s_end - a < 4 ? static_cast<uint32_t>(s_end - a) : 4u;
          cp_async4(slot_addr + St::kS + rs * St::kScaleRow + 4 * h, have ? reinterpret_cast<const void*>(a) : p.qw, have);
        }
      }
      w_step += stride;
    };
    auto copy_x = [&](uint32_t slot_addr) {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        cp_async16(slot_addr + x_dst + mt * 512, x_src[mt], x_have[mt]);
        if (PLANES == 2) cp_async16(slot_addr + x_dst + TOK * 64 + mt * 512, x_src[mt] + p.rows, x_have[mt]);
        x_src[mt] += 32 * stride;
      }
    };

    float acc[2 * CPW][MT][4];
#pragma unroll
    for (int t = 0; t < 2 * CPW; ++t)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][mt][i] = 0.f;

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
      if (s < count) copy_w(ring + s * St::kBytes);
    // Activations may be the previous kernel's output; weights never are.
    if (!waited) { pdl_wait(); waited = true; }
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
      if (s < count) copy_x(ring + s * St::kBytes);
      cp_async_commit();
    }

    uint32_t st = ring, fill = ring + (STAGES - 1) * St::kBytes;
    const uint32_t ring_end = ring + STAGES * St::kBytes;
#pragma unroll 1
    for (int i = 0; i < count; ++i) {
      cp_async_wait<STAGES - 2>();
      __syncwarp();  // step i has landed for every lane, and every lane is done with step i - 1
      if (i + STAGES - 1 < count) {
        copy_w(fill);
        copy_x(fill);
      }
      cp_async_commit();
      uint32_t w[8 * CPW];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const uint32_t a = st + (r * 4 + c) * St::kRow;
        if (RAGGED) {
          // row 8c + r starts `off` bytes into its first word
          const uint32_t off = static_cast<uint32_t>(
              (reinterpret_cast<uintptr_t>(p.qw) + (32ll * (first + i * stride) + 8 * c + r) * p.N + n0) & 3);
          w[r] = __funnelshift_r(lds32(a + 4 * g), lds32(a + 4 * g + 4), 8 * off);
        } else if (SHIFTED) {
          const uint32_t off = ((8 * c + r) * p.N) & 15;  // as in every step, and n0 is a multiple of 32
          const uint32_t b = a + ((off + 4 * g) & ~3u);
          w[r] = __funnelshift_r(lds32(b), lds32(b + 4), 8 * (off & 3));
        } else if (CPW == 1) {
          w[r] = lds32(a + 4 * g);
        } else {
          const uint2 v = lds64(a + 8 * g);
          w[2 * r] = v.x;
          w[2 * r + CPW - 1] = v.y;
        }
      }
      // Scales (and zero points) of this lane's columns, two bf16 per word.
      auto row4 = [&](int pl, int rs, const __nv_bfloat16* base, int wd) -> uint2 {
        const uint32_t a = st + St::kS + rs * St::kScaleRow;
        if (!RAGGED && !SHIFTED) return lds64(a + (4 * CPW * g + 4 * wd) * 2);
        const int s32 = first + i * stride + pl * p.steps;
        const uint32_t grp = p.group_shift >= 0 ? s32 >> p.group_shift : s32 / (p.group >> 5);
        const uint32_t off = (static_cast<uint32_t>(reinterpret_cast<uintptr_t>(base)) + 2 * (grp * p.N + n0)) & (SHIFTED ? 15 : 3);
        const uint32_t b = a + off + 8 * g;
        return make_uint2(lds16(b) | (lds16(b + 2) << 16), lds16(b + 4) | (lds16(b + 6) << 16));
      };
      uint2 scale[PLANES][CPW];
      uint2 zero8[CPW];  // int8: zero points as byte patterns, see deq8_zeros
      uint32_t any = 0, odd = 0;
#pragma unroll
      for (int pl = 0; pl < PLANES; ++pl)
#pragma unroll
        for (int wd = 0; wd < CPW; ++wd) {
          scale[pl][wd] = row4(pl, pl, p.scales, wd);
          any |= scale[pl][wd].x | scale[pl][wd].y;
          if (KIND == kSmallW8) {
            zero8[wd] = make_uint2(0x00800080u, 0x00800080u);
            if (has_zero) {
              const uint2 zv = row4(pl, PLANES + pl, p.zeros, wd);
              zero8[wd] = make_uint2(deq8_zeros(zv.x, odd), deq8_zeros(zv.y, odd));
            }
          }
        }
      auto products = [&](auto way) {
        constexpr bool LARGE = decltype(way)::value;
#pragma unroll
        for (int pl = 0; pl < PLANES; ++pl) {
          uint4 xv[MT];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) xv[mt] = lds128(st + St::kX + (pl * TOK + 8 * mt + g) * 64 + 16 * c);
#pragma unroll
          for (int wd = 0; wd < CPW; ++wd) {
            const uint2 sv = scale[pl][wd];
            uint2 zv = make_uint2(0u, 0u);
            if (has_zero && (W4 || LARGE)) zv = row4(pl, PLANES + pl, p.zeros, wd);
#pragma unroll
            for (int th = 0; th < 2; ++th) {  // 16 columns: 4g + 2 th and the next, of word wd
              const int t = 2 * wd + th;
              const uint32_t sp = th ? sv.y : sv.x;
              const uint32_t zp = th ? zv.y : zv.x;
              uint32_t s0, s1, z0, z1;
              if (W4) {
                s0 = dup_lo(sp); s1 = dup_hi(sp);
                z0 = has_zero ? dup_lo(zp) : 0x43084308u;
                z1 = has_zero ? dup_hi(zp) : 0x43084308u;
                if (KIND == kSmallW4Sym) {
                  z0 = sym4_offset(s0); z1 = sym4_offset(s1);
                  s0 = sym4_scale_low(s0); s1 = sym4_scale_mid(s1);
                } else if (KIND == kSmallW4Relaid) {  // odd columns of a word are converted where they stand
                  s1 = mid_scale(s1);
                  z1 = has_zero ? mid_zero(z1) : 0xC000C000u;
                }
              } else if (!LARGE) {
                const uint32_t sv8 = deq8_scale(sp), zv8 = th ? zero8[wd].y : zero8[wd].x;
                s0 = dup_lo(sv8); s1 = dup_hi(sv8);
                z0 = dup_lo(zv8); z1 = dup_hi(zv8);
              } else {
                s0 = __float_as_uint(bf16lo_f32(sp) / kSymAcc);
                s1 = __float_as_uint(bf16hi_f32(sp) / kSymAcc);
                z0 = has_zero ? zp << 16 : __float_as_uint(128.0f);
                z1 = has_zero ? zp & 0xFFFF0000u : __float_as_uint(128.0f);
              }
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                uint32_t a[4];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                  const int pr = 2 * h + j;  // pair of rows 2 pr, 2 pr + 1
                  const uint32_t we = w[(2 * pr) * CPW + wd], wo = w[(2 * pr + 1) * CPW + wd];
                  if (KIND == kSmallW4Sym) {
                    const uint32_t W = (pl == 0 ? we : wo) >> (8 * th);
                    a[2 * j] = LARGE ? sym4_any(W, z0) : sym4_low(W, s0, z0);
                    a[2 * j + 1] = LARGE ? sym4_any(W >> 4, z1) : sym4_mid(W, s1, z1);
                  } else if (KIND == kSmallW4Relaid) {
                    const uint32_t W = (pl == 0 ? we : wo) >> (8 * th);
                    a[2 * j] = deq4(W, z0, s0);
                    a[2 * j + 1] = deq4_mid(W, z1, s1);
                  } else if (KIND == kSmallW4) {
                    const uint32_t P = prmt(we, wo, th ? 0x7632u : 0x5410u) >> (4 * pl);
                    a[2 * j] = deq4(P, z0, s0);
                    a[2 * j + 1] = deq4(P >> 8, z1, s1);
                  } else if (!LARGE) {
                    const uint32_t pairs = byte_pairs(we, wo, th);
                    a[2 * j] = deq8_zero(byte_pair(pairs, 0), s0, z0);
                    a[2 * j + 1] = deq8_zero(byte_pair(pairs, 1), s1, z1);
                  } else {
                    a[2 * j] = deq8_any(we, wo, 2 * th, __uint_as_float(z0), __uint_as_float(s0));
                    a[2 * j + 1] = deq8_any(we, wo, 2 * th + 1, __uint_as_float(z1), __uint_as_float(s1));
                  }
                }
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
                  mma_m16n8k16(acc[t][mt], a[0], a[1], a[2], a[3], h ? xv[mt].z : xv[mt].x, h ? xv[mt].w : xv[mt].y);
              }
            }
          }
        }
      };
      // (see sym4_any and deq8_any)
      constexpr bool kTwoWays = KIND == kSmallW4Sym || KIND == kSmallW8;
      if (kTwoWays && __any_sync(0xffffffffu, sym4_large(any) || odd != 0))
        products(std::integral_constant<bool, kTwoWays>{});
      else
        products(std::false_type{});
      fill = st;
      st += St::kBytes;
      if (st == ring_end) st = ring;
    }
    cp_async_wait<0>();

    // Sum over the warps (fixed order), then over the cluster's CTAs.
    __syncthreads();  // every warp is through with its ring
#pragma unroll
    for (int t = 0; t < 2 * CPW; ++t)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        float* dst = red + (warp * TOK + 8 * mt + 2 * c) * kRedRow + 4 * CPW * g + 2 * t;
        dst[0] = acc[t][mt][0];
        dst[kRedRow] = acc[t][mt][1];
        dst[1] = acc[t][mt][2];
        dst[kRedRow + 1] = acc[t][mt][3];
      }
    __syncthreads();
    if (p.cluster > 1 && tile == tile_first) cluster_wait();
    for (int i = threadIdx.x; i < toks * BN; i += blockDim.x) {
      const int m = i / BN, col = i - m * BN;
      float v = red[m * kRedRow + col];
      for (int k = 1; k < warps; ++k) v += red[(k * TOK + m) * kRedRow + col];
      if (crank > 0) {
        const uint32_t a = dsmem_addr(smem_u32(recv + (crank - 1) * TOK * BN + i), 0);
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
      } else {
        red[m * kRedRow + col] = v;  // only this thread reads this cell again
      }
    }
    if (p.cluster > 1) cluster_sync_all();
    if (crank == 0) {
      for (int i = threadIdx.x; i < toks * BN; i += blockDim.x) {
        const int m = i / BN, col = i - m * BN;
        if (n0 + col < p.N) {
          float v = red[m * kRedRow + col];
          for (int k = 1; k < p.cluster; ++k) v += recv[(k - 1) * TOK * BN + i];
          if (KIND == kSmallW4Sym || KIND == kSmallW8) v *= kSymAcc;
          __nv_bfloat16 o = __float2bfloat16_rn(v);
          if (p.bias != nullptr) o = __float2bfloat16_rn(__bfloat162float(o) + __bfloat162float(p.bias[n0 + col]));
          if (p.epilogue == DXB_EPILOGUE_GELU_TANH) o = __float2bfloat16_rn(gelu_tanh(__bfloat162float(o)));
          p.out[static_cast<long long>(m0 + m) * p.ldo + n0 + col] = o;
        }
      }
    }
    if (tile + tile_step < p.tiles) {  // the rings and receive slots are about to be filled again
      if (p.cluster > 1) cluster_sync_all();
      else __syncthreads();
    }
  }
}

}  // namespace dx

// Shared pieces of the weight-only quantised GEMM kernels for sm_100a: tile and
// ring constants, the bit-pattern dequantisation arithmetic, the barrier slots of
// the warp-specialised pipeline, and the host helpers that encode TMA tensor maps.
#pragma once
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <cstdlib>
#include <mutex>
#include <unordered_map>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/dexter_b200.h"
#include "sm100_ptx.cuh"

namespace dx {
// ------------------------------------------------------------------ constants
constexpr int kTileN = 128;      // weight columns per tile (UMMA M)
constexpr int kUnitRows = 64;    // packed rows per plane of a unit (one plane = 64 logical k)
constexpr int kQBytes = kTileN * kUnitRows;  // 8192: bytes of 64 packed rows of a tile
constexpr int kWStage = kQBytes;
// Packed-weight ring, always a multiple of kAStages.  Deeper ones fit, but what they ask for ahead of time delays the
// activations: us with 16 stages / 12 / 8, int4 83 tokens 3072 x 20096 19.5 / 18.9 / 18.6, 3072 x 14336 11.0 in all
// three, int8 16 tokens 3072 x 9216 9.7 (12) / 8.7.
constexpr int kMaxWStages = 8;
constexpr int kAStages = 4;      // dequantised-tile ring in TMEM
constexpr int kACol0 = 256;      // TMEM column where that ring starts
constexpr int kThreads = 768;    // 24 warps
constexpr int kDequantThreads = 128;  // one team
constexpr int kTeamWarps = kDequantThreads / 32;
constexpr int kEpilogueThreads = 128;
constexpr int kSmemBudget = 227 * 1024 - 4096;
constexpr int kMaxTiles = 16384;  // tile counters reserved in every workspace

// -------------------------------------------------------------- dequant math
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
__device__ __forceinline__ uint32_t sub_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t cvt_bf16x2(float hi, float lo) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
// (w & mask) | bits in ONE instruction.  Written as a C expression, its two constants become immediates of two
// instructions (a three-input LOP3 takes one immediate only), which makes the conversion, bound by the integer
// pipe, 20 % slower: 405 against 325 cycles per 128 x 128 int4 weights with sixteen warps at it.
__device__ __forceinline__ uint32_t and_or(uint32_t w, uint32_t mask, uint32_t bits) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(w), "r"(mask), "r"(bits));
  return d;
}
// Two nibbles (bits 0..3 and 16..19 of `w`) -> two bf16 weights.  OR-ing a nibble
// into the mantissa of 0x4300 gives 128 + q exactly; `zero2` holds 128 + zero
// point in both halves (0x4308 = 136.0 for the symmetric midpoint 8), so the
// subtract is exact and the multiply is the only rounding.
__device__ __forceinline__ uint32_t deq4(uint32_t w, uint32_t zero2, uint32_t scale2) {
  const uint32_t v = and_or(w, 0x000F000Fu, 0x43004300u);
  return mul_bf16x2(sub_bf16x2(v, zero2), scale2);
}
// The same for nibbles at bits 4..7 and 20..23, without shifting them down: as bf16 such a pattern is at most
// in the first normal binade, whose step is that of the subnormals, so its value is 16 q * 2^-133 for
// all sixteen q.  One exact multiply-add makes (q - zero) / 4 of it (times 2^127, plus `zero4` =
// -zero / 4), `scale4` = 4 * scale (for scales below 2^126) puts the factor back, and its multiply is
// the only rounding.  Two of
// four shifts of a word of nibbles go: with them the conversion, bound by the integer pipe, loses 32 of
// 400 instructions per 128 x 128 weights.
__device__ __forceinline__ uint32_t deq4_mid(uint32_t w, uint32_t zero4, uint32_t scale4) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(w & 0x00F000F0u), "r"(0x7F007F00u), "r"(zero4));
  return mul_bf16x2(d, scale4);
}
__device__ __forceinline__ uint32_t mid_scale(uint32_t scale2) { return mul_bf16x2(scale2, 0x40804080u); }
__device__ __forceinline__ uint32_t mid_zero(uint32_t zero2) {  // from 128 + zero
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(zero2), "r"(0xBE80BE80u), "r"(0x42004200u));
  return d;
}
// Symmetric grid (zero point 8): ONE multiply-add per two weights.  With the nibbles read as above (16 q or
// q times 2^-133), q * scale - 8 * scale is exact up to the final rounding -- 8 * scale is a bf16, which
// zero * scale in general is not -- so (q - 8) * scale needs no subtraction of its own.  2^133 * scale would
// overflow, so the weights come out divided by 64, and so do the products and their fp32 sums, bit for
// bit; whoever reads an accumulator multiplies by kSymAcc.  (Weights below 2^-120 lose bits: divided, they are bf16
// subnormals.  The quantiser's scales are 1e-8 and more.)  2^127 * scale still
// overflows for |scale| >= 2, where sym4_any converts the long way (never with a model's weights, so the
// check is one OR of exponents per unit: sym4_large).  Measured against deq4 / deq4_mid: 83 tokens 3072 x 14336
// 10.9 -> 10.65 us, 14336 x 3072 12.4 -> 11.85, 16 tokens 9.25 -> 9.0; the check costs 0.25 us of it.
constexpr float kSymAcc = 64.0f;
__device__ __forceinline__ bool sym4_large(uint32_t scales) { return (scales & 0x40004000u) != 0; }
// `offset`: sym4_offset of the scale, from which the scale comes back exactly.
__device__ __forceinline__ uint32_t sym4_any(uint32_t w, uint32_t offset) {  // bits 0..3, 16..19
  return mul_bf16x2(deq4(w, 0x43084308u, mul_bf16x2(offset, 0xC100C100u)), 0x3C803C80u);
}
__device__ __forceinline__ uint32_t sym4_low(uint32_t w, uint32_t scale, uint32_t offset) {  // bits 0..3, 16..19
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(w & 0x000F000Fu), "r"(scale), "r"(offset));
  return d;
}
__device__ __forceinline__ uint32_t sym4_mid(uint32_t w, uint32_t scale, uint32_t offset) {  // bits 4..7, 20..23
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(w & 0x00F000F0u), "r"(scale), "r"(offset));
  return d;
}
__device__ __forceinline__ uint32_t sym4_scale_low(uint32_t s2) { return mul_bf16x2(s2, 0x7F007F00u); }  // 2^(133-6)
__device__ __forceinline__ uint32_t sym4_scale_mid(uint32_t s2) { return mul_bf16x2(s2, 0x7D007D00u); }  // 2^(129-6)
__device__ __forceinline__ uint32_t sym4_offset(uint32_t s2) { return mul_bf16x2(s2, 0xBE00BE00u); }     // -8 * 2^-6
// One byte -> fp32 by bit pattern: 0x4B0000qq = 8388608 + q.  8388608 and the zero point are taken off in turn: added up
// first, zero points that are no whole numbers would be rounded to one.  The difference is exact as far as fp32's 24
// bits go (zero points whose last bit is 2^-8 or more have 16 of them), its product with an 8-bit
// scale then too, and the later cvt.rn to bf16 is the only rounding.
__device__ __forceinline__ float deq8(uint32_t word, uint32_t byte_sel, float zero, float scale) {
  const float f = __uint_as_float(prmt(word, 0x4B000000u, 0x7650u + byte_sel));
  return ((f - 8388608.0f) - zero) * scale;
}
// Bytes in GEMMs.  As bf16 the pattern 0x00qq is q * 2^-133 for all 256 bytes (the first normal binade has the
// subnormals' step), so two byte permutes per four bytes pair them up, and
//   without zero points: ONE multiply-add makes (q - 128) * scale / 64 of a pair; 128 * scale is a bf16, so the
//     rounding of the result is the only one, as in sym4_low;
//   with zero points that are whole numbers from 0 to 255, which a quantiser's are: the difference is exact in
//     that range and the multiply by 2^127 * scale is the only rounding.
// Weights and sums are divided by kSymAcc as on int4's symmetric grid, in deq8_any as well, with the same limit: weights
// below 2^-120 lose bits (of all bytes and significands without zero points, none at a scale of 2^-120, 128 of
// 32768 at 2^-121, 7128 at 2^-126).  2.5 and 3.5 instructions per two
// weights, of which 1.5 are on the integer pipe.  Scales of 2 and more take deq8_sym_any, or with zero points, as do other
// zero points, deq8_any, in bodies of their own: 3.5 and 9 instructions per two weights.  Measured, us with a
// conversion of 5 instructions through fp32 / so: 83 tokens 3072 x 14336 13.9 / 13.2, 14336 x 3072 15.2 / 14.2, with zero
// points 13.7 / 12.9; 16 tokens 3072 x 9216 10.4 / 9.5; one token 3072 x 3072 6.1 / 5.4.  (125 tokens 3072 x 8192 on
// clusters of two: 12.7 either way.)
__device__ __forceinline__ uint32_t byte_pairs(uint32_t w0, uint32_t w1, bool high) {  // columns 0, 1 or 2, 3 of two rows
  return prmt(w0, w1, high ? 0x7632u : 0x5410u);
}
__device__ __forceinline__ uint32_t byte_pair(uint32_t pairs, uint32_t odd) {  // one column of them, as 0x00qq00qq
  return prmt(pairs, 0u, odd ? 0x4341u : 0x4240u);
}
__device__ __forceinline__ uint32_t deq8_sym(uint32_t pair, uint32_t scale, uint32_t offset) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(pair), "r"(scale), "r"(offset));
  return d;
}
__device__ __forceinline__ uint32_t deq8_zero(uint32_t pair, uint32_t scale, uint32_t zero) {
  return mul_bf16x2(sub_bf16x2(pair, zero), scale);
}
__device__ __forceinline__ uint32_t deq8_scale(uint32_t s2) { return mul_bf16x2(s2, 0x7F007F00u); }   // 2^(133-6)
__device__ __forceinline__ uint32_t deq8_offset(uint32_t s2) { return mul_bf16x2(s2, 0xC000C000u); }  // -128 * 2^-6
// Two zero points as byte patterns; `odd` collects bits where one of them is no whole number from 0 to 255.
__device__ __forceinline__ uint32_t deq8_zeros(uint32_t z2, uint32_t& odd) {
  const uint32_t r = mul_bf16x2(z2, 0x00010001u);  // times 2^-133: exact for those, and back below
  odd |= (r & 0xFF00FF00u) | (mul_bf16x2(r, 0x7F007F00u) ^ mul_bf16x2(z2, 0x3C803C80u));
  return r;
}
// Without zero points, any scale: the difference is a bf16, so it goes to bf16 (divided by kSymAcc) and is multiplied there.
__device__ __forceinline__ uint32_t deq8_sym_any(uint32_t pair, uint32_t scale) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(pair), "r"(0x7F007F00u), "r"(0xC000C000u));  // q / 64 - 2
  return mul_bf16x2(d, scale);
}
// Any scale and zero point.  Byte `b` of two words (consecutive k of one column) -> a bf16 pair; `scale` is divided by
// kSymAcc.
__device__ __forceinline__ uint32_t deq8_any(uint32_t w0, uint32_t w1, uint32_t b, float zero, float scale) {
  return cvt_bf16x2(deq8(w1, b, zero, scale), deq8(w0, b, zero, scale));
}

__device__ __forceinline__ uint32_t dup_lo(uint32_t w) { return prmt(w, w, 0x1010u); }
__device__ __forceinline__ uint32_t dup_hi(uint32_t w) { return prmt(w, w, 0x3232u); }
__device__ __forceinline__ float bf16lo_f32(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi_f32(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// Value 0..15 of logical row k, column n of an int4 weight in either layout.
__device__ __forceinline__ uint32_t fetch_q4(const uint8_t* __restrict__ qw, int N, int half, int k, int n,
                                             int relaid) {
  const int plane = k < half ? 0 : 1;
  const int r = k - plane * half;  // packed row
  if (!relaid) return (qw[static_cast<long long>(r) * N + n] >> (4 * plane)) & 0xFu;
  const uint32_t word = reinterpret_cast<const uint32_t*>(qw)[(static_cast<long long>(r & ~1) + plane) * (N >> 2) + (n >> 2)];
  return (word >> (16 * (r & 1) + 4 * (n & 3))) & 0xFu;
}

// tanh-GELU of a value that has already been rounded to bf16, as the reference applies it
// between the FFN linears (torch gelu(approximate="tanh") on the bf16 output of the up
// projection, python/dexter/models/dreamzero/model.py:279-285): evaluated in fp32, rounded once.
// 0.5 (1 + tanh u) is the logistic function of 2u, which needs one exponential and one division and does
// not cancel for negative u.  The fast forms' documented errors are 2 + 1.2 |2u| units of fp32 for the
// exponential and 2 for the division: 5e-6 relative where the result reaches 2^-100, against 2e-3 for half a step
// of bf16.  Over all bf16 inputs, 5 results (from -10.06 to -10.31, below 2^-122) are not the exact value's
// rounding; 155 are with tanhf, which cancels below -3.5.  (tanhf with its branches also made the
// epilogue of 83 x 14336 outputs 7 us longer and its code evicted the main loop's.)
__device__ __forceinline__ float gelu_tanh(float v) {
  const float u2 = -1.5957691216057308f * (v + 0.044715f * v * v * v);
  return __fdividef(v, 1.0f + __expf(u2));
}

__device__ __forceinline__ uint32_t gelu_tanh2(uint32_t v) {  // of a bf16 pair
  return cvt_bf16x2(gelu_tanh(bf16hi_f32(v)), gelu_tanh(bf16lo_f32(v)));
}

__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// The same barrier, telling every thread whether any of them says yes.
__device__ __forceinline__ bool named_bar_any(int id, int nthreads, bool yes) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %3, 0;\n\tbar.red.or.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(any)
      : "r"(id), "r"(nthreads), "r"(yes ? 1u : 0u)
      : "memory");
  return any != 0;
}

// First unit of CTA c and the CTA that owns unit u, for `total` units cut into
// `ctas` contiguous ranges.
__host__ __device__ inline long long range_begin(long long c, long long total, long long ctas) {
  return c * total / ctas;
}
__host__ __device__ inline int owner_of(long long u, long long total, long long ctas) {
  return static_cast<int>(((u + 1) * ctas - 1) / total);
}

// ----------------------------------------------------------------- the kernel
// Barrier slots in shared memory.
// ready[t]: unit slot t has its activations in shared memory (TMA bytes) AND its
// dequantised weights in TMEM (128 arrivals of one team); free[t]: the MMAs that
// read slot t are done (one tcgen05.commit), so both may be overwritten.
constexpr int kBarFullW = 0, kBarEmptyW = kMaxWStages, kBarReady = 2 * kMaxWStages, kBarFree = kBarReady + kAStages,
              kBarAccFull = kBarFree + kAStages, kBarAccEmpty = kBarAccFull + 2, kNumBars = kBarAccEmpty + 2;

__device__ __forceinline__ uint32_t bar_count(int i) {
  if (i < kBarEmptyW) return 1;                    // full_w: producer's expect_tx
  // One arrival per WARP, not per thread: 128 arrivals on one barrier word serialise in
  // the shared-memory atomic unit and put ~500 cycles on every hand-over.
  if (i < kBarReady) return kTeamWarps;            // empty_w: the four warps of one team
  if (i < kBarFree) return kTeamWarps + 1;         // ready: team warps + activation producer
  if (i < kBarAccEmpty) return 1;                  // free, acc_full: one tcgen05.commit
  return kEpilogueThreads / 32;                    // acc_empty: the four epilogue warps
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}

// rank-2 or rank-3 tiled map; dims/box innermost first, strides in bytes for dims 1..rank-1.
inline bool make_map(CUtensorMap* m, const void* base, CUtensorMapDataType dt, int rank,
                     const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box,
                     CUtensorMapSwizzle sw) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t d[3], st[2];
  cuuint32_t bx[3], es[3] = {1, 1, 1};
  for (int i = 0; i < rank; ++i) { d[i] = dims[i]; bx[i] = box[i]; }
  for (int i = 0; i + 1 < rank; ++i) st[i] = strides_bytes[i];
  return fn(m, dt, rank, const_cast<void*>(base), d, st, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct DeviceInfo {
  int sms = 0;
  int l2_bytes = 0;
};
inline DeviceInfo& device_info() {
  static std::mutex mu;
  static std::unordered_map<int, DeviceInfo> infos;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  DeviceInfo& d = infos[dev];
  if (d.sms == 0) {
    cudaDeviceGetAttribute(&d.l2_bytes, cudaDevAttrL2CacheSize, dev);
    cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return d;
}

// Shapes whose tiles the tcgen05 kernel takes (int8 also wants whole units, see gemm_tc_supported).  The others go
// to wq_gemm_small, or to wq_gemm_simt where that cannot take them either.
inline bool tc_supported(int M, int N, int K, int group, int bits) {
  if (M < 1) return false;
  if (N % 16 || N < 16) return false;
  const int rows = bits == 4 ? K / 2 : K;
  if (bits == 4 && (K % 2)) return false;
  if (rows % kUnitRows) return false;
  if (group % kUnitRows || K % group) return false;
  if (K / group < 1) return false;
  // tiles = column tiles x token blocks of 128
  if (static_cast<long long>((N + kTileN - 1) / kTileN) * ((M + 127) / 128) > kMaxTiles) return false;
  return true;
}

// Head of a workspace: the status word, and at this many ints from it the address of another status word that
// a kernel sets as well, or 0.
constexpr size_t kStatusBytes = 256;
constexpr int kStatusAlso = 2;

// Polls (of about a quarter of a microsecond) a wait on a flag written by ANOTHER GPU makes
// before it gives up; set through dxb_set_wait_limit_ms, about a second by default.
unsigned wait_tries();

}  // namespace dx

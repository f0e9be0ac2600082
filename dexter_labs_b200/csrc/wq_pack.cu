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
          const float lo = deq8(word, 2 * (h & 1), 8388608.0f + bf16lo_f32(z[h]), bf16lo_f32(s[h]));
          const float hi = deq8(word, 2 * (h & 1) + 1, 8388608.0f + bf16hi_f32(z[h]), bf16hi_f32(s[h]));
          v[h] = cvt_bf16x2(hi, lo);
        }
      }
      __stcs(reinterpret_cast<uint4*>(out + static_cast<long long>(k0 + i) * N + n),
             make_uint4(v[0], v[1], v[2], v[3]));
    }
  }
}

// Any shape (output widths that are no multiple of 8, odd groups): a thread takes 8 consecutive
// packed bytes in memory order, whatever rows they fall in, so loads and stores stay wide where the
// row length would misalign them; scales are looked up per element (they hit L1).
template <int BITS>
__global__ void __launch_bounds__(128)
wq_dequant_flat_kernel(const uint8_t* __restrict__ qw, const __nv_bfloat16* __restrict__ scales,
                       const __nv_bfloat16* __restrict__ zeros, __nv_bfloat16* __restrict__ out, int N, int K,
                       int group, int relaid) {
  const int rows = BITS == 4 ? K >> 1 : K;
  const long long total = static_cast<long long>(rows) * N;
  const long long f = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) << 3;
  if (f >= total) return;
  const int cnt = total - f < 8 ? static_cast<int>(total - f) : 8;
  const int r_first = static_cast<int>(f / N), n_first = static_cast<int>(f - static_cast<long long>(r_first) * N);
  const bool wide = cnt == 8 && (reinterpret_cast<uintptr_t>(qw) & 7) == 0;
  uint32_t raw[2] = {0u, 0u};
  if (BITS == 8 || !relaid) {
    if (wide) {
      const uint2 v = __ldcs(reinterpret_cast<const uint2*>(qw + f));
      raw[0] = v.x; raw[1] = v.y;
    } else {
      for (int j = 0; j < cnt; ++j) raw[j >> 2] |= static_cast<uint32_t>(qw[f + j]) << (8 * (j & 3));
    }
  }
  constexpr int PLANES = BITS == 4 ? 2 : 1;
#pragma unroll
  for (int pl = 0; pl < PLANES; ++pl) {
    uint32_t v[4] = {0u, 0u, 0u, 0u};
    int r = r_first, n = n_first, gi = (r + pl * rows) / group;
    int left = group - ((r + pl * rows) - gi * group);  // rows until the next group
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j < cnt) {
        const long long so = static_cast<long long>(gi) * N + n;
        const uint32_t sb = __bfloat16_as_ushort(scales[so]);
        uint32_t o;
        if (BITS == 4) {
          const uint32_t zb = zeros ? __bfloat16_as_ushort(zeros[so]) : 0x4308u;
          const uint32_t q = relaid ? fetch_q4(qw, N, rows, r + pl * rows, n, 1)
                                    : (raw[j >> 2] >> (8 * (j & 3) + 4 * pl)) & 0xFu;
          o = deq4(q, zb, sb) & 0xFFFFu;
        } else {
          const float cz = 8388608.0f + (zeros ? __bfloat162float(zeros[so]) : 128.0f);
          o = cvt_bf16x2(0.0f, deq8(raw[j >> 2], j & 3, cz, __uint_as_float(sb << 16))) & 0xFFFFu;
        }
        v[j >> 1] |= o << (16 * (j & 1));
        if (++n == N) {
          n = 0;
          ++r;
          if (--left == 0) { left = group; ++gi; }
        }
      }
    }
    __nv_bfloat16* dst = out + static_cast<long long>(pl) * total + f;
    if (cnt == 8 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
      __stcs(reinterpret_cast<uint4*>(dst), make_uint4(v[0], v[1], v[2], v[3]));
    } else {
      for (int j = 0; j < cnt; ++j)
        dst[j] = __ushort_as_bfloat16(static_cast<unsigned short>((v[j >> 1] >> (16 * (j & 1))) & 0xFFFFu));
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
    const long long total = static_cast<long long>(rows) * N;
    const unsigned grid = static_cast<unsigned>((total + 1023) / 1024);
    wq_dequant_flat_kernel<BITS><<<grid, 128, 0, stream>>>(q, s, z, o, N, K, group, relaid);
  }
  return cudaGetLastError() == cudaSuccess ? DXB_OK : DXB_ERR_CUDA;
}

}  // namespace dx

extern "C" {

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

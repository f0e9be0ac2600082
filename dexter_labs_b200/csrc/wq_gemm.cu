// Weight-only quantised GEMM for sm_100a:  Y[M,N] = X[M,K] @ dequant(Q)[K,N] (+ bias)
//
//   Q       packed weights exactly as the reference quantiser lays them out
//           (python/dexter/quant.py:62-133): int4 = [K/2, N] bytes, low nibble is
//           row i, high nibble is row i + K/2 ("split-half"); int8 = [K, N] bytes.
//   scales  [K/G, N] bf16, zeros [K/G, N] bf16 or absent (symmetric).
//   W[k,n]  = bf16( (q - zero) * scale ), one rounding, bit-identical to the
//           reference's torch dequantize (python/dexter/ops/reference/gemm.py:51-73).
//   Y       = bf16( sum_k X*W in fp32 ), then bf16( Y + bias ) as a second rounding,
//           as the reference does (gemm.py:76-79).
//
// Tensor-core kernel (wq_gemm_tc): the weight tile is the 128-row UMMA "M"
// operand and the tokens are the UMMA "N" (swap-AB), so M = 83 tokens costs a
// 96-wide MMA instead of a 128-row one.  24 warps per CTA, one CTA per SM; per unit
// of 128 logical k x 128 columns (64 packed rows of int4, 128 rows of int8):
//   warps 0, 3   TMA producers: packed bytes of alternate units land in a
//                shared-memory ring (128 B swizzle).
//   warp 2       TMA producer: the matching activation k-slices (both nibble planes
//                in one 3-D box for int4).
//   warps 8-23   four dequant teams of four warps, one unit each in flight:
//                ld.shared of packed words, values -> bf16 by bit pattern (deq4, sym4_low,
//                deq8_sym; no int->float convert), written straight into TMEM with
//                tcgen05.st.16x128b (the dequantised tile never touches shared memory);
//                scales and zero points come from global memory one unit ahead.
//   warp 1       one lane issues tcgen05.mma (A = weights from TMEM, B = activations
//                from shared memory, fp32 accumulators in TMEM, two accumulators).
//   warps 4-7    epilogue: tcgen05.ld, bias, bf16 stores; or fp32 partial sums.
// How the (tile, unit) space is handed to CTAs is chosen per launch (make_plan,
// launch_tc): whole tiles per CTA; equal contiguous unit ranges (stream-K), where a tile
// shared by several CTAs is finished by the one that holds its first units, which adds the
// others' partial sums in a fixed order; or, for few tiles, one
// thread-block cluster per tile that splits K and adds through distributed shared memory.
// More than 128 tokens: every (token block, column tile) pair is a tile, one launch; on single CTAs
// (blocks of 128 tokens) or on CTA pairs (256 columns x up to 256 tokens).
// Few tokens on small weights, and shapes off these tiles, take wq_gemm_small (wq_small.cuh) instead.
#include "wq_common.cuh"
#include "wq_small.cuh"

namespace dx {
#ifdef DXB_TRACE
#define DX_TRACE(role, i) do { if (p.trace && (i) < 32) p.trace[(static_cast<long long>(blockIdx.x) * 8 + (role)) * 32 + (i)] = clock64() - t_start; } while (0)
#else
#define DX_TRACE(role, i) do { } while (0)
#endif


// ---------------------------------------------------------------------------
// Sum over tensor-parallel ranks fused into the row-parallel GEMM (dxb_gemm_opts.peer_*).
// Every rank owns a region of peer-mapped memory with the same layout:
//   [ control: epoch, exit count ][ arrived: tiles x 8 u32 ][ base: tiles x 8 u32 ]
//   [ recv: 2 parities x world x capacity bf16 ]
// Whoever finishes rows of a 128-column tile (an epilogue warp group or a cluster's owner
// CTA) rounds its fp32 partial sums to bf16 and stores them into slot `rank` of EVERY rank's
// receive buffer (plain 8-byte stores over NVLink, own region included), fences at system
// scope, and adds the number of rows it delivered to arrived[tile][rank] on every rank
// (red.release.sys).  It then waits (bounded) until arrived[tile][s] - base[tile][s] has
// reached the tile's row count for every sender s -- rows are counted, not chunks, so ranks
// may cut their tiles differently -- adds the world slots in rank order in fp32 (every rank
// computes the same bits), applies bias / activation and writes bf16.  The last CTA to
// leave adds the row count to base[][] and advances the epoch (= receive-buffer parity), so
// a captured graph replays.  A rank can be at most one call ahead of a peer, and it then
// writes the other parity.  Only plain peer loads/stores and system-scope fences.
constexpr int kPeerMaxRanks = 8;
constexpr int kFusedMaxTiles = 512;
constexpr size_t kFusedControlBytes = 256;
constexpr size_t kFusedCounterBytes = static_cast<size_t>(kFusedMaxTiles) * kPeerMaxRanks * sizeof(unsigned);
constexpr size_t kFusedHeaderBytes = kFusedControlBytes + 2 * kFusedCounterBytes;

struct PeerFuse {
  unsigned char* region[kPeerMaxRanks];  // every rank's region as mapped in this process
  long long capacity;                    // bf16 elements per receive slot (>= M * N)
  int rank, world;
  unsigned wait_tries;                   // polls of ~0.25 us before a wait gives up
};

__device__ __forceinline__ unsigned* fused_arrived(unsigned char* region, int tile, int sender) {
  return reinterpret_cast<unsigned*>(region + kFusedControlBytes) + tile * kPeerMaxRanks + sender;
}
__device__ __forceinline__ unsigned* fused_base(unsigned char* region, int tile, int sender) {
  return reinterpret_cast<unsigned*>(region + kFusedControlBytes + kFusedCounterBytes) +
         tile * kPeerMaxRanks + sender;
}
__device__ __forceinline__ __nv_bfloat16* fused_recv(const PeerFuse& pf, int owner, unsigned parity, int sender) {
  return reinterpret_cast<__nv_bfloat16*>(pf.region[owner] + kFusedHeaderBytes) +
         (static_cast<long long>(parity) * pf.world + sender) * pf.capacity;
}
__device__ __forceinline__ void red_release_sys_add(unsigned* ptr, unsigned v) {
  asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(ptr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire_sys_u32(const unsigned* ptr) {
  unsigned v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
  return v;
}
// Deliver four consecutive columns of one token row to slot `rank` of every rank.
__device__ __forceinline__ void fused_push4(const PeerFuse& pf, unsigned parity, long long elem,
                                            float f0, float f1, float f2, float f3) {
  const uint2 pk = make_uint2(cvt_bf16x2(f1, f0), cvt_bf16x2(f3, f2));
  for (int r = 0; r < pf.world; ++r)
    *reinterpret_cast<uint2*>(fused_recv(pf, r, parity, pf.rank) + elem) = pk;
}
// Tell every rank that `rows` more rows of `tile` from this rank are in place (one thread
// per destination rank; the caller has fenced and synchronised the storing threads).
__device__ __forceinline__ void fused_signal(const PeerFuse& pf, int tile, int dest, unsigned rows) {
  red_release_sys_add(fused_arrived(pf.region[dest], tile, pf.rank), rows);
}
// One thread per sender: bounded wait until that sender's rows of `tile` have all arrived.
__device__ __forceinline__ bool fused_wait(const PeerFuse& pf, int tile, int sender, unsigned rows,
                                           volatile int* abort_flag) {
  unsigned char* mine = pf.region[pf.rank];
  const unsigned base = __ldcg(fused_base(mine, tile, sender));
  const unsigned* arrived = fused_arrived(mine, tile, sender);
  for (unsigned tries = 0; tries < pf.wait_tries; ++tries) {
    if (static_cast<int>(ld_acquire_sys_u32(arrived) - base - rows) >= 0) return true;
    if (*abort_flag) return false;
    __nanosleep(tries < 64 ? 32 : 256);
  }
  *abort_flag = 1;
  return false;
}
// Sum of the world slots for four consecutive columns of one token row, in rank order.
__device__ __forceinline__ float4 fused_sum4(const PeerFuse& pf, unsigned parity, long long elem) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s = 0; s < pf.world; ++s) {
    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(fused_recv(pf, pf.rank, parity, s) + elem));
    acc.x += bf16lo_f32(v.x); acc.y += bf16hi_f32(v.x);
    acc.z += bf16lo_f32(v.y); acc.w += bf16hi_f32(v.y);
  }
  return acc;
}

struct WqParams {
  const __nv_bfloat16* scales;
  const __nv_bfloat16* zeros;
  const __nv_bfloat16* bias;
  __nv_bfloat16* out;
  long long ldo;
  float* partials;
  int* counters;
  int* status;
  int M, N, K, group;
  int NU;              // tokens padded to a multiple of 16: the UMMA N
  int units_per_tile;  // packed rows / 64
  int tiles;           // ceil(N / 128) x token blocks: tile t is token block t / tiles_n,
                       // weight columns 128 * (t % tiles_n)
  int tiles_n;         // ceil(N / 128); CTA pairs: ceil(N / 256)
  int block;           // tokens per token block: 128; CTA pairs: at most 256
  int total_units;
  int half_k;          // int4: K/2 (first activation column of the high-nibble plane)
  int stages;          // activation (X) ring depth
  int w_stages;        // packed-weight ring depth, a multiple of 4 so that every
                       // stage is only ever used by one dequant team, in order
  uint64_t w_policy;   // L2 eviction priority of the packed weights, see weight_policy
  int x_stage_bytes;   // planes * rows of activations held * 128
  int max_slots;       // partial slots reserved per tile
  int nacc;            // accumulator buffers in TMEM: 2; CTA pairs with more than 128 tokens per block: 1
  int group_shift;     // log2(group / 64) when that is a power of two, else -1
  int sz_step;         // scale rows a dequant team moves on per unit inside a tile, in 4 x bf16; -1: no
                       // constant (the group does not divide the teams' stride)
  int split;           // CTA pairs per tile, each with a slice of its K units (kModeSplit; else 1)
  int cluster;         // CTAs per tile (thread-block cluster along x); 1 = no cluster
  int recv_off;        // cluster mode: byte offset of the receive buffers in shared memory
  int recv_alias;      // cluster mode: the receive buffers lie over the (then idle) rings, so
                       // partial rows are only sent once every CTA of the cluster has finished
                       // its main loop
  int rows_per;        // cluster mode: token rows each CTA of the cluster reduces
  int rows_inv;        // ceil(65536 / rows_per): row / rows_per == (row * rows_inv) >> 16
  int epilogue;        // DXB_EPILOGUE_*: what is applied to the bf16 result before it is stored
  int tile_ranges;     // CTAs take whole tiles (ranges cut in tiles, not in units)
  int range_q, range_r;  // quotient and remainder of the cut: units of a tile by the cluster
                         // size, or tiles by the grid size (see the kernel's range arithmetic)
  PeerFuse peer;       // peer.world > 1: the sum over ranks is part of this launch (see below)
  long long* trace;    // only used when built with -DDXB_TRACE
};


// Four fp32 sums of one token row -> four bf16 outputs, in the reference's order of
// roundings: round the matmul to bf16, add the bias in bf16 arithmetic (second rounding),
// then the optional activation on that bf16 value (third rounding).
__device__ __forceinline__ uint2 finish_row4(float f0, float f1, float f2, float f3,
                                             const float (&bias4)[4], bool has_bias, int epilogue) {
  uint32_t r01 = cvt_bf16x2(f1, f0), r23 = cvt_bf16x2(f3, f2);
  if (has_bias) {
    const uint32_t b01 = cvt_bf16x2(bf16hi_f32(r01) + bias4[1], bf16lo_f32(r01) + bias4[0]);
    const uint32_t b23 = cvt_bf16x2(bf16hi_f32(r23) + bias4[3], bf16lo_f32(r23) + bias4[2]);
    r01 = b01; r23 = b23;
  }
  if (epilogue == DXB_EPILOGUE_GELU_TANH) {
    r01 = gelu_tanh2(r01);
    r23 = gelu_tanh2(r23);
  }
  return make_uint2(r01, r23);
}

// MULTI: more than one token block (M > 128); a tile is then a (token block, column tile)
// pair.  The single-block kernel carries none of that bookkeeping.
// RELAID (int4 only): the packed bytes were rewritten by wq_relayout_w4_kernel so that one
// 32-bit word holds the k-pairs the TMEM store wants (see there); saves the byte permutes.
// MODE: the same pipeline compiled six times.  All but the general instance carry only what their
// launches execute, which keeps their code a third of the general instance's: these
// launches last 8-15 us, and a kernel whose code is larger than the instruction cache pays for
// fetching it again in every launch (measured: 12.6 against 13.5 us on the headline shape).
//   kModeGeneral  the sum over ranks, tiles shared between CTAs through global partial sums, clusters
//   kModeWhole    whole tiles per CTA, no cluster
//   kModeCluster  one tile per cluster (K split, sum through distributed shared memory)
//   kModePair     whole tiles of 256 columns per CTA PAIR (cta_group::2): each CTA converts 128 columns and
//                 loads half the tokens, one MMA multiplies both, so a converted weight serves up to
//                 256 tokens and an activation is read once per 256 columns
//   kModeGroup    several problems with the same activations' shape in one launch, one tile per CTA (dxb_wq_gemm_group)
//   kModeSplit    CTA pairs, several per tile: each takes a slice of K, the last one adds the sums (an instance
//                 of its own: inside kModePair its code made those launches 2 % longer)
// Units of a tile times its tokens (a unit's products take four cycles a token) from which on the activation function
// of the tile before goes beside them.  Measured at 913 tokens and 13824 columns, us before the next tile / beside it
// (zeros as activations, so that the power limit stays away): int4 K of 1024 40.5 / 40.6, 1536 47.7 / 46.1, 2048 54.6 / 49.7,
// 5120 94.7 / 84.1; int8 with K of 1024 41.9 / 43.5.
constexpr int kActivateLater = 3072;
enum : int { kModeGeneral = 0, kModeWhole = 1, kModeCluster = 2, kModePair = 3, kModeSplit = 4, kModeGroup = 5 };

// One problem of a grouped launch, beside what all of them share (WqParams).
constexpr int kMaxGroup = 8;
struct GroupItem {
  const __nv_bfloat16* scales;
  const __nv_bfloat16* zeros;
  const __nv_bfloat16* bias;
  __nv_bfloat16* out;
  long long ldo;
  int N;
  int tile0;    // its first tile in the launch
  int sz_step;  // see WqParams
};
template <bool GROUP>
struct GroupArgs {};
template <>
struct GroupArgs<true> {
  CUtensorMap q[kMaxGroup], x[kMaxGroup];
  GroupItem item[kMaxGroup];
  int count;
};
// What a CTA works on: the launch's one problem, or the one of a group that its tile belongs to.  (Read where it is
// used, as kernel parameters are; gathered in one struct up front, other launches took 0.05 us longer.)
template <int MODE>
struct Problem {
  const CUtensorMap &tm_q, &tm_x;
  const WqParams& p;
  const GroupArgs<MODE == kModeGroup>& group;
  int i;  // kModeGroup: the item
  __device__ __forceinline__ Problem(const CUtensorMap& q, const CUtensorMap& x, const WqParams& params,
                                     const GroupArgs<MODE == kModeGroup>& g)
      : tm_q(q), tm_x(x), p(params), group(g), i(0) {
    if constexpr (MODE == kModeGroup)
      for (int j = 1; j < group.count; ++j) i += static_cast<int>(blockIdx.x) >= group.item[j].tile0;
  }
#define DX_OF(type, name, one, item_of)                      \
  __device__ __forceinline__ type name() const {             \
    if constexpr (MODE == kModeGroup) return group.item_of;  \
    else return one;                                         \
  }
  DX_OF(const CUtensorMap*, q, &tm_q, q + i)
  DX_OF(const CUtensorMap*, x, &tm_x, x + i)
  DX_OF(const __nv_bfloat16*, scales, p.scales, item[i].scales)
  DX_OF(const __nv_bfloat16*, zeros, p.zeros, item[i].zeros)
  DX_OF(const __nv_bfloat16*, bias, p.bias, item[i].bias)
  DX_OF(__nv_bfloat16*, out, p.out, item[i].out)
  DX_OF(long long, ldo, p.ldo, item[i].ldo)
  DX_OF(int, N, p.N, item[i].N)
  DX_OF(int, sz_step, p.sz_step, item[i].sz_step)
  DX_OF(int, tile0, 0, item[i].tile0)
#undef DX_OF
};

template <int BITS, bool HAS_ZERO, bool MULTI, bool RELAID, int MODE>
__global__ void __launch_bounds__(kThreads, 1)
wq_gemm_tc(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_x,
           const WqParams p, const __grid_constant__ GroupArgs<MODE == kModeGroup> group) {
  // A unit is 128 logical k of 128 weight columns in two planes of 64: for int4 the low and the
  // high nibbles of 64 packed rows (k and k + K/2), for int8 two consecutive blocks of 64 rows.
  constexpr int PLANES = 2;
  constexpr int A_STAGE_COLS = PLANES * 32;
  constexpr int UNIT_ROWS = BITS == 4 ? 64 : 128;   // packed rows per unit
  constexpr int W_STAGE = UNIT_ROWS * kTileN;       // bytes of one packed-weight stage

#ifdef DXB_TRACE
  const long long t_entry = clock64();
#endif
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[kNumBars];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  __shared__ int left_tiles;  // unit ranges: 1 = left the shared tile it began in, 2 = the one it ended in
#ifdef DXB_TRACE
  __shared__ long long t_start;
#endif

  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t w_ring = smem0;
  const uint32_t x_ring = smem0 + p.w_stages * W_STAGE;
  const uint32_t bar0 = smem_u32(bars);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int SW = p.w_stages;

  const Problem<MODE> pb(tm_q, tm_x, p, group);

  // This CTA's contiguous range of (tile, unit) work.
  // Cluster mode: the `cluster` CTAs of one cluster share one tile, each taking a
  // contiguous slice of its K units; they add their partial sums through distributed
  // shared memory at the end (no global scratch, no counters).
  const int TU = p.total_units;
  const int G = static_cast<int>(gridDim.x);
  const int U = p.units_per_tile;
  constexpr bool SYM4 = BITS == 4 && !HAS_ZERO;  // weights and sums are divided by kSymAcc, see sym4_low
  constexpr float ACC = SYM4 || BITS == 8 ? kSymAcc : 1.0f;  // (int8: see deq8_sym)
  constexpr bool kLean = MODE != kModeGeneral;
  constexpr bool ksplit = MODE == kModeSplit;
  constexpr bool PAIR = MODE == kModePair || ksplit;
  constexpr bool GROUP = MODE == kModeGroup;
  constexpr bool WHOLE = MODE == kModeWhole || PAIR || GROUP;
  const int NACC = PAIR ? p.nacc : 2;
  const int C = WHOLE ? 1 : p.cluster;  // kModeCluster is only launched with C > 1
  const bool clustered = MODE == kModeCluster || (MODE == kModeGeneral && C > 1);
  const bool tile_ranges = WHOLE || (MODE == kModeGeneral && p.tile_ranges);
  // Ranges without a division on the way to the first weight load (a 64-bit division is a few
  // hundred cycles at the head of every launch): `range_q`, `range_r` are quotient and remainder
  // of what is being cut (a cluster's units by its size, or the tiles by the grid), so part i
  // starts at i * q + min(i, r).  Only unit ranges that cut tiles still divide.
  const int crank = clustered || PAIR ? static_cast<int>(cluster_cta_rank()) : 0;
  // Split pairs: the last slice's pairs, which wait for the others, are the last in the grid.
  const int slice = ksplit ? static_cast<int>(cluster_id_x()) / p.tiles : 0;
  const int ctile = clustered ? static_cast<int>(cluster_id_x())
                    : ksplit ? static_cast<int>(cluster_id_x()) - slice * p.tiles : 0;
  const int part = clustered ? crank : ksplit ? slice : PAIR ? static_cast<int>(cluster_id_x()) : static_cast<int>(blockIdx.x);
  const int cut_begin = GROUP ? static_cast<int>(blockIdx.x) - pb.tile0() : part * p.range_q + (part < p.range_r ? part : p.range_r);
  const int cut_end = cut_begin + (GROUP ? 1 : p.range_q + (part < p.range_r ? 1 : 0));
  const bool unit_ranges = MODE == kModeGeneral && !clustered && !tile_ranges;
  const bool sliced = clustered || ksplit;  // a slice of one tile
  const int u_begin = sliced ? ctile * U + cut_begin
                      : !unit_ranges ? cut_begin * U : static_cast<int>(range_begin(blockIdx.x, TU, G));
  const int u_end = sliced ? ctile * U + cut_end
                    : !unit_ranges ? cut_end * U : static_cast<int>(range_begin(blockIdx.x + 1, TU, G));
  const int tile_begin = sliced ? ctile : !unit_ranges ? cut_begin : u_begin / U;
  const int ku_begin = sliced ? cut_begin : !unit_ranges ? 0 : u_begin - tile_begin * U;
  // This CTA's 128 columns of a tile.
  auto column_of = [&](int ntile) { return (PAIR ? 2 * ntile + crank : ntile) * kTileN; };

  // Packed-weight producers (warps 0 and 3, alternate units): cursor of the next unit to load.
  // (Issuing the first loads before the CTA-wide set-up barrier, with the producers only
  // arriving at it, triggering the dependent launch earlier, staggering the teams' first
  // conversions, and a first conversion pass that only walks the code to fill the
  // instruction cache were all measured: none made the launch faster, so the plain order stays.)
  const int wp = warp == 0 ? 0 : 1;
  int w_u = u_begin + wp, w_tile = tile_begin, w_ku = ku_begin + wp, w_s = wp, w_ntile = 0;
  uint32_t w_ph = 0;
  auto w_issue = [&]() {
    if (elect_one()) {
      const uint32_t fw = bar0 + 8 * (kBarFullW + w_s);
      mbar_expect_tx(fw, W_STAGE);
      tma_load_2d_policy(w_ring + w_s * W_STAGE, pb.q(), fw, column_of(MULTI ? w_ntile : w_tile), w_ku * UNIT_ROWS, p.w_policy);
    }
    __syncwarp();
    w_u += 2;
    w_s += 2;
    if (w_s >= SW) { w_s -= SW; w_ph ^= 1u; }
    w_ku += 2;
    while (w_ku >= U) { w_ku -= U; ++w_tile; if (MULTI && ++w_ntile == p.tiles_n) w_ntile = 0; }
  };
  if (warp == 0 || warp == 3) {
    if (lane == 0) tma_prefetch_desc(pb.q());
    // Each producer initialises the full and empty barriers of its own stages (even stages:
    // warp 0, odd: warp 3), the only ones it ever waits on, so it needs nobody else's set-up;
    // warp 3 also initialises the remaining barriers, which nobody touches before the set-up
    // barrier below.  Both clear the abort flag (same value) before anybody can wait.
    constexpr int kOwn = kMaxWStages / 2;  // stages of each producer
    static_assert(kMaxWStages % kAStages == 0 && kNumBars - kBarReady <= 32 - kOwn, "one lane per barrier below");
    if (lane < kOwn) {
      mbar_init(bar0 + 8 * (kBarFullW + wp + 2 * lane), bar_count(kBarFullW + wp + 2 * lane));
      mbar_init(bar0 + 8 * (kBarEmptyW + wp + 2 * lane), bar_count(kBarEmptyW + wp + 2 * lane));
    } else if (warp == 3 && kBarReady + lane - kOwn < kNumBars) {
      const int i = kBarReady + lane - kOwn;
      // The leader of a pair issues for both: its slots are ready with both CTAs' conversions, its accumulators
      // empty with both CTAs' epilogue warps.
      const uint32_t more = !PAIR ? 0u : i < kBarFree ? kTeamWarps : i >= kBarAccEmpty ? bar_count(i) : 0u;
      mbar_init(bar0 + 8 * i, bar_count(i) + more);
    }
    if (lane == 0) {
      abort_flag = 0;
      if (MODE == kModeGeneral) left_tiles = 0;
#ifdef DXB_TRACE
      if (warp == 3) {
        t_start = t_entry;  // trace builds: every stamp counts from the thread's first instruction
        DX_TRACE(5, 0);     // barriers initialised
      }
#endif
    }
    mbar_init_fence();
    __syncwarp();
    while (w_ku >= U) { w_ku -= U; ++w_tile; }
    w_ntile = MULTI ? w_tile % p.tiles_n : 0;
  } else if (warp == 2 && lane == 0) {
    tma_prefetch_desc(pb.x());
  } else if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(smem_u32(&tmem_base_s), 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(&tmem_base_s), 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // the other CTA's barriers exist, its TMEM is allocated
  tc_fence_after();
  const uint32_t tmem0 = tmem_base_s;
  if (threadIdx.x == 0) DX_TRACE(5, 1);  // set-up barrier passed
  // The next kernel of the stream may start now: its weight loads and conversion do not
  // depend on this kernel; it waits (pdl_wait) before it touches activations or outputs.
  pdl_launch_dependents();

  volatile int* abortp = &abort_flag;
  // One lane's wait for MMAs (slots that are free again, accumulators that are complete): a pair's come from
  // the leader.
  auto wait_mma = [abortp](uint32_t bar, uint32_t parity) {
    return PAIR ? mbar_wait_pair<false>(bar, parity, abortp) : mbar_wait(bar, parity, abortp);
  };

  // Cluster mode: send this CTA's fp32 partial rows from accumulator `d_tmem` (already
  // offset to the calling warp's lane quadrant) to their owners' receive buffers.
  auto cluster_send = [&](uint32_t d_tmem, int c, int n_local, int m_rows, int wk, int nwk) {
    const uint32_t recv0 = smem0 + static_cast<uint32_t>(p.recv_off);
    for (int c0 = 16 * wk; c0 < p.NU; c0 += 16 * nwk) {
      uint32_t ra[8], rb[8];
      tmem_ld_16x128b_x4(d_tmem + c0, ra);
      tmem_ld_16x128b_x4(d_tmem + (16u << 16) + c0, rb);
      tc_wait_ld();
      if (threadIdx.x == 0) DX_TRACE(7, 7);  // accumulator chunk in registers
#pragma unroll
      for (int rep = 0; rep < 4; ++rep) {
        const int m = c0 + 4 * rep + c;
        if (m < m_rows) {
          const int owner = (m * p.rows_inv) >> 16;
          const int row = crank * p.rows_per + (m - owner * p.rows_per);
          st_dsmem_b32x4(dsmem_addr(recv0 + static_cast<uint32_t>(row * kTileN + n_local) * 4u, owner),
                         ra[2 * rep], ra[2 * rep + 1], rb[2 * rep], rb[2 * rep + 1]);
        }
      }
    }
  };

  // ------------------------------------------------------------------ epilogue of one segment
  // A segment = this CTA's units of one tile, summed in accumulator `b`; run by the four
  // epilogue warps (one per TMEM lane quadrant).  Accumulator lane 32q + 8b + g holds weight
  // column 32q + 4g + b (see the dequant mapping), so the 16x128b load shape hands thread
  // (g, c) the four consecutive columns 4g..4g+3 of token 4*rep + c: one 8-byte store each.
  // Returns false when a bounded wait ran out.
  // Bias of this thread's four columns of a tile (fetched before waiting for the accumulator,
  // so that its latency is not added to the tail of the tile).
  auto load_bias4 = [&](int tile, float (&bias4)[4]) {
    const int ntile = MULTI ? tile % p.tiles_n : tile;
    const int n = column_of(ntile) + 32 * (warp & 3) + 4 * (lane >> 2);
    bias4[0] = bias4[1] = bias4[2] = bias4[3] = 0.f;
    if (pb.bias() != nullptr && n < pb.N()) {
      const uint2 bb = __ldg(reinterpret_cast<const uint2*>(pb.bias() + n));
      bias4[0] = bf16lo_f32(bb.x); bias4[1] = bf16hi_f32(bb.x);
      bias4[2] = bf16lo_f32(bb.y); bias4[3] = bf16hi_f32(bb.y);
    }
  };
  // `wk` of `nwk`: which 16-token chunks of the accumulator the calling warp takes.
  auto epilogue_segment = [&](int tile, int ku0, int nun, int b, const float (&bias4)[4], const int wk,
                              const int nwk) -> bool {
    constexpr int nthr = kEpilogueThreads;  // (the sum over ranks and shared tiles: the four epilogue warps)
    const int wtid = (warp - 4) * 32 + lane;
    const int q = warp & 3;
    const int c = lane & 3;
    const int g = lane >> 2;
    const int n_local = 32 * q + 4 * g;
    const bool has_bias = pb.bias() != nullptr;
    const bool whole = WHOLE || (MODE == kModeGeneral && nun == U);
    const int tblock = MULTI ? tile / p.tiles_n : 0;  // token block of this tile
    const int ntile = tile - tblock * p.tiles_n;      // its 128 weight columns
    const int row0 = tblock * p.block;
    const int m_rows = MULTI ? ((p.M - row0) < p.block ? (p.M - row0) : p.block) : p.M;  // token rows in this block
    const int n = column_of(ntile) + n_local;
    const bool n_ok = n < pb.N();
    // Sum over ranks fused into this launch (one token block only): finished rows go to
    // every rank's receive buffer instead of `out`; fused_finish then completes the tile.
    const bool fused = !kLean && p.peer.world > 1;
    // One accumulator: the next tile's products wait until it has been read, and the activation function would
    // keep them waiting as long again.  So the rows are stored without it first (rounded and with their
    // bias, as it wants them), the accumulator is given back, and then each thread takes its own values
    // up again.  Only where the next tile lasts long enough to cover that.  (The dequant warps reading along as well: 84.1
    // -> 83.9 us at 913 x 5120 x 13824, and their registers spilled: 200 x 8192 x 20096 72 -> 77.)
    const bool later = MODE == kModePair && nwk == 1 && NACC == 1 && p.epilogue != DXB_EPILOGUE_NONE &&
                       U * p.NU >= kActivateLater;
    const bool plain = !fused && (p.epilogue == DXB_EPILOGUE_NONE || later);
    const unsigned parity =
        fused ? (__ldcg(reinterpret_cast<const unsigned*>(p.peer.region[p.peer.rank])) & 1u) : 0u;
    auto fused_finish = [&]() -> bool {
      // The barrier orders every participant's peer stores before the signalling threads;
      // their release at system scope is cumulative, so it covers all of them (a system
      // fence costs about 1.7 us on this machine: one per rank to signal, not one per thread).
      named_bar_sync(1, nthr);
      if (wtid < p.peer.world) {
        fused_signal(p.peer, ntile, wtid, static_cast<unsigned>(m_rows));
        fused_wait(p.peer, ntile, wtid, static_cast<unsigned>(m_rows), abortp);
      }
      if (named_bar_any(1, nthr, *abortp)) return false;
      const int c4 = (wtid & 31) * 4;
      const int nn = ntile * kTileN + c4;
      if (nn < pb.N()) {
        float b4[4] = {0.f, 0.f, 0.f, 0.f};
        if (has_bias) {
          const uint2 bb = __ldg(reinterpret_cast<const uint2*>(pb.bias() + nn));
          b4[0] = bf16lo_f32(bb.x); b4[1] = bf16hi_f32(bb.x);
          b4[2] = bf16lo_f32(bb.y); b4[3] = bf16hi_f32(bb.y);
        }
        for (int m = wtid >> 5; m < m_rows; m += nthr >> 5) {
          const float4 a = fused_sum4(p.peer, parity, static_cast<long long>(m) * pb.N() + nn);
          *reinterpret_cast<uint2*>(pb.out() + static_cast<long long>(m) * pb.ldo() + nn) =
              finish_row4(a.x, a.y, a.z, a.w, b4, has_bias, p.epilogue);
        }
      }
      return true;
    };
    const uint32_t d_tmem = tmem_addr(tmem0 + b * p.NU, 32 * q, 0);
    if (whole) {
      for (int c0 = 16 * wk; c0 < p.NU; c0 += 16 * nwk) {
        uint32_t ra[8], rb[8];
        tmem_ld_16x128b_x4(d_tmem + c0, ra);
        tmem_ld_16x128b_x4(d_tmem + (16u << 16) + c0, rb);
        tc_wait_ld();
#pragma unroll
        for (int rep = 0; rep < 4; ++rep) {
          const int m = c0 + 4 * rep + c;
          if (n_ok && m < m_rows) {
            const float f0 = ACC * __uint_as_float(ra[2 * rep]), f1 = ACC * __uint_as_float(ra[2 * rep + 1]);
            const float f2 = ACC * __uint_as_float(rb[2 * rep]), f3 = ACC * __uint_as_float(rb[2 * rep + 1]);
            uint2* dst = reinterpret_cast<uint2*>(pb.out() + static_cast<long long>(row0 + m) * pb.ldo() + n);
            if (plain) {  // the common case, kept free of the optional epilogues' code
              uint2 pk;
              if (has_bias) {
                // Reference order: round the matmul to bf16, then add the bias in bf16.
                const uint32_t r01 = cvt_bf16x2(f1, f0), r23 = cvt_bf16x2(f3, f2);
                pk.x = cvt_bf16x2(bf16hi_f32(r01) + bias4[1], bf16lo_f32(r01) + bias4[0]);
                pk.y = cvt_bf16x2(bf16hi_f32(r23) + bias4[3], bf16lo_f32(r23) + bias4[2]);
              } else {
                pk.x = cvt_bf16x2(f1, f0);
                pk.y = cvt_bf16x2(f3, f2);
              }
              *dst = pk;
            } else if (fused) {
              fused_push4(p.peer, parity, static_cast<long long>(m) * pb.N() + n, f0, f1, f2, f3);
            } else {
              *dst = finish_row4(f0, f1, f2, f3, bias4, has_bias, p.epilogue);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0 && nwk == 1) {
        if (PAIR) mbar_arrive_pair(dsmem_addr(bar0 + 8 * (kBarAccEmpty + b), 0));  // the leader issues for both
        else mbar_arrive(bar0 + 8 * (kBarAccEmpty + b));
      }
      if (later) {
        for (int m0 = c; m0 < m_rows; m0 += 32) {
          uint2 v[8];
          uint2* row = reinterpret_cast<uint2*>(pb.out() + static_cast<long long>(row0 + m0) * pb.ldo() + n);
          const long long step = pb.ldo();  // four rows further, in uint2
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (n_ok && m0 + 4 * j < m_rows) v[j] = row[j * step];
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (n_ok && m0 + 4 * j < m_rows)
              row[j * step] = make_uint2(gelu_tanh2(v[j].x), gelu_tanh2(v[j].y));
        }
      }
      if (fused && !fused_finish()) return false;
    } else if (clustered) {
      // Cluster mode: CTA r of the cluster finishes token rows [r*rows_per, (r+1)*rows_per)
      // of the tile.  Every CTA sends each owner its fp32 partial rows straight from the
      // accumulator registers into the owner's receive buffer `crank` (distributed shared
      // memory stores); one cluster barrier later the owner only reads its own memory.
      // A cluster CTA has exactly this one segment, in accumulator 0, at the very end of its
      // work, when every other warp is idle: the accumulator stays where it is and ALL warps
      // send it after the CTA-wide barrier below (six warps per TMEM lane quadrant, 16
      // token columns each, instead of the four epilogue warps walking all of them).
    } else if (!kLean) {
      // A tile shared by several CTAs (equal unit ranges cut it): the CTA that holds the
      // tile's first units finishes it.  Ranges are contiguous and worked through in
      // order, so a CTA contributes to a tile it does not finish as its FIRST segment
      // and finishes a shared tile as its LAST one: by then the contributions have
      // normally been waiting in global scratch for a while, and the finisher only adds
      // them to its own accumulator (own sum first, then the slots in CTA order: the
      // result does not depend on timing).
      const int c_first = owner_of(static_cast<long long>(tile) * U, TU, G);
      const int c_last = owner_of(static_cast<long long>(tile) * U + U - 1, TU, G);
      const long long slot_elems = static_cast<long long>(p.NU) * kTileN;
      float* tile_ws = p.partials + static_cast<long long>(tile) * p.max_slots * slot_elems;
      if (ku0 > 0) {
        // contributor: park the fp32 sums, publish, carry on
        float* ws = tile_ws + (static_cast<int>(blockIdx.x) - c_first - 1) * slot_elems;
        for (int c0 = 16 * wk; c0 < p.NU; c0 += 16 * nwk) {
          uint32_t ra[8], rb[8];
          tmem_ld_16x128b_x4(d_tmem + c0, ra);
          tmem_ld_16x128b_x4(d_tmem + (16u << 16) + c0, rb);
          tc_wait_ld();
#pragma unroll
          for (int rep = 0; rep < 4; ++rep) {
            const int m = c0 + 4 * rep + c;
            if (m < m_rows)
              __stcg(reinterpret_cast<float4*>(ws + m * kTileN + n_local),
                     make_float4(__uint_as_float(ra[2 * rep]), __uint_as_float(ra[2 * rep + 1]),
                                 __uint_as_float(rb[2 * rep]), __uint_as_float(rb[2 * rep + 1])));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && wk == 0) mbar_arrive(bar0 + 8 * (kBarAccEmpty + b));
        __threadfence();
        named_bar_sync(1, nthr);
        if (wtid == 0) {
          tile_leave(&p.counters[tile], c_last - c_first + 1, true);
          left_tiles |= 1;
        }
      } else {
        // finisher: wait (bounded) until every contributor has published
        const int ncontrib = c_last - c_first;
        if (wtid == 0) {
          if (wait_tile_parked(&p.counters[tile], ncontrib + 1, abortp))
            p.counters[tile] = 0;  // ready for the next launch / graph replay
          else
            tile_leave(&p.counters[tile], ncontrib + 1, false);
          left_tiles |= 2;
        }
        if (named_bar_any(1, nthr, *abortp)) return false;
        for (int c0 = 16 * wk; c0 < p.NU; c0 += 16 * nwk) {
          float4 v[4];
#pragma unroll
          for (int rep = 0; rep < 4; ++rep) v[rep] = make_float4(0.f, 0.f, 0.f, 0.f);
          // contributions in CTA order; the loads of one slot are in flight together
          for (int sl = 0; sl < ncontrib; ++sl) {
            float4 t4[4];
#pragma unroll
            for (int rep = 0; rep < 4; ++rep) {
              const int m = c0 + 4 * rep + c;
              t4[rep] = m < m_rows ? __ldcg(reinterpret_cast<const float4*>(
                                         tile_ws + sl * slot_elems + m * kTileN + n_local))
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int rep = 0; rep < 4; ++rep) {
              if (sl == 0) {
                v[rep] = t4[rep];
              } else {
                v[rep].x += t4[rep].x; v[rep].y += t4[rep].y;
                v[rep].z += t4[rep].z; v[rep].w += t4[rep].w;
              }
            }
          }
          uint32_t ra[8], rb[8];
          tmem_ld_16x128b_x4(d_tmem + c0, ra);
          tmem_ld_16x128b_x4(d_tmem + (16u << 16) + c0, rb);
          tc_wait_ld();
#pragma unroll
          for (int rep = 0; rep < 4; ++rep) {
            const int m = c0 + 4 * rep + c;
            if (n_ok && m < m_rows) {
              const float f0 = ACC * (__uint_as_float(ra[2 * rep]) + v[rep].x);
              const float f1 = ACC * (__uint_as_float(ra[2 * rep + 1]) + v[rep].y);
              const float f2 = ACC * (__uint_as_float(rb[2 * rep]) + v[rep].z);
              const float f3 = ACC * (__uint_as_float(rb[2 * rep + 1]) + v[rep].w);
              if (fused)
                fused_push4(p.peer, parity, static_cast<long long>(m) * pb.N() + n, f0, f1, f2, f3);
              else
                *reinterpret_cast<uint2*>(pb.out() + static_cast<long long>(row0 + m) * pb.ldo() + n) =
                    finish_row4(f0, f1, f2, f3, bias4, has_bias, p.epilogue);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && wk == 0) mbar_arrive(bar0 + 8 * (kBarAccEmpty + b));
        if (fused && !fused_finish()) return false;
      }
    }
    return true;
  };

  if (warp == 0 || warp == 3) {
    // ============================================ TMA producer: packed weights
    // Two producer warps (0 and 3) take alternate units, which doubles the issue rate.
    // The whole warp runs the loop (so addresses and coordinates stay in uniform
    // registers, which the TMA instruction wants); one elected lane issues.
    {
      bool ok = true;
      // first pass over the ring: every stage is free
      for (int first = 0; first < (SW >> 1) && w_u < u_end; ++first) {
        w_issue();
        if (warp == 0 && lane == 0 && first == 0) DX_TRACE(5, 2);  // first weight load issued
      }
      while (w_u < u_end) {
        ok = mbar_wait_warp(bar0 + 8 * (kBarEmptyW + w_s), w_ph ^ 1u, abortp);
        if (!ok) break;
        w_issue();
      }
      if (!ok && lane == 0) {
        // Leaving early: let the copies already issued land before the CTA exits.
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ============================================== TMA producer: activations
    // Activations may be the output of the previous kernel in the stream.
    pdl_wait();
    if (lane == 0) DX_TRACE(5, 3);  // the previous kernel of the stream is complete
    // One elected thread runs the whole loop, unrolled over the ring's stages (see the MMA issuer).
    if (elect_one()) {
      int ku = ku_begin;
      int ntile = MULTI ? tile_begin % p.tiles_n : 0;
      // first token row of the token block (a pair's CTAs load half of it each)
      int row0 = MULTI ? (tile_begin / p.tiles_n) * p.block + (PAIR ? crank * (p.NU >> 1) : 0) : 0;
      uint32_t ph = 1;
      int u = u_begin;
      bool ok = true;
      const uint32_t x_bytes = p.x_stage_bytes;
      // Four stages go with the four slots; with three (int8) the unit three ago has to be done.
      constexpr bool kMayBeThree = BITS == 8 && !MULTI;
      const bool three = kMayBeThree && p.stages == 3;
      uint32_t dst = x_ring;
      while (u < u_end && ok) {
#pragma unroll
        for (int t = 0; t < kAStages; ++t) {
          if (u < u_end && ok) {
            ok = three ? wait_mma(bar0 + 8 * (kBarFree + (t + 1) % kAStages), t < 3 ? ph : ph ^ 1u)
                       : wait_mma(bar0 + 8 * (kBarFree + t), ph);
            if (ok) {
              const uint32_t rb = bar0 + 8 * (kBarReady + t);
              if (!kMayBeThree) dst = x_ring + t * p.x_stage_bytes;
              // A pair: both CTAs' halves complete on the leader's barrier (this slot's free barrier is
              // the commit of the MMAs before, so the leader's is in this unit's phase).
              if (!PAIR) mbar_expect_tx(rb, x_bytes);
              else if (crank == 0) mbar_expect_tx(rb, 2 * x_bytes);
              if (PAIR && BITS == 4) {
                tma_load_3d_pair(dst, pb.x(), dsmem_addr(rb, 0), ku * 64, row0, 0);
              } else if (PAIR) {
                tma_load_2d_pair(dst, pb.x(), dsmem_addr(rb, 0), ku * 128, row0);
                tma_load_2d_pair(dst + (x_bytes >> 1), pb.x(), dsmem_addr(rb, 0), ku * 128 + 64, row0);
              } else if (BITS == 4) {
                tma_load_3d(dst, pb.x(), rb, ku * 64, row0, 0);
              } else {  // two k-blocks of 64, one per plane
                tma_load_2d(dst, pb.x(), rb, ku * 128, row0);
                tma_load_2d(dst + (x_bytes >> 1), pb.x(), rb, ku * 128 + 64, row0);
                if (kMayBeThree) {
                  dst += x_bytes;
                  if (dst == x_ring + p.stages * x_bytes) dst = x_ring;
                }
              }
              ++u;
              if (++ku == U) {
                ku = 0;
                if (MULTI && ++ntile == p.tiles_n) { ntile = 0; row0 += p.block; }
              }
            }
          }
        }
        ph ^= 1u;
      }
      if (!ok) {
        // Leaving early: give copies already issued time to land before the CTA exits.
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ======================================================= MMA issuer ====
    // One elected thread runs the whole loop, unrolled over the four slots so that every operand of a
    // slot is a constant away from its base.  This warp shares its scheduler with four dequant
    // warps that keep it about 80 % busy, so each of its instructions waits for a turn: as a
    // warp-uniform loop with a slot counter a unit's 8 products and its wait took 840 cycles beside
    // them, twice what the tensor pipe needs for 96 tokens; in this form they take 460.
    if ((!PAIR || crank == 0) && elect_one()) {
      const uint32_t idesc = idesc_bf16_f32(PAIR ? 2 * kTileN : kTileN, p.NU);
      const uint64_t xdesc0 = smem_desc_kmajor_sw128(x_ring);
      const uint32_t x_stage16 = static_cast<uint32_t>(p.x_stage_bytes) >> 4;
      const uint32_t plane16 = static_cast<uint32_t>(p.x_stage_bytes >> 1) >> 4;
      const uint32_t a_tmem0 = tmem0 + kACol0;
      int b = 0;
      const uint32_t x_lo0 = static_cast<uint32_t>(xdesc0), x_hi = static_cast<uint32_t>(xdesc0 >> 32);
      uint32_t x_lo = x_lo0;  // the half that holds the address
      const uint32_t x_lo_end = x_lo + p.stages * x_stage16;
      uint32_t ph = 0, accph = 1, accumulate = 0;
      int left = u_end - u_begin;                           // units of this CTA that are in no segment yet
      int seg = left < U - ku_begin ? left : U - ku_begin;  // units still to do in the current tile
      left -= seg;
      uint32_t d_tmem = tmem0;
      auto mma = [x_hi](uint32_t d, uint32_t a, uint32_t b, uint32_t id, uint32_t acc) {
        if (PAIR) mma_ts_pair(d, a, b, x_hi, id, acc);
        else mma_ts(d, a, b, x_hi, id, acc);
      };
      auto commit = [](uint32_t bar) {
        if (PAIR) tc_commit_pair(bar);
        else tc_commit(bar);
      };
      auto wait = [abortp](uint32_t bar, uint32_t parity) {
        return PAIR ? mbar_wait_pair<true>(bar, parity, abortp) : mbar_wait(bar, parity, abortp);
      };
      bool ok = seg > 0 && wait(bar0 + 8 * kBarAccEmpty, accph);  // there is more to do
      while (ok) {
#pragma unroll
        for (int t = 0; t < kAStages; ++t) {
          if (ok) {
            ok = wait(bar0 + 8 * (kBarReady + t), ph);
            if (ok) {
              tc_fence_after();
              if (BITS == 4 || MULTI) x_lo = x_lo0 + t * x_stage16;
              const uint32_t a_tmem = a_tmem0 + t * A_STAGE_COLS;
              mma(d_tmem, a_tmem, x_lo, idesc, accumulate);
#pragma unroll
              for (int kk = 1; kk < 4; ++kk) mma(d_tmem, a_tmem + kk * 8, x_lo + kk * 2, idesc, 1u);
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                mma(d_tmem, a_tmem + 32 + kk * 8, x_lo + plane16 + kk * 2, idesc, 1u);
              commit(bar0 + 8 * (kBarFree + t));
              accumulate = 1;
              if (BITS == 8 && !MULTI) {
                x_lo += x_stage16;
                if (x_lo == x_lo_end) x_lo = x_lo0;
              }
              if (--seg == 0) {
                commit(bar0 + 8 * (kBarAccFull + b));
                if (++b == NACC) { b = 0; accph ^= 1u; }
                ok = left > 0;
                if (ok) {
                  seg = left < U ? left : U;
                  left -= seg;
                  accumulate = 0;
                  d_tmem = tmem0 + b * p.NU;
                  ok = wait(bar0 + 8 * (kBarAccEmpty + b), accph);
                }
              }
            }
          }
        }
        ph ^= 1u;
      }
    }
    __syncwarp();
  } else if (warp >= 4 && warp < 8) {
    // ========================================================= epilogue ====
    pdl_wait();  // outputs / scratch may still be in use by the previous kernel
    const int etid = (warp - 4) * 32 + lane;
    int b = 0;
    uint32_t accph = 0;
    int u = u_begin, ku0 = ku_begin, tile = tile_begin;
    while (u < u_end) {
      const int left = u_end - u;
      const int nun = left < (U - ku0) ? left : (U - ku0);
      float bias4[4];
      load_bias4(tile, bias4);
      bool ok = __all_sync(0xffffffffu, wait_mma(bar0 + 8 * (kBarAccFull + b), accph));  // see mbar_wait_warp
      // Sums over ranks and shared tiles synchronise the four epilogue warps: they go on together or not at all.
      if (MODE == kModeGeneral) ok = !named_bar_any(1, kEpilogueThreads, !ok);
      if (!ok) break;
      if (etid == 0) DX_TRACE(0, tile - tile_begin);
      tc_fence_after();
      if (WHOLE && u + nun == u_end) break;  // the last tile is everybody's, see below
      if (!epilogue_segment(tile, ku0, nun, b, bias4, 0, 1)) break;
      if (etid == 0) DX_TRACE(1, tile - tile_begin);
      u += nun;
      ku0 = 0;
      ++tile;
      if (++b == NACC) { b = 0; accph ^= 1u; }
    }
  } else if (warp >= 8) {
    // ========================================================== dequant ====
    // Four teams of four warps; team j converts units j, j+4, j+8, ... of this CTA
    // into TMEM ring stage j, so four units are in flight and the per-unit chain
    // (barrier wake-up, shared-memory loads, TMEM store drain) of one team is
    // hidden behind the other three.
    // Thread (c = lane % 4, g = lane / 4) of quadrant q reads, for each slab of 8
    // packed rows, the 32-bit words at rows 2c and 2c+1, byte columns
    // 32q + 4g .. +3.  Byte b of the word is weight column 32q + 4g + b and goes to
    // TMEM lane 32q + 8b + g; rows (2c, 2c+1) form one bf16 pair = TMEM column c of
    // that slab: exactly the register layout of tcgen05.st.16x128b.
    const int team = (warp - 8) >> 2;
    const int q = warp & 3;
    const int c = lane & 3;
    const int g = lane >> 2;
    const uint32_t chunk = 2 * q + (g >> 2);
    const uint32_t off0 = (2 * c) * 128 + ((chunk ^ (2 * c)) << 4) + 4 * (g & 3);
    const uint32_t off1 = (2 * c + 1) * 128 + ((chunk ^ (2 * c + 1)) << 4) + 4 * (g & 3);
    const uint32_t lane_base = 32 * q;
    const int n_local = 32 * q + 4 * g;
    const int group_units = p.group / 64;   // quantisation group in planes of 64 k
    const int half_units = p.half_k / 64;    // int4: planes between the low and the high nibbles
    const uint32_t a_tmem = tmem0 + kACol0 + team * A_STAGE_COLS;
    const uint32_t a_full_bar = PAIR ? dsmem_addr(bar0 + 8 * (kBarReady + team), 0) : bar0 + 8 * (kBarReady + team);
    const uint32_t a_empty_bar = bar0 + 8 * (kBarFree + team);

    // What a unit costs here beyond its conversion counts: the sixteen warps keep the schedulers
    // about 80 % busy, and ten instructions more per unit made a launch 9 % longer.
    int left = (u_end - u_begin - team + kAStages - 1) / kAStages;  // units of this team still to do
    int tile = tile_begin, ku = ku_begin + team;
    while (ku >= U) { ku -= U; ++tile; }
    int s = team;  // SW is a multiple of the team count: stages j, j+4, ... belong to team j
    uint32_t ph = 0;
    uint32_t aph = 0;
    bool ok = true;
    // Scales / zero points come straight from global memory (they are tiny and stay in
    // L2), fetched one team-unit ahead so the load latency is never waited for.  Inside a tile their
    // row moves on by the same amount from unit to unit (sz_step) unless the group is no
    // divisor of the teams' stride.
    uint2 sc[PLANES], zr[PLANES];
    int sz[PLANES];  // offset of the current rows, in 4 x bf16
    const int n4_stride = pb.N() >> 2;
    auto seek_sz = [&]() {  // rows of unit (tile, ku); columns beyond N (last tile) re-read the last ones
      int n4 = (column_of(MULTI ? tile % p.tiles_n : tile) + n_local) >> 2;
      n4 = n4 < n4_stride ? n4 : n4_stride - 1;
#pragma unroll
      for (int pl = 0; pl < PLANES; ++pl) {
        const int kunit = BITS == 4 ? ku + pl * half_units : 2 * ku + pl;  // plane of 64 k
        sz[pl] = (p.group_shift >= 0 ? (kunit >> p.group_shift) : (kunit / group_units)) * n4_stride + n4;
      }
    };
    auto load_sz = [&]() {
#pragma unroll
      for (int pl = 0; pl < PLANES; ++pl) {
        sc[pl] = __ldg(reinterpret_cast<const uint2*>(pb.scales()) + sz[pl]);
        if (HAS_ZERO) zr[pl] = __ldg(reinterpret_cast<const uint2*>(pb.zeros()) + sz[pl]);
      }
    };
    if (left > 0) { seek_sz(); load_sz(); }
    while (left > 0) {
      // (Lanes that gave up carry on to the end of the unit, where the warp decides, see mbar_wait_warp: once per unit
      // and off its critical path.  A decision after each wait: FFN of 913 tokens 5120 x 13824 246.9 us, 236.4 so;
      // one after the second wait: int8 with zero points 160 tokens 14336 x 3072 31.4 against 30.2.)
      ok = mbar_wait(bar0 + 8 * (kBarFullW + s), ph, abortp);
      const uint32_t wsrc = w_ring + s * W_STAGE;
      uint32_t w0[8], w1[8];
#pragma unroll
      for (int sl = 0; sl < 8; ++sl) {
        w0[sl] = lds32(wsrc + off0 + sl * 1024);
        w1[sl] = lds32(wsrc + off1 + sl * 1024);
      }
      if (BITS == 4) {  // (int8 reads the second half of its stage further down)
        __syncwarp();  // every lane has its words in registers
        if (lane == 0) mbar_arrive(bar0 + 8 * (kBarEmptyW + s));
      }
      // This unit's scales and zero points as the conversion wants them (in both halves of a word; in
      // fp32 for deq8_any); then the next unit's rows.
      uint32_t s2[PLANES][4], z2[PLANES][4];
      // Constants outside the short conversions' range (never a model's): bodies of their own, so that the usual one is
      // scheduled as if they did not exist (a branch in front of each store made launches 6 % longer).
      bool large = false;
      uint32_t odd = 0;
      if (BITS == 8 && HAS_ZERO) {
#pragma unroll
        for (int pl = 0; pl < PLANES; ++pl) {
          z2[pl][0] = deq8_zeros(zr[pl].x, odd);
          z2[pl][2] = deq8_zeros(zr[pl].y, odd);
        }
      }
      if (SYM4 || BITS == 8)
        large = __any_sync(0xffffffffu, sym4_large(sc[0].x | sc[0].y | sc[1].x | sc[1].y) || odd != 0);
#pragma unroll
      for (int pl = 0; pl < PLANES; ++pl) {
        if (BITS == 4) {
          s2[pl][0] = dup_lo(sc[pl].x); s2[pl][1] = dup_hi(sc[pl].x);
          s2[pl][2] = dup_lo(sc[pl].y); s2[pl][3] = dup_hi(sc[pl].y);
          if (HAS_ZERO) {
            z2[pl][0] = dup_lo(zr[pl].x); z2[pl][1] = dup_hi(zr[pl].x);
            z2[pl][2] = dup_lo(zr[pl].y); z2[pl][3] = dup_hi(zr[pl].y);
          } else {
            // Repacked: columns 1 and 3 stand at bits 4..7; otherwise those of the high-nibble plane do.
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              z2[pl][i] = sym4_offset(s2[pl][i]);
              s2[pl][i] = (RELAID ? (i & 1) : pl) ? sym4_scale_mid(s2[pl][i]) : sym4_scale_low(s2[pl][i]);
            }
          }
          if (RELAID && HAS_ZERO) {  // columns 1 and 3 of a word are converted where they stand, see deq4_mid
#pragma unroll
            for (int i = 1; i < 4; i += 2) {
              s2[pl][i] = mid_scale(s2[pl][i]);
              z2[pl][i] = mid_zero(z2[pl][i]);
            }
          }
        } else {
          const uint32_t sx[2] = {sc[pl].x, sc[pl].y};
          if (large && HAS_ZERO) {
            const uint32_t zx[2] = {zr[pl].x, zr[pl].y};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              s2[pl][2 * i] = __float_as_uint(bf16lo_f32(sx[i]) / kSymAcc);
              s2[pl][2 * i + 1] = __float_as_uint(bf16hi_f32(sx[i]) / kSymAcc);
              z2[pl][2 * i] = zx[i] << 16;
              z2[pl][2 * i + 1] = zx[i] & 0xFFFF0000u;
            }
          } else if (large) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              s2[pl][2 * i] = dup_lo(sx[i]); s2[pl][2 * i + 1] = dup_hi(sx[i]);
              z2[pl][2 * i] = z2[pl][2 * i + 1] = 0u;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint32_t sv = deq8_scale(sx[i]), zv = HAS_ZERO ? z2[pl][2 * i] : deq8_offset(sx[i]);
              s2[pl][2 * i] = dup_lo(sv); s2[pl][2 * i + 1] = dup_hi(sv);
              z2[pl][2 * i] = dup_lo(zv); z2[pl][2 * i + 1] = dup_hi(zv);
            }
          }
        }
      }
      if (--left > 0) {
        ku += kAStages;
        if (ku >= U || pb.sz_step() < 0) {
          while (ku >= U) { ku -= U; ++tile; }
          seek_sz();
        } else {
#pragma unroll
          for (int pl = 0; pl < PLANES; ++pl) sz[pl] += pb.sz_step();
        }
        load_sz();
      }
      ok = wait_mma(a_empty_bar, aph ^ 1u) && ok;
      tc_fence_after();
      if (BITS == 4 && large) {
        // The same with scales of 2 and more, see sym4_any.
#pragma unroll
        for (int pl = 0; pl < 2; ++pl) {
#pragma unroll
          for (int rh = 0; rh < 2; ++rh) {
            uint32_t ra[8], rb[8];
#pragma unroll
            for (int sl = 0; sl < 4; ++sl) {
              uint32_t v[4];  // the four columns' pairs at bits 0..3 and 16..19
              if (RELAID) {
                const uint32_t W = pl == 0 ? w0[4 * rh + sl] : w1[4 * rh + sl];
                v[0] = W; v[1] = W >> 4; v[2] = W >> 8; v[3] = W >> 12;
              } else {
                v[0] = prmt(w0[4 * rh + sl], w1[4 * rh + sl], 0x5410u) >> (4 * pl);
                v[2] = prmt(w0[4 * rh + sl], w1[4 * rh + sl], 0x7632u) >> (4 * pl);
                v[1] = v[0] >> 8; v[3] = v[2] >> 8;
              }
              ra[2 * sl + 0] = sym4_any(v[0], z2[pl][0]);
              ra[2 * sl + 1] = sym4_any(v[1], z2[pl][1]);
              rb[2 * sl + 0] = sym4_any(v[2], z2[pl][2]);
              rb[2 * sl + 1] = sym4_any(v[3], z2[pl][3]);
            }
            tmem_st_16x128b_x4(tmem_addr(a_tmem + pl * 32 + 16 * rh, lane_base, 0), ra);
            tmem_st_16x128b_x4(tmem_addr(a_tmem + pl * 32 + 16 * rh, lane_base + 16, 0), rb);
          }
        }
      } else if (BITS == 4) {
#pragma unroll
        for (int pl = 0; pl < 2; ++pl) {
#pragma unroll
          for (int rh = 0; rh < 2; ++rh) {
            uint32_t ra[8], rb[8];
#pragma unroll
            for (int sl = 0; sl < 4; ++sl) {
              if (RELAID) {
                // The word of the even row holds the low-nibble plane, the word of the odd
                // row the high-nibble plane: nibble b is byte column b of the even row,
                // nibble 4 + b the same column of the odd row, so masking with 0x000F000F
                // after a shift by 4b (0x00F000F0 after 4b - 4) yields the k-pair of column b.
                const uint32_t W = pl == 0 ? w0[4 * rh + sl] : w1[4 * rh + sl];
                if (SYM4) {
                  ra[2 * sl + 0] = sym4_low(W, s2[pl][0], z2[pl][0]);
                  ra[2 * sl + 1] = sym4_mid(W, s2[pl][1], z2[pl][1]);
                  rb[2 * sl + 0] = sym4_low(W >> 8, s2[pl][2], z2[pl][2]);
                  rb[2 * sl + 1] = sym4_mid(W >> 8, s2[pl][3], z2[pl][3]);
                } else {
                  ra[2 * sl + 0] = deq4(W, z2[pl][0], s2[pl][0]);
                  ra[2 * sl + 1] = deq4_mid(W, z2[pl][1], s2[pl][1]);
                  rb[2 * sl + 0] = deq4(W >> 8, z2[pl][2], s2[pl][2]);
                  rb[2 * sl + 1] = deq4_mid(W >> 8, z2[pl][3], s2[pl][3]);
                }
              } else {
                const uint32_t P = prmt(w0[4 * rh + sl], w1[4 * rh + sl], 0x5410u);
                const uint32_t Q = prmt(w0[4 * rh + sl], w1[4 * rh + sl], 0x7632u);
                if (SYM4) {
                  auto sym4 = [&](uint32_t w, int i) {
                    return pl ? sym4_mid(w, s2[pl][i], z2[pl][i]) : sym4_low(w, s2[pl][i], z2[pl][i]);
                  };
                  ra[2 * sl + 0] = sym4(P, 0);
                  ra[2 * sl + 1] = sym4(P >> 8, 1);
                  rb[2 * sl + 0] = sym4(Q, 2);
                  rb[2 * sl + 1] = sym4(Q >> 8, 3);
                } else {
                  ra[2 * sl + 0] = deq4(P >> (4 * pl), z2[pl][0], s2[pl][0]);
                  ra[2 * sl + 1] = deq4(P >> (4 * pl + 8), z2[pl][1], s2[pl][1]);
                  rb[2 * sl + 0] = deq4(Q >> (4 * pl), z2[pl][2], s2[pl][2]);
                  rb[2 * sl + 1] = deq4(Q >> (4 * pl + 8), z2[pl][3], s2[pl][3]);
                }
              }
            }
            tmem_st_16x128b_x4(tmem_addr(a_tmem + pl * 32 + 16 * rh, lane_base, 0), ra);
            tmem_st_16x128b_x4(tmem_addr(a_tmem + pl * 32 + 16 * rh, lane_base + 16, 0), rb);
          }
        }
      } else {
        auto convert = [&](auto way) {
          constexpr bool ANY = decltype(way)::value;
#pragma unroll
          for (int pl = 0; pl < 2; ++pl) {
            if (pl == 1) {
              // rows 64..127 of the unit; after these loads the stage can be refilled
#pragma unroll
              for (int sl = 0; sl < 8; ++sl) {
                w0[sl] = lds32(wsrc + 8192 + off0 + sl * 1024);
                w1[sl] = lds32(wsrc + 8192 + off1 + sl * 1024);
              }
              __syncwarp();
              if (lane == 0) mbar_arrive(bar0 + 8 * (kBarEmptyW + s));
            }
#pragma unroll
            for (int rh = 0; rh < 2; ++rh) {
              uint32_t r[2][8];  // columns 0, 1 and 2, 3
#pragma unroll
              for (int sl = 0; sl < 4; ++sl) {
                const uint32_t x0 = w0[4 * rh + sl], x1 = w1[4 * rh + sl];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const uint32_t pairs = byte_pairs(x0, x1, h);
#pragma unroll
                  for (int o = 0; o < 2; ++o) {
                    const int i = 2 * h + o;
                    r[h][2 * sl + o] = ANY && HAS_ZERO ? deq8_any(x0, x1, i, __uint_as_float(z2[pl][i]), __uint_as_float(s2[pl][i]))
                                       : ANY ? deq8_sym_any(byte_pair(pairs, o), s2[pl][i])
                                       : HAS_ZERO ? deq8_zero(byte_pair(pairs, o), s2[pl][i], z2[pl][i])
                                                  : deq8_sym(byte_pair(pairs, o), s2[pl][i], z2[pl][i]);
                  }
                }
              }
              tmem_st_16x128b_x4(tmem_addr(a_tmem + pl * 32 + 16 * rh, lane_base, 0), r[0]);
              tmem_st_16x128b_x4(tmem_addr(a_tmem + pl * 32 + 16 * rh, lane_base + 16, 0), r[1]);
            }
          }
        };
        if (large) convert(std::true_type{});
        else convert(std::false_type{});
      }
      tc_wait_st();
      tc_fence_before();
      ok = __all_sync(0xffffffffu, ok);
      __syncwarp();
      if (!ok) break;
      if (lane == 0) {
        if (PAIR) mbar_arrive_pair(a_full_bar);
        else mbar_arrive(a_full_bar);
      }
      aph ^= 1u;
      s += kAStages;
      if (s >= SW) { s -= SW; ph ^= 1u; }
    }
  }

  tc_fence_before();
  const bool aborted = __syncthreads_or(abort_flag) != 0;  // one answer for all threads
  if (threadIdx.x == 0) DX_TRACE(7, 1);  // every role is through its loop
  if (ksplit && aborted) {
    if (threadIdx.x == 0) {
      pdl_wait();
      tile_leave(p.counters + 2 * ctile + crank, p.split, false);
    }
  } else if (ksplit) {
    // K split over pairs: all but the last slice park their fp32 sums in global scratch (each CTA its own
    // 128 columns) and leave; the last slice's CTAs add them to their own in slice order.
    const int slots = p.split - 1;
    const int q = warp & 3, c = lane & 3, n_local = 32 * q + 4 * (lane >> 2);
    const int tblock = ctile / p.tiles_n, ntile = ctile - tblock * p.tiles_n;
    const int row0 = tblock * p.block;
    const int m_rows = (p.M - row0) < p.block ? (p.M - row0) : p.block;
    const int n = column_of(ntile) + n_local;
    const long long slot_elems = static_cast<long long>(p.NU) * kTileN;
    float* slot0 = p.partials + static_cast<long long>(2 * ctile + crank) * slots * slot_elems;
    int* counter = p.counters + 2 * ctile + crank;
    float bias4[4];
    load_bias4(ctile, bias4);
    pdl_wait();
    tc_fence_after();
    const bool last = slice == slots;
    if (last) {
      if (threadIdx.x == 0) {
        if (wait_tile_parked(counter, p.split, abortp)) *counter = 0;  // ready for the next launch
        else tile_leave(counter, p.split, false);
      }
      __syncthreads();
    }
    const uint32_t d_tmem = tmem_addr(tmem0, 32 * q, 0);
    for (int c0 = 16 * (warp >> 2); c0 < p.NU && !abort_flag; c0 += 16 * (kThreads / 128)) {
      float4 v[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int sl = 0; last && sl < slots; ++sl) {
        float4 t4[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int m = c0 + 4 * r + c;
          t4[r] = m < m_rows ? __ldcg(reinterpret_cast<const float4*>(slot0 + sl * slot_elems + m * kTileN + n_local))
                             : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) { v[r].x += t4[r].x; v[r].y += t4[r].y; v[r].z += t4[r].z; v[r].w += t4[r].w; }
      }
      uint32_t ra[8], rb[8];
      tmem_ld_16x128b_x4(d_tmem + c0, ra);
      tmem_ld_16x128b_x4(d_tmem + (16u << 16) + c0, rb);
      tc_wait_ld();
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int m = c0 + 4 * r + c;
        if (m >= m_rows) continue;
        const float f0 = __uint_as_float(ra[2 * r]) + v[r].x, f1 = __uint_as_float(ra[2 * r + 1]) + v[r].y;
        const float f2 = __uint_as_float(rb[2 * r]) + v[r].z, f3 = __uint_as_float(rb[2 * r + 1]) + v[r].w;
        if (!last)
          __stcg(reinterpret_cast<float4*>(slot0 + slice * slot_elems + m * kTileN + n_local), make_float4(f0, f1, f2, f3));
        else if (n < pb.N())
          *reinterpret_cast<uint2*>(pb.out() + static_cast<long long>(row0 + m) * pb.ldo() + n) =
              finish_row4(ACC * f0, ACC * f1, ACC * f2, ACC * f3, bias4, pb.bias() != nullptr, p.epilogue);
      }
    }
    tc_fence_before();
    if (!last) __threadfence();
    __syncthreads();  // every store of this CTA is out; before the accumulator's TMEM is given back
    if (!last && threadIdx.x == 0) tile_leave(counter, p.split, true);
  } else if (WHOLE && !aborted) {
    // The CTA's last tile: its accumulator is complete (the epilogue warps have waited for it) and
    // every other warp is idle, so all 24 finish it, six per TMEM lane quadrant with a 16-token chunk
    // each, instead of four walking six chunks.
    const int tiles = cut_end - cut_begin;
    const int tile = cut_end - 1;
    float bias4[4];
    load_bias4(tile, bias4);
    pdl_wait();
    tc_fence_after();
    epilogue_segment(tile, 0, U, NACC == 2 ? (tiles - 1) & 1 : 0, bias4, warp >> 2, kThreads / 128);
    tc_fence_before();
    __syncthreads();  // before the accumulator's TMEM is given back
  }
  if (clustered) {
    // The cluster's tile: token block and column tile.
    const int tblock = MULTI ? ctile / p.tiles_n : 0;
    const int ntile = ctile - tblock * p.tiles_n;
    const int row0 = tblock * p.block;
    const int m_rows = MULTI ? ((p.M - row0) < p.block ? (p.M - row0) : p.block) : p.M;
    const int m_lo = crank * p.rows_per;
    const int m_hi = (m_lo + p.rows_per) < m_rows ? (m_lo + p.rows_per) : m_rows;
    const uint32_t recv0 = smem0 + static_cast<uint32_t>(p.recv_off);
    const uint32_t src_stride = static_cast<uint32_t>(p.rows_per * kTileN) * 4u;
    const bool has_bias = pb.bias() != nullptr;
    // Every item of one thread has the same four columns (kThreads is a multiple of 32):
    // their bias is fetched before the barrier, off the critical path.
    const int c4 = (threadIdx.x & 31) * 4;
    const int n = ntile * kTileN + c4;
    float bias4[4] = {0.f, 0.f, 0.f, 0.f};
    if (has_bias && n < pb.N()) {
      const uint2 bb = __ldg(reinterpret_cast<const uint2*>(pb.bias() + n));
      bias4[0] = bf16lo_f32(bb.x); bias4[1] = bf16hi_f32(bb.x);
      bias4[2] = bf16lo_f32(bb.y); bias4[3] = bf16hi_f32(bb.y);
    }
    if (p.recv_alias) {
      // The receive buffers lie over the rings, which the peers may still be using.  Every
      // CTA of the cluster is past its main loop after this barrier: nothing reads or writes
      // the rings any more, so the buffers may be filled.
      cluster_sync_all();
    }
    // The epilogue warps have seen the accumulator complete before the CTA-wide barrier above.
    tc_fence_after();
    if (threadIdx.x == 0) DX_TRACE(7, 6);  // about to send
    cluster_send(tmem_addr(tmem0, 32 * (warp & 3), 0), lane & 3, 32 * (warp & 3) + 4 * (lane >> 2), m_rows,
                 warp >> 2, kThreads / 128);
    tc_fence_before();
    if (threadIdx.x == 0) DX_TRACE(7, 2);  // partial sums sent
    // After this barrier every partial row of this CTA's share has arrived in its receive
    // buffers: sum them in rank order (deterministic), add the bias, write bf16.  Nothing
    // remote is touched any more, so CTAs leave independently.
    cluster_sync_all();
    if (threadIdx.x == 0) DX_TRACE(7, 3);  // cluster barrier passed
    pdl_wait();
    if (threadIdx.x == 0) DX_TRACE(7, 4);  // previous kernel complete
    const bool fused = !kLean && p.peer.world > 1;
    const int epi = p.epilogue;
    const unsigned parity =
        fused ? (__ldcg(reinterpret_cast<const unsigned*>(p.peer.region[p.peer.rank])) & 1u) : 0u;
    if (n < pb.N()) {
      for (int i = threadIdx.x; i < (m_hi - m_lo) * 32; i += kThreads) {
        const int j = i >> 5;
        const uint32_t a0 = recv0 + static_cast<uint32_t>(j * kTileN + c4) * 4u;
        float4 v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r)
          v[r] = r < C ? ld_smem_f4(a0 + r * src_stride) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < 8; ++r) {  // rank order: the sum does not depend on timing
          acc.x += v[r].x; acc.y += v[r].y; acc.z += v[r].z; acc.w += v[r].w;
        }
        acc.x *= ACC; acc.y *= ACC; acc.z *= ACC; acc.w *= ACC;
        if (fused)
          fused_push4(p.peer, parity, static_cast<long long>(m_lo + j) * pb.N() + n, acc.x, acc.y, acc.z, acc.w);
        else
          *reinterpret_cast<uint2*>(pb.out() + static_cast<long long>(row0 + m_lo + j) * pb.ldo() + n) =
              finish_row4(acc.x, acc.y, acc.z, acc.w, bias4, has_bias, epi);
      }
    }
    if (threadIdx.x == 0) DX_TRACE(7, 5);  // rows summed and stored
    if (fused) {
      // This CTA's rows of the tile are on their way to every rank: publish them (the
      // barrier orders all stores before the signalling threads' cumulative release), wait
      // for the whole tile from every rank, then finish this CTA's rows from the local slots.
      __syncthreads();
      if (threadIdx.x < p.peer.world && m_hi > m_lo) {  // a CTA without rows has nothing to do
        fused_signal(p.peer, ntile, threadIdx.x, static_cast<unsigned>(m_hi - m_lo));
        fused_wait(p.peer, ntile, threadIdx.x, static_cast<unsigned>(m_rows), abortp);
      }
      __syncthreads();
      if (!abort_flag && n < pb.N()) {
        for (int i = threadIdx.x; i < (m_hi - m_lo) * 32; i += kThreads) {
          const int m = m_lo + (i >> 5);
          const float4 a = fused_sum4(p.peer, parity, static_cast<long long>(m) * pb.N() + n);
          *reinterpret_cast<uint2*>(pb.out() + static_cast<long long>(m) * pb.ldo() + n) =
              finish_row4(a.x, a.y, a.z, a.w, bias4, has_bias, epi);
        }
      }
    }
  }
  if (!kLean && p.peer.world > 1) {
    // The last CTA to leave moves the per-tile row baselines and the epoch on for the next
    // call (every other CTA has finished reading them by then).
    __shared__ int is_last;
    __syncthreads();
    unsigned char* mine = p.peer.region[p.peer.rank];
    unsigned* control = reinterpret_cast<unsigned*>(mine);
    if (threadIdx.x == 0) {
      __threadfence();
      is_last = atomicAdd(control + 1, 1u) == gridDim.x - 1 ? 1 : 0;
    }
    __syncthreads();
    if (is_last) {
      __threadfence();
      for (int i = threadIdx.x; i < p.tiles_n * p.peer.world; i += kThreads) {
        unsigned* bp = fused_base(mine, i / p.peer.world, i % p.peer.world);
        *bp = __ldcg(bp) + static_cast<unsigned>(p.M);
      }
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) {
        control[1] = 0;
        control[0] = __ldcg(control) + 1;
      }
    }
  }
  if (threadIdx.x == 0) DX_TRACE(7, 0);
  // Neither CTA of a pair may leave while the other can still signal it or use its memory.
  if (PAIR) cluster_sync_all();
  if (warp == 1) {
    if (PAIR) tmem_dealloc_pair(tmem0, 512);
    else tmem_dealloc(tmem0, 512);
  }
  if (threadIdx.x == 0 && abort_flag) {
    pdl_wait();
    if (unit_ranges && u_begin < u_end) {
      // Shared tiles that this CTA has not got to: leave them, so that their counters end at zero.
      const int t1 = (u_end - 1) / U;
      auto leave = [&](int tile) {
        const int sharers = owner_of(static_cast<long long>(tile) * U + U - 1, TU, G) -
                            owner_of(static_cast<long long>(tile) * U, TU, G) + 1;
        tile_leave(&p.counters[tile], sharers, false);
      };
      if (ku_begin > 0 && !(left_tiles & 1)) leave(tile_begin);
      if (t1 * U >= u_begin && u_end < (t1 + 1) * U && !(left_tiles & 2)) leave(t1);
    }
    atomicExch(p.status, DXB_ERR_KERNEL_TIMEOUT);
    int* also = *reinterpret_cast<int**>(p.status + kStatusAlso);  // see dxb_workspace_init
    if (also != nullptr) atomicExch(also, DXB_ERR_KERNEL_TIMEOUT);
  }
}

// A workspace ready for its first call (see dxb_workspace_init).
__global__ void wq_workspace_init_kernel(uint4* ws, int vecs, int* also) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= vecs) return;
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (i == 0) {  // status word, its padding, the other status word's address
    const unsigned long long a = reinterpret_cast<unsigned long long>(also);
    v.z = static_cast<uint32_t>(a);
    v.w = static_cast<uint32_t>(a >> 32);
  }
  ws[i] = v;
}

// ------------------------------------------------ load-time weight re-layout
// int4 only.  The reference packs byte [i, n] = row i (low nibble) | row i + K/2 (high
// nibble) (python/dexter/quant.py:62-72).  For every aligned block of 2 packed rows x 4
// byte columns (the two 32-bit words one dequant thread reads per slab of 8 rows) the 16
// nibbles are regrouped: the word at the even row keeps the low-nibble plane, the word at
// the odd row the high-nibble plane; inside a word, nibble b (bits 4b..4b+3) is byte column b
// of the even row and nibble 4 + b the same column of the odd row.  `(word >> 4b) &
// 0x000F000F` is then the bf16x2 mantissa pair (k, k+1) of column b: no byte permute.
// Same shape, same strides, same tiles; the transform is its own inverse pair (forward /
// inverse below) and is applied once per weight, never per call.
__device__ __forceinline__ uint32_t squeeze_nibbles(uint32_t v) {  // nibbles at bits 0,8,16,24 -> 0,4,8,12
  return (v & 0xFu) | ((v >> 4) & 0xF0u) | ((v >> 8) & 0xF00u) | ((v >> 12) & 0xF000u);
}
__device__ __forceinline__ uint32_t spread_nibbles(uint32_t h) {   // nibbles at bits 0,4,8,12 -> 0,8,16,24
  return (h & 0xFu) | ((h & 0xF0u) << 4) | ((h & 0xF00u) << 8) | ((h & 0xF000u) << 12);
}
__global__ void wq_relayout_w4_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                      long long row_pairs, int n4, int inverse) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= row_pairs * n4) return;
  const long long rp = idx / n4;
  const int j = static_cast<int>(idx - rp * n4);
  const long long i0 = (2 * rp) * n4 + j, i1 = (2 * rp + 1) * n4 + j;
  const uint32_t w0 = in[i0], w1 = in[i1];
  if (!inverse) {
    out[i0] = squeeze_nibbles(w0 & 0x0F0F0F0Fu) | (squeeze_nibbles(w1 & 0x0F0F0F0Fu) << 16);
    out[i1] = squeeze_nibbles((w0 >> 4) & 0x0F0F0F0Fu) | (squeeze_nibbles((w1 >> 4) & 0x0F0F0F0Fu) << 16);
  } else {
    out[i0] = spread_nibbles(w0 & 0xFFFFu) | (spread_nibbles(w1 & 0xFFFFu) << 4);
    out[i1] = spread_nibbles(w0 >> 16) | (spread_nibbles(w1 >> 16) << 4);
  }
}

// ------------------------------------------------------ any-shape CUDA path
// Plain CUDA-core kernel for what neither wq_gemm_tc nor wq_gemm_small takes: groups or packed rows that are
// no multiple of 32, weights and activations off the alignment of their loads.  One thread per output
// column, 8 tokens per block row; slow but exact in the same sense (bit-identical W, fp32 accumulation).
template <int BITS>
__global__ void wq_gemm_simt(const __nv_bfloat16* __restrict__ x, long long ldx, const uint8_t* __restrict__ qw,
                             const __nv_bfloat16* __restrict__ scales, const __nv_bfloat16* __restrict__ zeros,
                             const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ out, long long ldo,
                             int M, int N, int K, int group, int relaid, int epilogue) {
  constexpr int MT = 8;
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int m0 = blockIdx.y * MT;
  if (n >= N) return;
  float acc[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i) acc[i] = 0.0f;
  const int half = K / 2;
  for (int k = 0; k < K; ++k) {
    const int gi = k / group;
    const uint32_t sbits = __bfloat16_as_ushort(scales[static_cast<long long>(gi) * N + n]);
    float w;
    if (BITS == 4) {
      const uint32_t byte = fetch_q4(qw, N, half, k, n, relaid);
      const uint32_t z = zeros ? __bfloat16_as_ushort(zeros[static_cast<long long>(gi) * N + n]) : 0x4308u;
      w = __uint_as_float(deq4(byte, z | (z << 16), sbits | (sbits << 16)) << 16);
    } else {
      const float zero = zeros ? __bfloat162float(zeros[static_cast<long long>(gi) * N + n]) : 128.0f;
      const float v = deq8(qw[static_cast<long long>(k) * N + n], 0, zero, __uint_as_float(sbits << 16));
      w = __uint_as_float((cvt_bf16x2(0.0f, v) & 0xFFFFu) << 16);
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
      if (m0 + i < M) acc[i] += __bfloat162float(x[static_cast<long long>(m0 + i) * ldx + k]) * w;
  }
#pragma unroll
  for (int i = 0; i < MT; ++i)
    if (m0 + i < M) {
      __nv_bfloat16 o = __float2bfloat16_rn(acc[i]);
      if (bias) o = __float2bfloat16_rn(__bfloat162float(o) + __bfloat162float(bias[n]));
      if (epilogue == DXB_EPILOGUE_GELU_TANH) o = __float2bfloat16_rn(gelu_tanh(__bfloat162float(o)));
      out[static_cast<long long>(m0 + i) * ldo + n] = o;
    }
}

// ------------------------------------------------------------------ host side
static long long* g_trace = nullptr;

// Upper bound of the polled waits on flags that another GPU writes, in polls of about a
// quarter of a microsecond (default: about a second).
static std::atomic<unsigned> g_wait_tries{4000000u};
unsigned wait_tries() { return g_wait_tries.load(std::memory_order_relaxed); }

// Programmatic dependent launch is on unless DEXTER_B200_PDL=0.
static bool pdl_enabled() {
  static const bool on = [] {
    const char* e = getenv("DEXTER_B200_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

// What a call asks for beyond the plain GEMM (dxb_gemm_opts, checked and copied).
struct Opts {
  int relaid = 0;
  int epilogue = DXB_EPILOGUE_NONE;
  int max_ctas = 0;
  int serialize = 0;
  PeerFuse peer = {};
};

struct Plan {
  int NU, planes, rows, unit_rows, w_stage_bytes, units_per_tile, tiles, tiles_n, total_units, stages,
      w_stages, x_stage_bytes, x_rows, ctas, block,
      max_slots, nacc, recv_bytes, recv_off, recv_alias, whole;
  size_t smem_bytes;
};

// Cost, in units, of finishing a tile that equal unit ranges cut between CTAs: the finisher
// reads the other CTAs' fp32 partial tiles from L2 and adds them to its accumulator.
static int fixup_units(int NU) {
  // Measured, us equal ranges / whole tiles, int4 with 83 tokens: 3072 x 14336 (112 tiles) 17.8 / 10.2, i.e. finishing
  // shared tiles costs about as much as 20 units; 157 tiles, a second round for nine of them: 3072 x 20096 18.9 /
  // 16.5 (the line lies a little early here), 8192 x 20096 32.2 / 40.5, 14336 x 20096 51.3 / 72.7; 128 tokens 3072 x
  // 20096 21.9 / 19.7, 8192 x 20096 39.1 / 46.0.
  return NU > 96 ? 32 : 20;
}

// int8 units are 16 KB: with four weight stages a team has one, and waits for HBM in every unit.  Three
// activation stages instead of four make room for eight with 89 to 120 tokens (83 tokens 3072 x 14336, when
// activations were held in sixteens: four weight stages 15.1 us, three activation stages 13.7; now both fit, 12.9 ->
// 12.1); elsewhere four fit anyway or the stage costs more than it brings (913 tokens: 66.8 -> 72.3 us; with two
// stages everything is slower).
static int activation_stages(int bits, int blocks, int x_stage_bytes, int reserved) {
  auto w_stages = [&](int x) { return (kSmemBudget - reserved - x * x_stage_bytes) / (128 * kTileN); };
  return bits == 8 && blocks == 1 && w_stages(4) < 2 * kAStages && w_stages(3) >= 2 * kAStages ? 3 : kAStages;
}

static Plan make_plan_uncached(int M, int N, int K, int bits, int sms, int max_ctas, bool allow_split) {
  Plan pl{};
  // More than 128 tokens: token blocks of 128, each (block, column tile) pair is a tile of
  // its own, so one launch covers all of them and every SM stays busy.
  const int blocks = (M + 127) / 128;
  pl.NU = blocks > 1 ? 128 : ((M + 15) / 16) * 16;
  // A unit is 128 logical k in two planes of 64: 64 packed rows of int4, 128 rows of int8.
  pl.planes = 2;
  pl.rows = bits == 4 ? K / 2 : K;
  pl.unit_rows = bits == 4 ? 64 : 128;
  pl.w_stage_bytes = pl.unit_rows * kTileN;
  pl.units_per_tile = pl.rows / pl.unit_rows;
  pl.tiles_n = (N + kTileN - 1) / kTileN;
  pl.tiles = pl.tiles_n * blocks;
  pl.total_units = pl.units_per_tile * pl.tiles;
  pl.block = 128;
  // Rows of activations that are loaded.  int8: whole swizzle atoms of 8, where the MMA takes whole sixteens, which
  // makes room for weights (see activation_stages).  What the MMA reads beyond them (the next rows in shared memory,
  // whatever they are) only reaches accumulator columns of tokens that do not exist.  (int4 has the room; FFN of
  // 83 tokens 24.6 us in sixteens, 24.9 in eights.)
  pl.x_rows = bits == 8 && blocks == 1 ? (M + 7) / 8 * 8 : pl.NU;
  pl.x_stage_bytes = pl.planes * pl.x_rows * 128;
  // Shared memory: four activation stages (one per unit slot, like the TMEM ring; int8: see above) and
  // as deep a ring of packed-weight stages as still fits: those come from HBM and
  // need the most bytes in flight.  The depth is a multiple of four so that every
  // stage is only ever used by one dequant team, in order.
  // Launches that may split tiles over a cluster keep room for its receive buffers
  // (at most NU + 8 token rows of 128 fp32) behind the two rings.
  const int budget_ctas = (max_ctas > 0 && max_ctas < sms) ? max_ctas : sms;
  pl.recv_bytes = (pl.tiles * 2 <= budget_ctas && pl.units_per_tile >= 2) ? (pl.NU + 8) * kTileN * 4 : 0;
  pl.stages = activation_stages(bits, blocks, pl.x_stage_bytes, pl.recv_bytes);
  int w_stages = (kSmemBudget - pl.recv_bytes - pl.stages * pl.x_stage_bytes) / pl.w_stage_bytes;
  pl.recv_alias = 0;
  // Units a cluster's CTA gets (the launcher may end up with a smaller cluster and more).
  const int share = pl.recv_bytes > 0 ? budget_ctas / pl.tiles : 1;
  const int cluster_units = pl.units_per_tile / (share > 8 ? 8 : share < 1 ? 1 : share);
  if (pl.recv_bytes > 0 && ((w_stages / kAStages) * kAStages * pl.w_stage_bytes < 2 * kAStages * kWStage ||
                            (w_stages < 2 * kAStages && bits == 8 && cluster_units >= 12))) {
    // Not enough room for a useful weight ring next to the receive buffers (more than 96
    // tokens; long shares of int8, which want eight stages of 16 KB): let them lie over the rings
    // instead.  The partial rows are then sent after a cluster barrier at the end of the main loop,
    // when the rings are idle.
    pl.stages = activation_stages(bits, blocks, pl.x_stage_bytes, 0);
    w_stages = (kSmemBudget - pl.stages * pl.x_stage_bytes) / pl.w_stage_bytes;
    pl.recv_alias = 1;
  }
  w_stages = (w_stages / kAStages) * kAStages;
  if (w_stages > kMaxWStages) w_stages = kMaxWStages;
  pl.w_stages = w_stages;
  const int rings = pl.w_stages * pl.w_stage_bytes + pl.stages * pl.x_stage_bytes;
  if (pl.recv_alias && pl.recv_bytes > rings) {  // does not fit there either: no cluster split
    pl.recv_alias = 0;
    pl.recv_bytes = 0;
  }
  pl.recv_off = pl.recv_alias ? 0 : rings;
  pl.smem_bytes = static_cast<size_t>(rings) + (pl.recv_alias ? 0 : pl.recv_bytes) + 1024 + (pl.NU - pl.x_rows) * 128;
  // Grid: `budget` CTAs at most (all SMs unless the caller caps it, e.g. to run several
  // GEMMs side by side).
  const int budget = budget_ctas;
  // Two ways to hand out the work.  Whole tiles: every CTA takes `rounds` complete tiles
  // (CTAs may idle, nothing is split).  Equal unit ranges over all CTAs: nobody idles, but
  // the tiles cut by a range boundary are finished through global scratch (see the
  // epilogue).  Take whichever ends sooner.  (Few tiles in one token block are split over
  // clusters instead; the launcher decides that, see launch_tc.)
  const int rounds = (pl.tiles + budget - 1) / budget;
  const int whole_ctas = (pl.tiles + rounds - 1) / rounds;
  const long long whole_units = static_cast<long long>(rounds) * pl.units_per_tile;
  const long long split_units = (pl.total_units + budget - 1) / budget + fixup_units(pl.NU);
  // whole tiles: CTA c takes tiles [c * tiles / ctas, (c + 1) * tiles / ctas), at most `rounds`
  const bool whole = !allow_split || whole_units <= split_units;
  int ctas = whole ? whole_ctas : budget;
  if (ctas > pl.total_units) ctas = pl.total_units;
  pl.ctas = ctas;
  pl.whole = whole ? 1 : 0;
  pl.nacc = 2;
  int max_slots = 1;
  for (int t = 0; t < pl.tiles && !whole; ++t) {
    const long long u0 = static_cast<long long>(t) * pl.units_per_tile;
    const int c0 = owner_of(u0, pl.total_units, ctas);
    const int c1 = owner_of(u0 + pl.units_per_tile - 1, pl.total_units, ctas);
    if (c1 - c0 + 1 > max_slots) max_slots = c1 - c0 + 1;
  }
  pl.max_slots = max_slots;
  return pl;
}

// Plan for CTA pairs over `pairs` clusters of two, tokens in `blocks` equal blocks of at most 256.
static Plan make_pair_plan(int M, int N, int K, int bits, int pairs, int blocks) {
  Plan pl{};
  if (blocks < (M + 255) / 256) blocks = (M + 255) / 256;  // more tokens than an MMA takes are not encodable
  pl.block = ((M + blocks - 1) / blocks + 31) / 32 * 32;  // a pair MMA takes its N in steps of 32
  pl.NU = pl.block;
  pl.planes = 2;
  pl.rows = bits == 4 ? K / 2 : K;
  pl.unit_rows = bits == 4 ? 64 : 128;
  pl.w_stage_bytes = pl.unit_rows * kTileN;
  pl.units_per_tile = pl.rows / pl.unit_rows;
  pl.tiles_n = (N + 2 * kTileN - 1) / (2 * kTileN);
  pl.tiles = pl.tiles_n * ((M + pl.block - 1) / pl.block);
  pl.total_units = pl.units_per_tile * pl.tiles;
  pl.x_rows = pl.NU / 2;
  pl.x_stage_bytes = pl.planes * pl.x_rows * 128;
  pl.stages = kAStages;
  int w_stages = (kSmemBudget - pl.stages * pl.x_stage_bytes) / pl.w_stage_bytes / kAStages * kAStages;
  pl.w_stages = w_stages > kMaxWStages ? kMaxWStages : w_stages;
  pl.smem_bytes = static_cast<size_t>(pl.w_stages) * pl.w_stage_bytes + pl.stages * pl.x_stage_bytes + 1024;
  const int rounds = (pl.tiles + pairs - 1) / pairs;
  pl.ctas = (pl.tiles + rounds - 1) / rounds;  // pairs
  pl.whole = 1;
  pl.nacc = pl.NU <= 128 ? 2 : 1;
  pl.max_slots = 1;
  return pl;
}

struct PlanKey {
  int M, N, K, bits, sms, max_ctas, split;
  bool operator==(const PlanKey& o) const {
    return M == o.M && N == o.N && K == o.K && bits == o.bits && sms == o.sms && max_ctas == o.max_ctas &&
           split == o.split;
  }
};
struct PlanKeyHash {
  size_t operator()(const PlanKey& k) const {
    size_t h = 1469598103934665603ull;
    for (int v : {k.M, k.N, k.K, k.bits, k.sms, k.max_ctas, k.split}) h = (h ^ static_cast<size_t>(v)) * 1099511628211ull;
    return h;
  }
};
// Plans only depend on the shape, so they are computed once per shape and thread.
static Plan make_plan(int M, int N, int K, int bits, int sms, int max_ctas, bool allow_split = true) {
  static thread_local std::unordered_map<PlanKey, Plan, PlanKeyHash> cache;
  const PlanKey key{M, N, K, bits, sms, max_ctas, allow_split ? 1 : 0};
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  if (cache.size() > 4096) cache.clear();
  return cache.emplace(key, make_plan_uncached(M, N, K, bits, sms, max_ctas, allow_split)).first->second;
}

// The counter block has one fixed size so that calls with different tile counts
// never let one call's partial sums land on another call's counters.
static size_t counters_bytes(int) { return static_cast<size_t>(kMaxTiles) * 4; }

// Shapes wq_gemm_tc takes: those of tc_supported, and for int8 whole units of 128 rows.
static bool gemm_tc_supported(int M, int N, int K, int group, int bits) {
  return tc_supported(M, N, K, group, bits) && (bits != 8 || K % 128 == 0);
}

// Workspace the tensor-core launch of this problem needs (status, counters, partial sums).
static size_t plan_workspace_bytes(int M, int N, int K, int bits, int max_ctas) {
  DeviceInfo& di = device_info();
  const Plan pl = make_plan(M, N, K, bits, di.sms > 0 ? di.sms : 148, max_ctas);
  return kStatusBytes + counters_bytes(pl.tiles) +
         static_cast<size_t>(pl.tiles) * pl.max_slots * pl.NU * kTileN * sizeof(float);
}

// TMA tensor maps are encoded once per (pointer, geometry) and thread, not per call.
struct MapKey {
  const void* ptr;
  long long a, b, c;
  int kind;
  bool operator==(const MapKey& o) const { return ptr == o.ptr && a == o.a && b == o.b && c == o.c && kind == o.kind; }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.ptr) * 1099511628211ull;
    for (long long v : {k.a, k.b, k.c, static_cast<long long>(k.kind)}) h = (h ^ static_cast<size_t>(v)) * 1099511628211ull;
    return h;
  }
};
template <class Encode>
static const CUtensorMap* cached_map(const MapKey& key, Encode&& encode) {
  static thread_local std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  auto it = cache.find(key);
  if (it != cache.end()) return &it->second;
  if (cache.size() > 16384) cache.clear();
  CUtensorMap m;
  if (!encode(&m)) return nullptr;
  return &cache.emplace(key, m).first->second;
}

using TcKernel = void (*)(const CUtensorMap, const CUtensorMap, const WqParams, const GroupArgs<false>);

template <int BITS, bool HAS_ZERO, bool MULTI, bool RELAID>
static TcKernel pick_mode(int mode) {
  switch (mode) {
    case kModeWhole: return wq_gemm_tc<BITS, HAS_ZERO, MULTI, RELAID, kModeWhole>;
    case kModeCluster: return wq_gemm_tc<BITS, HAS_ZERO, MULTI, RELAID, kModeCluster>;
    case kModePair: return wq_gemm_tc<BITS, HAS_ZERO, true, RELAID, kModePair>;
    case kModeSplit: return wq_gemm_tc<BITS, HAS_ZERO, true, RELAID, kModeSplit>;
    default: return wq_gemm_tc<BITS, HAS_ZERO, MULTI, RELAID, kModeGeneral>;
  }
}

template <int BITS, bool HAS_ZERO>
static TcKernel pick_kernel(bool multi, bool relaid, int mode) {
  if (BITS == 4 && relaid)
    return multi ? pick_mode<BITS, HAS_ZERO, true, BITS == 4>(mode) : pick_mode<BITS, HAS_ZERO, false, BITS == 4>(mode);
  return multi ? pick_mode<BITS, HAS_ZERO, true, false>(mode) : pick_mode<BITS, HAS_ZERO, false, false>(mode);
}

// CTA pairs that are resident at once, within a budget of CTAs.
static int resident_pairs(const void* kernel, int budget) {
  int dev = 0;
  cudaGetDevice(&dev);
  static thread_local std::unordered_map<size_t, int> cache;
  const size_t key = reinterpret_cast<size_t>(kernel) * 64 + static_cast<size_t>(dev);
  auto it = cache.find(key);
  if (it == cache.end()) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBudget + 1024;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
    it = cache.emplace(key, n).first;
  }
  return it->second < budget / 2 ? it->second : budget / 2;
}

// Scratch of a pair plan whose K is split: fp32 sums of all slices but one.
static size_t pair_split_bytes(const Plan& pp, int split) {
  return static_cast<size_t>(pp.tiles) * 2 * (split - 1) * pp.NU * kTileN * sizeof(float);
}

// What CTA pairs are to do: token blocks (0: the other plans are the better ones) and pairs per tile.
constexpr int kMaxPairSplit = 8;
struct PairChoice {
  int blocks = 0, split = 1;
};
// The shortest of the times below, all fitted to measurements on shapes between 160 x 3072 x 3072 and 913 x 13824 x
// 5120, before int8's conversion became shorter and before the activation function went beside the next tile's products.
// What they trade: a pair's unit takes as long as the MMA of its tokens (0.56 us at 256, 0.31 at
// 128), converted once for all of them, but its accumulator of more than 128 tokens is not
// double-buffered, so every further tile shows its epilogue; single CTAs convert a unit per 128
// tokens (0.36 us int4, 0.42 int8); few tiles are split over clusters instead, at 7.5 us for the
// exchange.  Which wins turns mostly on how full the last round of tiles is.
// How good the choice is: with pairs wherever they can be, without, and as chosen, over 15 weights of 2 to 157 x 2^20
// values, 10 token counts from 129 to 913 and both grids, it is within 4 % of the better at 269 of 300 points for int4
// and 267 of 300 for int8.  Furthest off, us as chosen / the other way: int8 256 tokens 1024 x 2048 8.5 / 6.6, 129
// 14336 x 3072 32.3 / 26.2, 768 1024 x 14336 29.5 / 24.1; int4 200 8192 x 20096 80.6 / 68.4, 160 14336 x 3072 24.5 / 22.0.
static PairChoice choose_pairs(const Plan& pl, int M, int N, int K, int bits, int pairs, int budget, bool may_split) {
  const int least = (M + 255) / 256;  // a block has at most 256 tokens
  PairChoice choice;
  if (pairs < 1) return choice;
  const double U = pl.units_per_tile, unit = bits == 4 ? 0.36 : 0.42;
  double best;
  if (pl.recv_bytes > 0 && pl.tiles * 2 <= budget && pl.units_per_tile >= 2) {
    int c = budget / pl.tiles;
    c = c > 8 ? 8 : c > pl.units_per_tile ? pl.units_per_tile : c;
    best = 7.5 + (U / c) * unit;
  } else {
    const int rounds = (pl.tiles + budget - 1) / budget;
    best = 2.5 + rounds * (U * unit + (bits == 4 ? 0.7 : 1.2));
  }
  for (int nb = least; nb <= least + 7; ++nb) {
    const Plan pp = make_pair_plan(M, N, K, bits, pairs, nb);
    const int rounds = (pp.tiles + pairs - 1) / pairs;
    double u = 0.02 + 0.0022 * pp.NU;
    const double least_unit = bits == 4 ? 0.30 : 0.46;
    if (u < least_unit) u = least_unit;
    const double t = 1.15 * (4.2 + rounds * U * u + (rounds - 1) * (pp.nacc == 1 ? 0.006 * pp.NU : 0.5));
    if (t < best) { best = t; choice.blocks = nb; choice.split = 1; }
    // Few tiles: several pairs per tile, with a slice of K each.  Parking and adding the sums measured
    // about 2.6 us per slice (512 tokens int8 14336 x 3072, 3 slices: 39.4 us, 48.8 without).
    for (int s = 2; may_split && s <= kMaxPairSplit && pp.tiles * s <= pairs && s <= pp.units_per_tile / 4; ++s) {
      const double ts = 1.15 * (4.2 + (U / s) * u + 0.8 + 2.6 * (s - 1));
      if (ts < best) { best = ts; choice.blocks = nb; choice.split = s; }
    }
  }
  return choice;
}

// Workspace that one launch of this problem wants because it shares tiles between CTAs (counters and partial
// sums); 0 where it leaves all but the status word alone.  (Tiles split over clusters add through distributed
// shared memory; where no cluster is resident, launch_tc hands out whole tiles.)
static size_t launch_scratch_bytes(int M, int N, int K, int bits, int max_ctas) {
  static thread_local std::unordered_map<PlanKey, size_t, PlanKeyHash> cache;
  const PlanKey key{M, N, K, bits, 0, max_ctas, 0};
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  const int sms = device_info().sms > 0 ? device_info().sms : 148;
  const int budget = (max_ctas > 0 && max_ctas < sms) ? max_ctas : sms;
  const Plan pl = make_plan(M, N, K, bits, sms, max_ctas);
  PairChoice choice;
  if (M > 128) choice = choose_pairs(pl, M, N, K, bits, budget / 2, budget, true);
  size_t need = 0;
  if (choice.blocks > 0) {
    if (choice.split > 1)
      need = kStatusBytes + counters_bytes(0) +
             pair_split_bytes(make_pair_plan(M, N, K, bits, budget / 2, choice.blocks), choice.split);
  } else if (pl.recv_bytes == 0 && pl.max_slots > 1) {
    need = plan_workspace_bytes(M, N, K, bits, max_ctas);
  }
  if (cache.size() > 4096) cache.clear();
  return cache.emplace(key, need).first->second;
}

// Boxes of one unit of packed weights, and of the activations that go with it.
static const CUtensorMap* weight_map(int bits, const void* qw, int N, int rows) {
  return cached_map(MapKey{qw, N, rows, 0, bits}, [&](CUtensorMap* m) {
    const uint64_t dims[2] = {static_cast<uint64_t>(N), static_cast<uint64_t>(rows)};
    const uint64_t strides[1] = {static_cast<uint64_t>(N)};
    const uint32_t box[2] = {kTileN, bits == 4 ? 64u : 128u};
    return make_map(m, qw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  });
}
static const CUtensorMap* activation_map(int bits, const void* x, long long ldx, int M, int K, int x_rows) {
  return cached_map(MapKey{x, ldx, (static_cast<long long>(M) << 32) | K, x_rows, 16 + bits}, [&](CUtensorMap* m) {
    if (bits == 4) {
      // X seen as [plane][token][k within the plane]: one box brings both k-slices of a unit.
      const uint64_t dims[3] = {static_cast<uint64_t>(K / 2), static_cast<uint64_t>(M), 2};
      const uint64_t strides[2] = {static_cast<uint64_t>(ldx) * 2, static_cast<uint64_t>(K / 2) * 2};
      const uint32_t box[3] = {64, static_cast<uint32_t>(x_rows), 2};
      return make_map(m, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    }
    const uint64_t dims[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(M)};
    const uint64_t strides[1] = {static_cast<uint64_t>(ldx) * 2};
    const uint32_t box[2] = {64, static_cast<uint32_t>(x_rows)};
    return make_map(m, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  });
}

// Streaming past, weights push activations, scales and results out of L2 before their next use, unless they are
// told to go first.  That costs where a weight would have been there again at its next use.  Whether it would depends on
// all that a program reads in between; the launch only knows one weight's size, so it goes by that: from a
// quarter of the L2 on all of its lines go first, from an eighth on half of them, below that none.  The lines are set for
// programs of few weights, which are those that lose: three sets in turn, us with normal priority / half / all: FFN of
// 83 tokens 3072 x 14336 int8 (44 MB a weight) 35.0 / 33.9 / 32.4, int4 (22 MB) 26.3 / 25.2 / 25.3; 125 tokens int8 3072 x
// 8192 (25 MB, three of them fit) 12.3 / 12.4 / 12.9; 8 tokens int4 3072 x 9216 (14 MB) 7.19 / 7.30 / -; eight of 83
// tokens 3072 x 3072 int4 (4.7 MB) 6.45 / - / 6.6.  Where a model's weights exceed the L2 by far, none of them is ever there
// again, and all lines first would be the better: two int4 blocks of width 3072, 125.7 us with
// this rule, 123.3 so.  Nobody tells the launch.  (Activations told to stay instead: half the gain, and they
// would stay after their use.  A prefetch of the activations into L2: a tenth of it.)
static uint64_t weight_policy(long long bytes, bool read_once) {
  const long long l2 = device_info().l2_bytes;
  if (!read_once || bytes < l2 / 8) return kL2EvictNormal;
  return bytes < l2 / 4 ? kL2EvictFirstHalf : kL2EvictFirst;
}

// The part of the parameters that follows from the plan.
static WqParams plan_params(const Plan& pl, int M, int K, int group, void* workspace) {
  WqParams p{};
  uint8_t* wsb = static_cast<uint8_t*>(workspace);
  p.status = reinterpret_cast<int*>(wsb);
  p.counters = reinterpret_cast<int*>(wsb + kStatusBytes);
  p.partials = reinterpret_cast<float*>(wsb + kStatusBytes + counters_bytes(pl.tiles));
  p.M = M; p.K = K; p.group = group;
  p.NU = pl.NU;
  p.units_per_tile = pl.units_per_tile;
  p.tiles = pl.tiles;
  p.tiles_n = pl.tiles_n;
  p.block = pl.block;
  p.total_units = pl.total_units;
  p.stages = pl.stages;
  p.w_stages = pl.w_stages;
  p.x_stage_bytes = pl.x_stage_bytes;
  p.max_slots = pl.max_slots;
  p.nacc = pl.nacc;
  const int gu = group / kUnitRows;
  p.group_shift = -1;
  for (int b = 0; b < 20; ++b) if ((1 << b) == gu) p.group_shift = b;
  return p;
}

// WqParams::sz_step: planes of 64 k from one of a team's units to its next, in quantisation groups.
static int scale_step(int bits, int N, int K, int group) {
  const int gu = group / kUnitRows, stride = kAStages * (bits == 4 ? 1 : 2);
  return group == K ? 0 : stride % gu == 0 ? stride / gu * (N / 4) : -1;
}

template <int BITS, bool HAS_ZERO>
static int launch_tc(const void* x, long long ldx, const void* qw, const void* scales,
                     const void* zeros, const void* bias, void* out, long long ldo, int M, int N,
                     int K, int group, void* workspace, size_t workspace_bytes, const Opts& opts,
                     cudaStream_t stream) {
  DeviceInfo& di = device_info();
  const int max_ctas = opts.max_ctas;
  Plan plan = make_plan(M, N, K, BITS, di.sms, max_ctas);
  const Plan* plp = &plan;
  const bool multi = plp->tiles > plp->tiles_n;
  if (plp->w_stages < kAStages) return DXB_ERR_UNSUPPORTED;
  // Status word and counters are always needed; the partial sums only if the launch ends up
  // splitting tiles through global scratch (checked below, once the cluster size is known).
  if (workspace == nullptr || workspace_bytes < kStatusBytes + counters_bytes(plp->tiles))
    return DXB_ERR_WORKSPACE;

  int dev = 0;
  cudaGetDevice(&dev);
  static thread_local int attr_dev = -1;
  if (attr_dev != dev) {
    bool ok = true;
    auto set = [&](auto kern) {
      ok = ok && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget + 2048) == cudaSuccess;
    };
    for (int multi = 0; multi < 2; ++multi)
      for (int relaid = 0; relaid < (BITS == 4 ? 2 : 1); ++relaid)
        for (int mode = 0; mode < 5; ++mode) set(pick_kernel<BITS, HAS_ZERO>(multi, relaid, mode));
    if (!ok) return DXB_ERR_CUDA;
    attr_dev = dev;
  }
  const bool relaid = BITS == 4 && opts.relaid;
  // The lean instances serve every launch without a sum over ranks; which of the two follows from the plan below.
  const bool lean = opts.peer.world <= 1;
  auto kernel = pick_kernel<BITS, HAS_ZERO>(multi, relaid, lean ? kModeCluster : kModeGeneral);

  // Few tiles: split each tile's K range over a thread-block cluster (<= 8 CTAs) that
  // reduces through distributed shared memory.  The cluster size is the largest one for
  // which all clusters are resident at once; the answer is cached per configuration.
  int cluster = 1;
  int pair_blocks = 0;  // > 0: CTA pairs, this many token blocks
  int pair_split = 1;   // and this many pairs per tile
  const int budget = (max_ctas > 0 && max_ctas < di.sms) ? max_ctas : di.sms;
  if (multi && lean) {
    const int pairs = resident_pairs(reinterpret_cast<const void*>(pick_kernel<BITS, HAS_ZERO>(true, relaid, kModePair)), budget);
    static thread_local std::unordered_map<size_t, PairChoice> chosen;
    const Plan base = *plp;
    auto choose = [&](bool may_split) {
      const size_t key = (((static_cast<size_t>(M) * 1000003u + static_cast<size_t>(N)) * 1000003u + static_cast<size_t>(K)) * 512u +
                          static_cast<size_t>(budget)) * 2u + (may_split ? 1u : 0u);
      auto it = chosen.find(key);
      if (it == chosen.end()) {
        if (chosen.size() > 4096) chosen.clear();
        it = chosen.emplace(key, choose_pairs(base, M, N, K, BITS, pairs, budget, may_split)).first;
      }
      return it->second;
    };
    PairChoice choice = choose(true);
    if (choice.split > 1) {  // only with room for the partial sums
      const Plan pp = make_pair_plan(M, N, K, BITS, pairs, choice.blocks);
      if (workspace_bytes < kStatusBytes + counters_bytes(0) + pair_split_bytes(pp, choice.split)) choice = choose(false);
    }
    pair_blocks = choice.blocks;
    pair_split = choice.split;
    if (pair_blocks > 0) {
      plan = make_pair_plan(M, N, K, BITS, pairs, pair_blocks);
      kernel = pick_kernel<BITS, HAS_ZERO>(true, relaid, pair_split > 1 ? kModeSplit : kModePair);
    }
  }
  if (pair_blocks == 0 && plp->recv_bytes > 0 && plp->tiles * 2 <= budget && plp->units_per_tile >= 2) {
    static thread_local std::unordered_map<long long, int> cache;
    const long long key = (static_cast<long long>(dev) << 48) ^ (static_cast<long long>(plp->tiles) << 28) ^
                          (static_cast<long long>(plp->units_per_tile) << 8) ^ static_cast<long long>(plp->NU >> 4) ^
                          (static_cast<long long>(budget) << 38) ^ (static_cast<long long>(multi) << 58) ^
                          (static_cast<long long>(relaid) << 59) ^ (static_cast<long long>(lean) << 60);
    auto it = cache.find(key);
    if (it != cache.end()) {
      cluster = it->second;
    } else {
      int cmax = budget / plp->tiles;
      if (cmax > 8) cmax = 8;
      if (cmax > plp->units_per_tile) cmax = plp->units_per_tile;
      for (int c = cmax; c >= 2; --c) {
        cudaLaunchConfig_t qcfg = {};
        qcfg.gridDim = dim3(plp->tiles * c);
        qcfg.blockDim = dim3(kThreads);
        qcfg.dynamicSmemBytes = plp->smem_bytes;
        cudaLaunchAttribute qattr[1];
        qattr[0].id = cudaLaunchAttributeClusterDimension;
        qattr[0].val.clusterDim.x = c;
        qattr[0].val.clusterDim.y = 1;
        qattr[0].val.clusterDim.z = 1;
        qcfg.attrs = qattr;
        qcfg.numAttrs = 1;
        int resident = 0;
        if (cudaOccupancyMaxActiveClusters(&resident, kernel, &qcfg) == cudaSuccess &&
            resident >= plp->tiles) {
          cluster = c;
          break;
        }
        cudaGetLastError();
      }
      cache[key] = cluster;
    }
    if (cluster == 1) plan = make_plan(M, N, K, BITS, di.sms, max_ctas, false);
  }
  if (cluster == 1 && pair_blocks == 0) {
    const size_t need = kStatusBytes + counters_bytes(plp->tiles) +
                        static_cast<size_t>(plp->tiles) * plp->max_slots * plp->NU * kTileN * sizeof(float);
    if (workspace_bytes < need) {
      // The workspace was sized for another grid cap: whole tiles need no partial sums.
      if (plp->max_slots > 1) plan = make_plan(M, N, K, BITS, di.sms, max_ctas, false);
      if (plp->max_slots > 1) return DXB_ERR_WORKSPACE;
    }
  }
  const Plan& pl = *plp;
  if (cluster == 1 && pair_blocks == 0)
    kernel = pick_kernel<BITS, HAS_ZERO>(multi, relaid, lean && pl.whole ? kModeWhole : kModeGeneral);

  const CUtensorMap* tq = weight_map(BITS, qw, N, pl.rows);
  const CUtensorMap* tx = activation_map(BITS, x, ldx, M, K, pl.x_rows);
  if (!tq || !tx) return DXB_ERR_TENSORMAP;

  WqParams p = plan_params(pl, M, K, group, workspace);
  p.scales = static_cast<const __nv_bfloat16*>(scales);
  p.zeros = static_cast<const __nv_bfloat16*>(zeros);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.ldo = ldo;
  p.N = N;
  p.half_k = BITS == 4 ? K / 2 : 0;
  p.sz_step = scale_step(BITS, N, K, group);
  p.trace = g_trace;
  p.epilogue = opts.epilogue;
  p.tile_ranges = (cluster == 1 && pl.whole) ? 1 : 0;
  p.peer = opts.peer;
  p.split = pair_blocks > 0 ? pair_split : 1;
  p.cluster = cluster;
  p.recv_off = pl.recv_off;
  p.recv_alias = cluster > 1 ? pl.recv_alias : 0;
  p.rows_per = ((M > 128 ? 128 : M) + cluster - 1) / cluster;  // token rows of one block per CTA
  {
    const int what = cluster > 1 || p.split > 1 ? pl.units_per_tile : pl.tiles;
    const int parts = cluster > 1 ? cluster : p.split > 1 ? p.split : pl.ctas;
    p.range_q = what / parts;
    p.range_r = what % parts;
  }
  // Each weight is read once, or by all token blocks at one time?
  const bool once = pl.tiles == pl.tiles_n || cluster > 1 || p.split > 1 || (pl.whole && pl.tiles <= pl.ctas);
  p.w_policy = weight_policy(static_cast<long long>(pl.rows) * N, once);
  p.rows_inv = (65536 + p.rows_per - 1) / p.rows_per;

  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.split > 1 ? 2 * pl.tiles * p.split : pair_blocks > 0 ? 2 * pl.ctas : cluster > 1 ? pl.tiles * cluster : pl.ctas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = pl.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int nattr = 0;
  if (cluster > 1 || pair_blocks > 0) {
    attr[nattr].id = cudaLaunchAttributeClusterDimension;
    attr[nattr].val.clusterDim.x = pair_blocks > 0 ? 2 : cluster;
    attr[nattr].val.clusterDim.y = 1;
    attr[nattr].val.clusterDim.z = 1;
    ++nattr;
  }
  if (pdl_enabled() && !opts.serialize) {
    // Let this launch begin while the previous kernel of the stream drains: the kernel
    // itself waits (griddepcontrol.wait) before touching anything that kernel may produce.
    attr[nattr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[nattr].val.programmaticStreamSerializationAllowed = 1;
    ++nattr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = nattr;
  if (cudaLaunchKernelEx(&cfg, kernel, *tq, *tx, p, GroupArgs<false>{}) != cudaSuccess) {
    cudaGetLastError();
    return DXB_ERR_CUDA;
  }
  return cudaGetLastError() == cudaSuccess ? DXB_OK : DXB_ERR_CUDA;
}

// Several problems as one launch of whole tiles, one per CTA (more tiles than SMs start as others end).
template <int BITS, bool HAS_ZERO>
static int launch_group(const dxb_group_item* items, int count, int M, int K, int group, void* workspace,
                        size_t workspace_bytes, const Opts& opts, cudaStream_t stream) {
  const bool relaid = BITS == 4 && opts.relaid;
  using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const WqParams, const GroupArgs<true>);
  Kernel kernel = wq_gemm_tc<BITS, HAS_ZERO, false, false, kModeGroup>;
  if constexpr (BITS == 4)
    if (relaid) kernel = wq_gemm_tc<BITS, HAS_ZERO, false, true, kModeGroup>;
  GroupArgs<true> g{};
  int tiles = 0;
  for (int i = 0; i < count; ++i) tiles += (items[i].n + kTileN - 1) / kTileN;
  const DeviceInfo& di = device_info();
  const Plan pl = make_plan(M, tiles * kTileN, K, BITS, di.sms, 0, false);
  if (pl.w_stages < kAStages) return DXB_ERR_UNSUPPORTED;
  if (workspace == nullptr || workspace_bytes < kStatusBytes) return DXB_ERR_WORKSPACE;
  int dev = 0;
  cudaGetDevice(&dev);
  static thread_local int attr_dev[2] = {-1, -1};
  if (attr_dev[relaid] != dev) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget + 2048) != cudaSuccess)
      return DXB_ERR_CUDA;
    attr_dev[relaid] = dev;
  }
  WqParams p = plan_params(pl, M, K, group, workspace);
  p.half_k = BITS == 4 ? K / 2 : 0;
  p.epilogue = opts.epilogue;
  p.split = p.cluster = p.tile_ranges = 1;
  p.peer = opts.peer;
  long long bytes = 0;
  g.count = count;
  tiles = 0;
  for (int i = 0; i < count; ++i) {
    const dxb_group_item& it = items[i];
    const CUtensorMap* tq = weight_map(BITS, it.qweight, it.n, pl.rows);
    if (!tq) return DXB_ERR_TENSORMAP;
    g.q[i] = *tq;
    const CUtensorMap* tx = activation_map(BITS, it.x, it.ldx, M, K, pl.x_rows);
    if (!tx) return DXB_ERR_TENSORMAP;
    g.x[i] = *tx;
    g.item[i] = {static_cast<const __nv_bfloat16*>(it.scales), static_cast<const __nv_bfloat16*>(it.zeros),
                 static_cast<const __nv_bfloat16*>(it.bias), static_cast<__nv_bfloat16*>(it.out), it.ldo, it.n, tiles,
                 scale_step(BITS, it.n, K, group)};
    tiles += (it.n + kTileN - 1) / kTileN;
    bytes += static_cast<long long>(pl.rows) * it.n;
  }
  p.w_policy = weight_policy(bytes, true);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = pl.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() && !opts.serialize ? 1 : 0;
  if (cudaLaunchKernelEx(&cfg, kernel, g.q[0], g.x[0], p, g) != cudaSuccess) {
    cudaGetLastError();
    return DXB_ERR_CUDA;
  }
  return DXB_OK;
}

// ------------------------------------------------------------- few tokens, odd shapes
// Shapes wq_gemm_small takes: whole steps of 32 packed rows with one scale row per plane each, and
// activations it can load 16 bytes at a time.
static bool small_supported(const void* x, long long ldx, int K, int group, int bits) {
  const int rows = bits == 4 ? K / 2 : K;
  return rows % 32 == 0 && group % 32 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 && ldx % 8 == 0;
}

struct SmallKernel {
  void (*fn)(const SmallParams);
  int warp_bytes;  // one warp's ring
};
template <int KIND, int ROWS, int CPW>
static SmallKernel pick_small(int mt) {
  using S1 = SmallStage<KIND, ROWS, CPW, 1>;
  using S2 = SmallStage<KIND, ROWS, CPW, 2>;
  return mt == 1 ? SmallKernel{wq_gemm_small<KIND, ROWS, CPW, 1>, S1::kBytes * S1::kStages}
                 : SmallKernel{wq_gemm_small<KIND, ROWS, CPW, 2>, S2::kBytes * S2::kStages};
}

// Shared memory a CTA may have (227 KB).
constexpr int kSmallSmem = 227 * 1024;

// Lets the kernel use more than 48 KB of shared memory; once per kernel, device and thread.
static bool small_smem_ready(void (*fn)(const SmallParams)) {
  int dev = 0;
  cudaGetDevice(&dev);
  static thread_local std::unordered_map<size_t, bool> done;
  const size_t key = reinterpret_cast<size_t>(fn) * 64 + static_cast<size_t>(dev);
  if (done.find(key) != done.end()) return true;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem) != cudaSuccess) return false;
  done[key] = true;
  return true;
}

static int launch_small(int bits, const void* x, long long ldx, const void* qw, const void* scales, const void* zeros,
                        const void* bias, void* out, long long ldo, int M, int N, int K, int group, const Opts& opts,
                        cudaStream_t stream) {
  const int sms = device_info().sms;
  const int budget = (opts.max_ctas > 0 && opts.max_ctas < sms) ? opts.max_ctas : sms;
  SmallParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.qw = static_cast<const uint8_t*>(qw);
  p.scales = static_cast<const __nv_bfloat16*>(scales);
  p.zeros = static_cast<const __nv_bfloat16*>(zeros);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.ldx = ldx; p.ldo = ldo;
  p.M = M; p.N = N; p.K = K; p.group = group;
  p.rows = bits == 4 ? K / 2 : K;
  p.steps = p.rows / 32;
  p.epilogue = opts.epilogue;
  const int mt = M <= 8 ? 1 : 2;
  const int blocks = (M + 8 * mt - 1) / (8 * mt);
  // Tiles of 32 columns.  Up to one per SM: sixteen warps each, and clusters that split K while SMs
  // are left over and every warp keeps at least two steps.  More: eight warps, two CTAs per SM.
  // (All of this fixes the order of the sums, so it must be the same for a weight and its repacked copy.)
  const long long tiles32 = static_cast<long long>((N + 31) / 32) * blocks;
  int warps = 8, cluster = 1;
  if (tiles32 <= budget) {
    warps = 16;
    while (cluster < 8 && tiles32 * cluster * 2 <= budget && p.steps >= 64 * cluster) cluster *= 2;
  }
  {
    const int g32 = group / 32;
    p.group_shift = -1;
    for (int b = 0; b < 20; ++b)
      if ((1 << b) == g32) p.group_shift = b;
  }
  const uintptr_t pq = reinterpret_cast<uintptr_t>(qw), ps = reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(zeros);
  const int how = ps % 16 == 0 && N % 8 == 0 && pq % 8 == 0 ? (N % 16 == 0 && pq % 16 == 0 ? kRows16 : kRows8)
                  : (pq | ps) % 16 == 0 ? kRowsShifted : kRowsWords;  // see there
  if (how != kRows16 && (opts.relaid || (pq | ps) % 4 != 0)) return DXB_ERR_UNSUPPORTED;
  const int kind = bits == 8 ? kSmallW8 : !opts.relaid ? kSmallW4 : zeros ? kSmallW4Relaid : kSmallW4Sym;
  // More tiles than two per SM: twice the width, so that they all still run at once.
  const bool wide = tiles32 > 2 * budget && how == kRows16 && kind != kSmallW4;
  SmallKernel k;
  if (how == kRowsWords) k = kind == kSmallW8 ? pick_small<kSmallW8, kRowsWords, 1>(mt) : pick_small<kSmallW4, kRowsWords, 1>(mt);
  else if (how == kRows8) k = kind == kSmallW8 ? pick_small<kSmallW8, kRows8, 1>(mt) : pick_small<kSmallW4, kRows8, 1>(mt);
  else if (how == kRowsShifted) k = kind == kSmallW8 ? pick_small<kSmallW8, kRowsShifted, 1>(mt) : pick_small<kSmallW4, kRowsShifted, 1>(mt);
  else if (wide) k = kind == kSmallW8 ? pick_small<kSmallW8, kRows16, 2>(mt)
                    : kind == kSmallW4Sym ? pick_small<kSmallW4Sym, kRows16, 2>(mt) : pick_small<kSmallW4Relaid, kRows16, 2>(mt);
  else k = kind == kSmallW8 ? pick_small<kSmallW8, kRows16, 1>(mt)
         : kind == kSmallW4 ? pick_small<kSmallW4, kRows16, 1>(mt)
         : kind == kSmallW4Sym ? pick_small<kSmallW4Sym, kRows16, 1>(mt) : pick_small<kSmallW4Relaid, kRows16, 1>(mt);
  const int bn = wide ? 64 : 32;
  p.tiles_n = (N + bn - 1) / bn;
  if (static_cast<long long>(p.tiles_n) * blocks > (1 << 30)) return DXB_ERR_SHAPE;
  p.tiles = p.tiles_n * blocks;
  p.ring_bytes = warps * k.warp_bytes;
  const int red_bytes = (warps * 8 * mt * (bn + 1) * 4 + 15) / 16 * 16;
  if (p.ring_bytes < red_bytes) p.ring_bytes = red_bytes;
  // A cluster's first CTA also has a receive slot for every other one.  Next to sixteen rings of int4 in words
  // (222,208 B with more than 8 tokens) there is room for three of 2 KB, so clusters of four.
  const int slot_bytes = 8 * mt * bn * 4;
  while (cluster > 1 && p.ring_bytes + (cluster - 1) * slot_bytes > kSmallSmem) cluster /= 2;
  p.cluster = cluster;
  // A caller's cap limits the CTAs, which then walk several tiles; without one every tile has its own.
  int grid = p.tiles;
  if (budget < sms && grid > budget * (16 / warps)) grid = budget * (16 / warps);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid) * cluster);
  cfg.blockDim = dim3(32 * warps);
  cfg.dynamicSmemBytes = static_cast<size_t>(p.ring_bytes) + static_cast<size_t>(cluster - 1) * slot_bytes;
  if (!small_smem_ready(k.fn)) return DXB_ERR_CUDA;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int nattr = 0;
  if (cluster > 1) {
    attr[nattr].id = cudaLaunchAttributeClusterDimension;
    attr[nattr].val.clusterDim.x = cluster;
    attr[nattr].val.clusterDim.y = 1;
    attr[nattr].val.clusterDim.z = 1;
    ++nattr;
  }
  if (pdl_enabled() && !opts.serialize) {
    attr[nattr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[nattr].val.programmaticStreamSerializationAllowed = 1;
    ++nattr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = nattr;
  if (cudaLaunchKernelEx(&cfg, k.fn, p) != cudaSuccess) {
    cudaGetLastError();
    return DXB_ERR_CUDA;
  }
  return DXB_OK;
}

template <int BITS>
static int launch_simt(const void* x, long long ldx, const void* qw, const void* scales,
                       const void* zeros, const void* bias, void* out, long long ldo, int M, int N,
                       int K, int group, const Opts& opts, cudaStream_t stream) {
  dim3 block(128), grid((N + 127) / 128, (M + 7) / 8);
  wq_gemm_simt<BITS><<<grid, block, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(x), ldx, static_cast<const uint8_t*>(qw),
      static_cast<const __nv_bfloat16*>(scales), static_cast<const __nv_bfloat16*>(zeros),
      static_cast<const __nv_bfloat16*>(bias), static_cast<__nv_bfloat16*>(out), ldo, M, N, K, group,
      opts.relaid, opts.epilogue);
  return cudaGetLastError() == cudaSuccess ? DXB_OK : DXB_ERR_CUDA;
}

static int check_args(int bits, const void* x, long long ldx, const void* qw, const void* scales,
                      void* out, long long ldo, int M, int N, int K, int group) {
  if (bits != 4 && bits != 8) return DXB_ERR_BITS;
  if (!x || !qw || !scales || !out) return DXB_ERR_NULL;
  if (M < 0 || N <= 0 || K <= 0 || group <= 0) return DXB_ERR_SHAPE;
  if (K % group) return DXB_ERR_SHAPE;
  if (bits == 4 && (K % 2)) return DXB_ERR_SHAPE;
  if (ldx < K || ldo < N) return DXB_ERR_SHAPE;
  return DXB_OK;
}

static bool pointers_aligned(int bits, const void* x, long long ldx, const void* qweight, const void* scales,
                             const void* zeros, const void* bias, const void* out, long long ldo, int K) {
  return (reinterpret_cast<uintptr_t>(x) % 16 == 0) && (ldx % 8 == 0) &&
         (reinterpret_cast<uintptr_t>(qweight) % 16 == 0) && (reinterpret_cast<uintptr_t>(scales) % 16 == 0) &&
         (zeros == nullptr || reinterpret_cast<uintptr_t>(zeros) % 16 == 0) &&
         (bias == nullptr || reinterpret_cast<uintptr_t>(bias) % 8 == 0) &&
         (reinterpret_cast<uintptr_t>(out) % 8 == 0) && (ldo % 4 == 0) && (bits != 4 || (K / 2) % 8 == 0);
}

// Checks dxb_gemm_opts against the problem and copies it.
static int read_opts(const dxb_gemm_opts* o, int bits, int M, int N, int K, Opts* out) {
  Opts r;
  if (o) {
    if (o->weight_layout != DXB_LAYOUT_DEXTER && o->weight_layout != DXB_LAYOUT_B200) return DXB_ERR_UNSUPPORTED;
    if (o->weight_layout == DXB_LAYOUT_B200 && (bits != 4 || (K / 2) % 2 || N % 4)) return DXB_ERR_UNSUPPORTED;
    if (o->epilogue != DXB_EPILOGUE_NONE && o->epilogue != DXB_EPILOGUE_GELU_TANH) return DXB_ERR_UNSUPPORTED;
    r.relaid = o->weight_layout == DXB_LAYOUT_B200;
    r.epilogue = o->epilogue;
    r.max_ctas = o->max_ctas;
    r.serialize = o->serialize;
    if (o->peer_world > 1) {
      if (o->peer_world > kPeerMaxRanks || o->peer_rank < 0 || o->peer_rank >= o->peer_world) return DXB_ERR_SHAPE;
      if (!o->peer_regions) return DXB_ERR_NULL;
      // one token block, whole 4-column groups, a counter per tile, room for the partial output
      if (M > 128 || N % 4 || (N + kTileN - 1) / kTileN > kFusedMaxTiles) return DXB_ERR_UNSUPPORTED;
      if (o->peer_capacity_elems < static_cast<int64_t>(M) * N) return DXB_ERR_SHAPE;
      for (int i = 0; i < o->peer_world; ++i) {
        if (!o->peer_regions[i] || reinterpret_cast<uintptr_t>(o->peer_regions[i]) % 16) return DXB_ERR_NULL;
        r.peer.region[i] = static_cast<unsigned char*>(o->peer_regions[i]);
      }
      r.peer.capacity = o->peer_capacity_elems;
      r.peer.rank = o->peer_rank;
      r.peer.world = o->peer_world;
      r.peer.wait_tries = wait_tries();
    }
  }
  *out = r;
  return DXB_OK;
}

// Few tokens and a weight that is read in little more than the fixed cost of a launch: there the kernel
// without set-up is ahead; with more to convert (once per 16 tokens, there) the tcgen05 pipeline is.
// The lines lie where the two crossed over 14 weights of 0.5 to 44 x 2^20 values and 18 token counts from 1 to 256, with
// both kernels on all of them (int8's before its conversion became shorter).  Near the lines, us small / tcgen05 on the
// symmetric grids: int4 1 token 3072 x 9216 6.6 / 7.2 and 3072 x 11264 8.7 / 8.6, 8 tokens 4096 x 4096 5.5 / 6.2 and 3072 x
// 6144 6.4 / 6.3, 16 tokens 3072 x 3072 5.1 / 5.4 and 4096 x 4096 6.6 / 6.2, 32 tokens 2048 x 2048 4.3 / 4.7 and 2048 x 3072
// 5.9 / 5.1, 96 tokens 1024 x 1024 4.1 / 5.1 and 1024 x 2048 6.2 / 5.5, 128 tokens 1024 x 2048 6.3 / 7.0 and 2048 x 2048 9.1 /
// 7.6 (from 97 tokens on the pipeline's clusters have their receive buffers over the rings, two more us), 160 tokens
// 512 x 1024 4.8 / 4.8; int8 8 tokens 3072 x 3072 5.6 / 5.9 and 4096 x 4096 7.2 / 7.1, 16 tokens 2048 x 2048 4.7 / 4.7 and
// 3072 x 3072 6.2 / 6.0, 80 tokens 1024 x 1024 4.6 / 4.8, 128 tokens 5.0 / 6.7 and 1024 x 2048 7.4 / 7.3.  With zero points
// as well, the choice is within 4 % of the better kernel at 981 of the 1008 points (int4 493 of 504, int8 488) and
// 14 % off at worst: up to 4 tokens 5120 x 5120 int4 (160 tiles, so CTAs of eight warps, of which a second one
// fits an SM but most SMs get one); int8 5 to 10 % at 12 and 16 tokens 2048 x 3072 and up to 8 tokens 3072 x 4096, 13 % at
// 96 tokens 1024 x 1024, where the line is a little low.
static bool small_is_faster(int M, int N, int K, int bits) {
  const long long weights = static_cast<long long>(N) * K, mega = 1 << 20;
  if (M <= 8) return weights <= (bits == 8 ? 10 : M <= 4 ? 30 : 16) * mega;
  const long long converted = weights * ((M + 15) / 16);
  if (bits == 4) return converted <= (M <= 16 ? 10 : M <= 96 ? 8 : M <= 128 ? 16 : 5) * mega;
  return converted <= (M <= 16 ? 4 : M <= 96 ? 5 : M <= 128 ? 9 : 5) * mega;
}

static int gemm_dispatch(int bits, const void* x, int64_t ldx, const void* qweight, const void* scales,
                         const void* zeros, const void* bias, void* out, int64_t ldo, int M, int N, int K,
                         int group_size, void* workspace, size_t workspace_bytes, const Opts& opts,
                         cudaStream_t stream) {
  const int max_ctas = opts.max_ctas;
  const bool aligned = pointers_aligned(bits, x, ldx, qweight, scales, zeros, bias, out, ldo, K);
  auto launch = [&](const char* xc, char* oc, int mc) -> int {
    if (bits == 4)
      return zeros ? launch_tc<4, true>(xc, ldx, qweight, scales, zeros, bias, oc, ldo, mc, N, K,
                                        group_size, workspace, workspace_bytes, opts, stream)
                   : launch_tc<4, false>(xc, ldx, qweight, scales, zeros, bias, oc, ldo, mc, N, K,
                                         group_size, workspace, workspace_bytes, opts, stream);
    return zeros ? launch_tc<8, true>(xc, ldx, qweight, scales, zeros, bias, oc, ldo, mc, N, K,
                                      group_size, workspace, workspace_bytes, opts, stream)
                 : launch_tc<8, false>(xc, ldx, qweight, scales, zeros, bias, oc, ldo, mc, N, K,
                                       group_size, workspace, workspace_bytes, opts, stream);
  };
  // The sum over ranks lives in the tensor-core kernel's epilogue only.
  if (opts.peer.world > 1 && !(aligned && gemm_tc_supported(M, N, K, group_size, bits)))
    return DXB_ERR_UNSUPPORTED;
  // Few tokens, and whatever the tensor-core pipeline cannot take.
  const bool tc = aligned && gemm_tc_supported(M <= 128 ? M : 128, N, K, group_size, bits);
  if (opts.peer.world <= 1 && (!tc || small_is_faster(M, N, K, bits)) && small_supported(x, ldx, K, group_size, bits)) {
    const int rc = launch_small(bits, x, ldx, qweight, scales, zeros, bias, out, ldo, M, N, K, group_size, opts, stream);
    if (rc != DXB_ERR_UNSUPPORTED) return rc;
  }
  // More than 128 tokens: one launch over all token blocks when the workspace holds the partial sums that it
  // parks, if any; a smaller workspace still works, block by block.
  if (M > 128 && aligned && gemm_tc_supported(M, N, K, group_size, bits) &&
      workspace_bytes >= launch_scratch_bytes(M, N, K, bits, max_ctas))
    return launch(static_cast<const char*>(x), static_cast<char*>(out), M);
  // Token blocks of at most 128 rows per launch (the UMMA N of one accumulator); 96 when the
  // weight has so few tiles that the launch splits them over clusters, whose receive buffers
  // only fit next to the activation ring up to 96 tokens.
  int chunk = M <= 128 ? M : 128;
  if (M > 128 && ((N + kTileN - 1) / kTileN) * 2 <= device_info().sms) chunk = 96;
  for (int m0 = 0; m0 < M; m0 += chunk) {
    const int mc = (M - m0) < chunk ? (M - m0) : chunk;
    const char* xc = static_cast<const char*>(x) + static_cast<long long>(m0) * ldx * 2;
    char* oc = static_cast<char*>(out) + static_cast<long long>(m0) * ldo * 2;
    int rc;
    if (aligned && gemm_tc_supported(mc, N, K, group_size, bits)) {
      rc = launch(xc, oc, mc);
    } else {
      rc = bits == 4 ? launch_simt<4>(xc, ldx, qweight, scales, zeros, bias, oc, ldo, mc, N, K,
                                      group_size, opts, stream)
                     : launch_simt<8>(xc, ldx, qweight, scales, zeros, bias, oc, ldo, mc, N, K,
                                      group_size, opts, stream);
    }
    if (rc != DXB_OK) return rc;
  }
  return DXB_OK;
}

}  // namespace dx

// =================================================================== C ABI ==
extern "C" {

#ifdef DXB_TRACE
void dxb_debug_set_trace(void* ptr) { dx::g_trace = static_cast<long long*>(ptr); }
#endif

int dxb_wq_gemm_ex(int bits, const void* x, int64_t ldx, const void* qweight, const void* scales,
                   const void* zeros, const void* bias, void* out, int64_t ldo, int M, int N, int K,
                   int group_size, void* workspace, size_t workspace_bytes, const dxb_gemm_opts* opts,
                   void* cuda_stream) {
  using namespace dx;
  int rc = check_args(bits, x, ldx, qweight, scales, out, ldo, M, N, K, group_size);
  if (rc != DXB_OK) return rc;
  Opts o;
  rc = read_opts(opts, bits, M, N, K, &o);
  if (rc != DXB_OK) return rc;
  if (M == 0) return DXB_OK;
  return gemm_dispatch(bits, x, ldx, qweight, scales, zeros, bias, out, ldo, M, N, K, group_size, workspace,
                       workspace_bytes, o, static_cast<cudaStream_t>(cuda_stream));
}

int dxb_wq_gemm_group(int bits, const dxb_group_item* items, int count, int M, int K, int group_size, void* workspace,
                      size_t workspace_bytes, const dxb_gemm_opts* opts, void* cuda_stream) {
  using namespace dx;
  if (items == nullptr) return DXB_ERR_NULL;
  if (count < 1 || count > kMaxGroup) return DXB_ERR_UNSUPPORTED;
  Opts o;
  bool together = M >= 1 && M <= 128;
  for (int i = 0; i < count; ++i) {
    const dxb_group_item& it = items[i];
    int rc = check_args(bits, it.x, it.ldx, it.qweight, it.scales, it.out, it.ldo, M, it.n, K, group_size);
    if (rc != DXB_OK) return rc;
    rc = read_opts(opts, bits, M, it.n, K, &o);
    if (rc != DXB_OK) return rc;
    together = together && gemm_tc_supported(M, it.n, K, group_size, bits) &&
               pointers_aligned(bits, it.x, it.ldx, it.qweight, it.scales, it.zeros, it.bias, it.out, it.ldo, K) &&
               (it.zeros == nullptr) == (items[0].zeros == nullptr);
  }
  if (!together || o.max_ctas > 0 || o.peer.world > 1) return DXB_ERR_UNSUPPORTED;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  const bool zeros = items[0].zeros != nullptr;
  if (bits == 4)
    return zeros ? launch_group<4, true>(items, count, M, K, group_size, workspace, workspace_bytes, o, stream)
                 : launch_group<4, false>(items, count, M, K, group_size, workspace, workspace_bytes, o, stream);
  return zeros ? launch_group<8, true>(items, count, M, K, group_size, workspace, workspace_bytes, o, stream)
               : launch_group<8, false>(items, count, M, K, group_size, workspace, workspace_bytes, o, stream);
}

int dxb_wq_gemm(int bits, const void* x, int64_t ldx, const void* qweight, const void* scales,
                const void* zeros, const void* bias, void* out, int64_t ldo, int M, int N, int K,
                int group_size, void* workspace, size_t workspace_bytes, int max_ctas,
                void* cuda_stream) {
  dxb_gemm_opts o = {};
  o.max_ctas = max_ctas;
  return dxb_wq_gemm_ex(bits, x, ldx, qweight, scales, zeros, bias, out, ldo, M, N, K, group_size, workspace,
                        workspace_bytes, &o, cuda_stream);
}

// ---------------------------------------------------------------------------
// Scratch that lives inside the library image, for callers that must not
// allocate device memory (see dxb_wq_gemm_static in the header).  Zero at load
// time; every GPU that loads the library keeps these 24 MiB until the process
// exits.  In host code the symbol below is only a stand-in: its device address
// has to be asked for with cudaGetSymbolAddress, per device.
constexpr size_t kStaticScratchBytes = static_cast<size_t>(24) << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// A status word (and counters that nobody uses) for launches that have no scratch, see dxb_shared_workspace.
static __device__ __align__(256) unsigned char g_shared_workspace[dx::kStatusBytes + dx::kMaxTiles * 4];

namespace dx {
constexpr int kMaxDevices = 64;
struct SymbolAddress {
  std::mutex mu;
  void* addr[kMaxDevices] = {};
};
// Device address of a symbol of this library on the CURRENT device, looked up once per device.
static int symbol_address(SymbolAddress& known, const void* symbol, void** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return DXB_ERR_CUDA;
  std::lock_guard<std::mutex> lock(known.mu);
  if (known.addr[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, symbol) != cudaSuccess || p == nullptr) {
      cudaGetLastError();  // clear the sticky-less error so later calls start clean
      return DXB_ERR_CUDA;
    }
    known.addr[dev] = p;
  }
  *out = known.addr[dev];
  return DXB_OK;
}
static int static_scratch_address(void** out) {
  static SymbolAddress known;
  return symbol_address(known, g_static_scratch, out);
}
}  // namespace dx

int dxb_wq_gemm_static(int bits, const void* x, int64_t ldx, const void* qweight,
                       const void* scales, const void* zeros, const void* bias, void* out,
                       int64_t ldo, int M, int N, int K, int group_size, void* cuda_stream) {
  using namespace dx;
  int rc = check_args(bits, x, ldx, qweight, scales, out, ldo, M, N, K, group_size);
  if (rc != DXB_OK) return rc;
  if (M == 0) return DXB_OK;
  // What one launch of at most 128 tokens needs; with more tokens dxb_wq_gemm takes the
  // one-launch plan when the array holds it and goes block by block otherwise.  Shapes that
  // run on the plain CUDA-core kernel use no scratch at all.
  const int mc = M <= 128 ? M : 128;
  if (pointers_aligned(bits, x, ldx, qweight, scales, zeros, bias, out, ldo, K) &&
      gemm_tc_supported(mc, N, K, group_size, bits) &&
      (plan_workspace_bytes(mc, N, K, bits, 0) > kStaticScratchBytes ||
       (M > 128 && plan_workspace_bytes(96, N, K, bits, 0) > kStaticScratchBytes)))
    return DXB_ERR_SCRATCH_LIMIT;
  void* scratch = nullptr;
  rc = static_scratch_address(&scratch);
  if (rc != DXB_OK) return rc;
  // The array keeps whatever the previous call left.  Partial sums are always written
  // before they are read, but the tile counters must start at zero.  The status word in
  // front of them is left alone: a timeout reported by an earlier call stays readable
  // (dxb_read_status(NULL, stream)) until it has been read.
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  if (cudaMemsetAsync(static_cast<unsigned char*>(scratch) + kStatusBytes, 0, counters_bytes(0), stream) !=
      cudaSuccess)
    return DXB_ERR_CUDA;
  return dxb_wq_gemm(bits, x, ldx, qweight, scales, zeros, bias, out, ldo, M, N, K, group_size,
                     scratch, kStaticScratchBytes, 0, cuda_stream);
}

int dxb_w4a16(const void* x, int64_t ldx, const void* qweight, const void* scales,
              const void* zeros, const void* bias, void* out, int64_t ldo, int M, int N, int K,
              int group_size, void* workspace, size_t workspace_bytes, void* cuda_stream) {
  return dxb_wq_gemm(4, x, ldx, qweight, scales, zeros, bias, out, ldo, M, N, K, group_size,
                     workspace, workspace_bytes, 0, cuda_stream);
}

int dxb_w8a16(const void* x, int64_t ldx, const void* qweight, const void* scales,
              const void* zeros, const void* bias, void* out, int64_t ldo, int M, int N, int K,
              int group_size, void* workspace, size_t workspace_bytes, void* cuda_stream) {
  return dxb_wq_gemm(8, x, ldx, qweight, scales, zeros, bias, out, ldo, M, N, K, group_size,
                     workspace, workspace_bytes, 0, cuda_stream);
}

size_t dxb_workspace_bytes_ex(int M, int N, int K, int bits, int max_ctas) {
  using namespace dx;
  if (M <= 0 || N <= 0 || K <= 0 || (bits != 4 && bits != 8)) return kStatusBytes;
  const int rows = bits == 4 ? K / 2 : K;
  if (rows < (bits == 4 ? 64 : 128)) return kStatusBytes;
  // Up to 128 tokens: that launch.  More: the larger of the one-launch plan over all token
  // blocks and the plan of a single block (used when the caller's workspace is smaller).
  size_t one_block = plan_workspace_bytes(M <= 128 ? M : 128, N, K, bits, max_ctas);
  if (M <= 128) return one_block;
  // block by block, few-tile weights go in blocks of 96 tokens (see dxb_wq_gemm)
  const size_t block96 = plan_workspace_bytes(96, N, K, bits, max_ctas);
  if (block96 > one_block) one_block = block96;
  if (static_cast<long long>((N + kTileN - 1) / kTileN) * ((M + 127) / 128) > kMaxTiles)
    return one_block;
  size_t all_blocks = plan_workspace_bytes(M, N, K, bits, max_ctas);
  // CTA pairs that split K park partial sums too; with less they do not split.
  const int sms = device_info().sms > 0 ? device_info().sms : 148;
  const int budget = (max_ctas > 0 && max_ctas < sms) ? max_ctas : sms;
  const PairChoice choice = choose_pairs(make_plan(M, N, K, bits, sms, max_ctas), M, N, K, bits, budget / 2, budget, true);
  if (choice.split > 1) {
    const Plan pp = make_pair_plan(M, N, K, bits, budget / 2, choice.blocks);
    const size_t split = kStatusBytes + counters_bytes(0) + pair_split_bytes(pp, choice.split);
    if (split > all_blocks) all_blocks = split;
  }
  return all_blocks > one_block ? all_blocks : one_block;
}

size_t dxb_workspace_bytes(int M, int N, int K, int bits) { return dxb_workspace_bytes_ex(M, N, K, bits, 0); }

size_t dxb_scratch_bytes(int M, int N, int K, int bits, int max_ctas) {
  using namespace dx;
  if (M <= 0 || N <= 0 || K <= 0 || (bits != 4 && bits != 8)) return 0;
  if ((bits == 4 ? K / 2 : K) < (bits == 4 ? 64 : 128)) return 0;
  const long long tiles = static_cast<long long>((N + kTileN - 1) / kTileN) * ((M + 127) / 128);
  if (tiles <= kMaxTiles) return launch_scratch_bytes(M, N, K, bits, max_ctas);
  const size_t a = launch_scratch_bytes(128, N, K, bits, max_ctas), b = launch_scratch_bytes(96, N, K, bits, max_ctas);
  return a > b ? a : b;  // block by block
}

int dxb_workspace_init(void* workspace, size_t workspace_bytes, void* status, void* cuda_stream) {
  using namespace dx;
  const size_t bytes = kStatusBytes + counters_bytes(0);
  if (!workspace) return DXB_ERR_NULL;
  if (workspace_bytes < bytes) return DXB_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(workspace) % 16 || reinterpret_cast<uintptr_t>(status) % 4) return DXB_ERR_UNSUPPORTED;
  const int vecs = static_cast<int>(bytes / 16);
  wq_workspace_init_kernel<<<(vecs + 255) / 256, 256, 0, static_cast<cudaStream_t>(cuda_stream)>>>(
      static_cast<uint4*>(workspace), vecs, static_cast<int*>(status));
  return cudaGetLastError() == cudaSuccess ? DXB_OK : DXB_ERR_CUDA;
}

int dxb_shared_workspace(void** workspace) {
  if (!workspace) return DXB_ERR_NULL;
  static dx::SymbolAddress known;
  // The first look-up on a device may load code there, which is refused while a stream is captured in the
  // usual mode, unless the thread is in this one.
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) { cudaGetLastError(); return DXB_ERR_CUDA; }
  const int rc = dx::symbol_address(known, g_shared_workspace, workspace);
  cudaThreadExchangeStreamCaptureMode(&mode);
  return rc;
}

int dxb_event_done(void* cuda_event) {
  // A query is refused while any stream is captured in the usual mode, unless its thread is in this one.
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) { cudaGetLastError(); return 0; }
  const cudaError_t rc = cudaEventQuery(static_cast<cudaEvent_t>(cuda_event));
  if (rc != cudaSuccess) cudaGetLastError();
  cudaThreadExchangeStreamCaptureMode(&mode);
  return rc == cudaSuccess ? 1 : 0;
}

unsigned long long dxb_capture_id(void* cuda_stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(static_cast<cudaStream_t>(cuda_stream), &status, &id) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return status == cudaStreamCaptureStatusNone ? 0 : id + 1;
}

int dxb_relayout_w4(const void* qweight, void* out, int K, int N, int inverse, void* cuda_stream) {
  using namespace dx;
  if (!qweight || !out) return DXB_ERR_NULL;
  if (K <= 0 || N <= 0 || K % 4 || N % 4) return DXB_ERR_SHAPE;  // whole row pairs, whole 32-bit words
  if (reinterpret_cast<uintptr_t>(qweight) % 4 || reinterpret_cast<uintptr_t>(out) % 4) return DXB_ERR_UNSUPPORTED;
  const long long row_pairs = K / 4;
  const int n4 = N / 4;
  const long long total = row_pairs * n4;
  const int block = 256;
  wq_relayout_w4_kernel<<<static_cast<unsigned>((total + block - 1) / block), block, 0,
                          static_cast<cudaStream_t>(cuda_stream)>>>(
      static_cast<const uint32_t*>(qweight), static_cast<uint32_t*>(out), row_pairs, n4, inverse ? 1 : 0);
  return cudaGetLastError() == cudaSuccess ? DXB_OK : DXB_ERR_CUDA;
}

size_t dxb_fused_reduce_bytes(int world, int64_t capacity_elems) {
  if (world < 1 || world > dx::kPeerMaxRanks || capacity_elems <= 0) return 0;
  const size_t cap = (static_cast<size_t>(capacity_elems) + 7) / 8 * 8;
  return dx::kFusedHeaderBytes + 2 * static_cast<size_t>(world) * cap * 2;
}

void dxb_set_wait_limit_ms(int ms) {
  const long long tries = static_cast<long long>(ms < 1 ? 1 : ms) * 4000;
  dx::g_wait_tries.store(static_cast<unsigned>(tries > 4000000000ll ? 4000000000ll : tries));
}

int dxb_uses_tensor_cores(int M, int N, int K, int group_size, int bits) {
  const int mc = M <= 128 ? M : 128;
  return dx::gemm_tc_supported(mc, N, K, group_size, bits) ? 1 : 0;
}

int dxb_read_status(void* workspace, void* cuda_stream) {
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  const bool builtin = workspace == nullptr;  // the scratch of dxb_wq_gemm_static
  if (builtin && dx::static_scratch_address(&workspace) != DXB_OK) return DXB_ERR_CUDA;
  int code = 0;
  if (cudaMemcpyAsync(&code, workspace, sizeof(int), cudaMemcpyDeviceToHost, stream) != cudaSuccess)
    return DXB_ERR_CUDA;
  // The built-in scratch has no owner who could clear its status word: reading it does.
  if (builtin && cudaMemsetAsync(workspace, 0, sizeof(int), stream) != cudaSuccess) return DXB_ERR_CUDA;
  if (cudaStreamSynchronize(stream) != cudaSuccess) return DXB_ERR_CUDA;
  return code;
}

const char* dxb_strerror(int code) {
  switch (code) {
    case DXB_OK: return "ok";
    case DXB_ERR_BITS: return "bits must be 4 or 8";
    case DXB_ERR_NULL: return "null pointer argument";
    case DXB_ERR_SHAPE: return "inconsistent shape, stride or group size";
    case DXB_ERR_UNSUPPORTED: return "shape or option not supported by this build";
    case DXB_ERR_WORKSPACE: return "workspace missing or too small (see dxb_workspace_bytes)";
    case DXB_ERR_TENSORMAP: return "could not encode a TMA tensor map";
    case DXB_ERR_CUDA: return "CUDA launch or runtime error";
    case DXB_ERR_KERNEL_TIMEOUT: return "a bounded wait inside the kernel ran out";
    case DXB_ERR_SCRATCH_LIMIT:
      return "problem needs more scratch than the 24 MiB built into the library "
             "(use dxb_wq_gemm with a caller-provided workspace)";
    default: return "unknown error";
  }
}

}  // extern "C"

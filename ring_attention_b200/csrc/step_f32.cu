// Blackwell (sm_100a) ring step for fp32 Q/K/V on the tensor cores: the same FlashAttention-style
// forward as step_tc.cu (TMA, tcgen05.mma, tensor memory) with every operand split into two fp16
// terms of a scaled value, x * 2^e ~ hi + lo (hi = fp16(x * 2^e), lo = fp16(x * 2^e - hi)), and
// every product taken as hi*hi + lo*hi + hi*lo with fp32 accumulation. Replaces the reference's
// fp32 step (src/attention_step.cu:114-282) for head_dim 32, 64 and 128.
//
// Precision. hi + lo carry 22 bits like a pair of TF32 terms, and kind::f16 runs at twice the rate
// of kind::tf32 with half the operand bytes and half the accumulations per product. What fp16
// lacks is range, so values are scaled by powers of two first (exact): Q by row, K by key, V by
// key tile, each so that the largest magnitude sits in [2^14, 2^15), and P by row and tile (see the unit
// of O in the softmax). An element keeps 22 bits down to 2^-17 of that largest one and an absolute 2^-40
// of it below; P keeps them down to 2^-11 of its largest and an absolute 2^-33. The row sums stay
// fp32. The dropped lo*lo and the rounding of lo are about 2^-22 of a product; what shows in the
// output is the tensor core's fp32 accumulation over the key tiles, as in any such kernel.
// Where the shared scales do not hold what single elements need, a tile is marked and taken in plain
// fp32 by the softmax threads: V tiles with a key or a column far below the tile's largest value, and
// tiles whose products with Q span too much (kKeyRange, kColRange, kScoreRange). B1 H4 S16384 D128 causal:
// 20 us for one marked tile in each head, 6.6 ms when a column of V lies 2^20 above the others (every
// tile), 28 ms when a channel of Q lies 2^24 above and that of K 2^24 below the others (2.6 ms each on
// TF32 pairs, which need no marks).
// RA_STEP_FORCE_SIMT selects the plain-fp32 kernel; head_dim 256 keeps it (its split Q tiles and key
// ring exceed shared memory).
//
// Work decomposition: grid = (batch * heads, 256-row query blocks), heavy blocks first; a block
// owns two 128-row query tiles and walks the visible 64-key tiles of every key segment. Calls with
// few query blocks cut the tile list over the blocks of a cluster (pick_key_split).
//
// Roles inside a block (640 threads)
//   warp 0        TMA producer: K_0, V_0, K_1, ... as 128B-swizzled fp32 tiles into a shared-memory
//                 ring (no multicast).
//   warps 1, 2    MMA issuers, one per query tile, at head_dim 128 warp 1 for both in turn (converged
//                 warp, one elected lane).
//   warps 4-11    softmax, one thread per row, a warpgroup per query tile. At the start each thread
//                 reads, scales and splits its row of Q into tensor memory, where the A operand
//                 costs the scores no shared-memory reads, which bound them otherwise (head_dim
//                 128: the hi term; lo goes as swizzled tiles into shared memory).
//   warps 12-19   splitters: a landed raw tile is read into registers, scaled, split and written
//                 back over itself, the hi tiles over the even 32-column boxes and the lo tiles over
//                 the odd ones, in the layout TMA would give 16-bit data. They also find the range of
//                 every tile; a marked V tile stays as it landed.
//   With a workspace, long calls split K and V once ahead (split_kv_kernel): no splitters, 384 threads.
//   Head_dim 32 / 64: S and P have buffers of their own, so the scores of tile t+1 are computed
//   while the softmax of tile t runs. Head_dim 128: P is written over S and the two query tiles take
//   turns on the tensor core.
//
// Tensor memory, 256 columns per query tile: S [0,64) P hi [64,96) P lo [96,128) O [128,192) Q hi
// [192,224) Q lo [224,256); head_dim 128: S and P [0,64) O [64,192) Q hi [192,256).
// What bounds it: at head_dim 128 the issue of the MMAs. A pair of tiles of 64 keys needs 3330 clocks of the tensor core, in 72
// instructions of 32 to 64; its queue holds a few of them, so whatever the issuing warp does between two batches is
// time in which the tensor core is idle (P is always written when the warp comes to it). A satisfied wait costs it 100 to
// 150 clocks, a sum of 64 bits in a descriptor half as much as an instruction. us, B1 H4 S16384 D128 causal: 824; descriptors
// as 32-bit words 781; without a wait for V and with one for K 740; K and V split ahead 719; a warp for each query tile then
// 686 (CUDA graphs). At head_dim 64 it is the softmax (hi and lo of P beside the exponentials). Against one 128-row tile per block on
// TF32 pairs: B1 H8 S1024 D64 dense 20.6 (37), H4/kvH1 8231 x 9075 rows D64 causal 161 (272).
//
// Every wait on an mbarrier is bounded (see tc_common.cuh); a wait that runs out reports into
// the device status word and the block unwinds.
#include <algorithm>
#include <atomic>

#include "tc_common.cuh"

namespace rab {

using namespace tcgen;

namespace {

constexpr int kBNf = 64;          // keys per tile
constexpr int kThreadsF = 640;
constexpr int kSplitThreads = 256;
constexpr int kTopExp = 14;       // scaled values have their largest magnitude in [2^14, 2^15)
constexpr int kPBits = 8;         // the largest P of a tile that sets a row's unit is 2^8
constexpr int kNoUnit = 1 << 20;  // nothing in O yet, or (as a tile's exponent) nothing but zeros in V
constexpr int kOTop = 116;        // O may be scaled up to 2^116
constexpr int kMinPExp = -60;     // (a P below 2^-25 adds nothing)
constexpr float kPSumLimit = 65000.f;  // of eight P: none of them then leaves fp16's range
// A V tile is wide if the largest value of some key (not all zeros) is below 2^-kKeyRange of the tile's, or
// that of some column among a splitter warp's eight keys below 2^-kColRange: what its elements lose
// below 2^-40 of the tile's largest (and P below 2^-33) could then show in a row or a column.
constexpr int kKeyRange = 9, kColRange = 16;
// The scores of a query block and a key tile whose largest magnitudes multiply to 2^kScoreRange or more are
// taken in plain fp32: what the terms lose (2^-40 of a row's or a key's largest element each) could
// reach 2^-20 in a score.
constexpr int kScoreRange = 17;
// A tile as v_exp holds it: V's exponent + kExpBias, or kNoUnit, or kWide with or without kPlain.
constexpr int kExpBias = 512, kWide = 1 << 12, kPlain = 1 << 13;

// What the softmax needs to know of a key tile besides its split K and V, as the form with split operands keeps it in
// the workspace and copies it with the tile: factors of the keys, exponents of V's keys, the V tile's as v_exp holds it,
// and the exponent of the largest magnitude of K.
constexpr int kMetaG = 0, kMetaVKey = kBNf * 4, kMetaVExp = kMetaVKey + kBNf, kMetaKTop = kMetaVExp + 4, kMetaBytes = 384;
// The split operands of a call in its workspace, by KV head (as the tensor map counts them) and tile.
struct SplitKV {
  unsigned char *k, *v, *meta;
  int tiles;               // of all key segments of a head
  int beg[RA_MAX_SEG];     // first tile of a segment
};

template <int DR, bool kSplit, bool kPre = false>
struct F32Cfg {
  static constexpr int kThreads = kPre ? 384 : kThreadsF;
  static constexpr int kTiles = 2;
  static constexpr int D = DR < 64 ? 64 : DR;           // columns of a split tile row
  // Where Q's terms go. Head_dim 32 / 64: both into tensor memory, beside S, P and O. Head_dim 128:
  // hi into tensor memory, lo as swizzled tiles into shared memory; P is then written over S, and
  // the 64 KB that Q's hi tiles do not take make the ring 5 slots instead of 3. (With Q all in
  // shared memory and P beside S, B1 H4 S16384 causal took 1032 us: every K tile waited for the
  // slot that P.V of the tile before last frees.)
  static constexpr bool kQLoInTmem = D == 64;
  static constexpr bool kAlias = D == 128;
  // There one warp issues for both query tiles in turn, or, where no splitters take issue slots, a warp for each (B1 H4
  // S16384 D128 causal: 686 against 719 with split operands, 770 against 740 us without).
  static constexpr bool kTurns = kAlias && kPre;
  static constexpr bool kOneIssuer = kAlias && !kTurns;
  static constexpr int kBoxes = DR / 32;                // raw boxes: 32 fp32 = 128 bytes of a row
  static constexpr int kGroups = D / 64;                // 64-column groups of a split tile
  static constexpr int kBoxBytes = kBNf * 128;
  static constexpr int kSlotBytes = 2 * kGroups * kBoxBytes;  // raw tile = hi + lo tiles
  static constexpr int kRawBytes = kBoxes * kBoxBytes;
  // (eight slots leave room for the staged rows without taking L1 from the second read of Q: with ten a call with
  // one key tile at head_dim 64 took 16.4 us, with eight 14.7)
  static constexpr int kStages = D == 128 ? (kSplit ? 4 : 5) : (kSplit ? 10 : 8);
  // per-key factors of K are read by the softmax of their tile while later tiles are split; the
  // ring holds the producer back far enough for this many copies
  static constexpr int kGDepth = D == 128 ? 4 : 8;
  static_assert(kGDepth > kStages / 2, "a key factor could be overwritten before it is read");
  static constexpr int kQBytes = kQLoInTmem ? 0 : kBM * D * 2;  // lo of one query tile
  static constexpr int kOffQ = 0;
  static constexpr int kOffKV = kTiles * kQBytes;
  static constexpr int kOffBar = kOffKV + kStages * kSlotBytes;
  static constexpr int kNumBars = 2 + 3 * kStages + 8 + 3;
  static constexpr int kOffSlot = kOffBar + kNumBars * 8;      // tensor-memory address, abort flag
  static constexpr int kOffRed = (kOffSlot + 8 + 15) & ~15;    // [2][2][8] range of a V tile by warp
  static constexpr int kOffVExp = kOffRed + 128;               // [16] exponents of V tiles
  static constexpr int kOffG = (kOffVExp + 64 + 15) & ~15;     // [kGDepth][kBNf] factors of K
  static constexpr int kOffVKey = kOffG + kGDepth * (kPre ? kMetaBytes : kBNf * 4);  // [8][kBNf] exponents of V's keys
  static constexpr int kOffQTop = kOffVKey + (kPre ? 0 : 8 * kBNf);  // [2][4] exponents of Q by softmax warp
  static constexpr int kOffMl = kOffQTop + 32;
  static constexpr int kMlBytes = kSplit ? kTiles * kBM * 8 : 0;
  // where the unsplit form stages its rows (see RowStore): over Q's lo tiles, else in a place of their own
  static constexpr int kRowStage = 4 * RowStore<DR>::kStageBytes;  // of a query tile
  static constexpr bool kOwnStage = !kSplit && kQBytes < kRowStage;
  static constexpr int kOffStage = kOwnStage ? (kOffMl + 15) & ~15 : kOffQ;
  static constexpr int kSmemBytes = kOwnStage ? kOffStage + kTiles * kRowStage : kOffMl + kMlBytes;
  // Registers of a thread of the producer / issuing, the softmax and the splitting warps; 640 threads start with 96
  // each, 61440 in all. Head_dim 128 spills 60 bytes so and 128 with 40 / 144 / 72: us per call B1 H4 S16384 causal 828 /
  // 848. The others spill next to nothing either way and gain from registers for the splitters: H8 S8192 D64 242 (247 with
  // the split of head_dim 128), H16/kvH8 978 rows on 5874 keys D32 93.8 (97.0).
  static constexpr int kRegsIssue = kPre ? 72 : D == 128 ? 64 : 40, kRegsSoftmax = kPre ? 216 : D == 128 ? 152 : 144,
                       kRegsSplit = kPre ? 0 : D == 128 ? 56 : 72;
  static_assert(128 * kRegsIssue + 256 * kRegsSoftmax + 256 * kRegsSplit <= (kPre ? 384 * 168 : 640 * 96), "setmaxnreg draws on the launch's registers");
  static constexpr int kColS = 0, kColP = kAlias ? 0 : 64, kColO = kAlias ? 64 : 128, kColQ = 192;
  static_assert(kSmemBytes <= 232448, "shared memory budget");
  static_assert(kTiles * kBM * ((DR + 4) * 4 + 8) <= kOffBar, "staging of the key-split merge");
};

// The power-of-two exponent that brings a largest magnitude (as its bits) to [2^14, 2^15); an
// infinity or a NaN counts as nothing (it stays what it is under any scale), zero gives zero.
// At least -113, at most `limit`. The limits keep the scale and its inverse normal numbers: below 2^-106
// (K: 2^-98) values lose bits gradually.
__device__ inline int scale_exp(unsigned max_bits, int limit) {
  return max_bits == 0 ? 0 : min(kTopExp + 127 - static_cast<int>(max_bits >> 23), limit);
}
constexpr int kMaxExp = 120;
// A score is scaled back in two steps, by 2^-(exponent of the key + kBias) and by 2^-(exponent of the row
// - kBias): neither factor nor the value between them leaves fp32 where the score does not, unless
// magnitudes of Q or K exceed 2^118.
constexpr int kBias = 14, kMaxExpK = 126 - kBias;
__device__ inline unsigned finite_abs_bits(float x) {
  const unsigned u = __float_as_uint(x) & 0x7fffffffu;
  return u < 0x7f800000u ? u : 0u;
}
__device__ inline float pow2i(int e) { return __int_as_float((e + 127) << 23); }  // -126 <= e <= 127
__device__ inline float pow2_any(int e) {                                          // -149 <= e <= 127
  return e >= -126 ? pow2i(e) : __int_as_float(1 << (e + 149));
}
// Two scaled values as packed hi and lo fp16 pairs.
__device__ inline void split_pair(float x0, float x1, unsigned& hi, unsigned& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 f = __half22float2(h);
  const __half2 r = __floats2half2_rn(x0 - f.x, x1 - f.y);
  hi = *reinterpret_cast<const unsigned*>(&h);
  lo = *reinterpret_cast<const unsigned*>(&r);
}
__device__ inline float2 fmul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return d;
}
__device__ inline unsigned ld_shared_u1(unsigned addr) {
  unsigned v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ inline uint4 ld_shared_u4(unsigned addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ inline float4 ld_shared_f4(unsigned addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}
__device__ inline void st_shared_u4(unsigned addr, unsigned a, unsigned b, unsigned c, unsigned d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}

// The range of a splitter warp's eight rows of V (x: this lane's pieces of one of them, mx: the largest magnitude
// among them, out: of all eight rows): returns what their tile's largest must not exceed, as the upper half of
// its bits, or the tile is wide. Also writes the exponents of the keys. The smallest nonzero maximum of a key and of
// a column count. No column lies below the warp's smallest element, which is near enough for most tiles.
template <int kUnits>
__device__ inline unsigned v_range(const float (&x)[kUnits][8], unsigned& mx, int lane, unsigned char* v_key) {
  const int r8 = lane & 7, p4 = lane >> 3;
  float fn = fabsf(x[0][0]);
#pragma unroll
  for (int u = 0; u < kUnits; ++u)
#pragma unroll
    for (int i = 0; i < 8; i += 2) fn = min3(fn, fabsf(x[u][i]), fabsf(x[u][i + 1]));
  mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
  mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
  if (p4 == 0) v_key[r8] = static_cast<unsigned char>(mx >> 23);
  unsigned low = (mx == 0 ? 0xffffu : mx >> 16) + (kKeyRange << 7);
  const unsigned least = __reduce_min_sync(0xffffffffu, __float_as_uint(fn)) >> 16;
  mx = __reduce_max_sync(0xffffffffu, mx);
  // (a zero says nothing: the rows behind a ragged end are zeros)
  if (__builtin_expect(least > 0 && least + ((kColRange - 1) << 7) >= mx >> 16, 1)) {
    low = min(low, least + (kColRange << 7));
  } else {
    // column by column, the upper halves of two magnitudes in a word; each lane ends with its
    // share of the columns (1 below, so that none is zero)
    unsigned c2[4 * kUnits];
#pragma unroll
    for (int i = 0; i < 4 * kUnits; ++i)
      c2[i] = __byte_perm(__float_as_uint(x[i / 4][2 * (i & 3)]), __float_as_uint(x[i / 4][2 * (i & 3) + 1]),
                          0x7632) & 0x7fff7fffu;
#pragma unroll
    for (int step = 0; step < 3; ++step) {
      const bool odd = (lane >> step) & 1;
      const int n = (4 * kUnits) >> (step + 1);
      if (n > 0) {
#pragma unroll
        for (int i = 0; i < 2 * kUnits; ++i)
          if (i < n)
            c2[i] = __vmaxu2(odd ? c2[i + n] : c2[i],
                             __shfl_xor_sync(0xffffffffu, odd ? c2[i] : c2[i + n], 1 << step));
      } else {
        c2[0] = __vmaxu2(c2[0], __shfl_xor_sync(0xffffffffu, c2[0], 1 << step));
      }
    }
    unsigned low2 = __vsub2(c2[0], 0x00010001u);
    if constexpr (kUnits == 4) low2 = __vminu2(low2, __vsub2(c2[1], 0x00010001u));
    low = min(low, min(low2 & 0xffffu, low2 >> 16) + (kColRange << 7));
  }
  return __reduce_min_sync(0xffffffffu, low);
}

template <int DR, bool kSplit, bool kPre>
__global__ void __launch_bounds__((F32Cfg<DR, kSplit, kPre>::kThreads), 1)
    step_f32_kernel(const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const float* q_g,
                    const float* k_g, long long kv_head_stride, const TcArgs a, const __grid_constant__ SplitKV pre) {
  using C = F32Cfg<DR, kSplit, kPre>;
  extern __shared__ __align__(1024) unsigned char smem[];  // 128B-swizzled tiles
  const unsigned s_base = smem_u32(smem);
  const unsigned s_q = s_base + C::kOffQ;
  const unsigned s_kv = s_base + C::kOffKV;
  const unsigned s_bar = s_base + C::kOffBar;
  const unsigned bar_q_full = s_bar;                             // [2] Q split
  const unsigned bar_kv_raw = s_bar + 16;                        // [kStages] TMA bytes
  const unsigned bar_kv_full = bar_kv_raw + 8 * C::kStages;      // [kStages] split
  const unsigned bar_kv_empty = bar_kv_full + 8 * C::kStages;    // [kStages] MMAs done
  const unsigned bar_s_full = bar_kv_empty + 8 * C::kStages;     // [2]
  const unsigned bar_s_free = bar_s_full + 16;                   // [2] S held in registers
  const unsigned bar_p_full = bar_s_free + 16;                   // [2]
  const unsigned bar_o_done = bar_p_full + 16;                   // [2] P.V done
  const unsigned bar_v_max = bar_o_done + 16;                    // a V tile's maxima by warp written
  const unsigned bar_turn = bar_v_max + 8;                       // [2] the MMAs of this query tile may go out
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(smem + C::kOffSlot);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile unsigned* red = reinterpret_cast<volatile unsigned*>(smem + C::kOffRed);
  volatile int* v_exp = reinterpret_cast<volatile int*>(smem + C::kOffVExp);
  volatile int* q_tops = reinterpret_cast<volatile int*>(smem + C::kOffQTop);

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  unsigned cta_rank = 0;
  if constexpr (kSplit) cta_rank = cluster_ctarank();

  const int gone = tid == 0 ? *reinterpret_cast<volatile int*>(a.status) : 0;
  let_next_start();

  const bool causal = (a.flags & RA_STEP_CAUSAL) != 0;
  const bool fresh = (a.flags & RA_STEP_FRESH) != 0;
  const bool finalize = (a.flags & RA_STEP_FINALIZE) != 0;

  const int bh = kSplit ? static_cast<int>(blockIdx.x) / a.key_split : static_cast<int>(blockIdx.x);
  const int qb_lin = static_cast<int>(gridDim.y) - 1 - static_cast<int>(blockIdx.y);
  const int sq = qb_lin / a.n_qblocks_per_seg;
  const int tq = qb_lin - sq * a.n_qblocks_per_seg;
  const int h = bh % a.H;
  const int b = bh / a.H;
  const int kv_bh = b * a.kvH + (h % a.kvH);
  const int q_seg_len = a.qmap.seg_len;
  constexpr int kQBlock = C::kTiles * kBM;
  const int row0 = tq * kQBlock;
  const int rows_in_block = min(kQBlock, q_seg_len - row0);
  const int qmin = a.qmap.base[sq] + row0 * a.stride;
  const int qmax = a.qmap.base[sq] + (row0 + rows_in_block - 1) * a.stride;
  const int live = rows_in_block > kBM ? 2 : 1;  // query tiles that hold a row

  int n_tiles = 0;
  for (int sk = 0; sk < a.kmap.n_seg; ++sk) {
    const TileRange r = tile_range<kBNf>(a.kmap, sk, a.stride, causal, a.doc_len, qmin, qmax);
    n_tiles += r.hi - r.lo;
  }
  if (n_tiles == 0) {  // (the blocks of a cluster agree)
    wait_for_previous();
    rows_without_keys<DR>(a, static_cast<size_t>(bh) * a.Sq + static_cast<size_t>(sq) * q_seg_len + row0, rows_in_block,
                          kSplit ? cta_rank : 0, kSplit ? a.key_split : 1, fresh, finalize);
    return;
  }
  int share_beg = 0, share_end = n_tiles;
  if constexpr (kSplit) {
    share_beg = static_cast<int>(static_cast<long long>(n_tiles) * cta_rank / a.key_split);
    share_end = static_cast<int>(static_cast<long long>(n_tiles) * (cta_rank + 1) / a.key_split);
    n_tiles = share_end - share_beg;
  }

  if (tid == 0) {
    for (int w = 0; w < 2; ++w) {
      mbar_init(bar_q_full + 8 * w, kBM);
      mbar_init(bar_s_full + 8 * w, 1);
      mbar_init(bar_s_free + 8 * w, kBM);
      mbar_init(bar_p_full + 8 * w, kBM);
      mbar_init(bar_o_done + 8 * w, 1);
      mbar_init(bar_turn + 8 * w, 1);
    }
    mbar_init(bar_v_max, kSplitThreads / 32);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(bar_kv_raw + 8 * s, 1);
      mbar_init(bar_kv_full + 8 * s, kPre ? 1 : kSplitThreads);
      mbar_init(bar_kv_empty + 8 * s, C::kOneIssuer ? 1 : live);  // (a commit is about its own thread's MMAs)
    }
    *abort_flag = gone != 0;
    if (s_base & 1023u) {  // the swizzle of TMA and the descriptors below count on it
      *abort_flag = 1;
      atomicCAS(&a.status[0], 0, RA_ERR_DEVICE_WAIT);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == 0 && lane == 0) {
    prefetch_map(&tmap_k);
    prefetch_map(&tmap_v);
  }
  tc_fence_before();
  // an earlier block gave up: leave at once; a cluster starts in the aborted state instead and
  // still meets at its barriers (see step_tc.cu)
  const bool leave = __syncthreads_or(gone) != 0 && !kSplit;
  tc_fence_after();
  const unsigned tmem_base = *tmem_slot;
  wait_for_previous();
  if (leave) {
    if (warp == 1)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    return;
  }

  // Split operands come as they are: the block's largest magnitude of Q meets each tile's of K where the tile is used.
  [[maybe_unused]] auto wait_q = [&](int* q_top) {
    bool ok = true;
    *q_top = 0;
    for (int w = 0; w < live && ok; ++w) {
      ok = mbar_wait(bar_q_full + 8 * w, 0, abort_flag, a.status, 3, w, a.wait_ns);
      if (ok) *q_top = max(*q_top, max(max(q_tops[4 * w], q_tops[4 * w + 1]), max(q_tops[4 * w + 2], q_tops[4 * w + 3])));
    }
    return ok;
  };
  [[maybe_unused]] const unsigned char* const meta_ring = smem + C::kOffG;
  [[maybe_unused]] auto tile_exp = [&](int j, int q_top) {  // as v_exp would hold it
    const unsigned char* const m = meta_ring + (j % C::kGDepth) * kMetaBytes;
    const int ve = *reinterpret_cast<const volatile int*>(m + kMetaVExp), k_top = *reinterpret_cast<const volatile int*>(m + kMetaKTop);
    return q_top + k_top - 254 >= kScoreRange ? kWide | kPlain : ve;
  };

  // (registers follow the work, see F32Cfg)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kRegsIssue));
    if (warp == 0) {
      // ---------------------------------------------------------- TMA producer ----
      if (lane == 0 && n_tiles > 0) {
        int it = 0;
        [[maybe_unused]] int k_top = 0, q_top = 0;
        bool ok = *abort_flag == 0;
        // (the status word once more, see step_tc.cu: behind a launch that gave up no V comes)
        const int lost = *reinterpret_cast<volatile int*>(a.status);
        TileShare share{share_beg, share_end, 0};
        for (int sk = 0; sk < a.kmap.n_seg && ok; ++sk) {
          const TileRange r =
              share.clip(tile_range<kBNf>(a.kmap, sk, a.stride, causal, a.doc_len, qmin, qmax));
          for (int t = r.lo; t < r.hi && ok; ++t) {
            const int k_row = a.kseg_row[sk] + t * kBNf;
            const int k_head = a.kseg_head[sk] + kv_bh;
            for (int which = 0; which < 2 && ok; ++which, ++it) {
              if (which == 1 && lost != 0) {
                *abort_flag = 1;
                ok = false;
                break;
              }
              const int slot = it % C::kStages;
              if (it >= C::kStages)
                ok = mbar_wait(bar_kv_empty + 8 * slot, ((it / C::kStages) + 1) & 1, abort_flag,
                               a.status, 1, it, a.wait_ns);
              if (!ok) break;
              if (a.stall_after >= 0 && it >= a.stall_after) {  // test hook, see step_tc.cu
                ok = false;
                break;
              }
              const CUtensorMap* map = which == 0 ? &tmap_k : &tmap_v;
              auto raw = [&](unsigned bar) {
                for (int bx = 0; bx < C::kBoxes; ++bx)
                  tma_load_3d(s_kv + slot * C::kSlotBytes + bx * C::kBoxBytes, map, bar, bx * 32, k_row, k_head);
              };
              if constexpr (kPre) {
                const unsigned bar = bar_kv_full + 8 * slot;
                const size_t tile = static_cast<size_t>(kv_bh) * pre.tiles + pre.beg[sk] + t;
                const unsigned char* const meta = pre.meta + tile * kMetaBytes;
                if (which == 0) {
                  mbar_expect_tx(bar, C::kSlotBytes);
                  bulk_load(s_kv + slot * C::kSlotBytes, pre.k + tile * C::kSlotBytes, C::kSlotBytes, bar);
                  k_top = *reinterpret_cast<const volatile int*>(meta + kMetaKTop);  // (used with V)
                } else {
                  // The meta data come with V, whose slot, other than K's, is not loaded again before the softmax of the
                  // tile is done: a wait for V's barrier can stand for them.
                  if (it == 1 && !(ok = wait_q(&q_top))) break;
                  const bool plain = q_top + k_top - 254 >= kScoreRange;  // P * V will be taken in plain fp32
                  mbar_expect_tx(bar, (plain ? C::kRawBytes : C::kSlotBytes) + kMetaBytes);
                  if (plain) raw(bar);
                  else bulk_load(s_kv + slot * C::kSlotBytes, pre.v + tile * C::kSlotBytes, C::kSlotBytes, bar);
                  bulk_load(s_base + C::kOffG + ((it >> 1) % C::kGDepth) * kMetaBytes, meta, kMetaBytes, bar);
                }
              } else {
                mbar_expect_tx(bar_kv_raw + 8 * slot, C::kRawBytes);
                raw(bar_kv_raw + 8 * slot);
              }
            }
          }
        }
      }
    } else if (warp == 1 || (!C::kOneIssuer && warp == 2 && live == 2)) {
      // ----------------------------------------------------------- MMA issuers ----
      if (n_tiles > 0) {
        constexpr unsigned idesc_s = make_idesc(0u, 0, kBNf, kBM);
        constexpr unsigned idesc_pv = make_idesc(0u, 1, DR, kBM);
        constexpr unsigned kQBox = (kBM * 128) >> 4;        // one 64-column box, 16-byte units
        constexpr unsigned kGroup = (2 * C::kBoxBytes) >> 4;  // hi and lo box of a 64-column group
        constexpr unsigned kLo = C::kBoxBytes >> 4;
        auto wait = [&](unsigned bar, unsigned parity, int which, int tile) {
          return __all_sync(0xffffffffu,
                            mbar_wait(bar, parity, abort_flag, a.status, which, tile, a.wait_ns)) != 0;
        };
        [[maybe_unused]] int q_top = 0;
        if constexpr (kPre) wait_q(&q_top);  // (one that runs out is met again below)
        // ring item of K_t: 2t, of V_t: 2t + 1 (which the softmax has waited for when its P is written: no wait here)
        auto wait_kv = [&](int it, int which, int t) {
          return wait(bar_kv_full + 8 * (it % C::kStages), (it / C::kStages) & 1, which, t);
        };
        // `last`: no other of this thread's MMAs reads the slot, which is free when they are done (or the caller sees to it)
        auto issue_s = [&](int t, int w, bool last) {
          const int slot = (2 * t) % C::kStages;
          const unsigned kd = static_cast<unsigned>(desc_kmajor(s_kv + slot * C::kSlotBytes));
          [[maybe_unused]] const unsigned qd = static_cast<unsigned>(desc_kmajor(s_q + w * C::kQBytes));
          const unsigned t_s = tmem_base + 256 * w + C::kColS, t_q = tmem_base + 256 * w + C::kColQ;
          if (elect_one()) {
            // small terms first: lo*hi, hi*lo, hi*hi
#pragma unroll
            for (int term = 0; term < 3; ++term) {
#pragma unroll
              for (int ks = 0; ks < DR / 16; ++ks) {  // 16 columns = 32 bytes, 4 steps per group
                const unsigned off_k = (ks / 4) * kGroup + (ks % 4) * 2 + (term == 1 ? kLo : 0);
                const unsigned acc = (term > 0 || ks > 0) ? 1u : 0u;
                if (C::kQLoInTmem || term > 0) {
                  mma_ts_lo(t_s, t_q + ks * 8 + (term == 0 ? 32 : 0), kd + off_k, kDescHi, idesc_s, acc);
                } else {
                  mma_ss_lo(t_s, qd + (ks / 4) * kQBox + (ks % 4) * 2, kd + off_k, kDescHi, idesc_s, acc);
                }
              }
            }
            tc_commit(bar_s_full + 8 * w);
            if (last) tc_commit(bar_kv_empty + 8 * slot);
          }
        };
        auto issue_pv = [&](int t, int w, bool last) {
          const int slot = (2 * t + 1) % C::kStages;
          // MN-major V: 64 columns per 128-byte row, groups 2 boxes apart, 16 keys per k-step
          const unsigned vd = static_cast<unsigned>(desc_mnmajor(s_kv + slot * C::kSlotBytes, 2 * C::kBoxBytes, 1024));
          const unsigned t_p = tmem_base + 256 * w + C::kColP, t_o = tmem_base + 256 * w + C::kColO;
          // (marked: the softmax threads have added this tile to O)
          const bool wide = ((kPre ? tile_exp(t, q_top) : v_exp[t & 15]) & kWide) != 0;
          if (elect_one()) {
            if (!wide) {
#pragma unroll
              for (int term = 0; term < 3; ++term) {
#pragma unroll
                for (int ks = 0; ks < kBNf / 16; ++ks)
                  mma_ts_lo(t_o, t_p + ks * 8 + (term == 0 ? 32 : 0),
                            vd + ks * (2048 >> 4) + (term == 1 ? kLo : 0), kDescHi, idesc_pv,
                            (t > 0 || term > 0 || ks > 0) ? 1u : 0u);
              }
            }
            tc_commit(bar_o_done + 8 * w);
            if (last) tc_commit(bar_kv_empty + 8 * slot);
          }
        };
        bool ok = true;
        if constexpr (C::kTurns) {
          // As below, but with a warp for each query tile, whose turn comes with the end of the other's batch: it has done its
          // waits by then. The tensor core's queue holds a few instructions, so a batch that follows at once leaves no gap.
          // A turn orders when batches are issued, not when they end, and a commit is about its own thread's MMAs: each warp
          // commits to the slots it has read, and a slot is free when both have. These commits go behind the turn, out of the
          // other warp's way: B1 H4 S16384 D128 causal 686 us in a CUDA graph, with each behind its MMAs 703, V's there and K's behind
          // the turn 694.
          const int w = warp - 1;
          auto turn = [&](int n) { return live == 1 || wait(bar_turn + 8 * w, n & 1, 12, n); };
          auto free_slot = [&](int it) {  // (nobody waits for the last ones, so nothing arrives late in a block that ends)
            if (it + C::kStages < 2 * n_tiles && elect_one()) tc_commit(bar_kv_empty + 8 * (it % C::kStages));
          };
          auto pass = [&]() {
            if (live == 2 && elect_one()) mbar_arrive(bar_turn + 8 * (1 - w));
          };
          ok = wait(bar_q_full + 8 * w, 0, 3, w) && wait_kv(0, 5, 0) && (w == 0 || turn(0));
          if (ok) {
            tc_fence_after();
            issue_s(0, w, false);
            pass();
            free_slot(0);
          }
          for (int t = 0; t < n_tiles && ok; ++t) {
            const bool more = t + 1 < n_tiles;
            ok = (!more || wait_kv(2 * t + 2, 5, t)) && wait(bar_p_full + 8 * w, t & 1, 6, t) && turn(t + w);
            if (!ok) break;
            tc_fence_after();
            issue_pv(t, w, false);
            if (more) issue_s(t + 1, w, false);
            pass();
            free_slot(2 * t + 1);
            if (more) free_slot(2 * t + 2);
          }
        } else if constexpr (C::kAlias) {
          // One warp issues for both query tiles, in turn: P.V of tile t and the scores of tile t + 1, which
          // overwrite P, of one query tile, then those of the other. The tensor core runs them in that
          // order, so one tile's softmax works under the other's MMAs. (Two issuing warps end in step:
          // the tensor core takes their instructions alternately, both batches end together, 3250 clocks
          // after they began, and both softmax groups run at once while it idles: 6400 clocks a tile.)
          for (int w = 0; w < live && ok; ++w) {
            ok = wait(bar_q_full + 8 * w, 0, 3, w) && wait_kv(0, 5, 0);
            if (!ok) break;
            tc_fence_after();
            issue_s(0, w, w == live - 1);
          }
          for (int t = 0; t < n_tiles && ok; ++t) {
            const bool more = t + 1 < n_tiles;
            ok = !more || wait_kv(2 * t + 2, 5, t);
            for (int w = 0; w < live && ok; ++w) {
              ok = wait(bar_p_full + 8 * w, t & 1, 6, t);
              if (!ok) break;
              tc_fence_after();
              issue_pv(t, w, w == live - 1);
              if (more) issue_s(t + 1, w, w == live - 1);
            }
          }
        } else {
          const int w = warp - 1;
          ok = wait(bar_q_full + 8 * w, 0, 3, w) && wait_kv(0, 5, 0);
          if (ok) {
            tc_fence_after();
            issue_s(0, w, true);
          }
          for (int t = 0; t < n_tiles && ok; ++t) {
            if (t + 1 < n_tiles) {
              ok = wait(bar_s_free + 8 * w, t & 1, 9, t) && wait_kv(2 * t + 2, 5, t);
              if (!ok) break;
              tc_fence_after();
              issue_s(t + 1, w, true);
            }
            ok = wait(bar_p_full + 8 * w, t & 1, 6, t);
            if (!ok) break;
            tc_fence_after();
            issue_pv(t, w, true);
          }
        }
      }
    }
    if constexpr (kSplit) {  // the three meetings of merge_key_split
      for (int i = 0; i < 3; ++i) cluster_sync_threads();
    }
  } else if (!kPre && warp >= 12) {
    if constexpr (!kPre) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kRegsSplit));
    // --------------------------------------------------------------- splitters ----
    // A warp owns eight rows of every tile; its lanes own 16-byte pieces of the split rows (8
    // values, 32 raw bytes): lane = (piece, row), so the eight lanes of a phase touch eight rows
    // at one swizzled column and no bank twice.
    if (n_tiles > 0) {
      constexpr int kUnits = DR / 32;  // pieces per lane
      const int sw = warp - 12, r8 = lane & 7, p4 = lane >> 3;
      const unsigned row_off = (sw * 8 + r8) * 128;
      bool ok = true;
      int q_top = 0, k_top = 0;  // exponents: of the query block, of the warp's eight keys of the tile
      for (int it = 0; it < 2 * n_tiles && ok; ++it) {
        const int slot = it % C::kStages;
        ok = __all_sync(0xffffffffu, mbar_wait(bar_kv_raw + 8 * slot, (it / C::kStages) & 1, abort_flag,
                                               a.status, 13, it, a.wait_ns)) != 0;
        if (!ok) break;
        const unsigned base = s_kv + slot * C::kSlotBytes + row_off;
        float x[kUnits][8];
        float fm = 0.f;
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
          const int piece = p4 + 4 * u;  // of the whole row; raw box = piece / 4, 2 chunks each
          const unsigned box = base + (piece >> 2) * C::kBoxBytes;
          const int c = (piece & 3) * 2;
          const float4 v0 = ld_shared_f4(box + ((c ^ r8) << 4));
          const float4 v1 = ld_shared_f4(box + (((c + 1) ^ r8) << 4));
          x[u][0] = v0.x, x[u][1] = v0.y, x[u][2] = v0.z, x[u][3] = v0.w;
          x[u][4] = v1.x, x[u][5] = v1.y, x[u][6] = v1.z, x[u][7] = v1.w;
#pragma unroll
          for (int i = 0; i < 8; i += 2) fm = max3(fm, fabsf(x[u][i]), fabsf(x[u][i + 1]));
        }
        unsigned mx = __float_as_uint(fm);  // (a maximum passes NaN by)
        if (mx >= 0x7f800000u) {            // an infinity among them: the finite ones count
          mx = 0;
#pragma unroll
          for (int u = 0; u < kUnits; ++u)
#pragma unroll
            for (int i = 0; i < 8; ++i) mx = max(mx, finite_abs_bits(x[u][i]));
        }
        int e;
        bool wide = false;
        if ((it & 1) == 0) {
          // K: by key. The row's pieces sit in the four lanes r8, r8 + 8, ...
          mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
          mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
          e = scale_exp(mx, kMaxExpK);
          if (p4 == 0) {
            const unsigned g = s_base + C::kOffG + (((it >> 1) % C::kGDepth) * kBNf + sw * 8 + r8) * 4;
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(g), "f"(pow2i(-e - kBias)) : "memory");
          }
          k_top = static_cast<int>(__reduce_max_sync(0xffffffffu, mx) >> 23);  // (the warp's rows have been read)
        } else {
          // V: by tile
          unsigned low = v_range<kUnits>(x, mx, lane, smem + C::kOffVKey + ((it >> 1) & 7) * kBNf + sw * 8);
          if (it == 1) {
            for (int w = 0; w < live && ok; ++w) {
              ok = __all_sync(0xffffffffu, mbar_wait(bar_q_full + 8 * w, 0, abort_flag, a.status, 3, w, a.wait_ns)) != 0;
              if (ok) q_top = max(q_top, max(max(q_tops[4 * w], q_tops[4 * w + 1]), max(q_tops[4 * w + 2], q_tops[4 * w + 3])));
            }
            if (!ok) break;
          }
          const bool plain = q_top + k_top - 254 >= kScoreRange;
          const int par = (it >> 1) & 1;
          if (lane == 0) {
            red[par * 16 + sw] = mx | (plain ? 0x80000000u : 0u);
            red[par * 16 + 8 + sw] = low;
            mbar_arrive(bar_v_max);
          }
          // (an mbarrier and not bar.sync: a warp that gives up must not leave the others waiting)
          ok = __all_sync(0xffffffffu,
                          mbar_wait(bar_v_max, par, abort_flag, a.status, 15, it, a.wait_ns)) != 0;
          if (!ok) break;
          const unsigned red_at = s_base + C::kOffRed + par * 64;
          const uint4 m0 = ld_shared_u4(red_at), m1 = ld_shared_u4(red_at + 16);
          const uint4 l0 = ld_shared_u4(red_at + 32), l1 = ld_shared_u4(red_at + 48);
          const unsigned marks = (m0.x | m0.y | m0.z | m0.w) | (m1.x | m1.y | m1.z | m1.w);
          constexpr unsigned kMag = 0x7fffffffu;
          mx = max(max(max(m0.x & kMag, m0.y & kMag), max(m0.z & kMag, m0.w & kMag)),
                   max(max(m1.x & kMag, m1.y & kMag), max(m1.z & kMag, m1.w & kMag)));
          low = min(min(min(l0.x, l0.y), min(l0.z, l0.w)), min(min(l1.x, l1.y), min(l1.z, l1.w)));
          e = scale_exp(mx, kMaxExp);
          wide = low < mx >> 16 || marks > kMag;
          if (sw == 0 && lane == 0)
            v_exp[(it >> 1) & 15] = wide ? (marks > kMag ? kWide | kPlain : kWide) : mx == 0 ? kNoUnit : e + kExpBias;
        }
        const float sc = pow2i(e);
        if (!wide) {  // (a wide tile stays as it is)
#pragma unroll
          for (int u = 0; u < kUnits; ++u) {
            const int piece = p4 + 4 * u;  // split box pair = piece / 8
            const unsigned hi_at = base + (piece >> 3) * 2 * C::kBoxBytes + (((piece & 7) ^ r8) << 4);
            unsigned hi[4], lo[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) split_pair(x[u][2 * i] * sc, x[u][2 * i + 1] * sc, hi[i], lo[i]);
            st_shared_u4(hi_at, hi[0], hi[1], hi[2], hi[3]);
            st_shared_u4(hi_at + C::kBoxBytes, lo[0], lo[1], lo[2], lo[3]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(bar_kv_full + 8 * slot);
      }
    }
    if constexpr (kSplit) {
      for (int i = 0; i < 3; ++i) cluster_sync_threads();
    }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kRegsSoftmax));
    // ----------------------------------------------------------------- softmax ----
    const int w = (warp - 4) >> 2;
    const int row = ((warp & 3) << 5) + lane;  // row of the tile = tensor-memory lane
    const unsigned t_w = tmem_base + (static_cast<unsigned>((warp & 3) << 5) << 16) + 256 * w;
    const unsigned t_s = t_w + C::kColS, t_p = t_w + C::kColP, t_o = t_w + C::kColO;
    const int r_in_seg = row0 + w * kBM + row;
    const bool row_valid = r_in_seg < q_seg_len;
    const int qpos = a.qmap.base[sq] + r_in_seg * a.stride;
    const long long qdoc = a.doc_len > 0 ? qpos / a.doc_len : 0;
    const size_t grow0 = static_cast<size_t>(bh) * a.Sq + static_cast<size_t>(sq) * q_seg_len + row0;
    const size_t grow = grow0 + (row_valid ? w * kBM + row : 0);
    const bool mine = w < live && n_tiles > 0;

    // ---- this row of Q: scale, split, hand to the MMA warp
    // 1 / sqrt(head_dim) in log2 units
    constexpr float kPlainF = (DR == 32 ? 0.17677669529663689f : DR == 64 ? 0.125f : 0.08838834764831845f) * kLog2e;
    float row_f = 0.f;  // turns a scaled score (K factor applied) into log2 units
    if (mine) {
      const float4* q4 = reinterpret_cast<const float4*>(q_g + grow * DR);
      unsigned mx = 0;
#pragma unroll 16
      for (int i = 0; i < DR / 4; ++i) {
        const float4 v = row_valid ? q4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        mx = max(max(max(mx, finite_abs_bits(v.x)), max(finite_abs_bits(v.y), finite_abs_bits(v.z))),
                 finite_abs_bits(v.w));
      }
      const int e = scale_exp(mx, kMaxExp);
      const float sc = pow2i(e);
      mx = __reduce_max_sync(0xffffffffu, mx);
      if (lane == 0) q_tops[warp - 4] = static_cast<int>(mx >> 23);
      row_f = kPlainF * pow2i(kBias - e);
#pragma unroll
      for (int g = 0; g < DR / 32; ++g) {  // 32 columns at a time (second read: L1 / L2)
        unsigned hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 v = row_valid ? q4[g * 8 + i] : make_float4(0.f, 0.f, 0.f, 0.f);
          split_pair(v.x * sc, v.y * sc, hi[2 * i], lo[2 * i]);
          split_pair(v.z * sc, v.w * sc, hi[2 * i + 1], lo[2 * i + 1]);
        }
        tmem_st16(t_w + C::kColQ + 16 * g, hi);
        if constexpr (C::kQLoInTmem) {
          tmem_st16(t_w + C::kColQ + 32 + 16 * g, lo);
        } else {
          const unsigned at = s_q + w * C::kQBytes + (g >> 1) * (kBM * 128) + row * 128;
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const unsigned off = ((((g & 1) * 4 + p) ^ (row & 7)) << 4);
            st_shared_u4(at + off, lo[4 * p], lo[4 * p + 1], lo[4 * p + 2], lo[4 * p + 3]);
          }
        }
      }
      tmem_wait_st();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_fence_before();
      mbar_arrive(bar_q_full + 8 * w);
    }

    float m_ref = -INFINITY;  // reference point of P, O and l, log2 units
    float l_run = 0.f;
    int unit = kNoUnit;       // O is in units of 2^-unit
    bool ok = true;
    int j = 0;
    const int n_seg = mine ? a.kmap.n_seg : 0;
    TileShare share{share_beg, share_end, 0};
    [[maybe_unused]] int q_top = 0;
    if constexpr (kPre) ok = __all_sync(0xffffffffu, !mine || wait_q(&q_top)) != 0;
    for (int sk = 0; sk < n_seg && ok; ++sk) {
      const TileRange tr =
          share.clip(tile_range<kBNf>(a.kmap, sk, a.stride, causal, a.doc_len, qmin, qmax));
      // visible local key indices [rel_lo, rel_hi) of this segment for this row
      int rel_lo = 0, rel_hi = row_valid ? a.kmap.seg_len : 0;
      {
        const long long kb = a.kmap.base[sk];
        if (causal) {
          const long long d = static_cast<long long>(qpos) - kb;
          rel_hi = d < 0 ? 0 : static_cast<int>(min(static_cast<long long>(rel_hi), d / a.stride + 1));
        }
        if (a.doc_len > 0) {
          const long long p_lo = qdoc * a.doc_len, p_hi = p_lo + a.doc_len - 1;
          if (p_hi < kb) {
            rel_hi = 0;
          } else {
            rel_hi = static_cast<int>(min(static_cast<long long>(rel_hi), (p_hi - kb) / a.stride + 1));
            if (p_lo > kb)
              rel_lo = static_cast<int>(min(static_cast<long long>(a.kmap.seg_len),
                                            (p_lo - kb + a.stride - 1) / a.stride));
          }
        }
      }
      for (int t = tr.lo; t < tr.hi && ok; ++t, ++j) {
        int c_lo = min(max(rel_lo - t * kBNf, 0), kBNf);
        int c_hi = min(max(rel_hi - t * kBNf, 0), kBNf);
        if (c_hi < c_lo) c_hi = c_lo;
        const bool full = __all_sync(0xffffffffu, c_lo == 0 && c_hi == kBNf);

        // the V tile's barrier stands for both: K_j is split before V_j, and V_j's slot is not
        // reused before this softmax is done
        const int vit = 2 * j + 1;
        ok = mbar_wait(bar_kv_full + 8 * (vit % C::kStages), (vit / C::kStages) & 1, abort_flag, a.status,
                       11, j, a.wait_ns);
        const int ve = kPre ? tile_exp(j, q_top) : v_exp[j & 15];
        ok = ok && mbar_wait(bar_s_full + 8 * w, j & 1, abort_flag, a.status, 7, j, a.wait_ns);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const unsigned g_at = s_base + C::kOffG + (j % C::kGDepth) * (kPre ? kMetaBytes : kBNf * 4);
        if (__builtin_expect((ve & kWide) != 0, 0)) {
          // A marked tile: P * V in plain fp32 from V as it landed in its slot (every lane reads the same
          // 16 bytes), and the scores too if Q and K ask for it. Short loops over tensor memory, so that
          // the registers of the common path do not suffer. The issuer only passes the barriers on.
          if (!C::kAlias && j > 0) {
            ok = mbar_wait(bar_o_done + 8 * w, (j - 1) & 1, abort_flag, a.status, 10, j, a.wait_ns);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
          }
          const bool any = __any_sync(0xffffffffu, c_hi > c_lo) != 0;
          if (any && (ve & kPlain) != 0) {
            // eight keys at a time, Q and K from memory (the K slot may have been given back), scaled as
            // the tensor core's scores are, in their place
            const float4* q4 = reinterpret_cast<const float4*>(q_g + grow * DR);
            const float* k_t = k_g + (a.kseg_head[sk] + kv_bh) * kv_head_stride +
                               static_cast<long long>(a.kseg_row[sk] + t * kBNf) * DR;
            const int last = min(kBNf, a.kmap.seg_len - t * kBNf) - 1;
            const float unscale = pow2i((__float_as_int(kPlainF) >> 23) - (__float_as_int(row_f) >> 23));
#pragma unroll 1
            for (int i0 = 0; i0 < kBNf; i0 += 8) {
              float x[8] = {};
#pragma unroll 1
              for (int c = 0; c < DR / 4; ++c) {
                const float4 qv = row_valid ? q4[c] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const float4 kv = *reinterpret_cast<const float4*>(k_t + min(i0 + i, last) * DR + 4 * c);
                  x[i] = fmaf(qv.w, kv.w, fmaf(qv.z, kv.z, fmaf(qv.y, kv.y, fmaf(qv.x, kv.x, x[i]))));
                }
              }
#pragma unroll
              for (int i = 0; i < 8; ++i)
                x[i] = x[i] * unscale * pow2i(127 - static_cast<int>(ld_shared_u1(g_at + (i0 + i) * 4) >> 23));
              tmem_st8(t_s + i0, x);
            }
            tmem_wait_st();
          }
          auto scores = [&](int i0, float (&x)[8]) {
            tmem_ld8(t_s + i0, x);
#pragma unroll
            for (int i = 0; i < 8; ++i)
              x[i] = i0 + i >= c_lo && i0 + i < c_hi ? x[i] * __uint_as_float(ld_shared_u1(g_at + (i0 + i) * 4)) : -INFINITY;
          };
          float alpha = 1.f;
          int c_top = 0;  // biased exponents of P and V of the largest product
          if (any) {
            float mx = -INFINITY, x[8];
#pragma unroll 1
            for (int i0 = 0; i0 < kBNf; i0 += 8) {
              scores(i0, x);
#pragma unroll
              for (int i = 0; i < 8; ++i) mx = fmaxf(mx, x[i]);
            }
            const float tile_max = mx * row_f;
            if (tile_max > m_ref) {
              if (m_ref > -INFINITY) alpha = ex2(m_ref - tile_max);
              m_ref = tile_max;
            }
            const float n = m_ref == -INFINITY ? 0.f : kPBits - m_ref;
            float sum = 0.f;
#pragma unroll 1
            for (int i0 = 0; i0 < kBNf; i0 += 8) {  // P as fp32 over the columns of its terms
              scores(i0, x);
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                x[i] = ex2(fmaf(x[i], row_f, n));
                sum += x[i];
                const int vk = kPre ? meta_ring[(j % C::kGDepth) * kMetaBytes + kMetaVKey + i0 + i]
                                    : smem[C::kOffVKey + (j & 7) * kBNf + i0 + i];
                if (x[i] > 0.f && vk > 0) c_top = max(c_top, (__float_as_int(x[i]) >> 23) + vk);
              }
              tmem_st8(t_p + i0, x);
            }
            tmem_wait_st();
            l_run = l_run * alpha + sum * pow2i(-kPBits);
          }
          if constexpr (!C::kAlias) {
            tc_fence_before();
            mbar_arrive(bar_s_free + 8 * w);
          }
          if (any || j == 0) {
            // unit: a product becomes at most 2^22
            const int to = c_top == 0 ? unit : min(unit, min(kMaxExp, 22 - (c_top - 252 - kPBits)));
            const float fac = unit == kNoUnit ? alpha : alpha * ex2(static_cast<float>(to - unit));
            unit = to;
            const float p_sc = to == kNoUnit ? 0.f : pow2i(to - kPBits);
            const unsigned v_at = s_kv + (vit % C::kStages) * C::kSlotBytes;
#pragma unroll 1
            for (int c = 0; c < DR; c += 16) {
              const unsigned box = v_at + (c >> 5) * C::kBoxBytes;
              float acc[16] = {};
#pragma unroll 1
              for (int i0 = 0; any && i0 < kBNf; i0 += 8) {
                float p[8];
                tmem_ld8(t_p + i0, p);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  p[i] *= p_sc;
#pragma unroll
                  for (int u = 0; u < 4; ++u) {  // 16-byte chunks of the row
                    const float4 v = ld_shared_f4(box + (i0 + i) * 128 + ((((c & 31) >> 2) + u) ^ i) * 16);
                    acc[4 * u] = fmaf(p[i], v.x, acc[4 * u]), acc[4 * u + 1] = fmaf(p[i], v.y, acc[4 * u + 1]);
                    acc[4 * u + 2] = fmaf(p[i], v.z, acc[4 * u + 2]), acc[4 * u + 3] = fmaf(p[i], v.w, acc[4 * u + 3]);
                  }
                }
              }
#pragma unroll
              for (int u = 0; u < 16; u += 8) {
                float o[8] = {};
                if (j > 0) tmem_ld8(t_o + c + u, o);
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = fmaf(o[i], fac, acc[u + i]);
                tmem_st8(t_o + c + u, o);
              }
            }
            tmem_wait_st();
          }
          tc_fence_before();
          mbar_arrive(bar_p_full + 8 * w);
          continue;
        }
        float s[kBNf];
        tmem_ld64(t_s, s);
        if constexpr (!C::kAlias) {
          tc_fence_before();
          mbar_arrive(bar_s_free + 8 * w);  // the tensor core may write the next scores
        }
#pragma unroll
        for (int i = 0; i < kBNf; i += 4) {
          const float4 g = ld_shared_f4(g_at + i * 4);
          const float2 x0 = fmul2(make_float2(s[i], s[i + 1]), make_float2(g.x, g.y));
          const float2 x1 = fmul2(make_float2(s[i + 2], s[i + 3]), make_float2(g.z, g.w));
          s[i] = x0.x, s[i + 1] = x0.y, s[i + 2] = x1.x, s[i + 3] = x1.y;
        }
        if (!full) {
#pragma unroll
          for (int i = 0; i < kBNf; ++i) s[i] = (i >= c_lo && i < c_hi) ? s[i] : -INFINITY;
        }

        // P of this tile is 2^p_exp at the reference point, so that P * V (scaled by 2^ev) lands in
        // the row's unit. The unit is the row's own and follows what the row adds to O: a V tile it sees no
        // key of says nothing, and one of larger values only once a P that it meets would leave fp16. The
        // two terms of P have an absolute floor of 2^-25, so a tile of much smaller values (p_exp < 0) moves
        // the unit as well.
        const int ev = ve - kExpBias;
        const bool adds = c_hi > c_lo && ve < kWide;
        if (adds && unit == kNoUnit) unit = kPBits + ev;
        int p_exp = adds ? unit - ev : kPBits;
        bool slow = __any_sync(0xffffffffu, p_exp < 0 || p_exp > 100 || (m_ref == -INFINITY && c_hi > c_lo)) != 0;
        // Wait for P.V of the previous tile: its P buffer is about to be written. (With P over S the
        // scores of this tile, issued behind it, stand for that.)
        if (!C::kAlias && j > 0) {
          ok = mbar_wait(bar_o_done + 8 * w, (j - 1) & 1, abort_flag, a.status, 10, j, a.wait_ns);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
        }
        const float2 f2 = make_float2(row_f, row_f);
        float row_sum = 0.f, oct_max = 0.f;
        // P = 2^(s * f - m_ref + p_exp) as hi + lo in tensor memory, 32 columns at a time; the sums
        // of eight columns each bound every P and add up to the row sum
        auto exponentials = [&]() {
          const float n = m_ref == -INFINITY ? 0.f : static_cast<float>(p_exp) - m_ref;
          const float2 n2 = make_float2(n, n);
          float2 sum[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) sum[i] = make_float2(0.f, 0.f);
#pragma unroll
          for (int c = 0; c < kBNf / 32; ++c) {
            unsigned hi[16], lo[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float2 x = ffma2(make_float2(s[32 * c + 2 * i], s[32 * c + 2 * i + 1]), f2, n2);
              const float2 p = make_float2(ex2(x.x), ex2(x.y));
              sum[i & 3] = fadd2(sum[i & 3], p);
              split_pair(p.x, p.y, hi[i], lo[i]);
            }
            tmem_st16(t_p + 16 * c, hi);
            tmem_st16(t_p + 32 + 16 * c, lo);
          }
          const float2 s01 = fadd2(sum[0], sum[1]), s23 = fadd2(sum[2], sum[3]);
          const float2 all = fadd2(s01, s23);
          oct_max = fmaxf(max3(fmaxf(sum[0].x, sum[0].y), sum[1].x, sum[1].y),
                          max3(fmaxf(sum[2].x, sum[2].y), sum[3].x, sum[3].y));
          row_sum = all.x + all.y;
        };
        if (!slow) {
          exponentials();
          slow = __any_sync(0xffffffffu, !(oct_max <= kPSumLimit) || !(row_sum == row_sum)) != 0;
        }
        if (slow) {
          float mx = s[0];
#pragma unroll
          for (int i = 1; i < kBNf - 1; i += 2) mx = max3(mx, s[i], s[i + 1]);
          mx = fmaxf(mx, s[kBNf - 1]);
          const float tile_max = mx * row_f;  // -inf stays -inf
          float alpha = 1.f;
          const float m_old = m_ref;
          if (tile_max > m_ref) {
            if (m_old > -INFINITY) alpha = ex2(m_old - tile_max);
            m_ref = tile_max;
          }
          l_run *= alpha;
          // O as it stands is in units of 2^-keep of the new reference point. This tile's largest P,
          // 2^-low of it, must not exceed 2^kPBits; and if its values are far smaller than the unit, O is
          // scaled up, as far as it cannot overflow.
          const int low = static_cast<int>(fminf(m_ref - tile_max, 100.f));
          const int keep = unit + (m_old > -INFINITY ? static_cast<int>(fminf(m_ref - m_old, 1000.f)) : 0);
          int to = adds ? min(keep, kPBits + ev + low) : unit;
          if (j > 0 && __any_sync(0xffffffffu, adds && to < ev)) {
            float top = 0.f;
#pragma unroll 1
            for (int c = 0; c < DR / 32; ++c) {
              float o[32];
              tmem_ld32(t_o + c * 32, o);
#pragma unroll
              for (int i = 0; i < 32; i += 2) top = max3(top, fabsf(o[i]), fabsf(o[i + 1]));
            }
            const int room = kOTop + 126 - (__float_as_int(top) >> 23);
            if (adds && to < ev) to = max(to, min(kPBits + ev, keep + room));
          }
          float oa = alpha;  // factor of O
          if (adds) {
            if (m_old > -INFINITY) oa = ex2(m_old - m_ref + static_cast<float>(to - unit));
            unit = to;
            p_exp = max(to - ev, kMinPExp);
          }
          if (j > 0 && __any_sync(0xffffffffu, oa != 1.f)) {
            // O is at rest: P.V of tile j - 1 has completed
#pragma unroll 1
            for (int c = 0; c < DR / 32; ++c) {
              float o[32];
              tmem_ld32(t_o + c * 32, o);
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] *= oa;
              tmem_st32(t_o + c * 32, o);
            }
          }
          exponentials();
        }
        l_run += row_sum * pow2i(-p_exp);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(bar_p_full + 8 * w);
      }
    }

    // ---------------------------------------------------------------- epilogue ----
    auto wait_o = [&]() {
      if (ok && mine)
        ok = mbar_wait(bar_o_done + 8 * w, (n_tiles - 1) & 1, abort_flag, a.status, 8, n_tiles, a.wait_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (ok && mine) tc_fence_after();
      return ok;
    };
    const float o_unit = pow2_any(unit == kNoUnit ? 0 : -unit);
    if constexpr (kSplit) {
      wait_o();
      const bool gave_up = __any_sync(0xffffffffu, !ok || *abort_flag != 0) != 0;
      merge_key_split<C, DR>(a, smem, s_base, t_o, w, row, row_valid, grow0, gave_up, !gave_up && mine, m_ref, l_run,
                             o_unit, cta_rank, fresh, finalize);
    } else {
      float m_old = -INFINITY, l_old = 0.f;
      if (!fresh && row_valid) {
        m_old = a.m[grow];
        l_old = a.l[grow];
      }
      RowStore<DR>::run(
          lane, a.out, grow0 + w * kBM + row - lane, __ballot_sync(0xffffffffu, row_valid),
          s_base + C::kOffStage + w * C::kRowStage + (warp & 3) * RowStore<DR>::kStageBytes, t_o, mine, fresh, wait_o, [&]() {
            const bool have = row_valid && mine && m_ref > -INFINITY;
            const float m_new = have ? m_ref * kLn2 : -INFINITY;  // natural-log units
            const float m_fin = fmaxf(m_old, m_new);
            const float ca = (m_old == -INFINITY) ? 0.f : expf(m_old - m_fin);
            const float cb = have ? expf(m_new - m_fin) : 0.f;
            const float l_fin = ca * l_old + cb * l_run;
            const float inv = finalize ? (l_fin > 0.f ? 1.f / l_fin : 0.f) : 1.f;
            const bool touch = row_valid && (have || fresh || finalize);
            if (touch) {
              a.m[grow] = m_fin;
              a.l[grow] = l_fin;
            }
            return RowOut{touch, have, ca * inv, cb * inv, o_unit};
          });
    }
  }

  // ---------------------------------------------------------------- teardown ----
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*abort_flag) {
      // give copies and MMAs still in flight time to land before tensor memory is released
      const unsigned long long t0 = global_ns();
      while (global_ns() - t0 < 1000000ull) __nanosleep(1000);
    }
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base)
                 : "memory");
  }
}

// Splits K and V once for all query blocks of a call: a block per key tile and KV head writes, to the workspace, what the
// splitter warps leave in a ring slot, byte for byte, and the tile's meta data. (At head_dim 32 a slot has room for 64 columns:
// the other half is not written, and nothing reads what the step copies of it.) The step then copies whole slots, and has
// neither splitter warps (two thirds of its issue slots at head_dim 64) nor their traffic in shared memory. Bound by
// memory: H4 S16384 D128, 67 MB read and as many written, 27 us.
template <int DR>
__global__ void __launch_bounds__(kSplitThreads) split_kv_kernel(const float* k, const float* v, long long kv_head_stride,
                                                                const __grid_constant__ TcArgs a,
                                                                const __grid_constant__ SplitKV pre, int k_rows) {
  using C = F32Cfg<DR, false, true>;
  constexpr int kUnits = DR / 32;
  __shared__ unsigned red[3][8];
  let_next_start();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r8 = lane & 7, p4 = lane >> 3;
  int sk = 0;
  while (sk + 1 < a.kmap.n_seg && pre.beg[sk + 1] <= static_cast<int>(blockIdx.x)) ++sk;
  const int row = a.kseg_row[sk] + (static_cast<int>(blockIdx.x) - pre.beg[sk]) * kBNf + warp * 8 + r8;
  const size_t tile = static_cast<size_t>(blockIdx.y) * pre.tiles + blockIdx.x;
  const long long src = (a.kseg_head[sk] + static_cast<long long>(blockIdx.y)) * kv_head_stride + static_cast<long long>(row) * DR;
  const unsigned row_off = (warp * 8 + r8) * 128;
  unsigned char* const meta = pre.meta + tile * kMetaBytes;
  wait_for_previous();
  float x[2][kUnits][8];
  unsigned mx[2];
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const float4* const p = reinterpret_cast<const float4*>((which == 0 ? k : v) + src);
#pragma unroll
    for (int u = 0; u < kUnits; ++u) {
      const int piece = p4 + 4 * u;
      const float4 v0 = row < k_rows ? p[2 * piece] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 v1 = row < k_rows ? p[2 * piece + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
      x[which][u][0] = v0.x, x[which][u][1] = v0.y, x[which][u][2] = v0.z, x[which][u][3] = v0.w;
      x[which][u][4] = v1.x, x[which][u][5] = v1.y, x[which][u][6] = v1.z, x[which][u][7] = v1.w;
    }
  }
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    mx[which] = 0;
#pragma unroll
    for (int u = 0; u < kUnits; ++u)
#pragma unroll
      for (int i = 0; i < 8; ++i) mx[which] = max(mx[which], finite_abs_bits(x[which][u][i]));
  }
  // K: by key
  unsigned key = max(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], 8));
  key = max(key, __shfl_xor_sync(0xffffffffu, key, 16));
  const int ek = scale_exp(key, kMaxExpK);
  if (p4 == 0) reinterpret_cast<float*>(meta + kMetaG)[warp * 8 + r8] = pow2i(-ek - kBias);
  const unsigned k_max = __reduce_max_sync(0xffffffffu, mx[0]);
  // V: by tile
  const unsigned low_w = v_range<kUnits>(x[1], mx[1], lane, meta + kMetaVKey + warp * 8);
  if (lane == 0) red[0][warp] = k_max, red[1][warp] = mx[1], red[2][warp] = low_w;
  __syncthreads();
  unsigned k_all = 0, v_all = 0, low = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    k_all = max(k_all, red[0][i]);
    v_all = max(v_all, red[1][i]);
    low = min(low, red[2][i]);
  }
  const int e = scale_exp(v_all, kMaxExp);
  const bool wide = low < v_all >> 16;
  if (threadIdx.x == 0) {
    *reinterpret_cast<int*>(meta + kMetaVExp) = wide ? kWide : v_all == 0 ? kNoUnit : e + kExpBias;
    *reinterpret_cast<int*>(meta + kMetaKTop) = static_cast<int>(k_all >> 23);
  }
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    unsigned char* const base = (which == 0 ? pre.k : pre.v) + tile * C::kSlotBytes + row_off;
    const float sc = pow2i(which == 0 ? ek : e);
#pragma unroll
    for (int u = 0; u < kUnits; ++u) {
      const int piece = p4 + 4 * u;
      if (which == 1 && wide) {  // as it is, in the layout in which the copy of an fp32 tile lands
        unsigned char* const box = base + (piece >> 2) * C::kBoxBytes;
        const int c = (piece & 3) * 2;
        *reinterpret_cast<float4*>(box + ((c ^ r8) << 4)) = make_float4(x[1][u][0], x[1][u][1], x[1][u][2], x[1][u][3]);
        *reinterpret_cast<float4*>(box + (((c + 1) ^ r8) << 4)) = make_float4(x[1][u][4], x[1][u][5], x[1][u][6], x[1][u][7]);
        continue;
      }
      unsigned char* const hi_at = base + (piece >> 3) * 2 * C::kBoxBytes + (((piece & 7) ^ r8) << 4);
      unsigned hi[4], lo[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) split_pair(x[which][u][2 * i] * sc, x[which][u][2 * i + 1] * sc, hi[i], lo[i]);
      *reinterpret_cast<uint4*>(hi_at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(hi_at + C::kBoxBytes) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

// ---- host side ----------------------------------------------------------------------

// Tiles of all key segments of a head, and the workspace of the form with split operands.
int split_tiles(const StepArgs& a) { return (a.kmap.seg_len + kBNf - 1) / kBNf * a.kmap.n_seg; }
template <int DR>
size_t split_bytes(const StepArgs& a) {
  using C = F32Cfg<DR, false, true>;
  return static_cast<size_t>(a.B) * a.kvH * split_tiles(a) * (2 * C::kSlotBytes + kMetaBytes);
}
// Whether K and V are split ahead, given a workspace: a pair of query tiles saves 0.3 us a key tile (0.35 at head_dim 128), and the
// launch ahead costs 5 us and the way of K, V and their terms through memory. us per call, split by every block / ahead:
// B1 H4 S16384 D128 causal 753 / 686, H8 S8192 D64 causal 241 / 217, H16/kvH8 B2 1000 rows on 6000 keys D32 168 / 152,
// H8/kvH1 3810 rows dense D64 117 / 101; not so H8 2048 rows causal D128 75 / 81, H8 1024 rows dense D64 21 / 27. Over 130
// random calls (300 to 16384 rows) the 53 taken ones 0.87 in the mean, 0.96 at worst.
// Not for more (batch, KV head) pairs than the launch ahead has blocks in y; the step itself has its heads in x.
template <int DR>
bool split_ahead(const StepArgs& a) {
  if (static_cast<long long>(a.B) * a.kvH > 65535) return false;
  long long steps = 0;  // of one head
  const int per_seg = (a.qmap.seg_len + 2 * kBM - 1) / (2 * kBM);
  for (int sq = 0; sq < a.qmap.n_seg; ++sq)
    for (int tq = 0; tq < per_seg; ++tq) {
      const int row0 = tq * 2 * kBM, rows = std::min(2 * kBM, a.qmap.seg_len - row0);
      const int qmin = a.qmap.base[sq] + row0 * a.stride;
      for (int sk = 0; sk < a.kmap.n_seg; ++sk) {
        const TileRange r = tile_range<kBNf>(a.kmap, sk, a.stride, (a.flags & RA_STEP_CAUSAL) != 0, a.doc_len, qmin,
                                             qmin + (rows - 1) * a.stride);
        steps += r.hi - r.lo;
      }
    }
  constexpr double kSaves = DR == 128 ? 0.35 : 0.3, kLaunch = 5, kBytesPerUs = 5e6;
  const double bytes = 16.0 * a.B * a.kvH * split_tiles(a) * kBNf * DR;  // read and written
  return kSaves * a.B * a.H * steps / sm_count() > kLaunch + bytes / kBytesPerUs;
}
template <int DR, bool kSplit, bool kPre>
int launch_f32(const StepArgs& a, cudaStream_t stream, int key_split) {
  using C = F32Cfg<DR, kSplit, kPre>;
  CUtensorMap mk, mv;
  int rc = make_map(&mk, RA_F32, a.k, a.D, a.k_rows, a.k_heads_total, a.kv_head_stride, kBNf);
  if (rc != RA_OK) return rc;
  rc = make_map(&mv, RA_F32, a.v, a.D, a.k_rows, a.k_heads_total, a.kv_head_stride, kBNf);
  if (rc != RA_OK) return rc;
  TcArgs t;
  t.kv_per_wave = 0;
  t.key_split = key_split;
  set_step_form(key_split | (kPre ? 256 : 0));
  t.out = a.out;
  t.m = a.m;
  t.l = a.l;
  t.H = a.H;
  t.kvH = a.kvH;
  t.Sq = a.Sq;
  t.n_qblocks_per_seg = (a.qmap.seg_len + 2 * kBM - 1) / (2 * kBM);
  t.qmap = a.qmap;
  t.kmap = a.kmap;
  for (int i = 0; i < RA_MAX_SEG; ++i) {
    t.kseg_head[i] = a.kseg_head[i];
    t.kseg_row[i] = a.kseg_row[i];
  }
  t.stride = a.stride;
  t.flags = a.flags;
  t.doc_len = a.doc_len;
  t.status = a.status;
  t.wait_ns = tc_wait_limit_ns();
  t.stall_after = tc_stall_after();
  const long long n_qblocks = static_cast<long long>(t.n_qblocks_per_seg) * a.qmap.n_seg;
  RAB_REQUIRE(n_qblocks <= 65535, RA_ERR_INVALID, "attention step: too many query blocks (%lld)",
              n_qblocks);
  SplitKV pre = {};
  if constexpr (kPre) {
    pre.tiles = split_tiles(a);
    const size_t n = static_cast<size_t>(a.B) * a.kvH * pre.tiles;
    pre.k = static_cast<unsigned char*>(a.workspace);
    pre.v = pre.k + n * C::kSlotBytes;
    pre.meta = pre.v + n * C::kSlotBytes;
    for (int i = 0; i < a.kmap.n_seg; ++i) pre.beg[i] = i * (pre.tiles / a.kmap.n_seg);
    RAB_CUDA(launch_overlapped(split_kv_kernel<DR>, dim3(pre.tiles, a.B * a.kvH), dim3(kSplitThreads), 0, stream,
                               static_cast<const float*>(a.k), static_cast<const float*>(a.v), a.kv_head_stride, t, pre, a.k_rows));
  }
  auto kern = step_f32_kernel<DR, kSplit, kPre>;
  static std::atomic<unsigned long long> smem_set{0};  // once per device, see step_tc.cu
  int dev = 0;
  RAB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !(smem_set.load(std::memory_order_acquire) >> dev & 1ull)) {
    RAB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
    if (dev >= 0 && dev < 64) smem_set.fetch_or(1ull << dev, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(a.B) * a.H * (kSplit ? key_split : 1),
                     static_cast<unsigned>(n_qblocks));
  cfg.blockDim = dim3(C::kThreads);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = key_split;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = kSplit ? 2 : 1;
  RAB_CUDA(cudaLaunchKernelEx(&cfg, kern, mk, mv, static_cast<const float*>(a.q), static_cast<const float*>(a.k),
                              a.kv_head_stride, t, pre));
  RAB_CUDA(cudaGetLastError());
  return RA_OK;
}

template <int DR>
int launch_f32_d(const StepArgs& a, cudaStream_t stream) {
  const int* slots = nullptr;
  const int rc = cluster_slots(step_f32_kernel<DR, true, false>, kThreadsF, F32Cfg<DR, true>::kSmemBytes, &slots);
  if (rc != RA_OK) return rc;
  // (a merge in tiles: those of head_dim 128 take longer)
  const int split = pick_key_split<kBNf>(a, 2 * kBM, DR == 128 ? 1.5 : 2.5, slots);
  if (a.workspace != nullptr && a.workspace_bytes >= split_bytes<DR>(a) && (reinterpret_cast<uintptr_t>(a.workspace) & 127u) == 0 &&
      split_ahead<DR>(a))
    return split > 1 ? launch_f32<DR, true, true>(a, stream, split) : launch_f32<DR, false, true>(a, stream, 1);
  return split > 1 ? launch_f32<DR, true, false>(a, stream, split) : launch_f32<DR, false, false>(a, stream, 1);
}

}  // namespace

bool step_f32_supported(int dtype, const StepArgs& a) {
  if (dtype != RA_F32) return false;
  if (a.D != 32 && a.D != 64 && a.D != 128) return false;
  if (a.Sq <= 0 || a.Sk <= 0) return false;
  if (a.qmap.n_seg * a.qmap.seg_len != a.Sq || a.kmap.n_seg * a.kmap.seg_len != a.Sk) return false;
  if ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) |
       reinterpret_cast<uintptr_t>(a.v) | reinterpret_cast<uintptr_t>(a.out)) & 15u)
    return false;
  return true;
}

size_t step_f32_workspace_bytes(const StepArgs& a) {
  if (a.D == 32) return split_ahead<32>(a) ? split_bytes<32>(a) : 0;
  if (a.D == 64) return split_ahead<64>(a) ? split_bytes<64>(a) : 0;
  return split_ahead<128>(a) ? split_bytes<128>(a) : 0;
}

int launch_step_f32(const StepArgs& a, cudaStream_t stream) {
  RAB_REQUIRE(a.status != nullptr, RA_ERR_CUDA, "attention step: no device status word");
  if (a.D == 32) return launch_f32_d<32>(a, stream);
  if (a.D == 64) return launch_f32_d<64>(a, stream);
  return launch_f32_d<128>(a, stream);
}

}  // namespace rab

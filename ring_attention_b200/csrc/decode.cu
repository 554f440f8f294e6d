// Split-K decode (seq_q == 1) against a KV cache read in place: the HBM-bound half of the
// hot path. Replaces the reference's split + reduce kernels (src/attention_decode.cu:73-277).
//
// What bounds it: every K and V row of the local shard is read exactly once from HBM, so
// the kernels are built around bytes in flight, not arithmetic.
//  - A block serves ALL query heads that map to that KV
//    head (h % kv_heads), so grouped-query attention reads each cached row once instead of
//    once per query head (the reference re-reads it per head, src/attention_decode.cu:88).
//  - How the cached rows are dealt to blocks: see Deal.
//  - decode_mma_kernel (fp16 / bf16 caches, head_dim >= 64) is the fast path: K/V rows stream
//    through a 3-6-stage shared-memory ring of 64-key stages filled with 16-byte cp.async
//    copies (fully coalesced, XOR-swizzled), and per 16-key block a warp does both
//    contractions on mma.sync m16n8k16 with the up to 16 grouped query heads as M rows
//    (ldmatrix / ldmatrix.trans), online softmax with warp-shuffle row maxima and a lazy
//    rescale; warps are merged through shared memory. The tensor cores are there to get under
//    the instruction-issue bound (about 5 instead of about 80 warp instructions per cached
//    row), the kernel is bound by the copy. Two blocks of 96 KB of ring per SM: the loads of one
//    run on through the barriers and the arithmetic of the other (B4 H32/kvH8 D128, 262144 rows:
//    one block of 160 KB 799 us, two of 96 KB 591-635 us = 6.8-7.25 TB/s).
//  - decode_split_kernel (fp32 caches, head_dim 32; one and two query heads to a KV head) is the SIMT form of the same structure
//    with a 4-stage ring: a group of `LPR` lanes owns a row, each lane keeps its slice of q
//    (pre-scaled) for every head of the group, the dot product finishes with log2(LPR)
//    shuffles, each lane group carries its own running (m, l, out), and a warp-shuffle
//    log-sum-exp merge plus one shared-memory pass combine lane groups and warps.
//  - decode_group_kernel: the same caches with more query heads to a KV head, four or eight a block. There the
//    instructions count, and one butterfly serves the scores of all heads.
// Partials (m, l, out) go to a workspace and a second small kernel folds them into the persistent
// state (src/attention_decode.cu:228-277 does the same for its fixed 8 splits); short calls merge
// them inside a cluster instead.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "tc_common.cuh"

namespace rab {

namespace {

using tcgen::cluster_addr;
using tcgen::cluster_ctarank;
using tcgen::cluster_sync_threads;
using tcgen::ex2;
using tcgen::fadd2;
using tcgen::ffma2;
using tcgen::kLn2;
using tcgen::kLog2e;
using tcgen::ld_cluster_f4;
using tcgen::smem_u32;

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kStages = 4;
constexpr int kMaxSplits = 128;

__device__ inline void cp_async16(void* smem_dst, const void* gsrc, int src_bytes) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gsrc),
               "r"(src_bytes)
               : "memory");
}
__device__ inline void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ inline void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Unpack one 16-byte piece into floats.
template <typename T>
struct Piece;
template <>
struct Piece<float> {
  static constexpr int kElems = 4;
  __device__ static void unpack(const uint4& u, float* f) {
    f[0] = __uint_as_float(u.x);
    f[1] = __uint_as_float(u.y);
    f[2] = __uint_as_float(u.z);
    f[3] = __uint_as_float(u.w);
  }
};
template <>
struct Piece<__half> {
  static constexpr int kElems = 8;
  __device__ static void unpack(const uint4& u, float* f) {
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      f[2 * i] = x.x;
      f[2 * i + 1] = x.y;
    }
  }
};
template <>
struct Piece<__nv_bfloat16> {
  static constexpr int kElems = 8;
  __device__ static void unpack(const uint4& u, float* f) {
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // bf16 -> fp32 is a 16-bit shift
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};

// decode_split_kernel: every lane owns 1..4 pieces of a row.
template <typename T, int D>
struct DecodeCfg {
  static constexpr int kRowBytes = D * static_cast<int>(sizeof(T));
  static constexpr int kPieces = kRowBytes / 16;  // 16-byte pieces per row
  static constexpr int kLPR = kPieces >= 32 ? 16 : (kPieces >= 8 ? 8 : 4);
  static constexpr int kVPT = kPieces / kLPR;               // pieces per lane
  static constexpr int kEPL = kVPT * Piece<T>::kElems;      // elements per lane
  static constexpr int kRowsPerWarpStep = 32 / kLPR;
  static constexpr int kRowsPerStep = kWarps * kRowsPerWarpStep;
  static constexpr int kSteps = 8192 / (kRowsPerStep * kRowBytes) > 0 ? 8192 / (kRowsPerStep * kRowBytes) : 1;
  static constexpr int kRowsPerStage = kRowsPerStep * kSteps;  // 8 KB per tensor and stage
  static constexpr int kStageBytes = kRowsPerStage * kRowBytes;  // per tensor
  static constexpr int kSmemBytes = 2 * kStages * kStageBytes;
};

// decode_group_kernel: a lane owns four columns of a row, or eight at head_dim 256, and a warp takes kSets times kRows rows of
// each of its 32 / kLPR lane groups at a time.
template <typename T, int D, int GB>
struct GroupCfg {
  static constexpr int kRowBytes = D * static_cast<int>(sizeof(T));
  static constexpr int kPieceBytes = 4 * static_cast<int>(sizeof(T));
  static constexpr int kLPR = D / 4 < 32 ? D / 4 : 32;
  static constexpr int kVPT = D / 4 / kLPR;
  static constexpr int kEPL = 4 * kVPT;
  static constexpr int kRows = D == 256 ? 2 : (kLPR / GB < 4 ? kLPR / GB : 4);
  static constexpr int kScores = kRows * GB;  // of a lane group; no more than it has lanes
  static constexpr int kGroups = 32 / kLPR;
  static constexpr int kSets = sizeof(T) == 2 ? 2 : 1;  // such sets of scores a step
  static constexpr int kRowsPerWarpStep = kGroups * kRows * kSets;
  static constexpr int kWarps =
      8192 / kRowBytes / kRowsPerWarpStep < 8 ? 8192 / kRowBytes / kRowsPerWarpStep : 8;
  static constexpr int kThreads = kWarps * 32;
  static constexpr int kRowsPerStep = kWarps * kRowsPerWarpStep;
  static constexpr int kSteps = 8192 / (kRowsPerStep * kRowBytes);
  static constexpr int kRowsPerStage = kRowsPerStep * kSteps;
  static constexpr int kStageBytes = kRowsPerStage * kRowBytes;  // per tensor
  static constexpr int kSmemBytes = 2 * kStages * kStageBytes;
  // Whether the rows of a step are added up by themselves before they reach the accumulators: fewer terms one after
  // another there. So where a block has fewer lane groups, or (at head_dim 32) an SM fewer blocks or a row more lanes, than in
  // the kernel above, whose error against 64 bits is not to be exceeded: 16 bits, head_dim 32, B5 H64/kvH16 150000 rows 4.8e-7
  // so, 6.5e-7 without, H64/kvH8 3.5e-7 and 5.0e-7. (Elsewhere the errors are those of before either way, and the
  // additions cost B5 H48/kvH6 D64, 55149 rows 175 us instead of 159.)
  static constexpr bool kSumFirst = kRows * kSets > 1 && (kWarps < 8 || D == 32);
  static_assert(kStageBytes == 8192 && kScores <= kLPR, "8 KB per tensor and stage, a score for each lane and set");
};

// ---- how the keys are dealt to blocks ----------------------------------------------------
//
// A group is one (batch row, KV head, batch of query heads); its visible rows are `stages` ring
// stages. Two forms of the same kernels:
//  * balanced: one block per resident slot of the GPU, block i takes the stages
//    [i T / G, (i + 1) T / G) of all T = groups * stages, whatever groups they belong to (one or
//    two, more when groups are short). Every block moves the same bytes, so there is no last wave:
//    with a fixed number of splits per group the long-context shape (B4 kvH8, 262144 rows) made
//    448 blocks for 148 SMs, three waves and four blocks. A block leaves one partial per
//    group it touches in the workspace and a second kernel folds them. Measured with 160 KB rings
//    it made no difference by itself (799 against 769 us); with two blocks per SM 1, 3 or 6 times as
//    many blocks were no faster either, and the B1 H8 D128 fp32 call on 16384 rows slower (37 us
//    against 31).
//  * cluster: the blocks of a cluster take equal shares of ONE group and merge
//    their partials through distributed shared memory into the state. No workspace and no second
//    launch: for calls that one wave finishes in a few microseconds (B1 H32/kvH8 D128 fp16 on 1061
//    rows 11.5 -> 9.3 us per call, most of it host time).
enum DealForm { kBalanced, kCluster };
struct Deal {
  int stages;          // per group
  int groups;
  int head_batches;
  int cap;             // partial slots per (batch, head) row
  int ring;            // ring slots (no more than a block's stages)
  unsigned flags;      // cluster form: RA_STEP_FRESH / RA_STEP_FINALIZE
};
// The block that owns stage x of the balanced form: the largest i with floor(i T / G) <= x.
__host__ __device__ inline int deal_owner(long long x, long long total, int ctas) {
  return static_cast<int>(((x + 1) * ctas - 1) / total);
}

__device__ inline float ld_cluster_f1(unsigned addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

constexpr int kMaxCluster = 8;

// Four floats of a workspace or a state, which need not be 16-byte aligned.
__device__ inline float4 ld4(const float* p, bool vec) {
  return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ inline void st4(float* p, float4 v, bool vec) {
  if (vec) *reinterpret_cast<float4*>(p) = v;
  else p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
}
__device__ inline void add_scaled(float4& a, float f, float4 v) {
  a.x += f * v.x;
  a.y += f * v.y;
  a.z += f * v.z;
  a.w += f * v.w;
}

// End of a block's share of a group: the warps' partials (red_*: [warps][ROWS], red_o [..][D]) of
// the ROWS query heads h = kvh + kvH * (hb * ROWS + r) become the block's, which goes to slot
// `part` of the workspace or is merged over the cluster and folded into the state.
template <int ROWS, int D, int NWARPS, DealForm kForm>
__device__ inline void finish_group(float* red_m, float* red_l, float* red_o, int b, int kvh, int hb, int H,
                                    int kvH, int part, const Deal& deal, float* Mp, float* Lp,
                                    float* Op) {
  constexpr int kThr = NWARPS * 32;
  const int tid = threadIdx.x;
  const int first = kvh + kvH * hb * ROWS;
  const int live = first < H ? min(ROWS, (H - first + kvH - 1) / kvH) : 0;
  float* blk_m = red_o + NWARPS * ROWS * D;  // [ROWS], [ROWS], [ROWS][D]: cluster form
  float* blk_l = blk_m + ROWS;
  float* blk_o = blk_m + ((2 * ROWS + 3) & ~3);
  for (int idx = 4 * tid; idx < live * D; idx += 4 * kThr) {  // four columns at a time
    const int r = idx / D;
    const int d = idx - r * D;
    float m_n = -INFINITY;
#pragma unroll
    for (int w = 0; w < NWARPS; ++w) m_n = fmaxf(m_n, red_m[w * ROWS + r]);
    float4 o_acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float l_acc = 0.f;
#pragma unroll
    for (int w = 0; w < NWARPS; ++w) {
      const float mw = red_m[w * ROWS + r];
      const float sc = (mw == -INFINITY) ? 0.f : ex2(mw - m_n);
      const float4 o = *reinterpret_cast<const float4*>(red_o + (w * ROWS + r) * D + d);
      o_acc.x += sc * o.x;
      o_acc.y += sc * o.y;
      o_acc.z += sc * o.z;
      o_acc.w += sc * o.w;
      l_acc += sc * red_l[w * ROWS + r];
    }
    // natural-log units, the unit of the persistent state
    if constexpr (kForm == kCluster) {
      *reinterpret_cast<float4*>(blk_o + idx) = o_acc;
      if (d == 0) {
        blk_m[r] = m_n * kLn2;
        blk_l[r] = l_acc;
      }
    } else {
      const size_t slot = (static_cast<size_t>(b) * H + first + kvH * r) * deal.cap + part;
      float* dst = Op + slot * D + d;
      st4(dst, o_acc, (reinterpret_cast<uintptr_t>(dst) & 15u) == 0);
      if (d == 0) {
        Mp[slot] = m_n * kLn2;
        Lp[slot] = l_acc;
      }
    }
  }
  if constexpr (kForm == kCluster) {
    // Mp / Lp / Op are the state itself here
    const bool fresh = (deal.flags & RA_STEP_FRESH) != 0, finalize = (deal.flags & RA_STEP_FINALIZE) != 0;
    const int n = static_cast<int>(gridDim.x), rank = static_cast<int>(cluster_ctarank());
    cluster_sync_threads();  // every block's partial is staged
    // (m, l) of row r in every block, all loads in flight at once; then what the maxima make of them:
    // the factors of the blocks' partials (f), the factor of the old state (returned), the sum
    auto load_ml = [&](int r, float (&f)[kMaxCluster], float (&ls)[kMaxCluster]) {
#pragma unroll
      for (int i = 0; i < kMaxCluster; ++i) {
        f[i] = i < n ? ld_cluster_f1(cluster_addr(smem_u32(blk_m + r), i)) : -INFINITY;
        ls[i] = i < n ? ld_cluster_f1(cluster_addr(smem_u32(blk_l + r), i)) : 0.f;
      }
    };
    auto factors = [&](size_t row, float (&f)[kMaxCluster], const float (&ls)[kMaxCluster], float& m_n, float& l_acc) {
      const float m_old = fresh ? -INFINITY : Mp[row];
      m_n = m_old;
#pragma unroll
      for (int i = 0; i < kMaxCluster; ++i) m_n = fmaxf(m_n, f[i]);
      const float a = (m_old == -INFINITY) ? 0.f : expf(m_old - m_n);
      l_acc = (m_old == -INFINITY) ? 0.f : a * Lp[row];
#pragma unroll
      for (int i = 0; i < kMaxCluster; ++i) {
        f[i] = (f[i] == -INFINITY) ? 0.f : expf(f[i] - m_n);
        l_acc += f[i] * ls[i];
      }
      return a;
    };
    for (int idx = 4 * (rank * kThr + tid); idx < live * D; idx += 4 * n * kThr) {
      const int r = idx / D;
      const size_t row = static_cast<size_t>(b) * H + first + kvH * r;
      float* dst = Op + row * D + (idx - r * D);
      const bool vec = (reinterpret_cast<uintptr_t>(dst) & 15u) == 0;
      float f[kMaxCluster], ls[kMaxCluster], m_n, l_acc;
      float4 o[kMaxCluster], acc = make_float4(0.f, 0.f, 0.f, 0.f);
      load_ml(r, f, ls);
#pragma unroll
      for (int i = 0; i < kMaxCluster; ++i) o[i] = i < n ? ld_cluster_f4(cluster_addr(smem_u32(blk_o + idx), i)) : acc;
      const float a = factors(row, f, ls, m_n, l_acc);
      if (m_n == -INFINITY) {
        // nothing visible anywhere: the state stays as it is (or is written empty)
        if (fresh || finalize) st4(dst, acc, vec);
        continue;
      }
      if (!fresh && Mp[row] > -INFINITY) add_scaled(acc, a, ld4(dst, vec));
#pragma unroll
      for (int i = 0; i < kMaxCluster; ++i) add_scaled(acc, f[i], o[i]);
      if (finalize) {
        const float inv = l_acc > 0.f ? 1.f / l_acc : 0.f;
        acc = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
      }
      st4(dst, acc, vec);
    }
    // (m, l) of a row once every block has read the old ones and nobody needs this block any more
    float m_n = -INFINITY, l_acc = 0.f;
    const bool owner = rank == 0 && tid < live;
    size_t row = 0;
    if (owner) {
      row = static_cast<size_t>(b) * H + first + kvH * tid;
      float f[kMaxCluster], ls[kMaxCluster];
      load_ml(tid, f, ls);
      factors(row, f, ls, m_n, l_acc);
    }
    cluster_sync_threads();
    if (owner && (m_n > -INFINITY || m_n != m_n || fresh)) {
      Mp[row] = m_n;
      Lp[row] = m_n == -INFINITY ? 0.f : l_acc;
    }
  }
}

// Floats of shared memory that a block's end takes: (m, l, O) by warp, then the block's.
constexpr size_t red_floats(int warps, int rows, int D) {
  return static_cast<size_t>(warps) * rows * (D + 2) + ((2 * rows + 3) & ~3) + static_cast<size_t>(rows) * D;
}

// A block's next share: stages [beg, end) of the group (b, kvh, hb), partial slot `part`. Only the balanced form
// has more than one.
struct Share {
  int beg, end, part, hb, kvh, b;
};
template <DealForm kForm>
struct Shares {
  long long total, at, at_end;
  int n, i;
  __device__ explicit Shares(const Deal& deal) {
    n = static_cast<int>(gridDim.x);
    i = static_cast<int>(blockIdx.x);
    total = static_cast<long long>(deal.groups) * deal.stages;
    at = kForm == kBalanced ? total * i / n : 0;
    at_end = kForm == kBalanced ? total * (i + 1ll) / n : 1;
    let_next_start();
    wait_for_previous();
  }
  __device__ bool next(const Deal& deal, int kvH, Share& s) {
    if (at >= at_end) return false;
    const int group = static_cast<int>(kForm == kBalanced ? at / deal.stages : blockIdx.y);
    if (kForm == kBalanced) {
      const long long first = static_cast<long long>(group) * deal.stages;
      s.beg = static_cast<int>(at - first);
      s.end = static_cast<int>(min(static_cast<long long>(deal.stages), s.beg + (at_end - at)));
      s.part = i - deal_owner(first, total, n);
      at += s.end - s.beg;
    } else {
      s.beg = static_cast<int>(static_cast<long long>(deal.stages) * i / n);
      s.end = static_cast<int>(static_cast<long long>(deal.stages) * (i + 1ll) / n);
      s.part = i;
      at = at_end;
    }
    s.hb = group % deal.head_batches;
    s.kvh = (group / deal.head_batches) % kvH;
    s.b = group / (deal.head_batches * kvH);
    return true;
  }
};

// GB = query heads handled per block. Grid: see Deal.
template <typename T, int D, int GB, DealForm kForm>
__global__ void __launch_bounds__(kThreads)
    decode_split_kernel(const T* Q, const T* K, const T* V,
                        float* Mp, float* Lp, float* Op, int H,
                        int kvH, int sk_eff, long long kv_head_stride, const Deal deal, float scale_log2) {
  using C = DecodeCfg<T, D>;
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char* k_ring = smem;
  unsigned char* v_ring = smem + deal.ring * C::kStageBytes;

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int lr = lane % C::kLPR;       // lane within the row group
  const int grp = lane / C::kLPR;      // row group within the warp
  Shares<kForm> shares(deal);
  Share share;
  while (shares.next(deal, kvH, share)) {
    const int b = share.b, kvh = share.kvh, hb = share.hb;

    // Query heads of this block: h = kvh + kvH * (hb * GB + g), while h < H.
    float q_reg[GB][C::kEPL];
    float o_reg[GB][C::kEPL];
    float m_run[GB], l_run[GB];
#pragma unroll
    for (int g = 0; g < GB; ++g) {
      const int h = kvh + kvH * (hb * GB + g);
      m_run[g] = -INFINITY;
      l_run[g] = 0.f;
#pragma unroll
      for (int v = 0; v < C::kVPT; ++v) {
        float f[Piece<T>::kElems];
        if (h < H) {
          const uint4 u = *reinterpret_cast<const uint4*>(
              reinterpret_cast<const unsigned char*>(Q + (static_cast<size_t>(b) * H + h) * D) +
              (v * C::kLPR + lr) * 16);
          Piece<T>::unpack(u, f);
        } else {
#pragma unroll
          for (int e = 0; e < Piece<T>::kElems; ++e) f[e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < Piece<T>::kElems; ++e) {
          q_reg[g][v * Piece<T>::kElems + e] = f[e] * scale_log2;
          o_reg[g][v * Piece<T>::kElems + e] = 0.f;
        }
      }
    }

    const int row_begin = share.beg * C::kRowsPerStage;
    const int row_end = min(static_cast<long long>(sk_eff), static_cast<long long>(share.end) * C::kRowsPerStage);
    const int n_rows = row_end - row_begin;
    const int n_stages = share.end - share.beg;
    const unsigned char* k_base = reinterpret_cast<const unsigned char*>(
        K + (static_cast<size_t>(b) * kvH + kvh) * kv_head_stride);
    const unsigned char* v_base = reinterpret_cast<const unsigned char*>(
        V + (static_cast<size_t>(b) * kvH + kvh) * kv_head_stride);

    auto issue = [&](int st) {
      if (st < n_stages) {
        const int slot = st % kStages;
        const long long first = static_cast<long long>(row_begin) + st * C::kRowsPerStage;
        const long long valid_bytes =
            (static_cast<long long>(row_end) - first) * C::kRowBytes;  // > 0
        const size_t goff = static_cast<size_t>(first) * C::kRowBytes;
        for (int p = tid; p < C::kStageBytes / 16; p += kThreads) {
          const long long off = static_cast<long long>(p) * 16;
          const bool ok = off < valid_bytes;
          // past the split: src-size 0 zero-fills the destination, the source is not read
          cp_async16(k_ring + slot * C::kStageBytes + off, ok ? k_base + goff + off : k_base,
                     ok ? 16 : 0);
          cp_async16(v_ring + slot * C::kStageBytes + off, ok ? v_base + goff + off : v_base,
                     ok ? 16 : 0);
        }
      }
      cp_async_commit();
    };

#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) issue(s);

    for (int st = 0; st < n_stages; ++st) {
      cp_async_wait<kStages - 2>();
      __syncthreads();
      issue(st + kStages - 1);
      const int slot = st % kStages;
      const int stage_row0 = st * C::kRowsPerStage;
#pragma unroll 1
      for (int step = 0; step < C::kSteps; ++step) {
        const int rl = step * C::kRowsPerStep + warp * C::kRowsPerWarpStep + grp;
        const bool valid = stage_row0 + rl < n_rows;
        const unsigned char* krow = k_ring + slot * C::kStageBytes + rl * C::kRowBytes;
        const unsigned char* vrow = v_ring + slot * C::kStageBytes + rl * C::kRowBytes;
        float kf[C::kEPL];
#pragma unroll
        for (int v = 0; v < C::kVPT; ++v) {
          const uint4 u = *reinterpret_cast<const uint4*>(krow + (v * C::kLPR + lr) * 16);
          Piece<T>::unpack(u, &kf[v * Piece<T>::kElems]);
        }
        float s[GB];
#pragma unroll
        for (int g = 0; g < GB; ++g) {
          float acc = 0.f;
#pragma unroll
          for (int e = 0; e < C::kEPL; ++e) acc = fmaf(q_reg[g][e], kf[e], acc);
          s[g] = acc;
        }
#pragma unroll
        for (int off = 1; off < C::kLPR; off <<= 1) {
#pragma unroll
          for (int g = 0; g < GB; ++g) s[g] += __shfl_xor_sync(0xffffffffu, s[g], off);
        }
        float vf[C::kEPL];
#pragma unroll
        for (int v = 0; v < C::kVPT; ++v) {
          const uint4 u = *reinterpret_cast<const uint4*>(vrow + (v * C::kLPR + lr) * 16);
          Piece<T>::unpack(u, &vf[v * Piece<T>::kElems]);
        }
        if (valid) {
#pragma unroll
          for (int g = 0; g < GB; ++g) {
            if (s[g] > m_run[g]) {  // rare after the first rows: rescale only when the max moves
              const float alpha = ex2(m_run[g] - s[g]);  // ex2(-inf) = 0 on the first row
              l_run[g] *= alpha;
#pragma unroll
              for (int e = 0; e < C::kEPL; ++e) o_reg[g][e] *= alpha;
              m_run[g] = s[g];
            }
            const float p = ex2(s[g] - m_run[g]);
            l_run[g] += p;
#pragma unroll
            for (int e = 0; e < C::kEPL; ++e) o_reg[g][e] = fmaf(p, vf[e], o_reg[g][e]);
          }
        }
      }
    }
    cp_async_wait<0>();

    // Merge the row groups of the warp (log-sum-exp merge through shuffles) ...
#pragma unroll
    for (int off = C::kLPR; off < 32; off <<= 1) {
#pragma unroll
      for (int g = 0; g < GB; ++g) {
        const float m_o = __shfl_xor_sync(0xffffffffu, m_run[g], off);
        const float l_o = __shfl_xor_sync(0xffffffffu, l_run[g], off);
        const float m_n = fmaxf(m_run[g], m_o);
        const float a = (m_run[g] == -INFINITY) ? 0.f : ex2(m_run[g] - m_n);
        const float c = (m_o == -INFINITY) ? 0.f : ex2(m_o - m_n);
        l_run[g] = a * l_run[g] + c * l_o;
#pragma unroll
        for (int e = 0; e < C::kEPL; ++e) {
          const float o_o = __shfl_xor_sync(0xffffffffu, o_reg[g][e], off);
          o_reg[g][e] = a * o_reg[g][e] + c * o_o;
        }
        m_run[g] = m_n;
      }
    }
    // ... then the warps of the block through shared memory (the ring is idle now).
    __syncthreads();
    float* red_m = reinterpret_cast<float*>(smem);            // [kWarps][GB]
    float* red_l = red_m + kWarps * GB;                        // [kWarps][GB]
    float* red_o = red_l + kWarps * GB;                        // [kWarps][GB][D]
    if (grp == 0) {
#pragma unroll
      for (int g = 0; g < GB; ++g) {
        if (lr == 0) {
          red_m[warp * GB + g] = m_run[g];
          red_l[warp * GB + g] = l_run[g];
        }
#pragma unroll
        for (int v = 0; v < C::kVPT; ++v)
#pragma unroll
          for (int e = 0; e < Piece<T>::kElems; ++e)
            red_o[(warp * GB + g) * D + (v * C::kLPR + lr) * Piece<T>::kElems + e] =
                o_reg[g][v * Piece<T>::kElems + e];
      }
    }
    __syncthreads();
    finish_group<GB, D, kWarps, kForm>(red_m, red_l, red_o, b, kvh, hb, H, kvH, share.part, deal, Mp, Lp, Op);
    if (kForm == kBalanced) __syncthreads();  // the ring is free again
  }
}

// ---- four and eight query heads to a KV head ---------------------------------------------------
//
// The kernel above finishes every head's dot product with a butterfly of its own and works out the
// softmax of every head in every lane. Here a lane's kRows x GB partial sums go through ONE butterfly that halves their
// number at each exchange and leaves one (row, head) score a lane. No value is selected on the way: register j of a
// lane holds head j ^ (lane % GB) and row i is row i ^ (lane / GB % kRows), so what a lane keeps and what it
// gives away are the same registers in all of them. The softmax is one exponential a lane, the
// weights go to all lanes through shared memory, both contractions are packed FMAs, and a step's rows are added up before they
// reach the accumulators where kSumFirst says so (without that the error against 64 bits grew from 2.4e-7 to 2.9e-7 on 40000 rows: an SM has fewer
// warps than before, so each adds more rows). With eight heads of 128 about 80 instead of 180 instructions a row and warp, 16
// instead of 40 of them shuffles. Two sets of rows a step, in 16 bits, share the maximum, the barrier and the reading of the
// weights (64 random calls of head_dim 32: 0.97 of the time with one). fp32, eight heads, before / now (floor of the copy): B1 H64/kvH8 D256 135081 rows 939 / 332 us
// (338), B3 H48/kvH6 D128 179592 rows 1073 / 508 (505), B1 H32/kvH4 D128 16049 rows 31 / 20 (10); bf16 rows of 32, B2 H32/kvH4
// 225843 rows 179 / 96 (35). Four heads were near the copy in long calls (B3 H64/kvH16 D64 162905 rows 578 / 548);
// short ones are 3 to 25 % faster (B2 H12/kvH4 D128 683 rows 8.2 / 6.9). 110 random calls: 0.85 in the mean, 0.99 at worst.
// One and two heads stay with the kernel above: a row costs it 17 to 35 instructions there, below what its copy takes.
template <typename T>
__device__ inline void load_four(const unsigned char* p, float (&f)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    f[0] = x.x, f[1] = x.y, f[2] = x.z, f[3] = x.w;
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    float g[8];
    Piece<T>::unpack(make_uint4(u.x, u.y, 0, 0), g);
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = g[e];
  }
}

template <typename T, int D, int GB, DealForm kForm>
__global__ void __launch_bounds__(GroupCfg<T, D, GB>::kThreads)
    decode_group_kernel(const T* Q, const T* K, const T* V, float* Mp, float* Lp, float* Op, int H, int kvH, int sk_eff,
                        long long kv_head_stride, const Deal deal, float scale_log2) {
  using C = GroupCfg<T, D, GB>;
  constexpr int kR = C::kRows, kAll = kR * C::kSets;
  extern __shared__ __align__(16) unsigned char smem[];
  // a warp's weights of one step; two buffers, so that one barrier a step is enough
  __shared__ __align__(16) float weights[C::kWarps][2][C::kGroups * C::kScores * C::kSets];
  unsigned char* k_ring = smem;
  unsigned char* v_ring = smem + deal.ring * C::kStageBytes;

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int lr = lane % C::kLPR;   // lane within the row group
  const int grp = lane / C::kLPR;  // row group within the warp
  const int my_head = lr % GB, my_row = lr / GB % kR;
  const int base = lane - lr;
  const bool lead = lr < C::kScores;
  Shares<kForm> shares(deal);
  Share share;
  int buf = 0;
  while (shares.next(deal, kvH, share)) {
    const int b = share.b, kvh = share.kvh, hb = share.hb;

    // Query heads of this block: h = kvh + kvH * (hb * GB + g), while h < H.
    float2 q2[GB][C::kEPL / 2];  // (column, column + 1) of head j ^ my_head
    float2 o2[GB / 2][C::kEPL];  // (head 2 j, head 2 j + 1) of a column
    float m_run = -INFINITY, l_run = 0.f;    // of my_head over the rows of this group of lanes; l_run of my_row only
#pragma unroll
    for (int j = 0; j < GB; ++j) {
      const int h = kvh + kvH * (hb * GB + (j ^ my_head));
#pragma unroll
      for (int v = 0; v < C::kVPT; ++v) {
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (h < H)
          load_four<T>(reinterpret_cast<const unsigned char*>(Q + (static_cast<size_t>(b) * H + h) * D) +
                           (v * C::kLPR + lr) * C::kPieceBytes,
                       f);
        q2[j][2 * v] = make_float2(f[0] * scale_log2, f[1] * scale_log2);
        q2[j][2 * v + 1] = make_float2(f[2] * scale_log2, f[3] * scale_log2);
      }
    }
#pragma unroll
    for (int j = 0; j < GB / 2; ++j)
#pragma unroll
      for (int e = 0; e < C::kEPL; ++e) o2[j][e] = make_float2(0.f, 0.f);

    const int row_begin = share.beg * C::kRowsPerStage;
    const int row_end = min(static_cast<long long>(sk_eff), static_cast<long long>(share.end) * C::kRowsPerStage);
    const int n_rows = row_end - row_begin;
    const int n_stages = share.end - share.beg;
    const unsigned char* k_base = reinterpret_cast<const unsigned char*>(
        K + (static_cast<size_t>(b) * kvH + kvh) * kv_head_stride + static_cast<size_t>(row_begin) * D);
    const unsigned char* v_base = reinterpret_cast<const unsigned char*>(
        V + (static_cast<size_t>(b) * kvH + kvh) * kv_head_stride + static_cast<size_t>(row_begin) * D);
    const long long share_bytes = static_cast<long long>(n_rows) * C::kRowBytes;

    auto issue = [&](int st) {
      if (st < n_stages) {
        const int slot = st % kStages;
        const long long first = static_cast<long long>(st) * C::kStageBytes;
#pragma unroll
        for (int p = 0; p < C::kStageBytes / 16 / C::kThreads; ++p) {
          const int off = (p * C::kThreads + tid) * 16;
          const bool ok = first + off < share_bytes;
          // past the share: src-size 0 zero-fills the destination, the source is not read
          cp_async16(k_ring + slot * C::kStageBytes + off, ok ? k_base + first + off : k_base, ok ? 16 : 0);
          cp_async16(v_ring + slot * C::kStageBytes + off, ok ? v_base + first + off : v_base, ok ? 16 : 0);
        }
      }
      cp_async_commit();
    };

#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) issue(s);

    for (int st = 0; st < n_stages; ++st) {
      cp_async_wait<kStages - 2>();
      __syncthreads();
      issue(st + kStages - 1);
      const int slot = st % kStages;
#pragma unroll 1
      for (int step = 0; step < C::kSteps; ++step) {
        // row i of lane group g: first + i * kGroups + g; kR of them make a set
        const int first = step * C::kRowsPerStep + warp * C::kRowsPerWarpStep + grp;
        const unsigned char* krow = k_ring + slot * C::kStageBytes + first * C::kRowBytes + lr * C::kPieceBytes;
        const unsigned char* vrow = v_ring + slot * C::kStageBytes + first * C::kRowBytes + lr * C::kPieceBytes;
        float score[C::kSets];
        bool valid[C::kSets];
        float m_new = -INFINITY;
#pragma unroll
        for (int set = 0; set < C::kSets; ++set) {
          float s[kR][GB];
#pragma unroll
          for (int i = 0; i < kR; ++i) {
            float2 acc[GB];
#pragma unroll
            for (int j = 0; j < GB; ++j) acc[j] = make_float2(0.f, 0.f);
#pragma unroll
            for (int v = 0; v < C::kVPT; ++v) {
              float f[4];
              load_four<T>(krow + (set * kR + (i ^ my_row)) * C::kGroups * C::kRowBytes + v * C::kLPR * C::kPieceBytes, f);
              const float2 k0 = make_float2(f[0], f[1]), k1 = make_float2(f[2], f[3]);
#pragma unroll
              for (int j = 0; j < GB; ++j) {
                acc[j] = ffma2(q2[j][2 * v], k0, acc[j]);
                acc[j] = ffma2(q2[j][2 * v + 1], k1, acc[j]);
              }
            }
#pragma unroll
            for (int j = 0; j < GB; ++j) s[i][j] = acc[j].x + acc[j].y;
          }
#pragma unroll
          for (int half = kR / 2; half > 0; half /= 2)
#pragma unroll
            for (int i = 0; i < half; ++i)
#pragma unroll
              for (int j = 0; j < GB; ++j) s[i][j] += __shfl_xor_sync(0xffffffffu, s[i + half][j], half * GB);
#pragma unroll
          for (int half = GB / 2; half > 0; half /= 2)
#pragma unroll
            for (int j = 0; j < half; ++j) s[0][j] += __shfl_xor_sync(0xffffffffu, s[0][j + half], half);
          score[set] = s[0][0];
#pragma unroll
          for (int off = C::kScores; off < C::kLPR; off *= 2) score[set] += __shfl_xor_sync(0xffffffffu, score[set], off);
          valid[set] = st * C::kRowsPerStage + first + (set * kR + my_row) * C::kGroups < n_rows;
          m_new = fmaxf(m_new, valid[set] ? score[set] : -INFINITY);
        }
#pragma unroll
        for (int off = GB; off < C::kScores; off *= 2) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, off));
        m_new = fmaxf(m_run, m_new);
        if (__any_sync(0xffffffffu, m_new > m_run)) {  // rare after the first rows: rescale only when a maximum moves
          const float alpha = m_new > m_run ? ex2(m_run - m_new) : 1.f;  // ex2(-inf) = 0 on the first row
          l_run *= alpha;
          m_run = m_new;
#pragma unroll
          for (int j = 0; j < GB / 2; ++j) {
            const float2 a = make_float2(__shfl_sync(0xffffffffu, alpha, base + 2 * j),
                                               __shfl_sync(0xffffffffu, alpha, base + 2 * j + 1));
#pragma unroll
            for (int e = 0; e < C::kEPL; ++e) o2[j][e] = ffma2(o2[j][e], a, make_float2(0.f, 0.f));
          }
        }
        float* w = weights[warp][buf];
        buf ^= 1;
        float l_step = 0.f;
#pragma unroll
        for (int set = 0; set < C::kSets; ++set) {
          const float p = valid[set] && score[set] != -INFINITY ? ex2(score[set] - m_run) : 0.f;
          l_step += p;
          if (lead) w[(grp * C::kSets + set) * C::kScores + lr] = p;
        }
        l_run += l_step;
        __syncwarp();
        float2 p2[kAll][GB / 2];
#pragma unroll
        for (int i = 0; i < kAll; ++i)
#pragma unroll
          for (int j = 0; j < GB / 4; ++j) {
            const float4 x = *reinterpret_cast<const float4*>(w + grp * C::kSets * C::kScores + i * GB + 4 * j);
            p2[i][2 * j] = make_float2(x.x, x.y);
            p2[i][2 * j + 1] = make_float2(x.z, x.w);
          }
#pragma unroll
        for (int v = 0; v < C::kVPT; ++v) {
          float f[kAll][4];
#pragma unroll
          for (int i = 0; i < kAll; ++i)
            load_four<T>(vrow + i * C::kGroups * C::kRowBytes + v * C::kLPR * C::kPieceBytes, f[i]);
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int j = 0; j < GB / 2; ++j) {
              float2& o = o2[j][4 * v + e];
              if constexpr (!C::kSumFirst) {
#pragma unroll
                for (int i = 0; i < kAll; ++i) o = ffma2(p2[i][j], make_float2(f[i][e], f[i][e]), o);
              } else {
                float2 sum = ffma2(p2[0][j], make_float2(f[0][e], f[0][e]), make_float2(0.f, 0.f));
#pragma unroll
                for (int i = 1; i < kAll; ++i) sum = ffma2(p2[i][j], make_float2(f[i][e], f[i][e]), sum);
                o = fadd2(o, sum);
              }
            }
        }
      }
    }
    cp_async_wait<0>();

    // Merge the rows of a lane group (they share m_run), then the groups of the warp (log-sum-exp merge) ...
#pragma unroll
    for (int off = GB; off < C::kScores; off *= 2) l_run += __shfl_xor_sync(0xffffffffu, l_run, off);
    __syncthreads();  // the ring is idle now
    float* red_m = reinterpret_cast<float*>(smem);  // [kWarps][GB]
    float* red_l = red_m + C::kWarps * GB;           // [kWarps][GB]
    float* red_o = red_l + C::kWarps * GB;           // [kWarps][GB][D]
#pragma unroll
    for (int g = 0; g < GB; ++g) {
      float m_g = __shfl_sync(0xffffffffu, m_run, base + g), l_g = __shfl_sync(0xffffffffu, l_run, base + g);
      float o_g[C::kEPL];
#pragma unroll
      for (int e = 0; e < C::kEPL; ++e) o_g[e] = g % 2 ? o2[g / 2][e].y : o2[g / 2][e].x;
#pragma unroll
      for (int off = C::kLPR; off < 32; off *= 2) {
        const float m_o = __shfl_xor_sync(0xffffffffu, m_g, off);
        const float l_o = __shfl_xor_sync(0xffffffffu, l_g, off);
        const float m_n = fmaxf(m_g, m_o);
        const float a = (m_g == -INFINITY) ? 0.f : ex2(m_g - m_n);
        const float c = (m_o == -INFINITY) ? 0.f : ex2(m_o - m_n);
        l_g = a * l_g + c * l_o;
#pragma unroll
        for (int e = 0; e < C::kEPL; ++e) {
          const float o_o = __shfl_xor_sync(0xffffffffu, o_g[e], off);
          o_g[e] = a * o_g[e] + c * o_o;
        }
        m_g = m_n;
      }
      // ... then the warps of the block through shared memory.
      if (grp == 0) {
        if (lr == 0) {
          red_m[warp * GB + g] = m_g;
          red_l[warp * GB + g] = l_g;
        }
#pragma unroll
        for (int v = 0; v < C::kVPT; ++v)
          *reinterpret_cast<float4*>(red_o + (warp * GB + g) * D + (v * C::kLPR + lr) * 4) =
              make_float4(o_g[4 * v], o_g[4 * v + 1], o_g[4 * v + 2], o_g[4 * v + 3]);
      }
    }
    __syncthreads();
    finish_group<GB, D, C::kWarps, kForm>(red_m, red_l, red_o, b, kvh, hb, H, kvH, share.part, deal, Mp, Lp, Op);
    if (kForm == kBalanced) __syncthreads();  // the ring is free again
  }
}

// ---- tensor-core variant for 16-bit caches ---------------------------------------------
//
// The SIMT kernel above spends ~80 warp instructions per cached row (a convert and one FMA
// per element per query head), which makes it issue-bound at well under HBM speed. For
// fp16 / bf16 caches both contractions of a block of 16 keys run on mma.sync m16n8k16
// instead: the (up to 16) query heads that share the KV head are the M rows, so a key row
// costs ~5 instructions and the kernel is bound by the copy into shared memory again.
// K/V rows go to shared memory with the same 16-byte cp.async copies, but each 16-byte
// piece c of row r is stored at piece c ^ (r & 7), so that the ldmatrix reads (8 rows at a
// fixed column) touch all banks once.
constexpr int kMmaKeysPerWarp = 16;

template <typename T>
__device__ inline void mma16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1);
template <>
__device__ inline void mma16816<__half>(float (&c)[4], const unsigned (&a)[4], unsigned b0,
                                        unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ inline void mma16816<__nv_bfloat16>(float (&c)[4], const unsigned (&a)[4], unsigned b0,
                                               unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ inline void ldmatrix_x4(unsigned (&r)[4], unsigned saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(saddr));
}
__device__ inline void ldmatrix_x4_trans(unsigned (&r)[4], unsigned saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(saddr));
}
template <typename T>
__device__ inline unsigned pack_pair(float lo, float hi);
template <>
__device__ inline unsigned pack_pair<__half>(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&h);
}
template <>
__device__ inline unsigned pack_pair<__nv_bfloat16>(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&h);
}

template <int D>
struct MmaCfg {
  static constexpr int kRowBytes = D * 2;
  static constexpr int kPieces = kRowBytes / 16;
  // head_dim 256: two warps and 32-key stages, so that three stages are 96 KB as well and two
  // blocks fit an SM (B3 kvH4 bf16, 34876 rows: 86 us with four warps and 192 KB, 74 so)
  static constexpr int kWarps = D == 256 ? 2 : 4;
  static constexpr int kThreads = kWarps * 32;
  static constexpr int kStageRows = kWarps * kMmaKeysPerWarp;
  static constexpr int kStageBytes = kStageRows * kRowBytes;  // per tensor
  static constexpr int kStages = (96 * 1024) / (2 * kStageBytes);
  static constexpr int kSmemBytes = 2 * kStages * kStageBytes;
};

// A block serves up to 16 query heads of one KV head (rows of the MMA tile; row r is head
// kvh + kv_heads * (16 * hb + r)). Grid: see Deal.
template <typename T, int D, DealForm kForm>
__global__ void __launch_bounds__(MmaCfg<D>::kThreads)
    decode_mma_kernel(const T* Q, const T* K, const T* V,
                      float* Mp, float* Lp, float* Op, int H,
                      int kvH, int sk_eff, long long kv_head_stride, const Deal deal, float scale_log2) {
  using C = MmaCfg<D>;
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char* k_ring = smem;
  unsigned char* v_ring = smem + deal.ring * C::kStageBytes;

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int g = lane >> 2;   // fragment row (and row + 8)
  const int tq = lane & 3;   // fragment column pair
  Shares<kForm> shares(deal);
  Share share;
  while (shares.next(deal, kvH, share)) {
    const int b = share.b, kvh = share.kvh, hb = share.hb;

    // Q as A fragments: reg0 (row g, k 2tq..), reg1 (row g+8, same k), reg2 / reg3 the same at k+8.
    const int h0 = kvh + kvH * (hb * 16 + g);
    const int h1 = kvh + kvH * (hb * 16 + g + 8);
    unsigned qa[D / 16][4];
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      const int d0 = ks * 16 + 2 * tq;
      const T* q0 = Q + (static_cast<size_t>(b) * H + (h0 < H ? h0 : 0)) * D + d0;
      const T* q1 = Q + (static_cast<size_t>(b) * H + (h1 < H ? h1 : 0)) * D + d0;
      qa[ks][0] = h0 < H ? *reinterpret_cast<const unsigned*>(q0) : 0u;
      qa[ks][1] = h1 < H ? *reinterpret_cast<const unsigned*>(q1) : 0u;
      qa[ks][2] = h0 < H ? *reinterpret_cast<const unsigned*>(q0 + 8) : 0u;
      qa[ks][3] = h1 < H ? *reinterpret_cast<const unsigned*>(q1 + 8) : 0u;
    }

    float o[D / 8][4];
#pragma unroll
    for (int n = 0; n < D / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    float m_run[2] = {-INFINITY, -INFINITY};
    float l_run[2] = {0.f, 0.f};  // this lane's share of the row sums (its four columns per block)

    const int row_begin = share.beg * C::kStageRows;
    const int row_end = min(static_cast<long long>(sk_eff), static_cast<long long>(share.end) * C::kStageRows);
    const int n_rows = row_end - row_begin;
    const int n_stages = share.end - share.beg;
    const unsigned char* k_base = reinterpret_cast<const unsigned char*>(
        K + (static_cast<size_t>(b) * kvH + kvh) * kv_head_stride);
    const unsigned char* v_base = reinterpret_cast<const unsigned char*>(
        V + (static_cast<size_t>(b) * kvH + kvh) * kv_head_stride);

    auto issue = [&](int st) {
      if (st < n_stages) {
        const int slot = st % C::kStages;
        const long long first = static_cast<long long>(row_begin) + st * C::kStageRows;
        const long long valid_bytes = (static_cast<long long>(row_end) - first) * C::kRowBytes;
        const size_t goff = static_cast<size_t>(first) * C::kRowBytes;
        for (int p = tid; p < C::kStageBytes / 16; p += C::kThreads) {
          const int r = p / C::kPieces;
          const int c = p - r * C::kPieces;
          const long long off = static_cast<long long>(p) * 16;
          const int dst = slot * C::kStageBytes + r * C::kRowBytes + ((c ^ (r & 7)) << 4);
          const bool ok = off < valid_bytes;
          cp_async16(k_ring + dst, ok ? k_base + goff + off : k_base, ok ? 16 : 0);
          cp_async16(v_ring + dst, ok ? v_base + goff + off : v_base, ok ? 16 : 0);
        }
      }
      cp_async_commit();
    };

#pragma unroll
    for (int s = 0; s < C::kStages - 1; ++s) issue(s);

    const int mi = lane >> 3, r8 = lane & 7;
    const int key0 = warp * kMmaKeysPerWarp;
    // per-lane row offsets of the ldmatrix addresses (piece index is XORed with r8 = key & 7)
    const unsigned k_row_off = static_cast<unsigned>((key0 + (mi >> 1) * 8 + r8) * C::kRowBytes);
    const unsigned v_row_off = static_cast<unsigned>((key0 + (mi & 1) * 8 + r8) * C::kRowBytes);

    for (int st = 0; st < n_stages; ++st) {
      cp_async_wait<C::kStages - 2>();
      __syncthreads();
      issue(st + C::kStages - 1);
      const int slot = st % C::kStages;
      const int n_valid = n_rows - (st * C::kStageRows + key0);  // valid keys of this warp's block
      if (n_valid <= 0) continue;
      const unsigned kt = static_cast<unsigned>(__cvta_generic_to_shared(k_ring + slot * C::kStageBytes));
      const unsigned vt = static_cast<unsigned>(__cvta_generic_to_shared(v_ring + slot * C::kStageBytes));

      // S = Q K^T for 16 keys: s0 = keys 0..7, s1 = keys 8..15
      float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        unsigned kb[4];
        ldmatrix_x4(kb, kt + k_row_off + (((2 * ks + (mi & 1)) ^ r8) << 4));
        mma16816<T>(s0, qa[ks], kb[0], kb[1]);
        mma16816<T>(s1, qa[ks], kb[2], kb[3]);
      }
      // scale, hide the keys past the end, row maxima (rows g and g + 8)
      float v[8] = {s0[0], s0[1], s1[0], s1[1], s0[2], s0[3], s1[2], s1[3]};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int col = ((i >> 1) & 1) * 8 + 2 * tq + (i & 1);
        v[i] = (col < n_valid) ? v[i] * scale_log2 : -INFINITY;
      }
      float mx0 = fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3]));
      float mx1 = fmaxf(fmaxf(v[4], v[5]), fmaxf(v[6], v[7]));
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
      const bool moved = mx0 > m_run[0] || mx1 > m_run[1];
      if (__any_sync(0xffffffffu, moved)) {  // rare after the first blocks
        const float mn0 = fmaxf(m_run[0], mx0), mn1 = fmaxf(m_run[1], mx1);
        const float a0 = (m_run[0] == -INFINITY) ? 0.f : ex2(m_run[0] - mn0);
        const float a1 = (m_run[1] == -INFINITY) ? 0.f : ex2(m_run[1] - mn1);
        l_run[0] *= a0;
        l_run[1] *= a1;
#pragma unroll
        for (int n = 0; n < D / 8; ++n) {
          o[n][0] *= a0;
          o[n][1] *= a0;
          o[n][2] *= a1;
          o[n][3] *= a1;
        }
        m_run[0] = mn0;
        m_run[1] = mn1;
      }
      const float ms0 = (m_run[0] == -INFINITY) ? 0.f : m_run[0];
      const float ms1 = (m_run[1] == -INFINITY) ? 0.f : m_run[1];
      float p[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        p[i] = ex2(v[i] - ms0);
        p[4 + i] = ex2(v[4 + i] - ms1);
      }
      l_run[0] += (p[0] + p[1]) + (p[2] + p[3]);
      l_run[1] += (p[4] + p[5]) + (p[6] + p[7]);
      // P as the A fragment of the second product
      unsigned pa[4];
      pa[0] = pack_pair<T>(p[0], p[1]);  // row g,     keys 2tq, 2tq+1
      pa[1] = pack_pair<T>(p[4], p[5]);  // row g + 8, same keys
      pa[2] = pack_pair<T>(p[2], p[3]);  // row g,     keys 8 + 2tq, ...
      pa[3] = pack_pair<T>(p[6], p[7]);  // row g + 8
#pragma unroll
      for (int c2 = 0; c2 < D / 16; ++c2) {
        unsigned vb[4];
        ldmatrix_x4_trans(vb, vt + v_row_off + (((2 * c2 + (mi >> 1)) ^ r8) << 4));
        mma16816<T>(o[2 * c2], pa, vb[0], vb[1]);
        mma16816<T>(o[2 * c2 + 1], pa, vb[2], vb[3]);
      }
    }
    cp_async_wait<0>();

    // row sums over the four lanes of a row, then the warps of the block through shared memory
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 1);
      l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 2);
    }
    __syncthreads();
    float* red_m = reinterpret_cast<float*>(smem);  // [warps][16]
    float* red_l = red_m + C::kWarps * 16;          // [warps][16]
    float* red_o = red_l + C::kWarps * 16;          // [warps][16][D]
    if (tq == 0) {
      red_m[warp * 16 + g] = m_run[0];
      red_m[warp * 16 + g + 8] = m_run[1];
      red_l[warp * 16 + g] = l_run[0];
      red_l[warp * 16 + g + 8] = l_run[1];
    }
#pragma unroll
    for (int n = 0; n < D / 8; ++n) {
      float* r0 = red_o + (warp * 16 + g) * D + n * 8 + 2 * tq;
      float* r1 = red_o + (warp * 16 + g + 8) * D + n * 8 + 2 * tq;
      r0[0] = o[n][0];
      r0[1] = o[n][1];
      r1[0] = o[n][2];
      r1[1] = o[n][3];
    }
    __syncthreads();
    finish_group<16, D, C::kWarps, kForm>(red_m, red_l, red_o, b, kvh, hb, H, kvH, share.part, deal, Mp, Lp, Op);
    if (kForm == kBalanced) __syncthreads();  // the ring is free again
  }
}

// Fold the partials of the balanced form into the persistent (out, m, l). grid = (H, B); a thread
// takes four columns of every n_grp-th partial (with one column and two groups at head_dim 256 the B1 H64/kvH1
// call on 6000 rows spent 17 of its 28 us of kernels on 38 loads in a row per thread), and (m, l) are read by
// lanes. Launched while the split kernel still runs (programmatic dependent launch): everything it
// reads comes after griddepcontrol.wait and through plain pointers, because the data changes while this
// kernel runs (const __restrict__ would allow loads through the read-only path and in front of the wait).
// RA_STEP_FRESH: the state is known to be empty (it is written, never read, which saves the
// caller an init launch); RA_STEP_FINALIZE: divide by l after folding (saves the finalize
// launch). vec: Op and O are 16-byte aligned (a caller's workspace and state need not be).
constexpr int kFoldGroups = 16, kFoldThreads = kFoldGroups * 64;
template <int kEach>  // partials a thread holds, a power of two: n_grp * kEach >= cap
__global__ void __launch_bounds__(kFoldThreads)
    decode_reduce_kernel(const float* Mp, const float* Lp, const float* Op, float* M, float* L, float* O, int H,
                         int kvH, int D, int head_rows, int ctas, bool vec, const Deal deal) {
  __shared__ float sc[kMaxSplits];
  __shared__ float4 part_o[kFoldThreads];
  const int h = blockIdx.x, b = blockIdx.y;
  const int cols = D / 4;
  const int d = threadIdx.x % cols * 4, grp = threadIdx.x / cols, n_grp = blockDim.x / cols;
  const int lane = threadIdx.x & 31;
  const size_t row = static_cast<size_t>(b) * H + h;
  const bool fresh = (deal.flags & RA_STEP_FRESH) != 0, finalize = (deal.flags & RA_STEP_FINALIZE) != 0;
  const long long total = static_cast<long long>(deal.groups) * deal.stages;
  const long long group =
      (static_cast<long long>(b) * kvH + h % kvH) * deal.head_batches + (h / kvH) / head_rows;
  const int n = deal_owner((group + 1) * deal.stages - 1, total, ctas) - deal_owner(group * deal.stages, total, ctas) + 1;
  wait_for_previous();
  const float* mp = Mp + row * deal.cap;
  const float* lp = Lp + row * deal.cap;
  const float* op = Op + row * deal.cap * D + d;
  float* o_row = O + row * D + d;
  // Everything the call reads is asked for at once: a thread's partials of O (no more than kEach), (m, l) of all partials in every warp, and the old state. One
  // behind the other the loads were most of the fold's time: fp16 B1 H2/kvH1 D64, 8391 rows 8.8 -> 6.5 us a call, fp32 B1
  // H24/kvH8 D128, 11229 rows 17.5 -> 16.3, B1 H8 16384 rows 27.0 -> 26.0; the same bits.
  constexpr int kML = (kFoldGroups * kEach + 31) / 32;
  float ms[kML], ls[kML];
#pragma unroll
  for (int i = 0; i < kML; ++i) {
    const int s = lane + 32 * i;
    ms[i] = s < n ? mp[s] : -INFINITY;
    ls[i] = s < n ? lp[s] : 0.f;
  }
  float4 o[kEach];
#pragma unroll
  for (int i = 0; i < kEach; ++i) {
    const int s = grp + i * n_grp;
    o[i] = s < n ? ld4(op + static_cast<size_t>(s) * D, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const float m_old = fresh ? -INFINITY : M[row], l_old = fresh ? 0.f : L[row];
  // every warp works out the same maximum and sum; the scales go to shared memory once
  float m_n = m_old;
#pragma unroll
  for (int i = 0; i < kML; ++i) m_n = fmaxf(m_n, ms[i]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m_n = fmaxf(m_n, __shfl_xor_sync(0xffffffffu, m_n, off));
  if (m_n == -INFINITY) {
    // nothing visible anywhere: the state stays as it is (or is written empty)
    if ((fresh || finalize) && grp == 0) {
      st4(o_row, make_float4(0.f, 0.f, 0.f, 0.f), vec);
      if (fresh && d == 0) {
        M[row] = -INFINITY;
        L[row] = 0.f;
      }
    }
    return;
  }
  float l_acc = 0.f;
#pragma unroll
  for (int i = 0; i < kML; ++i) {
    const float f = (ms[i] == -INFINITY) ? 0.f : expf(ms[i] - m_n);
    l_acc += f * ls[i];
    if (threadIdx.x < 32) sc[lane + 32 * i] = f;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) l_acc += __shfl_xor_sync(0xffffffffu, l_acc, off);
  const float a = (m_old == -INFINITY) ? 0.f : expf(m_old - m_n);
  if (m_old > -INFINITY) l_acc += a * l_old;
  __syncthreads();
  float4 o_acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < kEach; ++i)
    if (grp + i * n_grp < n) add_scaled(o_acc, sc[grp + i * n_grp], o[i]);
  part_o[threadIdx.x] = o_acc;
  __syncthreads();
  if (grp > 0) return;
  for (int i = 1; i < n_grp; ++i) add_scaled(o_acc, 1.f, part_o[i * cols + threadIdx.x]);
  if (m_old > -INFINITY) add_scaled(o_acc, a, ld4(o_row, vec));
  if (finalize) {
    const float inv = l_acc > 0.f ? 1.f / l_acc : 0.f;
    o_acc = make_float4(o_acc.x * inv, o_acc.y * inv, o_acc.z * inv, o_acc.w * inv);
  }
  st4(o_row, o_acc, vec);
  if (d == 0) {  // every thread has read M / L: two block barriers ago
    M[row] = m_n;
    L[row] = l_acc;
  }
}

struct DecodePlan {
  int cluster;  // > 0: the cluster form with this many blocks per group
  int ctas;     // balanced form: blocks
  Deal deal;
};

// What a kernel needs for a ring stage, in us: `alone` for one block on an SM, `share` of the SM's issue slots
// (k blocks on an SM take k times that if it is longer). Slopes of calls with few groups, one block each,
// between 6000 and 20000 rows: the mma kernel 0.53, 0.71 and 1.14 at head_dim 64, 128 (64 keys) and 256 (32);
// the SIMT kernel 0.34-0.49 for 16 KB with one head, 0.47-0.77 with four and 0.75-1.1 with eight. (The kernel that four and eight
// heads have now needs 0.38-0.48 and 0.49-0.64. Its stages count as its predecessor's because they stand against kFold,
// which is as much too high: a fold at 8.2 with the lower stages sends calls that fold well to clusters, 7.8 -> 10.8 us at
// worst. The two have to change together, see make_plan.)
struct StageCost {
  double alone, share;
};
constexpr StageCost mma_stage_cost(int D) { return {0.5 + 0.0038 * D, 0.0036 * D}; }
constexpr StageCost simt_stage_cost(int heads, size_t stage_bytes) {
  return {(0.46 + 0.12 * heads) * (stage_bytes / 16384.0), 0.145 * heads * (stage_bytes / 16384.0)};
}

// Which form, and how many blocks. `per_sm`: resident blocks per SM; `cap`: partial slots per row
// that the workspace holds; `rows`: (batch, head) rows; `head_rows`: rows of a group; `partials`: there is room for
// partials, or there can be; `long_share`: with more stages a block, twice as many blocks (0: never). Every estimate is the walk of a block, wave by wave, at what its SM or the
// memory (7 TB/s) allows, plus what the fold (a launch, and more the more rows it has) or the merge
// (columns of the group, blocks of the cluster, and a wave of clusters starts slower than one of blocks)
// adds. Constants fitted to 457 shapes (heads 8/8 to 64/1, batch 1 to 64, 200 to 100000 rows, fp16 and fp32,
// every head_dim) timed in each form when a fold was a launch of its own. Launches overlap now and a fold costs about 4:
// over 1700 calls the choice is 2.3 % from the best form on average (single calls of 3 to 100 MB by up to a third), with
// kFold = 4 it would be 0.7 %. kFold stays at 8.2 because the form also decides what a call without a workspace touches:
// a fold goes through the library's one buffer for partials, a merge in clusters through nothing that calls share, and a lower
// kFold moves calls of the second kind to the first.
DecodePlan make_plan(int groups, int stages, size_t stage_bytes, int per_sm, int cap, int ring_max,
                     StageCost cost, size_t rows, int head_rows, int D, bool partials, int long_share) {
  constexpr double kBytesPerUs = 7e6, kFold = 8.2, kFoldRow = 0.005, kMerge = 0.6, kMergeBlock = 0.15,
                   kMergeElement = 0.0005, kWave = 1.5, kClusterWave = 4.0;
  DecodePlan p;
  const int sms = sm_count();
  const double total = static_cast<double>(groups) * stages;
  const int slots = sms * per_sm;
  auto walk = [&](double blocks, double stages_each) {
    const double active = std::min<double>(blocks, slots), on_sm = std::min<double>(per_sm, std::ceil(blocks / sms));
    return std::ceil(blocks / slots) * stages_each *
           std::max(std::max(cost.alone, on_sm * cost.share), stage_bytes * active / kBytesPerUs);
  };
  // no more partials than the workspace holds: a group meets at most ceil(ctas / groups) + 1 blocks,
  // exactly one each when there are as many blocks as groups
  long long ctas = std::min<long long>(slots, static_cast<long long>(total));
  // (with few groups a row's partials are what limits the blocks, down to a second wave that is a quarter full: B3 H8/kvH1
  // D256, 60000 rows 69 -> 83 us; below that there is nothing to cut)
  if (long_share > 0 && total > static_cast<double>(long_share) * slots && (cap - 1.0) * groups > 1.2 * slots) ctas *= 2;
  ctas = cap > 1 ? std::min(ctas, (cap - 1ll) * groups) : groups;
  p.cluster = 0;
  p.ctas = static_cast<int>(ctas);
  double best = walk(static_cast<double>(ctas), std::ceil(total / ctas)) + kFold + kFoldRow * rows;
  if (!partials) best = 1e30;
  for (int c = 1; c <= kMaxCluster && groups <= 65535; c *= 2) {
    if (c > 1 && c > stages) break;
    const double blocks = static_cast<double>(groups) * c;
    const double t = walk(blocks, std::ceil(static_cast<double>(stages) / c)) + kMergeElement * head_rows * D +
                     (c > 1 ? kMerge + kMergeBlock * c : 0.0) +
                     (std::ceil(blocks / slots) - 1) * (c > 1 ? kClusterWave : kWave);
    if (t < best) {
      best = t;
      p.cluster = c;
    }
  }
  p.deal.stages = stages;
  p.deal.groups = groups;
  p.deal.cap = (p.ctas + groups - 1) / groups + (p.ctas == groups ? 0 : 1);
  const long long most = p.cluster ? (stages + p.cluster - 1) / p.cluster
                                   : std::min<long long>(stages, (static_cast<long long>(total) + ctas - 1) / ctas);
  p.deal.ring = static_cast<int>(std::max<long long>(1, std::min<long long>(ring_max, most)));
  return p;
}

// Per-device workspace that grows on demand, like the reference's process-static buffer
// (src/attention_decode.cu:55-65). Not safe for concurrent streams, as the reference's.
struct DevWorkspace {
  void* ptr = nullptr;
  size_t bytes = 0;
  bool recorded = false;  // a capture has seen `ptr`
};
DevWorkspace g_ws[64];
std::mutex g_ws_mu;

// At least `need` bytes. `record`: the address may become part of a CUDA graph, whose replays go on writing there when a
// larger call has made the workspace grow: such a buffer is never given back. Its successor is twice as large (or, if there
// is no room, as large as it must be), so that all buffers left behind take no more than the last one.
int grow_workspace(DevWorkspace& w, size_t need, bool record, void** out) {
  if (w.bytes < need) {
    const size_t old = w.recorded ? w.bytes : 0;
    if (w.ptr && !w.recorded) RAB_CUDA(cudaFree(w.ptr));
    if (!w.recorded) w = DevWorkspace();
    void* ptr = nullptr;
    size_t bytes = std::max(need, 2 * old);
    if (bytes > need && cudaMalloc(&ptr, bytes) != cudaSuccess) {
      cudaGetLastError();
      ptr = nullptr;
      bytes = need;
    }
    if (ptr == nullptr) RAB_CUDA(cudaMalloc(&ptr, bytes));
    w.ptr = ptr;
    w.bytes = bytes;
    w.recorded = false;
  }
  w.recorded = w.recorded || record;
  *out = w.ptr;
  return RA_OK;
}

int ensure_workspace(size_t need, bool record, void** out) {
  int dev = 0;
  RAB_CUDA(cudaGetDevice(&dev));
  RAB_REQUIRE(dev >= 0 && dev < 64, RA_ERR_INVALID, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lk(g_ws_mu);
  return grow_workspace(g_ws[dev], need, record, out);
}

bool workspace_holds(size_t need) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  std::lock_guard<std::mutex> lk(g_ws_mu);
  return g_ws[dev].bytes >= need;
}

}  // namespace

// (a few KB: asking whether the stream is captured would cost every call more than keeping the old ones)
int decode_ml_scratch(size_t floats, float** out) {
  static DevWorkspace ml[64];
  int dev = 0;
  RAB_CUDA(cudaGetDevice(&dev));
  RAB_REQUIRE(dev >= 0 && dev < 64, RA_ERR_INVALID, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lk(g_ws_mu);
  void* ptr = nullptr;
  const int rc = grow_workspace(ml[dev], floats * sizeof(float), true, &ptr);
  *out = static_cast<float*>(ptr);
  return rc;
}

namespace {

// Workspace of the balanced form: [row][slot] of O, m and l.
int partial_space(size_t rows, int D, int cap, void* workspace, bool record, float** Op, float** Mp, float** Lp) {
  const size_t need = rows * cap * (D + 2) * sizeof(float);
  if (workspace == nullptr) {
    const int rc = ensure_workspace(need, record, &workspace);
    if (rc != RA_OK) return rc;
  }
  *Op = static_cast<float*>(workspace);
  *Mp = *Op + rows * cap * D;
  *Lp = *Mp + rows * cap;
  return RA_OK;
}

// Everything both kernels' launches share: plan, workspace, dynamic shared memory, the fold.
// launch(cluster form?, config, deal, Mp, Lp, Op) sets the attribute and launches the kernel.
template <int D, int ROWS, typename Launch>
int run_plan(const ra_shape& s, int head_batches, int stages, size_t stage_bytes, int ring_max, int per_sm,
             StageCost cost, int long_share, size_t red_bytes, int old_splits, float* out, float* m, float* l, void* workspace,
             size_t workspace_bytes, int split_cap, unsigned flags, cudaStream_t stream, Launch launch) {
  const int kvH = kv_heads_of(s);
  const size_t rows = static_cast<size_t>(s.batch) * s.heads;
  const size_t slot_bytes = rows * (D + 2) * sizeof(float);
  int cap = split_cap;
  if (workspace != nullptr) {
    RAB_REQUIRE(workspace_bytes >= old_splits * slot_bytes, RA_ERR_OVERFLOW,
                "decode workspace too small: %zu < %zu bytes", workspace_bytes, old_splits * slot_bytes);
    cap = static_cast<int>(std::min<size_t>(cap, workspace_bytes / slot_bytes));
  }
  auto plan = [&](bool partials) {
    return make_plan(s.batch * kvH * head_batches, stages, stage_bytes, per_sm, cap, ring_max, cost, rows,
                     std::min(ROWS, (s.heads + kvH - 1) / kvH), D, partials, long_share);
  };
  DecodePlan p = plan(true);
  // a stream that is being captured allows no allocation: such a call merges in clusters instead
  bool captured = false;
  if (!p.cluster && workspace == nullptr) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) cudaGetLastError();
    captured = status != cudaStreamCaptureStatusNone;
    if (captured && p.deal.groups <= 65535 && !workspace_holds(p.deal.cap * slot_bytes)) p = plan(false);
  }
  p.deal.head_batches = head_batches;
  p.deal.flags = flags;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = stream;
  cfg.dynamicSmemBytes = std::max(p.deal.ring * stage_bytes, red_bytes);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  if (p.cluster) {
    // Blocks that start beside those of the kernel before go where there is room, two to an SM while
    // others stay empty; so only calls whose blocks leave half of the SMs free overlap it. 157 shapes of 1 to 48 KV
    // heads, 300 to 4000 rows, D64 and D128, fp16 and fp32, calls in a row in a CUDA graph, time beside / behind: up to
    // 74 blocks 0.94 in the median (0.89 to 1.04), 75 to 148 blocks 1.02 (0.94 to 1.23), more 1.00 (0.96 to 1.18).
    cfg.attrs = attr;
    cfg.numAttrs = 2 * p.deal.groups * p.cluster <= sm_count() ? 2 : 1;
    cfg.gridDim = dim3(p.cluster, p.deal.groups);
    return launch(true, cfg, p.deal, m, l, out);
  }
  float *Op, *Mp, *Lp;
  int rc = partial_space(rows, D, p.deal.cap, workspace, captured, &Op, &Mp, &Lp);
  if (rc != RA_OK) return rc;
  // (these fill every slot, so it makes no difference where one begins. The fold does not let the next call's
  // blocks start: they would take the slots around its own, and the last of them would begin behind it. B1 H8
  // D128 fp32, 16384 rows: 27.5 us so, 30.6 with that, 29.7 launched behind.)
  cfg.attrs = attr + 1;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(p.ctas);
  rc = launch(false, cfg, p.deal, Mp, Lp, Op);
  if (rc != RA_OK) return rc;
  // (no more thread groups than partials: with many rows and few partials each the idle ones cost, 2048
  // rows of D32 8 us)
  const int groups = std::min(kFoldGroups, p.deal.cap);
  const int each = (p.deal.cap + groups - 1) / groups;
  const auto fold = each > 4 ? decode_reduce_kernel<8> : each > 2 ? decode_reduce_kernel<4>
                    : each > 1 ? decode_reduce_kernel<2> : decode_reduce_kernel<1>;
  RAB_CUDA(launch_overlapped(fold, dim3(s.heads, s.batch), dim3(std::max(32, groups * (D / 4))), 0, stream, Mp, Lp, Op, m, l,
                             out, s.heads, kvH, D, ROWS, p.ctas,
                             ((reinterpret_cast<uintptr_t>(Op) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0, p.deal));
  RAB_CUDA(cudaGetLastError());
  return RA_OK;
}

// Partials per row that a caller's workspace has always been held to: three waves of equal splits of a group.
int fixed_splits(int blocks_per_split, int sk_eff, int rows_per_stage, int split_cap) {
  int want = (3 * sm_count() + blocks_per_split - 1) / blocks_per_split;
  want = std::max(1, std::min(std::min(want, std::max(1, sk_eff / (2 * rows_per_stage))), split_cap));
  long long rps = (sk_eff + want - 1ll) / want;
  rps = ((rps + rows_per_stage - 1) / rows_per_stage) * rows_per_stage;
  return static_cast<int>(std::max(1ll, (sk_eff + rps - 1) / rps));
}

template <typename K>
int resident_blocks(K kern, int threads, size_t smem) {
  int n = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem) != cudaSuccess)
    cudaGetLastError();
  return n > 0 ? n : 1;
}

template <typename T, int D>
int launch_decode_typed(const void* q, const void* k, const void* v, float* out, float* m,
                        float* l, const ra_shape& s, int sk_eff, long long kv_head_stride,
                        void* workspace, size_t workspace_bytes, cudaStream_t stream,
                        int split_cap = kMaxSplits, unsigned flags = 0) {
  const int kvH = kv_heads_of(s);
  const int group = (s.heads + kvH - 1) / kvH;  // query heads per KV head (largest group)
  const float scale_log2 = kLog2e / sqrtf(static_cast<float>(D));
  const T *qt = static_cast<const T*>(q), *kt = static_cast<const T*>(k), *vt = static_cast<const T*>(v);
  auto launch_with = [&](auto kern, size_t smem_max, std::atomic<unsigned long long>& smem_set,
                         cudaLaunchConfig_t& cfg, int threads, const Deal& deal, float* Mp, float* Lp,
                         float* Op) -> int {
    // once per device and instantiation
    int dev = 0;
    RAB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !(smem_set.load(std::memory_order_acquire) >> dev & 1ull)) {
      RAB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(smem_max)));
      if (dev >= 0 && dev < 64) smem_set.fetch_or(1ull << dev, std::memory_order_release);
    }
    cfg.blockDim = dim3(threads);
    RAB_CUDA(cudaLaunchKernelEx(&cfg, kern, qt, kt, vt, Mp, Lp, Op, s.heads, kvH, sk_eff, kv_head_stride,
                                deal, scale_log2));
    return RA_OK;
  };
  if constexpr (sizeof(T) == 2 && D >= 64) {
    // 16-bit caches: the tensor-core kernel (16 query heads per block)
    using M = MmaCfg<D>;
    constexpr size_t kRed = red_floats(M::kWarps, 16, D) * sizeof(float);
    constexpr size_t kSmem = M::kSmemBytes > kRed ? M::kSmemBytes : kRed;
    const int head_batches = (group + 15) / 16;
    const int stages = (sk_eff + M::kStageRows - 1) / M::kStageRows;
    static const int per_sm = resident_blocks(decode_mma_kernel<T, D, kBalanced>, M::kThreads, kSmem);
    return run_plan<D, 16>(
        s, head_batches, stages, 2 * M::kStageBytes, M::kStages, per_sm, mma_stage_cost(D), 0, kRed,
        fixed_splits(s.batch * kvH * head_batches, sk_eff, 64, split_cap), out,
        m, l, workspace, workspace_bytes, split_cap, flags, stream,
        [&](bool cluster, cudaLaunchConfig_t& cfg, const Deal& deal, float* Mp, float* Lp, float* Op) {
          static std::atomic<unsigned long long> set_c{0}, set_b{0};
          return cluster ? launch_with(decode_mma_kernel<T, D, kCluster>, kSmem, set_c, cfg, M::kThreads, deal,
                                       Mp, Lp, Op)
                         : launch_with(decode_mma_kernel<T, D, kBalanced>, kSmem, set_b, cfg, M::kThreads, deal,
                                       Mp, Lp, Op);
        });
  } else {
    // Rows to which a caller's workspace is held (see fixed_splits): a stage of the kernel with 8 warps and 16-byte pieces
    using Plan = DecodeCfg<T, D>;
    auto run = [&](auto gb_tag) {
      constexpr int GB = decltype(gb_tag)::value;
      using C = std::conditional_t<(GB >= 4), GroupCfg<T, D, GB < 4 ? 4 : GB>, DecodeCfg<T, D>>;
      constexpr int kBlockThreads = GB >= 4 ? GroupCfg<T, D, GB < 4 ? 4 : GB>::kThreads : kThreads;
      constexpr size_t kRed = red_floats(kBlockThreads / 32, GB, D) * sizeof(float);
      constexpr size_t kSmem = C::kSmemBytes > kRed ? C::kSmemBytes : kRed;
      const auto kernel = [](auto form) {
        if constexpr (GB >= 4) return decode_group_kernel<T, D, GB, decltype(form)::value>;
        else return decode_split_kernel<T, D, GB, decltype(form)::value>;
      };
      const auto balanced = kernel(std::integral_constant<DealForm, kBalanced>{});
      const auto clustered = kernel(std::integral_constant<DealForm, kCluster>{});
      const int head_batches = (group + GB - 1) / GB;
      const int stages = (sk_eff + C::kRowsPerStage - 1) / C::kRowsPerStage;
      // fp32, four and eight heads: two blocks an SM move 7.3 and 6.9 TB/s, three 6.9 and 6.9 (D128; B3 H32/kvH8, 200335 rows
      // 699 us with two, 731 with three). 16-bit rows of 32: as many as their registers allow (two; with four heads kept
      // to 80 registers three fit, 22 % faster to 22 % slower by shape and even in the mean)
      static const int per_sm = std::min(resident_blocks(balanced, kBlockThreads, kSmem), GB >= 4 && sizeof(T) == 4 ? 2 : 16);
      // Eight heads with rows of 32 in 16 bits or of 256: two blocks an SM are two thirds of the blocks that the kernel with a butterfly
      // for each head had, so a lane adds up half as many rows again, one after another. Blocks with more than 24 stages are
      // cut in two. Error against 64 bits in that kernel / uncut / so: fp16 D32 B5 H64/kvH8, 150000 rows 3.5e-7 / 3.9e-7 / 3.2e-7; fp32
      // D256 B3 H64/kvH8, 20000 rows 2.9e-7 / 3.2e-7 / 2.7e-7; with shorter shares they differ by 2 % at most. It costs such calls 2 to
      // 20 % (fp16 D32 B1 H64/kvH8, 175724 rows 72 -> 77 us, fp32 D256 B3 H64/kvH8, 20000 rows 160 -> 163, 5000 rows 50 -> 54).
      constexpr int kLongShare = GB == 8 && (sizeof(T) == 2 || D == 256) ? 24 : 0;
      return run_plan<D, GB>(
          s, head_batches, stages, 2 * C::kStageBytes, kStages, per_sm, simt_stage_cost(GB, 2 * C::kStageBytes), kLongShare, kRed,
          fixed_splits(s.batch * kvH * head_batches, sk_eff, Plan::kRowsPerStage, split_cap),
          out, m, l, workspace, workspace_bytes, split_cap, flags, stream,
          [&](bool cluster, cudaLaunchConfig_t& cfg, const Deal& deal, float* Mp, float* Lp, float* Op) {
            static std::atomic<unsigned long long> set_c{0}, set_b{0};
            return cluster ? launch_with(clustered, kSmem, set_c, cfg, kBlockThreads, deal, Mp, Lp, Op)
                           : launch_with(balanced, kSmem, set_b, cfg, kBlockThreads, deal, Mp, Lp, Op);
          });
    };
    // smallest of 1 / 2 / 4 / 8 that fits the group
    if (group > 4) return run(std::integral_constant<int, 8>{});
    if (group > 2) return run(std::integral_constant<int, 4>{});
    if (group > 1) return run(std::integral_constant<int, 2>{});
    return run(std::integral_constant<int, 1>{});
  }
}

template <typename T>
int launch_decode_dtype(const void* q, const void* k, const void* v, float* out, float* m,
                        float* l, const ra_shape& s, int sk_eff, long long kv_head_stride,
                        void* ws, size_t ws_bytes, cudaStream_t stream,
                        int split_cap = kMaxSplits, unsigned flags = 0) {
  switch (s.head_dim) {
    case 32:
      return launch_decode_typed<T, 32>(q, k, v, out, m, l, s, sk_eff, kv_head_stride, ws,
                                        ws_bytes, stream, split_cap, flags);
    case 64:
      return launch_decode_typed<T, 64>(q, k, v, out, m, l, s, sk_eff, kv_head_stride, ws,
                                        ws_bytes, stream, split_cap, flags);
    case 128:
      return launch_decode_typed<T, 128>(q, k, v, out, m, l, s, sk_eff, kv_head_stride, ws,
                                         ws_bytes, stream, split_cap, flags);
    case 256:
      return launch_decode_typed<T, 256>(q, k, v, out, m, l, s, sk_eff, kv_head_stride, ws,
                                         ws_bytes, stream, split_cap, flags);
  }
  set_error("attention_decode_step: unsupported head_dim=%d (supported: 32, 64, 128, 256)",
            s.head_dim);
  return RA_ERR_UNSUPPORTED;
}

}  // namespace

int decode_step(int dtype, const void* q, const void* k, const void* v, float* out, float* m,
                float* l, const ra_shape& s, int q_offset, int k_offset, int causal,
                cudaStream_t stream, int kv_row_stride, void* ws, size_t ws_bytes,
                unsigned flags) {
  RAB_REQUIRE(q && k && v && out && m && l, RA_ERR_INVALID, "decode step: null argument");
  RAB_REQUIRE(s.seq_q == 1, RA_ERR_INVALID, "decode step: seq_q must be 1 (got %d)", s.seq_q);
  RAB_REQUIRE(s.batch > 0 && s.heads > 0 && s.batch <= 65535, RA_ERR_INVALID,
              "decode step: bad batch/heads");
  RAB_REQUIRE((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
               reinterpret_cast<uintptr_t>(v)) % 16 == 0,
              RA_ERR_INVALID, "decode step: q, k and v must be 16-byte aligned");
  int sk_eff = s.seq_k;
  if (causal) {
    // rows [0, q_offset - k_offset] are visible (reference: src/attention_decode.cu:110-116)
    const long long vis = static_cast<long long>(q_offset) - k_offset + 1;
    if (vis < sk_eff) sk_eff = vis < 0 ? 0 : static_cast<int>(vis);
  }
  if (sk_eff <= 0) {
    // nothing visible: the state stays as it is, or is written empty / normalised on request
    const size_t rows = static_cast<size_t>(s.batch) * s.heads;
    if (flags & RA_STEP_FRESH) return launch_init(out, m, l, rows * s.head_dim, rows, stream);
    if (flags & RA_STEP_FINALIZE) return launch_finalize(out, l, rows, s.head_dim, stream);
    return RA_OK;
  }
  const int stride_rows = kv_row_stride > 0 ? kv_row_stride : s.seq_k;
  const long long kv_head_stride = static_cast<long long>(stride_rows) * s.head_dim;
  switch (dtype) {
    case RA_F32:
      return launch_decode_dtype<float>(q, k, v, out, m, l, s, sk_eff, kv_head_stride, ws,
                                        ws_bytes, stream, kMaxSplits, flags);
    case RA_F16:
      return launch_decode_dtype<__half>(q, k, v, out, m, l, s, sk_eff, kv_head_stride, ws,
                                         ws_bytes, stream, kMaxSplits, flags);
    case RA_BF16:
      return launch_decode_dtype<__nv_bfloat16>(q, k, v, out, m, l, s, sk_eff, kv_head_stride, ws,
                                                ws_bytes, stream, kMaxSplits, flags);
  }
  set_error("decode step: unknown dtype %d", dtype);
  return RA_ERR_INVALID;
}

// ---- decode step that never allocates --------------------------------------------------
//
// Some hosts of this library may not call cudaMalloc at all: a serving process that handed
// its whole memory budget to one arena at start-up, a caller inside a region where the
// allocator is locked (a stream being captured, a real-time loop that must not take the
// driver's allocation lock), or an embedder whose policy forbids a library to allocate behind
// its back. For them the split partials live in a fixed array that is part of the library
// image: every GPU that loads the library holds these kStaticScratchFloats * 4 bytes (1 MiB)
// until the process exits.
constexpr size_t kStaticScratchFloats = 262144;  // 1 MiB
static __device__ __align__(256) float g_decode_static_scratch[kStaticScratchFloats];

// Device address of the array on the CURRENT device. In host code the array's name is only a
// host-side handle for the symbol, never a device pointer, so the address is asked for once
// per device (with that device current) and cached.
int static_scratch_ptr(float** out) {
  static float* cache[64] = {};
  static std::mutex mu;
  int dev = 0;
  RAB_CUDA(cudaGetDevice(&dev));
  RAB_REQUIRE(dev >= 0 && dev < 64, RA_ERR_INVALID, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lk(mu);
  if (cache[dev] == nullptr) {
    void* p = nullptr;
    RAB_CUDA(cudaGetSymbolAddress(&p, g_decode_static_scratch));
    RAB_REQUIRE(p != nullptr, RA_ERR_CUDA, "no device address for the static decode scratch");
    cache[dev] = static_cast<float*>(p);
  }
  *out = cache[dev];
  return RA_OK;
}

int decode_step_noalloc(int dtype, const void* q, const void* k, const void* v, float* out,
                        float* m, float* l, const ra_shape& s, int q_offset, int k_offset,
                        int causal, cudaStream_t stream, int kv_row_stride) {
  RAB_REQUIRE(q && k && v && out && m && l, RA_ERR_INVALID, "decode step: null argument");
  RAB_REQUIRE(s.seq_q == 1, RA_ERR_INVALID, "decode step: seq_q must be 1 (got %d)", s.seq_q);
  RAB_REQUIRE(s.batch > 0 && s.heads > 0 && s.batch <= 65535, RA_ERR_INVALID,
              "decode step: bad batch/heads");
  RAB_REQUIRE(s.head_dim == 32 || s.head_dim == 64 || s.head_dim == 128 || s.head_dim == 256,
              RA_ERR_UNSUPPORTED,
              "attention_decode_step: unsupported head_dim=%d (supported: 32, 64, 128, 256)",
              s.head_dim);
  RAB_REQUIRE((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
               reinterpret_cast<uintptr_t>(v)) % 16 == 0,
              RA_ERR_INVALID, "decode step: q, k and v must be 16-byte aligned");
  // One split needs batch * heads * (head_dim + 2) floats; the array must hold at least one.
  const size_t per_split = static_cast<size_t>(s.batch) * s.heads * (s.head_dim + 2);
  RAB_REQUIRE(per_split <= kStaticScratchFloats, RA_ERR_OVERFLOW,
              "ra_attention_decode_step_noalloc: batch*heads*(head_dim+2) = %zu floats exceeds the "
              "built-in scratch of %zu floats (1 MiB); use ra_attention_decode_step with a "
              "caller-provided workspace",
              per_split, kStaticScratchFloats);
  const int split_cap =
      static_cast<int>(std::min<size_t>(kMaxSplits, kStaticScratchFloats / per_split));
  float* scratch = nullptr;
  const int rc = static_scratch_ptr(&scratch);
  if (rc != RA_OK) return rc;
  int sk_eff = s.seq_k;
  if (causal) {
    const long long vis = static_cast<long long>(q_offset) - k_offset + 1;
    if (vis < sk_eff) sk_eff = vis < 0 ? 0 : static_cast<int>(vis);
  }
  if (sk_eff <= 0) return RA_OK;
  const int stride_rows = kv_row_stride > 0 ? kv_row_stride : s.seq_k;
  const long long kv_head_stride = static_cast<long long>(stride_rows) * s.head_dim;
  const size_t bytes = kStaticScratchFloats * sizeof(float);
  // Nothing in the array has to start at zero: every (split, batch, head) slot the reduce
  // kernel reads is written by the split kernel of the same call first.
  switch (dtype) {
    case RA_F32:
      return launch_decode_dtype<float>(q, k, v, out, m, l, s, sk_eff, kv_head_stride, scratch,
                                        bytes, stream, split_cap);
    case RA_F16:
      return launch_decode_dtype<__half>(q, k, v, out, m, l, s, sk_eff, kv_head_stride, scratch,
                                         bytes, stream, split_cap);
    case RA_BF16:
      return launch_decode_dtype<__nv_bfloat16>(q, k, v, out, m, l, s, sk_eff, kv_head_stride,
                                                scratch, bytes, stream, split_cap);
  }
  set_error("decode step: unknown dtype %d", dtype);
  return RA_ERR_INVALID;
}

}  // namespace rab

extern "C" {

int ra_attention_decode_step_noalloc(int dtype, const void* q, const void* k, const void* v,
                                     float* out, float* m, float* l, const ra_shape* shape,
                                     int q_offset, int k_offset, int causal, ra_stream stream,
                                     int kv_row_stride) {
  RAB_REQUIRE(shape != nullptr, RA_ERR_INVALID, "ra_attention_decode_step_noalloc: null shape");
  return rab::decode_step_noalloc(dtype, q, k, v, out, m, l, *shape, q_offset, k_offset, causal,
                                  static_cast<cudaStream_t>(stream), kv_row_stride);
}

size_t ra_decode_workspace_bytes(const ra_shape* shape) {
  if (!shape) return 0;
  return static_cast<size_t>(rab::kMaxSplits) * shape->batch * shape->heads *
         (static_cast<size_t>(shape->head_dim) + 2) * sizeof(float);
}

int ra_attention_decode_step(int dtype, const void* q, const void* k, const void* v, float* out,
                             float* m, float* l, const ra_shape* shape, int q_offset, int k_offset,
                             int causal, ra_stream stream, int kv_row_stride, void* workspace,
                             size_t workspace_bytes) {
  RAB_REQUIRE(shape != nullptr, RA_ERR_INVALID, "ra_attention_decode_step: null shape");
  return rab::decode_step(dtype, q, k, v, out, m, l, *shape, q_offset, k_offset, causal,
                          static_cast<cudaStream_t>(stream), kv_row_stride, workspace,
                          workspace_bytes);
}

}  // extern "C"

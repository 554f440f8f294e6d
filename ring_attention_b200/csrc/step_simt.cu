// SIMT online-softmax ring step: fp32 arithmetic end to end, for fp32 / fp16 / bf16 inputs
// and every supported head_dim (32, 64, 128, 256). It is the fp32 path at head_dim 256 and for
// tensors that TMA does not take, the form a caller can ask for at every other shape, and what
// the tensor-core kernels are checked against.
//
// Same recurrence and state semantics as the reference's attention_step_kernel
// (src/attention_step.cu:114-282): per row, m/l/out are read, folded with one K/V chunk and
// written back unnormalised; a row with no visible key keeps its state. Positions come from
// piecewise-affine maps, which covers the affine call (one segment), the segmented call
// (src/attention_step.cu:305-460) and striped layouts (stride > 1).
//
// Layout of the work: 256 threads per block, 4 to 16 threads share a query row (16 elements of
// the head dimension each, 8 at head_dim 32) and every thread carries two rows, or four, so a K or V
// value read from shared memory feeds as many multiply-adds. What bounds it is what there is beside the
// multiply-adds (packed fp32x2; 72 TFLOP/s): reads of shared memory, shuffles, few warps. K/V tiles of
// 8192/D keys are staged in shared memory as fp32, in two buffers with four rows a thread; a score is a partial dot
// product per thread plus a transposing shuffle reduction over the row's threads, which leaves each complete
// score on exactly one lane: that lane masks and exponentiates it, and the weights travel back
// by shuffle for the second product. fp32 head_dim 256, H8 4096 causal: 10790 us with a lane's 16 columns in a row (four-way
// bank conflicts), 3681 with its pieces dealt over the row's lanes, 2865 with heavy blocks first, 2308 = 30 TFLOP/s with four
// rows a thread, sums merged early and asynchronous copies into a second buffer; the same error. H8 2048 dense, head_dim
// 128 2307 -> 780, 64 750 -> 514, 32 325 -> 335.
#include <cfloat>

#include "common.cuh"

namespace rab {

namespace {

constexpr int kThreads = 256;
constexpr int kChunk = 8;   // keys folded per online-softmax update

// kR: query rows per thread
template <int D, int kR>
struct SimtCfg {
  static constexpr int kTPR = D <= 64 ? 4 : D / 16;  // threads per row
  // Lane c of a row owns four columns in every kStep from c * kFirst on. With the lanes' pieces side by side a
  // read of shared memory touches every bank once; 16 columns in a row per lane were four-way conflicts. (At head_dim
  // 32 a lane's 8 columns have none either way, and side by side they measured 343 us instead of 325.)
  static constexpr int kStep = D == 32 ? 4 : 4 * kTPR, kFirst = D == 32 ? 8 : 4;
  static constexpr int kBufs = kR > 2 ? 2 : 1;  // tiles in shared memory
  static constexpr int kDQ = D / kTPR;               // head-dimension elements per thread
  static constexpr int kGroups = kThreads / kTPR;    // row groups per block
  static constexpr int kRows = kGroups * kR;         // query rows per block
  static constexpr int kBC = 8192 / D;               // keys per shared-memory tile (32 KiB each of K, V)
  static constexpr int kSmemBytes = kBufs * (2 * kBC * D * 4 + kBC * 4);
};

// packed fp32x2 multiply-add: one instruction for two lanes
__device__ inline float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return d;
}

template <typename T>
__device__ inline float load_as_float(const T* p);
template <>
__device__ inline float load_as_float<float>(const float* p) { return *p; }
template <>
__device__ inline float load_as_float<__half>(const __half* p) { return __half2float(*p); }
template <>
__device__ inline float load_as_float<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}

// Four consecutive elements as float4 (16-byte load for fp32, 8-byte for 16-bit types).
template <typename T>
__device__ inline float4 load4(const T* p);
template <>
__device__ inline float4 load4<float>(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
template <>
__device__ inline float4 load4<__half>(const __half* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const __half2 a = *reinterpret_cast<const __half2*>(&raw.x);
  const __half2 b = *reinterpret_cast<const __half2*>(&raw.y);
  const float2 fa = __half22float2(a), fb = __half22float2(b);
  return make_float4(fa.x, fa.y, fb.x, fb.y);
}
template <>
__device__ inline float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
  const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
  const float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
  return make_float4(fa.x, fa.y, fb.x, fb.y);
}

__device__ inline int pos_of(const PosMap& pm, int i, int stride) {
  const int seg = i / pm.seg_len;
  return pm.base[seg] + (i - seg * pm.seg_len) * stride;
}

__device__ inline void copy_async16(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(src_bytes)
               : "memory");
}

template <int kR>
struct Rows {
  float x[kR];
};
// Sum over the kLanes lanes of a row of dot(t), dot(t + kStride), ... (kLanes / kStride values): lane c keeps that of
// t + c % kLanes / kStride * kStride.
template <int kStride, int kLanes, int kR, typename Dot>
__device__ inline Rows<kR> transposed_sum(int t, int c, Dot& dot) {
  if constexpr (kStride == kLanes) {
    return dot(t);
  } else {
    const Rows<kR> a = transposed_sum<2 * kStride, kLanes, kR>(t, c, dot);
    const Rows<kR> b = transposed_sum<2 * kStride, kLanes, kR>(t + kStride, c, dot);
    const bool upper = (c & kStride) != 0;
    Rows<kR> r;
#pragma unroll
    for (int rr = 0; rr < kR; ++rr) {
      const float keep = upper ? b.x[rr] : a.x[rr];
      const float send = upper ? a.x[rr] : b.x[rr];
      r.x[rr] = keep + __shfl_xor_sync(0xffffffffu, send, kStride);
    }
    return r;
  }
}

template <typename T, int D, int kR>
__global__ void __launch_bounds__(kThreads, kR > 2 ? 1 : 2)
    step_simt_kernel(const T* __restrict__ Q, const T* __restrict__ K, const T* __restrict__ V,
                     float* __restrict__ O, float* __restrict__ M, float* __restrict__ L, int H,
                     int kvH, int Sq, int Sk, long long kv_head_stride, const __grid_constant__ PosMap qmap,
                     const __grid_constant__ PosMap kmap,
                     int stride, unsigned flags, long long doc_len) {
  using C = SimtCfg<D, kR>;
  constexpr int DQ = C::kDQ, BC = C::kBC, TPR = C::kTPR;
  constexpr int CH = kChunk > TPR ? kChunk : TPR;  // keys folded per online-softmax update
  constexpr int KPL = CH / TPR;                    // of which this lane scores KPL
  static_assert(BC % CH == 0, "tile must be a whole number of chunks");
  static_assert(DQ % 4 == 0, "float4 loads");
  extern __shared__ __align__(16) unsigned char simt_smem[];
  float* const tiles = reinterpret_cast<float*>(simt_smem);  // [kBufs][K, V][BC][D]
  int* const positions = reinterpret_cast<int*>(tiles + C::kBufs * 2 * BC * D);  // [kBufs][BC]
  __shared__ int qmax_s;
  static_assert(BC <= kThreads, "one thread per key computes the tile's positions");

  const bool causal = (flags & RA_STEP_CAUSAL) != 0;
  const bool fresh = (flags & RA_STEP_FRESH) != 0;
  const int tid = threadIdx.x;
  const int g = tid / TPR;  // row group; its rows are g and g + kGroups of the block
  const int c = tid % TPR;
  // (batch, head) fastest and the last query rows first: under a causal mask they take longest, and begun last they
  // would run on alone
  const unsigned heads = gridDim.y * gridDim.z;
  const unsigned long long at =
      blockIdx.x + static_cast<unsigned long long>(gridDim.x) * (blockIdx.y + gridDim.y * blockIdx.z);
  const int row_block = static_cast<int>(gridDim.x - 1 - at / heads);
  const int h = static_cast<int>(at % heads % gridDim.y);
  const int b = static_cast<int>(at % heads / gridDim.y);
  const float scale = rsqrtf(static_cast<float>(D));

  const size_t q_head = (static_cast<size_t>(b) * H + h) * static_cast<size_t>(Sq) * D;
  const size_t kv_head = (static_cast<size_t>(b) * kvH + (h % kvH)) * kv_head_stride;

  int row[kR], qpos[kR];
  long long qdoc[kR];
  bool active[kR];
  size_t row_idx[kR];
  float2 q2[kR][DQ / 2], o2[kR][DQ / 2];
  float m_i[kR], l_i[kR];

  if (tid == 0) qmax_s = INT_MIN;
  __syncthreads();
#pragma unroll
  for (int rr = 0; rr < kR; ++rr) {
    row[rr] = row_block * C::kRows + rr * C::kGroups + g;
    active[rr] = row[rr] < Sq;
    row_idx[rr] = (static_cast<size_t>(b) * H + h) * Sq + (active[rr] ? row[rr] : 0);
    qpos[rr] = active[rr] ? pos_of(qmap, row[rr], stride) : INT_MIN;
    qdoc[rr] = (doc_len > 0 && active[rr]) ? qpos[rr] / doc_len : 0;
    m_i[rr] = -INFINITY;
    l_i[rr] = 0.f;
#pragma unroll
    for (int d = 0; d < DQ / 2; ++d) {
      q2[rr][d] = make_float2(0.f, 0.f);
      o2[rr][d] = make_float2(0.f, 0.f);
    }
    if (active[rr]) {
      if (c == 0) atomicMax(&qmax_s, qpos[rr]);
      const T* qp = Q + q_head + static_cast<size_t>(row[rr]) * D + c * C::kFirst;
#pragma unroll
      for (int d = 0; d < DQ; d += 4) {
        const float4 x = load4<T>(qp + d / 4 * C::kStep);
        q2[rr][d / 2] = make_float2(x.x, x.y);
        q2[rr][d / 2 + 1] = make_float2(x.z, x.w);
      }
      if (!fresh) {
        const float* op = O + q_head + static_cast<size_t>(row[rr]) * D + c * C::kFirst;
#pragma unroll
        for (int d = 0; d < DQ; d += 4) {
          const float4 x = *reinterpret_cast<const float4*>(op + d / 4 * C::kStep);
          o2[rr][d / 2] = make_float2(x.x, x.y);
          o2[rr][d / 2 + 1] = make_float2(x.z, x.w);
        }
        m_i[rr] = M[row_idx[rr]];
        l_i[rr] = c == 0 ? L[row_idx[rr]] : 0.f;  // the row sum is kept as per-lane shares
      }
    }
  }
  __syncthreads();
  const int qmax = qmax_s;

  // The next tile from j0 on that any row of this block can see, or Sk; its keys' positions go to buffer `buf`. All
  // threads have left the tile that used the buffer before, and the barrier publishes the positions.
  auto find = [&](int j0, int buf) {
    for (; j0 < Sk; j0 += BC) {
      // Global position of each key of the tile (INT_MAX marks rows past the chunk).
      int any = 0;
      if (tid < BC) {
        const int j = j0 + tid;
        const int kp = j < Sk ? pos_of(kmap, j, stride) : INT_MAX;
        any = (j < Sk) && (!causal || kp <= qmax);
        positions[buf * BC + tid] = kp;
      }
      if (__syncthreads_or(any)) return j0;
    }
    return Sk;
  };
  // Stage K and V as fp32, zero-filled past the chunk: fp32 by asynchronous copies, where two buffers let them run under
  // the tile before.
  auto stage = [&](int j0, int buf) {
    float* const Kd = tiles + buf * 2 * BC * D;
    float* const Vd = Kd + BC * D;
    for (int e = tid * 4; e < BC * D; e += kThreads * 4) {
      const int jl = e / D;
      const int d = e - jl * D;
      const int j = j0 + jl;
      const size_t off = kv_head + static_cast<size_t>(j < Sk ? j : 0) * D + d;
      if constexpr (sizeof(T) == 4 && C::kBufs > 1) {
        copy_async16(Kd + e, K + off, j < Sk ? 16 : 0);
        copy_async16(Vd + e, V + off, j < Sk ? 16 : 0);
      } else {
        float4 kx = make_float4(0.f, 0.f, 0.f, 0.f), vx = kx;
        if (j < Sk) {
          kx = load4<T>(K + off);
          vx = load4<T>(V + off);
        }
        *reinterpret_cast<float4*>(&Kd[e]) = kx;
        *reinterpret_cast<float4*>(&Vd[e]) = vx;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  int buf = 0, j_now = find(0, 0);
  if (C::kBufs > 1 && j_now < Sk) stage(j_now, 0);
  for (; j_now < Sk;) {
    int j_next = Sk;
    if constexpr (C::kBufs > 1) {
      j_next = find(j_now + BC, buf ^ 1);
      if (j_next < Sk) {
        stage(j_next, buf ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
    } else {
      stage(j_now, 0);
    }
    __syncthreads();
    const float* const Ks = tiles + buf * 2 * BC * D;
    const float* const Vs = Ks + BC * D;
    const int* const kpos_s = positions + buf * BC;

#pragma unroll 1
    for (int jc = 0; jc < BC; jc += CH) {
      // Scores of CH keys for all rows. The partial dot products of a group of TPR keys are
      // summed with a transposing reduction (TPR - 1 shuffles per group and row): afterwards
      // lane c of the row holds the complete score of key c of the group, so the mask, the
      // maximum and the exponential of a key are computed once, not once per lane. Two partial sums are
      // merged as soon as both are there, so that log2(TPR) of them are alive and not TPR.
      float sc[kR][KPL];  // this lane's keys: group gi, key gi * TPR + c of the chunk
#pragma unroll
      for (int gi = 0; gi < KPL; ++gi) {
        auto dot = [&](int t) {
          const float* kr = &Ks[(jc + gi * TPR + t) * D + c * C::kFirst];
          float2 acc[kR];
#pragma unroll
          for (int rr = 0; rr < kR; ++rr) acc[rr] = make_float2(0.f, 0.f);
#pragma unroll
          for (int d = 0; d < DQ; d += 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(kr + d / 4 * C::kStep);
            const float2 ka = make_float2(k4.x, k4.y), kb = make_float2(k4.z, k4.w);
#pragma unroll
            for (int rr = 0; rr < kR; ++rr) {
              acc[rr] = ffma2(q2[rr][d / 2], ka, acc[rr]);
              acc[rr] = ffma2(q2[rr][d / 2 + 1], kb, acc[rr]);
            }
          }
          Rows<kR> part;
#pragma unroll
          for (int rr = 0; rr < kR; ++rr) part.x[rr] = acc[rr].x + acc[rr].y;
          return part;
        };
        const Rows<kR> sum = transposed_sum<1, TPR, kR>(0, c, dot);
#pragma unroll
        for (int rr = 0; rr < kR; ++rr) sc[rr][gi] = sum.x[rr];
      }
      bool live[kR];
#pragma unroll
      for (int rr = 0; rr < kR; ++rr) {
        float m_new = -INFINITY;
#pragma unroll
        for (int gi = 0; gi < KPL; ++gi) {
          const int kp = kpos_s[jc + gi * TPR + c];
          bool vis = (kp != INT_MAX) && (!causal || kp <= qpos[rr]);
          if (doc_len > 0 && vis) vis = (kp / doc_len) == qdoc[rr];
          sc[rr][gi] = vis ? sc[rr][gi] * scale : -INFINITY;
          m_new = fmaxf(m_new, sc[rr][gi]);
        }
#pragma unroll
        for (int o = 1; o < TPR; o <<= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, o));
        m_new = fmaxf(m_new, m_i[rr]);
        live[rr] = m_new != -INFINITY;  // false: nothing visible so far, state unchanged
        const float alpha = live[rr] ? expf(m_i[rr] - m_new) : 1.f;
        float part_sum = 0.f;
#pragma unroll
        for (int gi = 0; gi < KPL; ++gi) {
          sc[rr][gi] = (sc[rr][gi] == -INFINITY) ? 0.f : expf(sc[rr][gi] - m_new);
          part_sum += sc[rr][gi];
        }
        if (live[rr]) {
          l_i[rr] = alpha * l_i[rr] + part_sum;  // per-lane share of the row sum
          m_i[rr] = m_new;
#pragma unroll
          for (int d = 0; d < DQ / 2; ++d)
            o2[rr][d] = make_float2(o2[rr][d].x * alpha, o2[rr][d].y * alpha);
        }
      }
      bool any_live = false;
#pragma unroll
      for (int rr = 0; rr < kR; ++rr) any_live |= live[rr];
      // the weights are fetched from their owner lanes with warp shuffles below, so the whole
      // warp takes this branch together
      if (!__any_sync(0xffffffffu, any_live)) continue;
#pragma unroll
      for (int jj = 0; jj < CH; ++jj) {
        const float* vr = &Vs[(jc + jj) * D + c * C::kFirst];
        float2 p2[kR];
#pragma unroll
        for (int rr = 0; rr < kR; ++rr) {
          const float pw = __shfl_sync(0xffffffffu, sc[rr][jj / TPR], jj % TPR, TPR);
          p2[rr] = make_float2(pw, pw);
        }
#pragma unroll
        for (int d = 0; d < DQ; d += 4) {
          const float4 v4 = *reinterpret_cast<const float4*>(vr + d / 4 * C::kStep);
          const float2 va = make_float2(v4.x, v4.y), vb = make_float2(v4.z, v4.w);
#pragma unroll
          for (int rr = 0; rr < kR; ++rr) {
            o2[rr][d / 2] = ffma2(p2[rr], va, o2[rr][d / 2]);
            o2[rr][d / 2 + 1] = ffma2(p2[rr], vb, o2[rr][d / 2 + 1]);
          }
        }
      }
    }
    if constexpr (C::kBufs > 1) {
      j_now = j_next;
      buf ^= 1;
      if (j_now < Sk) __syncthreads();  // everyone is done with this tile's buffer, which the next search writes to
    } else {
      __syncthreads();
      j_now = find(j_now + BC, 0);
    }
  }

#pragma unroll
  for (int rr = 0; rr < kR; ++rr) {
#pragma unroll
    for (int o = 1; o < TPR; o <<= 1) l_i[rr] += __shfl_xor_sync(0xffffffffu, l_i[rr], o);
  }
#pragma unroll
  for (int rr = 0; rr < kR; ++rr) {
    if (!active[rr]) continue;
    float inv = 1.f;
    if (flags & RA_STEP_FINALIZE) inv = l_i[rr] > 0.f ? 1.f / l_i[rr] : 0.f;
    float* op = O + q_head + static_cast<size_t>(row[rr]) * D + c * C::kFirst;
#pragma unroll
    for (int d = 0; d < DQ; d += 4) {
      *reinterpret_cast<float4*>(op + d / 4 * C::kStep) =
          make_float4(o2[rr][d / 2].x * inv, o2[rr][d / 2].y * inv, o2[rr][d / 2 + 1].x * inv,
                      o2[rr][d / 2 + 1].y * inv);
    }
    if (c == 0) {
      M[row_idx[rr]] = m_i[rr];
      L[row_idx[rr]] = l_i[rr];
    }
  }
}

template <typename T>
int launch_typed(const StepArgs& a, cudaStream_t stream) {
  const dim3 block(kThreads);
  const T* q = static_cast<const T*>(a.q);
  const T* k = static_cast<const T*>(a.k);
  const T* v = static_cast<const T*>(a.v);
  auto launch = [&](auto kern, int rows, size_t smem) -> int {
    const dim3 grid((a.Sq + rows - 1) / rows, a.H, a.B);
    RAB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    kern<<<grid, block, smem, stream>>>(q, k, v, a.out, a.m, a.l, a.H, a.kvH, a.Sq, a.Sk, a.kv_head_stride, a.qmap,
                                        a.kmap, a.stride, a.flags, a.doc_len);
    return RA_OK;
  };
  int rc = RA_OK;
#define RAB_SIMT_CASE(DD, ROWS)                                                                \
  case DD:                                                                                     \
    rc = launch(step_simt_kernel<T, DD, ROWS>, SimtCfg<DD, ROWS>::kRows, SimtCfg<DD, ROWS>::kSmemBytes); \
    break;
  // fp32 at head_dim 256: four rows a thread halve the reads of shared memory, but a block takes an SM's registers for 64
  // rows. Two rows / four, H8 4096 causal 2865 / 2308 us, H16 1000 dense 784 / 624, H2 2432 dense (76 blocks of four) 936 / 735;
  // fewer blocks leave SMs empty, and under a causal mask the first to go have half the work: H4 1000 dense (64)
  // 273 / 313, H2 2700 causal (86) 740 / 808, H4 2500 causal (160) 852 / 751.
  const long long blocks4 = (a.Sq + SimtCfg<256, 4>::kRows - 1ll) / SimtCfg<256, 4>::kRows * a.H * a.B;
  const bool four = sizeof(T) == 4 && blocks4 * ((a.flags & RA_STEP_CAUSAL) ? 1 : 2) >= sm_count();
  switch (a.D) {
    RAB_SIMT_CASE(32, 2)
    RAB_SIMT_CASE(64, 2)
    RAB_SIMT_CASE(128, 2)
    case 256:
      if (four)
        rc = launch(step_simt_kernel<T, 256, sizeof(T) == 4 ? 4 : 2>, SimtCfg<256, 4>::kRows, SimtCfg<256, 4>::kSmemBytes);
      else
        rc = launch(step_simt_kernel<T, 256, 2>, SimtCfg<256, 2>::kRows, SimtCfg<256, 2>::kSmemBytes);
      break;
    default:
      set_error("attention step: unsupported head_dim=%d (supported: 32, 64, 128, 256)", a.D);
      return RA_ERR_UNSUPPORTED;
  }
#undef RAB_SIMT_CASE
  RAB_CUDA(cudaGetLastError());
  return rc;
}

}  // namespace

int launch_step_simt(int dtype, const StepArgs& a, cudaStream_t stream) {
  if (a.Sq <= 0 || a.B <= 0 || a.H <= 0) return RA_OK;
  RAB_REQUIRE(a.H <= 65535 && a.B <= 65535, RA_ERR_INVALID,
              "attention step: heads/batch exceed the grid limit");
  switch (dtype) {
    case RA_F32:
      return launch_typed<float>(a, stream);
    case RA_F16:
      return launch_typed<__half>(a, stream);
    case RA_BF16:
      return launch_typed<__nv_bfloat16>(a, stream);
  }
  set_error("attention step: unknown dtype %d", dtype);
  return RA_ERR_INVALID;
}

}  // namespace rab

// Multi-head attention (head dim 64, all-ones mask) on tcgen05 tensor cores.
//
// One CTA serves one (sequence, head) and loops over its 128-query tiles.
//   scores = Q . K^T      tcgen05.mma, M=128, N=128 per key block, K=64, fp32 in TMEM
//   P = softmax(scores)   8 or 16 warps, 1/2 or 1/4 of a query row per thread, from TMEM,
//                         written as bf16 into 128-byte-swizzled shared memory
//   O = P . V             tcgen05.mma, M=128, N=64, K=SEQ, fp32 in TMEM
// With several tiles the scores of tile t+1 are issued before the P.V of tile t, and the output of tile t-1 leaves while
// they are computed (two output accumulators): what stays in series per tile of 384 keys is scores (0.8 us with the hand-over),
// maxima and their exchange (0.6 us) and the exponentials (2.0 us; 1.6 us of the special-function unit).  16 x 384 tokens of
// 16 heads, two rounds of CTAs: 32.2 us with each tile's steps in sequence, 31.2 with the scores first, 29.3 with the
// output behind them; 1 x 384: 15.7 -> 14.4.
// All operands arrive by TMA (no multicast) from this GPU's memory:
//   Q and K from the [tokens, 2*hidden] output of the fused Q|K projection,
//   V^T from the [hidden, tokens] output of the V projection computed with
//   swapped GEMM operands, so that it is already K-major for the second product.
// The V bias is added to the output instead (softmax rows sum to one).
// Replaces the attention subgraph the original runs inside ONNX Runtime
// (reference src/apps/ort_defs.h:141-190).  Waits are bounded; a timeout sets
// *status, the CTA stops, frees its tensor memory and returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstring>

#include "driver_api.h"
#include "nn_kernels.h"
#include "pdl_launch.h"
#include "ptx.cuh"
#include "per_device.h"

namespace {

constexpr int HD = 64;          // head dim
constexpr int QT = 128;         // queries per tile
// Softmax warps per tensor-memory lane quarter; one more warp issues TMA and MMAs.  Long rows take four: 384 keys need the
// warps to keep the special-function unit busy (one CTA per SM).  With 128 keys three CTAs share an SM and two are enough.
template <int SEQ>
struct AttThreads {
  static constexpr int SHARES = SEQ == QT ? 2 : 4;  // a thread has one query row and 1/SHARES of its keys
  static constexpr int SOFT = SHARES * 128, TOTAL = SOFT + 32;
};

template <int SEQ>
struct AttSmem {
  static constexpr int Q_BYTES = QT * 128;            // 128 rows x 64 bf16
  static constexpr int K_BYTES = SEQ * 128;           // SEQ rows x 64 bf16
  static constexpr int VT_BYTES = (SEQ / 64) * 64 * 128;  // SEQ/64 atoms of 64 rows x 64 keys
  static constexpr int P_BYTES = (SEQ / 64) * QT * 128;   // SEQ/64 atoms of 128 rows x 64 keys
  // With a single query tile (SEQ == 128) Q and K are dead once the scores exist, and the scores are dead once P is
  // written: P takes the place of Q|K in shared memory and the output accumulator the place of the scores in tensor
  // memory.  48 KB, 128 columns and the launch bounds let three CTAs share an SM, so every (sequence, head) of a 32 x 12
  // batch is resident at once (384 of 444) and the SM interleaves their load -> MMA -> softmax -> MMA chains.
  static constexpr bool ALIAS = SEQ == QT;
  static constexpr int P_OFFSET = ALIAS ? 0 : Q_BYTES + K_BYTES + VT_BYTES;
  static constexpr int TOTAL = ALIAS ? Q_BYTES + K_BYTES + VT_BYTES : Q_BYTES + K_BYTES + VT_BYTES + P_BYTES;
  static constexpr int TMEM_COLS = ALIAS ? 128 : ((SEQ + 2 * HD) <= 256 ? 256 : 512);
  static_assert(!ALIAS || P_BYTES <= Q_BYTES + K_BYTES, "P must fit over Q and K");
};

// Barrier of the softmax warps with the AND of their threads' predicates.
template <int SOFT_THREADS>
__device__ __forceinline__ bool soft_all(bool pred) {
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
      "barrier.cta.red.and.pred p, 1, %1, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(out)
      : "n"(SOFT_THREADS), "r"((uint32_t)pred)
      : "memory");
  return out != 0;
}

// VMN = true: V is read in place from the fused Q|K|V projection ([tokens, 3*hidden], V in the last third).  A V tile
// is then [keys, 64] with the head dimension contiguous, i.e. an MN-major B operand of the second product: same
// 128-byte-swizzled shared-memory tile and descriptor, "B is MN-major" in the instruction descriptor, and a step of 16
// keys along K is 2048 bytes (two 8-row groups) instead of 32.  No transposed copy of V and no separate V GEMM.
template <int SEQ, bool VMN>
__global__ void __launch_bounds__(AttThreads<SEQ>::TOTAL, SEQ == QT ? 3 : 1)
attention_tc(const __grid_constant__ CUtensorMap tmap_qk, const __grid_constant__ CUtensorMap tmap_vt,
             __nv_bfloat16* out, int ld_out, const float* v_bias, int hidden, float scale_log2e,
             uint32_t* status) {
  using L = AttSmem<SEQ>;
  constexpr int SOFT_THREADS = AttThreads<SEQ>::SOFT, SHARES = AttThreads<SEQ>::SHARES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + L::Q_BYTES;
  uint8_t* sVT = sK + L::K_BYTES;
  uint8_t* sP = smem + L::P_OFFSET;
  __shared__ __align__(8) uint64_t bar_k, bar_v, bar_q, bar_s, bar_p, bar_o;
  __shared__ uint32_t tmem_base_smem;
  __shared__ uint32_t s_error;
  __shared__ float s_max[SHARES][QT], s_sum[2][SHARES][QT];  // sums of alternating tiles

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = blockIdx.x, seq_idx = blockIdx.y;
  const int tok0 = seq_idx * SEQ;
  constexpr int NQT = SEQ / QT;

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bar_k, 1);
    ptx::mbar_init(&bar_v, 1);
    ptx::mbar_init(&bar_q, 1);
    ptx::mbar_init(&bar_s, 1);
    ptx::mbar_init(&bar_p, SOFT_THREADS / 32);
    ptx::mbar_init(&bar_o, 1);
    ptx::fence_mbar_init();
    s_error = 0;
    ptx::prefetch_tmap(&tmap_qk);
    ptx::prefetch_tmap(&tmap_vt);
  }
  if (warp == SOFT_THREADS / 32) {
    ptx::tmem_alloc(&tmem_base_smem, L::TMEM_COLS);
    ptx::tmem_relinquish();
    ptx::grid_dep_launch();  // after the allocation, see pdl_launch.h
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::grid_dep_wait();
  ptx::tc_fence_after();
  const uint32_t tmem_s = tmem_base_smem;          // scores: columns [0, SEQ)
  // Outputs of alternating tiles: columns [SEQ, SEQ+64) and [SEQ+64, SEQ+128), or, with one tile, over the scores.
  auto tmem_o = [&](int qt) { return tmem_base_smem + (L::ALIAS ? 0 : SEQ + (qt & 1) * HD); };

  if (warp == SOFT_THREADS / 32) {
    // The warp walks the tiles together, one elected lane issues: descriptors and addresses stay in uniform registers
    // (see gemm_persistent.cu).  K and V^T of this head stay resident for all query tiles; the first Q tile does not wait
    // for V^T.
    const bool elected = ptx::elect_one();
    auto load_q = [&](int qt) {
      ptx::mbar_expect_tx(&bar_q, L::Q_BYTES);
      ptx::tma_load_2d(sQ, &tmap_qk, &bar_q, head * HD, tok0 + qt * QT);
    };
    if (elected) {
      load_q(0);
      ptx::mbar_expect_tx(&bar_k, L::K_BYTES);
      for (int nb = 0; nb < SEQ / 128; nb++)
        ptx::tma_load_2d(sK + nb * 128 * 128, &tmap_qk, &bar_k, hidden + head * HD, tok0 + nb * 128);
      ptx::mbar_expect_tx(&bar_v, L::VT_BYTES);
      if constexpr (VMN) {
        for (int nb = 0; nb < SEQ / 128; nb++)
          ptx::tma_load_2d(sVT + nb * 128 * 128, &tmap_qk, &bar_v, 2 * hidden + head * HD, tok0 + nb * 128);
      } else {
        for (int a = 0; a < SEQ / 64; a++) ptx::tma_load_2d(sVT + a * 64 * 128, &tmap_vt, &bar_v, tok0 + a * 64, head * HD);
      }
    }
    const uint32_t idesc_s = ptx::umma_idesc_bf16(QT, 128);
    const uint32_t idesc_o = ptx::umma_idesc_bf16(QT, HD) | (VMN ? (1u << 16) : 0u);  // bit 16: B is MN-major
    const uint32_t q_lo = ptx::umma_desc_lo(ptx::smem_u32(sQ)), k_lo = ptx::umma_desc_lo(ptx::smem_u32(sK)),
                   p_lo = ptx::umma_desc_lo(ptx::smem_u32(sP)), v_lo = ptx::umma_desc_lo(ptx::smem_u32(sVT));
    auto scores = [&]() {
      if (!elected) return;
#pragma unroll
      for (int nb = 0; nb < SEQ / 128; nb++)
#pragma unroll
        for (int k = 0; k < HD / 16; k++)
          ptx::umma_bf16(tmem_s + nb * 128, ptx::umma_desc_join(q_lo + k * 2), ptx::umma_desc_join(k_lo + nb * (128 * 128 / 16) + k * 2),
                         idesc_s, k != 0 ? 1u : 0u);
      ptx::umma_commit(&bar_s);
    };
    bool ok = ptx::mbar_wait_warp(&bar_q, 0) && ptx::mbar_wait_warp(&bar_k, 0);
    if (ok) scores();
    ok = ok && ptx::mbar_wait_warp(&bar_v, 0);
    for (int qt = 0; qt < NQT && ok; qt++) {
      const uint32_t ph = (uint32_t)qt & 1u;
      // The next Q tile takes this one's place as soon as its scores exist, while the softmax runs.
      if (qt + 1 < NQT) {
        if (!(ok = ptx::mbar_wait_warp(&bar_s, ph))) break;
        if (elected) load_q(qt + 1);
      }
      // P ready (written by the softmax warps, which have read all scores by then)
      if (!(ok = ptx::mbar_wait_warp(&bar_p, ph))) break;
      ptx::tc_fence_after();
      // The next tile's scores go first: its maxima are looked for while P.V runs.
      if (qt + 1 < NQT) {
        if (!(ok = ptx::mbar_wait_warp(&bar_q, ph ^ 1u))) break;
        scores();
      }
      if (elected) {
#pragma unroll
        for (int kk = 0; kk < SEQ / 16; kk++) {
          const uint32_t atom = (uint32_t)kk >> 2, sub = (uint32_t)kk & 3u;
          const uint32_t v_at = VMN ? (uint32_t)kk * (2048 / 16) : atom * (64 * 128 / 16) + sub * 2;
          ptx::umma_bf16(tmem_o(qt), ptx::umma_desc_join(p_lo + atom * (QT * 128 / 16) + sub * 2), ptx::umma_desc_join(v_lo + v_at),
                         idesc_o, kk != 0 ? 1u : 0u);
        }
        ptx::umma_commit(&bar_o);
      }
    }
    if (!ok && elected) atomicCAS(&s_error, 0u, 1u);
  } else {
    // A thread has one query row and a share of its keys; the shares' maxima and sums meet in shared memory.
    const int share = warp >> 2, row = (warp & 3) * 32 + lane;
    constexpr int COLS = SEQ / SHARES;
    const int c0 = share * COLS;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    // Output of tile qt: every share writes its part of the head's 64 columns.
    auto output = [&](int qt) {
      constexpr int OC = HD / SHARES;
      float total = s_sum[qt & 1][0][row];
#pragma unroll
      for (int k = 1; k < SHARES; k++) total += s_sum[qt & 1][k][row];
      const float inv = 1.f / total;
      __nv_bfloat16* orow = out + (size_t)(tok0 + qt * QT + row) * ld_out + head * HD;
      const int c = share * OC;
      uint32_t r[OC];
      if constexpr (OC == 32) ptx::tmem_ld_32x32b_x32(tmem_o(qt) + lane_base + c, r);
      else ptx::tmem_ld_32x32b_x16(tmem_o(qt) + lane_base + c, r);
      ptx::tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < OC / 8; j++) {
        uint4 q;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
        for (int t = 0; t < 4; t++) {
          const int d = c + j * 8 + 2 * t;
          const float b0 = v_bias ? *(v_bias + head * HD + d) : 0.f;
          const float b1 = v_bias ? *(v_bias + head * HD + d + 1) : 0.f;
          h[t] = __floats2bfloat162_rn(__uint_as_float(r[j * 8 + 2 * t]) * inv + b0,
                                       __uint_as_float(r[j * 8 + 2 * t + 1]) * inv + b1);
        }
        *reinterpret_cast<uint4*>(orow + c + j * 8) = q;
      }
    };
    bool ok = true;
    for (int qt = 0; qt < NQT; qt++) {
      const uint32_t ph = (uint32_t)qt & 1u;
      ok = *(volatile uint32_t*)&s_error == 0 && ptx::mbar_wait(&bar_s, ph);
      if (!(ok = soft_all<SOFT_THREADS>(ok))) {
        if (lane == 0) atomicCAS(&s_error, 0u, 2u);
        break;
      }
      ptx::tc_fence_after();
      // pass 1: row maximum
      float mx = -3.0e38f;
      for (int c = 0; c < COLS; c += 32) {
        uint32_t r[32];
        ptx::tmem_ld_32x32b_x32(tmem_s + lane_base + c0 + c, r);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j += 2) mx = ptx::max3(mx, __uint_as_float(r[j]), __uint_as_float(r[j + 1]));
      }
      s_max[share][row] = mx;
      // behind the barrier the previous tile's P.V is through as well, and P may be written again
      if (!(ok = soft_all<SOFT_THREADS>(qt == 0 || ptx::mbar_wait(&bar_o, ph ^ 1u)))) {
        if (lane == 0) atomicCAS(&s_error, 0u, 3u);
        break;
      }
      ptx::tc_fence_after();
#pragma unroll
      for (int k = 0; k < SHARES; k++) mx = fmaxf(mx, s_max[k][row]);
      // pass 2: exponentials, row sum, P in bf16 to swizzled shared memory.  Packed differences and products; the fast exponential
      // flushes subnormal results, so 32 weights of which one may be subnormal (below 2^-126 of the row's largest) are made
      // again with exp2f.
      float2 sum = make_float2(0.f, 0.f);
      const float2 neg_mx = make_float2(-mx, -mx), scale2 = make_float2(scale_log2e, scale_log2e);
      for (int c = c0; c < c0 + COLS; c += 32) {
        uint32_t r[32];
        ptx::tmem_ld_32x32b_x32(tmem_s + lane_base + c, r);
        ptx::tmem_ld_wait();
        uint8_t* prow = sP + (size_t)(c >> 6) * QT * 128 + (size_t)row * 128;
        const int chunk0 = (c & 63) >> 3;
        const float2 sum_before = sum;
        float least = 0.f;  // smallest exponent
        auto weights = [&](auto exponential) {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            uint4 q;
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
            for (int t = 0; t < 4; t++) {
              const float2 x = make_float2(__uint_as_float(r[j * 8 + 2 * t]), __uint_as_float(r[j * 8 + 2 * t + 1]));
              const float2 y = __fmul2_rn(__fadd2_rn(x, neg_mx), scale2);
              h[t] = __floats2bfloat162_rn(exponential(y.x), exponential(y.y));
              least = ptx::min3(least, y.x, y.y);
              sum = __fadd2_rn(sum, __bfloat1622float2(h[t]));  // of the rounded values that the second product will see
            }
            *reinterpret_cast<uint4*>(prow + (((chunk0 + j) ^ (row & 7)) << 4)) = q;
          }
        };
        weights([](float y) {
          float e;
          asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(y));
          return e;
        });
        if (least < -126.f) {
          sum = sum_before;
          weights([](float y) { return exp2f(y); });
        }
      }
      s_sum[qt & 1][share][row] = sum.x + sum.y;
      ptx::tc_fence_before();
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bar_p);
      // The previous tile's output leaves while the tensor core works on the next scores.
      if (qt > 0) output(qt - 1);
      ptx::tc_fence_before();
    }
    if (ok) {
      ok = soft_all<SOFT_THREADS>(ptx::mbar_wait(&bar_o, (uint32_t)(NQT - 1) & 1u));
      if (!ok && lane == 0) atomicCAS(&s_error, 0u, 3u);
      ptx::tc_fence_after();
      if (ok) output(NQT - 1);
      ptx::tc_fence_before();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (s_error != 0) {
    if (threadIdx.x == 0 && status) atomicExch(status, 0x100u | s_error);
    __nanosleep(1000000);
    __syncthreads();
  }
  if (warp == SOFT_THREADS / 32) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base_smem, L::TMEM_COLS);
  }
}

cudaError_t encode(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t outer, uint64_t stride_bytes, uint32_t box_inner,
                   uint32_t box_outer) {
  const SrpcDriverApi* d = srpc_driver_api();
  if (!d->TensorMapEncodeTiled) return cudaErrorNotSupported;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t st[1] = {stride_bytes};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t es[2] = {1, 1};
  CUresult r = d->TensorMapEncodeTiled(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, st, box, es,
                                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int SEQ, bool VMN>
cudaError_t launch(const CUtensorMap& tqk, const CUtensorMap& tvt, void* out, int ld_out, const float* v_bias, int hidden,
                   int batch, int heads, uint32_t* status, cudaStream_t s) {
  static PerDeviceFlag attr;
  const int dev = PerDeviceFlag::current();
  const int smem = AttSmem<SEQ>::TOTAL + 1024;
  if (attr.needed(dev)) {
    cudaError_t e = cudaFuncSetAttribute(attention_tc<SEQ, VMN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    attr.set(dev);
  }
  const float scale_log2e = 0.125f * 1.4426950408889634f;
  return launch_pdl(attention_tc<SEQ, VMN>, dim3(heads, batch), dim3(AttThreads<SEQ>::TOTAL), smem, s, tqk, tvt, (__nv_bfloat16*)out, ld_out, v_bias,
                    hidden, scale_log2e, status);
}

}  // namespace

cudaError_t nn_attention_tc(const void* qk, int ld_qk, const void* vt, int ld_vt, void* out, int ld_out, const float* v_bias,
                            int batch, int seq, int heads, uint32_t* status, cudaStream_t s) {
  const int hidden = heads * HD;
  const int tokens = batch * seq;
  if ((ld_qk % 8) || (ld_out % 8) || ((uintptr_t)qk & 15) || ((uintptr_t)out & 15)) return cudaErrorInvalidValue;
  CUtensorMap tqk, tvt;
  if (!vt) {  // V in place: qk is the [tokens, 3*hidden] output of the fused Q|K|V projection
    cudaError_t e = encode(&tqk, qk, (uint64_t)3 * hidden, (uint64_t)tokens, (uint64_t)ld_qk * 2, 64, 128);
    if (e != cudaSuccess) return e;
    if (seq == 128) return launch<128, true>(tqk, tqk, out, ld_out, v_bias, hidden, batch, heads, status, s);
    if (seq == 384) return launch<384, true>(tqk, tqk, out, ld_out, v_bias, hidden, batch, heads, status, s);
    return cudaErrorInvalidValue;
  }
  if ((ld_vt % 8) || ((uintptr_t)vt & 15)) return cudaErrorInvalidValue;
  cudaError_t e = encode(&tqk, qk, (uint64_t)2 * hidden, (uint64_t)tokens, (uint64_t)ld_qk * 2, 64, 128);
  if (e != cudaSuccess) return e;
  e = encode(&tvt, vt, (uint64_t)tokens, (uint64_t)hidden, (uint64_t)ld_vt * 2, 64, 64);
  if (e != cudaSuccess) return e;
  if (seq == 128) return launch<128, false>(tqk, tvt, out, ld_out, v_bias, hidden, batch, heads, status, s);
  if (seq == 384) return launch<384, false>(tqk, tvt, out, ld_out, v_bias, hidden, batch, heads, status, s);
  return cudaErrorInvalidValue;
}

// Two pointwise convolutions of a bottleneck chain in one kernel: the expansion that ends a block and the reduction that begins
// the next one, for blocks of 64 channels (56 x 56 pixels in ResNet-50).
//
//   wide   = relu(W3 . x [+ W3' . x2] + b3 [+ residual])     [M, 256]
//   narrow = relu(W1 . wide + b1)                            [M, 64 or 128]
//
// Both are bound by memory: the wide tensor is 103 MB for 64 images, and a kernel of its own for the reduction reads it
// again.  Here a CTA keeps both filters in shared memory and walks over tiles of 128 pixels in chunks of 64 wide channels.  A
// chunk's buffer takes the residual (TMA), then the finished wide values in its place (bf16, 128-byte swizzle), and in that
// form it is at once the source of the TMA store and an A operand of the second product: one k-block of it.
//   warp 0       loads: filters once, then per tile x [x2] and the chunks of the residual
//   warp 1       tcgen05.mma of the expansion, 64 columns into one of four accumulators at a time
//   warp 3       tcgen05.mma of the reduction, a k-block per finished chunk.  One warp for both products took 1300 - 1600 cycles
//                per chunk for its waits and issues in sequence and set the pace (16 images, cached: 13.6 us, now 11.9)
//   warp 2       stores of finished chunks; hands their buffers back
//   warps 4-11   chunks, four warps for every second one: accumulator + bias + residual, relu, bf16
//   warps 12-15  the narrow tile: accumulator + bias, relu, bf16, store
// Each value is computed with the same operations in the same order as by the separate kernels, k-block by k-block, and the
// second product reads the same rounded values, so the results are the same bits.
// 64 images: expansion with residual and reduction 40.6 + 18.5 us apart in the network,
// 40.5 here (257 MB, 39 us at the copy rate); with 128 narrow channels 41.3 + 23.3 and 47.6, with two inputs 24.7 + 18.5 and 39.1.  4
// images, cached: 10.9 -> 6.5, 11.6 -> 7.5, 9.0 -> 6.3; one image: 6.7 -> 6.0, 7.1 -> 6.9, 6.5 -> 6.0: no size is better apart.  ResNet-50,
// 64 images: 931 -> 884.
// Waits are bounded; a timeout sets *status, the CTA stops, frees its tensor memory and returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "gemm_tcgen05.h"
#include "pdl_launch.h"
#include "per_device.h"
#include "ptx.cuh"

cudaError_t srpc_tensor_map_2d(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                               uint32_t box_inner, uint32_t box_outer);

namespace {

constexpr int TM = 128;              // pixels per tile
constexpr int WIDE = 256, CHUNKS = WIDE / 64;
constexpr int BLOCK_BYTES = TM * 128;  // 128 pixels x 64 channels
constexpr int ACC = CHUNKS;          // accumulators of 64 wide columns; the two narrow ones lie behind them
constexpr int THREADS = 512;

// N2 = 64 or 128 narrow channels; DUAL: two inputs of 64 channels and no residual.  The ring has as many chunk buffers as
// fit beside the filters: a buffer is held from the request for its residual to the end of its store, about 4 us.
template <int N2, bool DUAL>
struct Chain {
  static constexpr int KB = DUAL ? 2 : 1;           // k-blocks of the expansion
  static constexpr int A_SLOTS = DUAL ? 3 : 2;
  static constexpr int RING = DUAL ? 4 : N2 == 64 ? 7 : 5;
  static constexpr int W3_BYTES = KB * WIDE * 128, W1_BYTES = CHUNKS * N2 * 128;
  static constexpr int W1_AT = W3_BYTES, A_AT = W1_AT + W1_BYTES, RING_AT = A_AT + A_SLOTS * BLOCK_BYTES,
                       T_AT = RING_AT + RING * BLOCK_BYTES;
  static constexpr int SMEM = T_AT + BLOCK_BYTES + 1024;
};

struct ChainMaps {
  CUtensorMap x, x2, w3, w1, residual, wide, narrow;
};

// relu of 32 accumulator columns + bias (+ residual) to the swizzled row of a 64-channel block.  All loads come before the first
// store: behind one, the compiler has to keep them in order, and eight round trips to shared memory take longer than the rest.
template <bool RES>
__device__ __forceinline__ void finish_32(const uint32_t* r, const float* bias, const uint4* res, uint8_t* row_base, int chunk0, int row) {
  float4 b4[8];
#pragma unroll
  for (int j = 0; j < 8; j++) b4[j] = *reinterpret_cast<const float4*>(bias + j * 4);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    float v[8];
#pragma unroll
    for (int t = 0; t < 2; t++) {
      v[4 * t] = __uint_as_float(r[j * 8 + 4 * t]) + b4[2 * j + t].x;
      v[4 * t + 1] = __uint_as_float(r[j * 8 + 4 * t + 1]) + b4[2 * j + t].y;
      v[4 * t + 2] = __uint_as_float(r[j * 8 + 4 * t + 2]) + b4[2 * j + t].z;
      v[4 * t + 3] = __uint_as_float(r[j * 8 + 4 * t + 3]) + b4[2 * j + t].w;
    }
    if (RES) {
      const __nv_bfloat162* f2 = reinterpret_cast<const __nv_bfloat162*>(&res[j]);
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const float2 f = __bfloat1622float2(f2[t]);
        v[2 * t] += f.x;
        v[2 * t + 1] += f.y;
      }
    }
    uint4 q;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
    for (int t = 0; t < 4; t++) h[t] = __floats2bfloat162_rn(fmaxf(v[2 * t], 0.f), fmaxf(v[2 * t + 1], 0.f));
    *reinterpret_cast<uint4*>(row_base + (((chunk0 + j) ^ (row & 7)) << 4)) = q;
  }
}

template <int N2, bool DUAL>
__global__ void __launch_bounds__(THREADS, 1)
conv_chain_kernel(const __grid_constant__ ChainMaps maps, int M, const float* b3, const float* b1, int late_trigger, uint32_t* status) {
  using C = Chain<N2, DUAL>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t w_full, a_full[C::A_SLOTS], a_free[C::A_SLOTS], r_full[C::RING], p_full[C::RING], r_free[C::RING],
      acc_full[ACC], acc_free[ACC], nar_full[2], nar_free[2];
  __shared__ uint32_t tmem_base_smem, s_error;
  __shared__ __align__(16) float s_b3[WIDE], s_b1[N2];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = (M + TM - 1) / TM;
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // tiles blockIdx.x, + gridDim.x, ...
  const int chunks = mine * CHUNKS;

  if (threadIdx.x == 0) {
    ptx::mbar_init(&w_full, 1);
    for (int i = 0; i < C::A_SLOTS; i++) {
      ptx::mbar_init(&a_full[i], 1);
      ptx::mbar_init(&a_free[i], 1);
    }
    for (int i = 0; i < C::RING; i++) {
      ptx::mbar_init(&r_full[i], 1);
      ptx::mbar_init(&p_full[i], 4);
      ptx::mbar_init(&r_free[i], 2);  // the reduction has read the chunk, and so has its store
    }
    for (int i = 0; i < ACC; i++) {
      ptx::mbar_init(&acc_full[i], 1);
      ptx::mbar_init(&acc_free[i], 4);
    }
    for (int i = 0; i < 2; i++) {
      ptx::mbar_init(&nar_full[i], 1);
      ptx::mbar_init(&nar_free[i], 4);
    }
    ptx::fence_mbar_init();
    s_error = 0;
  }
  if (warp == 3) {
    ptx::tmem_alloc(&tmem_base_smem, 512);
    ptx::tmem_relinquish();
    if (!late_trigger) ptx::grid_dep_launch();  // after the allocation, see pdl_launch.h
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::grid_dep_wait();
  for (int i = threadIdx.x; i < WIDE; i += THREADS) s_b3[i] = *(b3 + i);
  for (int i = threadIdx.x; i < N2; i += THREADS) s_b1[i] = *(b1 + i);
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = tmem_base_smem, tmem_narrow = tmem + ACC * 64;
  auto healthy = [&]() { return *(volatile uint32_t*)&s_error == 0; };

  if (warp == 0) {
    const bool elected = ptx::elect_one();
    if (elected) {
      ptx::mbar_expect_tx(&w_full, C::W3_BYTES + C::W1_BYTES);
      for (int kb = 0; kb < C::KB; kb++) ptx::tma_load_2d(smem + kb * WIDE * 128, &maps.w3, &w_full, kb * 64, 0);
      for (int kb = 0; kb < CHUNKS; kb++) ptx::tma_load_2d(smem + C::W1_AT + kb * N2 * 128, &maps.w1, &w_full, kb * 64, 0);
    }
    int as = 0, rs = 0;
    uint32_t a_ph = 1, r_ph = 1;  // the first turn of each ring does not wait
    auto load_input = [&](int t) {
      const int y = ((int)blockIdx.x + t * (int)gridDim.x) * TM;
#pragma unroll
      for (int kb = 0; kb < C::KB; kb++) {
        if (!ptx::mbar_wait_warp(&a_free[as], a_ph)) return false;
        if (elected) {
          ptx::mbar_expect_tx(&a_full[as], BLOCK_BYTES);
          ptx::tma_load_2d(smem + C::A_AT + as * BLOCK_BYTES, kb ? &maps.x2 : &maps.x, &a_full[as], 0, y);
        }
        if (++as == C::A_SLOTS) as = 0, a_ph ^= 1u;
      }
      return true;
    };
    bool ok = mine == 0 || load_input(0);
    for (int t = 0; t < mine && ok; t++) {
      if (t + 1 < mine) ok = load_input(t + 1);
      if (!DUAL) {
        const int y = ((int)blockIdx.x + t * (int)gridDim.x) * TM;
        for (int c = 0; c < CHUNKS && ok; c++) {
          if (!(ok = ptx::mbar_wait_warp(&r_free[rs], r_ph))) break;
          if (elected) {
            ptx::mbar_expect_tx(&r_full[rs], BLOCK_BYTES);
            ptx::tma_load_2d(smem + C::RING_AT + rs * BLOCK_BYTES, &maps.residual, &r_full[rs], c * 64, y);
          }
          if (++rs == C::RING) rs = 0, r_ph ^= 1u;
        }
      }
      ok = __all_sync(0xffffffffu, ok && healthy());
    }
    if (!ok && elected) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_PRODUCER_WAIT);
    if (late_trigger) ptx::grid_dep_launch();
  } else if (warp == 1) {
    const bool elected = ptx::elect_one();
    constexpr uint32_t idesc = ptx::umma_idesc_bf16(TM, 64);
    const uint32_t w3_lo = ptx::umma_desc_lo(ptx::smem_u32(smem)), a_lo = ptx::umma_desc_lo(ptx::smem_u32(smem) + C::A_AT);
    int as = 0;
    uint32_t a_ph = 0;
    bool ok = ptx::mbar_wait_warp(&w_full, 0);
    for (int t = 0; t < mine && ok; t++) {
      int slots[C::KB];
#pragma unroll
      for (int kb = 0; kb < C::KB; kb++) {
        ok = ok && ptx::mbar_wait_warp(&a_full[as], a_ph);
        slots[kb] = as;
        if (++as == C::A_SLOTS) as = 0, a_ph ^= 1u;
      }
#pragma unroll
      for (int c = 0; c < CHUNKS; c++) {
        ok = ok && ptx::mbar_wait_warp(&acc_free[c], ((uint32_t)t & 1u) ^ 1u);
        if (!ok) break;
        ptx::tc_fence_after();
        if (elected) {
#pragma unroll
          for (int kb = 0; kb < C::KB; kb++)
#pragma unroll
            for (int k = 0; k < 4; k++)
              ptx::umma_bf16(tmem + c * 64, ptx::umma_desc_join(a_lo + slots[kb] * (BLOCK_BYTES / 16) + k * 2),
                             ptx::umma_desc_join(w3_lo + kb * (WIDE * 128 / 16) + c * (64 * 128 / 16) + k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
          ptx::umma_commit(&acc_full[c]);
        }
      }
      if (!ok) break;
      if (elected) {
#pragma unroll
        for (int kb = 0; kb < C::KB; kb++) ptx::umma_commit(&a_free[slots[kb]]);
      }
      ok = __all_sync(0xffffffffu, healthy());
    }
    if (!ok && elected) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_MMA_WAIT);
  } else if (warp == 3) {
    const bool elected = ptx::elect_one();
    constexpr uint32_t idesc = ptx::umma_idesc_bf16(TM, N2);
    const uint32_t w1_lo = ptx::umma_desc_lo(ptx::smem_u32(smem) + C::W1_AT), ring_lo = ptx::umma_desc_lo(ptx::smem_u32(smem) + C::RING_AT);
    int ps = 0;
    uint32_t p_ph = 0;
    bool ok = ptx::mbar_wait_warp(&w_full, 0);
    for (int t = 0; t < mine && ok; t++) {
      ok = ptx::mbar_wait_warp(&nar_free[t & 1], (((uint32_t)t >> 1) & 1u) ^ 1u);
      const uint32_t d = tmem_narrow + (t & 1) * 128;
#pragma unroll
      for (int c = 0; c < CHUNKS; c++) {
        ok = ok && ptx::mbar_wait_warp(&p_full[ps], p_ph);
        if (!ok) break;
        ptx::tc_fence_after();
        if (elected) {
#pragma unroll
          for (int k = 0; k < 4; k++)
            ptx::umma_bf16(d, ptx::umma_desc_join(ring_lo + ps * (BLOCK_BYTES / 16) + k * 2),
                           ptx::umma_desc_join(w1_lo + c * (N2 * 128 / 16) + k * 2), idesc, (c | k) != 0 ? 1u : 0u);
          ptx::umma_commit(&r_free[ps]);
        }
        if (++ps == C::RING) ps = 0, p_ph ^= 1u;
      }
      if (!ok) break;
      if (elected) ptx::umma_commit(&nar_full[t & 1]);
      ok = __all_sync(0xffffffffu, healthy());
    }
    if (!ok && elected) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_MMA_WAIT);
  } else if (warp == 2) {
    if (lane == 0) {
      int s = 0, before = 0;
      uint32_t ph = 0;
      for (int j = 0; j < chunks && healthy(); j++) {
        if (!ptx::mbar_wait(&p_full[s], ph)) {
          atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_EPILOGUE_WAIT);
          break;
        }
        const int y = ((int)blockIdx.x + (j / CHUNKS) * (int)gridDim.x) * TM;
        ptx::tma_store_2d(&maps.wide, smem + C::RING_AT + s * BLOCK_BYTES, (j & (CHUNKS - 1)) * 64, y);
        ptx::bulk_commit();
        ptx::bulk_wait_read<1>();  // the store before this one has been read
        if (j >= 1) ptx::mbar_arrive(&r_free[before]);
        before = s;
        if (++s == C::RING) s = 0, ph ^= 1u;
      }
      ptx::bulk_wait_all<0>();
    }
  } else if (warp >= 4 && warp < 12) {
    const int group = (warp - 4) >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    bool ok = true;
    for (int j = group; j < chunks && ok; j += 2) {
      const int slot = j & (ACC - 1), rs = j % C::RING;
      const uint32_t turn = (uint32_t)(j / C::RING);
      uint8_t* row_base = smem + C::RING_AT + rs * BLOCK_BYTES + row * 128;
      // the buffer: with the residual in it, or free
      ok = healthy() && (DUAL ? ptx::mbar_wait(&r_free[rs], (turn & 1u) ^ 1u) : ptx::mbar_wait(&r_full[rs], turn & 1u));
      uint4 res[8];
      if (!DUAL && ok) {
#pragma unroll
        for (int i = 0; i < 8; i++) res[i] = *reinterpret_cast<const uint4*>(row_base + ((i ^ (row & 7)) << 4));
      }
      ok = ok && ptx::mbar_wait(&acc_full[slot], ((uint32_t)j / ACC) & 1u);
      if (!(ok = __all_sync(0xffffffffu, ok))) break;
      ptx::tc_fence_after();
      const float* bias = s_b3 + (j & (CHUNKS - 1)) * 64;
      const uint32_t acc = tmem + slot * 64 + lane_base;
      uint32_t r[32];
      ptx::tmem_ld_32x32b_x32(acc, r);
      ptx::tmem_ld_wait();
      finish_32<!DUAL>(r, bias, res, row_base, 0, row);
      ptx::tmem_ld_32x32b_x32(acc + 32, r);
      ptx::tmem_ld_wait();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&acc_free[slot]);
      finish_32<!DUAL>(r, bias + 32, res + 4, row_base, 4, row);
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&p_full[rs]);
    }
    if (!ok && lane == 0) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_EPILOGUE_WAIT);
  } else if (warp >= 12) {
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    uint8_t* stage = smem + C::T_AT;
    bool ok = true;
    for (int t = 0; t < mine; t++) {
      const int buf = t & 1, y = ((int)blockIdx.x + t * (int)gridDim.x) * TM;
      ok = ptx::named_bar_all(1, 128, healthy() && ptx::mbar_wait(&nar_full[buf], ((uint32_t)t >> 1) & 1u));
      if (!ok) break;
      ptx::tc_fence_after();
#pragma unroll
      for (int h = 0; h < N2 / 64; h++) {
        uint32_t r[64];
        ptx::tmem_ld_32x32b_x32(tmem_narrow + buf * 128 + h * 64 + lane_base, r);
        ptx::tmem_ld_32x32b_x32(tmem_narrow + buf * 128 + h * 64 + lane_base + 32, r + 32);
        ptx::tmem_ld_wait();
        if (h == N2 / 64 - 1) {
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&nar_free[buf]);
        }
        // the staging block: the store before this one has been read
        if (threadIdx.x == 12 * 32) ptx::bulk_wait_read<0>();
        ptx::named_bar_all(1, 128, true);
        finish_32<false>(r, s_b1 + h * 64, nullptr, stage + row * 128, 0, row);
        finish_32<false>(r + 32, s_b1 + h * 64 + 32, nullptr, stage + row * 128, 4, row);
        ptx::fence_proxy_async_smem();
        ptx::named_bar_all(1, 128, true);
        if (threadIdx.x == 12 * 32) {
          ptx::tma_store_2d(&maps.narrow, stage, h * 64, y);
          ptx::bulk_commit();
        }
      }
    }
    if (threadIdx.x == 12 * 32) ptx::bulk_wait_all<0>();
    if (!ok && lane == 0) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_EPILOGUE_WAIT);
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (s_error != 0) {
    if (threadIdx.x == 0 && status) atomicExch(status, s_error);
    __nanosleep(1000000);  // let loads that are still in flight land before the block leaves
    __syncthreads();
  }
  if (warp == 3) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

template <int N2, bool DUAL>
cudaError_t launch_chain(const ConvChain& c, uint32_t* status, cudaStream_t stream) {
  using C = Chain<N2, DUAL>;
  static PerDeviceFlag attr;
  const int dev = PerDeviceFlag::current();
  if (attr.needed(dev)) {
    const cudaError_t e = cudaFuncSetAttribute(conv_chain_kernel<N2, DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return e;
    attr.set(dev);
  }
  ChainMaps m;
  const uint64_t rows = (uint64_t)c.pixels;
  cudaError_t e = srpc_tensor_map_2d(&m.x, c.x, 64, rows, 128, 64, TM);
  if (e == cudaSuccess) e = srpc_tensor_map_2d(&m.x2, DUAL ? c.x2 : c.x, 64, rows, 128, 64, TM);
  if (e == cudaSuccess) e = srpc_tensor_map_2d(&m.w3, c.w_wide, 64 * C::KB, WIDE, 128 * C::KB, 64, WIDE);
  if (e == cudaSuccess) e = srpc_tensor_map_2d(&m.w1, c.w_narrow, WIDE, N2, WIDE * 2, 64, N2);
  if (e == cudaSuccess) e = srpc_tensor_map_2d(&m.wide, c.wide, WIDE, rows, WIDE * 2, 64, TM);
  if (e == cudaSuccess) e = srpc_tensor_map_2d(&m.residual, DUAL ? c.wide : c.residual, WIDE, rows, WIDE * 2, 64, TM);
  if (e == cudaSuccess) e = srpc_tensor_map_2d(&m.narrow, c.narrow, N2, rows, N2 * 2, 64, TM);
  if (e != cudaSuccess) return e;
  const int grid = std::min((c.pixels + TM - 1) / TM, srpc_gemm_grid_sms());
  return launch_pdl(conv_chain_kernel<N2, DUAL>, dim3(grid), dim3(THREADS), C::SMEM, stream, m, c.pixels, c.b_wide, c.b_narrow,
                    (int)(srpc_gemm_reserved_sms() > 0), status);
}

}  // namespace

cudaError_t srpc_conv_chain(const ConvChain& c, uint32_t* status, cudaStream_t stream) {
  const void* aligned[] = {c.x, c.x2, c.w_wide, c.w_narrow, c.residual, c.wide, c.narrow};
  for (const void* p : aligned)
    if ((uintptr_t)p & 15) return cudaErrorInvalidValue;
  if (c.pixels < 1 || !c.b_wide || !c.b_narrow || !c.x2 == !c.residual) return cudaErrorInvalidValue;
  if (c.narrow_channels == 64) return c.x2 ? launch_chain<64, true>(c, status, stream) : launch_chain<64, false>(c, status, stream);
  if (c.narrow_channels == 128 && !c.x2) return launch_chain<128, false>(c, status, stream);
  return cudaErrorInvalidValue;
}

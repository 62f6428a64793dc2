// Linear layer for a few rows (the classifier of a batch): out[M, N] = a[M, K] . w[N, K]^T + bias in fp32, K up to 2048.
//
// The weights are the M operand of the tensor core: a cluster of eight CTAs makes 128 output columns of up to 32 rows, and each
// CTA takes an eighth of K.  64 x 1000 x 2048 is 128 short loads side by side (two CTAs fit an SM) instead of 126 long loops.
//
// The tensor core keeps fewer bits of a long sum than chains of fp32 additions do: one accumulator over K = 2048 is 25 times further
// from the exact sum than chains of fp32 FMAs.  So an accumulator gets one instruction only, 16 products per output (a sum of 16 products
// of one sign comes out 1.6e-8 low on average), and everything beyond is added in pairs in fp32.  The last four levels weigh most; there
// the rounding errors are kept and added at the end.  Relative error against 64 bits, 64 x 1000 outputs, chains of FMAs (fc_skinny) / here /
// here without the kept errors, K = 2048: operands of both signs 7.9e-8 / 6.3e-8 / 7.4e-8, one operand positive 7.9e-8 / 6.3e-8 / 7.5e-8, both
// positive 3.2e-8 / 2.8e-8 / 3.5e-8; K = 1544: 7.5e-8 / 6.3e-8 / 7.4e-8, 7.5e-8 / 6.3e-8 / 7.4e-8, 3.5e-8 / 3.3e-8 / 4.7e-8.
//
// The CTAs' sums travel by st.async: CTA r finishes rows r*4 .. r*4+3 for all 128 columns, and its mbarrier counts the bytes.
// 64 x 1000 x 2048: 11.8 (fc_skinny) -> 5.0 us, 32 rows 9.0 -> 4.3, 32 x 4096 x 2048 28.0 -> 5.5; most of it is the chain of load, product, exchange
// and store.  All sixteen accumulators of a CTA at once (512 columns, one CTA per SM) put 64 rows into two rounds: 6.8; 64 rows per CTA
// with 32 products: 4.7.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>

#include "gemm_tcgen05.h"
#include "nn_kernels.h"
#include "pdl_launch.h"
#include "per_device.h"
#include "ptx.cuh"

cudaError_t srpc_tensor_map_2d(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                               uint32_t box_inner, uint32_t box_outer);

namespace {

constexpr int CLUSTER = 8, COLS = 128, ROWS = 32, MAX_KB = 4;  // k-blocks of 64 per CTA
constexpr int THREADS = 256;
constexpr int W_BYTES = COLS * 128, A_BYTES = ROWS * 128, STAGE = W_BYTES + A_BYTES;
constexpr int RECV_BYTES = CLUSTER * COLS * 16;                // [source][column] of four rows
constexpr int SMEM = MAX_KB * STAGE + RECV_BYTES + 1024;
constexpr int TMEM_COLS = 2 * 4 * ROWS;                        // two k-blocks of four accumulators

__device__ __forceinline__ void st_async_v4(uint32_t addr, float4 v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "f"(v.x),
               "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
               : "memory");
}

// a + b, and what the rounding took away is added to err (Knuth's TwoSum).
__device__ __forceinline__ float add_keep_error(float a, float b, float& err) {
  const float s = a + b, t = s - a;
  err += (a - (s - t)) + (b - t);
  return s;
}

__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(THREADS, 2)
fc_cluster(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a, const float* bias, float* out, int ldo,
           int M, int N, int num_kb, int kb_per_cta, uint32_t* status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float4* recv = reinterpret_cast<float4*>(smem + MAX_KB * STAGE);
  __shared__ __align__(8) uint64_t full[MAX_KB], acc_full[2], acc_free, recv_full;
  __shared__ uint32_t tmem_base_smem, s_error;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const int n0 = ((int)blockIdx.x / CLUSTER) * COLS, m0 = (int)blockIdx.y * ROWS;
  const int kb0 = (int)rank * kb_per_cta, kbs = min(kb_per_cta, num_kb - kb0);  // may be <= 0: nothing to add

  if (threadIdx.x == 0) {
    for (int i = 0; i < MAX_KB; i++) ptx::mbar_init(&full[i], 1);
    ptx::mbar_init(&acc_full[0], 1);
    ptx::mbar_init(&acc_full[1], 1);
    ptx::mbar_init(&acc_free, THREADS / 32);
    ptx::mbar_init(&recv_full, 1);
    ptx::fence_mbar_init();
    ptx::mbar_expect_tx(&recv_full, RECV_BYTES);
    s_error = 0;
  }
  if (warp == 1) {
    ptx::tmem_alloc(&tmem_base_smem, TMEM_COLS);
    ptx::tmem_relinquish();
    ptx::grid_dep_launch();  // after the allocation, see pdl_launch.h
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_arrive_relaxed();  // the peers' barriers exist before anything is sent to them
  ptx::grid_dep_wait();
  ptx::tc_fence_after();
  const uint32_t tmem = tmem_base_smem;

  bool ok = true;
  const bool elected = ptx::elect_one();
  if (warp == 0 && elected) {
    for (int i = 0; i < kbs; i++) {
      ptx::mbar_expect_tx(&full[i], STAGE);
      ptx::tma_load_2d(smem + i * STAGE, &tmap_w, &full[i], (kb0 + i) * 64, n0);
      ptx::tma_load_2d(smem + i * STAGE + W_BYTES, &tmap_a, &full[i], (kb0 + i) * 64, m0);
    }
  }
  __syncwarp();
  // This warp adds up 32 output columns (accumulator rows) x 16 rows of the batch, in pairs: a k-block's four accumulators, k-blocks,
  // pairs of k-blocks.  A k-block that this CTA does not have adds nothing.
  const int quarter = warp & 3, half = warp >> 2;
  const uint32_t t_addr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 16);
  const uint32_t w_lo = ptx::umma_desc_lo(ptx::smem_u32(smem));
  constexpr uint32_t idesc = ptx::umma_idesc_bf16(COLS, ROWS);
  float sum[16];
#pragma unroll
  for (int j = 0; j < 16; j++) sum[j] = 0.f;
#pragma unroll
  for (int p = 0; p < MAX_KB / 2; p++) {
    if (2 * p >= kbs) break;
    if (warp == 1) {
      if (p > 0) ok = ok && ptx::mbar_wait_warp(&acc_free, 0);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        if (2 * p + i >= kbs) break;
        ok = ok && ptx::mbar_wait_warp(&full[2 * p + i], 0);
        ptx::tc_fence_after();
        if (ok && elected) {
#pragma unroll
          for (int k = 0; k < 4; k++)
            ptx::umma_bf16(tmem + (uint32_t)(i * 4 + k) * ROWS, ptx::umma_desc_join(w_lo + (2 * p + i) * (STAGE / 16) + k * 2),
                           ptx::umma_desc_join(w_lo + (2 * p + i) * (STAGE / 16) + W_BYTES / 16 + k * 2), idesc, 0u);
        }
      }
      if (elected) ptx::umma_commit(&acc_full[p]);
      __syncwarp();
    }
    ok = ptx::mbar_wait_warp(&acc_full[p], 0) && ok;
    ptx::tc_fence_after();
    float v[2][16];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      if (2 * p + i >= kbs) break;
      uint32_t r[4][16];
#pragma unroll
      for (int k = 0; k < 4; k++) ptx::tmem_ld_32x32b_x16(t_addr + (uint32_t)(4 * i + k) * ROWS, r[k]);
      ptx::tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; j++)
        v[i][j] = (__uint_as_float(r[0][j]) + __uint_as_float(r[1][j])) + (__uint_as_float(r[2][j]) + __uint_as_float(r[3][j]));
    }
    ptx::tc_fence_before();
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(&acc_free);
#pragma unroll
    for (int j = 0; j < 16; j++) sum[j] += 2 * p + 1 < kbs ? v[0][j] + v[1][j] : v[0][j];
  }
  ptx::cluster_wait();
  {
    // CTA r gets rows r*4 .. r*4+3
    const uint32_t dst = ptx::smem_u32(recv) + (rank * COLS + quarter * 32 + lane) * 16, bar = ptx::smem_u32(&recv_full);
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const uint32_t to = (uint32_t)(half * 4 + g);
      st_async_v4(ptx::mapa_shared(dst, to), make_float4(sum[g * 4], sum[g * 4 + 1], sum[g * 4 + 2], sum[g * 4 + 3]),
                  ptx::mapa_shared(bar, to));
    }
  }
  ptx::cluster_arrive_relaxed();  // nothing more goes to a peer
  // The peers' sums; every lane acquires for itself what it reads below.
  ok = __all_sync(0xffffffffu, ptx::mbar_wait<ptx::mbar_try_wait_cluster>(&recv_full, 0)) && ok;
  if (!ok && lane == 0) atomicExch(&s_error, (uint32_t)GEMM_ERR_EPILOGUE_WAIT);
  if (threadIdx.x < COLS) {
    const int c = threadIdx.x, n = n0 + c, m = m0 + (int)rank * 4;
    float v[CLUSTER][4], err[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < CLUSTER; s++) {
      const float4 q = recv[s * COLS + c];
      v[s][0] = q.x, v[s][1] = q.y, v[s][2] = q.z, v[s][3] = q.w;
    }
#pragma unroll
    for (int d = 1; d < CLUSTER; d *= 2)
#pragma unroll
      for (int s = 0; s < CLUSTER; s += 2 * d)
#pragma unroll
        for (int k = 0; k < 4; k++) v[s][k] = add_keep_error(v[s][k], v[s + d][k], err[k]);
    if (ok && n < N) {
      const float b = bias ? *(bias + n) : 0.f;
      float* o = out + (size_t)m * ldo + n;
      float r[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        r[k] = add_keep_error(v[0][k], b, err[k]);
        r[k] += err[k] == err[k] ? err[k] : 0.f;  // (not a number beside infinities; r is right then)
      }
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (m + k < M) o[(size_t)k * ldo] = r[k];
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (s_error != 0) {
    if (threadIdx.x == 0 && status) atomicExch(status, s_error);
    __nanosleep(1000000);  // let loads that are still in flight land before the block leaves
    __syncthreads();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, TMEM_COLS);
  }
  ptx::cluster_wait();  // no peer sends to a block that has left
}

cudaError_t prepare(int dev) {
  static PerDeviceFlag attr;
  if (!attr.needed(dev)) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(fc_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e == cudaSuccess) attr.set(dev);
  return e;
}

}  // namespace

bool nn_fc_cluster_fits() {
  static std::atomic<int> fits[64];  // per device: 0 not asked yet, 1 yes, 2 no
  const int dev = PerDeviceFlag::current();
  int f = fits[dev].load(std::memory_order_relaxed);
  if (f == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CLUSTER);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM;
    int n = 0;
    const bool ok = prepare(dev) == cudaSuccess && cudaOccupancyMaxActiveClusters(&n, fc_cluster, &cfg) == cudaSuccess && n >= 1;
    if (!ok) (void)cudaGetLastError();  // the other kernel runs; nothing is left behind for a later check
    fits[dev].store(f = ok ? 1 : 2, std::memory_order_relaxed);
  }
  return f == 1;
}

cudaError_t nn_fc_cluster(const void* a, int lda, const void* w, int ldw, const float* bias, float* out, int ldo, int M, int N, int K,
                          uint32_t* status, cudaStream_t s) {
  const int num_kb = (K + 63) / 64, kb_per_cta = (num_kb + CLUSTER - 1) / CLUSTER;
  if (kb_per_cta > MAX_KB || M < 1 || N < 1) return cudaErrorInvalidValue;
  CUtensorMap tw, ta;
  cudaError_t e = prepare(PerDeviceFlag::current());
  if (e == cudaSuccess) e = srpc_tensor_map_2d(&tw, w, (uint64_t)K, (uint64_t)N, (uint64_t)ldw * 2, 64, COLS);
  if (e == cudaSuccess) e = srpc_tensor_map_2d(&ta, a, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, 64, ROWS);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((N + COLS - 1) / COLS) * CLUSTER, (unsigned)((M + ROWS - 1) / ROWS));
  return launch_pdl(fc_cluster, grid, dim3(THREADS), (size_t)SMEM, s, tw, ta, bias, out, ldo, M, N, num_kb, kb_per_cta, status);
}

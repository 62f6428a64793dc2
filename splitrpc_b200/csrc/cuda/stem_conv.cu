// Convolution over overlapping 64-channel windows of 16-channel pixels: four row taps, 64 output channels (the ResNet stem on
// the space-to-depth image, see stem_s2d in nn_kernels.cu).
//
//   out[n, y, x, :] = act(sum over fr < 4, j < 4 of W[:, fr, j*16 .. j*16+15] . in[n, y + fr, x + j, :] + bias)
//
// As an ordinary implicit GEMM every output pixel pulls its 4 x 128-byte windows through the TMA unit and into shared
// memory, 16 times the bytes of the input, in 128-byte pieces that start off the 128-byte lines: 71 us for 64 images.  Here an
// input pixel enters shared memory once per chunk, split into two planes of 16 bytes per pixel.  Eight pixels of a
// plane are then one 8 x 16-byte core matrix of an unswizzled K-major operand, whatever pixel they start at, so the operand
// of tap (fr, j) is the same memory read from another start address, and overlapping windows cost nothing.
// Output positions are numbered along the padded row (width + 3 pixels): 128 consecutive positions are one tile whose operand
// is one run of memory; the three positions per row that lie past the output's width are computed and dropped.
//
// One persistent CTA per SM.  A work item is a chunk of up to MAX_TILES tiles of one image.
//   warp 0      weights by TMA once, then one elected lane issues 16 MMAs (128 x 64 x 16) per tile into one of eight
//               accumulators, taps in the order of the generic kernel, so that results are bit-identical to it
//   warps 1-3   move the next chunk's pixels through registers into the other of two buffers
//   warps 4-15  read accumulators as 8 x 8 fragments (four warps per tile, three tiles at a time), bias from registers,
//               activation, bf16, transpose through a swizzled 4 KB buffer per warp (stmatrix), 512-byte coalesced stores
// 64 images: 37.8 us, 32 images 19.7 (71 us for 64 in the generic kernel; the output alone takes 16 us of memory time).  What
// bounds it is shared memory: 48.2 us with a bias read from shared memory per value and pixels copied by cp.async, 41.8 with
// the fragment epilogue alone; without the pixel copies it would be 31.5, with a quarter of the MMAs 33, without stores 39.
// Waits are bounded as in gemm_persistent.cu.
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

constexpr int BM = 128, COUT = 64, TAPS = 4, WIN = 4;  // window: 4 pixels of 16 channels
constexpr int MAX_TILES = 8;
constexpr int MAX_PITCH = 115;                          // padded row width a chunk's buffer is sized for
constexpr int MAX_PIX = MAX_TILES * BM + (TAPS - 1) * MAX_PITCH + WIN - 1;
constexpr int PLANE = (MAX_PIX * 16 + 127) / 128 * 128;
constexpr int BUF_BYTES = 2 * PLANE;
constexpr int W_BYTES = TAPS * COUT * 128;
constexpr int LOADERS = 96, EPI_WARPS = 12, THREADS = 32 + LOADERS + EPI_WARPS * 32;
constexpr int STAGE_BYTES = 32 * 128;                   // per epilogue warp: 32 pixels x 64 channels
constexpr int SMEM_BYTES = W_BYTES + 2 * BUF_BYTES + EPI_WARPS * STAGE_BYTES;
constexpr int ACC = 8;

struct StemParams {
  const uint8_t* in;            // image 0 (or the ring's base with in_stub)
  const void* in_stub;          // its first word names the first image when the kernel runs
  unsigned long long img_bytes; // distance between images
  int pitch, in_rows;           // pixels per padded row, rows of an image
  int ow, oh, n;
  int tiles;                    // tiles of the largest chunk
  int chunks_per_img;
  int relu;
  int late_trigger;             // the next kernel starts behind this CTA's last load only (pdl_launch.h)
  const float* bias;
  __nv_bfloat16* out;
};

__global__ void __launch_bounds__(THREADS, 1) stem_conv_kernel(const __grid_constant__ CUtensorMap tmap_w, const StemParams p, uint32_t* status) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* s_w = smem;
  uint8_t* s_in = smem + W_BYTES;
  uint8_t* s_out = smem + W_BYTES + 2 * BUF_BYTES;
  __shared__ __align__(8) uint64_t w_bar, full_bar[2], empty_bar[2], acc_full[ACC], acc_empty[ACC];
  __shared__ __align__(16) float s_bias[COUT];
  __shared__ uint32_t tmem_base_smem, s_error;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool layout_ok = (ptx::smem_u32(smem) & 1023u) == 0;
  if (threadIdx.x == 0) {
    ptx::mbar_init(&w_bar, 1);
    for (int i = 0; i < 2; i++) {
      ptx::mbar_init(&full_bar[i], LOADERS);
      ptx::mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < ACC; i++) {
      ptx::mbar_init(&acc_full[i], 1);
      ptx::mbar_init(&acc_empty[i], 4);
    }
    ptx::fence_mbar_init();
    s_error = layout_ok ? 0u : (uint32_t)GEMM_ERR_PRODUCER_WAIT;
    ptx::prefetch_tmap(&tmap_w);
  }
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_alloc(&tmem_base_smem, ACC * COUT);
    ptx::tmem_relinquish();
    if (!p.late_trigger) ptx::grid_dep_launch();  // after the allocation, see pdl_launch.h
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = tmem_base_smem;
  ptx::grid_dep_wait();
  if (threadIdx.x < COUT) s_bias[threadIdx.x] = p.bias ? p.bias[threadIdx.x] : 0.f;
  __syncthreads();

  const int n_chunks = p.n * p.chunks_per_img, n_pos = p.oh * p.pitch;
  const int chunk_pos = p.tiles * BM;
  auto tiles_of = [&](int c) {  // tiles of chunk c (the last of an image may be shorter)
    const int left = n_pos - (c % p.chunks_per_img) * chunk_pos;
    return min(p.tiles, (left + BM - 1) / BM);
  };
  if (layout_ok) {
    if (warp == 0) {
      // ---------------- weights, MMA
      const bool elected = ptx::elect_one();
      if (elected) {
        ptx::mbar_expect_tx(&w_bar, W_BYTES);
        for (int fr = 0; fr < TAPS; fr++) ptx::tma_load_2d(s_w + fr * COUT * 128, &tmap_w, &w_bar, fr * 64, 0);
      }
      bool ok = ptx::mbar_wait_warp(&w_bar, 0);
      const uint32_t idesc = ptx::umma_idesc_bf16(BM, COUT);
      const uint32_t w_lo = ptx::umma_desc_lo(ptx::smem_u32(s_w));
      // unswizzled K-major operand: core matrices along K are a plane apart, 8-pixel groups 128 bytes
      constexpr uint32_t a_hi = (128u >> 4) | (1u << 14);
      const uint32_t pitch = (uint32_t)p.pitch;
      uint32_t tile = 0;
      int it = 0;
      for (int c = blockIdx.x; ok && c < n_chunks; c += gridDim.x, it++) {
        const int buf = it & 1;
        ok = ptx::mbar_wait_warp(&full_bar[buf], (it >> 1) & 1);
        if (!ok) break;
        const uint32_t a_lo = (ptx::smem_u32(s_in + buf * BUF_BYTES) >> 4) | ((uint32_t)(PLANE >> 4) << 16);
        const int nt = tiles_of(c);
        for (int r = 0; r < nt; r++, tile++) {
          const uint32_t acc = tile & (ACC - 1);
          ok = ptx::mbar_wait_warp(&acc_empty[acc], ((tile / ACC) & 1u) ^ 1u);
          if (!ok) break;
          ptx::tc_fence_after();
          const uint32_t a0 = a_lo + (uint32_t)(r * BM);
          if (elected) {
#pragma unroll
            for (int fr = 0; fr < TAPS; fr++)
#pragma unroll
              for (int j = 0; j < WIN; j++)
                ptx::umma_bf16(tmem + acc * COUT, ((uint64_t)a_hi << 32) | (a0 + fr * pitch + j),
                               ptx::umma_desc_join(w_lo + (uint32_t)(fr * COUT * 128 / 16 + j * 2)), idesc, (fr | j) != 0 ? 1u : 0u);
            ptx::umma_commit(&acc_full[acc]);
          }
        }
        if (ok && elected) ptx::umma_commit(&empty_bar[buf]);
      }
      if (!ok && elected) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_MMA_WAIT);
    } else if (warp < 1 + LOADERS / 32) {
      // ---------------- pixels of chunk c into buffer it & 1.  A warp moves 16 pixels at a time through registers: its eight-lane
      // groups store 128 bytes of one plane each.  (cp.async writes a pixel's two halves, which lie in different planes, 16 bytes
      // at a time: 10 us of 64 images' 42 were that.)
      const int lw = warp - 1, plane = (lane >> 3) & 1, px_in_unit = (lane & 7) + ((lane >> 4) << 3);
      const uint8_t* img0 = p.in_stub ? *reinterpret_cast<uint8_t* const*>(p.in_stub) : p.in;
      const int img_pix = p.pitch * p.in_rows;
      int it = 0;
      for (int c = blockIdx.x; c < n_chunks; c += gridDim.x, it++) {
        if (!ptx::mbar_wait_warp(&empty_bar[it & 1], ((it >> 1) & 1) ^ 1u)) {
          if (lane == 0) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_PRODUCER_WAIT);
          break;
        }
        const int img = c / p.chunks_per_img, first = (c - img * p.chunks_per_img) * chunk_pos;
        const int n_pix = tiles_of(c) * BM + (TAPS - 1) * p.pitch + WIN - 1;
        const int inside = min(n_pix, img_pix - first);  // past the image: zeros
        const uint8_t* src = img0 + (size_t)img * p.img_bytes + (size_t)first * 32 + plane * 16;
        uint8_t* dst = s_in + (it & 1) * BUF_BYTES + plane * PLANE;
        constexpr int AHEAD = 8;  // loads in flight per thread
        for (int base = lw * 16 + px_in_unit; base < n_pix; base += AHEAD * LOADERS / 2) {
          uint4 q[AHEAD];
#pragma unroll
          for (int k = 0; k < AHEAD; k++) {
            const int px = base + k * (LOADERS / 2);
            q[k] = px < inside ? *reinterpret_cast<const uint4*>(src + (size_t)px * 32) : make_uint4(0u, 0u, 0u, 0u);
          }
#pragma unroll
          for (int k = 0; k < AHEAD; k++) {
            const int px = base + k * (LOADERS / 2);
            if (px < n_pix) *reinterpret_cast<uint4*>(dst + px * 16) = q[k];
          }
        }
        ptx::fence_proxy_async_smem();
        ptx::mbar_arrive(&full_bar[it & 1]);
      }
      if (p.late_trigger && warp == 1) {
        __syncwarp();
        ptx::grid_dep_launch();
      }
    } else {
      // ---------------- epilogue: each set of four warps takes every third tile; a warp has 32 positions
      const int ew = warp - 4, set = ew >> 2, quarter = warp & 3;
      uint8_t* stage = s_out + ew * STAGE_BYTES;
      float2 bias[8];
#pragma unroll
      for (int g = 0; g < 8; g++) bias[g] = make_float2(s_bias[g * 8 + (lane & 3) * 2], s_bias[g * 8 + (lane & 3) * 2 + 1]);
      uint32_t tile = 0;
      bool ok = true;
      for (int c = blockIdx.x; ok && c < n_chunks; c += gridDim.x) {
        const int img = c / p.chunks_per_img, first = (c - img * p.chunks_per_img) * chunk_pos;
        const int nt = tiles_of(c);
        for (int r = 0; r < nt; r++, tile++) {
          if ((int)(tile % 3u) != set) continue;
          const uint32_t acc = tile & (ACC - 1);
          ok = ptx::mbar_wait_warp(&acc_full[acc], (tile / ACC) & 1u);
          if (!ok) break;
          ptx::tc_fence_after();
          // 32 positions x 64 channels as 8 x 8 fragments (see gemm_2sm.cu): a thread's bias is 16 values for the whole launch
          uint32_t v[4][16];  // [half of the channels][half of the positions]
          const uint32_t at = tmem + acc * COUT + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
          for (int q = 0; q < 4; q++) ptx::tmem_ld_16x256b_x4(at + (q >> 1) * 32 + ((uint32_t)((q & 1) * 16) << 16), v[q]);
          ptx::tmem_ld_wait();
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&acc_empty[acc]);
#pragma unroll
          for (int q = 0; q < 4; q++) {
            uint32_t o[8];  // [channel group][position group of 8]
#pragma unroll
            for (int k = 0; k < 8; k++) {
              float2 f = __fadd2_rn(make_float2(__uint_as_float(v[q][2 * k]), __uint_as_float(v[q][2 * k + 1])), bias[(q >> 1) * 4 + (k >> 1)]);
              if (p.relu) f = make_float2(fmaxf(f.x, 0.f), fmaxf(f.y, 0.f));
              const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
              o[k] = *reinterpret_cast<const uint32_t*>(&h);
            }
            const int row = (q & 1) * 16 + (lane & 15);
#pragma unroll
            for (int g = 0; g < 4; g += 2)  // the two position groups of channel groups g, g + 1
              ptx::stmatrix_x4(ptx::smem_u32(stage) + row * 128 + ((((q >> 1) * 4 + g + (lane >> 4)) ^ (row & 7)) << 4), o[2 * g], o[2 * g + 1],
                               o[2 * g + 2], o[2 * g + 3]);
          }
          __syncwarp();
          const int pos0 = first + r * BM + quarter * 32 + (lane >> 3);
          int y = pos0 / p.pitch, x = pos0 - y * p.pitch;
#pragma unroll
          for (int i = 0; i < 8; i++) {  // four positions of 128 bytes per store
            const int row = i * 4 + (lane >> 3);
            const uint4 o = *reinterpret_cast<const uint4*>(stage + row * 128 + (((lane & 7) ^ (row & 7)) << 4));
            if (x < p.ow && y < p.oh)
              *reinterpret_cast<uint4*>(p.out + (((size_t)img * p.oh + y) * p.ow + x) * COUT + (lane & 7) * 8) = o;
            x += 4;
            if (x >= p.pitch) {
              x -= p.pitch;
              y++;
            }
          }
          __syncwarp();
        }
      }
      if (!ok && lane == 0) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_EPILOGUE_WAIT);
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (s_error != 0) {
    if (threadIdx.x == 0 && status) atomicExch(status, s_error);
    __nanosleep(1000000);  // let loads that are still in flight land before the block leaves
    __syncthreads();
  }
  if (warp == 0) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, ACC * COUT);
  }
}

}  // namespace

// Takes the convolutions of the form in this file's header; everything else stays with the generic kernel.
bool srpc_stem_conv_eligible(const ConvShape& cs, const GemmEpilogue& ep) {
  static const int allow = [] { const char* e = getenv("SPLITRPC_STEM_CONV"); return e ? atoi(e) : 1; }();
  return allow && cs.r == TAPS && cs.s == 1 && cs.stride == 1 && cs.pad == 0 && cs.cin == WIN * 16 && cs.cout == COUT && !cs.in2 &&
         cs.in_pix_stride == 16 && cs.in_row_stride == (long)(cs.w + WIN - 1) * 16 && cs.w + WIN - 1 <= MAX_PITCH &&
         cs.in_img_stride >= (long)cs.h * cs.in_row_stride && cs.in_img_stride % 8 == 0 && !ep.residual && (ep.act == GEMM_ACT_NONE || ep.act == GEMM_ACT_RELU);
}

cudaError_t srpc_stem_conv(const void* in, const void* weight, const ConvShape& cs, const GemmEpilogue& ep, uint32_t* status,
                           cudaStream_t stream) {
  static PerDeviceFlag attr;
  const int dev = PerDeviceFlag::current();
  if (attr.needed(dev)) {
    const cudaError_t e = cudaFuncSetAttribute(stem_conv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return e;
    attr.set(dev);
  }
  CUtensorMap tw;
  const cudaError_t e = srpc_tensor_map_2d(&tw, weight, (uint64_t)TAPS * 64, COUT, (uint64_t)TAPS * 128, 64, COUT);
  if (e != cudaSuccess) return e;
  StemParams p{};
  p.in = (const uint8_t*)in;
  p.in_stub = cs.in_stub;
  p.img_bytes = (unsigned long long)cs.in_img_stride * 2;
  p.pitch = cs.w + WIN - 1;
  p.in_rows = cs.h;
  p.ow = cs.ow;
  p.oh = cs.oh;
  p.n = cs.n;
  p.relu = ep.act == GEMM_ACT_RELU;
  p.late_trigger = srpc_gemm_reserved_sms() > 0;
  p.bias = ep.bias;
  p.out = (__nv_bfloat16*)ep.out;
  // Tiles per chunk: few for small batches, so that every SM has a chunk; a chunk costs the rows shared with its neighbour
  // and a hand-over, about one tile's time.
  const int sms = srpc_gemm_grid_sms(), tiles_img = (p.oh * p.pitch + BM - 1) / BM;
  long best = 1l << 60;
  for (int t = MAX_TILES; t >= 1; t--) {
    const long per_img = (tiles_img + t - 1) / t, rounds = (per_img * cs.n + sms - 1) / sms, cost = rounds * (t + 1);
    if (cost < best) {
      best = cost;
      p.tiles = t;
      p.chunks_per_img = (int)per_img;
    }
  }
  const int grid = std::min(sms, cs.n * p.chunks_per_img);
  return launch_pdl(stem_conv_kernel, dim3(grid), dim3(THREADS), (size_t)SMEM_BYTES, stream, tw, p, status);
}

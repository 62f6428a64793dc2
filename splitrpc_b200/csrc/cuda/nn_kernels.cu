// Memory-bound layers around the tensor-core kernels: request deserialisation,
// pooling, normalisation, softmax/argmax response writers, embedding and attention.
//
// These stand in for the cuDNN/TensorRT layers the original reaches through ONNX
// Runtime (reference src/apps/ort_app.h:511-516).  Activations are bf16 (NHWC for
// images, [tokens, hidden] for sequences); statistics are computed in fp32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "../host/p2p_rpc_app.h"
#include "gemm_tcgen05.h"
#include "nn_kernels.h"
#include "pdl_launch.h"
#include "per_device.h"
#include "ptx.cuh"
#include "resp_push.cuh"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int s = 16; s; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int s = 16; s; s >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, s));
  return v;
}

// Block-wide sum of one value per thread (blockDim.x <= 1024, multiple of 32).
__device__ __forceinline__ float block_sum(float v, float* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float t = (l < nw) ? sh[l] : 0.f;
  t = warp_sum(t);
  return t;
}

// ------------------------------------------------------------------ ResNet stem input
// Request = fp32 CHW image (3 x 224 x 224).  Writes the im2col matrix of the 7x7
// stride-2 pad-3 stem convolution: row = output pixel (n, oy, ox), 192 bf16
// columns ordered k = ky*24 + c*8 + kx (kx = 7 and k >= 168 are zero), after
// (x - mean[c]) * inv_std[c].  With this order one 16-byte chunk of a row is 7
// consecutive input pixels of one image row and channel, so a thread reads 28
// contiguous bytes and writes one 16-byte store.
__global__ void __launch_bounds__(256) stem_im2col(const g_params* stub, const float* direct_in, int batch,
                                                   __nv_bfloat16* out, float3 mean, float3 inv_std) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const float* in = direct_in ? direct_in : reinterpret_cast<const float*>(stub->req);
  const size_t total = (size_t)batch * 112 * 112 * 24;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int kc = (int)(i % 24);
    const size_t pix = i / 24;
    uint4 o = make_uint4(0u, 0u, 0u, 0u);
    if (kc < 21) {
      const int ky = kc / 3, c = kc - ky * 3;
      const int ox = (int)(pix % 112), oy = (int)((pix / 112) % 112), n = (int)(pix / (112 * 112));
      const int iy = oy * 2 - 3 + ky, ix0 = ox * 2 - 3;
      if (iy >= 0 && iy < 224) {
        const float m = c == 0 ? mean.x : (c == 1 ? mean.y : mean.z);
        const float s = c == 0 ? inv_std.x : (c == 1 ? inv_std.y : inv_std.z);
        const float* row = in + (((size_t)n * 3 + c) * 224 + iy) * 224;
        float v[8];
#pragma unroll
        for (int j = 0; j < 7; j++) {
          const int ix = ix0 + j;
          v[j] = (ix >= 0 && ix < 224) ? (*(row + ix) - m) * s : 0.f;
        }
        v[7] = 0.f;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int t = 0; t < 4; t++) h[t] = __floats2bfloat162_rn(v[2 * t], v[2 * t + 1]);
      }
    }
    *reinterpret_cast<uint4*>(out + pix * 192 + kc * 8) = o;
  }
}

// Space-to-depth form of the stem input.  The 7x7 stride-2 pad-3 convolution over 3 channels equals a 4x4 stride-1
// convolution over the 2x2 space-to-depth transform of the zero-padded (230 x 230) image.  Writes
// out[n][Y][X][16] bf16 with Y, X < 115 and channel dy*8 + dx*3 + c = normalised input pixel (2Y+dy-3, 2X+dx-3) of
// channel c (zero outside the image; channels 6, 7, 14, 15 are zero).  Four horizontally adjacent pixels are 64
// contiguous channels, so the convolution reads its rows straight from this array through a tensor map whose pixel
// stride is 16 elements: no im2col matrix is ever written (27 MB per 64 images instead of 308 MB).
__global__ void __launch_bounds__(256) stem_s2d(const g_params* stub, const float* direct_in, int batch,
                                                __nv_bfloat16* out, float3 mean, float3 inv_std) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const float* in = direct_in ? direct_in : reinterpret_cast<const float*>(stub->req);
  const size_t total = (size_t)batch * 115 * 115 * 2;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int dy = (int)(i & 1);
    const size_t pix = i >> 1;
    const int X = (int)(pix % 115), Y = (int)((pix / 115) % 115), n = (int)(pix / (115 * 115));
    const int iy = 2 * Y + dy - 3, ix0 = 2 * X - 3;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = 0.f;
    if (iy >= 0 && iy < 224) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const float m = c == 0 ? mean.x : (c == 1 ? mean.y : mean.z);
        const float s = c == 0 ? inv_std.x : (c == 1 ? inv_std.y : inv_std.z);
        const float* row = in + (((size_t)n * 3 + c) * 224 + iy) * 224;
#pragma unroll
        for (int dx = 0; dx < 2; dx++) {
          const int ix = ix0 + dx;
          if (ix >= 0 && ix < 224) v[dx * 3 + c] = (*(row + ix) - m) * s;
        }
      }
    }
    uint4 o;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int t = 0; t < 4; t++) h[t] = __floats2bfloat162_rn(v[2 * t], v[2 * t + 1]);
    *reinterpret_cast<uint4*>(out + pix * 16 + dy * 8) = o;
  }
}

// 3x3 stride-2 pad-1 max pooling, NHWC bf16, 8 channels per thread.  Window positions outside the image are clamped
// to the nearest pixel inside (a duplicate does not change a maximum), so the nine 16-byte loads of a thread carry no
// branches and are all in flight together.
__global__ void __launch_bounds__(256) maxpool3x3s2(const __nv_bfloat16* in, __nv_bfloat16* out,
                                                    int n, int h, int w, int c) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const int oh = (h + 2 - 3) / 2 + 1, ow = (w + 2 - 3) / 2 + 1, cv = c / 8;
  const size_t total = (size_t)n * oh * ow * cv;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int cc = (int)(i % cv);
    size_t p = i / cv;
    const int ox = (int)(p % ow);
    p /= ow;
    const int oy = (int)(p % oh), b = (int)(p / oh);
    uint4 q[9];
#pragma unroll
    for (int dy = 0; dy < 3; dy++) {
      const int iy = min(max(oy * 2 - 1 + dy, 0), h - 1);
#pragma unroll
      for (int dx = 0; dx < 3; dx++) {
        const int ix = min(max(ox * 2 - 1 + dx, 0), w - 1);
        q[dy * 3 + dx] = *(reinterpret_cast<const uint4*>(in + (((size_t)b * h + iy) * w + ix) * c + cc * 8));
      }
    }
    __nv_bfloat162 m[4];
    {
      const __nv_bfloat162* h0 = reinterpret_cast<const __nv_bfloat162*>(&q[0]);
#pragma unroll
      for (int t = 0; t < 4; t++) m[t] = h0[t];
    }
#pragma unroll
    for (int k = 1; k < 9; k++) {
      const __nv_bfloat162* hq = reinterpret_cast<const __nv_bfloat162*>(&q[k]);
#pragma unroll
      for (int t = 0; t < 4; t++) m[t] = __hmax2(m[t], hq[t]);
    }
    uint4 o;
    __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int t = 0; t < 4; t++) ho[t] = m[t];
    *reinterpret_cast<uint4*>(out + (((size_t)b * oh + oy) * ow + ox) * c + cc * 8) = o;
  }
}

// Global average pooling NHWC -> [n, c]; block (x = channel chunk of 512, y = image), two channels per thread, the
// pixel loop unrolled so that several loads are in flight.
__global__ void __launch_bounds__(256) global_avgpool(const __nv_bfloat16* in, __nv_bfloat16* out,
                                                      int hw, int c) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const int b = blockIdx.y, ch = (blockIdx.x * 256 + threadIdx.x) * 2;
  if (ch >= c) return;
  const __nv_bfloat16* src = in + (size_t)b * hw * c + ch;
  float s0 = 0.f, s1 = 0.f;
  int p = 0;
  for (; p + 7 <= hw; p += 7) {
    __nv_bfloat162 v[7];
#pragma unroll
    for (int j = 0; j < 7; j++) v[j] = *reinterpret_cast<const __nv_bfloat162*>(src + (size_t)(p + j) * c);
#pragma unroll
    for (int j = 0; j < 7; j++) {
      float2 f = __bfloat1622float2(v[j]);
      s0 += f.x;
      s1 += f.y;
    }
  }
  for (; p < hw; p++) {
    float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(src + (size_t)p * c));
    s0 += f.x;
    s1 += f.y;
  }
  *reinterpret_cast<__nv_bfloat162*>(out + (size_t)b * c + ch) = __floats2bfloat162_rn(s0 / hw, s1 / hw);
}

// Skinny fully connected layer: out[m, n] = sum_k a[m, k] * w[n, k] + bias[n] for a handful of rows, fp32 output and fp32 sums
// (the tensor cores' accumulator rounds more).  A block owns FC_NB output columns and 16 * RPT rows: a warp copies the weights of
// one column into shared memory, in four parts of K that arrive behind one another, so that the arithmetic starts with the first;
// thread (row group, kq) walks every sixteenth 8-element slice of its RPT rows of `a` with the next slice's loads in flight, and
// the sixteen partial sums of a row meet through shuffles that halve the list of values at every step.  A slice's weights are
// read from shared memory and converted once for the RPT rows.  Two rows stay for up to 32 rows, where there are enough of them
// for one block per column group anyway.  PER_SM: blocks that the registers leave room for on an SM, see nn_fc_skinny.
// Us, before (weights staged whole, as fp32, before any arithmetic; 128 shuffles per thread) and now: 64 x 1000 x 2048 12.85 and
// 11.75, 64 x 1192 x 512 9.9 and 7.4, 128 x 1000 x 512 10.1 and 7.6, 64 x 8192 x 768 38 and 31, 32 x 1192 x 512 6.4 and 5.2.  The loop
// is bound by what it reads through the L1 / shared-memory path (9.5 of the first, the FMAs are 4.2): deeper prefetch, twice the
// warps or scalar FMAs change nothing.  The order of every sum is the same in all forms.  K from 1537 to 2048 goes to fc_cluster.cu,
// see nn_fc_skinny.
constexpr int FC_NB = 8, FC_PARTS = 4;
template <int RPT, int PER_SM>
__global__ void __launch_bounds__(256, PER_SM) fc_skinny(const __nv_bfloat16* a, int lda, const __nv_bfloat16* w,
                                                 int ldw, const float* bias, float* out, int ldo, int M,
                                                 int N, int K) {
  static_assert(FC_NB == 8 && FC_PARTS == 4, "one warp per column, three steps over the columns; four waits below");
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  extern __shared__ __align__(16) uint4 s_w[];  // [FC_NB][K/8]
  const int n0 = blockIdx.x * FC_NB, kvn = K / 8, turns = (kvn + 15) / 16;
  const int kq = threadIdx.x & 15;
  const int row0 = blockIdx.y * (16 * RPT) + (threadIdx.x >> 4) * RPT;
  {
    const int col = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool in = n0 + col < N;
    const __nv_bfloat16* wr = w + (size_t)(in ? n0 + col : 0) * ldw;
#pragma unroll
    for (int part = 0; part < FC_PARTS; part++) {
      const int end = min(kvn, turns * (part + 1) / FC_PARTS * 16);
      for (int kv = turns * part / FC_PARTS * 16 + lane; kv < end; kv += 32) ptx::cp_async_16(s_w + col * kvn + kv, wr + kv * 8, in);
      ptx::cp_async_commit();
    }
  }
  // rows past M read row M-1 again (their results are not stored): no branch inside the loop
  const __nv_bfloat16* ar[RPT];
#pragma unroll
  for (int r = 0; r < RPT; r++) ar[r] = a + (size_t)min(row0 + r, M - 1) * lda;
  auto load = [&](const __nv_bfloat16* r, int kv) {
    return kv < kvn ? *(reinterpret_cast<const uint4*>(r + kv * 8)) : make_uint4(0, 0, 0, 0);
  };
  // AHEAD slices of every row are in flight, the first ones beside the weights.
  constexpr int AHEAD = RPT == 2 ? 2 : 1;
  uint4 qa[AHEAD][RPT];
#pragma unroll
  for (int d = 0; d < AHEAD; d++)
#pragma unroll
    for (int r = 0; r < RPT; r++) qa[d][r] = load(ar[r], kq + 16 * d);
  // packed fp32 FMAs (two per instruction): element x of an accumulator sums the even k, element y the odd k
  float2 acc[RPT][FC_NB];
#pragma unroll
  for (int r = 0; r < RPT; r++)
#pragma unroll
    for (int j = 0; j < FC_NB; j++) acc[r][j] = make_float2(0.f, 0.f);
  auto slice = [&](int kv, uint4 (&q)[RPT]) {
    float2 x[RPT][4];
#pragma unroll
    for (int r = 0; r < RPT; r++) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q[r]);
#pragma unroll
      for (int t = 0; t < 4; t++) x[r][t] = __bfloat1622float2(h[t]);
    }
#pragma unroll
    for (int r = 0; r < RPT; r++) q[r] = load(ar[r], kv + 16 * AHEAD);  // in flight during the arithmetic
#pragma unroll
    for (int j = 0; j < FC_NB; j++) {
      const uint4 wv = s_w[j * kvn + kv];
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const float2 wq = __bfloat1622float2(h[t]);
#pragma unroll
        for (int r = 0; r < RPT; r++) acc[r][j] = __ffma2_rn(x[r][t], wq, acc[r][j]);
      }
    }
  };
  int turn = 0;
#pragma unroll
  for (int part = 0; part < FC_PARTS; part++) {
    if (part == 0) ptx::cp_async_wait<3>();
    else if (part == 1) ptx::cp_async_wait<2>();
    else if (part == 2) ptx::cp_async_wait<1>();
    else ptx::cp_async_wait<0>();
    __syncthreads();
    const int end = turns * (part + 1) / FC_PARTS;
#pragma unroll 1
    for (; turn < end; turn++) {
      if (turn * 16 + kq >= kvn) continue;
      if (AHEAD > 1 && (turn & 1)) slice(turn * 16 + kq, qa[AHEAD - 1]);  // slice `turn` is in qa[turn mod AHEAD]
      else slice(turn * 16 + kq, qa[0]);
    }
  }
  // The sums over the sixteen lanes of a row group: at every step a lane keeps the half of its values that its lane number names
  // and gets the partner's share of them.  Lane kq ends with column kq & 7 of the rows r with r mod 2 = kq >> 3.
  float s[RPT][FC_NB];
#pragma unroll
  for (int r = 0; r < RPT; r++)
#pragma unroll
    for (int j = 0; j < FC_NB; j++) s[r][j] = acc[r][j].x + acc[r][j].y;
#pragma unroll
  for (int d = 1, n = FC_NB / 2; d < 8; d <<= 1, n >>= 1)
#pragma unroll
    for (int r = 0; r < RPT; r++)
#pragma unroll
      for (int j = 0; j < FC_NB / 2; j++)
        if (j < n) {
          const float even = s[r][2 * j], odd = s[r][2 * j + 1];
          s[r][j] = ((kq & d) ? odd : even) + __shfl_xor_sync(0xffffffffu, (kq & d) ? even : odd, d);
        }
  const int col = n0 + (kq & 7);
#pragma unroll
  for (int r = 0; r < RPT; r += 2) {
    const float v = ((kq & 8) ? s[r + 1][0] : s[r][0]) + __shfl_xor_sync(0xffffffffu, (kq & 8) ? s[r][0] : s[r + 1][0], 8);
    const int row = row0 + r + (kq >> 3);
    if (col < N && row < M) out[(size_t)row * ldo + col] = v + (bias ? bias[col] : 0.f);
  }
}

// ------------------------------------------------------------------ response writers
// Softmax over `n` fp32 logits per row written as fp32 into the response slot of
// each request (stub->resp + row * resp_stride), optionally followed by the
// argmax class as int32.  When `flag` is set, the block that finishes last
// publishes `flag_value` with a system-scope release store: the response is in
// place (possibly in a peer GPU's or the host's memory) before the flag is seen.
// With a response-push block (`push`, see resp_push.cuh) each row goes straight to
// the place the producer named for its slot (the ingress transmit arena, in another
// process's pinned memory or on a peer GPU) and the row's block completes the slot.
__global__ void __launch_bounds__(256) softmax_response(const float* logits, int n, int ld, const g_params* stub,
                                                        uint8_t* direct_out, size_t resp_stride, int write_argmax,
                                                        uint32_t* counter, volatile uint32_t* flag, uint32_t flag_value,
                                                        const RespPushCtx* push) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  __shared__ float sh_max[8], sh_sum[8];
  __shared__ int sh_arg[8];
  const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* x = logits + (size_t)row * ld;
  // One thread reads the stub and the push block (mapped host memory: every read is a PCIe round trip) for the block; the target is
  // needed behind the last barrier.  The logits stay in registers (a row of up to 2048), and every thread puts the warps'
  // shares together by itself: two barriers instead of eight and one read of the row instead of three (64 x 1000: 3.2 -> 1.85 us).
  __shared__ RespPushTarget s_target;
  if (threadIdx.x == 0) {
    uint8_t* b = (direct_out ? direct_out : stub->resp) + (size_t)row * resp_stride;
    s_target = (!direct_out && push) ? resp_push_target(push, (uint32_t)row, b) : RespPushTarget{b, nullptr, nullptr};
  }
  constexpr int REGS = 8;
  float v[REGS];
  float m = -FLT_MAX;
  int am = 0;
#pragma unroll
  for (int k = 0; k < REGS; k++) {
    const int i = threadIdx.x + k * 256;
    v[k] = i < n ? x[i] : -INFINITY;
  }
#pragma unroll
  for (int k = 0; k < REGS; k++)
    if (v[k] > m) {
      m = v[k];
      am = threadIdx.x + k * 256;
    }
  for (int i = threadIdx.x + REGS * 256; i < n; i += 256)
    if (x[i] > m) {
      m = x[i];
      am = i;
    }
  const float wm = warp_max(m);
  const int src = __ffs(__ballot_sync(0xffffffffu, m == wm)) - 1;
  const int wam = __shfl_sync(0xffffffffu, am, src);
  if (lane == 0) {
    sh_max[warp] = wm;
    sh_arg[warp] = wam;
  }
  __syncthreads();
  float mx = sh_max[0];
  int arg = sh_arg[0];
#pragma unroll
  for (int k = 1; k < 8; k++)
    if (sh_max[k] > mx) {
      mx = sh_max[k];
      arg = sh_arg[k];
    }
  float sum = 0.f;
#pragma unroll
  for (int k = 0; k < REGS; k++) {
    v[k] = __expf(v[k] - mx);
    if (threadIdx.x + k * 256 < n) sum += v[k];
  }
  for (int i = threadIdx.x + REGS * 256; i < n; i += 256) sum += __expf(x[i] - mx);
  sum = warp_sum(sum);
  if (lane == 0) sh_sum[warp] = sum;
  __syncthreads();
  sum = sh_sum[0];
#pragma unroll
  for (int k = 1; k < 8; k++) sum += sh_sum[k];
  const float inv = 1.f / sum;
  const RespPushTarget target = s_target;
  uint8_t* base = target.dst;
  float* o = reinterpret_cast<float*>(base);
#pragma unroll
  for (int k = 0; k < REGS; k++)
    if (threadIdx.x + k * 256 < n) o[threadIdx.x + k * 256] = v[k] * inv;
  for (int i = threadIdx.x + REGS * 256; i < n; i += 256) o[i] = __expf(x[i] - mx) * inv;
  if (write_argmax && threadIdx.x == 0) reinterpret_cast<int*>(base)[n] = arg;
  if (target.state) {
    __syncthreads();
    if (threadIdx.x == 0) resp_push_complete(target);
  }
  if (flag) {
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t prev = atomicAdd(counter, 1u);
      if (prev + 1 == gridDim.x) {
        atomicExch(counter, 0u);
        __threadfence_system();
        ptx::st_release_sys(flag, flag_value);
      }
    }
  }
}

// ------------------------------------------------------------------ LayerNorm (+ residual)
// y = LN(x + residual) * gamma + beta, one row per block; hidden <= 8 * blockDim.x.
__global__ void __launch_bounds__(256) layernorm_rows(const __nv_bfloat16* x,
                                                      const __nv_bfloat16* residual,
                                                      const float* gamma, const float* beta,
                                                      __nv_bfloat16* y, int hidden, float eps) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  __shared__ float sh[32];
  const size_t row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * hidden;
  const __nv_bfloat16* rr = residual ? residual + row * hidden : nullptr;
  float v[8];
  int cnt = 0;
  float s = 0.f;
  for (int i = threadIdx.x; i < hidden && cnt < 8; i += blockDim.x, cnt++) {
    float f = __bfloat162float(xr[i]);
    if (rr) f += __bfloat162float(rr[i]);
    v[cnt] = f;
    s += f;
  }
  const float mean = block_sum(s, sh) / hidden;
  float q = 0.f;
  for (int k = 0; k < cnt; k++) q += (v[k] - mean) * (v[k] - mean);
  const float var = block_sum(q, sh) / hidden;
  const float rstd = rsqrtf(var + eps);
  cnt = 0;
  for (int i = threadIdx.x; i < hidden && cnt < 8; i += blockDim.x, cnt++)
    y[row * hidden + i] = __float2bfloat16((v[cnt] - mean) * rstd * gamma[i] + beta[i]);
}

// LayerNorm for hidden sizes of 256, 512, 768 and 1024: a thread has eight columns of R rows, so that a row's 8 bytes of
// parameters per column are read once for R rows (a warp with a row of its own read twice as many bytes of parameters as of the
// row); rows never leave registers, both reductions halve their list of rows at every step through the warp and meet in
// shared memory.  Us with the product of hidden columns before it, a warp per row against this: 6144 x 1024 20.1 and 18.5, 4096 x 768
// 11.6 and 11.0, 2368 x 1024 13.1 and 11.3, 1184 x 768 8.65 and 7.7, 128 x 768 6.0 and 5.6, 6144 x 512 10.65 and 9.8, 4096 x 256 7.1 and 6.85.
// (Alone, one after the other, a warp per row wins where its blocks fill the SMs exactly: 1184 x 768 2.0 and 2.4, 1176 x 768 3.2 and 2.4.)
// v[r]: this thread's eight columns of rows row0 + r (values of rows behind the last one are not stored).  One warp per 256 columns,
// and for the narrow rows several groups of warps per block (row_groups), each with rows of its own: 12288 x 256 9.2 us with four
// groups, 12.3 with one, 6144 x 512 9.8 and 10.6.
constexpr int row_groups(int vpl) { return vpl == 1 ? 4 : vpl == 2 ? 2 : 1; }
template <int VPL>
__device__ __forceinline__ int row_group() {
  return row_groups(VPL) == 1 ? 0 : threadIdx.x / (32 * VPL);
}
template <int VPL, int R>
__device__ __forceinline__ void normalise_rows(float (&v)[R][8], float (&s)[R], const float* gamma, const float* beta, __nv_bfloat16* y,
                                               int row0, int rows, float eps) {
  static_assert(R == 2 || R == 4, "a power of two; the steps of the reduction below");
  constexpr int HIDDEN = VPL * 256;
  __shared__ __align__(16) float shared[2][row_groups(VPL)][VPL][R];
  const int group = row_group<VPL>(), warp = (threadIdx.x >> 5) - group * VPL, lane = threadIdx.x & 31, c0 = (warp * 32 + lane) * 8;
  float4 g4[2], b4[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    g4[i] = *reinterpret_cast<const float4*>(gamma + c0 + 4 * i);
    b4[i] = *reinterpret_cast<const float4*>(beta + c0 + 4 * i);
  }
  // Sums of s[r] over the block: lane l of a warp ends with row l mod R, the warps' shares meet in shared memory.
  auto block_sums = [&](float (&s)[R], int buf) {
#pragma unroll
    for (int d = 1, n = R / 2; d < 32; d <<= 1, n >>= 1) {
      if (n >= 1) {
#pragma unroll
        for (int r = 0; r < R / 2; r++)
          if (r < n) {
            const float even = s[2 * r], odd = s[2 * r + 1];
            s[r] = ((lane & d) ? odd : even) + __shfl_xor_sync(0xffffffffu, (lane & d) ? even : odd, d);
          }
      } else {
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], d);
      }
    }
    float(*sh)[R] = shared[buf][group];
    if (lane < R) sh[warp][lane] = s[0];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; r++) {
      s[r] = sh[0][r];
#pragma unroll
      for (int w = 1; w < VPL; w++) s[r] += sh[w][r];
    }
  };
  block_sums(s, 0);
  float u[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const float mean = s[r] * (1.f / HIDDEN);
    u[r] = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      v[r][k] -= mean;
      u[r] += v[r][k] * v[r][k];
    }
  }
  block_sums(u, 1);
  const float gg[8] = {g4[0].x, g4[0].y, g4[0].z, g4[0].w, g4[1].x, g4[1].y, g4[1].z, g4[1].w};
  const float bb[8] = {b4[0].x, b4[0].y, b4[0].z, b4[0].w, b4[1].x, b4[1].y, b4[1].z, b4[1].w};
#pragma unroll
  for (int r = 0; r < R; r++) {
    if (row0 + r >= rows) break;
    const float rstd = rsqrtf(u[r] * (1.f / HIDDEN) + eps);
    uint4 o;
    __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int t = 0; t < 4; t++)
      ho[t] = __floats2bfloat162_rn(v[r][2 * t] * rstd * gg[2 * t] + bb[2 * t], v[r][2 * t + 1] * rstd * gg[2 * t + 1] + bb[2 * t + 1]);
    *reinterpret_cast<uint4*>(y + (size_t)(row0 + r) * HIDDEN + c0) = o;
  }
}

template <int VPL, int R>  // hidden = VPL * 256
__global__ void __launch_bounds__(32 * VPL * row_groups(VPL)) layernorm_rows_vec(const __nv_bfloat16* x, const __nv_bfloat16* residual, const float* gamma,
                                                               const float* beta, __nv_bfloat16* y, int rows, float eps) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const int group = row_group<VPL>(), row0 = (blockIdx.x * row_groups(VPL) + group) * R, c0 = (threadIdx.x - group * 32 * VPL) * 8;
  uint4 q[R], q2[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const size_t at = (size_t)min(row0 + r, rows - 1) * (VPL * 256) + c0;
    q[r] = *reinterpret_cast<const uint4*>(x + at);
    q2[r] = residual ? *reinterpret_cast<const uint4*>(residual + at) : make_uint4(0u, 0u, 0u, 0u);
  }
  float v[R][8], s[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162*>(&q[r]), *h2 = reinterpret_cast<const __nv_bfloat162*>(&q2[r]);
    s[r] = 0.f;
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const float2 f = __bfloat1622float2(h[t]), g = __bfloat1622float2(h2[t]);
      v[r][2 * t] = f.x + g.x;
      v[r][2 * t + 1] = f.y + g.y;
      s[r] += v[r][2 * t] + v[r][2 * t + 1];
    }
  }
  normalise_rows<VPL, R>(v, s, gamma, beta, y, row0, rows, eps);
}

// ------------------------------------------------------------------ BERT embedding
// Request = seq int32 token ids per sequence.  y[token] = LN(word[id] + pos[t] + type[0]).
// Reads ids through the stub (ring window) or from `direct_ids`.
__global__ void __launch_bounds__(256) bert_embed_ln(const g_params* stub, const int* direct_ids, size_t req_stride,
                                                     int seq, const __nv_bfloat16* word,
                                                     const __nv_bfloat16* pos,
                                                     const __nv_bfloat16* type, const float* gamma,
                                                     const float* beta, __nv_bfloat16* y, int hidden,
                                                     int vocab, float eps) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  __shared__ float sh[32];
  const int tok = blockIdx.x, b = tok / seq, t = tok - b * seq;
  const int* ids = direct_ids ? direct_ids + (size_t)b * seq
                              : reinterpret_cast<const int*>(stub->req + (size_t)b * req_stride);
  int id = ids[t];
  id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
  float v[8];
  int cnt = 0;
  float s = 0.f;
  for (int i = threadIdx.x; i < hidden && cnt < 8; i += blockDim.x, cnt++) {
    float f = __bfloat162float(word[(size_t)id * hidden + i]) + __bfloat162float(pos[(size_t)t * hidden + i]) +
              __bfloat162float(type[i]);
    v[cnt] = f;
    s += f;
  }
  const float mean = block_sum(s, sh) / hidden;
  float q = 0.f;
  for (int k = 0; k < cnt; k++) q += (v[k] - mean) * (v[k] - mean);
  const float rstd = rsqrtf(block_sum(q, sh) / hidden + eps);
  cnt = 0;
  for (int i = threadIdx.x; i < hidden && cnt < 8; i += blockDim.x, cnt++)
    y[(size_t)tok * hidden + i] = __float2bfloat16((v[cnt] - mean) * rstd * gamma[i] + beta[i]);
}

// The same with eight columns of R tokens per thread (see layernorm_rows_vec).  Us, a block per token against this: 4096 tokens of
// 768 12.6 and 4.5, 6144 of 1024 20.8 and 6.5, 128 of 768 3.1 and 1.9, 4096 of 512 10.6 and 3.9, 4096 of 256 8.6 and 3.3, 128 of 256 2.1 and 1.8.
template <int VPL, int R>
__global__ void __launch_bounds__(32 * VPL * row_groups(VPL)) bert_embed_ln_vec(const g_params* stub, const int* direct_ids, size_t req_stride, int seq,
                                                              int tokens, const __nv_bfloat16* word, const __nv_bfloat16* pos,
                                                              const __nv_bfloat16* type, const float* gamma, const float* beta,
                                                              __nv_bfloat16* y, int vocab, float eps) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  constexpr int HIDDEN = VPL * 256;
  const int group = row_group<VPL>(), row0 = (blockIdx.x * row_groups(VPL) + group) * R, c0 = (threadIdx.x - group * 32 * VPL) * 8;
  uint4 q[R], q2[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int tok = min(row0 + r, tokens - 1), b = tok / seq, t = tok - b * seq;
    const int* ids = direct_ids ? direct_ids + (size_t)b * seq : reinterpret_cast<const int*>(stub->req + (size_t)b * req_stride);
    int id = ids[t];
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    q[r] = *reinterpret_cast<const uint4*>(word + (size_t)id * HIDDEN + c0);
    q2[r] = *reinterpret_cast<const uint4*>(pos + (size_t)t * HIDDEN + c0);
  }
  const uint4 q3 = *reinterpret_cast<const uint4*>(type + c0);
  const __nv_bfloat162* h3 = reinterpret_cast<const __nv_bfloat162*>(&q3);
  float v[R][8], s[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162*>(&q[r]), *h2 = reinterpret_cast<const __nv_bfloat162*>(&q2[r]);
    s[r] = 0.f;
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const float2 f = __bfloat1622float2(h[t]), g = __bfloat1622float2(h2[t]), k = __bfloat1622float2(h3[t]);
      v[r][2 * t] = f.x + g.x + k.x;
      v[r][2 * t + 1] = f.y + g.y + k.y;
      s[r] += v[r][2 * t] + v[r][2 * t + 1];
    }
  }
  normalise_rows<VPL, R>(v, s, gamma, beta, y, row0, tokens, eps);
}

// ------------------------------------------------------------------ attention (head dim 64)
// qkv: [tokens, 3*hidden] bf16 with q | k | v blocks; out: [tokens, hidden].
// One block = one (sequence, head, tile of 32 queries); K and V of the head sit in
// shared memory; one warp handles 4 queries at a time with fp32 accumulation.
// This is the simple SIMT form of the operator; it keeps every intermediate on chip.
template <int SEQ>
__global__ void __launch_bounds__(256) attention_d64(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* __restrict__ out,
                                                     int heads, int ld_qkv, int q_off, int k_off, int v_off, int ld_out,
                                                     float scale) {
  extern __shared__ __align__(16) uint8_t att_smem[];
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(att_smem);        // [SEQ][64+2] padded rows
  __nv_bfloat16* sV = sK + SEQ * 66;                                     // [SEQ][64]
  float* sP = reinterpret_cast<float*>(sV + SEQ * 64);                   // [8 warps][SEQ]
  const int qt = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t tok0 = (size_t)b * SEQ;
  for (int i = threadIdx.x; i < SEQ * 32; i += blockDim.x) {
    const int r = i >> 5, c = (i & 31) * 2;
    const __nv_bfloat16* row = qkv + (tok0 + r) * ld_qkv + h * 64 + c;
    *reinterpret_cast<__nv_bfloat162*>(sK + r * 66 + c) = *reinterpret_cast<const __nv_bfloat162*>(row + k_off);
    *reinterpret_cast<__nv_bfloat162*>(sV + r * 64 + c) = *reinterpret_cast<const __nv_bfloat162*>(row + v_off);
  }
  __syncthreads();
  float* p = sP + warp * SEQ;
  for (int qi = warp; qi < 32; qi += 8) {
    const int q = qt * 32 + qi;
    if (q >= SEQ) break;
    const __nv_bfloat16* qrow = qkv + (tok0 + q) * ld_qkv + q_off + h * 64;
    float2 qv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(qrow + lane * 2));
    // scores: each lane owns keys lane, lane+32, ...
    float mx = -FLT_MAX;
    for (int k0 = 0; k0 < SEQ; k0 += 32) {
      const int k = k0 + lane;
      float acc = 0.f;
#pragma unroll 8
      for (int d = 0; d < 64; d += 2) {
        float2 kv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sK + k * 66 + d));
        const float qx = __shfl_sync(0xffffffffu, qv.x, d >> 1), qy = __shfl_sync(0xffffffffu, qv.y, d >> 1);
        acc += qx * kv.x + qy * kv.y;
      }
      acc *= scale;
      p[k] = acc;
      mx = fmaxf(mx, acc);
    }
    mx = warp_max(mx);
    float sum = 0.f;
    for (int k = lane; k < SEQ; k += 32) {
      const float e = __expf(p[k] - mx);
      p[k] = e;
      sum += e;
    }
    sum = warp_sum(sum);
    __syncwarp();
    // out: each lane owns dims 2*lane, 2*lane+1
    float o0 = 0.f, o1 = 0.f;
    for (int k = 0; k < SEQ; k++) {
      const float pk = p[k];
      float2 vv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sV + k * 64 + lane * 2));
      o0 += pk * vv.x;
      o1 += pk * vv.y;
    }
    const float inv = 1.f / sum;
    *reinterpret_cast<__nv_bfloat162*>(out + (tok0 + q) * ld_out + h * 64 + lane * 2) = __floats2bfloat162_rn(o0 * inv, o1 * inv);
    __syncwarp();
  }
}

int grid_for(size_t total, int threads) {
  size_t b = (total + threads - 1) / threads;
  size_t cap = 148 * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

cudaError_t nn_stem_im2col(const void* d_stub, const float* direct_in, int batch, void* out, const float mean[3],
                           const float inv_std[3], cudaStream_t s) {
  size_t total = (size_t)batch * 112 * 112 * 24;
  return launch_pdl(stem_im2col, dim3(grid_for(total, 256)), dim3(256), 0, s, (const g_params*)d_stub, direct_in, batch,
                    (__nv_bfloat16*)out, make_float3(mean[0], mean[1], mean[2]), make_float3(inv_std[0], inv_std[1],
                    inv_std[2]));
}
cudaError_t nn_stem_s2d(const void* d_stub, const float* direct_in, int batch, void* out, const float mean[3],
                        const float inv_std[3], cudaStream_t s) {
  size_t total = (size_t)batch * 115 * 115 * 2;
  return launch_pdl(stem_s2d, dim3(grid_for(total, 256)), dim3(256), 0, s, (const g_params*)d_stub, direct_in, batch,
                    (__nv_bfloat16*)out, make_float3(mean[0], mean[1], mean[2]), make_float3(inv_std[0], inv_std[1],
                    inv_std[2]));
}
cudaError_t nn_maxpool3x3s2(const void* in, void* out, int n, int h, int w, int c, cudaStream_t s) {
  if (c % 8) return cudaErrorInvalidValue;
  int oh = (h - 1) / 2 + 1, ow = (w - 1) / 2 + 1;
  return launch_pdl(maxpool3x3s2, dim3(grid_for((size_t)n * oh * ow * (c / 8), 256)), dim3(256), 0, s, (const __nv_bfloat16*)in,
                    (__nv_bfloat16*)out, n, h, w, c);
}
cudaError_t nn_global_avgpool(const void* in, void* out, int n, int hw, int c, cudaStream_t s) {
  if (c % 2) return cudaErrorInvalidValue;
  return launch_pdl(global_avgpool, dim3((c + 511) / 512, n), dim3(256), 0, s, (const __nv_bfloat16*)in, (__nv_bfloat16*)out,
                    hw, c);
}
cudaError_t nn_fc_skinny(const void* a, int lda, const void* w, int ldw, const float* bias, float* out, int ldo, int M, int N, int K,
                         uint32_t* status, cudaStream_t s) {
  const size_t smem = (size_t)FC_NB * K * sizeof(__nv_bfloat16);
  if (K % 8 || lda % 8 || ldw % 8 || (((uintptr_t)a | (uintptr_t)w) & 15) || smem > 100 * 1024 || M <= 0) return cudaErrorInvalidValue;
  // Above 1536 the sums of 16 products that the tensor core makes are both faster and closer (us here / there: 32 x 1000 x 2048 9.0 / 4.3,
  // 64 x 1000 x 2048 11.8 / 5.0; errors in fc_cluster.cu).  Below, they were faster too (64 x 1192 x 512 7.5 / 3.8), but up to 2 % further from
  // the exact sums than the short chains of FMAs per lane (K = 512: 5.2e-8 / 5.3e-8) when the line was drawn, before rounding errors were
  // kept there.  Rows that overlap (broadcast ones, say) have no tensor map.
  if (K > 1536 && K <= 2048 && lda >= K && ldw >= K && M <= (1 << 20) && nn_fc_cluster_fits())
    return nn_fc_cluster(a, lda, w, ldw, bias, out, ldo, M, N, K, status, s);
  static PerDeviceFlag attr_set;
  const int dev = PerDeviceFlag::current();
  if (attr_set.needed(dev)) {
    cudaError_t e = cudaFuncSetAttribute(fc_skinny<2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 116 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fc_skinny<4, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 116 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fc_skinny<2, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 116 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fc_skinny<4, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 116 * 1024);
    if (e != cudaSuccess) return e;
    attr_set.set(dev);
  }
  // While the blocks fit the SMs one each, a block takes the registers it likes, and up to 32 rows also more than half of an
  // SM's shared memory: blocks that start while the kernel before still runs would otherwise be stacked two to an SM
  // beside empty ones (32 x 1000 x 2048: 13.6 us then, 8.9 us now).  With more blocks than SMs two share an SM, at 128
  // registers.  One per SM against two, us (weights staged whole): 32 x 1192 x 512 8.2 / 6.4, 32 x 4096 x 2048 32.9 / 28.4,
  // 64 x 1192 x 512 12.6 / 10.0, 128 x 1000 x 512 12.9 / 10.2, 64 x 8192 x 768 50.4 / 38.3.
  const size_t spread = 116 * 1024;
  const int sms = srpc_gemm_grid_sms(), rpt = M <= 32 ? 2 : 4;
  const dim3 grid((unsigned)((N + FC_NB - 1) / FC_NB), (unsigned)((M + 16 * rpt - 1) / (16 * rpt)));
  const bool one_each = (uint64_t)grid.x * grid.y <= (uint64_t)sms;
  auto go = [&](auto* kernel, size_t shared) {
    return launch_pdl(kernel, grid, dim3(256), shared, s, (const __nv_bfloat16*)a, lda, (const __nv_bfloat16*)w, ldw, bias, out, ldo, M, N, K);
  };
  if (rpt == 2) return one_each ? go(fc_skinny<2, 1>, spread) : go(fc_skinny<2, 2>, smem);
  return one_each ? go(fc_skinny<4, 1>, smem) : go(fc_skinny<4, 2>, smem);
}
cudaError_t nn_softmax_response(const float* logits, int rows, int n, int ld, const void* d_stub, void* direct_out,
                                size_t resp_stride, int write_argmax, uint32_t* counter, uint32_t* flag, uint32_t flag_value,
                                cudaStream_t s, const void* d_push) {
  if (rows <= 0) return cudaSuccess;
  return launch_pdl(softmax_response, dim3(rows), dim3(256), 0, s, logits, n, ld, (const g_params*)d_stub, (uint8_t*)direct_out,
                    resp_stride, write_argmax, counter, flag, flag_value, (const RespPushCtx*)d_push);
}
// Four rows per block instead of two once there is enough for every SM: about 4000 rows of 768, 3000 of 1024, 7500 of 512, never for 256 (us,
// two against four, with the product of hidden columns before it: 3072 x 768 9.3 / 9.9, 4096 x 768 11.06 / 11.01, 4736 x 768 12.44 / 12.34, 2368 x
// 1024 11.3 / 11.9, 4096 x 1024 14.3 / 13.8, 6144 x 512 9.8 / 10.4, 8192 x 512 11.7 / 11.5, 12288 x 256 9.2 / 9.6; embedding 2560 x 768 10.1 / 10.8,
// 5120 x 768 13.75 / 13.4, 6144 x 512 10.7 / 11.2).  Eight: 5.8 for 6144 x 1024 alone against 5.35, 121 registers.
static bool four_rows(int rows, int hidden) {
  return hidden > 256 && (size_t)rows * hidden >= (hidden == 512 ? 26000u : 20480u) * (size_t)srpc_gemm_grid_sms();
}
cudaError_t nn_layernorm(const void* x, const void* residual, const float* gamma, const float* beta, void* y, int rows,
                         int hidden, float eps, cudaStream_t s) {
  if (hidden > 2048) return cudaErrorInvalidValue;
  const bool aligned = (((uintptr_t)x | (uintptr_t)y | (uintptr_t)residual | (uintptr_t)gamma | (uintptr_t)beta) & 15) == 0;
  const __nv_bfloat16 *xp = (const __nv_bfloat16*)x, *rp = (const __nv_bfloat16*)residual;
  __nv_bfloat16* yp = (__nv_bfloat16*)y;
  if (aligned && rows > 0 && hidden % 256 == 0 && hidden <= 1024) {
    const bool many = four_rows(rows, hidden);
    auto go = [&](auto* kernel, int vpl, int r) {
      const int per_block = r * row_groups(vpl);
      return launch_pdl(kernel, dim3((rows + per_block - 1) / per_block), dim3(32 * vpl * row_groups(vpl)), 0, s, xp, rp, gamma, beta, yp, rows, eps);
    };
    if (hidden == 256) return go(layernorm_rows_vec<1, 2>, 1, 2);
    if (hidden == 512) return many ? go(layernorm_rows_vec<2, 4>, 2, 4) : go(layernorm_rows_vec<2, 2>, 2, 2);
    if (hidden == 768) return many ? go(layernorm_rows_vec<3, 4>, 3, 4) : go(layernorm_rows_vec<3, 2>, 3, 2);
    return many ? go(layernorm_rows_vec<4, 4>, 4, 4) : go(layernorm_rows_vec<4, 2>, 4, 2);
  }
  return launch_pdl(layernorm_rows, dim3(rows), dim3(256), 0, s, xp, rp, gamma, beta, yp, hidden, eps);
}
cudaError_t nn_bert_embed_ln(const void* d_stub, const int* direct_ids, size_t req_stride, int batch, int seq, const void* word,
                             const void* pos, const void* type, const float* gamma, const float* beta, void* y, int hidden,
                             int vocab, float eps, cudaStream_t s) {
  if (hidden > 2048) return cudaErrorInvalidValue;
  const int tokens = batch * seq;
  const uintptr_t all = (uintptr_t)word | (uintptr_t)pos | (uintptr_t)type | (uintptr_t)gamma | (uintptr_t)beta | (uintptr_t)y;
  if ((all & 15) == 0 && tokens > 0 && hidden % 256 == 0 && hidden <= 1024) {
    const bool many = four_rows(tokens, hidden);
    auto go = [&](auto* kernel, int vpl, int r) {
      const int per_block = r * row_groups(vpl);
      return launch_pdl(kernel, dim3((tokens + per_block - 1) / per_block), dim3(32 * vpl * row_groups(vpl)), 0, s, (const g_params*)d_stub,
                        direct_ids, req_stride, seq, tokens, (const __nv_bfloat16*)word, (const __nv_bfloat16*)pos,
                        (const __nv_bfloat16*)type, gamma, beta, (__nv_bfloat16*)y, vocab, eps);
    };
    if (hidden == 256) return go(bert_embed_ln_vec<1, 2>, 1, 2);
    if (hidden == 512) return many ? go(bert_embed_ln_vec<2, 4>, 2, 4) : go(bert_embed_ln_vec<2, 2>, 2, 2);
    if (hidden == 768) return many ? go(bert_embed_ln_vec<3, 4>, 3, 4) : go(bert_embed_ln_vec<3, 2>, 3, 2);
    return many ? go(bert_embed_ln_vec<4, 4>, 4, 4) : go(bert_embed_ln_vec<4, 2>, 4, 2);
  }
  return launch_pdl(bert_embed_ln, dim3(tokens), dim3(256), 0, s, (const g_params*)d_stub, direct_ids, req_stride, seq,
                    (const __nv_bfloat16*)word, (const __nv_bfloat16*)pos, (const __nv_bfloat16*)type, gamma, beta,
                    (__nv_bfloat16*)y, hidden, vocab, eps);
}
cudaError_t nn_attention_d64(const void* qkv, void* out, int batch, int seq, int heads, int ld_qkv, int q_off, int k_off,
                             int v_off, int ld_out, cudaStream_t s) {
  const float scale = 0.125f;
  dim3 grid((seq + 31) / 32, heads, batch);
  if (seq == 128) {
    const int smem = 128 * 66 * 2 + 128 * 64 * 2 + 8 * 128 * 4;
    attention_d64<128><<<grid, 256, smem, s>>>((const __nv_bfloat16*)qkv, (__nv_bfloat16*)out, heads, ld_qkv, q_off, k_off,
                                               v_off, ld_out, scale);
  } else if (seq == 384) {
    const int smem = 384 * 66 * 2 + 384 * 64 * 2 + 8 * 384 * 4;
    static PerDeviceFlag attr;
    const int dev = PerDeviceFlag::current();
    if (attr.needed(dev)) {
      cudaFuncSetAttribute(attention_d64<384>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      attr.set(dev);
    }
    attention_d64<384><<<grid, 256, smem, s>>>((const __nv_bfloat16*)qkv, (__nv_bfloat16*)out, heads, ld_qkv, q_off, k_off,
                                               v_off, ld_out, scale);
  } else {
    return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

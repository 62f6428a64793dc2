// Remaining device-side pieces of the original system, rebuilt for sm_100a:
//   swap_hdrs        reply-header construction on the GPU for headers that live in
//                    GPU-visible memory (reference src/transport/g_udp_handler.cu:96-178)
//   lenet_ref        the 20/50/10 LeNet of reference src/apps/lenet/lenet_vanilla.cu:17-192
//                    (uint8 pixels, (x-127)/128, conv 5x5 pad 1, tanh, 2x2 max pool, dense, softmax)
//                    as one kernel per batch instead of twelve launches per image
//   lstm_wavefront   the 8-layer x 8-step stacked LSTM (hidden 256) of reference
//                    src/apps/nnfusion_lstm/nnfusion_rt.cu:13870-13877,1213-1283 as one
//                    cluster launch per batch: the 8 blocks of a cluster own one layer
//                    each and advance along anti-diagonals with a cluster barrier per step
//                    (32 launches per inference in the original)
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <atomic>
#include <math.h>

#include "../host/p2p_rpc.h"
#include "../host/p2p_rpc_app.h"
#include "parity_kernels.h"
#include "per_device.h"
#include "ptx.cuh"

namespace cg = cooperative_groups;

namespace {

// ------------------------------------------------------------------ header swap
__global__ void swap_hdrs_kernel(p2p_rpc_hdr* const* hdrs, int n, int clear_sockperf) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  p2p_rpc_hdr* h = hdrs[i];
  swap_eth_hdr(h);
  if (clear_sockperf) set_sockperf_header(h);
  add_udp_cksum(h);
}

__global__ void swap_hdrs_contig_kernel(p2p_rpc_hdr* hdrs, int n, int clear_sockperf) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  p2p_rpc_hdr* h = hdrs + i;
  swap_eth_hdr(h);
  if (clear_sockperf) set_sockperf_header(h);
  add_udp_cksum(h);
}

// Resident header processor (launch type 2 of the GPU header-processing API): one block stays on the GPU and serves
// bursts of header pointers that the host posts in a mapped control block.  The doorbell is a sequence number, every
// poll also looks at the exit flag and the idle limit, and a burst is acknowledged by publishing its number in `done`.
__global__ void __launch_bounds__(1024) persistent_swap_hdrs(pp_params* stub, volatile uint32_t* door_bell, volatile uint32_t* done,
                                                             volatile uint32_t* exit_flag, volatile uint32_t* exited,
                                                             uint64_t idle_ns) {
  __shared__ uint32_t s_cmd, s_seq, s_n;
  uint32_t seen = *done;
  uint64_t last = ptx::globaltimer_ns();
  for (;;) {
    if (threadIdx.x == 0) {
      uint32_t cmd = 0;
      for (int spin = 0; spin < 4096; spin++) {
        if (ptx::ld_relaxed_sys(exit_flag) || ptx::globaltimer_ns() - last > idle_ns) {
          cmd = 2;
          break;
        }
        const uint32_t db = ptx::ld_acquire_sys(door_bell);
        if ((int32_t)(db - seen) > 0) {
          s_seq = db;
          s_n = ptx::ld_relaxed_sys(reinterpret_cast<const volatile uint32_t*>(&stub->num_items));
          cmd = 1;
          break;
        }
        __nanosleep(200);
      }
      s_cmd = cmd;
    }
    __syncthreads();
    const uint32_t cmd = s_cmd, seq = s_seq;
    uint32_t n = s_n;
    __syncthreads();
    if (cmd == 2) break;
    if (cmd == 0) continue;
    seen = seq;
    if (n > MAX_BI_SIZE) n = MAX_BI_SIZE;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      p2p_rpc_hdr* h = reinterpret_cast<p2p_rpc_hdr*>(ptx::ld_relaxed_sys_u64(reinterpret_cast<const uint64_t*>(&stub->hdr_ptrs[i])));
      swap_eth_hdr(h);
      if (stub->clear_sockperf) set_sockperf_header(h);
      add_udp_cksum(h);
    }
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
      ptx::st_release_sys(done, seen);
      last = ptx::globaltimer_ns();
    }
  }
  if (threadIdx.x == 0) ptx::st_release_sys(exited, 1u);
}

__global__ void swap_hdrs_stub_kernel(const pp_params* stub) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= stub->num_items) return;
  p2p_rpc_hdr* h = reinterpret_cast<p2p_rpc_hdr*>(stub->hdr_ptrs[i]);
  swap_eth_hdr(h);
  if (stub->clear_sockperf) set_sockperf_header(h);
  add_udp_cksum(h);
}

// ------------------------------------------------------------------ reference-format LeNet
struct LenetRefW {
  const float *c1, *c2, *fc, *fb;
};

// A cluster of eight blocks per image.
//   conv1   every block computes an eighth of the 20 x 13 x 13 pooled outputs (one thread each: the four window
//           positions from a 6 x 6 patch of the zero-bordered image, the 25 weights in registers) and stores them into
//           all eight blocks' copies through distributed shared memory;
//   conv2   2.5 of the 2.9 million multiply-adds of an inference.  Every block takes 6 or 7 of the 50 filters, weights
//           staged in shared memory once per block.  A warp is one pooled pixel; its lanes are (filter, quarter of the
//           input channels), so that the 6 x 6 input patch is a broadcast read and the weights fall into 28 different
//           banks; the quarters meet in shared-memory atomics.  0.6 shared-memory reads per multiply-add;
//   fc      every block multiplies its own 150 or 175 pooled values into the ten logits and adds them to block 0's,
//           block 0 writes the softmax.
// tanh is monotonic, so it is taken once, after the max over the window.  (One block per image with a thread per pooled
// output and weights read from global memory took 420 us per image, a cluster of four with redundant conv1 52 us.)
constexpr int LENET_REF_THREADS = 1024;
constexpr int LENET_REF_CLUSTER = 8;
constexpr int LENET_REF_KMAX = 7;      // filters of the second convolution per block (7, 7, 6, 6, 6, 6, 6, 6)
constexpr int LENET_P1_CH = 15 * 15;   // one zero-bordered 13 x 13 map

__device__ __forceinline__ float tanh_fast(float v) { return 1.f - __fdividef(2.f, 1.f + __expf(2.f * v)); }

__global__ void __cluster_dims__(LENET_REF_CLUSTER, 1, 1) __launch_bounds__(LENET_REF_THREADS, 1)
lenet_ref_kernel(const g_params* stub, const uint8_t* direct_in, float* direct_out, LenetRefW w, int batch) {
  cg::cluster_group cluster = cg::this_cluster();
  const int q = (int)cluster.block_rank();
  const int k_lo = q * 6 + (q < 2 ? q : 2), k_n = q < 2 ? 7 : 6;
  __shared__ __align__(16) float wc2[LENET_REF_KMAX * 500];  // [k_n][20][5][5]
  __shared__ float c2o[LENET_REF_KMAX * 100];                // [pixel][filter][2][2]: conv2 sums before max and tanh
  __shared__ float xp[30 * 32];                              // image with a zero border, rows 32 apart
  __shared__ float p1[20 * LENET_P1_CH];                     // conv1 output with a zero border
  __shared__ float p2[LENET_REF_KMAX * 25];
  __shared__ float lg[10];  // block 0: the logits
  __shared__ float wc1[500];
  const int t = threadIdx.x, warp = t / 32, lane = t % 32;
  for (int i = t; i < 500; i += LENET_REF_THREADS) wc1[i] = w.c1[i];
  for (int i = t; i < k_n * 125; i += LENET_REF_THREADS)
    reinterpret_cast<float4*>(wc2)[i] = __ldg(reinterpret_cast<const float4*>(w.c2 + (size_t)k_lo * 500) + i);
  for (int i = t; i < 30 * 32; i += LENET_REF_THREADS) xp[i] = 0.f;
  for (int i = t; i < 20 * LENET_P1_CH; i += LENET_REF_THREADS) p1[i] = 0.f;
  const uint8_t* in_base = direct_in ? direct_in : stub->req;
  float* out_base = direct_out ? direct_out : reinterpret_cast<float*>(stub->resp);
  float* lg_block0 = cluster.map_shared_rank(lg, 0);
  const int n_clusters = gridDim.x / LENET_REF_CLUSTER;
  cluster.sync();  // nobody stores into a block's p1 before that block has zeroed it
  for (int b = blockIdx.x / LENET_REF_CLUSTER; b < batch; b += n_clusters) {
    const uint8_t* in = in_base + (size_t)b * 784;
    float* out = out_base + (size_t)b * 10;
    if (t < 784) xp[(t / 28 + 1) * 32 + t % 28 + 1] = ((float)in[t] - 127.f) / 128.f;
    if (t < LENET_REF_KMAX * 100) c2o[t] = 0.f;
    if (q == 0 && t < 10) lg[t] = w.fb[t];
    __syncthreads();
    // conv1 (1->20, 5x5, pad 1: 28->26) + 2x2 max pool (->13) + tanh: this block's eighth, stored into every block
    {
      const int o = q * 423 + t;
      if (t < 423 && o < 20 * 169) {
        const int k = o / 169, r = (o % 169) / 13, c = o % 13;
        float wk[25];
#pragma unroll
        for (int i = 0; i < 25; i++) wk[i] = wc1[k * 25 + i];
        const float* xs = xp + (2 * r) * 32 + 2 * c;
        float a00 = 0.f, a01 = 0.f, a10 = 0.f, a11 = 0.f;
#pragma unroll
        for (int i = 0; i < 6; i++)
#pragma unroll
          for (int j = 0; j < 6; j++) {
            const float v = xs[i * 32 + j];
            if (i < 5 && j < 5) a00 += v * wk[i * 5 + j];
            if (i < 5 && j > 0) a01 += v * wk[i * 5 + j - 1];
            if (i > 0 && j < 5) a10 += v * wk[(i - 1) * 5 + j];
            if (i > 0 && j > 0) a11 += v * wk[(i - 1) * 5 + j - 1];
          }
        const float v = tanh_fast(fmaxf(fmaxf(a00, a01), fmaxf(a10, a11)));
        const int at = k * LENET_P1_CH + (r + 1) * 15 + c + 1;
#pragma unroll
        for (int d = 0; d < LENET_REF_CLUSTER; d++) cluster.map_shared_rank(p1, d)[at] = v;
      }
    }
    cluster.sync();  // every block holds the whole conv1 output
    // conv2 (20->50, 5x5, pad 1: 13->11) at the 10 x 10 positions that the pooling uses
    if (warp < 25) {
      const int pix = warp, quarter = lane & 3, kk = lane >> 2, r = pix / 5, c = pix % 5;
      if (kk < k_n) {
        float a00 = 0.f, a01 = 0.f, a10 = 0.f, a11 = 0.f;
        for (int ch = quarter * 5; ch < quarter * 5 + 5; ch++) {
          const float* ps = p1 + ch * LENET_P1_CH + (2 * r) * 15 + 2 * c;
          const float* wk = wc2 + (kk * 20 + ch) * 25;
#pragma unroll
          for (int i = 0; i < 6; i++)
#pragma unroll
            for (int j = 0; j < 6; j++) {
              const float v = ps[i * 15 + j];
              if (i < 5 && j < 5) a00 += v * wk[i * 5 + j];
              if (i < 5 && j > 0) a01 += v * wk[i * 5 + j - 1];
              if (i > 0 && j < 5) a10 += v * wk[(i - 1) * 5 + j];
              if (i > 0 && j > 0) a11 += v * wk[(i - 1) * 5 + j - 1];
            }
        }
        float* dst = c2o + (pix * LENET_REF_KMAX + kk) * 4;
        atomicAdd(dst, a00);
        atomicAdd(dst + 1, a01);
        atomicAdd(dst + 2, a10);
        atomicAdd(dst + 3, a11);
      }
    }
    __syncthreads();
    // 2x2 max pool + tanh, in the classifier's order [filter][pixel]
    if (t < k_n * 25) {
      const int kk = t / 25, pix = t % 25;
      const float* qv = c2o + (pix * LENET_REF_KMAX + kk) * 4;
      p2[t] = tanh_fast(fmaxf(fmaxf(qv[0], qv[1]), fmaxf(qv[2], qv[3])));
    }
    __syncthreads();
    // this block's share of the ten logits: one warp per output
    if (warp < 10) {
      float acc = 0.f;
      const float* fw = w.fc + warp * 1250 + k_lo * 25;
      for (int i = lane; i < k_n * 25; i += 32) acc += p2[i] * __ldg(fw + i);
      for (int sh = 16; sh; sh >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, sh);
      if (lane == 0) atomicAdd(lg_block0 + warp, acc);
    }
    cluster.sync();  // all shares are in; p1, c2o and p2 are free for the next image
    if (q == 0 && t == 0) {
      float m = lg[0];
      for (int i = 1; i < 10; i++) m = fmaxf(m, lg[i]);
      float e[10], sum = 0.f;
      for (int i = 0; i < 10; i++) {
        e[i] = expf(lg[i] - m);
        sum += e[i];
      }
      for (int i = 0; i < 10; i++) out[i] = e[i] / sum;
    }
    __syncthreads();  // block 0: the logits are read before the next image's bias goes in
  }
  cluster.sync();  // no block leaves while another may still store into its shared memory
}

// ------------------------------------------------------------------ LSTM wavefront
constexpr int LH = 256, LLAYERS = 8, LSTEPS = 8;

__device__ __forceinline__ float sigmoidf_(float v) { return 1.f / (1.f + __expf(-v)); }

// One cluster (8 blocks) per request; block l owns layer l.  At wave w block l computes cell (l, t = w - l):
//   gates = W_l . in + U_l . h_prev + b_l   (in = request step t for layer 0, else h of layer l-1 at step t)
// Layer outputs cross blocks through a small global scratch [request][layer][step][256]; the cluster barrier
// between waves orders the writes of wave w before the reads of wave w+1.
__global__ void __cluster_dims__(LLAYERS, 1, 1) __launch_bounds__(1024)
lstm_wavefront_kernel(const g_params* stub, const float* direct_in, float* direct_out, const float* __restrict__ weights,
                      float* __restrict__ scratch, int batch, float forget_bias) {
  cg::cluster_group cluster = cg::this_cluster();
  const int l = (int)cluster.block_rank();
  __shared__ float s_in[LH], s_h[LH], s_c[LH], s_g[4 * LH];
  const int t = threadIdx.x;
  const size_t per_layer = (size_t)8 * LH * LH + 4 * LH;
  const float* W = weights + (size_t)l * per_layer;
  const float* U = W + (size_t)4 * LH * LH;
  const float* B = U + (size_t)4 * LH * LH;
  const int n_clusters = gridDim.x / LLAYERS;
  const float* in_base = direct_in ? direct_in : reinterpret_cast<const float*>(stub->req);
  float* out_base = direct_out ? direct_out : reinterpret_cast<float*>(stub->resp);
  for (int req = blockIdx.x / LLAYERS; req < batch; req += n_clusters) {
    const float* x = in_base + (size_t)req * LSTEPS * LH;
    float* y = out_base + (size_t)req * LH;
    float* sc = scratch + (size_t)(blockIdx.x / LLAYERS) * LLAYERS * LSTEPS * LH;
    if (t < LH) {
      s_h[t] = 0.f;
      s_c[t] = 0.f;
    }
    __syncthreads();
    for (int w = 0; w < LLAYERS + LSTEPS - 1; w++) {
      const int step = w - l;
      if (step >= 0 && step < LSTEPS) {
        if (t < LH) s_in[t] = (l == 0) ? x[step * LH + t] : sc[((l - 1) * LSTEPS + step) * LH + t];
        __syncthreads();
        // 1024 threads = 4 gates x 256 outputs; each thread one dot product of length 512
        {
          const int g = t >> 8, o = t & 255;
          const float4* wr = reinterpret_cast<const float4*>(W + ((size_t)g * LH + o) * LH);
          const float4* ur = reinterpret_cast<const float4*>(U + ((size_t)g * LH + o) * LH);
          float acc = B[g * LH + o];
#pragma unroll 4
          for (int k = 0; k < LH / 4; k++) {
            const float4 a = __ldg(wr + k), b = __ldg(ur + k);
            acc += a.x * s_in[4 * k] + a.y * s_in[4 * k + 1] + a.z * s_in[4 * k + 2] + a.w * s_in[4 * k + 3];
            acc += b.x * s_h[4 * k] + b.y * s_h[4 * k + 1] + b.z * s_h[4 * k + 2] + b.w * s_h[4 * k + 3];
          }
          s_g[t] = acc;
        }
        __syncthreads();
        if (t < LH) {
          const float ig = s_g[t], gg = s_g[LH + t], fg = s_g[2 * LH + t], og = s_g[3 * LH + t];
          const float c = sigmoidf_(fg + forget_bias) * s_c[t] + sigmoidf_(ig) * tanhf(gg);
          const float h = tanhf(c) * sigmoidf_(og);
          s_c[t] = c;
          s_h[t] = h;
          sc[(l * LSTEPS + step) * LH + t] = h;
          if (l == LLAYERS - 1 && step == LSTEPS - 1) y[t] = h;
        }
        __syncthreads();
      }
      cluster.sync();
    }
  }
}

// ------------------------------------------------------------------ LSTM, whole-GPU dataflow
// The cluster kernel above gives a layer one SM, whose threads each walk one 1 KB weight row: a wave takes 74 us.  Here a
// layer has LSTM_LAYER_BLOCKS SMs and a warp owns two hidden units for the whole kernel: their eight gate rows of W and U each
// (16 KB) are loaded once and stay in its registers, so the weights cross the memory system once per launch instead of once per
// step.  What is left is the chain of 15 exchanges along the anti-diagonals (layer l, step t needs all 256 outputs of
// (l-1, t) and of (l, t-1)).  Outputs travel as 8-byte {value, tag} words through L2, stored and read whole: a reader that
// finds the launch's tag has the value with it, so an exchange is one store and one read, with no counter, no fence
// and no grid-wide barrier, and layers run apart as far as their inputs allow.  The tag is a launch counter in device memory
// (lstm_bump_kernel adds one before every launch; graph replays count too), so nothing has to be cleared in between.
// A block stages the vectors of a step in shared memory for its warps; the 8 x NB gate sums of a warp are reduced together
// (values are halved between lane pairs as they are added).  Two units per warp read every vector from shared memory half as often
// as one (16 warps): 29.8 / 34.3 / 46.4 / 77.0 us for 1 / 2 / 4 / 8 requests then, 28.0 / 33.9 / 41.2 / 69.1 now; the sums are the same bits.  The kernel is launched cooperatively: all blocks are resident,
// and every wait is bounded.  61.8 / 84.0 / 128.9 / 216.7 us with a grid barrier per wave.  What is left
// is the exchange latency, 1.9 us per step for one request, and 0.3 - 0.4 us per further request.
constexpr int LSTM_GROUP = 8;          // requests per launch
constexpr int LSTM_LAYER_BLOCKS = 16;  // 8 x 16 = 128 of 148 SMs
constexpr int LSTM_UNITS = LH / LSTM_LAYER_BLOCKS;  // hidden units per block
static_assert(LH % LSTM_LAYER_BLOCKS == 0, "every warp has its units");
// A cooperative launch waits until all its blocks fit, and the blocks of resident copy engines (16 each) do not leave between
// requests: a block that took all of its SM left two engines' LSTM 116 SMs.  256 threads x 216 registers leave room for one
// engine block on every SM (256 threads, held to 32 registers by its launch bounds, sg_kernels.cu); the 20 SMs that no block
// needs may hold any number.  128 of the registers hold weights; two requests' sums at a time keep a warp within the rest.
constexpr int LSTM_PER_WARP = 2;       // hidden units per warp
constexpr int LSTM_WARPS = LSTM_UNITS / LSTM_PER_WARP, LSTM_THREADS = LSTM_WARPS * 32, LSTM_REGS = 216;
static_assert(LSTM_THREADS * LSTM_REGS + 256 * 32 <= 65536, "a block and a resident copy block share an SM's registers");

struct LstmGridArgs {
  const g_params* stub;
  const float* direct_in;
  float* direct_out;
  const float* weights;
  unsigned long long* hbuf;  // [LLAYERS][LSTEPS][LSTM_GROUP][LH] words {value, tag}
  const unsigned* epoch;     // this launch's tag
  volatile uint32_t* status; // may be null
  long long wait_cycles;     // limit of one wait
  int first;                 // request of the window that this launch starts with
  int batch;                 // requests of this launch, 1 .. NB
  float forget_bias;
};

__device__ __forceinline__ float dot4(const float4& a, const float4& b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }

__device__ __forceinline__ void ld_two_words(const unsigned long long* p, unsigned long long* w0, unsigned long long* w1) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(*w0), "=l"(*w1) : "l"(p) : "memory");
}

// One step of a sum over the warp: of 2 x half values a lane keeps half, those of its side of `off`, and adds its partner's
// share of them; with one value left both add the whole.
template <int N>
__device__ __forceinline__ void keep_half(float (&v)[N], int half, int off) {
  const bool upper = (threadIdx.x & off) != 0;
  if (half == 0) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
#pragma unroll
  for (int k = 0; k < N / 2; k++) {
    if (k >= half) break;
    const float mine = upper ? v[k + half] : v[k], give = upper ? v[k] : v[k + half];
    v[k] = mine + __shfl_xor_sync(0xffffffffu, give, off);
  }
}

__global__ void lstm_bump_kernel(unsigned* epoch) { *epoch += 1; }

template <int NB>
__global__ void __maxnreg__(LSTM_REGS) lstm_grid_kernel(const LstmGridArgs a) {
  constexpr int PW = LSTM_PER_WARP;
  constexpr int P = NB == 1 ? 1 : 2, PASSES = NB / P;            // requests whose sums a warp forms together
  constexpr int PV = 4 * P * PW, REP = 32 / PV;                  // their gate sums, lanes per sum after the reduction
  constexpr int SUMS = PASSES > REP ? PASSES / REP : 1, LPP = PASSES > REP ? 1 : REP / PASSES;  // sums per lane at the end, lanes per sum
  constexpr int ROWS = LSTM_THREADS / (LH / 2);                  // vectors that the block stages at once
  constexpr int MAXQ = (2 * NB + ROWS - 1) / ROWS;               // word pairs a thread stages per step
  static_assert(LSTM_THREADS % (LH / 2) == 0 && (NB % ROWS == 0 || MAXQ == 1), "constant distance between a thread's vectors");
  __shared__ __align__(16) float s_vec[2][2][NB][LH];            // [buffer][input, own layer's previous output][request][unit]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int l = blockIdx.x / LSTM_LAYER_BLOCKS, part = blockIdx.x - l * LSTM_LAYER_BLOCKS;
  const int j0 = part * LSTM_UNITS + warp * PW;                     // this warp's first hidden unit
  const unsigned tag = *a.epoch;
  const float* in_base = (a.direct_in ? a.direct_in : reinterpret_cast<const float*>(a.stub->req)) + (size_t)a.first * LSTEPS * LH;
  float* out_base = (a.direct_out ? a.direct_out : reinterpret_cast<float*>(a.stub->resp)) + (size_t)a.first * LH;
  const float* W = a.weights + (size_t)l * ((size_t)8 * LH * LH + 4 * LH);
  const float* U = W + (size_t)4 * LH * LH;
  const float* B = U + (size_t)4 * LH * LH;
  float4 w[PW][4][2], u[PW][4][2];
#pragma unroll
  for (int n = 0; n < PW; n++)
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const float4* wr = reinterpret_cast<const float4*>(W + ((size_t)g * LH + j0 + n) * LH);
      const float4* ur = reinterpret_cast<const float4*>(U + ((size_t)g * LH + j0 + n) * LH);
      w[n][g][0] = __ldg(wr + lane);
      w[n][g][1] = __ldg(wr + 32 + lane);
      u[n][g][0] = __ldg(ur + lane);
      u[n][g][1] = __ldg(ur + 32 + lane);
    }
  // After the reductions a lane has gate `gate` of unit `j` for SUMS requests; with the other gates it computes their cells.
  const int lane_of_sum = lane & (REP - 1), gate = (lane / REP) & 3, src_lane = lane - gate * REP;
  const int item = lane / (4 * REP), req0 = lane_of_sum / LPP * SUMS * P + item % P, j = j0 + item / P;  // sum k: request req0 + k * P
  const bool stores = gate == 0 && lane_of_sum % LPP == 0;
  const float bias = B[gate * LH + j] + (gate == 2 ? a.forget_bias : 0.f);
  // Staging: a thread takes two units of every ROWS-th of the step's 2 x NB vectors.  Both sources lie on one line through
  // hbuf, so each further vector of a thread is the first one's address plus a constant.
  const int row0 = (int)threadIdx.x / (LH / 2), pr2 = 2 * ((int)threadIdx.x % (LH / 2));
  const int from0 = row0 / NB, b0 = row0 % NB;
  const int words0 = (((l - 1 + from0) * LSTEPS - from0) * LSTM_GROUP + b0) * LH + pr2;  // at step 0; + LSTM_GROUP * LH per step
  float cell[SUMS];
#pragma unroll
  for (int k = 0; k < SUMS; k++) cell[k] = 0.f;
  for (int t = 0; t < LSTEPS; t++) {
    float(*vec)[NB][LH] = s_vec[t & 1];
    // ---- stage the step's vectors (source 0: the layer below or the request, 1: this layer's previous output)
    bool open[MAXQ], any = false;
#pragma unroll
    for (int k = 0; k < MAXQ; k++) {
      const int from = from0 + k * ROWS / NB, b = b0 + k * ROWS % NB;
      open[k] = from <= (t > 0 ? 1 : 0) && b < a.batch;
      if (open[k] && from == 0 && l == 0) {
        *reinterpret_cast<float2*>(&vec[0][b][pr2]) = *reinterpret_cast<const float2*>(in_base + ((size_t)b * LSTEPS + t) * LH + pr2);
        open[k] = false;
      }
      any |= open[k];
    }
    const unsigned long long* words = a.hbuf + (words0 + t * LSTM_GROUP * LH);
    bool late = false;
    const long long t0 = clock64();
    while (any) {
      unsigned long long w0[MAXQ], w1[MAXQ];
#pragma unroll
      for (int k = 0; k < MAXQ; k++)
        if (open[k])
          ld_two_words(words + (k * ROWS / NB) * ((LSTEPS - 1) * LSTM_GROUP * LH) + (k * ROWS % NB) * LH, &w0[k], &w1[k]);
      any = false;
#pragma unroll
      for (int k = 0; k < MAXQ; k++) {
        if (!open[k]) continue;
        if ((unsigned)(w0[k] >> 32) == tag && (unsigned)(w1[k] >> 32) == tag) {
          *reinterpret_cast<float2*>(&vec[from0 + k * ROWS / NB][b0 + k * ROWS % NB][pr2]) =
              make_float2(__uint_as_float((unsigned)w0[k]), __uint_as_float((unsigned)w1[k]));
          open[k] = false;
        } else {
          any = true;
        }
      }
      if (any && clock64() - t0 > a.wait_cycles) {
        late = true;
        break;
      }
    }
    if (__syncthreads_or(late ? 1 : 0)) {
      // Every block that waits for this one's words gives up in turn; the last layer's blocks leave no number of an earlier
      // batch behind in the rows that they do not compute.
      if (l == LLAYERS - 1)
        for (int i = (int)threadIdx.x; i < a.batch * LSTM_UNITS; i += LSTM_THREADS)
          out_base[(size_t)(i / LSTM_UNITS) * LH + part * LSTM_UNITS + i % LSTM_UNITS] = __int_as_float(0x7fffffff);
      if (threadIdx.x == 0 && a.status) *a.status = 0x4C53u;  // 'LS': a wait of the LSTM ran out
      return;
    }
    // The buffers alternate: a warp overwrites a vector only after the barrier above of the next step, which every warp
    // reaches when it has read this step's vectors.
    // Sums over the warp: while a lane holds several values it keeps one half of them and adds its partner's share of that
    // half, first among the PV sums of P requests, then among the passes; what is left of the 32 lanes are replicas.
    float sum[PASSES];
#pragma unroll
    for (int p = 0; p < PASSES; p++) {
      float v[PV];
#pragma unroll
      for (int b = 0; b < P; b++) {
        if (p * P + b > NB / 2 && p * P + b >= a.batch) {  // (a launch has more than NB / 2 requests)
#pragma unroll
          for (int n = 0; n < PW; n++)
#pragma unroll
            for (int g = 0; g < 4; g++) v[(n * P + b) * 4 + g] = 0.f;
          continue;
        }
        const float4* xv = reinterpret_cast<const float4*>(vec[0][p * P + b]);
        const float4 x0 = xv[lane], x1 = xv[32 + lane];
#pragma unroll
        for (int n = 0; n < PW; n++)
#pragma unroll
          for (int g = 0; g < 4; g++) v[(n * P + b) * 4 + g] = dot4(w[n][g][0], x0) + dot4(w[n][g][1], x1);
        if (t > 0) {
          const float4* hv = reinterpret_cast<const float4*>(vec[1][p * P + b]);
          const float4 h0 = hv[lane], h1 = hv[32 + lane];
#pragma unroll
          for (int n = 0; n < PW; n++)
#pragma unroll
            for (int g = 0; g < 4; g++) v[(n * P + b) * 4 + g] += dot4(u[n][g][0], h0) + dot4(u[n][g][1], h1);
        }
      }
#pragma unroll
      for (int half = PV / 2, off = 16; half > 0; half /= 2, off /= 2) keep_half(v, half, off);
      sum[p] = v[0];
    }
#pragma unroll
    for (int half = PASSES / 2, off = REP / 2; off > 0; half /= 2, off /= 2) keep_half(sum, half, off);
#pragma unroll
    for (int k = 0; k < SUMS; k++) {
      sum[k] += bias;
      const float gi = __shfl_sync(0xffffffffu, sum[k], src_lane);
      const float gg = __shfl_sync(0xffffffffu, sum[k], src_lane + REP);
      const float gf = __shfl_sync(0xffffffffu, sum[k], src_lane + 2 * REP);
      const float go = __shfl_sync(0xffffffffu, sum[k], src_lane + 3 * REP);
      cell[k] = sigmoidf_(gf) * cell[k] + sigmoidf_(gi) * tanhf(gg);
      const float h = tanhf(cell[k]) * sigmoidf_(go);
      const int req = req0 + k * P;
      if (stores && req < a.batch) {
        unsigned long long* dst = a.hbuf + (((size_t)l * LSTEPS + t) * LSTM_GROUP + req) * LH + j;
        const unsigned long long word = ((unsigned long long)tag << 32) | __float_as_uint(h);
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(dst), "l"(word) : "memory");
        if (l == LLAYERS - 1 && t == LSTEPS - 1) out_base[(size_t)req * LH + j] = h;
      }
    }
  }
}

}  // namespace

cudaError_t srpc_swap_hdrs(void* const* d_hdr_ptrs, void* d_hdrs_contig, int n, int clear_sockperf, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (d_hdr_ptrs) swap_hdrs_kernel<<<(n + 255) / 256, 256, 0, s>>>((p2p_rpc_hdr* const*)d_hdr_ptrs, n, clear_sockperf);
  else swap_hdrs_contig_kernel<<<(n + 255) / 256, 256, 0, s>>>((p2p_rpc_hdr*)d_hdrs_contig, n, clear_sockperf);
  return cudaGetLastError();
}

cudaError_t srpc_lenet_ref(const void* d_stub, const void* direct_in, float* direct_out, const float* c1, const float* c2,
                           const float* fc, const float* fb, int batch, cudaStream_t s) {
  LenetRefW w{c1, c2, fc, fb};
  if (batch <= 0) return cudaSuccess;
  const int clusters = batch < 16 ? batch : 16;  // 16 clusters of eight blocks of 1024 threads fill the 148 SMs
  lenet_ref_kernel<<<LENET_REF_CLUSTER * clusters, LENET_REF_THREADS, 0, s>>>((const g_params*)d_stub, (const uint8_t*)direct_in, direct_out, w, batch);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ GPU header-processing API
struct pp_handler_ctx {
  pp_params* h_stub = nullptr;  // mapped pinned: the burst the host posts
  pp_params* d_stub = nullptr;
  volatile uint32_t* h_words = nullptr;  // [0] doorbell, [1] done, [2] exit flag, [3] exited
  uint32_t* d_words = nullptr;
  cudaStream_t g_stream = nullptr;
  uint8_t launch_type = 0;  // 0 none, 1 one kernel launch per burst, 2 resident kernel
  int device = 0;
  uint32_t seq = 0;
  bool resident = false;
  uint64_t idle_ns = 200000000ull, wait_ns = 2000000000ull;
  uint64_t bursts = 0, rearmed = 0, timeouts = 0;
};

static bool g_pp_stop_resident(pp_handler_ctx* c) {
  if (!c->resident) return true;
  __atomic_store_n(&c->h_words[2], 1u, __ATOMIC_RELEASE);
  const uint64_t t0 = getCurNs();
  while (__atomic_load_n(&c->h_words[3], __ATOMIC_ACQUIRE) == 0) {
    if (getCurNs() - t0 > c->wait_ns) return false;
  }
  cudaStreamSynchronize(c->g_stream);
  c->resident = false;
  return true;
}
static bool g_pp_ensure_resident(pp_handler_ctx* c) {
  if (c->resident && __atomic_load_n(&c->h_words[3], __ATOMIC_ACQUIRE) == 0) return true;
  if (!g_pp_stop_resident(c)) return false;  // it left after its idle limit: collect it, then launch again
  if (c->bursts) c->rearmed++;
  c->h_words[0] = c->seq;
  c->h_words[1] = c->seq;
  c->h_words[2] = 0;
  c->h_words[3] = 0;
  std::atomic_thread_fence(std::memory_order_seq_cst);
  persistent_swap_hdrs<<<1, 1024, 0, c->g_stream>>>(c->d_stub, c->d_words, c->d_words + 1, c->d_words + 2, c->d_words + 3, c->idle_ns);
  if (cudaGetLastError() != cudaSuccess) return false;
  c->resident = true;
  return true;
}

pp_handler_ctx* setup_g_pp(int device, int launch_type) {
  if (launch_type < 0) launch_type = (int)readEnvInfo<uint16_t>("P2P_RPC_G_PP_LAUNCH_TYPE", 2);
  if (cudaSetDevice(device) != cudaSuccess) return nullptr;
  srpc_parity_preload();
  pp_handler_ctx* c = new pp_handler_ctx;
  c->device = device;
  c->launch_type = (uint8_t)((launch_type == 1 || launch_type == 2) ? launch_type : 0);
  c->idle_ns = (uint64_t)readEnvInfo<uint64_t>("P2P_RPC_G_PP_IDLE_MS", 200) * 1000000ull;
  void *h = nullptr, *w = nullptr;
  if (cudaStreamCreateWithFlags(&c->g_stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaHostAlloc(&h, sizeof(pp_params), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess ||
      cudaHostAlloc(&w, 64, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
    delete c;
    return nullptr;
  }
  std::memset(h, 0, sizeof(pp_params));
  std::memset(w, 0, 64);
  c->h_stub = (pp_params*)h;
  c->h_words = (volatile uint32_t*)w;
  cudaHostGetDevicePointer((void**)&c->d_stub, h, 0);
  cudaHostGetDevicePointer((void**)&c->d_words, w, 0);
  if (c->launch_type == 2 && !g_pp_ensure_resident(c)) c->launch_type = 1;
  return c;
}

int do_g_pp(pp_handler_ctx* c, const p2p_hbufs* h_wi, int clear_sockperf) {
  if (!c || c->launch_type == 0 || !h_wi || h_wi->num_items == 0) return 0;
  cudaSetDevice(c->device);
  const uint32_t n = h_wi->num_items;
  for (uint32_t i = 0; i < n; i++) c->h_stub->hdr_ptrs[i] = h_wi->burst_items[i];
  c->h_stub->num_items = n;
  c->h_stub->clear_sockperf = (uint32_t)clear_sockperf;
  std::atomic_thread_fence(std::memory_order_release);
  c->bursts++;
  if (c->launch_type == 2) {
    for (int attempt = 0; attempt < 2; attempt++) {
      if (!g_pp_ensure_resident(c)) return -2;
      const uint32_t s = ++c->seq;
      __atomic_store_n(&c->h_words[0], s, __ATOMIC_RELEASE);
      const uint64_t t0 = getCurNs();
      bool gone = false;
      for (;;) {
        if (__atomic_load_n(&c->h_words[1], __ATOMIC_ACQUIRE) == s) return 0;
        if (__atomic_load_n(&c->h_words[3], __ATOMIC_ACQUIRE) != 0) {
          gone = true;
          break;
        }
        if (getCurNs() - t0 > c->wait_ns) break;
      }
      // it left (idle limit) around the doorbell, or the wait ran out: stop it for good before anything else.  A header
      // swap is not idempotent, so the burst is only repeated when the kernel left without having touched it.
      const bool served = __atomic_load_n(&c->h_words[1], __ATOMIC_ACQUIRE) == s;
      if (!g_pp_stop_resident(c)) return -2;
      if (served || __atomic_load_n(&c->h_words[1], __ATOMIC_ACQUIRE) == s) return 0;
      if (!gone) {
        c->timeouts++;
        return -1;
      }
    }
    c->timeouts++;
    return -1;
  }
  swap_hdrs_stub_kernel<<<(n + 255) / 256, 256, 0, c->g_stream>>>(c->d_stub);
  if (cudaGetLastError() != cudaSuccess) return -3;
  return cudaStreamSynchronize(c->g_stream) == cudaSuccess ? 0 : -3;
}

void g_pp_counters(const pp_handler_ctx* c, uint64_t* bursts, uint64_t* rearmed, uint64_t* timeouts, int* launch_type) {
  *bursts = c->bursts;
  *rearmed = c->rearmed;
  *timeouts = c->timeouts;
  *launch_type = c->launch_type;
}

void stop_g_pp(pp_handler_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  g_pp_stop_resident(c);
  cudaStreamSynchronize(c->g_stream);
  cudaStreamDestroy(c->g_stream);
  cudaFreeHost(c->h_stub);
  cudaFreeHost((void*)c->h_words);
  delete c;
}

void srpc_parity_preload() {
  cudaFuncAttributes fa;
  (void)cudaFuncGetAttributes(&fa, persistent_swap_hdrs);
  (void)cudaFuncGetAttributes(&fa, swap_hdrs_stub_kernel);
  (void)cudaFuncGetAttributes(&fa, swap_hdrs_kernel);
  (void)cudaFuncGetAttributes(&fa, swap_hdrs_contig_kernel);
  (void)cudaFuncGetAttributes(&fa, lenet_ref_kernel);
  (void)cudaFuncGetAttributes(&fa, lstm_wavefront_kernel);
  (void)cudaFuncGetAttributes(&fa, lstm_bump_kernel);
  (void)cudaFuncGetAttributes(&fa, lstm_grid_kernel<1>);
  (void)cudaFuncGetAttributes(&fa, lstm_grid_kernel<2>);
  (void)cudaFuncGetAttributes(&fa, lstm_grid_kernel<4>);
  (void)cudaFuncGetAttributes(&fa, lstm_grid_kernel<8>);
  (void)cudaGetLastError();
}

static constexpr size_t kLstmWords = (size_t)LLAYERS * LSTEPS * LSTM_GROUP * LH;

size_t srpc_lstm_scratch_bytes(int max_clusters) {
  const size_t cluster_form = (size_t)max_clusters * LLAYERS * LSTEPS * LH * sizeof(float);
  const size_t grid_form = kLstmWords * sizeof(unsigned long long) + 256;
  return cluster_form > grid_form ? cluster_form : grid_form;
}

cudaError_t srpc_lstm(const void* d_stub, const float* direct_in, float* direct_out, const float* weights, float* scratch,
                      int max_clusters, int batch, float forget_bias, uint32_t* status, uint64_t wait_ms, cudaStream_t s) {
  if (batch < 1) return cudaSuccess;
  // Whole-GPU dataflow (cooperative launches, LSTM_GROUP requests each); SPLITRPC_LSTM_CLUSTER=1 or a refused cooperative
  // launch falls back to the one-cluster-per-request kernel.
  static const int use_cluster = [] { const char* e = getenv("SPLITRPC_LSTM_CLUSTER"); return e ? atoi(e) : 0; }();
  static std::atomic<signed char> grid_forms[64];  // per device: 1 all blocks fit it, -1 they do not, 0 not known yet
  std::atomic<signed char>& grid_ok = grid_forms[PerDeviceFlag::current()];
  int done = 0;
  if (!use_cluster) {
    if (!grid_ok.load(std::memory_order_acquire)) {
      int dev = 0, sms = 0, per_sm = 0, coop = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lstm_grid_kernel<LSTM_GROUP>, LSTM_THREADS, 0);
      grid_ok.store(coop && sms * per_sm >= LLAYERS * LSTM_LAYER_BLOCKS ? 1 : -1, std::memory_order_release);
    }
    if (grid_ok.load(std::memory_order_acquire) > 0) {
      LstmGridArgs a;
      a.stub = (const g_params*)d_stub;
      a.direct_in = direct_in;
      a.direct_out = direct_out;
      a.weights = weights;
      a.hbuf = reinterpret_cast<unsigned long long*>(scratch);
      unsigned* epoch = reinterpret_cast<unsigned*>(a.hbuf + kLstmWords);
      a.epoch = epoch;
      a.status = status;
      a.wait_cycles = (long long)(wait_ms < 1000000 ? wait_ms : 1000000) * 2000000;  // at 2 GHz
      a.forget_bias = forget_bias;
      for (; done < batch; done += LSTM_GROUP) {
        a.first = done;
        a.batch = batch - done < LSTM_GROUP ? batch - done : LSTM_GROUP;
        lstm_bump_kernel<<<1, 1, 0, s>>>(epoch);
        if (const cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;  // the words of the launch before would pass for this one's
        void* args[] = {&a};
        const void* fn = a.batch == 1   ? (const void*)lstm_grid_kernel<1>
                         : a.batch == 2 ? (const void*)lstm_grid_kernel<2>
                         : a.batch <= 4 ? (const void*)lstm_grid_kernel<4>
                                        : (const void*)lstm_grid_kernel<8>;
        const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(LLAYERS * LSTM_LAYER_BLOCKS), dim3(LSTM_THREADS), args, 0, s);
        if (e == cudaSuccess) continue;
        (void)cudaGetLastError();
        if (done) return e;
        grid_ok.store(-1, std::memory_order_release);  // not possible on this device: use the cluster kernel from now on
        break;
      }
      if (done) return cudaSuccess;
    }
  }
  int clusters = batch < max_clusters ? batch : max_clusters;
  if (clusters < 1) return cudaSuccess;
  lstm_wavefront_kernel<<<clusters * LLAYERS, 1024, 0, s>>>((const g_params*)d_stub, direct_in, direct_out, weights, scratch,
                                                           batch, forget_bias);
  return cudaGetLastError();
}

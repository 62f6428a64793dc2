// Two-SM persistent GEMM:  D[M,N] = act(A[M,K] . B[N,K]^T + bias + residual), bf16 in and out, fp32 accumulation.
//
// The compute-bound shapes of the one-SM kernel (gemm_persistent.cu) stall on shared memory: for a 128 x 256 tile and a
// 64-deep k-block the loads write 48 KB and the MMAs read 48 KB, 768 cycles at 128 bytes per clock where the tensor pipe takes
// 512.  Here two CTAs of a cluster (an SM pair) compute one 256 x 256 tile with tcgen05.mma.cta_group::2: each CTA loads its own
// 128 rows of A and only HALF of the B rows (32 KB per k-block), one instruction of the leader CTA reads both CTAs' shared
// memory and writes 128 accumulator rows into each CTA's tensor memory.
//
// Protocol (both CTAs run the same code; rank 0 of the pair is the leader):
//   producer   two warps of each CTA, in turn, load its A rows and its half of B for every k-block into a stage ring.  The
//              "full" barrier of a stage is the LEADER's: the leader's producer posts the expected byte count of both
//              CTAs, and both CTAs' TMA loads (cp.async.bulk.tensor ... cta_group::2, no multicast) count on it.
//   MMA        one warp of the leader waits for a full stage, issues four 256 x 256 x 16 MMAs and commits them to
//              the stage's "empty" barrier in BOTH CTAs (tcgen05.commit with a two-CTA mask), then, per tile, to both
//              CTAs' "accumulator full" barriers.  Two accumulators (2 x 256 columns) alternate between tiles.
//   epilogue   16 warps per CTA read their CTA's 128 accumulator rows (tcgen05.ld), 32 rows x 64 columns each, add bias
//              and residual, apply the activation, stage the bf16 tile in swizzled shared memory and hand it to TMA
//              stores; each warp releases the accumulator by arriving on the LEADER's "accumulator empty" barrier.
// Every mbarrier wait is bounded; on a timeout the CTA records an error code and winds down; both CTAs always reach
// the two cluster barriers (after set-up and before tensor memory is freed).  All operands live in this GPU's memory.
//
// Tensor-parallel variant (template flag TP, entry point srpc_gemm_tp_2sm): the same pair tiles with
//   all-gather   copier clusters appended to the grid pull the peers' row shards of A over NVLink into this GPU's
//                gathered buffer (bulk copies through shared memory, no multicast) and publish each 128-row block; the
//                producer of a CTA waits (bounded) for the block its tile needs.  Tiles are ordered so that the rows
//                this rank already holds come first.
//   reduce-scatter  the epilogue stores the staged bf16 tile with 16-byte stores into the slot this rank owns in the
//                memory of the rank that owns the rows (its own slot for its own rows), fences, counts the tile and,
//                when the last tile for an owner is through, publishes the step number there.  Rows owned by peers
//                come first, so that their transfer overlaps the rest of the GEMM.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "fast_div.h"
#include "gemm_tcgen05.h"
#include "pdl_launch.h"
#include "per_device.h"
#include "ptx.cuh"
#include "tp_device.cuh"

cudaError_t srpc_tensor_map_2d(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                               uint32_t box_inner, uint32_t box_outer);
cudaError_t srpc_tensor_map_im2col(CUtensorMap* m, const void* ptr, int n, int h, int w, int c, int r, int s, int stride, int pad,
                                   int pixels);

namespace {

constexpr int BM = 128;   // rows per CTA; a pair computes 256
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int OUT_HALF_BYTES = BM * 128;    // 128 rows x 64 bf16 columns
constexpr int OUT_CHUNK_BYTES = 32 * 64;    // 32 rows x 32 bf16 columns

// Tile widths 128 / 192 / 256: one epilogue warp per 64 columns and TMEM lane quarter, as many stages as fit.
//
// What bounds the k loop: shared memory.  Loads write (128 + BN / 2) x 128 bytes per k-block and SM, MMAs read (128 + BN) x
// 128, and both together move 128 bytes per clock: 640 cycles for BN = 256 against 512 of the tensor pipe.
//
// What a launch costs beside it, and what was done about it (4096 x 2304 x 768, two tiles of 3.5 us each per pair): a
// cluster barrier with release / acquire takes 0.85 us, twice per launch, and so does every release to the peer, 0.6 us per
// tile: none of the three orders memory here (relaxed forms, see ptx.cuh).  The epilogue reads the accumulator as 8 x 8
// fragments: bias and residual are then packed pairs of columns, where a thread with a whole row needs every bias value of
// the tile broadcast to it through the pipe that the MMAs' operands take; with stmatrix behind it the last
// tile's epilogue takes 2.4 us instead of 3.9.  Together (us before -> now): 4096 x 2304 x 768 14.9 -> 12.4, 4096 x 3072 x 768
// with GELU 24.0 -> 20.0, 4096 x 768 x 3072 with residual 18.9 -> 15.8, 6144 x 1024 x 1024 16.2 -> 12.9, 12544 x 256 x 1024 12.0 -> 10.3.
// Not better: stores of 32 bytes per lane instead of TMA stores (17.5 us for the first), 64 columns per store (one operand
// stage less, 13.2 us).
//
// Output staging: every epilogue warp has a block of its own, one or two chunks of 32 rows x 32 columns (2 KB), so that no warp
// waits for another one between reading its part of the accumulator and handing it to its TMA store.  The 256-wide tile has
// one chunk per warp: the memory goes to a sixth operand stage.  (Peer stores use the same memory as one block of PASS_COLS
// columns per pass.)
// Rows per CTA: 128, or 64 for products with few tiles (RPC).  With 64 rows the accumulator's columns lie in two halves one
// below the other in tensor memory (lanes 0 - 63: columns 0 .. BN / 2 - 1, lanes 64 - 127: the others), a k-block takes 55 - 76 ns of
// the tensor pipe instead of 150, and two of them share a stage, since a turn of the MMA loop takes 134 ns whatever it issues.
template <int BN, int RPC, bool TP>
struct Cfg {
  static constexpr int KPS = RPC == 64 || BN == 64 ? 2 : 1;         // k-blocks per stage
  static constexpr int A_BYTES = RPC * BK * 2;
  static constexpr int KB_BYTES = A_BYTES + (BN / 2) * BK * 2;      // A rows and this CTA's half of the B rows
  static constexpr int STAGE_BYTES = KPS * KB_BYTES;
  static constexpr int PASSES = BN == 256 ? 2 : 1;
  static constexpr int PASS_COLS = BN / PASSES;
  static constexpr int QC = RPC == 128 ? BN : BN / 2;               // columns of a TMEM lane quarter
  static constexpr int NCH = RPC == 128 && BN >= 128 ? 2 : 1;       // 32-column chunks per epilogue warp
  static constexpr int EPI_WARPS = 4 * QC / (32 * NCH);
  static constexpr int CHUNK_BUFS = BN == 256 ? 1 : 2;
  static constexpr int OUT_BYTES = EPI_WARPS * CHUNK_BUFS * OUT_CHUNK_BYTES;
  static constexpr int STAGES = (224 * 1024 - OUT_BYTES) / STAGE_BYTES;
  static constexpr int EPI_THREADS = 32 * EPI_WARPS;
  static constexpr int THREADS = 64 + EPI_THREADS + 32;  // TMA, MMA, epilogue, second TMA warp
  static constexpr int ACC_STRIDE = QC == 192 ? 256 : QC;  // TMEM columns between the two accumulators
  static constexpr int TMEM_COLS = 2 * ACC_STRIDE;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + OUT_BYTES;
  static_assert(!TP || (RPC == 128 && OUT_BYTES == (PASS_COLS / 64) * OUT_HALF_BYTES), "peer stores stage whole passes");
};

__device__ __forceinline__ void named_bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
// Optional phase time stamps of block 0 (build with -DSRPC_GEMM_TRACE), read back through srpc_gemm_trace_read.
#ifdef SRPC_GEMM_TRACE
__device__ unsigned long long g_gemm2_trace[16];
#define GEMM2_TRACE(slot)                                             \
  do {                                                                \
    if (blockIdx.x == 0) g_gemm2_trace[slot] = ptx::globaltimer_ns(); \
  } while (0)
#else
#define GEMM2_TRACE(slot) ((void)0)
#endif

struct PairTile {
  int m2, n;  // 256-row block, 256-column block
};

struct TileOrder {
  int clusters;  // clusters that compute tiles (the grid may hold copier clusters after them)
  int tiles_m2, tiles_n;
  int group_m;   // pair row blocks per group
  // From the last tile to the first.  Products that read more than they write go this way: the rows that the kernel before wrote
  // last are still in the L2 cache, and the rows read last are again when a later product takes them as its residual, in order
  // (200704 x 64 x 256 behind the layer that writes its 103 MB 21.7 -> 18.5 us; ResNet-50, 64 images 936 -> 930).  Behind a copy that has written
  // A front to back, forward / backward without the copy: 200704 x 64 x 256 20.5 / 18.8, 200704 x 128 x 256 24.9 / 24.2, 60000 x 256 x 1024 33.1 / 31.1,
  // 24576 x 1024 x 4096 142.5 / 141.1, 50176 x 128 x 512, 12544 x 256 x 1024 and 40000 x 768 x 3072 within 2 %; none is slower.
  int reverse;
  int m_rot2;    // rotation of the pair row blocks (tensor-parallel: which rank's rows come first)
  int late_trigger;  // the next kernel starts behind this CTA's last load only (pdl_launch.h)
  FastDiv fd_group, fd_gm;  // by group_m * tiles_n and group_m
};

// j-th tile of this cluster, grouped so that tiles in flight share A and B blocks in L2 (see row_blocks_per_group).
__device__ __forceinline__ bool pair_tile(int j, const TileOrder& o, PairTile* out) {
  int tile = (int)(blockIdx.x >> 1) + j * o.clusters;
  if (tile >= o.tiles_m2 * o.tiles_n) return false;
  if (o.reverse) tile = o.tiles_m2 * o.tiles_n - 1 - tile;
  const int g = (int)fdiv(o.fd_group, (uint32_t)tile), in_g = tile - g * o.group_m * o.tiles_n;
  const int m_first = g * o.group_m;
  int m2;
  if (o.tiles_m2 - m_first >= o.group_m) {
    out->n = (int)fdiv(o.fd_gm, (uint32_t)in_g);
    m2 = m_first + in_g - out->n * o.group_m;
  } else {  // last, shorter group
    const int gm = o.tiles_m2 - m_first;
    out->n = in_g / gm;
    m2 = m_first + in_g - out->n * gm;
  }
  m2 += o.m_rot2;
  out->m2 = m2 >= o.tiles_m2 ? m2 - o.tiles_m2 : m2;
  return true;
}

// Where the rows of A come from.  GEMM: a matrix.  Convolution: row i of the product is output pixel i (rows and images in
// sequence), its A row for filter tap (fr, fs) the pixel that the tap meets, read through an im2col tensor map; k-blocks from
// kb_split on come from a second input (two-input 1x1 convolution) by tmap_a2.
enum { MATRIX, CONVOLUTION, TWO_INPUTS };
struct ASource {
  int im2col, im2col2;  // of the first / second input
  int kb_split;
  int stride, pad, stride2;
  FastDiv fd_img, fd_ow;      // by output pixels per image and per row
  FastDiv fd_cblocks, fd_s;   // by channel blocks and filter columns
  FastDiv fd_rows;            // by filter rows where they are innermost (srpc_conv_rows_innermost), by 1 otherwise
};

// Channels of A, filter tap and columns of the weights that k-block kb of a convolution multiplies (the second input's: columns only).
struct KBlock {
  int c, w;
  uint16_t fs, fr;
};
__device__ __forceinline__ KBlock conv_kblock(const ASource& src, int kb) {
  const int group = (int)fdiv(src.fd_rows, (uint32_t)kb), tap = (int)fdiv(src.fd_cblocks, (uint32_t)group);
  const int cb = group - tap * (int)src.fd_cblocks.d;
  int fr, fs;
  if (src.fd_rows.d > 1) {
    fr = kb - group * (int)src.fd_rows.d;
    fs = tap;
  } else {
    fr = (int)fdiv(src.fd_s, (uint32_t)tap);
    fs = tap - fr * (int)src.fd_s.d;
  }
  const int at = src.fd_rows.d > 1 ? (fr * (int)src.fd_s.d + fs) * (int)src.fd_cblocks.d + cb : kb;
  return KBlock{cb * BK, at * BK, (uint16_t)fs, (uint16_t)fr};
}

// The tensor-parallel part of the arguments; the plain kernel's launches do not carry its 288 bytes.
struct NoTp {};
template <bool TP>
using TpArg = std::conditional_t<TP, TpParams, NoTp>;

template <int BN, int RPC, bool TP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Cfg<BN, RPC, TP>::THREADS, 1)
gemm_2sm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ CUtensorMap tmap_a2, int M, int N, int K,
                const TileOrder order, const ASource src, GemmEpilogue ep, uint32_t* status, const TpArg<TP> tp_in) {
  using C = Cfg<BN, RPC, TP>;
  constexpr int A_BYTES = C::A_BYTES, KB_BYTES = C::KB_BYTES, KPS = C::KPS, STAGE_BYTES = C::STAGE_BYTES, STAGES = C::STAGES;
  constexpr int EPI_THREADS = C::EPI_THREADS, ACC_STRIDE = C::ACC_STRIDE, NCH = C::NCH;
  constexpr int PASSES = C::PASSES, PASS_COLS = C::PASS_COLS;
  extern __shared__ __align__(1024) uint8_t smem[];
  TpArg<TP> tp = tp_in;
  if constexpr (TP) {
    if (tp.epoch_base) tp.epoch += *tp.epoch_base;
    if ((int)(blockIdx.x >> 1) >= order.clusters) {
      // Copier CTA: neither of the pair takes part in the cluster barriers below, nor holds tensor memory.
      tpdev::copier(tp, (int)blockIdx.x - 2 * order.clusters, smem, status);
      return;
    }
  }
  uint8_t* stage_out = smem + (size_t)STAGES * STAGE_BYTES;
  __shared__ __align__(8) uint64_t full_bar[STAGES];   // used in the leader only
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t tmem_full_bar[2];
  __shared__ __align__(8) uint64_t tmem_empty_bar[2];  // used in the leader only: arrivals from both CTAs' epilogue warps
  __shared__ uint32_t tmem_base_smem;
  __shared__ uint32_t s_error;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const bool leader = rank == 0;
  const int num_kb = (K + BK - 1) / BK, num_st = (num_kb + KPS - 1) / KPS;  // k-blocks, stages of them
  // The swizzled tiles and their descriptors need a 1024-byte aligned base; the layout is the same in both CTAs, so
  // both take the same decision.
  const bool layout_ok = (ptx::smem_u32(smem) & 1023u) == 0;

  if (threadIdx.x == 0) {
    GEMM2_TRACE(0);
    for (int s = 0; s < STAGES; s++) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; a++) {
      ptx::mbar_init(&tmem_full_bar[a], 1);
      ptx::mbar_init(&tmem_empty_bar[a], 2 * (EPI_THREADS / 32));
    }
    ptx::fence_mbar_init();
    s_error = layout_ok ? 0u : (uint32_t)GEMM_ERR_PRODUCER_WAIT;
    ptx::prefetch_tmap(&tmap_a);
    ptx::prefetch_tmap(&tmap_b);
    ptx::prefetch_tmap(&tmap_out);
    if (src.kb_split < num_kb) ptx::prefetch_tmap(&tmap_a2);
  }
  if (warp == 1) {
    ptx::tmem_alloc_2sm(&tmem_base_smem, C::TMEM_COLS);
    ptx::tmem_relinquish_2sm();
    if (!order.late_trigger) ptx::grid_dep_launch();  // after the allocation, see pdl_launch.h
  }
  ptx::tc_fence_before();
  __syncthreads();
  // The peer's barriers must exist before anything signals them; every role waits for that where it first matters.
  ptx::cluster_arrive_relaxed();
  ptx::tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;

  if (warp == 0 || warp == C::THREADS / 32 - 1) {
    // ---------------- producers: two warps per CTA take the k-blocks in turn (see gemm_persistent.cu).  Each walks the schedule
    // as one and an elected lane issues, so that the operands of the loads stay in uniform registers (an iteration of
    // the loads alone: 240 ns in one lane's branch, 200 ns this way).
    constexpr int PRODUCERS = 2;
    const bool elected = ptx::elect_one();
    int st = warp == 0 ? 0 : 1, s = st, j = 0, seq = st;  // stage of the tile; seq: position in this cluster's sequence of stages
    uint32_t ph = 0;
    PairTile t;
    bool ok = layout_ok, first = true;
    // The rest of a tile's stages.  A matrix, a convolution and one with a second input have a loop each: with the choices inside one
    // loop a stage took 50 ns more of the issuing warps' time (128 x 768 x 3072 8.1 us, now 6.8; 3x3 over 32 x 56 x 56 x 64 13.9 and 11.6,
    // 64 x 28 x 28 x 128 16.9 and 14.7).
    auto stages = [&](auto source, int row0, int brow0, int img, int y, int x, bool first_tile) {
      constexpr int SOURCE = decltype(source)::value;
      for (; st < num_st; st += PRODUCERS) {
        // Which tap, channels and weights the stage takes: worked out before the wait (behind it, 1 % of a 3x3 convolution).
        KBlock at[KPS];
        if (SOURCE == CONVOLUTION || (SOURCE == TWO_INPUTS && src.im2col)) {
#pragma unroll
          for (int b = 0; b < KPS; b++) at[b] = conv_kblock(src, st * KPS + b);
        }
        ok = ptx::mbar_wait_warp(&empty_bar[s], ph ^ 1u);
        if (!ok) {
          if (elected) atomicExch(&s_error, GEMM_ERR_PRODUCER_WAIT);
          break;
        }
        const uint32_t full_leader = ptx::mapa_shared(ptx::smem_u32(&full_bar[s]), 0);
        uint8_t* sa = smem + (size_t)s * STAGE_BYTES;
        if (first) {
          // everything above overlaps the kernel before; its results are read below
          ptx::cluster_wait();
          if (lane == 0 && warp == 0) GEMM2_TRACE(1);
          ptx::grid_dep_wait();
          first = false;
        }
        const int blocks = KPS == 1 || st * KPS + 1 < num_kb ? KPS : 1;
        if (elected && leader) ptx::mbar_expect_tx(&full_bar[s], 2u * KB_BYTES * blocks);
#pragma unroll
        for (int b = 0; b < KPS; b++) {
          if (b >= blocks) break;
          const int kb = st * KPS + b;
          if (SOURCE == MATRIX || (SOURCE == TWO_INPUTS && !src.im2col && kb < src.kb_split)) {
            if (elected) ptx::tma_load_2d_2sm(sa + b * KB_BYTES, &tmap_a, full_leader, kb * BK, row0);
          } else if (SOURCE == CONVOLUTION || kb < src.kb_split) {
            if (elected)
              ptx::tma_load_im2col_2sm(sa + b * KB_BYTES, &tmap_a, full_leader, at[b].c, x * src.stride - src.pad, y * src.stride - src.pad,
                                       img, at[b].fs, at[b].fr);
          } else if (src.im2col2) {
            if (elected)
              ptx::tma_load_im2col_2sm(sa + b * KB_BYTES, &tmap_a2, full_leader, (kb - src.kb_split) * BK, x * src.stride2, y * src.stride2, img,
                                       0, 0);
          } else if (elected) {
            ptx::tma_load_2d_2sm(sa + b * KB_BYTES, &tmap_a2, full_leader, (kb - src.kb_split) * BK, row0);
          }
          if (elected) ptx::tma_load_2d_2sm(sa + b * KB_BYTES + A_BYTES, &tmap_b, full_leader, SOURCE == CONVOLUTION || (SOURCE == TWO_INPUTS && src.im2col) ? at[b].w : kb * BK, brow0);
        }
        if (first_tile && st == 0 && lane == 0) GEMM2_TRACE(2);
        seq += PRODUCERS;
        s += PRODUCERS;
        if (s >= STAGES) {
          s -= STAGES;
          ph ^= 1u;
        }
      }
    };
    const int source = src.kb_split < num_kb ? TWO_INPUTS : src.im2col ? CONVOLUTION : MATRIX;
    while (ok) {
      for (; st >= num_st; st -= num_st) j++;
      ok = __all_sync(0xffffffffu, *(volatile uint32_t*)&s_error == 0);
      if (!ok || !pair_tile(j, order, &t)) break;
      const int row0 = (t.m2 * 2 + (int)rank) * RPC;
      const int brow0 = t.n * BN + (int)rank * (BN / 2);
      int img = 0, y = 0, x = 0;  // output pixel of the first row
      if ((src.im2col | src.im2col2) && row0 < M) {  // (rows behind the last pixel: any pixels, the results are not stored)
        img = (int)fdiv(src.fd_img, (uint32_t)row0);
        const int in_img = row0 - img * (int)src.fd_img.d;
        y = (int)fdiv(src.fd_ow, (uint32_t)in_img);
        x = in_img - y * (int)src.fd_ow.d;
      }
      if constexpr (TP) {
        if (tp.mblock_ready) {
          // Rows of a peer arrive through the copier clusters of this launch, one 128-row block at a time.
          const int m_idx = t.m2 * 2 + (int)rank;
          if (m_idx / tp.mblocks_per_rank != tp.rank) {
            if (elected) {
              ok = tpdev::wait_flag_gpu(tp.mblock_ready + m_idx, tp.epoch);
              ptx::fence_proxy_async_all();  // the copier's writes -> this thread's TMA reads
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
              if (elected) atomicExch(&s_error, GEMM_ERR_TP_BLOCK_WAIT);
              break;
            }
          }
        }
      }
      if (source == MATRIX) stages(std::integral_constant<int, MATRIX>{}, row0, brow0, img, y, x, j == 0);
      else if (source == CONVOLUTION) stages(std::integral_constant<int, CONVOLUTION>{}, row0, brow0, img, y, x, j == 0);
      else stages(std::integral_constant<int, TWO_INPUTS>{}, row0, brow0, img, y, x, j == 0);
    }
    if (order.late_trigger && warp == 0) {
      __syncwarp();
      ptx::grid_dep_launch();
    }
    if (first) ptx::cluster_wait();  // this warp had no k-block
    // The leader's MMAs signal the stages of both CTAs, and none of those signals may still be on its way when this CTA leaves:
    // wait as for the STAGES stages behind the last one (this warp's share of them).
    if (ok) {
      const int tiles = order.tiles_m2 * order.tiles_n, first_tile = (int)(blockIdx.x >> 1);
      const int total = first_tile < tiles ? ((tiles - first_tile + order.clusters - 1) / order.clusters) * num_st : 0;
      for (int i = seq - total; ok && i < STAGES; i += PRODUCERS) {
        ok = ptx::mbar_wait_warp(&empty_bar[s], ph ^ 1u);
        s += PRODUCERS;
        if (s >= STAGES) {
          s -= STAGES;
          ph ^= 1u;
        }
      }
      if (!ok && elected) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_PRODUCER_WAIT);
    }
  } else if (warp == 1) {
    // ---------------- MMA issue (leader only): the warp walks the schedule together, one elected lane issues, so that
    // descriptors and addresses stay in uniform registers (see gemm_persistent.cu)
    ptx::cluster_wait();
    if (leader) {
      const bool elected = ptx::elect_one();
      const uint32_t idesc = ptx::umma_idesc_bf16(2 * RPC, BN);
      const uint32_t ring_lo = ptx::umma_desc_lo(ptx::smem_u32(smem));
      constexpr uint32_t K_LO = UMMA_K * 2 / 16;
      int s = 0;
      uint32_t ph = 0, local = 0;
      PairTile t;
      bool ok = layout_ok;
      for (int j = 0; ok && pair_tile(j, order, &t); j++, local++) {
        const uint32_t acc = local & 1u;
        ok = ptx::mbar_wait_warp(&tmem_empty_bar[acc], ((local >> 1) & 1u) ^ 1u);
        if (!ok) break;
        ptx::tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * ACC_STRIDE;
        for (int st = 0; st < num_st; st++) {
          ok = ptx::mbar_wait_warp(&full_bar[s], ph);
          if (!ok) break;
          if (j == 0 && st == 0 && lane == 0) GEMM2_TRACE(3);
          if (j == 0 && st == 8 && lane == 0) GEMM2_TRACE(10);
          if (j == 0 && st == 24 && lane == 0) GEMM2_TRACE(11);
          const uint32_t sa = ring_lo + (uint32_t)s * (STAGE_BYTES / 16), sb = sa + A_BYTES / 16;
          if (elected) {
#pragma unroll
            for (int b = 0; b < KPS; b++) {
              if (KPS > 1 && b > 0 && st * KPS + b >= num_kb) break;
#pragma unroll
              for (int k = 0; k < BK / UMMA_K; k++)
                ptx::umma_bf16_2sm(d_tmem, ptx::umma_desc_join(sa + b * (KB_BYTES / 16) + k * K_LO),
                                   ptx::umma_desc_join(sb + b * (KB_BYTES / 16) + k * K_LO), idesc, (st | b | k) != 0 ? 1u : 0u);
            }
            ptx::umma_commit_2sm(&empty_bar[s], 3);  // frees the stage in both CTAs
          }
          if (++s == STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
        if (!ok) break;
        if (elected) ptx::umma_commit_2sm(&tmem_full_bar[acc], 3);
        if (j == 0 && lane == 0) GEMM2_TRACE(4);
        ok = *(volatile uint32_t*)&s_error == 0;
        ok = __all_sync(0xffffffffu, ok);
      }
      // the peer's last hand-backs have arrived before this CTA leaves
      for (int i = 0; ok && i < 2; i++, local++) ok = ptx::mbar_wait_warp(&tmem_empty_bar[local & 1u], ((local >> 1) & 1u) ^ 1u);
      if (!ok && elected) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_MMA_WAIT);
    }
  } else {
    // ---------------- epilogue: a warp has 32 rows (its TMEM lane quarter) x two chunks of 32 columns of the tile and goes through
    // them on its own: residual and bias on their way before the accumulator is ready, its own TMA stores.
    ptx::grid_dep_wait();
    ptx::cluster_wait();
    const int warp_q = warp & 3;
    const int cgroup = (warp - 2) >> 2;      // 0 .. EPI_THREADS/128 - 1
    // first row and column of this warp's lane quarter in the CTA's part of the tile
    const int q_row = RPC == 128 ? warp_q * 32 : (warp_q & 1) * 32, q_col = RPC == 128 ? 0 : (warp_q >> 1) * (BN / 2);
    const int et = threadIdx.x - 64;
    // This thread's accumulator elements: columns 8 g + fc, + 1 (g = 0 .. 3) of rows fr + 8 i (i = 0 .. 3) of the warp's 32 rows.
    const int fr = lane >> 2, fc = (lane & 3) * 2;
    // pairs of residual columns (a pair is inside the matrix or outside)
    const bool vec_res = ep.residual && (((ep.ldr | N) & 1) == 0) && (((uintptr_t)ep.residual & 3) == 0);
    // column of chunk ch inside the lane quarter
    auto chunk_col = [&](int ch) { return PASSES == 2 && TP ? ch * PASS_COLS + cgroup * 32 : (cgroup * NCH + ch) * 32; };
    uint8_t* stage = stage_out + (size_t)(warp - 2) * C::CHUNK_BUFS * OUT_CHUNK_BYTES;
    // what this lane names in stmatrix: matrices 0, 1 = rows 0 .. 7, 8 .. 15 of one column group, 2, 3 = of the next one
    const int st_row = (lane & 7) + (lane & 8), st_cg = lane >> 4;
    uint32_t local = 0;
    PairTile t;
    bool peer_store = false;
    if constexpr (TP) peer_store = tp.rs != 0;
    bool ok = layout_ok;
    for (int j = 0; ok && pair_tile(j, order, &t); j++, local++) {
      const uint32_t acc = local & 1u;
      const int m0 = (t.m2 * 2 + (int)rank) * RPC + q_row;  // first row of this warp
      const int n0 = t.n * BN + q_col;
      // Residual and bias arrive before the accumulator is ready.
      uint32_t rq[NCH][16];
      if (vec_res) {
#pragma unroll
        for (int ch = 0; ch < NCH; ch++) {
          const int col = n0 + chunk_col(ch) + fc;
          const bool whole = n0 + chunk_col(ch) + 32 <= N;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const int m = m0 + fr + 8 * i;
            if (m < M) {
              const __nv_bfloat16* rp = ep.residual + (size_t)m * ep.ldr + col;
              if (whole) {
#pragma unroll
                for (int g = 0; g < 4; g++) rq[ch][i * 4 + g] = *reinterpret_cast<const uint32_t*>(rp + g * 8);
              } else {
#pragma unroll
                for (int g = 0; g < 4; g++)
                  if (col + g * 8 < N) rq[ch][i * 4 + g] = *reinterpret_cast<const uint32_t*>(rp + g * 8);
              }
            }
          }
        }
      }
      float2 b2[NCH][4];
      if (ep.bias) {
#pragma unroll
        for (int ch = 0; ch < NCH; ch++)
#pragma unroll
          for (int g = 0; g < 4; g++) {
            const int col = n0 + chunk_col(ch) + g * 8 + fc;
            if (col + 1 < N) b2[ch][g] = *reinterpret_cast<const float2*>(ep.bias + col);
            else b2[ch][g] = make_float2(col < N ? ep.bias[col] : 0.f, 0.f);
          }
      }
      ok = *(volatile uint32_t*)&s_error == 0 && ptx::mbar_wait(&tmem_full_bar[acc], (local >> 1) & 1u);
      ok = __all_sync(0xffffffffu, ok);
      if (TP && peer_store) ok = ptx::named_bar_all(2, EPI_THREADS, ok);
      if (!ok) {
        if (lane == 0) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_EPILOGUE_WAIT);
        break;
      }
      ptx::tc_fence_after();
      if (j == 0 && et == 0) GEMM2_TRACE(5);
#pragma unroll
      for (int ch = 0; ch < NCH; ch++) {
        const int c = chunk_col(ch);  // column inside the lane quarter
        const int col0 = n0 + c;
        const uint32_t t_addr = tmem_base + acc * ACC_STRIDE + ((uint32_t)(warp_q * 32) << 16) + (uint32_t)c;
        uint32_t r[32];
        ptx::tmem_ld_16x256b_x4(t_addr, r);
        ptx::tmem_ld_16x256b_x4(t_addr + (16u << 16), r + 16);
        ptx::tmem_ld_wait();
        if (ch == NCH - 1) {  // last read: hand the accumulator back to the leader's MMA warp
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster(ptx::mapa_shared(ptx::smem_u32(&tmem_empty_bar[acc]), 0));
        }
        float2 v[16];  // [row group i][column group g]
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int g = 0; g < 4; g++) {
            const int at = (i >> 1) * 16 + g * 4 + (i & 1) * 2;
            v[i * 4 + g] = make_float2(__uint_as_float(r[at]), __uint_as_float(r[at + 1]));
          }
        if (ep.bias) {
#pragma unroll
          for (int q = 0; q < 16; q++) v[q] = __fadd2_rn(v[q], b2[ch][q & 3]);
        }
        if (vec_res) {
#pragma unroll
          for (int q = 0; q < 16; q++) v[q] = __fadd2_rn(v[q], __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&rq[ch][q])));
        } else if (ep.residual) {
#pragma unroll
          for (int q = 0; q < 16; q++) {
            const int m = m0 + fr + 8 * (q >> 2), col = col0 + (q & 3) * 8 + fc;
            const __nv_bfloat16* rp = ep.residual + (size_t)m * ep.ldr + col;
            if (m < M && col < N) v[q].x += __bfloat162float(rp[0]);
            if (m < M && col + 1 < N) v[q].y += __bfloat162float(rp[1]);
          }
        }
        if (ep.act == GEMM_ACT_RELU) {
#pragma unroll
          for (int q = 0; q < 16; q++) v[q] = make_float2(fmaxf(v[q].x, 0.f), fmaxf(v[q].y, 0.f));
        } else if (ep.act == GEMM_ACT_GELU) {
#pragma unroll
          for (int q = 0; q < 16; q++) v[q] = ptx::gelu_erf_fast2(v[q]);
        } else if (ep.act == GEMM_ACT_TANH) {
#pragma unroll
          for (int q = 0; q < 16; q++) v[q] = make_float2(tanhf(v[q].x), tanhf(v[q].y));
        }
        uint32_t o[16];
#pragma unroll
        for (int q = 0; q < 16; q++) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(v[q].x, v[q].y);
          o[q] = *reinterpret_cast<const uint32_t*>(&h);
        }
        // Rows of `row_bytes`, 16-byte pieces exchanged within a row by piece XOR swz(row): piece `first` + column group.
        auto put = [&](uint8_t* base, int row_bytes, int first, auto swz) {
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int g = 0; g < 4; g += 2) {
              const int rr = h * 16 + st_row;
              const uint32_t addr = ptx::smem_u32(base) + (uint32_t)(rr * row_bytes + (((first + g + st_cg) ^ swz(rr)) << 4));
              ptx::stmatrix_x4(addr, o[(2 * h) * 4 + g], o[(2 * h + 1) * 4 + g], o[(2 * h) * 4 + g + 1], o[(2 * h + 1) * 4 + g + 1]);
            }
        };
        if constexpr (TP) {
          if (peer_store) {
            // The tile goes to the slot this rank owns on the rank that owns these rows (rows per rank are a multiple
            // of 128, so a CTA's half tile has one owner), PASS_COLS columns at a time.
            const int pass = PASSES == 2 ? ch : 0, cp = c - pass * PASS_COLS;  // column inside the pass
            if (PASSES == 2 || ch == 0) named_bar_sync(1, EPI_THREADS);        // the previous pass has been read
            put(stage_out + (size_t)(cp >> 6) * OUT_HALF_BYTES + (size_t)(warp_q * 32) * 128, 128, (cp & 63) >> 3, [](int rr) { return rr & 7; });
            if (PASSES == 1 && ch == 0) continue;
            named_bar_sync(1, EPI_THREADS);
            const int m_idx = t.m2 * 2 + (int)rank;
            const int owner = m_idx / tp.mblocks_per_rank;
            const int local_m0 = (m_idx - owner * tp.mblocks_per_rank) * BM;
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(tp.dst[owner]);
            constexpr int SEGS = PASS_COLS / 8;  // 16-byte segments per row of this pass
#pragma unroll 4
            for (int q = et; q < BM * SEGS; q += EPI_THREADS) {
              const int rr = q / SEGS, seg = q - rr * SEGS;
              const int col = n0 + pass * PASS_COLS + seg * 8;
              if (col < N) {
                const uint8_t* src = stage_out + (size_t)(seg >> 3) * OUT_HALF_BYTES + (size_t)rr * 128 + (((seg & 7) ^ (rr & 7)) << 4);
                *reinterpret_cast<uint4*>(dst + (size_t)(local_m0 + rr) * ep.ldo + col) = *reinterpret_cast<const uint4*>(src);
              }
            }
            if (ch == 1) {
              // Every thread's stores of every pass are ordered before the barrier; the one system-scope fence behind
              // it (fences are cumulative) then makes the whole half tile visible on the owner before the count, and
              // through the count before the flag.  A fence per thread costs hundreds of them per tile.
              named_bar_sync(1, EPI_THREADS);
              if (et == 0) {
                __threadfence_system();
                const uint32_t done = atomicAdd(tp.owner_count + owner, 1u) + 1u;
                if (done == (uint32_t)tp.tiles_per_owner) {
                  atomicExch(tp.owner_count + owner, 0u);
                  __threadfence_system();
                  ptx::st_release_sys(tp.dst_flag[owner], tp.epoch);
                }
              }
            }
            continue;
          }
        }
        // A chunk is a block of 32 rows of 64 bytes under the 64-byte swizzle; its last store must have been read.
        uint8_t* block = stage + (C::CHUNK_BUFS == 2 ? (NCH == 2 ? ch : (int)(local & 1u)) * OUT_CHUNK_BYTES : 0);
        if (lane == 0) ptx::bulk_wait_read<C::CHUNK_BUFS - 1>();
        __syncwarp();
        put(block, 64, 0, [](int rr) { return (rr >> 1) & 3; });
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (col0 < N && m0 < M) ptx::tma_store_2d(&tmap_out, block, col0, m0);
          ptx::bulk_commit();
        }
        if (j == 0 && et == 0 && ch == NCH - 1) GEMM2_TRACE(6);
      }
    }
    if (et == 0) GEMM2_TRACE(7);
    if (lane == 0) ptx::bulk_wait_read<0>();
    if (et == 0) GEMM2_TRACE(8);
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (s_error != 0) {
    if (threadIdx.x == 0 && status) atomicExch(status, s_error);
    __nanosleep(1000000);  // let loads that are still in flight land before the block leaves
  }
  // Every signal to this CTA has arrived (above) and the peer's MMAs no longer read its shared memory (its last accumulator was
  // complete); tensor memory is given back by both CTAs together.
  ptx::cluster_arrive_relaxed();
  ptx::cluster_wait();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_2sm(tmem_base, C::TMEM_COLS);
  }
}


// Clusters of two CTAs that can be resident at once (queried once per instantiation and device).
template <int BN, int RPC, bool TP>
cudaError_t max_clusters_2sm(int* out) {
  using C = Cfg<BN, RPC, TP>;
  static std::atomic<int> per_device[64];
  const int dev = PerDeviceFlag::current();
  int max_clusters = per_device[dev].load(std::memory_order_acquire);
  if (!max_clusters) {
    cudaError_t e = cudaFuncSetAttribute(gemm_2sm_kernel<BN, RPC, TP>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * 74);
    cfg.blockDim = dim3(C::THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, gemm_2sm_kernel<BN, RPC, TP>, &cfg);
    if (e != cudaSuccess) return e;
    if (n < 1) return cudaErrorInvalidConfiguration;
    max_clusters = n;
    per_device[dev].store(n, std::memory_order_release);
  }
  *out = max_clusters;
  return cudaSuccess;
}

// A matrix of rows as the only source.
ASource matrix_source(int num_kb) {
  ASource src = {};
  src.kb_split = num_kb;
  src.stride = src.stride2 = 1;
  src.fd_img = src.fd_ow = src.fd_cblocks = src.fd_s = src.fd_rows = make_fastdiv(1);
  return src;
}

void order_tiles(TileOrder* o, int M, int N, int rows, int bn, int max_clusters, int group_m) {
  o->tiles_m2 = (M + rows - 1) / rows;
  o->tiles_n = (N + bn - 1) / bn;
  o->clusters = std::min(o->tiles_m2 * o->tiles_n, max_clusters);
  o->group_m = group_m;
  o->fd_group = make_fastdiv((uint32_t)(group_m * o->tiles_n));
  o->fd_gm = make_fastdiv((uint32_t)group_m);
}

// Row blocks that walk the columns together.  B is read again for every group: while it stays in L2 four are best, and once it takes
// more than half of the 126 MB eight save reads from DRAM, and with them power that the tensor cores have instead.  Us with four /
// eight, sustained: 8192^3 911 / 858, 8192 x 8192 x 4096 445 / 415, 6000^3 368 / 354; 16384 x 4096 x 4096 401 / 414, 8192 x 1024 x
// 8192 114.0 / 116.5, 8192 x 8192 x 1024 113.1 / 114.9; 5000^3 and 4096 x 4096 x 8192 (50 and 67 MB) alike.
int row_blocks_per_group(int N, int K) { return (uint64_t)N * K * 2 > 63u * 1000 * 1000 ? 8 : 4; }

// What a launch reads its A rows from: makes the tensor maps for tiles of `rows_per_cta` rows per CTA.
struct AInput {
  const void* a = nullptr;
  int lda = 0;
  const ConvShape* cs = nullptr;
};
cudaError_t a_maps(const AInput& in, int M, int K, int rows_per_cta, ASource* src, CUtensorMap* ta, CUtensorMap* ta2) {
  *src = matrix_source((K + BK - 1) / BK);
  if (!in.cs) {
    cudaError_t e = srpc_tensor_map_2d(ta, in.a, (uint64_t)K, (uint64_t)M, (uint64_t)in.lda * 2, BK, (uint32_t)rows_per_cta);
    *ta2 = *ta;
    return e;
  }
  const ConvShape& cs = *in.cs;
  src->kb_split = cs.r * cs.s * cs.cin / BK;
  src->im2col = cs.r != 1 || cs.s != 1 || cs.stride != 1 || cs.pad != 0;
  src->stride = cs.stride;
  src->pad = cs.pad;
  src->fd_img = make_fastdiv((uint32_t)(cs.oh * cs.ow));
  src->fd_ow = make_fastdiv((uint32_t)cs.ow);
  src->fd_cblocks = make_fastdiv((uint32_t)(cs.cin / BK));
  src->fd_s = make_fastdiv((uint32_t)cs.s);
  src->fd_rows = make_fastdiv(srpc_conv_rows_innermost(cs) ? (uint32_t)cs.r : 1u);
  cudaError_t e = src->im2col ? srpc_tensor_map_im2col(ta, in.a, cs.n, cs.h, cs.w, cs.cin, cs.r, cs.s, cs.stride, cs.pad, rows_per_cta)
                              : srpc_tensor_map_2d(ta, in.a, (uint64_t)cs.cin, (uint64_t)M, (uint64_t)cs.cin * 2, BK, (uint32_t)rows_per_cta);
  *ta2 = *ta;
  if (e != cudaSuccess || !cs.in2) return e;
  src->im2col2 = cs.stride2 != 1;
  src->stride2 = cs.stride2;
  return src->im2col2 ? srpc_tensor_map_im2col(ta2, cs.in2, cs.n, cs.h2, cs.w2, cs.cin2, 1, 1, cs.stride2, 0, rows_per_cta)
                      : srpc_tensor_map_2d(ta2, cs.in2, (uint64_t)cs.cin2, (uint64_t)M, (uint64_t)cs.cin2 * 2, BK, (uint32_t)rows_per_cta);
}

template <int BN, int RPC>
cudaError_t launch_2sm(const AInput& in, const void* B, int ldb, int M, int N, int K, const GemmEpilogue& ep, uint32_t* status,
                       cudaStream_t stream) {
  using C = Cfg<BN, RPC, false>;
  int max_clusters = 0;
  cudaError_t e = max_clusters_2sm<BN, RPC, false>(&max_clusters);
  if (e != cudaSuccess) return e;
  CUtensorMap ta, tb, to, ta2;
  ASource src;
  e = a_maps(in, M, K, RPC, &src, &ta, &ta2);
  if (e != cudaSuccess) return e;
  e = srpc_tensor_map_2d(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, BK, BN / 2);
  if (e != cudaSuccess) return e;
  e = srpc_tensor_map_2d(&to, ep.out, (uint64_t)N, (uint64_t)M, (uint64_t)ep.ldo * 2, 32, 32);
  if (e != cudaSuccess) return e;
  TileOrder o;
  order_tiles(&o, M, N, 2 * RPC, BN, std::min(max_clusters, srpc_gemm_grid_sms() / 2), row_blocks_per_group(N, K));
  o.m_rot2 = 0;
  o.reverse = K > N;
  o.late_trigger = srpc_gemm_reserved_sms() > 0;
  return launch_pdl(gemm_2sm_kernel<BN, RPC, false>, dim3(2 * o.clusters), dim3(C::THREADS), C::SMEM_BYTES, stream, ta, tb, to, ta2, M,
                    N, K, o, src, ep, status, TpArg<false>{});
}

cudaError_t launch_shape(int bn, int rows, const AInput& in, const void* B, int ldb, int M, int N, int K, const GemmEpilogue& ep,
                         uint32_t* status, cudaStream_t stream) {
  if (rows == 256) {
    if (bn == 256) return launch_2sm<256, 128>(in, B, ldb, M, N, K, ep, status, stream);
    if (bn == 192) return launch_2sm<192, 128>(in, B, ldb, M, N, K, ep, status, stream);
    if (bn == 128) return launch_2sm<128, 128>(in, B, ldb, M, N, K, ep, status, stream);
    if (bn == 64) return launch_2sm<64, 128>(in, B, ldb, M, N, K, ep, status, stream);
  } else if (rows == 128) {
    if (bn == 128) return launch_2sm<128, 64>(in, B, ldb, M, N, K, ep, status, stream);
    if (bn == 64) return launch_2sm<64, 64>(in, B, ldb, M, N, K, ep, status, stream);
  }
  return cudaErrorInvalidValue;
}

// Tensor-parallel launch: `tp` arrives with mblocks_per_rank / mblock_bytes filled in and an even n_copy.
template <int BN>
cudaError_t launch_2sm_tp(const void* A, int lda, const void* B, int ldb, int M, int N, int K, const GemmEpilogue& ep,
                          TpParams tp, uint32_t* status, cudaStream_t stream) {
  using C = Cfg<BN, BM, true>;
  static_assert(C::SMEM_BYTES >= tpdev::COPY_SLOTS * tpdev::COPY_CHUNK, "the copier's ring lives in the operand stages");
  int max_clusters = 0;
  cudaError_t e = max_clusters_2sm<BN, BM, true>(&max_clusters);
  if (e != cudaSuccess) return e;
  max_clusters = std::min(max_clusters, srpc_gemm_grid_sms() / 2);
  const int copy_clusters = tp.n_copy / 2;
  if (max_clusters - copy_clusters < 1) return cudaErrorInvalidValue;
  CUtensorMap ta, tb, to;
  e = srpc_tensor_map_2d(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, BM);
  if (e != cudaSuccess) return e;
  e = srpc_tensor_map_2d(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, BK, BN / 2);
  if (e != cudaSuccess) return e;
  if (!tp.rs) {
    e = srpc_tensor_map_2d(&to, ep.out, (uint64_t)N, (uint64_t)M, (uint64_t)ep.ldo * 2, 32, 32);
    if (e != cudaSuccess) return e;
  } else {
    to = ta;  // never used: the epilogue stores to the owners' slots
  }
  const int m2_per_rank = tp.mblocks_per_rank / 2;
  int group_m = 1;
  for (int g = 2; g <= 4; g++)
    if (m2_per_rank % g == 0) group_m = g;  // groups never straddle two ranks' rows
  TileOrder o;
  order_tiles(&o, M, N, 2 * BM, BN, max_clusters - copy_clusters, group_m);
  o.late_trigger = 0;
  o.reverse = 0;
  // all-gather: own rows first (they are here already); reduce-scatter: own rows last (the peers' cross NVLink)
  o.m_rot2 = (tp.rs ? (tp.rank + 1) % tp.tp : tp.rank) * m2_per_rank;
  tp.tiles_per_owner = tp.mblocks_per_rank * o.tiles_n;
  gemm_2sm_kernel<BN, BM, true><<<2 * (o.clusters + copy_clusters), C::THREADS, C::SMEM_BYTES, stream>>>(
      ta, tb, to, ta, M, N, K, o, matrix_source((K + BK - 1) / BK), ep, status, tp);
  return cudaGetLastError();
}

}  // namespace

int srpc_gemm2_trace_read(unsigned long long* out, int n) {
#ifdef SRPC_GEMM_TRACE
  if (n > 16) n = 16;
  if (cudaMemcpyFromSymbol(out, g_gemm2_trace, n * sizeof(unsigned long long)) != cudaSuccess) return 0;
  return n;
#else
  (void)out;
  (void)n;
  return 0;
#endif
}

bool srpc_gemm_2sm_eligible(int K, const GemmEpilogue& ep) {
  static const int allow = [] { const char* e = getenv("SPLITRPC_GEMM_2SM"); return e ? atoi(e) : 1; }();
  if (!allow || ep.out_fp32 || (ep.ldo % 8) || ((uintptr_t)ep.out & 15)) return false;
  if (ep.bias && ((uintptr_t)ep.bias & 15)) return false;
  return K >= 64;
}

cudaError_t srpc_gemm_bf16_2sm(const void* A, int lda, const void* B, int ldb, int M, int N, int K, int bn, int rows,
                               const GemmEpilogue& ep, uint32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return cudaErrorInvalidValue;
  if ((lda % 8) || (ldb % 8) || (K % 8) || ((uintptr_t)A & 15) || ((uintptr_t)B & 15)) return cudaErrorInvalidValue;
  if (!srpc_gemm_2sm_eligible(K, ep)) return cudaErrorInvalidValue;
  AInput in;
  in.a = A;
  in.lda = lda;
  return launch_shape(bn, rows, in, B, ldb, M, N, K, ep, status, stream);
}

// Dense inputs only: no window that overlaps its neighbours, no request ring; corners and steps within what an im2col tensor map holds.
bool srpc_conv_2sm_eligible(const ConvShape& cs, const GemmEpilogue& ep) {
  if (cs.in_stub || cs.in_pix_stride || cs.in_row_stride || cs.in_img_stride || (cs.cin % BK) || (cs.in2 && (cs.cin2 % BK))) return false;
  if (cs.stride < 1 || cs.stride > 8 || cs.pad < 0 || cs.pad > 127 || cs.r < 1 || cs.s < 1 || cs.r > 128 || cs.s > 128) return false;
  if (cs.in2 && (cs.stride2 < 1 || cs.stride2 > 8)) return false;
  if (cs.oh != (cs.h + 2 * cs.pad - cs.r) / cs.stride + 1 || cs.ow != (cs.w + 2 * cs.pad - cs.s) / cs.stride + 1) return false;
  return srpc_gemm_2sm_eligible(cs.r * cs.s * cs.cin, ep);
}

cudaError_t srpc_conv_bf16_2sm(const void* input, const void* weight, const ConvShape& cs, int bn, int rows, const GemmEpilogue& ep,
                               uint32_t* status, cudaStream_t stream) {
  if (!srpc_conv_2sm_eligible(cs, ep) || cs.n <= 0 || cs.cout <= 0) return cudaErrorInvalidValue;
  AInput in;
  in.a = input;
  in.cs = &cs;
  const int K = cs.r * cs.s * cs.cin + (cs.in2 ? cs.cin2 : 0);
  return launch_shape(bn, rows, in, weight, K, cs.n * cs.oh * cs.ow, cs.cout, K, ep, status, stream);
}

// Tensor-parallel entry point (see gemm_tp.h).  Takes the shapes where a rank's rows are whole 256-row pair tiles.
bool srpc_gemm_tp_2sm_eligible(int M, int N, int K, const GemmEpilogue& ep, const TpParams& tp) {
  static const int allow = [] { const char* e = getenv("SPLITRPC_TP_2SM"); return e ? atoi(e) : 1; }();
  if (!allow || tp.tp < 1 || N < 128 || (N % 8) || K < 64 || ep.out_fp32 || (ep.ldo % 8)) return false;
  if (ep.bias && ((uintptr_t)ep.bias & 15)) return false;
  if (!tp.rs && ((uintptr_t)ep.out & 15)) return false;
  return M % (2 * BM * tp.tp) == 0;
}

cudaError_t srpc_gemm_tp_2sm(const void* A, int lda, const void* B, int ldb, int M, int N, int K, const GemmEpilogue& ep,
                             const TpParams& tp_in, uint32_t* status, cudaStream_t stream) {
  if (!srpc_gemm_tp_2sm_eligible(M, N, K, ep, tp_in)) return cudaErrorInvalidValue;
  TpParams tp = tp_in;
  tp.mblocks_per_rank = (M / BM) / tp.tp;
  tp.m_rot = 0;
  tp.mblock_bytes = (size_t)BM * lda * 2;
  // a copier takes whole 128-row blocks: more copiers than remote blocks would idle on SMs the GEMM could use
  tp.n_copy = tp.mblock_ready ? (std::min(tp.n_copy, (tp.tp - 1) * tp.mblocks_per_rank) + 1) & ~1 : 0;
  if (tp.rs)
    for (int o = 0; o < tp.tp; o++)
      if ((uintptr_t)tp.dst[o] & 15) return cudaErrorInvalidValue;
  const int bn = (N % 256 == 0) ? 256 : ((N % 192 == 0) ? 192 : (N % 128 == 0 ? 128 : (N >= 1024 ? 256 : 128)));
  if (bn == 256) return launch_2sm_tp<256>(A, lda, B, ldb, M, N, K, ep, tp, status, stream);
  if (bn == 192) return launch_2sm_tp<192>(A, lda, B, ldb, M, N, K, ep, tp, status, stream);
  return launch_2sm_tp<128>(A, lda, B, ldb, M, N, K, ep, tp, status, stream);
}

cudaError_t srpc_gemm_tp_2sm_set_wait_ns(uint64_t ns) { return tpdev::set_wait_ns_here(ns); }

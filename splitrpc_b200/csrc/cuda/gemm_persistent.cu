// Persistent tcgen05 GEMM / convolution kernel on single SMs, and the choice between it and CTA pairs.
//
//   D[M,N] = act(A[M,K] . B[N,K]^T + bias + residual)          (GEMM mode)
//   out = act(conv(in NHWC, filter [Cout][R][S][Cin]) + bias + residual)   (convolution mode)
//
// One CTA per SM loops over output tiles (128 x BN).  Warp roles:
//   warp 0 and the last warp   walk the schedule as one; an elected lane of each
//            issues the TMA loads of every second k-block of this CTA's tiles,
//            running ahead through a STAGES-deep shared-memory ring that is not
//            drained at tile boundaries;
//   warp 1   walks the schedule as one and waits; one elected lane issues
//            tcgen05.mma into one of ACC TMEM accumulators (BN columns each), so
//            tile i+1 accumulates while tile i is being written out;
//   warps from 2 on (8, 12 or 16 of them, two to four per TMEM lane quarter, see
//            Threads) read the accumulator with tcgen05.ld, release it at once,
//            apply bias / residual (prefetched before the accumulator is ready) /
//            activation and stage the bf16 tile in one of OB 128-byte-swizzled
//            shared-memory buffers;
//   the warp after them hands finished tiles to TMA stores (full-line coalesced
//            writes, bounds clipped by the tensor map) and prefetches residual tiles.
// In convolution mode the A operand needs no im2col and no gather: a tile is a
// PW x PH x PN patch of output pixels, and the rows for filter tap (fr, fs) are
// one 4-D TMA box over the NHWC input shifted by the tap offset, with element
// strides equal to the convolution stride; out-of-image coordinates are
// zero-filled by the TMA unit, which is exactly the padding.  Dense inputs go
// to CTA pairs (gemm_2sm.cu); this form has the inputs with pixel strides or in
// a request ring that stem_conv.cu does not take, and every input when
// SPLITRPC_GEMM_2SM=0 turns pairs off.
// All operands live in this GPU's memory; no load uses multicast.  Every wait
// is bounded; on a timeout the kernel records an error code, stops issuing work,
// frees its tensor memory and returns.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <unordered_map>

#include "fast_div.h"
#include "gemm_tcgen05.h"
#include "pdl_launch.h"
#include "ptx.cuh"
#include "per_device.h"

namespace {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
// Epilogue threads of the 128-wide tile: 512 (four warps per TMEM lane quarter, 32 columns each) measured 2-4 %
// faster than 256 on the memory-bound shapes once the TMA stores had moved to their own warp.
#ifndef SRPC_EPI128
#define SRPC_EPI128 512
#endif
// Output staging buffers per CTA.  A TMA store holds its buffer until the write has drained, which takes a few
// microseconds under load; with too few buffers the epilogue stalls on them and the store stream, not DRAM, sets
// the pace of memory-bound shapes.
constexpr int OUT_BUFS = 3;
constexpr int MAX_OUT_BUFS = 4;
// Width of the output patch of convolutions with row-tap reuse: an image row inside the box is one swizzle atom.
constexpr int REUSE_PW = 8;
// How many tiles ahead the residual tile is loaded (see TileParams::res_tma).
constexpr int RES_DIST = 2;
// warp 0 TMA, warp 1 MMA, then two to four epilogue warps per TMEM lane quarter (they share the tile's columns)
template <int BN>
struct Threads {
  // BN = 256 / 192: four / three warps per quarter, 64 columns each
  static constexpr int EPI = BN == 256 ? 512 : (BN == 192 ? 384 : (BN == 128 ? SRPC_EPI128 : 256));
  static constexpr int TOTAL = 64 + EPI + 64;  // + the store warp, the second producer warp
};

struct TileParams {
  int mode;          // 0 GEMM, 1 convolution
  int M, N, K;       // GEMM view (M = rows, N = columns)
  int num_kb;
  int tiles_m, tiles_n;
  // convolution
  int pw, ph, pn;            // output patch of one tile
  int tiles_w, tiles_h;      // tiles along W and H (tiles_m = tiles_w * tiles_h * tiles_img)
  int oh, ow, nimg;
  int r, s, cblocks, stride, pad;
  uint32_t a_box_bytes;      // bytes one A box writes
  int rows_used;             // pw * ph * pn
  // B-stationary schedule (few k-blocks): every CTA keeps one column block for its whole life, loads that B panel into
  // shared memory once and streams only A.  Without it every tile re-reads the same few KB of weights from L2 and the
  // handful of L2 lines that hold them becomes the bottleneck of the whole GPU.
  int b_stationary;
  int ctas_per_n;            // CTAs that share one column block (grid = ctas_per_n * tiles_n)
  // Residual through TMA: the residual tile of a later tile is loaded into that tile's output staging buffer while
  // earlier tiles are still in their epilogue; the epilogue then adds the accumulator to it in place.  Plain loads
  // of the residual from the epilogue threads leave each of them waiting a full DRAM round trip per tile.
  int res_tma;
  // Row-tap reuse (stride-1 convolutions, patch width a multiple of 8): one A box per (filter column, channel block)
  // holds the patch rows with their halo (ph + r - 1 image rows), and the r filter rows are r groups of MMAs whose A
  // descriptors start fr * pw rows further into that box: a third of the loads (and of the round trips that pace a
  // short-tile k loop) for a 3 x 3 filter.  num_kb then counts load groups (s * cblocks); panel_kb counts all k-blocks.
  int reuse;
  int panel_kb;
  FastDiv fd_tiles_n, fd_group, fd_tiles_w, fd_tiles_h, fd_cblocks, fd_s;  // filled in by launch()
  // Input that lives in a request ring (convolution mode): the tensor map covers the whole ring, one "image" per slot,
  // and the batch starts at the slot that the app stub's request pointer names when the kernel runs, so one captured
  // graph serves every ring position.  in_stub == nullptr: the input starts at image 0.
  const void* in_stub;
  unsigned long long in_ring_base;
  unsigned int in_slot_bytes;
  int late_trigger;  // the next kernel starts behind this CTA's last load only (pdl_launch.h); filled in by launch()
  // two-input 1x1 convolution: k-blocks from kb_split on come from the second input (pixel stride2, no padding)
  int kb_split, stride2;
};

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* smem_src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(m),
               "r"(ptx::smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}

// Optional phase time stamps of block 0 (build with -DSRPC_GEMM_TRACE): where a short kernel spends its time.
#ifdef SRPC_GEMM_TRACE
__device__ unsigned long long g_gemm_trace[16];
#define GEMM_TRACE(slot)                                                         \
  do {                                                                           \
    if (blockIdx.x == 0) g_gemm_trace[slot] = ptx::globaltimer_ns();             \
  } while (0)
#else
#define GEMM_TRACE(slot) ((void)0)
#endif

struct TileCoord {
  int m_idx, n_idx;
  int w0, h0, img0;  // convolution patch origin (output pixels)
};

// j-th tile of this CTA; false when the CTA has no more tiles.
__device__ __forceinline__ bool get_tile(const TileParams& p, int j, TileCoord* out) {
  TileCoord t;
  if (p.b_stationary) {
    const uint32_t q = fdiv(p.fd_tiles_n, blockIdx.x);
    t.n_idx = (int)(blockIdx.x - q * (uint32_t)p.tiles_n);
    t.m_idx = (int)q + j * p.ctas_per_n;
    if (t.m_idx >= p.tiles_m) return false;
  } else {
    const int tile = (int)blockIdx.x + j * (int)gridDim.x;
    if (tile >= p.tiles_m * p.tiles_n) return false;
    // Grouped order: the ~148 tiles in flight at any time cover GROUP_M row blocks x ~18 column blocks, so the A and
    // B blocks they share are read from DRAM once and then hit in L2.
    constexpr int GROUP_M = 8;
    const int per_group = GROUP_M * p.tiles_n;
    const int g = (int)fdiv(p.fd_group, (uint32_t)tile), in_g = tile - g * per_group;
    const int m_first = g * GROUP_M;
    const int gm = (p.tiles_m - m_first) < GROUP_M ? (p.tiles_m - m_first) : GROUP_M;
    if (gm == GROUP_M) {
      t.m_idx = m_first + (in_g & (GROUP_M - 1));
      t.n_idx = in_g >> 3;
    } else {  // last, shorter group
      t.m_idx = m_first + in_g % gm;
      t.n_idx = in_g / gm;
    }
  }
  t.w0 = t.h0 = t.img0 = 0;
  if (p.mode == 1) {
    const int rest = (int)fdiv(p.fd_tiles_w, (uint32_t)t.m_idx);
    const int tw = t.m_idx - rest * p.tiles_w;
    const int ti = (int)fdiv(p.fd_tiles_h, (uint32_t)rest);
    const int th = rest - ti * p.tiles_h;
    t.w0 = tw * p.pw;
    t.h0 = th * p.ph;
    t.img0 = ti * p.pn;
  }
  *out = t;
  return true;
}

template <int BN, int STAGES, int OB>
__global__ void __launch_bounds__(Threads<BN>::TOTAL, 1)
gemm_conv_persistent(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ CUtensorMap tmap_res, TileParams p,
                     GemmEpilogue ep, int use_tma_store, uint32_t* status) {
  constexpr int A_BYTES = BM * BK * 2;
  constexpr int B_BYTES = BN * BK * 2;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int OUT_HALF_BYTES = BM * 128;       // 128 rows x 64 bf16 columns
  constexpr int OUT_BYTES = (BN / 64) * OUT_HALF_BYTES;
  // No slack for manual alignment: the widest configuration then leaves 2 KB of the SM's shared memory, which is what
  // one small block of another stream (the scatter-gather kernel) needs to share the SM; a block that takes all of
  // it keeps every other block off its SM.
  extern __shared__ __align__(1024) uint8_t smem[];
  const bool layout_ok = (ptx::smem_u32(smem) & 1023u) == 0;
  uint8_t* stage_out = smem + (size_t)STAGES * STAGE_BYTES;
  constexpr int MAX_STAGES = 8;
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t empty_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t bpanel_bar;
  // Streaming: STAGES stages of {A tile, B tile}.  B-stationary: the B panel (num_kb tiles) first, then a ring of A tiles.
  const int panel_bytes = p.b_stationary ? p.panel_kb * B_BYTES : 0;
  const int b_per_stage = p.b_stationary ? 0 : (p.reuse ? p.r : 1);  // B tiles that travel with every A box
  const int a_stride = A_BYTES + b_per_stage * B_BYTES;
  int nst_calc = (STAGES * STAGE_BYTES - panel_bytes) / a_stride;
  const int nst = nst_calc > MAX_STAGES ? MAX_STAGES : nst_calc;
  uint8_t* a_ring = smem + panel_bytes;
  // Four TMEM accumulators: up to four tiles can be between "MMA issued" and "accumulator read back", which hides
  // the commit -> wake-up -> tcgen05.ld -> release round trip of short (few k-block) tiles.
  constexpr int ACC = BN >= 192 ? 2 : 4;
  constexpr int ACC_LOG2 = BN >= 192 ? 1 : 2;
  constexpr int ACC_STRIDE = BN == 192 ? 256 : BN;  // TMEM columns between accumulators (allocation is a power of two)
  static_assert(OB >= 1 && OB <= MAX_OUT_BUFS, "output staging buffers");
  __shared__ __align__(8) uint64_t tmem_full_bar[ACC];
  __shared__ __align__(8) uint64_t tmem_empty_bar[ACC];
  __shared__ __align__(8) uint64_t res_full_bar[MAX_OUT_BUFS];
  // Staging buffers: the epilogue warps announce a finished tile on out_full, the store warp's thread issues the TMA
  // stores (and the next residual loads) and hands the buffer back on out_empty once the store has read it.  The
  // epilogue warps never wait for a TMA instruction to issue: that took 0.6 - 0.7 us per tile on their critical path.
  __shared__ __align__(8) uint64_t out_full_bar[MAX_OUT_BUFS];
  __shared__ __align__(8) uint64_t out_empty_bar[MAX_OUT_BUFS];
  __shared__ uint32_t tmem_base_smem;
  __shared__ uint32_t s_error;
  // Bias of the current tile's columns, double-buffered over consecutive tiles: fetched while the accumulator is still
  // being computed, then read as broadcasts (a global load per chunk would sit on the epilogue's critical path).
  __shared__ __align__(16) float s_bias[2][BN];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    GEMM_TRACE(0);
    ptx::mbar_init(&bpanel_bar, 1);
    for (int s = 0; s < MAX_STAGES; s++) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < ACC; a++) {
      ptx::mbar_init(&tmem_full_bar[a], 1);
      ptx::mbar_init(&tmem_empty_bar[a], Threads<BN>::EPI / 32);  // one arrival per epilogue warp
    }
    for (int b = 0; b < MAX_OUT_BUFS; b++) {
      ptx::mbar_init(&res_full_bar[b], 1);
      ptx::mbar_init(&out_full_bar[b], Threads<BN>::EPI / 32);
      ptx::mbar_init(&out_empty_bar[b], 1);
    }
    ptx::fence_mbar_init();
    s_error = layout_ok ? 0u : (uint32_t)GEMM_ERR_PRODUCER_WAIT;
    ptx::prefetch_tmap(&tmap_a);
    ptx::prefetch_tmap(&tmap_b);
    if (use_tma_store) ptx::prefetch_tmap(&tmap_out);
    if (p.res_tma) ptx::prefetch_tmap(&tmap_res);
  }
  // TMA producers: warp 0 and the last warp take the k-blocks of this CTA's schedule in turn (even ones, odd ones).  Each walks
  // the schedule as one and an elected lane issues, so that the operands of the loads stay in uniform registers: an iteration
  // (wait for the stage, post the byte count, two loads) takes 200 ns this way and 240 ns in one lane's branch, and a k-block of
  // the narrow tiles is consumed in 150 - 250 ns.  One producer instead of two: 258 ns per k-block of a lone 128 x 128 tile.
  // The state lives across two calls: the first fills one (initially free) stage right after the barriers exist,
  // before the block-wide set-up barrier, so that the first operands are already in flight while tensor memory is being
  // allocated; the second runs the rest of the schedule.
  // (A ring of one stage, which the widest load groups of a short filter leave, has one producer.)
  const int producers = nst >= 2 ? 2 : 1;
  const int producer = warp == 0 ? 0 : (warp == Threads<BN>::TOTAL / 32 - 1 && producers == 2 ? 1 : -1);
  int pr_s = producer, pr_kb = producer, pr_j = 0;
  uint32_t pr_ph = 0;
  int img_off = 0;
  TileCoord pr_tc;
  bool pr_more = false;
  const bool pr_elected = producer >= 0 && ptx::elect_one();
  // Moves to the tile that holds k-block pr_kb; false when the schedule is through.
  auto producer_tile = [&]() {
    while (pr_kb >= p.num_kb) {
      pr_kb -= p.num_kb;
      pr_j++;
    }
    return get_tile(p, pr_j, &pr_tc) && __all_sync(0xffffffffu, *(volatile uint32_t*)&s_error == 0);
  };
  const uint32_t b_tx = (uint32_t)(b_per_stage * B_BYTES);
  auto produce_one = [&]() {
    if (!ptx::mbar_wait_warp(&empty_bar[pr_s], pr_ph ^ 1u)) {
      if (pr_elected) atomicExch(&s_error, GEMM_ERR_PRODUCER_WAIT);
      pr_more = false;
      return;
    }
    uint8_t* sa = a_ring + (size_t)pr_s * a_stride;
    uint64_t* full = &full_bar[pr_s];
    if (p.mode == 0) {
      if (pr_elected) {
        ptx::mbar_expect_tx(full, (uint32_t)A_BYTES + b_tx);
        ptx::tma_load_2d(sa, &tmap_a, full, pr_kb * BK, pr_tc.m_idx * BM);
        if (!p.b_stationary) ptx::tma_load_2d(sa + A_BYTES, &tmap_b, full, pr_kb * BK, pr_tc.n_idx * BN);
      }
    } else {
      const int tap = (int)fdiv(p.fd_cblocks, (uint32_t)pr_kb), cb = pr_kb - tap * p.cblocks;
      if (p.reuse) {
        // load group (fs, cb): the box covers filter rows 0 .. r-1 at once
        const int fs = tap;
        if (pr_elected) {
          ptx::mbar_expect_tx(full, p.a_box_bytes + b_tx);
          ptx::tma_load_4d(sa, &tmap_a, full, cb * BK, pr_tc.w0 + fs - p.pad, pr_tc.h0 - p.pad, pr_tc.img0 + img_off);
          if (!p.b_stationary)
            for (int fr = 0; fr < p.r; fr++)
              ptx::tma_load_2d(sa + A_BYTES + fr * B_BYTES, &tmap_b, full, ((fr * p.s + fs) * p.cblocks + cb) * BK, pr_tc.n_idx * BN);
        }
      } else if (pr_elected) {
        ptx::mbar_expect_tx(full, p.a_box_bytes + b_tx);
        if (pr_kb >= p.kb_split) {
          // second input of a two-input 1x1 convolution (its map travels in the residual map's place)
          ptx::tma_load_4d(sa, &tmap_res, full, (pr_kb - p.kb_split) * BK, pr_tc.w0 * p.stride2, pr_tc.h0 * p.stride2, pr_tc.img0);
        } else {
          const int fr = (int)fdiv(p.fd_s, (uint32_t)tap), fs = tap - fr * p.s;
          ptx::tma_load_4d(sa, &tmap_a, full, cb * BK, pr_tc.w0 * p.stride + fs - p.pad, pr_tc.h0 * p.stride + fr - p.pad,
                           pr_tc.img0 + img_off);
        }
        if (!p.b_stationary) ptx::tma_load_2d(sa + A_BYTES, &tmap_b, full, pr_kb * BK, pr_tc.n_idx * BN);
      }
    }
    if (pr_j == 0 && pr_kb == 0 && lane == 0) GEMM_TRACE(2);
    pr_kb += producers;
    pr_s += producers;
    if (pr_s >= nst) {
      pr_s -= nst;
      pr_ph ^= 1u;
    }
  };
  if (producer == 0) {
    pr_more = layout_ok && producer_tile();
    ptx::grid_dep_wait();  // set-up above overlaps the kernel before; its results are read below
    if (p.in_stub)
      img_off = (int)((*reinterpret_cast<const unsigned long long*>(p.in_stub) - p.in_ring_base) / p.in_slot_bytes);
    if (pr_more && p.b_stationary && pr_elected) {
      ptx::mbar_expect_tx(&bpanel_bar, (uint32_t)panel_bytes);
      for (int kb = 0; kb < p.panel_kb; kb++)
        ptx::tma_load_2d(smem + (size_t)kb * B_BYTES, &tmap_b, &bpanel_bar, kb * BK, pr_tc.n_idx * BN);
    }
    if (pr_more) produce_one();
  }
  if (warp == 1) {
    ptx::tmem_alloc(&tmem_base_smem, ACC * ACC_STRIDE);
    ptx::tmem_relinquish();
    if (!p.late_trigger) ptx::grid_dep_launch();  // after the allocation, see pdl_launch.h
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::grid_dep_wait();
  ptx::tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  if (threadIdx.x == 0) GEMM_TRACE(1);

  if (producer >= 0) {
    if (producer == 1) {
      if (p.in_stub)
        img_off = (int)((*reinterpret_cast<const unsigned long long*>(p.in_stub) - p.in_ring_base) / p.in_slot_bytes);
      pr_more = true;
    }
    // the rest of this producer's k-blocks, paced by the MMA warp through the empty barriers
    if (layout_ok && pr_more)
      while (producer_tile()) {
        const int j = pr_j;
        while (pr_more && pr_j == j && pr_kb < p.num_kb) produce_one();
        if (!pr_more) break;
      }
    if (producer == 0 && p.late_trigger) {
      __syncwarp();
      ptx::grid_dep_launch();
    }
  } else if (warp == 1) {
    // The whole warp walks the schedule and waits together; one elected lane issues.  Every value that a tcgen05
    // instruction takes lives in uniform registers then; with the loop inside the elected lane's branch each of them was
    // moved there one by one, and issuing a k-block (four MMAs) took 260 ns whatever the tile's width, up to three times
    // the tensor pipe's own time.  No tcgen05 fence per k-block: the operands arrive through TMA and an mbarrier, no
    // tcgen05 instruction of another thread has to be ordered before the MMAs here.
    const bool elected = ptx::elect_one();
    const uint32_t idesc = ptx::umma_idesc_bf16(BM, BN);
    const uint32_t ring_lo = ptx::umma_desc_lo(ptx::smem_u32(a_ring)), stride_lo = (uint32_t)a_stride >> 4;
    const uint32_t panel_lo = ptx::umma_desc_lo(ptx::smem_u32(smem));
    constexpr uint32_t K_LO = UMMA_K * 2 / 16;  // descriptor step from one 16-deep slice to the next
    constexpr uint32_t REUSE_ROW_LO = REUSE_PW * 128 / 16;  // to the next image row inside a reused box
    const uint32_t b_row_lo = (uint32_t)(p.b_stationary ? p.num_kb * B_BYTES : B_BYTES) / 16;  // to the next filter row
    uint32_t local = 0;
    int s = 0;
    uint32_t ph = 0;
    TileCoord tc;
    bool ok = true;
    if (p.b_stationary && get_tile(p, 0, &tc)) ok = ptx::mbar_wait_warp(&bpanel_bar, 0);
    for (int j = 0; ok && get_tile(p, j, &tc); j++, local++) {
      const uint32_t acc = local & (ACC - 1);
      ok = ptx::mbar_wait_warp(&tmem_empty_bar[acc], ((local >> ACC_LOG2) & 1u) ^ 1u);
      if (!ok) break;
      ptx::tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * ACC_STRIDE;
      for (int kb = 0; kb < p.num_kb; kb++) {
        ok = ptx::mbar_wait_warp(&full_bar[s], ph);
        if (!ok) break;
        if (j == 0 && kb == 0 && lane == 0) GEMM_TRACE(3);
        const uint32_t sa = ring_lo + (uint32_t)s * stride_lo;
        if (p.reuse) {
          // r filter rows: A a patch row further into the box, B the next filter row of this (filter column, channel block).
          // One unrolled run of MMAs per load group: issuing them was what a 64-wide tile took its time for (56 ns per MMA, 27 now;
          // 64 images with pairs turned off: 28 x 28 x 128 22.2 -> 20.3 us, 14 x 14 x 256 21.6 -> 18.7; pairs 13.9 and 15.6).
          const uint32_t sb = p.b_stationary ? panel_lo + (uint32_t)kb * (B_BYTES / 16) : sa + A_BYTES / 16;
          if (elected) {
            if (p.r == 3) {
#pragma unroll
              for (int fr = 0; fr < 3; fr++)
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; k++)
                  ptx::umma_bf16(d_tmem, ptx::umma_desc_join(sa + fr * REUSE_ROW_LO + k * K_LO),
                                 ptx::umma_desc_join(sb + fr * b_row_lo + k * K_LO), idesc, (kb | fr | k) != 0 ? 1u : 0u);
            } else {
              for (int fr = 0; fr < p.r; fr++)
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; k++)
                  ptx::umma_bf16(d_tmem, ptx::umma_desc_join(sa + fr * REUSE_ROW_LO + k * K_LO),
                                 ptx::umma_desc_join(sb + fr * b_row_lo + k * K_LO), idesc, (kb | fr | k) != 0 ? 1u : 0u);
            }
          }
        } else {
          const uint32_t sb = p.b_stationary ? panel_lo + (uint32_t)kb * (B_BYTES / 16) : sa + A_BYTES / 16;
          if (elected) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; k++)
              ptx::umma_bf16(d_tmem, ptx::umma_desc_join(sa + k * K_LO), ptx::umma_desc_join(sb + k * K_LO), idesc,
                             (kb | k) != 0 ? 1u : 0u);
          }
        }
        if (elected) ptx::umma_commit(&empty_bar[s]);
        if (++s == nst) {
          s = 0;
          ph ^= 1u;
        }
      }
      if (!ok) break;
      if (elected) ptx::umma_commit(&tmem_full_bar[acc]);
      if (j == 0 && lane == 0) GEMM_TRACE(4);
      ok = *(volatile uint32_t*)&s_error == 0;
      ok = __all_sync(0xffffffffu, ok);
    }
    if (!ok && elected) atomicCAS(&s_error, 0u, (uint32_t)GEMM_ERR_MMA_WAIT);
  } else if (warp < 2 + Threads<BN>::EPI / 32) {
    // ---------------- epilogue warps: those of one TMEM lane quarter (w, w+4, ...) split the columns
    constexpr int CPW = BN / (Threads<BN>::EPI / 128);  // columns per warp
    constexpr bool LEAN = BN >= 192 || Threads<BN>::EPI > 256;     // 14-18 warps per CTA: keep the accumulator in registers one chunk at a time
    constexpr int NCH = CPW / 32;        // 32-column chunks per warp
    constexpr int EPI_THREADS = Threads<BN>::EPI;
    const int warp_q = warp & 3;
    const int chalf = (warp - 2) >> 2;   // which 32-column group of the tile this warp takes
    const int row = warp_q * 32 + lane;  // row of the tile this thread owns
    const int et = threadIdx.x - 64;     // 0..255 among the epilogue threads
    const bool res_tma = OB > RES_DIST && p.res_tma != 0;
    const bool vec_res = !res_tma && ep.residual && ((ep.ldr & 7) == 0) && (((uintptr_t)ep.residual & 15) == 0);
    uint32_t local = 0;
    TileCoord tc;
    // Position of this thread's row inside a convolution patch (the same for every tile).
    int pw_i = 0, ph_i = 0, pn_i = 0;
    if (p.mode == 1) {
      const int rest = row / p.pw;
      pw_i = row - rest * p.pw;
      pn_i = rest / p.ph;
      ph_i = rest - pn_i * p.ph;
    }
    for (int j = 0; get_tile(p, j, &tc); j++, local++) {
      const uint32_t acc = local & (ACC - 1);
      // Where this thread's row lives in the output.
      bool row_ok;
      size_t row_off;  // pixel / row index (leading dimension not yet applied)
      if (p.mode == 0) {
        const int m = tc.m_idx * BM + row;
        row_ok = m < p.M;
        row_off = (size_t)m;
      } else {
        const int x = tc.w0 + pw_i, y = tc.h0 + ph_i, img = tc.img0 + pn_i;
        row_ok = row < p.rows_used && x < p.ow && y < p.oh && img < p.nimg;
        row_off = ((size_t)img * p.oh + y) * p.ow + x;
      }
      const int n0 = tc.n_idx * BN;
      const int cbase = chalf * CPW;  // first tile column of this warp
      // Residual rows are fetched before the accumulator is awaited, so their latency hides behind the MMAs.
      uint4 resq[LEAN ? 1 : CPW / 8];
      const bool res_vec_tile = vec_res && row_ok && (n0 + cbase + CPW <= p.N);
      if (!LEAN && res_vec_tile) {
        const __nv_bfloat16* rp = ep.residual + row_off * ep.ldr + n0 + cbase;
#pragma unroll
        for (int j = 0; j < CPW / 8; j++) resq[j] = *(reinterpret_cast<const uint4*>(rp) + j);
      }
      if (j == 5 && et == 0) GEMM_TRACE(10);
      float* bias_s = s_bias[local & 1u];
      if (ep.bias && et < BN) bias_s[et] = (n0 + et < p.N) ? *(ep.bias + n0 + et) : 0.f;
      // One warp waits for the accumulator and the staging buffer, the others for that warp at a hardware barrier: a
      // dozen warps polling the same barrier words keep the shared-memory pipe busy that the producer's and the MMA
      // warp's hand-offs go through.  Its wait is bounded; the vote makes the outcome uniform so that no thread is left
      // alone at a later barrier, and orders the wait and the bias writes before what follows.
      bool mine = true;
      if (warp == 2) {
        mine = (*(volatile uint32_t*)&s_error == 0) && ptx::mbar_wait(&tmem_full_bar[acc], (local >> ACC_LOG2) & 1u);
        // The staging buffer: with a prefetched residual it is ready when the residual has landed (the store warp loads
        // it only into a buffer whose last store has been read); otherwise when the store warp has handed it back.
        if (res_tma && mine) mine = ptx::mbar_wait(&res_full_bar[local % OB], (local / OB) & 1u);
        else if (use_tma_store && mine) mine = ptx::mbar_wait(&out_empty_bar[local % OB], ((local / OB) & 1u) ^ 1u);
      }
      if (!ptx::named_bar_all(2, EPI_THREADS, mine)) {
        if (lane == 0) atomicExch(&s_error, GEMM_ERR_EPILOGUE_WAIT);
        break;
      }
      ptx::tc_fence_after();
      if (j == 0 && et == 0) GEMM_TRACE(5);
      if (j == 5 && et == 0) GEMM_TRACE(11);
      uint32_t r[LEAN ? 32 : CPW];
      const uint32_t t_addr = tmem_base + acc * ACC_STRIDE + ((uint32_t)(warp_q * 32) << 16) + (uint32_t)cbase;
      if (!LEAN) {
#pragma unroll
        for (int ch = 0; ch < NCH; ch++) ptx::tmem_ld_32x32b_x32(t_addr + ch * 32, r + ch * 32);
        ptx::tmem_ld_wait();
        // Accumulator is in registers: give it back to the MMA warp right away.
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&tmem_empty_bar[acc]);
      }
      if (j == 5 && et == 0) GEMM_TRACE(12);
      uint8_t* sbuf = stage_out + (size_t)(local % OB) * OUT_BYTES;
#pragma unroll
      for (int ch = 0; ch < NCH; ch++) {
        const int c = cbase + ch * 32;  // tile column of this chunk
        const int col0 = n0 + c;
        if (LEAN) {
          ptx::tmem_ld_32x32b_x32(t_addr + ch * 32, r);
          ptx::tmem_ld_wait();
          if (ch == NCH - 1) {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&tmem_empty_bar[acc]);
          }
        }
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[(LEAN ? 0 : ch * 32) + j]);
        if (ep.bias) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 b4 = *reinterpret_cast<const float4*>(bias_s + c + j);
            v[j] += b4.x;
            v[j + 1] += b4.y;
            v[j + 2] += b4.z;
            v[j + 3] += b4.w;
          }
        }
        if (res_tma) {
          const uint8_t* half = sbuf + (size_t)(c >> 6) * OUT_HALF_BYTES + (size_t)row * 128;
          const int chunk0 = (c & 63) >> 3;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const uint4 q = *reinterpret_cast<const uint4*>(half + (((chunk0 + j) ^ (row & 7)) << 4));
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
            for (int t = 0; t < 4; t++) {
              float2 f = __bfloat1622float2(h[t]);
              v[j * 8 + 2 * t] += f.x;
              v[j * 8 + 2 * t + 1] += f.y;
            }
          }
        } else if (ep.residual && row_ok && col0 < p.N) {
          if (res_vec_tile) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
              if (LEAN) resq[0] = *(reinterpret_cast<const uint4*>(ep.residual + row_off * ep.ldr + col0) + j);
              const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&resq[LEAN ? 0 : ch * 4 + j]);
#pragma unroll
              for (int t = 0; t < 4; t++) {
                float2 f = __bfloat1622float2(h[t]);
                v[j * 8 + 2 * t] += f.x;
                v[j * 8 + 2 * t + 1] += f.y;
              }
            }
          } else {
            const __nv_bfloat16* rp = ep.residual + row_off * ep.ldr + col0;
            #pragma unroll
            for (int j = 0; j < 32; j++)
              if (col0 + j < p.N) v[j] += __bfloat162float(rp[j]);
          }
        }
        if (ep.act == GEMM_ACT_RELU) {
#pragma unroll
          for (int j = 0; j < 32; j++) v[j] = fmaxf(v[j], 0.f);
        } else if (ep.act == GEMM_ACT_GELU) {
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 g = ptx::gelu_erf_fast2(make_float2(v[j], v[j + 1]));
            v[j] = g.x;
            v[j + 1] = g.y;
          }
        } else if (ep.act == GEMM_ACT_TANH) {
#pragma unroll
          for (int j = 0; j < 32; j++) v[j] = tanhf(v[j]);
        }
        if (use_tma_store) {
          uint8_t* half = sbuf + (size_t)(c >> 6) * OUT_HALF_BYTES + (size_t)row * 128;
          const int chunk0 = (c & 63) >> 3;  // first 16-byte chunk of this 32-column group inside the 128-byte row
#pragma unroll
          for (int j = 0; j < 4; j++) {
            uint4 q;
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
            for (int t = 0; t < 4; t++) h[t] = __floats2bfloat162_rn(v[j * 8 + 2 * t], v[j * 8 + 2 * t + 1]);
            *reinterpret_cast<uint4*>(half + (((chunk0 + j) ^ (row & 7)) << 4)) = q;
          }
        } else if (row_ok && col0 < p.N) {
          if (ep.out_fp32) {
            float* op = reinterpret_cast<float*>(ep.out) + row_off * ep.ldo + col0;
            #pragma unroll
            for (int j = 0; j < 32; j++)
              if (col0 + j < p.N) op[j] = v[j];
          } else {
            __nv_bfloat16* op = reinterpret_cast<__nv_bfloat16*>(ep.out) + row_off * ep.ldo + col0;
            #pragma unroll
            for (int j = 0; j < 32; j++)
              if (col0 + j < p.N) op[j] = __float2bfloat16(v[j]);
          }
        }
      }
      if (j == 5 && et == 0) GEMM_TRACE(13);
      if (use_tma_store) {
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&out_full_bar[local % OB]);
      }
    }
  } else if (warp == 2 + Threads<BN>::EPI / 32 && lane == 0 && use_tma_store) {
    // ---------------- store warp (one thread): TMA stores of finished tiles, residual prefetch, buffer hand-back
    const bool res_tma = OB > RES_DIST && p.res_tma != 0;
    // Loads the residual tile of this CTA's jj-th tile into staging buffer jj % OB (one elected thread).
    auto load_residual = [&](int jj) {
      TileCoord tn;
      if (!get_tile(p, jj, &tn)) return;
      const int b = jj % OB;
      uint8_t* dst = stage_out + (size_t)b * OUT_BYTES;
      int boxes = 0;
      for (int hcol = 0; hcol < BN / 64; hcol++)
        if (tn.n_idx * BN + hcol * 64 < p.N) boxes++;
      ptx::mbar_expect_tx(&res_full_bar[b], (uint32_t)(boxes * OUT_HALF_BYTES));
      for (int hcol = 0; hcol < boxes; hcol++)
        ptx::tma_load_2d(dst + (size_t)hcol * OUT_HALF_BYTES, &tmap_res, &res_full_bar[b], tn.n_idx * BN + hcol * 64,
                         tn.m_idx * BM);
    };
    if (res_tma) {
      for (int jj = 0; jj < RES_DIST; jj++) load_residual(jj);
    }
    uint32_t local = 0;
    TileCoord tc;
    for (int j = 0; get_tile(p, j, &tc) && *(volatile uint32_t*)&s_error == 0; j++, local++) {
      const int b = (int)(local % OB);
      if (!ptx::mbar_wait(&out_full_bar[b], (local / OB) & 1u)) {
        atomicExch(&s_error, GEMM_ERR_EPILOGUE_WAIT);
        break;
      }
      const int n0 = tc.n_idx * BN;
      const uint8_t* sbuf = stage_out + (size_t)b * OUT_BYTES;
#pragma unroll
      for (int hcol = 0; hcol < BN / 64; hcol++) {
        if (n0 + hcol * 64 >= p.N) break;
        const void* src = sbuf + (size_t)hcol * OUT_HALF_BYTES;
        if (p.mode == 0) ptx::tma_store_2d(&tmap_out, src, n0 + hcol * 64, tc.m_idx * BM);
        else tma_store_4d(&tmap_out, src, n0 + hcol * 64, tc.w0, tc.h0, tc.img0);
      }
      ptx::bulk_commit();
      if (j == 0) GEMM_TRACE(6);
      if (res_tma) {
        // The tile RES_DIST ahead takes the buffer of the tile OB - RES_DIST back, so all stores but the last
        // OB - RES_DIST must have been read.
        ptx::bulk_wait_read<(OB > RES_DIST ? OB - RES_DIST : 0)>();
        load_residual(j + RES_DIST);
      } else if (OB == 1) {
        ptx::bulk_wait_read<0>();
        ptx::mbar_arrive(&out_empty_bar[0]);
      } else {
        // all stores but this one have been read: the previous tile's buffer is free again
        ptx::bulk_wait_read<1>();
        if (j >= 1) ptx::mbar_arrive(&out_empty_bar[(local - 1) % OB]);
      }
    }
    GEMM_TRACE(7);
    ptx::bulk_wait_all<0>();
    GEMM_TRACE(8);
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) GEMM_TRACE(9);
  if (s_error != 0) {
    if (threadIdx.x == 0 && status) atomicExch(status, s_error);
    __nanosleep(1000000);  // let loads that are still in flight land before the block leaves
    __syncthreads();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, ACC * ACC_STRIDE);
  }
}

// ------------------------------------------------------------------ host side
struct MapKey {
  const void* ptr;
  uint64_t d[5];
  uint64_t st[4];
  uint32_t box[5];
  uint32_t es[5];
  int rank;
  uint32_t swizzle;
  bool operator==(const MapKey& o) const { return std::memcmp(this, &o, sizeof(MapKey)) == 0; }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    const uint64_t* w = reinterpret_cast<const uint64_t*>(&k);
    size_t h = 1469598103934665603ull;
    for (size_t i = 0; i < sizeof(MapKey) / 8; i++) h = (h ^ w[i]) * 1099511628211ull;
    return h;
  }
};

// Tensor maps are cached: encoding costs microseconds and the same layers run
// for every batch.
template <typename Encode>
cudaError_t cached_map(CUtensorMap* out, const MapKey& k, Encode encode) {
  static std::mutex mu;
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(k);
  if (it != cache.end()) {
    *out = it->second;
    return cudaSuccess;
  }
  const cudaError_t e = encode(out);
  if (e != cudaSuccess) return e;
  if (cache.size() > 4096) cache.clear();
  cache.emplace(k, *out);
  return cudaSuccess;
}

cudaError_t get_map(CUtensorMap* out, const void* ptr, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                    const uint32_t* box, const uint32_t* estr, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  MapKey k;
  std::memset(&k, 0, sizeof(k));
  k.ptr = ptr;
  k.rank = rank;
  k.swizzle = (uint32_t)swizzle;
  for (int i = 0; i < rank; i++) {
    k.d[i] = dims[i];
    k.box[i] = box[i];
    k.es[i] = estr[i];
    if (i + 1 < rank) k.st[i] = strides_bytes[i];
  }
  return cached_map(out, k, [&](CUtensorMap* m) {
    const SrpcDriverApi* d = srpc_driver_api();
    if (!d->TensorMapEncodeTiled) return cudaErrorNotSupported;
    cuuint64_t gd[5], gs[4];
    cuuint32_t bx[5], es[5];
    for (int i = 0; i < rank; i++) {
      gd[i] = dims[i];
      bx[i] = box[i];
      es[i] = estr[i];
      if (i + 1 < rank) gs[i] = strides_bytes[i];
    }
    const CUresult r = d->TensorMapEncodeTiled(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(ptr), gd, gs,
                                               bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
  });
}

// Rows of the box are 128 bytes of shared memory under the 128-byte swizzle and 64 bytes under the 64-byte one.
cudaError_t map_2d(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                   uint32_t box_inner, uint32_t box_outer) {
  uint64_t dims[2] = {inner, outer}, st[1] = {row_stride_bytes};
  uint32_t box[2] = {box_inner, box_outer}, es[2] = {1, 1};
  return get_map(m, ptr, 2, dims, st, box, es, box_inner == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B);
}

// SMs that the persistent kernels size their grids for.  A persistent kernel has one block per SM and a fixed tile
// schedule; if a block of another stream (the scatter-gather kernel that runs beside the model) holds an SM, one of
// this kernel's blocks starts only when another has finished and the whole kernel takes twice as long.  Leaving a
// few SMs out of the grid keeps room for such blocks (srpc_gemm_reserve_sms, or SPLITRPC_GEMM_RESERVE_SMS).
int g_reserve_sms = -1;
int num_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  if (g_reserve_sms < 0) {
    const char* e = getenv("SPLITRPC_GEMM_RESERVE_SMS");
    g_reserve_sms = e ? atoi(e) : 0;
  }
  const int r = g_reserve_sms < n / 2 ? g_reserve_sms : n / 2;
  return n - r;
}

template <int BN, int STAGES, int OB>
cudaError_t launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& to, const CUtensorMap& tr,
                   const TileParams& p_in, const GemmEpilogue& ep, int use_tma_store, uint32_t* status, cudaStream_t st) {
  static PerDeviceFlag attr;
  const int dev = PerDeviceFlag::current();
  const int smem = STAGES * (BM * BK * 2 + BN * BK * 2) + OB * (BN / 64) * BM * 128;
  if (attr.needed(dev)) {
    cudaError_t e = cudaFuncSetAttribute(gemm_conv_persistent<BN, STAGES, OB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    attr.set(dev);
  }
  TileParams p = p_in;
  const int tiles = p.tiles_m * p.tiles_n;
  int grid = std::min(tiles, num_sms());
  p.b_stationary = 0;
  p.ctas_per_n = 0;
  p.fd_tiles_n = make_fastdiv((uint32_t)p.tiles_n);
  p.fd_group = make_fastdiv((uint32_t)(8 * p.tiles_n));  // GROUP_M row blocks x all column blocks (see get_tile)
  p.fd_tiles_w = make_fastdiv((uint32_t)(p.tiles_w > 0 ? p.tiles_w : 1));
  p.fd_tiles_h = make_fastdiv((uint32_t)(p.tiles_h > 0 ? p.tiles_h : 1));
  p.fd_cblocks = make_fastdiv((uint32_t)(p.cblocks > 0 ? p.cblocks : 1));
  p.fd_s = make_fastdiv((uint32_t)(p.s > 0 ? p.s : 1));
  p.late_trigger = srpc_gemm_reserved_sms() > 0;
  static const int allow_bs = [] { const char* e = getenv("SPLITRPC_GEMM_BSTAT"); return e ? atoi(e) : 1; }();
  // The panel may take the ring's memory as long as three A stages remain (a 3x3 convolution over 64 channels keeps its
  // nine 8 KB filter taps resident: otherwise every CTA re-reads the same few L2 lines for every tile).
  const int panel = p.panel_kb * BN * BK * 2, ring = STAGES * (BM * BK * 2 + BN * BK * 2);
  const bool panel_fits = p.mode == 1 ? panel + 3 * BM * BK * 2 <= ring : p.num_kb <= (BN >= 192 ? 2 : 4);
  if (allow_bs && panel_fits && p.tiles_n <= num_sms()) {
    const int per_n = std::min(num_sms() / p.tiles_n, p.tiles_m);
    if (per_n >= 1 && p.tiles_m >= 2 * per_n) {  // at least two tiles per CTA to pay for the panel load
      p.b_stationary = 1;
      p.ctas_per_n = per_n;
      grid = per_n * p.tiles_n;
    }
  }
  return launch_pdl(gemm_conv_persistent<BN, STAGES, OB>, dim3(grid), dim3(Threads<BN>::TOTAL), smem, st, ta, tb, to, tr, p, ep,
                    use_tma_store, status);
}

cudaError_t dispatch(int bn, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& to, const CUtensorMap& tr,
                     const TileParams& p, const GemmEpilogue& ep, int use_tma_store, uint32_t* status, cudaStream_t st) {
  // Long k loops run at (round trip MMA done -> stage free -> TMA -> stage full) / (stages): give them the staging
  // buffers' memory as extra stages.  Short k loops are bound by the output stream and keep three staging buffers.
  static const int allow_deep = [] { const char* e = getenv("SPLITRPC_GEMM_DEEP"); return e ? atoi(e) : 1; }();
  const bool deep = allow_deep && !p.res_tma && p.panel_kb >= 8;
  if (bn == 64) {
    if (deep) return launch<64, 8, 1>(ta, tb, to, tr, p, ep, use_tma_store, status, st);
    return launch<64, 6, OUT_BUFS>(ta, tb, to, tr, p, ep, use_tma_store, status, st);
  }
  if (bn == 256) return launch<256, 3, 1>(ta, tb, to, tr, p, ep, use_tma_store, status, st);
  if (bn == 192) return launch<192, 4, 1>(ta, tb, to, tr, p, ep, use_tma_store, status, st);
  if (deep) return launch<128, 6, 1>(ta, tb, to, tr, p, ep, use_tma_store, status, st);
  return launch<128, 4, OUT_BUFS>(ta, tb, to, tr, p, ep, use_tma_store, status, st);
}

}  // namespace

void srpc_gemm_reserve_sms(int n) { g_reserve_sms = n < 0 ? 0 : n; }
int srpc_gemm_grid_sms() { return num_sms(); }
int srpc_gemm_reserved_sms() {
  (void)num_sms();
  return g_reserve_sms > 0 ? g_reserve_sms : 0;
}

cudaError_t srpc_tensor_map_2d(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                               uint32_t box_inner, uint32_t box_outer) {
  return map_2d(m, ptr, inner, outer, row_stride_bytes, box_inner, box_outer);
}

// Dense NHWC tensor read by an r x s filter: `pixels` output pixels x 64 channels per load, zero outside the image.
cudaError_t srpc_tensor_map_im2col(CUtensorMap* m, const void* ptr, int n, int h, int w, int c, int r, int s, int stride, int pad,
                                   int pixels) {
  MapKey k;
  std::memset(&k, 0, sizeof(k));
  k.ptr = ptr;
  k.rank = 4 | 0x100;  // no tiled map has this rank
  const uint64_t dims[4] = {(uint64_t)c, (uint64_t)w, (uint64_t)h, (uint64_t)n};
  for (int i = 0; i < 4; i++) k.d[i] = dims[i];
  const uint32_t shape[5] = {(uint32_t)r, (uint32_t)s, (uint32_t)stride, (uint32_t)pad, (uint32_t)pixels};
  for (int i = 0; i < 5; i++) k.box[i] = shape[i];
  return cached_map(m, k, [&](CUtensorMap* out) {
    const SrpcDriverApi* d = srpc_driver_api();
    if (!d->TensorMapEncodeIm2col) return cudaErrorNotSupported;
    const cuuint64_t gd[4] = {dims[0], dims[1], dims[2], dims[3]};
    const cuuint64_t gs[3] = {(cuuint64_t)c * 2, (cuuint64_t)w * c * 2, (cuuint64_t)h * w * c * 2};
    // first and last filter position over the image, as offsets from its corners (w, then h)
    const int lower[2] = {-pad, -pad}, upper[2] = {pad - (s - 1), pad - (r - 1)};
    const cuuint32_t es[4] = {1, (cuuint32_t)stride, (cuuint32_t)stride, 1};
    const CUresult e = d->TensorMapEncodeIm2col(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), gd, gs, lower, upper, BK,
                                                (cuuint32_t)pixels, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return e == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
  });
}

int srpc_gemm_trace_read(unsigned long long* out, int n) {
#ifdef SRPC_GEMM_TRACE
  if (n > 16) n = 16;
  if (cudaMemcpyFromSymbol(out, g_gemm_trace, n * sizeof(unsigned long long)) != cudaSuccess) return 0;
  return n;
#else
  (void)out;
  (void)n;
  return 0;
#endif
}

// Tile shape: the one with the lowest estimated time, a launch plus rounds of tiles over the SMs (or SM pairs) x (k-blocks x time
// per k-block + hand-over, more with a residual or GELU).  The figures are a fit to 200 products and convolutions of 49 .. 200704 rows,
// 8 .. 8192 columns and K 64 .. 8192, each measured with every shape.  On 1050 others the choice is within 1.2 % of the best one on average, and
// 15 - 30 % behind where a few rows meet thousands of columns (10 x 4696 x 4720 15.6 us, 128 x 128 tiles 11.7); a fit to those with the
// producers' present loops (128 x 128 tiles 0.095 us per k-block instead of 0.123) makes that 1.0 %, but ResNet-50 888 -> 899 us.
// Pairs win nearly everywhere (us, one-SM against pairs): 128 x 768 x 3072 14.2 against 6.8, 512 x 768 x 768 6.8 and 4.4,
// 4096 x 768 x 768 10.8 and 7.6; the one-SM kernel is left with fp32 and unaligned outputs and with the shapes that stream a
// residual (srpc_gemm_bf16_v2).  The residual of a 256-wide pair tile hides only behind long k loops, except in the first round
// (13144 x 1024 x 768 31.5 us, 192 wide 25.4; 9953 x 1024 x 2048 40.2, 192 wide 41.5).  Every shape sums a result's products in the same order, so that a row does not depend on the
// batch that it is computed in.
struct TileShape {
  int bn, rows;  // columns; rows of a CTA pair, 0: the one-SM kernel (128 rows)
};
static TileShape pick_tile(int M, int N, int num_kb, const GemmEpilogue& ep, bool one_sm, bool pairs) {
  static const int allow256 = [] { const char* e = getenv("SPLITRPC_GEMM_BN256"); return e ? atoi(e) : 1; }();
  static const int allow192 = [] { const char* e = getenv("SPLITRPC_GEMM_BN192"); return e ? atoi(e) : 1; }();
  struct Cand {
    int bn, rows;
    double fixed, kb, round, res, gelu;  // microseconds per launch, k-block, tile; more per tile with a residual, with GELU
  };
  static const Cand cands[10] = {
      {256, 256, 3.26, 0.269, 1.34, 2.23, 1.53}, {192, 256, 2.97, 0.208, 1.14, 0.86, 0.95}, {128, 256, 2.62, 0.160, 1.07, 0.67, 0.60},
      {64, 256, 2.69, 0.132, 0.67, 0.40, 0.40},  {128, 128, 2.52, 0.123, 0.64, 0.33, 0.29}, {64, 128, 2.43, 0.116, 0.52, 0.17, 0.10},
      {256, 0, 4.30, 0.309, 1.69, 2.89, 1.38},   {192, 0, 4.13, 0.231, 1.30, 2.19, 1.01},   {128, 0, 3.82, 0.213, 0.88, 1.39, 0.61},
      {64, 0, 3.49, 0.192, 0.72, 0.61, 0.36}};
  const int sms = num_sms();
  const bool bf16_out = ep.out_fp32 == 0;
  TileShape best = {N <= 64 ? 64 : 128, 0};
  double best_cost = 1e30;
  for (const Cand& c : cands) {
    if (c.rows ? !pairs : !one_sm) continue;
    if (c.bn > 64 && N <= c.bn - 64) continue;  // more than a third of the tile would be empty
    if (c.bn == 256 && !(allow256 && bf16_out)) continue;
    if (c.bn == 192 && !(allow192 && bf16_out)) continue;
    const int rows = c.rows ? c.rows : BM, units = c.rows ? sms / 2 : sms;
    const long tiles = (long)((M + rows - 1) / rows) * ((N + c.bn - 1) / c.bn);
    const long rounds = (tiles + units - 1) / units;
    const double res = c.bn == 256 && c.rows && rounds > 1 ? std::max(c.res, 4.0 - 0.05 * num_kb) : c.res;
    const double cost = c.fixed + (double)rounds * (num_kb * c.kb + c.round + (ep.residual ? res : 0) + (ep.act == GEMM_ACT_GELU ? c.gelu : 0));
    if (cost < best_cost) {
      best_cost = cost;
      best = {c.bn, c.rows};
    }
  }
  return best;
}

cudaError_t srpc_gemm_bf16_v2(const void* A, int lda, const void* B, int ldb, int M, int N, int K, const GemmEpilogue& ep,
                              uint32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return cudaErrorInvalidValue;
  if ((lda % 8) || (ldb % 8) || (K % 8) || ((uintptr_t)A & 15) || ((uintptr_t)B & 15)) return cudaErrorInvalidValue;
  if (ep.bias && ((uintptr_t)ep.bias & 15)) return cudaErrorInvalidValue;
  int use_tma_store = (!ep.out_fp32 && (ep.ldo % 8) == 0 && ((uintptr_t)ep.out & 15) == 0) ? 1 : 0;
  static const int allow_res_tma = [] { const char* e = getenv("SPLITRPC_GEMM_RES_TMA"); return e ? atoi(e) : 1; }();
  static const int res_tma_max_k = [] { const char* e = getenv("SPLITRPC_GEMM_RES_TMA_MAXK"); return e ? atoi(e) : 512; }();
  // Short-K shapes of many tiles are bound by memory and gain from the residual that TMA prefetches tiles ahead; few rounds of tiles
  // are bound by the launch and the first and last tile, and with a long K the plain residual loads of the epilogue hide behind the
  // next tile's MMAs.  The line, in rounds of full tiles, us by TMA and with the best pair tiles: K up to 256 from two rounds on
  // (25088 x 256 x 64 7.8 and 10.2, 28331 x 256 x 256 9.3 and 10.9, 6326 x 1000 x 64 11.0 and 13.1; 1.7 rounds: 4154 x 1000 x 128
  // 8.9 and 8.1, 200704 x 256 x 64 42 and 63), up to 512 from three (12544 x 1024 x 256 14.2 and 15.4; 5616 x 1000 x 512 14.0 and 10.6).
  const int rt_bn = N <= 64 ? 64 : 128;
  const bool many_tiles = (long)M * N > (K <= 256 ? 2l : 3l) * num_sms() * BM * rt_bn;
  const bool pairs = srpc_gemm_2sm_eligible(K, ep);
  const bool res_tma = allow_res_tma && use_tma_store == 1 && ep.residual && (ep.ldr % 8) == 0 &&
                       ((uintptr_t)ep.residual & 15) == 0 && K <= res_tma_max_k && (many_tiles || !pairs);
  // The residual ring lives in the output staging buffers, which the wide tiles have only one of.
  const TileShape ts = res_tma ? TileShape{rt_bn, 0} : pick_tile(M, N, (K + BK - 1) / BK, ep, true, pairs);
  const int bn = ts.bn;
  if (ts.rows) return srpc_gemm_bf16_2sm(A, lda, B, ldb, M, N, K, bn, ts.rows, ep, status, stream);
  TileParams p{};
  p.mode = 0;
  p.res_tma = res_tma ? 1 : 0;
  p.M = M;
  p.N = N;
  p.K = K;
  p.num_kb = (K + BK - 1) / BK;
  p.panel_kb = p.num_kb;
  p.tiles_m = (M + BM - 1) / BM;
  p.tiles_n = (N + bn - 1) / bn;
  CUtensorMap ta, tb, to;
  cudaError_t e = map_2d(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, BM);
  if (e != cudaSuccess) return e;
  e = map_2d(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, BK, (uint32_t)bn);
  if (e != cudaSuccess) return e;
  CUtensorMap tr = ta;
  if (use_tma_store == 1) {
    e = map_2d(&to, ep.out, (uint64_t)N, (uint64_t)M, (uint64_t)ep.ldo * 2, 64, BM);
    if (e != cudaSuccess) return e;
    if (res_tma) {
      e = map_2d(&tr, ep.residual, (uint64_t)N, (uint64_t)M, (uint64_t)ep.ldr * 2, 64, BM);
      if (e != cudaSuccess) return e;
    }
  } else {
    to = ta;
  }
  return dispatch(bn, ta, tb, to, tr, p, ep, use_tma_store, status, stream);
}

// Picks the output patch (pw x ph x pn <= 128 pixels) that wastes the fewest tile rows.
static void pick_patch(int ow, int oh, int nimg, int* pw, int* ph, int* pn) {
  if (const char* e = getenv("SPLITRPC_CONV_PATCH")) {  // "w,h,n": experiments with the patch shape
    int w = 0, h = 0, n = 0;
    if (sscanf(e, "%d,%d,%d", &w, &h, &n) == 3 && w >= 1 && h >= 1 && n >= 1 && w * h * n <= 128 && w <= ow && h <= oh && n <= nimg) {
      *pw = w;
      *ph = h;
      *pn = n;
      return;
    }
  }
  double best = -1;
  for (int w = 1; w <= std::min(ow, 64); w++)
    for (int h = 1; h <= std::min(oh, 128 / w); h++) {
      int n = std::min(nimg, 128 / (w * h));
      if (n < 1) continue;
      long tiles = (long)((ow + w - 1) / w) * ((oh + h - 1) / h) * ((nimg + n - 1) / n);
      double eff = (double)ow * oh * nimg / ((double)tiles * 128.0);
      double score = eff + 1e-4 * w;  // ties: longer contiguous runs
      if (score > best) {
        best = score;
        *pw = w;
        *ph = h;
        *pn = n;
      }
    }
}

cudaError_t srpc_conv_bf16_tma(const void* in, const void* weight, const ConvShape& cs, const GemmEpilogue& ep,
                               uint32_t* status, cudaStream_t stream) {
  if (cs.cin % BK || cs.cout % 8) return cudaErrorInvalidValue;
  if (((uintptr_t)in & 15) || ((uintptr_t)weight & 15) || ((uintptr_t)ep.out & 15) || ep.out_fp32) return cudaErrorInvalidValue;
  if (ep.bias && ((uintptr_t)ep.bias & 15)) return cudaErrorInvalidValue;
  if (srpc_stem_conv_eligible(cs, ep)) {
    if (cs.in_stub && (cs.in_ring_slots < cs.n || !cs.in_slot_bytes || cs.in_img_stride * 2 != (long)cs.in_slot_bytes))
      return cudaErrorInvalidValue;
    return srpc_stem_conv(in, weight, cs, ep, status, stream);
  }
  GemmEpilogue ep2 = ep;
  ep2.ldo = cs.cout;
  if (ep2.residual) ep2.ldr = cs.cout;
  if (cs.in2) {
    // out = act(W1 . in + W2 . in2(strided) + bias): the weight rows hold [W1 | W2]
    if (cs.r != 1 || cs.s != 1 || cs.pad != 0 || cs.in_stub || cs.cin2 % BK || cs.stride2 < 1 || ((uintptr_t)cs.in2 & 15))
      return cudaErrorInvalidValue;
    if ((cs.h2 - 1) / cs.stride2 + 1 != cs.oh || (cs.w2 - 1) / cs.stride2 + 1 != cs.ow) return cudaErrorInvalidValue;
  }
  // A dense pointwise convolution is a matrix product and takes its routes, the residual by TMA among them (us as runs of pixels on
  // pairs, 200704 x 256 x 256 with residual 94, 53 as a product; 64 x 28 x 28 pixels, 64 -> 256 18.6 and 12.2; the same bits).
  const bool dense = !cs.in_stub && !cs.in_pix_stride && !cs.in_row_stride && !cs.in_img_stride;
  if (dense && !cs.in2 && cs.r == 1 && cs.s == 1 && cs.stride == 1 && cs.pad == 0)
    return srpc_gemm_bf16_v2(in, cs.cin, weight, cs.cin, cs.n * cs.h * cs.w, cs.cout, cs.cin, ep2, status, stream);
  // Every other dense convolution goes to pairs: on 745 (filters of 1 to 5 rows, steps of 1 and 2, 7 .. 224 pixels wide, 64 .. 512 channels, 1 .. 64
  // images) the one-SM form takes 1.5 times as long on average; it is ahead by up to 10 % on a few of the largest (8 x 28 x 28 x 512, 5x5 65 and 60 us;
  // 32 x 56 x 56, 64 -> 128, 3x3 20.9 and 19.9).
  if (srpc_conv_2sm_eligible(cs, ep2)) {
    const TileShape ts = pick_tile(cs.n * cs.oh * cs.ow, cs.cout, (cs.r * cs.s * cs.cin + (cs.in2 ? cs.cin2 : 0)) / BK, ep2, false, true);
    return srpc_conv_bf16_2sm(in, weight, cs, ts.bn, ts.rows, ep2, status, stream);
  }
  TileParams p{};
  p.mode = 1;
  p.oh = cs.oh;
  p.ow = cs.ow;
  p.nimg = cs.n;
  p.M = cs.n * cs.oh * cs.ow;
  p.N = cs.cout;
  p.K = cs.r * cs.s * cs.cin;
  p.r = cs.r;
  p.s = cs.s;
  p.cblocks = cs.cin / BK;
  p.num_kb = cs.r * cs.s * p.cblocks;
  p.kb_split = p.num_kb;
  p.stride2 = 1;
  if (cs.in2) {
    p.K += cs.cin2;
    p.num_kb += cs.cin2 / BK;
    p.stride2 = cs.stride2;
  }
  p.panel_kb = p.num_kb;
  p.stride = cs.stride;
  p.pad = cs.pad;
  // Row-tap reuse: 8-pixel-wide patches, so that a step of one image row inside the box is 1024 bytes (one swizzle
  // atom) and the shifted A descriptors stay aligned; the box (ph + r - 1 rows) must fit the 128-row A slot.
  static const int allow_reuse = [] { const char* e = getenv("SPLITRPC_CONV_REUSE"); return e ? atoi(e) : 1; }();
  const bool reuse = allow_reuse && srpc_conv_rows_innermost(cs);
  int bn;
  if (reuse) {
    p.reuse = 1;
    p.pw = REUSE_PW;
    p.ph = std::min(cs.oh, 16 - (cs.r - 1));
    p.pn = 1;
    p.num_kb = cs.s * p.cblocks;  // load groups
  } else {
    pick_patch(cs.ow, cs.oh, cs.n, &p.pw, &p.ph, &p.pn);
  }
  p.rows_used = p.pw * p.ph * p.pn;
  p.tiles_w = (cs.ow + p.pw - 1) / p.pw;
  p.tiles_h = (cs.oh + p.ph - 1) / p.ph;
  p.tiles_m = p.tiles_w * p.tiles_h * ((cs.n + p.pn - 1) / p.pn);
  if (reuse) bn = cs.cout <= 64 ? 64 : 128;  // r B tiles travel with every A box: wider tiles leave too few stages
  else bn = pick_tile(p.tiles_m * BM, cs.cout, p.num_kb, ep2, true, false).bn;
  p.tiles_n = (cs.cout + bn - 1) / bn;
  const int box_rows = reuse ? p.ph + cs.r - 1 : p.ph * cs.stride;
  p.a_box_bytes = reuse ? (uint32_t)(box_rows * p.pw) * 128u : (uint32_t)p.rows_used * 128u;
  CUtensorMap ta, tb, to;
  {
    const uint64_t pix = cs.in_pix_stride ? (uint64_t)cs.in_pix_stride : (uint64_t)cs.cin;
    const uint64_t rowst = cs.in_row_stride ? (uint64_t)cs.in_row_stride : (uint64_t)cs.w * pix;
    const uint64_t imgst = cs.in_img_stride ? (uint64_t)cs.in_img_stride : (uint64_t)cs.h * rowst;
    if ((pix % 8) || (rowst % 8) || (imgst % 8)) return cudaErrorInvalidValue;
    if (cs.in_stub && (cs.in_ring_slots < cs.n || !cs.in_slot_bytes || imgst * 2 != cs.in_slot_bytes)) return cudaErrorInvalidValue;
    uint64_t dims[4] = {(uint64_t)cs.cin, (uint64_t)cs.w, (uint64_t)cs.h, (uint64_t)(cs.in_stub ? cs.in_ring_slots : cs.n)};
    uint64_t st[3] = {pix * 2, rowst * 2, imgst * 2};
    p.in_stub = cs.in_stub;
    p.in_ring_base = (unsigned long long)(uintptr_t)in;
    p.in_slot_bytes = cs.in_slot_bytes;
    uint32_t box[4] = {BK, (uint32_t)(p.pw * cs.stride), (uint32_t)box_rows, (uint32_t)p.pn};
    uint32_t es[4] = {1, (uint32_t)cs.stride, (uint32_t)cs.stride, 1};
    if (box[1] > 256 || box[2] > 256) return cudaErrorInvalidValue;
    cudaError_t e = get_map(&ta, in, 4, dims, st, box, es);
    if (e != cudaSuccess) return e;
  }
  CUtensorMap ta2 = ta;
  if (cs.in2) {
    uint64_t dims[4] = {(uint64_t)cs.cin2, (uint64_t)cs.w2, (uint64_t)cs.h2, (uint64_t)cs.n};
    uint64_t st[3] = {(uint64_t)cs.cin2 * 2, (uint64_t)cs.w2 * cs.cin2 * 2, (uint64_t)cs.h2 * cs.w2 * cs.cin2 * 2};
    uint32_t box[4] = {BK, (uint32_t)(p.pw * cs.stride2), (uint32_t)(p.ph * cs.stride2), (uint32_t)p.pn};
    uint32_t es[4] = {1, (uint32_t)cs.stride2, (uint32_t)cs.stride2, 1};
    if (box[1] > 256 || box[2] > 256) return cudaErrorInvalidValue;
    cudaError_t e2 = get_map(&ta2, cs.in2, 4, dims, st, box, es);
    if (e2 != cudaSuccess) return e2;
  }
  cudaError_t e = map_2d(&tb, weight, (uint64_t)p.K, (uint64_t)cs.cout, (uint64_t)p.K * 2, BK, (uint32_t)bn);
  if (e != cudaSuccess) return e;
  {
    uint64_t dims[4] = {(uint64_t)cs.cout, (uint64_t)cs.ow, (uint64_t)cs.oh, (uint64_t)cs.n};
    uint64_t st[3] = {(uint64_t)cs.cout * 2, (uint64_t)cs.ow * cs.cout * 2, (uint64_t)cs.oh * cs.ow * cs.cout * 2};
    uint32_t box[4] = {64, (uint32_t)p.pw, (uint32_t)p.ph, (uint32_t)p.pn};
    uint32_t es[4] = {1, 1, 1, 1};
    e = get_map(&to, ep.out, 4, dims, st, box, es);
    if (e != cudaSuccess) return e;
  }
  return dispatch(bn, ta, tb, to, ta2, p, ep2, 1, status, stream);
}

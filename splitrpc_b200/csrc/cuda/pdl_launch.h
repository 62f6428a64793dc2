// Launches that may start while the kernel before them in the stream is still running (programmatic stream
// serialisation).  The layers of a model are chains of 50 - 90 kernels of 5 - 75 us: with ordinary launches every one
// of them pays the launch latency, its barrier / tensor-memory / tensor-map set-up and the wait for the slowest block of
// the kernel before it one after the other.  Launched this way a block takes its SM as soon as the previous kernel's
// block has left it, does its set-up there and waits at ptx::grid_dep_wait() for the data.
//
// Measured (graph replays): a BERT-base encoder layer for 128 tokens (seven launches) 60.1 -> 55.3 us, BERT-base for 32 x 128
// tokens (88 launches) 1268 -> 1227 us, ResNet-50 for 64 images (54 launches) 1315 -> 1284 us.
//
// What a kernel launched through launch_pdl must do:
//   * every thread calls ptx::grid_dep_wait() before its first access to global memory that another kernel may touch
//     (reads AND writes: a buffer may still be read by the kernel before); the wait returns when the kernel before has
//     finished and its writes are visible, and that kernel waited for its own predecessor in the same way, so the
//     order of the whole stream is kept;
//   * data that another kernel may have written is read with ordinary loads: no __ldg and no __restrict__ on the pointer,
//     since a non-coherent load may be moved above the wait;
//   * ptx::grid_dep_launch() comes AFTER the block has allocated its tensor memory: a block of the next kernel that
//     allocated first would hold the columns while it waits for this kernel, and this kernel would wait for the columns;
//   * a kernel whose grid leaves the reserved SMs free (srpc_gemm_reserve_sms) calls it behind its last load instead while
//     SMs are reserved.  The SMs left free are the only place where the next kernel's blocks fit; triggered early they
//     sat there for the whole length of this kernel, and the copy kernel that the SMs are reserved for waited for a kernel
//     boundary.  ResNet-50, 64 images, 12 SMs reserved, end to end: 46,400 req/s, p99 5.3 ms, 53 requests per batch with
//     the early trigger; 51,150 req/s, p99 4.0 ms, 63.7 per batch with the late one; 51,600 req/s, p99 3.9 ms with ordinary
//     launches, which cost the timed step 1.254 -> 1.307 ms.
// Kernels without these calls, copies and event nodes on either side keep the ordinary full dependency.
#pragma once

#include <cuda_runtime.h>

#include <utility>

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  if (e != cudaSuccess) (void)cudaGetLastError();  // reported to the caller; not left behind for a later check
  return e;
}

// reduce.cu -- hgb_reduce: single-pass global reductions (kernels in
// reduce_kernels.cuh) with the per-device library workspace as scratch.
#include "reduce_kernels.cuh"

using namespace hgb;

namespace {

// Where the kernel leaves a host result: eight bytes of pinned host memory per
// calling thread (a call returns after its stream is done, so a thread needs one),
// freed with the thread.  Writing it from the kernel saves the copy back: 20 us
// with a queued copy of 8 bytes through the C ABI, 13 us without (a call through
// hipacc_gb300.api 26 -> 16 us; the first call of a thread that lives for two calls
// 69 -> 55 us, from its start to its end 258 -> 224 us, pinning included).
struct HostSlot {
  unsigned long long *p = nullptr;
  ~HostSlot() {
    if (!p) return;
    const RelaxedCapture relaxed;
    if (cudaFreeHost(p) != cudaSuccess) cudaGetLastError();
  }
  unsigned long long *get() {
    if (!p) {
      const RelaxedCapture relaxed;
      if (cudaHostAlloc((void **)&p, sizeof(*p), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
        p = nullptr;
        cudaGetLastError();
      }
    }
    return p;  // unified addressing: the same address on every device
  }
};
thread_local HostSlot t_slot;

}  // namespace

extern "C" int hgb_reduce(const hgb_view *in, const hgb_window *winp, int op, void *result_dev, void *result_host,
                          void *stream) {
  HGB_REQUIRE(result_dev || result_host, "hgb_reduce: no result destination");
  RedParams p;
  int grid = 0;
  int rc = reduce_setup(in, winp, op, &p, &grid);
  if (rc) return rc;
  Workspace ws;
  rc = workspace_get((size_t)grid * 16 + 64, &ws);
  if (rc) return rc;
  p.partials = ws.base;
  // the 8-byte result slot sits behind the partials when no device result is given
  unsigned long long *slot = (unsigned long long *)((char *)ws.base + (size_t)grid * 16);
  unsigned long long *direct = result_host && !result_dev ? t_slot.get() : nullptr;
  p.result_dev = result_dev ? (unsigned long long *)result_dev : (direct ? direct : slot);
  p.ticket = ws.tickets + 1;
  p.acc = ws.acc + kSlotReduce;
  cudaStream_t st = (cudaStream_t)stream;
  rc = reduce_launch(in->dtype, op, p, grid, st);
  if (rc) return rc;
  if (direct) {
    HGB_CHECK_CUDA(cudaStreamSynchronize(st));
    memcpy(result_host, direct, 8);
  } else if (result_host) {
    HGB_CHECK_CUDA(cudaMemcpyAsync(result_host, p.result_dev, 8, cudaMemcpyDeviceToHost, st));
    HGB_CHECK_CUDA(cudaStreamSynchronize(st));
  }
  return HGB_OK;
}

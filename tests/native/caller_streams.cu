// A caller's side of the stream contract, for tests/test_caller_streams_gpu.py:
// kernels in front of the library's on the same stream, streams with implicit
// ordering, and stream capture.  Built by the test with nvcc; its own runtime
// instance shares the process's primary context, and streams cross as handles.
#include <cuda_runtime.h>

#include <cstdint>

namespace {

constexpr unsigned COPY_BLOCKS = 8, COPY_THREADS = 256;

// dst = src after about `delay_us`; the next kernel of the stream may start at once
__global__ void __launch_bounds__(COPY_THREADS) delayed_copy_kernel(const uint4 *src, uint4 *dst, unsigned long long words, unsigned delay_us) {
  asm volatile("griddepcontrol.launch_dependents;");
  for (unsigned k = 0; k < delay_us; k++)
    __nanosleep(1000);
  for (unsigned long long i = blockIdx.x * (unsigned long long)COPY_THREADS + threadIdx.x; i < words; i += (unsigned long long)COPY_BLOCKS * COPY_THREADS)
    dst[i] = src[i];
}

// lets the next kernel start and ends, without waiting for the one before it
__global__ void passing_kernel() { asm volatile("griddepcontrol.launch_dependents;"); }

cudaError_t launch_passing(cudaStream_t stream) {
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = 1;
  config.blockDim = 32;
  config.stream = stream;
  config.attrs = &early;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, passing_kernel);
}

} // namespace

extern "C" {

int caller_delayed_copy(void *stream, const void *src, void *dst, unsigned long long bytes, unsigned delay_us) {
  delayed_copy_kernel<<<COPY_BLOCKS, COPY_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint4 *>(src), static_cast<uint4 *>(dst),
                                                                                         bytes / 16, delay_us);
  return cudaGetLastError();
}
int caller_passing(void *stream) { return launch_passing(static_cast<cudaStream_t>(stream)); }

// a stream that is ordered with the legacy default stream
int caller_blocking_stream(void **stream) { return cudaStreamCreateWithFlags(reinterpret_cast<cudaStream_t *>(stream), cudaStreamDefault); }
int caller_stream_destroy(void *stream) { return cudaStreamDestroy(static_cast<cudaStream_t>(stream)); }

int caller_capture_begin(void *stream) { return cudaStreamBeginCapture(static_cast<cudaStream_t>(stream), cudaStreamCaptureModeThreadLocal); }
int caller_capture_end(void *stream, void **graph) {
  cudaGraph_t captured = nullptr;
  cudaError_t e = cudaStreamEndCapture(static_cast<cudaStream_t>(stream), &captured);
  if (e == cudaSuccess)
    e = cudaGraphInstantiate(reinterpret_cast<cudaGraphExec_t *>(graph), captured, 0);
  if (captured)
    cudaGraphDestroy(captured);
  return e;
}
int caller_graph_launch(void *graph, void *stream) { return cudaGraphLaunch(static_cast<cudaGraphExec_t>(graph), static_cast<cudaStream_t>(stream)); }
int caller_graph_destroy(void *graph) { return cudaGraphExecDestroy(static_cast<cudaGraphExec_t>(graph)); }

} // extern "C"

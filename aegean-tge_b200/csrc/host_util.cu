// Host-side error plumbing shared by every library built from this folder.
// An entry point that refuses its arguments stores a message here and returns
// a negative code; the Python binding raises it.
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>

#include "common.cuh"

static thread_local char g_error[768] = "";

void tge_set_error(const char* fmt, ...) {
  va_list args;
  va_start(args, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, args);
  va_end(args);
}

int tge_check_launch(const char* what) {
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    tge_set_error("%s: launch failed: %s", what, cudaGetErrorString(err));
    return -2;
  }
  return 0;
}

bool tge_pdl_enabled() {
  static int enabled = -1;
  if (enabled < 0) {
    const char* off = getenv("TGE_NO_PDL");
    enabled = (off != nullptr && off[0] != '\0') ? 0 : 1;
  }
  return enabled == 1;
}

int tge_sm_count() {
  static int count = 0;
  if (count == 0) {
    int device = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device);
    if (count <= 0) count = 1;
  }
  return count;
}

TGE_API int tge_device_sm_count() { return tge_sm_count(); }

// What a step does around its kernels, on the raw stream: torch's own calls look up a stream object and build event and
// copy objects each time (5 to 9 us apiece, against 1 to 2 here, three copies and two events to a step of a small model).
static int checked(const char* what, cudaError_t err) {
  if (err == cudaSuccess) return 0;
  cudaGetLastError();
  tge_set_error("%s: %s", what, cudaGetErrorString(err));
  return -2;
}
TGE_API int tge_event_create(void** event) {
  return checked("event", cudaEventCreateWithFlags(reinterpret_cast<cudaEvent_t*>(event), cudaEventDisableTiming));
}
TGE_API int tge_event_record(void* event, cudaStream_t stream) { return checked("event record", cudaEventRecord((cudaEvent_t)event, stream)); }
TGE_API int tge_event_synchronize(void* event) { return checked("event wait", cudaEventSynchronize((cudaEvent_t)event)); }
// 1: what was queued before the last record is done, 0: not yet
TGE_API int tge_event_query(void* event) {
  const cudaError_t err = cudaEventQuery((cudaEvent_t)event);
  if (err == cudaErrorNotReady) {
    cudaGetLastError();
    return 0;
  }
  return err == cudaSuccess ? 1 : checked("event query", err);
}
TGE_API int tge_event_wait(void* event, cudaStream_t stream) { return checked("wait of a stream", cudaStreamWaitEvent(stream, (cudaEvent_t)event, 0)); }
TGE_API int tge_event_destroy(void* event) { return checked("event", cudaEventDestroy((cudaEvent_t)event)); }
// The caller keeps both ends alive until the copy is done.
TGE_API int tge_copy(void* dst, const void* src, long long bytes, cudaStream_t stream) {
  return checked("copy", cudaMemcpyAsync(dst, src, (size_t)bytes, cudaMemcpyDefault, stream));
}

// A captured step's replay as one call: the step's index arrays go to the device (`copied` is recorded behind that copy), token ids that are
// on the device already go over them, the graph is launched.
TGE_API int tge_replay_step(void* dev, const void* host, long long bytes, void* copied, void* tokens_at, const void* tokens, long long token_bytes,
                            void* graph, cudaStream_t stream) {
  int rc = checked("copy of a step", cudaMemcpyAsync(dev, host, (size_t)bytes, cudaMemcpyHostToDevice, stream));
  if (rc == 0) rc = checked("event record", cudaEventRecord((cudaEvent_t)copied, stream));
  if (rc == 0 && token_bytes > 0) rc = checked("copy of a step's tokens", cudaMemcpyAsync(tokens_at, tokens, (size_t)token_bytes, cudaMemcpyDeviceToDevice, stream));
  return rc != 0 ? rc : checked("graph launch", cudaGraphLaunch((cudaGraphExec_t)graph, stream));
}

TGE_API const char* tge_last_error() { return g_error; }

TGE_API int tge_abi_version() { return 1; }

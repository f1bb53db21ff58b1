// A product whose rows come from the host and whose result goes back there, piece by piece (one GPU): piece i + 1 on its way in
// while piece i is multiplied and piece i - 1 is on its way out, on three streams.
//
// Host code only.  Bound by the link (53 GB/s each way).  Beside the longer direction the first piece's way in, the last one's product
// and its way out are exposed, and a pair of copies that run at the same time takes both directions some 12 us more than the link.
// So few pieces, whose sizes fall or rise by the ratio of the directions (`_pieces` in ops/gemm.py).  A piece takes eight
// runtime calls, 10 us here and 45 us through torch's streams and events (256 x 1024 x 1024 in four pieces: 254 us, all on the host).
#include <cuda_runtime.h>

#include "../common/host_util.h"
#include "../include/kb200.h"

namespace {

constexpr int MAX_PIECES = 64;
// events: three of the whole call, then of piece i: its rows are there, its product is done
constexpr int FINISHED = 0, STARTED = 1, LEFT = 2;
int ready_of(int i) { return 3 + 2 * i; }
int done_of(int i) { return 4 + 2 * i; }

cudaEvent_t event(const KbGemmStreamArgs* s, int i) { return static_cast<cudaEvent_t>(s->events[i]); }
cudaStream_t stream(void* p) { return static_cast<cudaStream_t>(p); }

int check(const KbGemmStreamArgs* s) {
  if (s == nullptr || s->events == nullptr || s->rows == nullptr || s->pieces < 1 || s->pieces > MAX_PIECES || s->product.kind != KB_LOCAL_DENSE ||
      s->product.a_mn != 0 || s->product.b_mn != 0 || s->a_host == nullptr || s->out_host == nullptr) {
    kb::set_error("kb_gemm_stream: a dense product of rows in 1 to %d pieces", MAX_PIECES);
    return KB_ERR_ARG;
  }
  long long rows = 0;
  for (int i = 0; i < s->pieces; ++i) rows += s->rows[i] > 0 ? s->rows[i] : s->product.M + 1ll;
  if (rows != s->product.M) {
    kb::set_error("kb_gemm_stream: the pieces are not the product's %d rows", s->product.M);
    return KB_ERR_ARG;
  }
  return KB_OK;
}

}  // namespace

extern "C" int kb_gemm_stream_events(int pieces) { return 2 * pieces + 3; }

extern "C" int kb_events_create(int n, void** events) {
  for (int i = 0; i < n; ++i) events[i] = nullptr;
  for (int i = 0; i < n; ++i) {
    cudaEvent_t e = nullptr;
    KB_CUDA_OK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    events[i] = e;
  }
  return KB_OK;
}

extern "C" int kb_events_destroy(int n, void** events) {
  for (int i = 0; i < n; ++i) {
    if (events[i] != nullptr) cudaEventDestroy(static_cast<cudaEvent_t>(events[i]));
    events[i] = nullptr;
  }
  return KB_OK;
}

extern "C" int kb_gemm_stream_begin(const KbGemmStreamArgs* s) {
  const int rc = check(s);
  if (rc != KB_OK) return rc;
  // A call on another stream than the last one's finds that one's buffers in use.  A graph does not wait for
  // calls before it, nor they for its replays: that order is the program's.
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  KB_CUDA_OK(cudaStreamIsCapturing(stream(s->stream), &capturing));
  if (capturing == cudaStreamCaptureStatusNone && s->again) KB_CUDA_OK(cudaStreamWaitEvent(stream(s->stream), event(s, FINISHED), 0));
  KB_CUDA_OK(cudaEventRecord(event(s, STARTED), stream(s->stream)));
  KB_CUDA_OK(cudaStreamWaitEvent(stream(s->in), event(s, STARTED), 0));
  return KB_OK;
}

extern "C" int kb_gemm_stream_run(const KbGemmStreamArgs* s) {
  int rc = check(s);
  if (rc != KB_OK) return rc;
  const cudaStream_t cur = stream(s->stream), in = stream(s->in), out = stream(s->out);
  KbLocalGemmArgs a = s->product;
  const size_t in_row = static_cast<size_t>(a.K) * 2, out_row = static_cast<size_t>(a.N) * 2;
  char* const in_dev = static_cast<char*>(const_cast<void*>(s->product.A));
  char* const out_dev = static_cast<char*>(s->product.out);
  size_t first = 0;
  for (int i = 0; i < s->pieces; ++i) {
    const int rows = s->rows[i];
    if (i > 0) {
      KB_CUDA_OK(cudaMemcpyAsync(in_dev + first * in_row, static_cast<const char*>(s->a_host) + first * in_row, rows * in_row, cudaMemcpyHostToDevice, in));
    }
    KB_CUDA_OK(cudaEventRecord(event(s, ready_of(i)), in));
    KB_CUDA_OK(cudaStreamWaitEvent(cur, event(s, ready_of(i)), 0));
    a.M = rows;
    a.A = in_dev + first * in_row;
    a.out = out_dev + first * out_row;
    rc = kb_gemm_local(&a, s->stream);
    if (rc != KB_OK) return rc;
    KB_CUDA_OK(cudaEventRecord(event(s, done_of(i)), cur));
    KB_CUDA_OK(cudaStreamWaitEvent(out, event(s, done_of(i)), 0));
    if (i + 1 < s->pieces) {
      KB_CUDA_OK(cudaMemcpyAsync(static_cast<char*>(s->out_host) + first * out_row, out_dev + first * out_row, rows * out_row, cudaMemcpyDeviceToHost, out));
    }
    first += rows;
  }
  return KB_OK;
}

extern "C" int kb_gemm_stream_end(KbGemmStreamArgs* s) {
  const int rc = check(s);
  if (rc != KB_OK) return rc;
  KB_CUDA_OK(cudaEventRecord(event(s, LEFT), stream(s->out)));
  KB_CUDA_OK(cudaStreamWaitEvent(stream(s->stream), event(s, LEFT), 0));
  // An event of a graph is nothing to wait for outside of it: a captured call leaves the chain of the others as it was.
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  KB_CUDA_OK(cudaStreamIsCapturing(stream(s->stream), &capturing));
  if (capturing != cudaStreamCaptureStatusNone) return KB_OK;
  KB_CUDA_OK(cudaEventRecord(event(s, FINISHED), stream(s->stream)));
  s->again = 1;
  return KB_OK;
}

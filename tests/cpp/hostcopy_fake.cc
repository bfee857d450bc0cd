// Host check of the threaded host copies (tg_hostcopy.cu) against a fake CUDA runtime whose streams run
// nothing until they are waited for.  A stream is a queue of operations; cudaStreamPerThread names another
// queue in every thread.  Each scenario (argv[1]) exits 0 when the copy did what it has to.
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <thread>
#include <utility>
#include <vector>

#include "tg_hostcopy.h"

namespace {

using Key = std::pair<cudaStream_t, std::thread::id>;
struct Queue {
  std::vector<std::function<void()>> ops;
  size_t done = 0;
};
struct Event {
  Queue* q = nullptr;
  size_t upto = 0;
};

std::mutex mu;
std::map<Key, Queue> queues;
std::thread::id caller;
int staged_copies = 0;     // transfers queued by a thread that is not the caller
int allocs = 0;            // of page-locked memory
int records = 0, fail_record = -1;
cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;

Queue* queue_of(cudaStream_t s) {
  return &queues[Key(s, s == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id())];
}
void run(Queue* q, size_t upto) {
  for (; q->done < upto; ++q->done) q->ops[q->done]();
}
size_t in_flight() {
  size_t n = 0;
  for (auto& kv : queues) n += kv.second.ops.size() - kv.second.done;
  return n;
}

}  // namespace

extern "C" {
int get_nprocs() { return 16; }  // what std::thread::hardware_concurrency reads
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::malloc(n);
  ++allocs;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new Event);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<Event*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::mutex> lk(mu);
  if (fail_record >= 0 && records++ >= fail_record) return cudaErrorUnknown;
  Event* ev = reinterpret_cast<Event*>(e);
  ev->q = queue_of(s);
  ev->upto = ev->q->ops.size();
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::mutex> lk(mu);
  Event* ev = reinterpret_cast<Event*>(e);
  run(ev->q, ev->upto);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  std::lock_guard<std::mutex> lk(mu);
  if (std::this_thread::get_id() != caller) ++staged_copies;
  queue_of(st)->ops.push_back([=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::mutex> lk(mu);
  if (capture != cudaStreamCaptureStatusNone) return cudaErrorStreamCaptureUnsupported;
  Queue* q = queue_of(s);
  run(q, q->ops.size());
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* st) {
  *st = capture;
  return cudaSuccess;
}
}

#define CHECK(c)                                             \
  do {                                                       \
    if (!(c)) {                                              \
      std::printf("line %d: %s\n", __LINE__, #c);            \
      return 1;                                              \
    }                                                        \
  } while (0)

int main(int argc, char** argv) {
  const char* what = argc > 1 ? argv[1] : "";
  const size_t n = (9 << 20) + 123;
  std::vector<unsigned char> dev(n, 0), host(n, 0), want(n);
  for (size_t i = 0; i < n; ++i) want[i] = (unsigned char)(i * 2654435761u >> 13);
  caller = std::this_thread::get_id();
  cudaStream_t s = std::strstr(what, "per_thread") ? cudaStreamPerThread : reinterpret_cast<cudaStream_t>(0x1000);
  tg::host_copy_retain();
  // the threads come once enough has been copied to pay for them
  if (std::strcmp(what, "short_use")) {
    const cudaStream_t other = reinterpret_cast<cudaStream_t>(0x2000);
    for (int i = 0; i < 30; ++i) CHECK(tg::host_copy(dev.data(), host.data(), n, true, 0, other) == cudaSuccess);
    CHECK(staged_copies > 0);
    staged_copies = 0;
  }

  if (!std::strcmp(what, "download") || !std::strcmp(what, "download_per_thread")) {
    // work queued before the copy on the caller's stream fills the device buffer
    for (int i = 0; i < 3; ++i) {
      {
        std::lock_guard<std::mutex> lk(mu);
        queue_of(s)->ops.push_back([&, i] {
          for (size_t k = 0; k < n; ++k) dev[k] = (unsigned char)(want[k] + i);
        });
      }
      CHECK(tg::host_copy(host.data(), dev.data(), n, false, 0, s) == cudaSuccess);
      for (size_t k = 0; k < n; ++k) CHECK(host[k] == (unsigned char)(want[k] + i));
    }
    CHECK(s == cudaStreamPerThread || staged_copies > 0);
  } else if (!std::strcmp(what, "upload") || !std::strcmp(what, "upload_per_thread")) {
    // work queued before the copy still reads the device buffer's former contents
    std::vector<unsigned char> seen(n, 1);
    {
      std::lock_guard<std::mutex> lk(mu);
      queue_of(s)->ops.push_back([&] { seen = dev; });
    }
    CHECK(tg::host_copy(dev.data(), want.data(), n, true, 0, s) == cudaSuccess);
    CHECK(cudaStreamSynchronize(s) == cudaSuccess);
    CHECK(dev == want);
    CHECK(seen == std::vector<unsigned char>(n, 0));
    CHECK(s == cudaStreamPerThread || staged_copies > 0);
  } else if (!std::strcmp(what, "record_fails")) {
    // events that cannot be recorded: the call fails, and no transfer is left in flight on the slots
    for (int at : {0, 2, 5}) {
      records = 0;
      fail_record = at;
      CHECK(tg::host_copy(dev.data(), want.data(), n, true, 0, s) != cudaSuccess);
      CHECK(in_flight() == 0);
      fail_record = -1;
      CHECK(tg::host_copy(dev.data(), want.data(), n, true, 0, s) == cudaSuccess);
      CHECK(dev == want);
    }
    CHECK(staged_copies > 0);
  } else if (!std::strcmp(what, "short_use")) {
    // a few copies of fields that are there: owners that come and go never set the threads up
    for (int round = 0; round < 3; ++round) {
      for (int i = 0; i < 13; ++i) {
        CHECK(tg::host_copy(host.data(), want.data(), n, false, 0, s) == cudaSuccess);
        CHECK(host == want);
      }
      for (int i = 0; i < 5; ++i) CHECK(tg::host_copy(dev.data(), want.data(), n, true, 0, s) == cudaSuccess);
      CHECK(staged_copies == 0 && allocs == 0);
      tg::host_copy_release();
      tg::host_copy_retain();
    }
    // three downloads into pages that are not there yet do
    for (int i = 0; i < 3; ++i) {
      void* f = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
      CHECK(tg::host_copy(f, want.data(), n, false, 0, s) == cudaSuccess);
      CHECK(std::memcmp(f, want.data(), n) == 0);
      munmap(f, n);
    }
    CHECK(staged_copies > 0 && allocs == 1);
  } else if (!std::strcmp(what, "capture")) {
    // a stream in capture: no other thread adds to the caller's graph, and the call is refused as a
    // plain copy with its wait is
    capture = cudaStreamCaptureStatusActive;
    CHECK(tg::host_copy(dev.data(), want.data(), n, true, 0, s) == cudaErrorStreamCaptureUnsupported);
    CHECK(staged_copies == 0);
  } else {
    return 2;
  }
  tg::host_copy_release();
  return 0;
}

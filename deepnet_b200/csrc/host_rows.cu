// Results written out to ordinary (pageable) host memory behind the work that produces them.
//
// A device-to-host copy into pageable memory goes through the driver's own pinned buffer on the calling thread, which meanwhile
// issues nothing: 110 us a megabyte, most of a minibatch's time where representations are written out
// (deepnet/extract_rbm_representation.py).  Here the copy lands in pinned pieces on a stream of its own and a few threads
// carry the pieces to where they belong, while the caller goes on to the next minibatch: eight of 250 x 1000 with their
// reconstruction error 1154 -> 540 us, and 365 with several minibatches a product and pieces copied several at a time.
// One staging area per process (4 MB and four threads, made on first use, given back by cublas_shutdown): whoever
// begins while another thread holds it is told so and copies the plain way.
//
// Every carrier takes a piece before it has landed, so that it is awake in time.  The two whose pieces land next wait busily
// (with blocking waits the call above took 603 us and more, against 556), the others look every ten microseconds.  Cores
// occupied with all four waiting busily / so: 4.1 / 3.3 in the call above, 4.4 / 3.6 in eight minibatches of 500 x 2048
// (1418 / 1297 us).  Fewer carriers, asleep until a piece has landed, gained as much on large results and lost up to 8 % on
// small ones; six lost 16 % where the result's pages are large.
#include <sys/prctl.h>
#include <time.h>

#include <atomic>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"

using namespace b200;

namespace {

// A copy from the device fills up to kRun neighbouring pieces, as many as are free (256 KB take 13 us one by one, 1 MB 24).  A
// thread carries a piece at a time, of a matrix of no more than one piece a part of it, so that all threads have one (100 x 500: 142 ->
// 65 us; parts of 64 KB cost large results up to a third).
constexpr int kPieces = 16, kRun = 4, kCarriers = 4, kBusy = 2;
constexpr size_t kPieceBytes = 256 * 1024, kPartBytes = 64 * 1024;
static_assert((1ull << 32) % kPieces == 0, "the counter of copies wraps to the same turn");

struct RowsStaging {
  std::mutex mu;
  std::condition_variable work, freed;
  struct Job {
    int piece, event;
    size_t from;           // in the pinned area
    float* dst;
    size_t bytes;
  };
  std::deque<Job> jobs;
  std::vector<std::thread> carriers;
  char* pinned = nullptr;
  cudaEvent_t landed[kPieces] = {nullptr}, ready = nullptr, done[2] = {nullptr, nullptr};
  cudaStream_t copies = nullptr;
  bool free_piece[kPieces];
  int parts[kPieces] = {0};      // of a piece, still to be carried
  int device = 0, in_flight = 0, adds = 0;
  unsigned copied = 0;           // copies so far; each has the next event in turn
  std::atomic<long> taken{0}, seen{0};     // pieces carriers have taken, and seen land
  bool held = false, stop = false, made = false, failed = false;

  // The order-th piece (of all ever taken) has landed.
  bool wait_for(cudaEvent_t event, long order) {
    for (;;) {
      const cudaError_t e = cudaEventQuery(event);
      if (e != cudaErrorNotReady) return e == cudaSuccess;
      if (order - seen < kBusy) return cudaEventSynchronize(event) == cudaSuccess;
      const timespec ten_us = {0, 10000};
      nanosleep(&ten_us, nullptr);
    }
  }
  void carry() {
    cudaSetDevice(device);
    prctl(PR_SET_TIMERSLACK, 1000ul);     // (of this thread: a nap of 10 us takes 60 by default)
    std::unique_lock<std::mutex> lock(mu);
    for (;;) {
      work.wait(lock, [&] { return stop || !jobs.empty(); });
      if (jobs.empty()) return;
      const Job j = jobs.front();
      jobs.pop_front();
      const long order = taken++;
      lock.unlock();
      const bool ok = wait_for(landed[j.event], order);
      seen++;
      if (ok) memcpy(j.dst, pinned + j.from, j.bytes);
      lock.lock();
      failed |= !ok;
      if (--parts[j.piece] == 0) free_piece[j.piece] = true;
      in_flight--;
      freed.notify_all();
    }
  }
  void give_back() {
    {
      std::lock_guard<std::mutex> lock(mu);
      stop = true;
    }
    work.notify_all();
    for (std::thread& t : carriers) t.join();
    carriers.clear();
    if (pinned) cudaFreeHost(pinned);
    pinned = nullptr;
    for (cudaEvent_t* e : {&ready, &done[0], &done[1]}) {
      if (*e) cudaEventDestroy(*e);
      *e = nullptr;
    }
    for (cudaEvent_t& e : landed) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
    if (copies) cudaStreamDestroy(copies);
    copies = nullptr;
    made = stop = false;
  }
  bool make() {
    bool ok = cudaGetDevice(&device) == cudaSuccess && cudaMallocHost((void**)&pinned, kPieces * kPieceBytes) == cudaSuccess &&
              cudaStreamCreateWithFlags(&copies, cudaStreamNonBlocking) == cudaSuccess;
    for (cudaEvent_t* e : {&ready, &done[0], &done[1]}) ok = ok && cudaEventCreateWithFlags(e, cudaEventDisableTiming) == cudaSuccess;
    for (cudaEvent_t& e : landed) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    for (bool& f : free_piece) f = true;
    try {
      for (int i = 0; ok && i < kCarriers; i++) carriers.emplace_back([this] { carry(); });
    } catch (...) {
      ok = false;
    }
    made = true;
    if (!ok) {
      cudaGetLastError();
      give_back();
    }
    return ok;
  }
};
// (never destroyed: the threads of a process that skips cublas_shutdown outlive its static objects)
RowsStaging& staging() {
  static RowsStaging* s = new RowsStaging;
  return *s;
}
std::mutex g_holder;     // guards `held` and the making of the staging area

}  // namespace

namespace b200 {
void free_rows_staging() {
  std::lock_guard<std::mutex> lock(g_holder);
  RowsStaging& s = staging();
  if (s.made && !s.held) s.give_back();
}
}  // namespace b200

extern "C" {

// 1: the staging area is the caller's until b200_rows_end; 0: it is taken, or cannot be had (copy the plain way).
int b200_rows_begin(void) {
  if (!initialised() || stream_capturing()) return 0;
  std::lock_guard<std::mutex> lock(g_holder);
  RowsStaging& s = staging();
  int device = -1;
  if (s.held || cudaGetDevice(&device) != cudaSuccess || (s.made && s.device != device)) return 0;
  if (!s.made && !s.make()) return 0;
  s.held = true;
  s.failed = false;
  s.adds = 0;
  return 1;
}

// The matrix into `dst` (numel floats), behind the work enqueued so far.  Work enqueued after this call may rewrite the matrix
// of the call before; this one's only after the next call or b200_rows_end.
int b200_rows_add(cudamat* src, float* dst) {
  RowsStaging& s = staging();
  if (!s.held) return ERROR_GENERIC;
  if (!src->on_device) return ERROR_NOT_ON_DEVICE;
  if (cudaEventRecord(s.ready, stream()) != cudaSuccess || cudaStreamWaitEvent(s.copies, s.ready, 0) != cudaSuccess)
    return set_error(cudaGetErrorString(cudaGetLastError()));
  const size_t bytes = (size_t)numel(src) * sizeof(float);
  for (size_t at = 0; at < bytes;) {
    int first = 0, pieces = 0;
    {
      std::unique_lock<std::mutex> lock(s.mu);
      s.freed.wait(lock, [&] {
        for (first = 0; first < kPieces && !s.free_piece[first];) first++;
        return first < kPieces;
      });
      while (pieces < kRun && first + pieces < kPieces && s.free_piece[first + pieces] && at + pieces * kPieceBytes < bytes)
        s.free_piece[first + pieces++] = false;
    }
    const size_t run = bytes - at < pieces * kPieceBytes ? bytes - at : pieces * kPieceBytes;
    // A job may still wait for this event, that of a copy kPieces copies ago: all copies are on one stream, so what it then waits
    // for landed later than its own.
    const int event = (int)(s.copied++ % kPieces);
    const bool ok = cudaMemcpyAsync(s.pinned + first * kPieceBytes, (const char*)src->data_device + at, run, cudaMemcpyDeviceToHost,
                                    s.copies) == cudaSuccess &&
                    cudaEventRecord(s.landed[event], s.copies) == cudaSuccess;
    std::lock_guard<std::mutex> lock(s.mu);
    if (!ok) {
      for (int i = 0; i < pieces; i++) s.free_piece[first + i] = true;
      s.failed = true;
      return set_error(cudaGetErrorString(cudaGetLastError()));
    }
    const size_t part = bytes <= kPieceBytes ? kPartBytes : kPieceBytes;
    for (size_t from = 0; from < run; from += part) {
      const int piece = first + (int)(from / kPieceBytes);
      s.jobs.push_back({piece, event, first * kPieceBytes + from, (float*)((char*)dst + at + from), run - from < part ? run - from : part});
      s.parts[piece]++;
      s.in_flight++;
      s.work.notify_one();
    }
    at += run;
  }
  // the matrix of the call before has been read once this stream is past its copies
  if (s.adds > 0 && cudaStreamWaitEvent(stream(), s.done[(s.adds - 1) & 1], 0) != cudaSuccess)
    return set_error(cudaGetErrorString(cudaGetLastError()));
  if (cudaEventRecord(s.done[s.adds & 1], s.copies) != cudaSuccess) return set_error(cudaGetErrorString(cudaGetLastError()));
  s.adds++;
  return 0;
}

// Returns when everything added is where it belongs.
int b200_rows_end(void) {
  RowsStaging& s = staging();
  if (!s.held) return ERROR_GENERIC;
  bool failed;
  {
    std::unique_lock<std::mutex> lock(s.mu);
    s.freed.wait(lock, [&] { return s.in_flight == 0; });
    failed = s.failed;
  }
  if (s.adds > 0 && cudaStreamWaitEvent(stream(), s.done[(s.adds - 1) & 1], 0) != cudaSuccess) failed = true;
  std::lock_guard<std::mutex> lock(g_holder);
  s.held = false;
  return failed ? set_error("a copy to the host failed") : 0;
}

}  // extern "C"

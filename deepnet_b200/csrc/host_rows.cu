// Results written out to ordinary (pageable) host memory behind the work that produces them.
//
// A device-to-host copy into pageable memory goes through the driver's own pinned buffer on the calling thread, which meanwhile
// issues nothing: 110 us a megabyte, most of a minibatch's time where representations are written out
// (deepnet/extract_rbm_representation.py).  Here the copy lands in pinned pieces on a stream of its own and a few threads
// carry the pieces to where they belong, while the caller goes on to the next minibatch: eight of 250 x 1000 with their
// reconstruction error 1154 -> 540 us.
// One staging area per process (4 MB and four threads, made on first use, given back by cublas_shutdown): whoever
// begins while another thread holds it is told so and copies the plain way.
//
// The carriers are bound by the page faults of the fresh result, which more than two or three threads only make dearer, unless its
// matrices are large.  At most two wait for their piece (busily: with blocking waits the call took twice as long); the others
// sleep until pieces have landed.  us a call and cores busy, by carriers / of them waiting:
//                                        2 / 2        3 / 2        4 / 2        4 / 4        6 / 2
//   eight minibatches of 250 x 1000      504, 2.5     552, 3.1     579, 3.3     556, 4.0     602, 3.4
//   eight of 500 x 2048                  1259, 2.4    1217, 3.5    1381, 3.9    1316, 4.4    1517, 4.0
//   two of 1024 x 8192                   9588, 2.0    7849, 2.9    7075, 3.6    7231, 4.0    6013, 4.8
//   two of 4096 x 2048, large pages                                             2627, 4.4    3062, 4.3
#include <condition_variable>
#include <cstring>
#include <deque>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"

using namespace b200;

namespace {

constexpr int kPieces = 16, kCarriers = 4, kWaiting = 2;
constexpr int kFewCarriers = 3;                     // ... of matrices below
constexpr size_t kManyCarriersBytes = 16 << 20;
constexpr size_t kPieceBytes = 256 * 1024;

struct RowsStaging {
  std::mutex mu;
  std::condition_variable work, more_work, freed;     // of the first carriers, of the others, of the caller
  struct Job {
    int piece;
    float* dst;
    size_t bytes;
  };
  std::deque<Job> jobs;
  std::vector<std::thread> carriers;
  char* pinned = nullptr;
  cudaEvent_t landed[kPieces] = {nullptr}, ready = nullptr, done[2] = {nullptr, nullptr};
  cudaStream_t copies = nullptr;
  bool free_piece[kPieces];
  int device = 0, in_flight = 0, adds = 0, waiting = 0, carrying = kFewCarriers;   // (threads that may carry)
  bool held = false, stop = false, made = false, failed = false;

  void wake_one() {
    work.notify_one();
    if (carrying > kFewCarriers) more_work.notify_one();
  }
  void carry(int self) {
    cudaSetDevice(device);
    std::unique_lock<std::mutex> lock(mu);
    for (;;) {
      (self < kFewCarriers ? work : more_work).wait(lock, [&] {
        return stop || (!jobs.empty() && waiting < kWaiting && self < carrying);
      });
      if (jobs.empty()) return;
      const Job j = jobs.front();
      jobs.pop_front();
      waiting++;
      lock.unlock();
      const bool ok = cudaEventSynchronize(landed[j.piece]) == cudaSuccess;
      lock.lock();
      waiting--;
      if (!jobs.empty()) wake_one();
      lock.unlock();
      if (ok) memcpy(j.dst, pinned + j.piece * kPieceBytes, j.bytes);
      lock.lock();
      failed |= !ok;
      free_piece[j.piece] = true;
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
    more_work.notify_all();
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
      for (int i = 0; ok && i < kCarriers; i++) carriers.emplace_back([this, i] { carry(i); });
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
  {
    std::lock_guard<std::mutex> lock(s.mu);
    s.carrying = bytes < kManyCarriersBytes ? kFewCarriers : kCarriers;
  }
  for (size_t at = 0; at < bytes; at += kPieceBytes) {
    const size_t n = bytes - at < kPieceBytes ? bytes - at : kPieceBytes;
    int piece = -1;
    {
      std::unique_lock<std::mutex> lock(s.mu);
      s.freed.wait(lock, [&] {
        for (piece = 0; piece < kPieces; piece++)
          if (s.free_piece[piece]) return true;
        return false;
      });
      s.free_piece[piece] = false;
    }
    const bool ok = cudaMemcpyAsync(s.pinned + piece * kPieceBytes, (const char*)src->data_device + at, n, cudaMemcpyDeviceToHost,
                                    s.copies) == cudaSuccess &&
                    cudaEventRecord(s.landed[piece], s.copies) == cudaSuccess;
    std::lock_guard<std::mutex> lock(s.mu);
    if (!ok) {
      s.free_piece[piece] = true;
      s.failed = true;
      return set_error(cudaGetErrorString(cudaGetLastError()));
    }
    s.jobs.push_back({piece, (float*)((char*)dst + at), n});
    s.in_flight++;
    s.wake_one();
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

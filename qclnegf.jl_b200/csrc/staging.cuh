// Transfers between pageable host arrays and the device through pinned
// buffers filled and emptied by several host threads.
//
// A copy from or to pageable memory goes through the driver's own pinned
// buffer on the calling thread: one core's copy and, for a fresh result array,
// its page faults, at 4 GB/s both ways together where the link carries 48 GB/s
// each way.  Here the threads of a CopyTeam share that work.
#pragma once
#include <atomic>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

#include "kernels.cuh"

namespace qcl {

// A 2D copy between host buffers: `rows` runs of `width` bytes.
struct CopyPiece {
  char* dst;
  const char* src;
  size_t dpitch, spitch, width, rows;
};

// Threads that copy lists of pieces together with the caller.  Lives for one
// call; without threads (none could be started) the caller copies alone.
// Between lists a thread sleeps after a short spin (other processes of the host
// have a use for its core), and one that wakes late is not waited for.
class CopyTeam {
 public:
  explicit CopyTeam(int threads);
  ~CopyTeam();
  CopyTeam(const CopyTeam&) = delete;
  CopyTeam& operator=(const CopyTeam&) = delete;
  void copy(const std::vector<CopyPiece>& pieces);  // returns when all are done

 private:
  struct Unit {
    size_t piece, first, count;  // rows of a piece
  };
  void work();
  std::vector<std::thread> threads_;
  const std::vector<CopyPiece>* pieces_ = nullptr;
  std::vector<Unit> units_;
  std::mutex m_;
  std::condition_variable start_, done_;
  // written under m_; atomic for the spins
  std::atomic<unsigned> round_{0};  // of the current list
  std::atomic<int> active_{0};      // threads that take part in it
  std::atomic<bool> stop_{false};
  bool open_ = false;               // the list may still be joined
  std::atomic<size_t> next_{0};
};

// Host threads worth using for `bytes` (0: leave the copy to the driver).
int copy_threads(size_t bytes);
// What p points to.
enum HostKind { HOST_PAGEABLE, HOST_PINNED, HOST_NOT };
HostKind host_kind(const void* p);

}  // namespace qcl

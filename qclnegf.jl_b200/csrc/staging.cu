#include "staging.cuh"

#include <sched.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <exception>

namespace qcl {

constexpr size_t kUnitBytes = (size_t)256 << 10;
constexpr int kSpins = 2000;  // yields before a wait sleeps: longer than the gaps between slabs

// Cores that this process may use: its affinity and its CPU quota.
static int usable_cores() {
  cpu_set_t set;
  int n = sched_getaffinity(0, sizeof(set), &set) == 0 ? CPU_COUNT(&set) : (int)std::thread::hardware_concurrency();
  if (FILE* f = fopen("/sys/fs/cgroup/cpu.max", "r")) {
    double quota, period;
    if (fscanf(f, "%lf %lf", &quota, &period) == 2 && period > 0) n = std::min(n, std::max(1, (int)(quota / period)));
    fclose(f);
  }
  return n;
}

int copy_threads(size_t bytes) {
  // Below 8 MB starting threads costs what they save.
  if (bytes < ((size_t)8 << 20)) return 0;
  return std::min(std::max(usable_cores() - 1, 0), 11);
}

HostKind host_kind(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return HOST_NOT;
  }
  return a.type == cudaMemoryTypeUnregistered ? HOST_PAGEABLE : a.type == cudaMemoryTypeHost ? HOST_PINNED : HOST_NOT;
}

CopyTeam::CopyTeam(int threads) {
  try {
    threads_.reserve(threads > 0 ? threads : 0);
    for (int i = 0; i < threads; ++i)
      threads_.emplace_back([this] {
        for (unsigned seen = 0;;) {
          for (int q = 0; q < kSpins && round_ == seen && !stop_; ++q) std::this_thread::yield();
          std::unique_lock<std::mutex> lock(m_);
          start_.wait(lock, [&] { return stop_ || round_ != seen; });
          if (stop_) return;
          seen = round_;
          if (!open_) continue;
          ++active_;
          lock.unlock();
          work();
          lock.lock();
          if (--active_ == 0) done_.notify_one();
        }
      });
  } catch (const std::exception&) {  // fewer threads, or none
  }
}

CopyTeam::~CopyTeam() {
  {
    std::lock_guard<std::mutex> lock(m_);
    stop_ = true;
  }
  start_.notify_all();
  for (auto& t : threads_) t.join();
}

void CopyTeam::work() {
  for (;;) {
    const size_t i = next_.fetch_add(1, std::memory_order_relaxed);
    if (i >= units_.size()) return;
    const Unit& u = units_[i];
    const CopyPiece& p = (*pieces_)[u.piece];
    for (size_t r = u.first; r < u.first + u.count; ++r) memcpy(p.dst + r * p.dpitch, p.src + r * p.spitch, p.width);
  }
}

void CopyTeam::copy(const std::vector<CopyPiece>& pieces) {
  // contiguous runs are cut, narrow rows grouped, to units of about kUnitBytes
  std::vector<CopyPiece> cut;
  for (const CopyPiece& p : pieces) {
    if (p.width == 0 || p.rows == 0) continue;
    if (p.width <= kUnitBytes) {
      cut.push_back(p);
      continue;
    }
    for (size_t r = 0; r < p.rows; ++r)
      for (size_t o = 0; o < p.width; o += kUnitBytes)
        cut.push_back({p.dst + r * p.dpitch + o, p.src + r * p.spitch + o, 0, 0, std::min(kUnitBytes, p.width - o), 1});
  }
  units_.clear();
  for (size_t i = 0; i < cut.size(); ++i) {
    const size_t per = std::max<size_t>(1, kUnitBytes / cut[i].width);
    for (size_t r = 0; r < cut[i].rows; r += per) units_.push_back({i, r, std::min(per, cut[i].rows - r)});
  }
  pieces_ = &cut;
  next_.store(0, std::memory_order_relaxed);
  if (!threads_.empty()) {
    {
      std::lock_guard<std::mutex> lock(m_);
      open_ = true;
      ++round_;
    }
    start_.notify_all();
  }
  work();
  if (threads_.empty()) return;
  std::unique_lock<std::mutex> lock(m_);
  open_ = false;
  for (int q = 0; q < kSpins && active_ != 0; ++q) {
    lock.unlock();
    std::this_thread::yield();
    lock.lock();
  }
  done_.wait(lock, [&] { return active_ == 0; });
}

}  // namespace qcl

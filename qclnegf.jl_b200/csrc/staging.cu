#include "staging.cuh"

#include <string.h>

#include <algorithm>
#include <system_error>

namespace qcl {

constexpr size_t kUnitBytes = (size_t)256 << 10;

int copy_threads(size_t bytes) {
  // Below 8 MB starting threads costs what they save.
  if (bytes < ((size_t)8 << 20)) return 0;
  const unsigned n = std::thread::hardware_concurrency();
  return (int)std::min(n > 1 ? n - 1 : 0u, 11u);
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
        unsigned seen = 0;
        for (;;) {
          unsigned r;
          while ((r = round_.load(std::memory_order_acquire)) == seen) {
            if (stop_.load(std::memory_order_relaxed)) return;
            std::this_thread::yield();
          }
          seen = r;
          work();
          busy_.fetch_sub(1, std::memory_order_release);
        }
      });
  } catch (const std::system_error&) {  // fewer threads, or none
  }
}

CopyTeam::~CopyTeam() {
  stop_.store(true);
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
  busy_.store((int)threads_.size(), std::memory_order_relaxed);
  round_.fetch_add(1, std::memory_order_release);
  work();
  while (busy_.load(std::memory_order_acquire) != 0) std::this_thread::yield();
}

}  // namespace qcl

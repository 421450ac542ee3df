// prefault.h -- see prefault.cpp.
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <thread>

namespace bvhgb {

// Starts making the pages of `count` buffers present that are about to be overwritten whole; finish() (or the
// destructor) helps and waits.  Buffers of less than kLeast bytes, those already present and memory
// that is not ordinary (page-locked, say) are left alone; contents never change.
class Prefault {
 public:
  Prefault(void* const* ptrs, const size_t* sizes, int count);
  ~Prefault() { finish(); }
  Prefault(const Prefault&) = delete;
  Prefault& operator=(const Prefault&) = delete;
  void finish();

 private:
  static constexpr int kThreads = 4, kMaxPieces = 4;
  static constexpr size_t kLeast = 2u << 20;  // below that the faults cost less than starting threads
  static constexpr size_t kChunk = 1u << 20;
  struct Piece {
    uintptr_t begin, end;
    size_t chunk;
  };
  void work();
  Piece piece_[kMaxPieces];
  int pieces_ = 0;
  std::atomic<size_t> next_[kMaxPieces] = {};
  std::thread workers_[kThreads - 1];
};

}  // namespace bvhgb

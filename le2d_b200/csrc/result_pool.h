// Host memory of a server's results (host logic without CUDA calls; Lock::lock / Lock::unlock
// get and give back page-locked memory).
//
// Reading a result back into fresh pageable memory keeps the worker from launching its next
// window meanwhile; page-locked memory that is used again does not.  But page-locking costs
// about 0.3 ms per MB, and a hundred times that when the host is busy, so none of it may stand
// between two windows: results take and return pieces of one size, which any later result can
// use, and the pool grows only while the worker has nothing to do (grow()), by one slab per
// call.  It grows to what two busy periods in a row held at once, at most kHeld bytes, and is
// given back with the server.  What the pool does not hold is malloc'd and freed with its
// ticket, so a server that is never idle runs as one without a pool.  Measured (FP32): bursts of
// 24 requests of 64 to 1024 nodes a side, 25 MB of fields, 22.5 ms a server's first and 13.3 ms
// once the pool holds them; 48 requests of 64 to 4096 a side at 200 / 1000 a second, ten runs
// each, 53 to 56 / 80 to 82 solves/s, where locking and unlocking blocks between the windows gave
// 40 to 55 / 58 to 80 and no pool at all (with the 64-row tiles of then) 51 / 76.
// Nothing is locked, unlocked or freed under the pool's mutex.
#pragma once

#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

namespace le2d {

template <typename Lock>
class ResultPool {
 public:
  static constexpr size_t kPiece = (size_t)512 << 10, kSlabPieces = 8, kHeld = (size_t)256 << 20;

  ResultPool() = default;
  ResultPool(const ResultPool&) = delete;
  ResultPool& operator=(const ResultPool&) = delete;
  ~ResultPool() {
    for (void* s : slabs_) Lock::unlock(s);
  }

  // `n` pieces, or none when the pool has not that many.
  std::vector<char*> take(size_t n) {
    std::vector<char*> out;
    std::lock_guard<std::mutex> lk(mu_);
    if (n <= kHeld / kPiece) {  // a larger result never fits: it asks for nothing
      asked_ += n;
      if (asked_ > peak_) peak_ = asked_;
    }
    if (n > free_.size()) return out;
    out.assign(free_.end() - n, free_.end());
    free_.resize(free_.size() - n);
    return out;
  }
  // Returns a result's pieces, or (empty) says that a malloc'd result of n pieces is gone.
  void give_back(const std::vector<char*>& pieces, size_t n) {
    std::lock_guard<std::mutex> lk(mu_);
    if (n <= kHeld / kPiece) asked_ -= n;
    free_.insert(free_.end(), pieces.begin(), pieces.end());
  }

  // The worker has nothing to do: a busy period is over.
  void idle() {
    std::lock_guard<std::mutex> lk(mu_);
    if (peak_ == 0) return;
    size_t both = peak_ < last_peak_ ? peak_ : last_peak_;
    if (both > kHeld / kPiece) both = kHeld / kPiece;
    if (both > target_) target_ = both;
    last_peak_ = peak_;
    peak_ = 0;
  }
  bool wants_more() {
    std::lock_guard<std::mutex> lk(mu_);
    return slabs_.size() * kSlabPieces < target_;
  }
  // One more slab (called by one thread, without any lock held).
  void grow() {
    char* s = static_cast<char*>(Lock::lock(kPiece * kSlabPieces));
    std::lock_guard<std::mutex> lk(mu_);
    if (!s) {  // none to be had: no more tries for what was wanted so far
      target_ = 0;
      return;
    }
    slabs_.push_back(s);
    for (size_t k = kSlabPieces; k > 0; --k) free_.push_back(s + (k - 1) * kPiece);
  }

 private:
  std::mutex mu_;
  std::vector<char*> free_;
  std::vector<void*> slabs_;
  size_t asked_ = 0;                  // pieces that the results held now take or would take
  size_t peak_ = 0, last_peak_ = 0;   // the most of them in this busy period and the one before
  size_t target_ = 0;                 // pieces to hold
};

// One result: pieces of the pool (all but the last full), or one malloc'd block.
template <typename Lock>
class PooledResult {
 public:
  using Pool = ResultPool<Lock>;
  PooledResult() = default;
  PooledResult(const PooledResult&) = delete;
  PooledResult& operator=(const PooledResult&) = delete;
  ~PooledResult() {
    free(block_);
    if (pool_) pool_->give_back(pieces_, count_);
  }
  // Memory for `bytes`; false when there is none.  `contiguous`: in one block (a piece or malloc).
  bool make(const std::shared_ptr<Pool>& pool, size_t bytes, bool contiguous) {
    const size_t n = bytes > 0 ? (bytes + Pool::kPiece - 1) / Pool::kPiece : 1;
    if (n == 1 || !contiguous) {
      pool_ = pool;
      count_ = n;
      pieces_ = pool->take(n);
    }
    if (pieces_.empty() && !(block_ = static_cast<char*>(malloc(bytes > 0 ? bytes : 1)))) return false;
    bytes_ = bytes;
    return true;
  }
  size_t bytes() const { return bytes_; }
  // The memory in order, as (address, bytes); a piece each, since a copy must not span two slabs.
  std::vector<std::pair<char*, size_t>> parts() const {
    std::vector<std::pair<char*, size_t>> out;
    if (pieces_.empty()) {
      if (bytes_) out.push_back({block_, bytes_});
      return out;
    }
    size_t left = bytes_;
    for (size_t k = 0; k < pieces_.size() && left > 0; ++k) {
      const size_t n = left < Pool::kPiece ? left : Pool::kPiece;
      out.push_back({pieces_[k], n});
      left -= n;
    }
    return out;
  }
  void copy_to(void* dst) const {
    char* to = static_cast<char*>(dst);
    for (const auto& p : parts()) {
      memcpy(to, p.first, p.second);
      to += p.second;
    }
  }

 private:
  std::shared_ptr<Pool> pool_;
  std::vector<char*> pieces_;
  char* block_ = nullptr;
  size_t count_ = 0, bytes_ = 0;
};

}  // namespace le2d

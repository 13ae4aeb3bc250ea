// eddy_pool.h -- host memory for the sets' kept outputs (networks, likelihoods,
// edge lists).
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>

#include <algorithm>
#include <vector>

namespace eddy {

// Chunks that the batches' packed outputs are copied into, as they are, and
// that hold them until clear().  The first kPinnedBytes of a pool are
// page-locked (Pinned::alloc, null when there is none; Pinned::release), which
// the copies run fastest into; what a context keeps beyond them, or where
// page-locked memory has run out, is ordinary memory.  clear() keeps one
// page-locked chunk at most, as large as all of them were, so a context's
// later sets find room and a large run gives its memory back.
template <class Pinned>
class ChunkPool {
 public:
  static constexpr size_t kPinnedBytes = (size_t)256 << 20;
  static constexpr size_t kMinChunk = (size_t)64 << 10;

  ChunkPool() = default;
  ChunkPool(const ChunkPool &) = delete;
  ChunkPool &operator=(const ChunkPool &) = delete;
  ~ChunkPool() { release(); }

  // room for `bytes` (null: no memory)
  uint8_t *take(size_t bytes) {
    bytes = (bytes + 255) & ~(size_t)255;
    if (chunks_.empty() || used_ + bytes > chunks_.back().n) {
      // (a chunk that holds nothing and is too small makes way)
      if (!chunks_.empty() && used_ == 0) {
        drop(chunks_.size() - 1);
        used_ = chunks_.empty() ? 0 : chunks_.back().n;
      }
      const size_t want = std::max(bytes, kMinChunk);
      if (!add(pinned_ + grow_ <= kPinnedBytes ? std::max(want, grow_) : want) && !add(bytes))
        return nullptr;
      used_ = 0;
    }
    uint8_t *p = chunks_.back().p + used_;
    used_ += bytes;
    return p;
  }

  // What is taken after mark() can be given back at once: rewind() keeps one
  // of the chunks added since, the last one, for the next.
  struct Mark {
    size_t chunks, used;  // chunks that hold something, bytes of the last one
  };
  Mark mark() const {
    const bool empty = !chunks_.empty() && used_ == 0;
    return {chunks_.size() - (empty ? 1 : 0), used_};
  }
  void rewind(const Mark &m) {
    if (chunks_.size() <= m.chunks) {
      used_ = m.used;
      return;
    }
    while (chunks_.size() > m.chunks + 1) drop(chunks_.size() - 2);
    used_ = 0;
  }

  void clear() {
    grow_ = std::min(pinned_, kPinnedBytes);
    if (chunks_.size() != 1 || !chunks_[0].pinned) release();
    used_ = 0;
  }
  void release() {
    while (!chunks_.empty()) drop(chunks_.size() - 1);
    used_ = 0;
  }

 private:
  struct Chunk {
    uint8_t *p;
    size_t n;
    bool pinned;
  };
  bool add(size_t n) {
    Chunk c{nullptr, n, false};
    if (pinned_ + n <= kPinnedBytes) {
      c.p = (uint8_t *)Pinned::alloc(n);
      c.pinned = c.p != nullptr;
    }
    if (!c.p) c.p = (uint8_t *)malloc(n);
    if (!c.p) return false;
    if (c.pinned) pinned_ += n;
    chunks_.push_back(c);
    return true;
  }
  void drop(size_t i) {
    const Chunk c = chunks_[i];
    chunks_.erase(chunks_.begin() + (ptrdiff_t)i);
    if (c.pinned) {
      pinned_ -= c.n;
      Pinned::release(c.p);
    } else {
      free(c.p);
    }
  }
  std::vector<Chunk> chunks_;
  size_t used_ = 0, grow_ = 0, pinned_ = 0;
};

}  // namespace eddy

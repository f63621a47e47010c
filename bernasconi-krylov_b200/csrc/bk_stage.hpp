// Host memory of a call's uploads, kept warm between calls.
//
// Pageable: a small copy from it is staged at once, and pinning memory costs milliseconds
// per context. Whether an asynchronous copy has read its pageable source when it returns is
// the driver's choice, and one call can upload twice (a gradient: its forward run, then its
// reverse sweep), so the room is handed out again only when the copies made from it are
// behind: `Fence::mark` follows them on the stream, `Fence::wait` waits for the mark.
// Not initialised: zero-filling touched every page once more.
#pragma once
#include <cstddef>
#include <memory>
#include <new>

namespace bk {

template <class Fence>
class StageRoom {
 public:
  explicit StageRoom(Fence fence = Fence()) : fence_(fence) {}
  // At least `bytes`, or nullptr: no memory, or the copies from it failed.
  char* take(size_t bytes) {
    if (sent_ && !fence_.wait()) return nullptr;
    sent_ = false;
    if (bytes > size_) {
      room_.reset();
      size_ = 0;
      room_.reset(new (std::nothrow) char[bytes]);
      if (!room_) return nullptr;
      size_ = bytes;
    }
    return room_.get();
  }
  // The copies that read what `take` gave have been enqueued.
  bool sent() {
    sent_ = true;
    return fence_.mark();
  }
  Fence& fence() { return fence_; }

 private:
  Fence fence_;
  std::unique_ptr<char[]> room_;
  size_t size_ = 0;
  bool sent_ = false;
};

}  // namespace bk

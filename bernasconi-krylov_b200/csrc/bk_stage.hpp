// Host memory of a call's uploads, kept warm between calls.
//
// Pageable: a small copy from it is staged at once, and pinning memory costs milliseconds
// per context. Whether an asynchronous copy has read its pageable source when it returns is
// the driver's choice, so the room is handed out again only when the copies made from it are
// behind: the caller says `settled` where it has waited for the stream anyway, and a `take`
// that finds them unsettled (a call that ended in an error) waits with `Fence::wait`. A call
// with two uploads before its first wait (a gradient) has a room for each: an event behind
// every upload cost each call a microsecond. Not initialised: zero-filling touched every
// page once more.
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
    sent_ = true;  // until settled: copies from it may be on their way
    if (bytes > size_) {
      room_.reset();
      size_ = 0;
      room_.reset(new (std::nothrow) char[bytes]);
      if (!room_) return nullptr;
      size_ = bytes;
    }
    return room_.get();
  }
  // The stream has been waited for since the last `take`.
  void settled() { sent_ = false; }
  Fence& fence() { return fence_; }

 private:
  Fence fence_;
  std::unique_ptr<char[]> room_;
  size_t size_ = 0;
  bool sent_ = false;
};

}  // namespace bk

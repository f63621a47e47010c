// The staging room (csrc/bk_stage.hpp) against a copy engine that reads its source late, as
// an asynchronous copy from pageable memory may.
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "bk_stage.hpp"

struct Engine {
  struct Copy {
    const char* src;
    size_t bytes;
    std::string* dst;
  };
  std::vector<Copy> queue;
  int waits = 0;
  void copy(const char* src, size_t bytes, std::string* dst) { queue.push_back({src, bytes, dst}); }
  void run() {
    for (auto& c : queue) c.dst->assign(c.src, c.bytes);
    queue.clear();
  }
};
struct LateFence {
  Engine* e = nullptr;
  bool wait() {
    ++e->waits;
    e->run();
    return true;
  }
};

static int failures = 0;
#define CHECK(x)                                       \
  do {                                                 \
    if (!(x)) {                                        \
      std::printf("line %d: %s\n", __LINE__, #x);      \
      ++failures;                                      \
    }                                                  \
  } while (0)

int main() {
  Engine e;
  bk::StageRoom<LateFence> room(LateFence{&e});
  std::string a, b, c;
  // two uploads before anybody waits for the stream: same size, then a larger one (a new room)
  char* p = room.take(64);
  std::memset(p, 'a', 64);
  e.copy(p, 64, &a);
  p = room.take(64);
  std::memset(p, 'b', 64);
  e.copy(p, 64, &b);
  p = room.take(1 << 20);
  std::memset(p, 'c', 1 << 20);
  e.copy(p, 1 << 20, &c);
  e.run();
  CHECK(a == std::string(64, 'a'));
  CHECK(b == std::string(64, 'b'));
  CHECK(c == std::string(1 << 20, 'c'));
  CHECK(e.waits == 2);
  // settled by the caller: nothing to wait for, and the room stays where it is
  room.settled();
  p = room.take(10);
  room.settled();
  CHECK(room.take(1 << 20) == p && e.waits == 2);
  room.settled();
  // a request no machine can meet is an answer, not an exception
  CHECK(room.take(~(size_t)0 >> 2) == nullptr);
  CHECK(room.take(16) != nullptr);
  return failures;
}

// mv_host.cu -- copies of result arrays into a program's own memory, on several threads.
//
// A build's host result stays in the context's pinned arena until its next build, so a
// program that keeps it copies it, widening indices to its own types on the way.  What
// bounds such a copy is the first touch of the destination (a page fault per page, on one
// thread about 5 GB/s); the pages are therefore touched by several threads.  200 MB of a
// 64^3 build: 44 ms in one thread (numpy), 7 ms here on a machine with 16 processors.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

#include "../../include/mvgpu.h"

namespace {

constexpr int64_t BLOCK = 1 << 16;  // elements a thread takes at a time

int src_size(int kind) { return kind == MV_COPY_8 ? 8 : (kind == MV_COPY_U8_TO_I32 || kind == MV_COPY_1 ? 1 : 4); }
int dst_size(int kind) { return kind == MV_COPY_8 || kind == MV_COPY_I32_TO_I64 ? 8 : (kind == MV_COPY_1 ? 1 : 4); }

void copy_block(const mv_copy& c, int64_t first, int64_t n) {
  const char* s = static_cast<const char*>(c.src) + first * src_size(c.kind);
  char* d = static_cast<char*>(c.dst) + first * dst_size(c.kind);
  if (c.kind == MV_COPY_I32_TO_I64) {
    const int32_t* a = reinterpret_cast<const int32_t*>(s);
    int64_t* b = reinterpret_cast<int64_t*>(d);
    for (int64_t i = 0; i < n; i++) b[i] = a[i];
  } else if (c.kind == MV_COPY_U8_TO_I32) {
    const uint8_t* a = reinterpret_cast<const uint8_t*>(s);
    int32_t* b = reinterpret_cast<int32_t*>(d);
    for (int64_t i = 0; i < n; i++) b[i] = a[i];
  } else {
    std::memcpy(d, s, (size_t)n * dst_size(c.kind));
  }
}

}  // namespace

extern "C" int mv_copy_arrays(const mv_copy* copies, int count) {
  if (count < 0 || (count > 0 && !copies)) return MV_ERR_ARG;
  int64_t bytes = 0, blocks = 0;
  for (int i = 0; i < count; i++) {
    const mv_copy& c = copies[i];
    if (c.kind < MV_COPY_1 || c.kind > MV_COPY_U8_TO_I32 || c.count < 0 || (c.count > 0 && (!c.src || !c.dst)))
      return MV_ERR_ARG;
    bytes += c.count * dst_size(c.kind);
    blocks += (c.count + BLOCK - 1) / BLOCK;
  }
  std::atomic<int64_t> next{0};
  auto work = [&]() {
    int i = 0;
    int64_t first = 0;  // number of copies[i]'s first block
    for (;;) {
      const int64_t b = next.fetch_add(1, std::memory_order_relaxed);
      if (b >= blocks) return;
      for (;; i++) {
        const int64_t mine = (copies[i].count + BLOCK - 1) / BLOCK;
        if (b < first + mine) break;
        first += mine;
      }
      const int64_t at = (b - first) * BLOCK;
      copy_block(copies[i], at, std::min(BLOCK, copies[i].count - at));
    }
  };
  // a thread per 2 MB (starting one costs about 30 us, as long as it takes to copy 0.2 MB),
  // at most 16 and the machine's number
  const int64_t most = std::min<int64_t>(16, std::max(1u, std::thread::hardware_concurrency()));
  const int64_t threads = std::min(most, bytes >> 21);
  std::vector<std::thread> pool;
  try {
    pool.reserve((size_t)std::max<int64_t>(threads, 1));
    for (int64_t t = 1; t < threads; t++) pool.emplace_back(work);
  } catch (const std::exception&) {
    // fewer threads than wanted: the rest of the blocks falls to those that run
  }
  work();
  for (std::thread& t : pool) t.join();
  return MV_OK;
}

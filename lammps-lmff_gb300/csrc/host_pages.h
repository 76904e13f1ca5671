// Host memory of the callers' output arrays: copies by several threads, and pages mapped ahead
// of the GPU's copies.
#pragma once

#include <stdint.h>
#include <string.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <exception>
#include <memory>
#include <new>
#include <thread>

namespace lmff {

// f(begin, end) over [0, bytes): from 4 MiB on in up to 8 pieces, each on its host thread.
// A piece whose thread cannot be had is done here.
template <class F>
void in_pieces(size_t bytes, const F &f) {
  const int nth = (int)std::min<size_t>(8, std::max(1u, std::thread::hardware_concurrency()));
  if (nth <= 1 || bytes < ((size_t)4 << 20)) {
    f((size_t)0, bytes);
    return;
  }
  const size_t piece = ((bytes / nth) + 63) & ~(size_t)63;
  std::thread pool[8];
  for (int k = 0; k < nth; k++) {
    const size_t b = (size_t)k * piece;
    if (b >= bytes) break;
    const size_t e = std::min(bytes, b + piece);
    try {
      pool[k] = std::thread([=, &f] { f(b, e); });
    } catch (const std::exception &) {
      f(b, e);
    }
  }
  for (auto &t : pool)
    if (t.joinable()) t.join();
}

// memcpy on up to 8 host threads, in 64-byte aligned pieces
inline void parallel_copy(void *dst, const void *src, size_t bytes) {
  in_pieces(bytes, [=](size_t b, size_t e) { memcpy((char *)dst + b, (const char *)src + b, e - b); });
}

// Maps the pages of a caller's output array that the call overwrites as a whole.  An array
// the program has just allocated has no pages yet; the GPU's copy into it then takes a fault
// of ~40 us for every 64 KB (490k atoms, lmff_download: 20-30 ms, with its pages there 0.9
// ms), where the host takes a few us, on several threads at once and, where a call's kernels
// are already queued, while they run.
// keep: the call may yet fail, and the array's contents stay as they are (a page of a file, or
// one swapped out, has some): the pages are populated as a write would, without one, 1 MB at a
// time so that the threads' own stacks can be mapped in between.  Otherwise a byte of each
// is written, which is faster (490k atoms, lmff_download: 52.6 against 53.2 ms with its 40
// steps).  (Reading that byte first maps the zero page, and replacing that is a second fault
// with a flush of every thread's translations, 70 ms for 2.7M atoms.)
inline void map_pages(void *p, size_t bytes, bool keep) {
  if (!p || !bytes) return;
  static const size_t page = (size_t)std::max(4096L, sysconf(_SC_PAGESIZE));
  const uintptr_t p0 = (uintptr_t)p / page * page, p1 = ((uintptr_t)p + bytes + page - 1) / page * page;
  const size_t pages = (p1 - p0) / page;
  const std::unique_ptr<unsigned char[]> in(new (std::nothrow) unsigned char[pages]);
  const unsigned char *there = in.get();
  if (!in || mincore((void *)p0, p1 - p0, in.get()) != 0) return;
  if (std::all_of(there, there + pages, [](unsigned char c) { return c & 1; })) return;
  if (!keep) {
    in_pieces(bytes, [=](size_t b, size_t e) {
      for (size_t q = b; q < e; q = ((uintptr_t)p + q) / page * page + page - (uintptr_t)p)
        if (!(there[((uintptr_t)p + q - p0) / page] & 1)) *((volatile char *)p + q) = 0;
    });
    return;
  }
#ifdef MADV_POPULATE_WRITE
  in_pieces(p1 - p0, [=](size_t b, size_t e) {
    const size_t step = std::max((size_t)1 << 20, page);
    b = b / page * page;
    e = e == p1 - p0 ? e : e / page * page;
    for (; b < e; b += step) madvise((void *)(p0 + b), std::min(step, e - b), MADV_POPULATE_WRITE);
  });
#endif
}

}  // namespace lmff

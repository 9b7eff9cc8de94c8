// How a download to pageable memory is shared (download_rows in engine.cu): threads, page-locked buffers and chunks.
#pragma once

#include <cstddef>

namespace b2 {

constexpr int DL_WORKERS = 12;  // threads at most, and buffers
constexpr size_t DL_CHUNK = 128 << 10, DL_LARGE_CHUNK = 512 << 10;
constexpr size_t DL_MIN_BYTES = 2 << 20, DL_MANY_BYTES = 12 << 20, DL_LARGE_BYTES = 32 << 20;
constexpr size_t DL_LARGE_AFTER = (size_t)256 << 20;

// A matrix of up to 2.5 MB comes over in one copy into page-locked memory made with the handle (making any takes 1 to 4 ms
// whatever its size up to here, so it is one block with the words that blocking calls read) and goes on to its place from there: in
// one thread up to 1.5 MB, whose destination gets its pages meanwhile, else in six, which take the faults as they go (asking
// for pages holds the others up). us per matrix into fresh memory, against the driver's copy or the chunks below: 128 KB 67 -> 22,
// 512 KB 110 -> 58, 1 MB 350 -> 200, 2 MB 540 -> 245 (1 MB into pages that are there: 96 and 104). At 4 MB it gains nothing (515, 505) and making the block takes 2 ms longer.
constexpr size_t DL_LANDING_BYTES = 5 << 19, DL_PIECE = 128 << 10;
inline int landing_threads(size_t bytes, int cores) {
  const int threads = bytes < 3 << 19 ? 1 : 6;
  return threads < cores ? threads : cores > 1 ? cores : 1;
}

// Page-locked buffers of a handle for larger ones, DL_WORKERS chunks.
struct DownloadBuffers {
  char* at = nullptr;
  size_t bytes = 0;
  size_t large_read = 0;  // bytes of the matrices of DL_LARGE_BYTES and more read so far
  bool no_large = false;  // there was no memory for the larger chunks: not asked for again
};

struct DownloadPlan {
  int threads;   // 0: one plain copy
  int bufs;      // buffers of each
  size_t chunk;  // bytes of a buffer
};

// A chunk costs about 8 us whatever its size, starting a thread 10 us. So a few MB get six threads with two buffers of 128 KB
// each (one copied to while the other is emptied), and from 12 MB on twelve threads share the same 1.5 MB, one buffer each
// (us per matrix into fresh memory: 3072 x 3072 3490 -> 3040, 4096 x 4096 6050 -> 5150). Fewer than twelve cores run a thread
// each, six at most, with two buffers: 2048 x 2048 and 4096 x 4096 on eight cores 1110 and 6000, as eight threads with one
// buffer each 1160 and 6400; on four 1080 and 7100 (twelve threads 1300 and 8300), on two 1250 and 9600 (2200 and 12400).
// Chunks of 512 KB from 32 MB on are faster still (3040 -> 2250, 5150 -> 3850, 8192 x 8192 19000 -> 12800), but their 6 MB of
// page-locked memory take 3 to 9 ms to make and 1.3 to give back. That is gained over some 256 MB, so they are made with the
// matrix that makes it as much for a handle.
inline DownloadPlan plan_download(size_t width, size_t rows, int cores, const DownloadBuffers& b) {
  const size_t total = width * rows;
  const bool large = total >= DL_LARGE_BYTES && b.large_read + total >= DL_LARGE_AFTER && !b.no_large;
  DownloadPlan p{0, 0, large ? DL_LARGE_CHUNK : DL_CHUNK};
  if (total < DL_MIN_BYTES || width > p.chunk) return p;
  const size_t per = p.chunk / width, chunks = (rows + per - 1) / per;
  p.threads = total >= DL_MANY_BYTES && cores >= DL_WORKERS ? DL_WORKERS : DL_WORKERS / 2;
  if (p.threads > cores) p.threads = cores > 1 ? cores : 1;
  if ((size_t)p.threads > chunks) p.threads = (int)chunks;
  p.bufs = p.threads <= DL_WORKERS / 2 ? 2 : 1;
  return p;
}

// The plan of a download with its buffers made: without memory for larger chunks the ones that are there serve, without
// memory for any the plain copy. `alloc(bytes)` returns null when there is none.
template <class Alloc, class Free>
DownloadPlan ready_download(size_t width, size_t rows, int cores, DownloadBuffers& b, Alloc alloc, Free release) {
  for (;;) {
    DownloadPlan p = plan_download(width, rows, cores, b);
    const size_t need = DL_WORKERS * p.chunk;
    if (p.threads > 0 && b.bytes < need) {
      char* fresh = alloc(need);
      if (!fresh && p.chunk == DL_LARGE_CHUNK) {
        b.no_large = true;
        continue;
      }
      if (fresh) {
        if (b.at) release(b.at);
        b.at = fresh;
        b.bytes = need;
      } else {
        p.threads = 0;
      }
    }
    if (width * rows >= DL_LARGE_BYTES && b.large_read < DL_LARGE_AFTER) b.large_read += width * rows;
    return p;
  }
}

}  // namespace b2
